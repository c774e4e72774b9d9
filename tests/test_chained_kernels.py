"""Contract of the chained launches (chain_enter in tn_device.cuh), read off the sources: every kernel launched with
launch_chained waits, and the kernel and the device functions it calls read no memory that another kernel of the stream
writes through a path the compiler may take as invariant (__ldg, ld.global.nc, __restrict__), since such a load may move
above the wait. Mesh tables, written once when the mesh is made, may be read that way."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "terra-ng_b200", "csrc")
MESH_TABLES = {"off", "mem", "owned"}


def _functions(text):
    """name -> signature and body of the device functions and kernels of one source."""
    text = re.sub(r"__launch_bounds__\([^()]*(?:\([^()]*\)[^()]*)*\)", "", text)
    out = {}
    for m in re.finditer(r"__(?:global|device)__\s[^;{}()]*?\b(\w+)\s*\(([^;{}]*)\)\s*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        out[m.group(1)] = text[m.start():i]
    return out


def _reachable(name, funcs, seen):
    if name in seen or name not in funcs:
        return seen
    seen.add(name)
    for callee in re.findall(r"\b(\w+)\s*(?:<[^;(){}]*>)?\s*\(", funcs[name]):
        _reachable(callee, funcs, seen)
    return seen


def test_chained_kernels_read_mutable_memory_coherently():
    texts = {f: re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read()) for f in os.listdir(CSRC)
             if f.endswith((".cu", ".cuh"))}
    shared = {}
    for f, t in texts.items():
        if f.endswith(".cuh"):
            shared.update(_functions(t))
    checked = set()
    for f, t in texts.items():
        if not f.endswith(".cu") or "launch_chained(" not in t:
            continue
        funcs = {**shared, **_functions(t)}
        names = {n for n in re.findall(r"\b(\w+_kernel)\b", t) if n in funcs and "chain_enter()" in funcs[n]}
        for arg in re.findall(r"launch_chained\((\w+)", t):  # kernels passed by name; others through a variable
            assert arg in names or arg not in funcs, f"{f}: {arg} is launched chained and does not wait"
        for n in names:
            for g in _reachable(n, funcs, set()):
                body = funcs[g]
                assert ".nc" not in body, f"{f}: {n} reads through {g} (ld.global.nc)"
                for a in re.findall(r"__ldg\(\s*(?:\w+<[^>]*>\()?(\w+)", body):
                    assert a in MESH_TABLES, f"{f}: {n} reads {a} through __ldg in {g}"
                for a in re.findall(r"__restrict__\s+(\w+)", body):
                    assert a in MESH_TABLES, f"{f}: {n} takes {a} as __restrict__ in {g}"
            checked.add(n)
    assert checked >= {"epsdivdiv_kernel", "gca_apply_compact_kernel", "cheb_kernel", "iface_kernel", "restrict_kernel",
                       "prolongate_kernel"}
