"""GPU parity of the epsilon-div-div apply against the oracle.

Bar: FP64 within 1e-12 relative (max norm) of the oracle's reference slow path
(element matrices); FP32 within 2e-5 relative of the FP64 oracle.
"""
import numpy as np
import pytest

import oracle as O
import terra_b200 as T
from helpers import BC_COMBOS, consistent, rel_err, smooth_viscosity

pytestmark = pytest.mark.gpu

TOL64 = 1e-12
TOL32 = 2e-5


def _setup(level, seed=0):
    sh = O.Shell(level)
    k = smooth_viscosity(sh, seed, contrast=100.0)
    u = consistent(sh, O.seeded_normal(sh.vec_shape, seed + 1))
    return sh, k, u


@pytest.mark.parametrize("level", [2, 3, 4])
@pytest.mark.parametrize("bcs", BC_COMBOS)
def test_apply_f64_matches_oracle(cuda, level, bcs):
    import torch

    sh, k, u = _setup(level, seed=level)
    ref = O.EpsDivDiv(sh, k=k, bc_cmb=bcs[0], bc_surface=bcs[1]).apply(u, path="slow")
    gsh = T.Shell(level)
    op = T.EpsDivDiv(gsh, k=torch.tensor(k, device=cuda), bc_cmb=bcs[0], bc_surface=bcs[1])
    src = torch.tensor(u, device=cuda)
    dst = torch.full_like(src, float("nan"))
    op.apply(src, dst)
    torch.cuda.synchronize()
    assert gsh.check_device_error() == 0
    assert rel_err(dst.cpu().numpy(), ref) < TOL64


@pytest.mark.parametrize("level", [2, 4])
@pytest.mark.parametrize("bcs", BC_COMBOS)
def test_diagonal_f64_matches_oracle(cuda, level, bcs):
    import torch

    sh, k, u = _setup(level, seed=10 + level)
    ref = O.EpsDivDiv(sh, k=k, bc_cmb=bcs[0], bc_surface=bcs[1]).apply(u, path="slow", diagonal=True)
    gsh = T.Shell(level)
    op = T.EpsDivDiv(gsh, k=torch.tensor(k, device=cuda), bc_cmb=bcs[0], bc_surface=bcs[1], diagonal=True)
    dst = torch.zeros((3,) + sh.scalar_shape, dtype=torch.float64, device=cuda)
    op.apply(torch.tensor(u, device=cuda), dst)
    assert rel_err(dst.cpu().numpy(), ref) < TOL64


@pytest.mark.parametrize("bcs", [(1, 1), (1, 2)])
def test_q0_coefficient(cuda, bcs):
    import torch

    level = 3
    sh = O.Shell(level)
    kq = np.exp(np.random.default_rng(5).uniform(0, np.log(1e4), sh.cell_shape))
    u = consistent(sh, O.seeded_normal(sh.vec_shape, 6))
    ref = O.EpsDivDiv(sh, k_q0=kq, bc_cmb=bcs[0], bc_surface=bcs[1]).apply(u, path="slow")
    gsh = T.Shell(level)
    op = T.EpsDivDiv(gsh, k_cell=torch.tensor(kq, device=cuda), bc_cmb=bcs[0], bc_surface=bcs[1])
    dst = torch.zeros((3,) + sh.scalar_shape, dtype=torch.float64, device=cuda)
    op.apply(torch.tensor(u, device=cuda), dst)
    assert rel_err(dst.cpu().numpy(), ref) < TOL64


def test_modes_add_and_skip_communication(cuda):
    """Replace+Skip leaves per-diamond partial sums; Add accumulates; the
    interface sum of the partial result equals the communicated apply."""
    import torch

    level = 3
    sh, k, u = _setup(level, seed=21)
    gsh = T.Shell(level)
    op = T.EpsDivDiv(gsh, k=torch.tensor(k, device=cuda))
    src = torch.tensor(u, device=cuda)
    full = torch.zeros_like(src)
    op.apply(src, full)
    op.set_modes(T.REPLACE, T.SKIP_COMMUNICATION)
    part = torch.zeros_like(src)
    op.apply(src, part)
    ref_part = O.EpsDivDiv(sh, k=k).apply(u, path="slow", comm=False)
    assert rel_err(part.cpu().numpy(), ref_part) < TOL64
    gsh.interface_sum(part)
    assert rel_err(part.cpu().numpy(), full.cpu().numpy()) < 1e-14
    op.set_modes(T.ADD, T.SKIP_COMMUNICATION)
    acc = torch.tensor(u, device=cuda)
    op.apply(src, acc)
    assert rel_err(acc.cpu().numpy(), u + ref_part) < TOL64


@pytest.mark.parametrize("tile", [(1, 1), (2, 3), (3, 5), (7, 9), (5, 64)])
def test_tile_shapes(cuda, tile):
    import torch

    level = 4
    sh, k, u = _setup(level, seed=31)
    ref = O.EpsDivDiv(sh, k=k, bc_cmb=1, bc_surface=2).apply(u, path="fast")
    gsh = T.Shell(level)
    op = T.EpsDivDiv(gsh, k=torch.tensor(k, device=cuda), bc_cmb=1, bc_surface=2)
    op.set_tile(*tile)
    dst = torch.zeros((3,) + sh.scalar_shape, dtype=torch.float64, device=cuda)
    op.apply(torch.tensor(u, device=cuda), dst)
    assert rel_err(dst.cpu().numpy(), ref) < TOL64


@pytest.mark.parametrize("level", [5, 6])
def test_large_levels_f64(cuda, level):
    """Two and one radial cells per lane (levels 5/6) against the oracle fast path."""
    import torch

    sh, k, u = _setup(level, seed=41)
    ref = O.EpsDivDiv(sh, k=k, bc_cmb=1, bc_surface=2).apply(u, path="fast")
    gsh = T.Shell(level)
    op = T.EpsDivDiv(gsh, k=torch.tensor(k, device=cuda), bc_cmb=1, bc_surface=2)
    dst = torch.zeros((3,) + sh.scalar_shape, dtype=torch.float64, device=cuda)
    op.apply(torch.tensor(u, device=cuda), dst)
    assert rel_err(dst.cpu().numpy(), ref) < TOL64


@pytest.mark.parametrize("level", [3, 5, 6])
@pytest.mark.parametrize("bcs", [(1, 1), (1, 2)])
def test_apply_f32(cuda, level, bcs):
    import torch

    sh, k, u = _setup(level, seed=51)
    ref = O.EpsDivDiv(sh, k=k, bc_cmb=bcs[0], bc_surface=bcs[1]).apply(u, path="fast")
    gsh = T.Shell(level)
    op = T.EpsDivDiv(gsh, k=torch.tensor(k, dtype=torch.float32, device=cuda), bc_cmb=bcs[0], bc_surface=bcs[1])
    dst = torch.zeros((3,) + sh.scalar_shape, dtype=torch.float32, device=cuda)
    op.apply(torch.tensor(u, dtype=torch.float32, device=cuda), dst)
    assert rel_err(dst.cpu().numpy(), ref) < TOL32


def test_level7_consistency(cuda):
    """Four radial cells per lane (level 7): FP32 vs FP64 agreement and symmetry."""
    import torch

    level = 7
    gsh = T.Shell(level)
    nl, nr = gsh.dims()
    g = torch.Generator(device=cuda).manual_seed(3)
    k = torch.exp(0.3 * torch.randn((10, nl, nl, nr), generator=g, device=cuda, dtype=torch.float64))
    u = torch.randn((3, 10, nl, nl, nr), generator=g, device=cuda, dtype=torch.float64)
    v = torch.randn((3, 10, nl, nl, nr), generator=g, device=cuda, dtype=torch.float64)
    gsh.interface_sum(u)  # any assembled vectors will do
    gsh.interface_sum(v)
    op = T.EpsDivDiv(gsh, k=k)
    Au, Av = torch.zeros_like(u), torch.zeros_like(v)
    op.apply(u, Au)
    op.apply(v, Av)
    a, b = gsh.dot(v, Au), gsh.dot(u, Av)
    assert abs(a - b) <= 1e-10 * abs(a)
    op32 = T.EpsDivDiv(gsh, k=k.float())
    Au32 = torch.zeros_like(u, dtype=torch.float32)
    op32.apply(u.float(), Au32)
    assert rel_err(Au32.double().cpu().numpy(), Au.cpu().numpy()) < 1e-4


@pytest.mark.parametrize("level", [2, 4, 6])
def test_apply_is_deterministic(cuda, level):
    """No atomics: repeated applies are bitwise identical."""
    import torch

    sh, k, u = _setup(level, seed=61)
    gsh = T.Shell(level)
    op = T.EpsDivDiv(gsh, k=torch.tensor(k, device=cuda), bc_cmb=1, bc_surface=2)
    src = torch.tensor(u, device=cuda)
    first = torch.zeros_like(src)
    op.apply(src, first)
    for _ in range(20):
        again = torch.full_like(src, float("nan"))
        op.apply(src, again)
        assert torch.equal(again, first)


@pytest.mark.parametrize("lat,rad", [(0, 1), (1, 1), (2, 1), (1, 4), (5, 2), (3, 5), (2, 6), (4, 6), (1, 7)])
@pytest.mark.parametrize("bcs", [(1, 2), (2, 1), (0, 0)])
def test_lateral_and_radial_levels(cuda, lat, rad, bcs):
    """Strips that share a warp, fill one or take several, tiles with a single line, and nodal / cell coefficients in
    both precisions, Replace and Add. Tolerances as in the equal-level tests."""
    import torch

    sh = O.Shell(lat, rad)
    rng = np.random.default_rng(100 * lat + 10 * rad + bcs[0])
    X = sh.physical_coords()
    k = np.exp(np.log(10.0) * np.sin(X @ np.array([1.3, -0.7, 2.1])))
    kc = np.exp(rng.uniform(-2.0, 2.0, (10, sh.nl - 1, sh.nl - 1, sh.nr - 1)))
    u = consistent(sh, rng.standard_normal(sh.vec_shape))
    g = T.Shell(lat, rad)
    for q0 in (False, True):
        ref = O.EpsDivDiv(sh, **({"k_q0": kc} if q0 else {"k": k}), bc_cmb=bcs[0], bc_surface=bcs[1]).apply(u)
        for dt, tol in ((torch.float64, TOL64), (torch.float32, TOL32)):
            coef = torch.tensor(kc if q0 else k, dtype=dt, device=cuda)
            op = T.EpsDivDiv(g, **({"k_cell": coef} if q0 else {"k": coef}), bc_cmb=bcs[0], bc_surface=bcs[1])
            src = torch.tensor(u, dtype=dt, device=cuda)
            dst = torch.full_like(src, float("nan"))
            op.apply(src, dst)
            assert rel_err(dst.double().cpu().numpy(), ref) < tol
            op.set_modes(T.ADD, T.SKIP_COMMUNICATION)
            part, acc = torch.zeros_like(src), src.clone()
            op.apply(src, part)
            op.apply(src, acc)
            assert rel_err(acc.double().cpu().numpy(), (src + part).double().cpu().numpy()) < tol


@pytest.mark.parametrize("level", [2, 5])
def test_chained_applies_equal_synchronised(cuda, level):
    """Back-to-back launches overlap at their ends; a chain of dependent applies gives the bits of one that waits."""
    import torch

    g = T.Shell(level)
    nl, nr = g.dims(-1)
    A = T.EpsDivDiv(g, -1, k=torch.ones((10, nl, nl, nr), dtype=torch.float64, device=cuda), bc_cmb=1, bc_surface=2)
    out = []
    for wait in (False, True):
        u = torch.tensor(O.seeded_normal((3, 10, nl, nl, nr), 48), device=cuda)
        v = torch.empty_like(u)
        torch.cuda.synchronize()
        for _ in range(24):
            A.apply(u, v)
            if wait:
                torch.cuda.synchronize()
            u, v = v, u
        torch.cuda.synchronize()
        out.append(u)
    assert torch.isfinite(out[0]).all() and torch.equal(out[0], out[1])


@pytest.mark.parametrize("lat,rad", [(0, 1), (1, 1), (2, 3), (3, 1), (1, 6)])
@pytest.mark.parametrize("bcs", [(0, 0), (1, 2), (2, 2), (2, 0)])
@pytest.mark.parametrize("q0", [False, True])
def test_diagonal_shapes(cuda, lat, rad, bcs, q0):
    """Diagonal mode on levels of two radial layers and many, both coefficients, with and without free-slip nodes (a launch
    of their own), replacing and adding: FP64 1e-12 as above, FP32 1e-5 (sums of 12 terms at 6e-8)."""
    import torch

    sh, gsh = O.Shell(lat, rad), T.Shell(lat, rad)
    rng = np.random.default_rng(lat + 10 * rad)
    k = np.exp(rng.uniform(-1.0, 1.0, sh.cell_shape)) if q0 else smooth_viscosity(sh, 12, 50.0)
    u = O.seeded_normal(sh.vec_shape, 13)
    ref = O.EpsDivDiv(sh, **({"k_q0": k} if q0 else {"k": k}), bc_cmb=bcs[0], bc_surface=bcs[1]).apply(
        u, path="slow", diagonal=True)
    for dt, tol in ((torch.float64, 1e-12), (torch.float32, 1e-5)):
        kt, ut = (torch.tensor(a, dtype=dt, device=cuda) for a in (k, u))
        op = T.EpsDivDiv(gsh, **({"k_cell": kt} if q0 else {"k": kt}), bc_cmb=bcs[0], bc_surface=bcs[1], diagonal=True)
        out = torch.zeros_like(ut)
        op.apply(ut, out)
        assert rel_err(out.double().cpu().numpy(), ref) < tol
        op.set_modes(T.ADD, T.SKIP_COMMUNICATION)
        once = torch.zeros_like(ut)
        op.apply(ut, once)
        twice = once.clone()
        op.apply(ut, twice)
        assert torch.equal(twice, 2 * once)
