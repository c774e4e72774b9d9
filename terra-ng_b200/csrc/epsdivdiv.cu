// epsilon-div-div wedge operator apply for sm_100a (FP64 and FP32).
//
// Semantics follow the reference's EpsilonDivDivKerngen (src/terra/fe/wedge/
// operators/shell/epsilon_divdiv_kerngen.hpp): 1-point centroid quadrature,
// k_eval = mean of the six nodal coefficients (or a per-cell Q0 value),
// Dirichlet rows reduced to their diagonal (:1569-1602), free-slip as
// P A P + diag_nn(A) n n^T on boundary nodes (:1638-2198), and a diagonal mode
// that applies diag(A) (rotated diagonal on free-slip nodes, :2008-2102).
//
// Formulation. The wedge Jacobian factorises as J = M diag(r_mid, r_mid, dr/2)
// with M = [p1-p0, p2-p0, (p0+p1+p2)/3] built from unit-sphere corners only
// (kernel_helpers.hpp:179-258). With M^{-T} = [e1 e2 e3] the physical gradient
// of node (m, side s) is g = alpha L_m + s beta e3, alpha = 1/(2 r_mid),
// beta = 1/(3 dr), L_1 = e1, L_2 = e2, L_0 = -(e1 + e2). With the corner sums
// S = u_top + u_bot and differences D = u_top - u_bot the velocity gradient is
//   G / alpha = e1 (x) (S1 - S0) + e2 (x) (S2 - S0) + e3 (x) rho (D0 + D1 + D2),
// rho = beta / alpha, and the nodal forces are sigma g. Two scalings move out of
// the wedge loop: sqrt|det M| goes into the lateral vectors (g_i = sqrt|det M| e_i,
// a table per level), and alpha^2 r_mid^2 dr/2 = dr/8 goes into the coefficient.
// A wedge is then 65 multiply-adds on nine lateral numbers: symmetric gradient 27,
// stress 11, sigma g_i 27.
//
// Every corner collects a lateral part L = sum sigma g_1,2 and a radial part
// R = sum sigma g_3 over the cells around its node line; only the sums are turned
// into node values, bottom = L - rho R and top = L + rho R. So the lateral sums
// run on six numbers per (node line, radial cell) and the radial neighbours meet
// once per node (three shuffles) instead of once per cell corner (twelve).
//
// Work decomposition:
//   * one cell per lane, lanes along r. A cell strip (fixed y) of nrc radial cells takes nrc / 32 warps ("chunks"), or,
//     below 32 radial cells, several strips share a warp.
//   * a CTA owns ty node lines (ty + 1 strips: the one left of the tile is recomputed) and sweeps x. Sums between strips
//     go through shared memory, one barrier a row; the column behind is kept in registers, inputs (S, D, k) as well as
//     outputs (L, R), so each row is read from shared memory once.
//   * the sweep is flattened over all tiles: CTA b takes rows [b n, (b + 1) n) of the sequence (diamond, tile, x), so all
//     SMs finish together; only the first row of a range repeats a cell column.
//   * two more warps stage: one issues the TMA bulk copies (no multicast) of whole rows and of the strips' geometry into
//     a 6-deep ring, the other applies the input side of the boundary treatment to the two boundary node planes in
//     shared memory, two rows ahead of use, and leaves the output-side record of each boundary node (normal and
//     Ann (n.u), or diag u). So the compute warps treat a boundary node with one add. The diagonals of the boundary
//     rows come from a table built with the operator.
// Every node value is written once by its owner: no atomics, no zeroing pass.
// Diamond-edge duplicates hold this diamond's partial sums afterwards; the interface-sum kernel completes them.
//
// What bounds it: in FP32 issue (0.70 of the slots), in FP64 the wait for the row barrier and for results with 12 warps
// (issue 0.49, FP64 pipe 0.46), both at 510 and 570 thread instructions per cell, half of them floating point. With
// radial sums per cell corner, radial factors and boundary code in every lane and a chunked grid the same apply took
// 820 / 1070 instructions per cell. Measured on the level-6 apply with interface sum (L2 flushed): FP32 115 -> 69 us,
// FP64 199 -> 100 us; level 7, FP64, per-cell coefficient: 1.29 -> 0.71 ms. Tried and slower, same measure: FP32 pairs on
// the packed FP32x2 instructions (12 warps of 152 registers: half the instructions per cell, but 0.48 instead of 0.70
// issue; 71 us), mbarriers between neighbouring warps instead of the row barrier (79 us FP32, 126 us FP64),
// 14 FP64 warps of 128 registers (116 us), 20 FP32 warps of 80 registers (71 us).
#include "tn_device.cuh"
#include "tn_kernels.hpp"
#include "tn_wedge_math.cuh"

#include <algorithm>
#include <atomic>
#include <mutex>
#include <type_traits>

namespace tn {
namespace {

constexpr int kMaxDevices = 64;  // devices a process can drive (per-device launch caches)

// Block shape per precision. FP32: 24 compute warps at 72 registers (six a scheduler). FP64: three warpgroups of
// compute warps and one for staging; launched with 128 registers a thread, the compute warpgroups grow to 152 out of
// what the staging warpgroup gives up (3 x 152 + 56 = 4 x 128, so no more is asked for than the block holds).
template <typename T>
struct Shape;
template <>
struct Shape<double> {
    static constexpr int  kComputeWarps = 12, kThreads = 512, kGeo = 20;
    static constexpr bool kSplit        = true;
    static constexpr int  kComputeRegs = 152, kStageRegs = 56;
    static_assert(3 * kComputeRegs + kStageRegs <= 4 * 128, "register split");
};
template <>
struct Shape<float> {
    static constexpr int  kComputeWarps = 24, kThreads = 896, kGeo = 24;
    static constexpr bool kSplit        = false;
    static constexpr int  kComputeRegs = 72, kStageRegs = 72;
};
constexpr int      kRing      = 6;  // staged rows
constexpr uint32_t kSmemLimit = 227 * 1024;

template <typename T>
struct EddArgs {
    int         nl, nr;
    const T*    geo;     // lateral table [10][nl - 1][nl][kGeo], entry y of a column x is strip y - 1
    const T*    radii;
    const T*    bdiag;   // [2 sides][10 nl nl][8]: diagonal (3), normal stiffness and normal (3) of the boundary nodes
    const T*    k;       // nodal coefficient or nullptr
    const T*    kq0;     // per-cell coefficient or nullptr
    const T*    src[3];
    T*          dst[3];
    int         bc_cmb, bc_surf;
    int         warps;       // compute warps
    int         strips, ty;  // strips of a CTA (slots / nrc) and node lines it owns (<= strips - 1)
    int         ytiles, rows, total_rows;
    int*        err;
};

template <typename T>
struct EddSmem {
    uint32_t bar, off, rec, edge, xch, ring, total;
    uint32_t rowcap, slot, geo;  // bytes of one field of a staged row, of a ring slot and of its geometry
};

template <typename T>
__host__ __device__ inline EddSmem<T> edd_smem(int nr, int warps, int strips)
{
    EddSmem<T>     L;
    constexpr uint32_t t = sizeof(T);
    const uint32_t     nw = static_cast<uint32_t>(warps), ns = static_cast<uint32_t>(strips);
    L.bar    = 0;                                        // row landed, per ring slot
    L.off    = 64;                                       // int4 per ring slot
    L.rec    = L.off + kRing * 16;                       // [slot][column][side][4] T
    L.edge   = L.rec + kRing * (ns + 1) * 8 * t;         // [parity][warp][6] T
    L.xch    = (L.edge + 2 * nw * 6 * t + 15) / 16 * 16;  // [parity][warp][6][32] T
    L.ring   = L.xch + 2 * nw * 6 * 32 * t;
    L.rowcap = ((ns + 1) * static_cast<uint32_t>(nr) * t + 16 + 15) / 16 * 16;
    L.geo    = ns * Shape<T>::kGeo * t;
    L.slot   = L.geo + 4 * L.rowcap;                     // geometry, then 4 fields
    L.total  = L.ring + kRing * L.slot;
    return L;
}

// Position in the ring: slot and the parity of its current use.
struct RingPos {
    uint32_t slot = 0, parity = 0;
    __device__ __forceinline__ void next()
    {
        if (++slot == kRing) {
            slot = 0;
            parity ^= 1u;
        }
    }
};

// One wedge: v1 = sigma g1, v2 = sigma g2, wv = sigma g3 for the lateral differences a, b, the scaled radial
// difference D and the weight kw; g holds the wedge's nine table values.
template <typename T>
__device__ __forceinline__ void wedge_forces(const T (&g)[9], const T (&a)[3], const T (&b)[3], const T (&D)[3], T kw,
                                             T (&v1)[3], T (&v2)[3], T (&wv)[3])
{
    T d[3], h[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) d[i] = fma(g[6 + i], D[i], fma(g[3 + i], b[i], g[i] * a[i]));
#pragma unroll
    for (int k = 0; k < 3; ++k) {  // pairs (0, 1), (0, 2), (1, 2)
        const int i = k == 2 ? 1 : 0, j = k == 0 ? 1 : 2;
        T         t = g[i] * a[j];
        t           = fma(g[j], a[i], t);
        t           = fma(g[3 + i], b[j], t);
        t           = fma(g[3 + j], b[i], t);
        t           = fma(g[6 + i], D[j], t);
        h[k]        = fma(g[6 + j], D[i], t);
    }
    const T k2 = kw + kw;
    const T tr = (T(-1) / T(3)) * k2 * (d[0] + d[1] + d[2]);
    const T s0 = fma(k2, d[0], tr), s1 = fma(k2, d[1], tr), s2 = fma(k2, d[2], tr);
    const T s01 = kw * h[0], s02 = kw * h[1], s12 = kw * h[2];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        T(&o)[3] = m == 0 ? v1 : (m == 1 ? v2 : wv);
        const T x = g[3 * m], y = g[3 * m + 1], z = g[3 * m + 2];
        o[0] = fma(s02, z, fma(s01, y, s0 * x));
        o[1] = fma(s12, z, fma(s1, y, s01 * x));
        o[2] = fma(s2, z, fma(s12, y, s02 * x));
    }
}

// MULTI: several strips share a warp (fewer than 32 radial cells); otherwise a strip takes nrc / 32 warps ("chunks").
template <typename T, bool Q0, bool MULTI, bool ADD>
__global__ void __launch_bounds__(Shape<T>::kThreads, 1) epsdivdiv_kernel(const __grid_constant__ EddArgs<T> A)
{
    using Sh              = Shape<T>;
    constexpr int kGeo    = Sh::kGeo;
    constexpr int kMaxW   = Sh::kComputeWarps;
    constexpr int kIssueWarp = kMaxW, kTreatWarp = kMaxW + 1;
    extern __shared__ __align__(16) unsigned char smem[];
    const int        nl = A.nl, nr = A.nr, nrc = nr - 1;
    const int        lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int        strips = A.strips, ty = A.ty, ytiles = A.ytiles;
    const EddSmem<T> L      = edd_smem<T>(nr, A.warps, strips);
    uint64_t*        landed = reinterpret_cast<uint64_t*>(smem + L.bar);
    int*             off    = reinterpret_cast<int*>(smem + L.off);
    T*               rec    = reinterpret_cast<T*>(smem + L.rec);
    const int        nchunks = MULTI ? 1 : nrc / 32;

    // rows [R0, R1) of the flattened sequence (diamond, tile, x); staged: from one row before (unless the range
    // starts a tile) to one row after (unless it ends one)
    const int R0 = blockIdx.x * A.rows, R1 = min(R0 + A.rows, A.total_rows);
    const int F0 = R0 - (R0 % nl != 0 ? 1 : 0);
    const int F1 = R1 - 1 + ((R1 - 1) % nl < nl - 1 ? 1 : 0);

    if (threadIdx.x == 0) {
        for (int s = 0; s < kRing; ++s) mbar_init(&landed[s], 1);
        fence_barrier_init();
    }
    // strips past the last cell column read their geometry from whatever the slot holds: start it at zero
    for (uint32_t i = threadIdx.x; i < kRing * (L.geo / 4); i += Sh::kThreads) {
        const uint32_t s = i / (L.geo / 4), e = i % (L.geo / 4);
        *reinterpret_cast<uint32_t*>(smem + L.ring + s * L.slot + 4 * e) = 0u;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    chain_enter();

    // One barrier a row for the compute warps and the two staging warps. Barrier B(f) ends the cells of row f: the
    // exchange sums of row f are written, the reads of staged row f are done, row f + 2 has been treated.
    const int  members     = 32 * (A.warps + 2);
    const auto row_barrier = [&] { asm volatile("barrier.sync 1, %0;" ::"r"(members) : "memory"); };

    if (w >= kMaxW) {
        // ------------------------------------------------------------------
        // Staging warps
        // ------------------------------------------------------------------
        if constexpr (Sh::kSplit) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Sh::kStageRegs));
        if (w == kIssueWarp) {
            const T* fields[4] = {A.src[0], A.src[1], A.src[2], A.k};
            int      tile = F0 / nl, x = F0 - tile * nl, d = tile / ytiles, y0 = (tile - d * ytiles) * ty;
            RingPos  pos;
            bool     first_row = true;
            auto     issue = [&] {
                const int     ylo = max(y0 - 1, 0), ncols = min(y0 + strips - 1, nl - 1) - ylo + 1;
                const int64_t e0  = node_index(nl, nr, d, x, ylo, 0);
                // field i into the slot: 16-byte aligned copy around n elements from p; returns the bytes
                const uint32_t first = L.ring + pos.slot * L.slot + L.geo;
                uint32_t       total = 0;
                auto bytes_of = [&](const T* p, int n) {
                    return ((static_cast<uint32_t>(reinterpret_cast<uint64_t>(p)) & 15u) + static_cast<uint32_t>(n * static_cast<int>(sizeof(T))) + 15u) & ~15u;
                };
                // the cell column behind this row: geometry of its strips, and their coefficients (Q0)
                const bool column = x > 0 && !first_row;
                const T*   q0p    = nullptr;
                int        nq     = 0;
                if (Q0 && column) {
                    q0p = A.kq0 + node_index(nl - 1, nrc, d, x - 1, ylo, 0);
                    nq  = (min(y0 + strips - 2, nl - 2) - ylo + 1) * nrc;
                }
                const int ngeo = column ? min(strips, nl - y0) : 0;  // entries y0 .. (entry y is strip y - 1)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const T* p = Q0 && i == 3 ? q0p : fields[i] + e0;
                    const int n = Q0 && i == 3 ? nq : ncols * nr;
                    if (n > 0) total += bytes_of(p, n);
                    off[4 * pos.slot + i] = static_cast<int>(first + i * L.rowcap + (static_cast<uint32_t>(reinterpret_cast<uint64_t>(p)) & 15u));
                }
                total += static_cast<uint32_t>(ngeo * kGeo * static_cast<int>(sizeof(T)));
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                mbar_arrive_expect_tx(&landed[pos.slot], total);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const T* p = Q0 && i == 3 ? q0p : fields[i] + e0;
                    const int n = Q0 && i == 3 ? nq : ncols * nr;
                    if (n > 0)
                        bulk_copy_g2s(smem + first + i * L.rowcap,
                                      reinterpret_cast<const void*>(reinterpret_cast<uint64_t>(p) & ~uint64_t(15)),
                                      bytes_of(p, n), &landed[pos.slot]);
                }
                if (ngeo > 0)
                    bulk_copy_g2s(smem + first - L.geo,
                                  A.geo + ((static_cast<int64_t>(d) * (nl - 1) + (x - 1)) * nl + y0) * kGeo,
                                  static_cast<uint32_t>(ngeo * kGeo * static_cast<int>(sizeof(T))), &landed[pos.slot]);
                first_row = false;
                pos.next();
                if (++x == nl) {
                    x = 0;
                    if (++tile % ytiles == 0) {
                        ++d;
                        y0 = 0;
                    } else {
                        y0 += ty;
                    }
                }
            };
            int next = F0;
            if (lane == 0)
                for (int i = 0; i < kRing && next <= F1; ++i, ++next) issue();
            row_barrier();
            for (int f = F0; f < R1; ++f) {
                // the slot of row f - 1 is free: its last readers have passed B(f - 1)
                if (lane == 0 && f > F0 && next <= F1) {
                    issue();
                    ++next;
                }
                row_barrier();
            }
            return;
        }
        if (w != kTreatWarp) return;
        // Rows in order: wait for the copies and apply the input side of the boundary treatment to the two boundary
        // planes (Dirichlet: input 0, record diag u; free slip: tangential part, record (n, Ann n.u)).
        const bool any_bc = A.bc_cmb != 0 || A.bc_surf != 0;
        int        tile = F0 / nl, x = F0 - tile * nl, d = tile / ytiles, y0 = (tile - d * ytiles) * ty;
        RingPos    pos;
        bool       ok = true;
        auto       treat = [&] {
            const int ylo = max(y0 - 1, 0), ncols = min(y0 + strips - 1, nl - 1) - ylo + 1;
            bool      waited = false;
            for (int i = lane; i - lane < (any_bc ? 2 * ncols : 1); i += 32) {
                const bool on   = any_bc && i < 2 * ncols;
                const int  col  = on ? i >> 1 : 0, side = i & 1;
                const int  bc   = side == 0 ? A.bc_cmb : A.bc_surf;
                T          t[8] = {};  // diagonal, normal stiffness, normal
                if (on && bc != 0) {
                    const T* p = A.bdiag + (static_cast<int64_t>(side) * 10 * nl * nl + lat_index3(nl, d, x, ylo + col)) * 8;
#pragma unroll
                    for (int q = 0; q < 7; ++q) t[q] = p[q];
                }
                if (!waited) {
                    waited = true;
                    if (ok) ok = mbar_wait_bounded(&landed[pos.slot], pos.parity);
                    if (!ok) report_error(A.err, kDevMbarrierTimeout);
                }
                if (!on || bc == 0) continue;
                T* u[3];
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    u[c] = reinterpret_cast<T*>(smem + off[4 * pos.slot + c]) + col * nr + (side == 0 ? 0 : nrc);
                const T u0 = *u[0], u1 = *u[1], u2 = *u[2];
                T*      o  = rec + (pos.slot * static_cast<uint32_t>(strips + 1) + (ylo - (y0 - 1)) + col) * 8 + side * 4;
                if (bc == 1) {
                    o[0] = t[0] * u0, o[1] = t[1] * u1, o[2] = t[2] * u2;
                    *u[0] = T(0), *u[1] = T(0), *u[2] = T(0);
                } else {
                    const T un = t[4] * u0 + t[5] * u1 + t[6] * u2;
                    o[0] = t[4], o[1] = t[5], o[2] = t[6], o[3] = t[3] * un;
                    *u[0] = u0 - un * t[4], *u[1] = u1 - un * t[5], *u[2] = u2 - un * t[6];
                }
            }
            // these writes precede the slot's next copy
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            pos.next();
            if (++x == nl) {
                x = 0;
                if (++tile % ytiles == 0) {
                    ++d;
                    y0 = 0;
                } else {
                    y0 += ty;
                }
            }
        };
        treat();
        if (F1 > F0) treat();
        row_barrier();
        for (int f = F0; f < R1; ++f) {
            if (f + 2 <= F1) treat();
            row_barrier();
        }
        // every copy has landed: all rows were waited for above, or, after a timeout, here
        if (!ok)
            for (int s = 0; s < kRing; ++s) (void)mbar_wait_bounded(&landed[s], 0, 100000000ull);
        return;
    }

    if constexpr (Sh::kSplit) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Sh::kComputeRegs));
    if (w >= A.warps) return;
    // ----------------------------------------------------------------------
    // Compute warps: one cell per lane.
    // ----------------------------------------------------------------------
    T*         xch   = reinterpret_cast<T*>(smem + L.xch);
    T*         edge  = reinterpret_cast<T*>(smem + L.edge);
    const int  chunk = MULTI ? 0 : w % nchunks;
    const int  spw   = MULTI ? 32 / nrc : 1;
    const int  strip = MULTI ? w * spw + lane / nrc : w / nchunks;
    const int  rc    = MULTI ? lane % nrc : chunk * 32 + lane;
    const int  below = MULTI ? max(strip - 1, 0) : 0;
    // (strip - 1, rc) in the exchange buffer of one parity; the lane whose top is below this lane's cell
    const int  prev       = MULTI ? (below / spw) * 6 * 32 + (below % spw) * nrc + rc : max(w - nchunks, 0) * 6 * 32 + lane;
    const int  below_lane = MULTI ? (lane & ~(nrc - 1)) | ((lane + nrc - 1) & (nrc - 1)) : (lane + 31) & 31;
    const bool last_chunk = chunk + 1 == nchunks;
    const bool first_node = rc == 0, last_node = rc == nrc - 1;  // this lane holds the strip's node 0 / nr - 1

    // radial constants: rho = beta / alpha = 2 r_mid / (3 dr), weight dr / 8 (/ 6 for the nodal mean)
    auto rho_of = [&](int c) { return (A.radii[c] + A.radii[c + 1]) / (T(3) * (A.radii[c + 1] - A.radii[c])); };
    const T rho = rho_of(rc);
    const T wr  = (A.radii[rc + 1] - A.radii[rc]) / (Q0 ? T(8) : T(48));

    const T rho_low = !MULTI && chunk > 0 ? rho_of(rc - 1) : T(0);  // of the cell below the chunk

    // a node column of the sweep: corner sums / differences / coefficients of nodes y (0) and y + 1 (1)
    struct Column {
        T S[2][3], D[2][3], k[2];
    } o = {};
    // forces the column's cells left on it (lateral part of node y + 1 with opposite sign)
    T         cL[2][3], cR[2][3];
    T         kL[3], kR[3];  // this warp's sums of node (x, y)
    int       x = 0;
    int       e0 = 0, q0 = 0;  // byte offsets of the cell's bottom node y (and cell coefficient) in a staged field
    int       id = 0;          // node (x, y, rc)
    bool      valid = false, own = false, some = true, any_own = true;
    const int pitch = nr * static_cast<int>(sizeof(T));
    uint32_t  slot = 0, par = 0;  // ring slot of row f, exchange parity of the step
    const uint32_t half = A.warps * (6 * 32);
    T* const       out  = xch + w * (6 * 32) + lane;
    const T* const in   = xch + prev;

    auto put = [&](int c, int i, T v) {
        T* p = A.dst[c] + i;
        if (ADD) v += *p;
        *p = v;
    };
    auto load_column = [&](uint32_t rslot, Column& C) {
        const int4 o4    = *reinterpret_cast<const int4*>(off + 4 * rslot);
        const int  at[4] = {o4.x, o4.y, o4.z, o4.w};
#pragma unroll
        for (int fld = 0; fld < (Q0 ? 3 : 4); ++fld) {
            const unsigned char* p0 = smem + at[fld] + e0;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const T* p   = reinterpret_cast<const T*>(p0 + q * pitch);
                T        bot = p[0], top = p[1];
                if (MULTI && !valid) bot = top = T(0);
                if (fld < 3) {
                    C.S[q][fld] = top + bot;
                    C.D[q][fld] = top - bot;
                } else {
                    C.k[q] = wr * (top + bot);
                }
            }
        }
    };
    // Cells between rows f and f + 1 (slot n1): sums of row f into kL / kR and the exchange, of row f + 1 into cL / cR.
    auto cells = [&](uint32_t n1) {
        Column n;
        load_column(n1, n);
        T kw0, kw1;
        if constexpr (Q0) {
            T kc = *reinterpret_cast<const T*>(smem + off[4 * n1 + 3] + q0);
            if (MULTI && !valid) kc = T(0);
            kw0 = kw1 = wr * kc;
        } else {
            const T k12 = n.k[0] + o.k[1];
            kw0         = o.k[0] + k12;
            kw1         = n.k[1] + k12;
        }
        // corners: 0 = (x, y) old 0, 2 = (x, y + 1) old 1, 1 = (x + 1, y) new 0, 3 = (x + 1, y + 1) new 1;
        // wedge 0 has nodes 0, 1, 2, wedge 1 has nodes 3, 2, 1
        T a[3], b[3], D[3], m[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            a[c] = n.S[0][c] - o.S[0][c];
            b[c] = o.S[1][c] - o.S[0][c];
            m[c] = rho * (n.D[0][c] + o.D[1][c]);
            D[c] = fma(rho, o.D[0][c], m[c]);
        }
        const T* gp = reinterpret_cast<const T*>(smem + L.ring + n1 * L.slot) + strip * kGeo;
        auto     load_geo = [&](int w2, T (&g)[9]) {
            const T* q = gp + w2 * (kGeo / 2);
            if constexpr (sizeof(T) == 8) {
#pragma unroll
                for (int i = 0; i < 8; i += 2) {
                    const double2 t = *reinterpret_cast<const double2*>(q + i);
                    g[i] = t.x, g[i + 1] = t.y;
                }
            } else {
#pragma unroll
                for (int i = 0; i < 8; i += 4) {
                    const float4 t = *reinterpret_cast<const float4*>(q + i);
                    g[i] = t.x, g[i + 1] = t.y, g[i + 2] = t.z, g[i + 3] = t.w;
                }
            }
            g[8] = q[8];
        };
        T g[9], v1[3], v2[3], wv[3], r0[3], sL[3];
        load_geo(0, g);
        wedge_forces(g, a, b, D, kw0, v1, v2, wv);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            kL[c]    = cL[0][c] - (v1[c] + v2[c]);
            kR[c]    = cR[0][c] + wv[c];
            sL[c]    = v2[c] - cL[1][c];
            cL[0][c] = v1[c];
            r0[c]    = wv[c];
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            a[c] = o.S[1][c] - n.S[1][c];
            b[c] = n.S[0][c] - n.S[1][c];
            D[c] = fma(rho, n.D[1][c], m[c]);
        }
        load_geo(1, g);
        wedge_forces(g, a, b, D, kw1, v1, v2, wv);
        T* so = out + par;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const T rad      = r0[c] + wv[c];
            so[c * 32]       = sL[c] + v1[c];
            so[(3 + c) * 32] = cR[1][c] + rad;
            cL[0][c] += v2[c];
            cR[0][c] = rad;
            cL[1][c] = v1[c] + v2[c];
            cR[1][c] = wv[c];
        }
        o = n;
    };
    // no cells beyond row f: what the column before left
    auto no_cells = [&] {
        T* so = out + par;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            kL[c]            = cL[0][c];
            kR[c]            = cR[0][c];
            so[c * 32]       = -cL[1][c];
            so[(3 + c) * 32] = cR[1][c];
        }
    };
    // Node values of row f: own sums plus those of the strip below in y.
    auto nodes = [&](bool write) {
        if (!MULTI && !last_chunk && lane == 31) {  // own sums of the chunk's last cell for the chunk above
            T* q = edge + (par == 0 ? 0 : A.warps * 6) + w * 6;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                q[c]     = kL[c];
                q[3 + c] = kR[c];
            }
        }
        row_barrier();
        if (write && any_own) {
            const T* ps = in + par;
            T        bot[3], top[3], low[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const T l = kL[c] + ps[c * 32], r = kR[c] + ps[(3 + c) * 32];
                bot[c] = fma(-rho, r, l);
                top[c] = fma(rho, r, l);
                low[c] = __shfl_sync(0xffffffffu, top[c], below_lane);
                if (MULTI ? first_node : lane == 0) low[c] = T(0);
            }
            if (!MULTI && chunk > 0 && lane == 0) {  // the cell below belongs to the warp before
                const T* q  = edge + (par == 0 ? 0 : A.warps * 6) + (w - 1) * 6;
                const T* q2 = ps - 6 * 32 + 31;
#pragma unroll
                for (int c = 0; c < 3; ++c) low[c] = fma(rho_low, q[3 + c] + q2[(3 + c) * 32], q[c] + q2[c * 32]);
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) bot[c] += low[c];
            if (!MULTI || own) {
                if (first_node || last_node) {  // nrc >= 2: never both
                    const int bc = first_node ? A.bc_cmb : A.bc_surf;
                    const T*  q  = rec + (slot * static_cast<uint32_t>(strips + 1) + strip) * 8 + (first_node ? 0 : 4);
                    T         v[3];
#pragma unroll
                    for (int c = 0; c < 3; ++c) v[c] = first_node ? bot[c] : top[c];
                    if (bc == 1) {
                        v[0] = q[0], v[1] = q[1], v[2] = q[2];
                    } else if (bc == 2) {
                        const T cr = q[3] - (q[0] * v[0] + q[1] * v[1] + q[2] * v[2]);
                        v[0] += cr * q[0], v[1] += cr * q[1], v[2] += cr * q[2];
                    }
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        if (first_node)
                            bot[c] = v[c];
                        else
                            put(c, id + 1, v[c]);
                    }
                }
#pragma unroll
                for (int c = 0; c < 3; ++c) put(c, id, bot[c]);
            }
        }
        par = half - par;
        id += nl * nr;
    };

    row_barrier();
    for (int f = F0; f < R1;) {
        // rows of one tile: x .. xe - 1
        const int tile = f / nl, d = tile / ytiles, y0 = (tile - d * ytiles) * ty;
        x            = f - tile * nl;
        const int xe = min(nl, x + R1 - f), yc = y0 - 1 + strip, col0 = max(strip - (y0 == 0 ? 1 : 0), 0);
        valid   = yc >= 0 && yc < nl - 1;
        own     = strip >= 1 && strip <= ty && yc < nl;
        e0      = (col0 * nr + rc) * static_cast<int>(sizeof(T));
        q0      = (col0 * nrc + rc) * static_cast<int>(sizeof(T));
        id      = ((d * nl + x) * nl + yc) * nr + rc;  // 32-bit: the host limits a level to 2^31 nodes
        some    = MULTI ? __any_sync(0xffffffffu, valid) : valid;
        any_own = MULTI ? __any_sync(0xffffffffu, own) : own;
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int c = 0; c < 3; ++c) cL[q][c] = cR[q][c] = T(0);
        if (some && x < nl - 1) load_column(slot, o);
        const int cols = min(xe, nl - 1);
        // FP64 has registers for two columns a trip, which saves copying the column behind (105 -> 102 us at level 6).
        // FP32, which spills 36 to 52 bytes at its 72 registers, spills more with it (69 -> 73 us).
#pragma unroll(sizeof(T) == 8 ? 2 : 1)
        for (; x < cols; ++x, ++f) {
            const uint32_t n1 = slot + 1 == kRing ? 0 : slot + 1;
            if (some)
                cells(n1);
            else
                no_cells();
            nodes(f >= R0);
            slot = n1;
        }
        if (x < xe) {  // the tile's last row
            no_cells();
            nodes(f >= R0);
            slot = slot + 1 == kRing ? 0 : slot + 1;
            ++f;
        }
    }
}

// ---------------------------------------------------------------------------
// Diagonal. f(g, kw) for every wedge around node (d, x, y, r) of this diamond: physical gradient g of the node's
// shape function and weight kw = k |det J|. Bound by issue and load latency: the two cells of a wedge column share its
// geometry, and the nodal coefficients are taken once a node instead of once a wedge (21 loads instead of 72).
// ---------------------------------------------------------------------------
template <typename G, typename K, typename F>
__device__ __forceinline__ void node_wedges(int nl, int nr, const G* colgeo, const G* radgeo, const K* k, const K* kq0,
                                            int d, int x, int y, int r, F&& f)
{
    // cells above (0: the node is at the bottom, cell r) and below (1: at the top, cell r - 1)
    const bool has[2] = {r < nr - 1, r > 0};
    G          alpha[2], beta[2], dfac[2];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const G* rg = radgeo + 3 * (r - s);
        alpha[s]    = has[s] ? rg[0] : G(0);
        beta[s]     = has[s] ? (s == 0 ? -rg[1] : rg[1]) : G(0);
        dfac[s]     = has[s] ? rg[2] : G(0);
    }
    // nodal coefficient of the seven lateral nodes around, bottom plus top of either cell: each value is loaded once
    G S[3][3][2] = {};
    if (!kq0) {
        const K* kb = k + node_index(nl, nr, d, x, y, r);
#pragma unroll
        for (int dx = -1; dx <= 1; ++dx)
#pragma unroll
            for (int dy = -1; dy <= 1; ++dy) {
                if (dx != 0 && dx == dy) continue;  // not in a wedge with the node
                const bool in = x + dx >= 0 && x + dx < nl && y + dy >= 0 && y + dy < nl;
                const K*   q  = kb + (dx * nl + dy) * nr;
                const G    up = in && has[0] ? static_cast<G>(q[1]) : G(0), at = in ? static_cast<G>(q[0]) : G(0),
                        down    = in && has[1] ? static_cast<G>(q[-1]) : G(0);
                S[dx + 1][dy + 1][0] = at + up;
                S[dx + 1][dy + 1][1] = at + down;
            }
    }
    const int col = (d * (nl - 1) + x) * (nl - 1) + y;  // 20 values a column: below 2^31 on every level
    const K*  kc  = kq0 ? kq0 + (static_cast<int64_t>(col) * (nr - 1) + r) : nullptr;
#pragma unroll
    for (int ab = 0; ab < 4; ++ab) {
        const int ox = ab & 1, oy = ab >> 1;
        if (x - ox < 0 || y - oy < 0 || x - ox > nl - 2 || y - oy > nl - 2) continue;
        const int back = ox * (nl - 1) + oy;
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            const int m = w == 0 ? ab : 3 - ab;  // lateral index of corner ab in wedge w
            if (m > 2) continue;
            const G* gw = colgeo + (col - back) * 20 + 10 * w;
            G        lat[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) lat[i] = m == 0 ? -(gw[i] + gw[3 + i]) : (m == 1 ? gw[i] : gw[3 + i]);
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                if (!has[s]) continue;
                G kv;
                if (kq0) {
                    kv = static_cast<G>(kc[-back * (nr - 1) - s]);
                } else {
                    kv = G(0);
#pragma unroll
                    for (int j = 0; j < 3; ++j) {
                        const int q = wedge_corner(w, j);
                        kv += S[(q & 1) - ox + 1][(q >> 1) - oy + 1][s];
                    }
                    kv *= G(1) / G(6);
                }
                G g[3];
#pragma unroll
                for (int i = 0; i < 3; ++i) g[i] = alpha[s] * lat[i] + beta[s] * gw[6 + i];
                f(g, kv * gw[9] * dfac[s]);
            }
        }
    }
}

// Diagonal mode: dst = diag(A) src, one thread per node; FRAME: the free-slip nodes, one thread per node of the two
// boundary planes, with the diagonal in the node's normal-tangential frame. In a kernel of their own those nodes cost the
// others neither registers nor branches. Level 7 (64 layers), no boundary treatment, nodal coefficient: FP64 508 us,
// FP32 285 us (in one kernel, with the coefficients loaded per wedge, 780 and 691; in the sweep of the apply 643 and 361).
template <typename T, bool FRAME>
__global__ void __launch_bounds__(256, FRAME ? 1 : 3) edd_diagonal_kernel(EddLaunch<T> A, int n, Decoder rad, Decoder lat)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int d, x, y, r, col;
    if (FRAME) {
        const int side = i & 1;
        i              = (i >> 1) * A.nr + (side ? A.nr - 1 : 0);
    }
    decode4(i, rad, lat, d, x, y, r, col);
    const int bc = r == 0 ? A.bc_cmb : (r == A.nr - 1 ? A.bc_surf : 0);
    if ((bc == 2) != FRAME) return;
    const T u[3] = {A.src[0][i], A.src[1][i], A.src[2][i]};
    T       o[3], dg[3] = {T(0), T(0), T(0)};
    if constexpr (FRAME) {
        const T* c  = A.coords + static_cast<int64_t>(col) * 3;
        const T  in = T(1) / sqrt(c[0] * c[0] + c[1] * c[1] + c[2] * c[2]);
        const T  nv[3] = {c[0] * in, c[1] * in, c[2] * in};
        T        R[3][3];
        trafo_nt(nv, R);
        node_wedges(A.nl, A.nr, A.colgeo, A.radgeo, A.k, A.kq0, d, x, y, r, [&](const T(&g)[3], T kw) {
            const T gg = g[0] * g[0] + g[1] * g[1] + g[2] * g[2];
            for (int c2 = 0; c2 < 3; ++c2) {
                const T q = R[c2][0] * g[0] + R[c2][1] * g[1] + R[c2][2] * g[2];
                dg[c2] += kw * (gg + q * q * (T(1) / T(3)));
            }
        });
        T v[3];
        for (int a = 0; a < 3; ++a) v[a] = dg[a] * (R[a][0] * u[0] + R[a][1] * u[1] + R[a][2] * u[2]);
        for (int c2 = 0; c2 < 3; ++c2) o[c2] = R[0][c2] * v[0] + R[1][c2] * v[1] + R[2][c2] * v[2];
    } else {
        node_wedges(A.nl, A.nr, A.colgeo, A.radgeo, A.k, A.kq0, d, x, y, r, [&](const T(&g)[3], T kw) {
            const T gg = g[0] * g[0] + g[1] * g[1] + g[2] * g[2];
            for (int c = 0; c < 3; ++c) dg[c] += kw * (gg + g[c] * g[c] * (T(1) / T(3)));
        });
        for (int c = 0; c < 3; ++c) o[c] = dg[c] * u[c];
    }
    for (int c = 0; c < 3; ++c) A.dst[c][i] = A.add ? A.dst[c][i] + o[c] : o[c];
}

// Boundary rows: for each node of the two boundary planes the diagonal (3 values) and the normal stiffness
// sum kw (|g|^2 + (n.g)^2 / 3), of this diamond's cells, and the unit normal. Independent of the boundary conditions.
template <typename T>
__global__ void __launch_bounds__(256) edd_boundary_kernel(int nl, int nr, const double* coords, const double* colgeo,
                                                           const double* radgeo, const T* k, const T* kq0, T* out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x, n = 10 * nl * nl;
    if (i >= 2 * n) return;
    const int    side = i / n, c = i % n;
    const int    y = c % nl, x = (c / nl) % nl, d = c / (nl * nl);
    const double p0 = coords[3 * c], p1 = coords[3 * c + 1], p2 = coords[3 * c + 2];
    const double in = 1.0 / sqrt(p0 * p0 + p1 * p1 + p2 * p2);
    double       dg[3] = {0.0, 0.0, 0.0}, ann = 0.0;
    node_wedges(nl, nr, colgeo, radgeo, k, kq0, d, x, y, side == 0 ? 0 : nr - 1, [&](const double(&g)[3], double kw) {
        const double gg = g[0] * g[0] + g[1] * g[1] + g[2] * g[2];
        for (int q = 0; q < 3; ++q) dg[q] += kw * (gg + g[q] * g[q] * (1.0 / 3.0));
        const double ng = (p0 * g[0] + p1 * g[1] + p2 * g[2]) * in;
        ann += kw * (gg + ng * ng * (1.0 / 3.0));
    });
    T* o = out + static_cast<int64_t>(i) * 8;
    for (int q = 0; q < 3; ++q) o[q] = static_cast<T>(dg[q]);
    o[3] = static_cast<T>(ann);
    o[4] = static_cast<T>(p0 * in), o[5] = static_cast<T>(p1 * in), o[6] = static_cast<T>(p2 * in), o[7] = T(0);
}

// Double-double arithmetic for the lateral table (Dekker, Numer. Math. 18, 1971; products by fused multiply-add), so
// that its entries are the rounded exact values: they enter the apply twice, on the input and on the output side.
struct Dd {
    double h, l;
};
__device__ __forceinline__ Dd dd_norm(double a, double b)
{
    const double s = a + b;
    return {s, b - (s - a)};
}
__device__ __forceinline__ Dd dd_add(Dd a, Dd b)
{
    const double s = a.h + b.h, v = s - a.h;
    return dd_norm(s, ((a.h - (s - v)) + (b.h - v)) + (a.l + b.l));
}
__device__ __forceinline__ Dd dd_neg(Dd a) { return {-a.h, -a.l}; }
__device__ __forceinline__ Dd dd_mul(Dd a, Dd b)
{
    const double p = a.h * b.h;
    return dd_norm(p, fma(a.h, b.h, -p) + (a.h * b.l + a.l * b.h));
}
__device__ __forceinline__ Dd dd_div(Dd a, Dd b)
{
    const double q = a.h / b.h;
    const Dd     r = dd_add(a, dd_neg(dd_mul(b, {q, 0.0})));
    return dd_norm(q, (r.h + r.l) / b.h);
}
__device__ __forceinline__ Dd dd_sqrt(Dd a)
{
    const double q = sqrt(a.h);
    const Dd     r = dd_add(a, dd_neg(dd_mul({q, 0.0}, {q, 0.0})));
    return dd_norm(q, (r.h + r.l) / (2.0 * q));
}

// Lateral table: entry (d, x, e) holds sqrt|det M| (e1, e2, e3) of both wedges of column y = e - 1 (zeros off the mesh).
// e1 = a2 x a3 / det and so on, so sqrt|det M| e1 = a2 x a3 / (sign(det) sqrt|det M|).
template <typename T>
__global__ void __launch_bounds__(128) edd_lateral_kernel(int nl, const double* coords, T* out)
{
    constexpr int kGeo = Shape<T>::kGeo;
    const int     i    = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 10 * (nl - 1) * nl) return;
    const int e = i % nl, x = (i / nl) % (nl - 1), d = i / (nl * (nl - 1));
    T*        o = out + static_cast<int64_t>(i) * kGeo;
    for (int v = 0; v < kGeo; ++v) o[v] = T(0);
    if (e == 0) return;
    for (int w = 0; w < 2; ++w) {
        Dd a[3][3];
        for (int c = 0; c < 3; ++c) {
            Dd p[3];
            for (int m = 0; m < 3; ++m) {
                const int q = wedge_corner(w, m);
                p[m]        = {coords[lat_index3(nl, d, x + (q & 1), e - 1 + (q >> 1)) * 3 + c], 0.0};
            }
            a[0][c] = dd_add(p[1], dd_neg(p[0]));
            a[1][c] = dd_add(p[2], dd_neg(p[0]));
            a[2][c] = dd_div(dd_add(dd_add(p[0], p[1]), p[2]), {3.0, 0.0});
        }
        Dd n[3][3], det = {0.0, 0.0};
        for (int k = 0; k < 3; ++k)
            for (int c = 0; c < 3; ++c) {
                const Dd *u = a[(k + 1) % 3], *v = a[(k + 2) % 3];
                n[k][c] = dd_add(dd_mul(u[(c + 1) % 3], v[(c + 2) % 3]), dd_neg(dd_mul(u[(c + 2) % 3], v[(c + 1) % 3])));
            }
        for (int c = 0; c < 3; ++c) det = dd_add(det, dd_mul(a[0][c], n[0][c]));
        const Dd s = det.h < 0.0 ? dd_neg(dd_sqrt(dd_neg(det))) : dd_sqrt(det);
        for (int k = 0; k < 3; ++k)
            for (int c = 0; c < 3; ++c) o[w * (kGeo / 2) + 3 * k + c] = static_cast<T>(dd_div(n[k][c], s).h);
    }
}

template <typename T, bool Q0, bool MULTI, bool ADD>
int launch_cfg(const EddArgs<T>& a, size_t smem, int ctas, cudaStream_t st)
{
    auto k = epsdivdiv_kernel<T, Q0, MULTI, ADD>;
    // the dynamic shared-memory limit is a per-device attribute of the kernel:
    // raise it once per device, only upwards; the check, the attribute call
    // and the record happen under one lock so racing threads cannot lower it
    static std::mutex mu;
    static size_t     configured[kMaxDevices];
    int               dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return -1;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (smem > configured[dev]) {
            // the compute warps wait for registers that the block must hold from its launch
            cudaFuncAttributes at;
            if (cudaFuncGetAttributes(&at, k) != cudaSuccess || (Shape<T>::kSplit && at.numRegs * 4 < 3 * Shape<T>::kComputeRegs + Shape<T>::kStageRegs))
                return -7;
            if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) !=
                cudaSuccess)
                return -1;
            configured[dev] = smem;
        }
    }
    launch_chained(k, ctas, Shape<T>::kThreads, smem, st, a);
    note_launch();
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int sm_count()
{
    static std::atomic<int> counts[kMaxDevices];
    int                     dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return -1;
    int sms = counts[dev].load(std::memory_order_relaxed);
    if (sms == 0) {
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
        counts[dev].store(sms, std::memory_order_relaxed);
    }
    return sms;
}

}  // namespace

template <typename T>
EddPlan edd_plan(int nl, int nr, int sms, int tile_y, int chunk_x)
{
    // Warps come in whole strips. The cost of a shape is rows per CTA (plus the repeated column) times the time of a
    // row: the issue time of its warps, four schedulers at a time, plus a latency floor of about five warps. It picks
    // 12 strips at level 6 in FP32 (69 us; 11 strips 80 us) and 6 in FP64 (105 us, with one column a trip; 4 strips
    // 140 us).
    const int nrc = nr - 1, slots = 32;
    const int wps = nrc > slots ? nrc / slots : 1;  // warps per strip
    const int spw = nrc < slots ? slots / nrc : 1;  // strips per warp
    EddPlan   best;
    double    cost = -1.0;
    for (int w = wps; w <= Shape<T>::kComputeWarps; w += wps) {
        const int strips = w / wps * spw;
        if (strips < 2) continue;
        if (edd_smem<T>(nr, w, strips).total > kSmemLimit) break;
        EddPlan p;
        p.warps  = w;
        p.strips = strips;
        p.ty     = std::min(strips - 1, nl);
        if (tile_y > 0) {
            p.ty = std::min(p.ty, tile_y);
            if (p.ty < std::min(tile_y, nl) && w + wps <= Shape<T>::kComputeWarps) continue;  // a larger CTA holds the asked tile
        }
        p.ytiles     = (nl + p.ty - 1) / p.ty;
        p.total_rows = 10 * p.ytiles * nl;
        p.rows       = chunk_x > 0 ? std::min(chunk_x, p.total_rows) : (p.total_rows + sms - 1) / sms;
        p.ctas       = (p.total_rows + p.rows - 1) / p.rows;
        const double waves = static_cast<double>((p.ctas + sms - 1) / sms);
        const double c     = waves * (p.rows + 1) * ((w + 3) / 4 * 4 + 5.0);
        if (cost < 0.0 || c < cost) {
            cost = c;
            best = p;
        }
        if (strips > nl) break;  // one tile holds every line
    }
    return best;
}

template <typename T>
int epsdivdiv_apply(const EddLaunch<T>& p, cudaStream_t stream)
{
    if (10LL * p.nl * p.nl * p.nr >= (1LL << 31)) return -6;  // the kernels index nodes in 32 bits
    const int nrc = p.nr - 1;
    if (p.diagonal) {
        const int n = 10 * p.nl * p.nl * p.nr;
        edd_diagonal_kernel<T, false><<<(n + 255) / 256, 256, 0, stream>>>(p, n, Decoder(p.nr), Decoder(p.nl));
        note_launch();
        if (p.bc_cmb == 2 || p.bc_surf == 2) {
            const int m = 2 * 10 * p.nl * p.nl;
            edd_diagonal_kernel<T, true><<<(m + 255) / 256, 256, 0, stream>>>(p, m, Decoder(p.nr), Decoder(p.nl));
            note_launch();
        }
        return cudaGetLastError() == cudaSuccess ? 0 : -2;
    }
    if (nrc < 2 || nrc > 128 || (nrc & (nrc - 1)) != 0) return -3;
    if (!p.lateral || !p.boundary) return -4;
    const int sms = sm_count();
    if (sms <= 0) return -1;
    const EddPlan plan = edd_plan<T>(p.nl, p.nr, sms, p.tile_y, p.chunk_x);
    if (plan.warps == 0) return -5;
    EddArgs<T> a;
    a.nl     = p.nl;
    a.nr     = p.nr;
    a.geo    = p.lateral;
    a.radii  = p.radii;
    a.bdiag  = p.boundary;
    a.k      = p.k;
    a.kq0    = p.kq0;
    for (int c = 0; c < 3; ++c) {
        a.src[c] = p.src[c];
        a.dst[c] = p.dst[c];
    }
    a.bc_cmb     = p.bc_cmb;
    a.bc_surf    = p.bc_surf;
    a.err        = p.err;
    a.warps      = plan.warps;
    a.strips     = plan.strips;
    a.ty         = plan.ty;
    a.ytiles     = plan.ytiles;
    a.rows       = plan.rows;
    a.total_rows = plan.total_rows;
    const size_t smem = edd_smem<T>(p.nr, plan.warps, plan.strips).total;
    auto go = [&](auto q0, auto multi) {
        constexpr bool Q = decltype(q0)::value, M = decltype(multi)::value;
        return p.add ? launch_cfg<T, Q, M, true>(a, smem, plan.ctas, stream)
                     : launch_cfg<T, Q, M, false>(a, smem, plan.ctas, stream);
    };
    using Yes = std::true_type;
    using No  = std::false_type;
    if (nrc < 32) return p.kq0 ? go(Yes{}, Yes{}) : go(No{}, Yes{});
    return p.kq0 ? go(Yes{}, No{}) : go(No{}, No{});
}

template <typename T>
size_t edd_lateral_values(int nl)
{
    return static_cast<size_t>(10) * (nl - 1) * nl * Shape<T>::kGeo;
}

template <typename T>
int edd_lateral_table(int nl, const double* coords, T* out, cudaStream_t st)
{
    const int n = 10 * (nl - 1) * nl;
    edd_lateral_kernel<T><<<(n + 127) / 128, 128, 0, st>>>(nl, coords, out);
    note_launch();
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

template <typename T>
int edd_boundary_table(int nl, int nr, const double* coords, const double* colgeo, const double* radgeo, const T* k,
                       const T* kq0, T* out, cudaStream_t st)
{
    const int n = 2 * 10 * nl * nl;
    edd_boundary_kernel<T><<<(n + 255) / 256, 256, 0, st>>>(nl, nr, coords, colgeo, radgeo, k, kq0, out);
    note_launch();
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

#define TN_INST(T)                                                                                                   \
    template EddPlan edd_plan<T>(int, int, int, int, int);                                                          \
    template int epsdivdiv_apply<T>(const EddLaunch<T>&, cudaStream_t);                                             \
    template size_t edd_lateral_values<T>(int);                                                                    \
    template int edd_lateral_table<T>(int, const double*, T*, cudaStream_t);                                      \
    template int edd_boundary_table<T>(int, int, const double*, const double*, const double*, const T*, const T*, T*, \
                                       cudaStream_t);
TN_INST(double)
TN_INST(float)
#undef TN_INST

}  // namespace tn
