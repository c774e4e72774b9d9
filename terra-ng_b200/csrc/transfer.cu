// Constant-weight multigrid transfers between level l (fine) and l-1 (coarse).
//
// Weights are prolongation_constant_weight (fe/wedge/shell/
// grid_transfer_constant.hpp:24-89): linear interpolation on the anti-diagonal
// triangulation of each diamond, tensor product with linear interpolation in r.
//   prolongate_add : fine += P coarse   (ProlongationVecConstant, Add mode,
//                    prolongation_constant.hpp:146-191), here as a gather: one
//                    thread per fine node reading its 1..8 coarse parents, no atomics.
//   restrict_owned : coarse = P^T (owned fine)  (RestrictionVecConstant,
//                    restriction_constant.hpp:190-249): one thread per coarse
//                    node over its 21-point fine stencil, non-owned fine
//                    duplicates masked; the caller completes it with the coarse
//                    interface sum.
#include "tn_device.cuh"
#include "tn_kernels.hpp"
#include "tn_wedge_math.cuh"

namespace tn {
namespace {

constexpr int kMaxComp = 4;
template <typename T>
struct PtrSet {
    const T* in[kMaxComp];
    const T* b[kMaxComp];
    T*       out[kMaxComp];
};

// Flat grids: one thread per fine node (prolongation) or coarse node (restriction) in storage order and component
// (grid.y), 256 threads per CTA, indices decoded with Decoder, so no thread of a radial column idles. Bound by load
// latency: on the small levels a kernel is one dependent chain, on the large ones it needs many loads in flight. So no
// load hangs on another (masks and values are read together, the mask applied after), and components run in
// different threads. Before (components in a loop of run-time length, loads behind the ownership test), cold caches:
// restriction 42 / 19 / 18 us to level 5 / 4 / 3 in FP32, prolongation 38 us to level 6. With the residual formed in the
// restriction instead of a pass of its own the level-6 mixed preconditioner went from 3.55 to 3.52 ms. The pointer set is a
// __grid_constant__: indexed by blockIdx.y, a plain parameter is copied to the stack by every thread (prolongation of three
// components to level 6: FP32 102 us instead of 34, FP64 107 instead of 37; a loop over the components in the thread 37 / 47).
constexpr int kTransferThreads = 256;

template <typename T>
__global__ void __launch_bounds__(kTransferThreads) prolongate_kernel(int nlf, int nrf,
                                                                      const __grid_constant__ PtrSet<T> P, int n,
                                                                      Decoder rad, Decoder lat)
{
    const int nlc = (nlf + 1) / 2, nrc = (nrf + 1) / 2;
    const int i   = blockIdx.x * blockDim.x + threadIdx.x;
    chain_enter();
    if (i >= n) return;
    const T* in  = P.in[blockIdx.y];
    T*       out = P.out[blockIdx.y];
    int d, x, y, r, col;
    decode4(i, rad, lat, d, x, y, r, col);
    // lateral parents: one, or two across an edge (along x, along y, or the anti-diagonal), and radial parents
    const int     x0 = (x + ((x & y) & 1)) / 2, y0 = y / 2;
    const int     x1 = (x & y & 1) ? (x - 1) / 2 : (x + 1) / 2, y1 = (y + 1) / 2;
    const bool    two = ((x | y) & 1) != 0, mid = (r & 1) != 0;
    const int64_t p0 = node_index(nlc, nrc, d, x0, y0, r / 2), p1 = node_index(nlc, nrc, d, x1, y1, r / 2);
    const T       old = out[i];
    const T       a0  = in[p0];
    const T       b0  = two ? in[p1] : T(0);
    const T       a1  = mid ? in[p0 + 1] : T(0);
    const T       b1  = two && mid ? in[p1 + 1] : T(0);
    // Copies of a diamond-edge node in different diamonds list their two
    // lateral parents in different orders. Summing the lateral pair first
    // (a two-term sum is the same in either order) and then the radial pair
    // (same order everywhere) gives every copy identical bits, so prolonged
    // vectors stay consistent on interface duplicates in FP32 as in FP64.
    T acc = two ? a0 + b0 : a0;
    if (mid) acc += two ? a1 + b1 : a1;
    out[i] = old + (two ? T(0.5) : T(1)) * (mid ? T(0.5) : T(1)) * acc;
}

// RESIDUAL: restricts b - in instead of in.
template <typename T, bool RESIDUAL>
__global__ void __launch_bounds__(kTransferThreads) restrict_kernel(int nlf, int nrf, const uint8_t* __restrict__ owned,
                                                                    const __grid_constant__ PtrSet<T> P, int n,
                                                                    Decoder rad, Decoder lat)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    chain_enter();
    if (i >= n) return;
    const T* in = P.in[blockIdx.y];
    const T* b  = RESIDUAL ? P.b[blockIdx.y] : nullptr;
    int d, xc, yc, rc, col;
    decode4(i, rad, lat, d, xc, yc, rc, col);
    // 7-point lateral stencil (prolongation_constant_fine_grid_stencil_offsets_at_coarse_vertex)
    constexpr int ox[7] = {-1, -1, 0, 1, 1, 0, 0};
    constexpr int oy[7] = {0, 1, 1, 0, -1, -1, 0};
    bool          on[7];
    T             v[7][3], q[7][3];
#pragma unroll
    for (int o = 0; o < 7; ++o) {
        const int  xf = 2 * xc + ox[o], yf = 2 * yc + oy[o];
        const bool inside = xf >= 0 && xf < nlf && yf >= 0 && yf < nlf;
        on[o]             = inside && owned[lat_index3(nlf, d, xf, yf)] != 0;
        const int64_t fi  = node_index(nlf, nrf, d, xf, yf, 2 * rc);
#pragma unroll
        for (int dr = -1; dr <= 1; ++dr) {
            const int  rf = 2 * rc + dr;
            const bool ok = inside && rf >= 0 && rf < nrf;
            v[o][dr + 1]  = ok ? in[fi + dr] : T(0);
            if (RESIDUAL) q[o][dr + 1] = ok ? b[fi + dr] : T(0);
        }
    }
    T acc = T(0);
#pragma unroll
    for (int o = 0; o < 7; ++o) {
        const T wl = (o == 6) ? T(1) : T(0.5);
#pragma unroll
        for (int dr = -1; dr <= 1; ++dr) {
            const T f = RESIDUAL ? q[o][dr + 1] - v[o][dr + 1] : v[o][dr + 1];
            if (on[o]) acc += (dr == 0 ? wl : T(0.5) * wl) * f;
        }
    }
    P.out[blockIdx.y][i] = acc;
}

inline int launch_status(int kernels = 1)
{
    note_launch(kernels);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace

template <typename T>
int prolongate_add(int nlf, int nrf, int ncomp, const T* const* coarse, T* const* fine, cudaStream_t st)
{
    if (ncomp < 1 || ncomp > kMaxComp) return -1;
    PtrSet<T> P{};
    for (int c = 0; c < ncomp; ++c) {
        P.in[c]  = coarse[c];
        P.out[c] = fine[c];
    }
    const int n = 10 * nlf * nlf * nrf;
    const dim3 g((n + kTransferThreads - 1) / kTransferThreads, ncomp);
    launch_chained(prolongate_kernel<T>, g, kTransferThreads, 0, st, nlf, nrf, P, n, Decoder(nrf), Decoder(nlf));
    return launch_status();
}

template <typename T>
int restrict_owned(int nlf, int nrf, int ncomp, const uint8_t* owned_lat_fine, const T* const* b, const T* const* fine,
                   T* const* coarse, cudaStream_t st)
{
    if (ncomp < 1 || ncomp > kMaxComp) return -1;
    PtrSet<T> P{};
    for (int c = 0; c < ncomp; ++c) {
        P.in[c]  = fine[c];
        P.b[c]   = b ? b[c] : nullptr;
        P.out[c] = coarse[c];
    }
    const int  nlc = (nlf + 1) / 2, nrc = (nrf + 1) / 2;
    const int  n = 10 * nlc * nlc * nrc;
    const dim3 g((n + kTransferThreads - 1) / kTransferThreads, ncomp);
    if (b)
        launch_chained(restrict_kernel<T, true>, g, kTransferThreads, 0, st, nlf, nrf, owned_lat_fine, P, n, Decoder(nrc),
                       Decoder(nlc));
    else
        launch_chained(restrict_kernel<T, false>, g, kTransferThreads, 0, st, nlf, nrf, owned_lat_fine, P, n, Decoder(nrc),
                       Decoder(nlc));
    return launch_status();
}

template int prolongate_add<double>(int, int, int, const double* const*, double* const*, cudaStream_t);
template int prolongate_add<float>(int, int, int, const float* const*, float* const*, cudaStream_t);
template int restrict_owned<double>(int, int, int, const uint8_t*, const double* const*, const double* const*,
                                    double* const*, cudaStream_t);
template int restrict_owned<float>(int, int, int, const uint8_t*, const float* const*, const float* const*,
                                   float* const*, cudaStream_t);

}  // namespace tn
