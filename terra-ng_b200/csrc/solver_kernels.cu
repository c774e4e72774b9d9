// Kernels of the Krylov / multigrid solver layer.
//
// * Owned-node dot products over (block) vectors laid out as segments of
//   components (velocity on level L, pressure on level L-1), reduced in a fixed
//   order by the last block to finish (no second launch, bitwise reproducible),
//   with the result left in device memory so that the host does not wait.
// * The FGMRES modified Gram-Schmidt of one iteration in two passes over the basis
//   (fgmres.hpp:230-240 takes two launches per basis vector, dot then lincomb).
// * The Chebyshev-Jacobi update d = alpha D^-1 (b - A x) + beta d, x += d in one
//   pass (chebyshev.hpp:102-176 uses four BLAS-1 launches per step).
// * The coarsest-grid CG (pcg.hpp:81-169, identity preconditioner) as a single
//   thread-block-cluster kernel over assembled rows, or over stored element matrices
//   on levels too large for that: the CTAs of one cluster synchronise with the
//   hardware cluster barrier, so the whole solve is one launch.
#include <algorithm>
#include <cfloat>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>

#include <cooperative_groups.h>

#include "tn_device.cuh"
#include "tn_kernels.hpp"

namespace tn {
namespace {
namespace cg = cooperative_groups;

constexpr int kThreads = 256;
constexpr int kBlocks  = 592;  // 4 x 148 SMs

__device__ __forceinline__ double warp_sum(double v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Block sum, then the last block of the grid sums the per-block partials in
// index order and writes *out (sqrt of it when take_sqrt).
__device__ void block_finish(double v, RedScratch rs, double* out, int take_sqrt)
{
    __shared__ double red[kThreads / 32];
    __shared__ int    is_last;
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int k = 0; k < kThreads / 32; ++k) s += red[k];
        rs.partials[blockIdx.x] = s;
        __threadfence();
        const unsigned t = atomicAdd(rs.counter, 1u);
        is_last          = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (is_last) {
        __threadfence();
        double s = 0.0;
        for (int k = threadIdx.x; k < static_cast<int>(gridDim.x); k += blockDim.x) s += __ldcg(rs.partials + k);
        s = warp_sum(s);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
        __syncthreads();
        if (threadIdx.x == 0) {
            double tot = 0.0;
            for (int k = 0; k < kThreads / 32; ++k) tot += red[k];
            *out        = take_sqrt ? sqrt(tot) : tot;
            *rs.counter = 0u;
        }
    }
}

__device__ __forceinline__ uint32_t lat_of(int64_t i, uint64_t rdiv)
{
    return static_cast<uint32_t>((static_cast<uint64_t>(i) * rdiv) >> 40);
}

template <typename T>
__global__ void __launch_bounds__(kThreads) vdot_kernel(VecDesc L, const T* __restrict__ a, const T* __restrict__ b,
                                                         RedScratch rs, double* out, int take_sqrt)
{
    double        acc    = 0.0;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int s = 0; s < L.nseg; ++s) {
        const VecSeg S = L.seg[s];
        for (int c = 0; c < S.ncomp; ++c) {
            const T* pa = a + S.offset + c * S.stride;
            const T* pb = b + S.offset + c * S.stride;
            for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < S.n; i += stride)
                if (S.owned[lat_of(i, S.rdiv)]) acc += static_cast<double>(pa[i]) * static_cast<double>(pb[i]);
        }
    }
    block_finish(acc, rs, out, take_sqrt);
}

// ---------------------------------------------------------------------------
// Gram-Schmidt of w against the m = j + 1 basis vectors v_0 .. v_j in two passes.
//
// Modified Gram-Schmidt (fgmres.hpp:230-240) is h_i = <w_i, v_i>, w_{i+1} = w_i - h_i v_i. Since
// w_i = w - sum_{k<i} h_k v_k, its coefficients solve the unit lower triangular system
//   h_i = <w, v_i> - sum_{k<i} <v_k, v_i> h_k
// with the basis vectors' own inner products (Swirydowicz, Langou, Ananthan, Yang, Thomas: Low synchronization
// Gram-Schmidt and GMRES algorithms, Numer. Linear Algebra Appl. 2021). Pass 1 takes all <w, v_i> and the new row
// <v_j, v_k> of that matrix together; its last block solves for h. Pass 2 subtracts sum h_i v_i in order and takes
// the norm. Each basis vector is read twice per iteration, as in the vector-by-vector form, but w and v_j once per pass
// instead of w once per vector, and 2 launches replace m + 1.
//
// What bounds it: the DRAM reads of the basis. A lane takes four 16-byte pieces of two basis vectors at a time, all
// loaded before use. The inner products of a warp's 256 entries are reduced at once (two vectors share the shuffles) and
// summed per warp in shared memory, then per block and over blocks in index order: results are reproducible. One
// 64-bit word per 64 entries says which are owned (components start at multiples of 64 entries).
// ---------------------------------------------------------------------------
constexpr int kGsBlocks = 296;  // 2 x 148 SMs
constexpr int kGsWarps  = kThreads / 32;
constexpr int kGsPieces = 4;

__global__ void owned_mask_kernel(VecDesc L, uint64_t* __restrict__ mask, int64_t words)
{
    const int64_t k = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (k >= words) return;
    uint64_t m = 0;
    for (int b = 0; b < 64; ++b) {
        const int64_t e = k * 64 + b;
        for (int s = 0; s < L.nseg; ++s) {
            const VecSeg& S = L.seg[s];
            if (e < S.offset || e >= S.offset + S.ncomp * S.stride) continue;
            const int64_t i = (e - S.offset) % S.stride;
            if (i < S.n && S.owned[i / S.nr]) m |= uint64_t(1) << b;
        }
    }
    mask[k] = m;
}

__device__ __forceinline__ double2 masked(double2 v, uint64_t word, int lane)
{
    const uint32_t bits = static_cast<uint32_t>(word >> (2 * lane)) & 3u;
    return make_double2((bits & 1u) ? v.x : 0.0, (bits & 2u) ? v.y : 0.0);
}

__global__ void __launch_bounds__(kThreads, 2) gs_dots_kernel(int64_t words, const uint64_t* __restrict__ mask,
                                                              const double* __restrict__ w, BasisList B,
                                                              RedScratch rs, double* gram, int ld, double* h)
{
    __shared__ double acc[kGsWarps][2 * kMaxAxpy];  // [2 i]: <w, v_i>, [2 i + 1]: <v_j, v_i>
    __shared__ double hs;
    __shared__ int    is_last;
    const int     lane = threadIdx.x & 31, warp = threadIdx.x >> 5, m = B.m;
    const double* vj   = B.v[m - 1];
    for (int i = lane; i < 2 * m; i += 32) acc[warp][i] = 0.0;
    __syncwarp();
    const int64_t chunks = (words + kGsPieces - 1) / kGsPieces;
    for (int64_t c = static_cast<int64_t>(blockIdx.x) * kGsWarps + warp; c < chunks;
         c += static_cast<int64_t>(kGsBlocks) * kGsWarps) {
        const int64_t first = c * kGsPieces, e = first * 64 + 2 * lane;
        double2       wm[kGsPieces], jm[kGsPieces];
#pragma unroll
        for (int u = 0; u < kGsPieces; ++u) {
            wm[u] = jm[u] = make_double2(0.0, 0.0);
            if (first + u < words) {
                const uint64_t bits = mask[first + u];
                wm[u] = masked(*reinterpret_cast<const double2*>(w + e + 64 * u), bits, lane);
                jm[u] = masked(*reinterpret_cast<const double2*>(vj + e + 64 * u), bits, lane);
            }
        }
        for (int i = 0; i < m; i += 2) {
            const double* p0 = B.v[i] + e;
            const double* p1 = B.v[i + 1 < m ? i + 1 : i] + e;
            double2       a0[kGsPieces], a1[kGsPieces];
#pragma unroll
            for (int u = 0; u < kGsPieces; ++u) {
                a0[u] = a1[u] = make_double2(0.0, 0.0);
                if (first + u < words) {
                    a0[u] = *reinterpret_cast<const double2*>(p0 + 64 * u);
                    a1[u] = *reinterpret_cast<const double2*>(p1 + 64 * u);
                }
            }
            double t0 = 0.0, t1 = 0.0, g0 = 0.0, g1 = 0.0;
#pragma unroll
            for (int u = 0; u < kGsPieces; ++u) {
                t0 = fma(wm[u].y, a0[u].y, fma(wm[u].x, a0[u].x, t0));
                g0 = fma(jm[u].y, a0[u].y, fma(jm[u].x, a0[u].x, g0));
                t1 = fma(wm[u].y, a1[u].y, fma(wm[u].x, a1[u].x, t1));
                g1 = fma(jm[u].y, a1[u].y, fma(jm[u].x, a1[u].x, g1));
            }
            // lanes 0-15 go on with t, 16-31 with g; then bit 3 selects the vector
            const bool hi = lane & 16, second = lane & 8;
            double     k0 = hi ? g0 : t0, k1 = hi ? g1 : t1;
            k0 += __shfl_xor_sync(0xffffffffu, hi ? t0 : g0, 16);
            k1 += __shfl_xor_sync(0xffffffffu, hi ? t1 : g1, 16);
            double k = second ? k1 : k0;
            k += __shfl_xor_sync(0xffffffffu, second ? k0 : k1, 8);
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) k += __shfl_xor_sync(0xffffffffu, k, o);
            const int idx = 2 * (i + (second ? 1 : 0)) + (hi ? 1 : 0);
            if ((lane & 7) == 0 && idx < 2 * m) acc[warp][idx] += k;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * m; i += kThreads) {
        double s = 0.0;
        for (int k = 0; k < kGsWarps; ++k) s += acc[k][i];
        rs.partials[static_cast<int64_t>(i) * kGsBlocks + blockIdx.x] = s;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) is_last = atomicAdd(rs.counter, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    for (int i = warp; i < 2 * m; i += kGsWarps) {
        double s = 0.0;
        for (int k = lane; k < kGsBlocks; k += 32) s += __ldcg(rs.partials + static_cast<int64_t>(i) * kGsBlocks + k);
        s = warp_sum(s);
        if (lane == 0) acc[0][i] = s;
    }
    __syncthreads();
    // row j of the inner products, then forward substitution: thread k holds h_k once all h_i, i < k, are subtracted
    const int k = threadIdx.x;
    if (k < m - 1) gram[static_cast<int64_t>(m - 1) * ld + k] = acc[0][2 * k + 1];
    double hk = k < m ? acc[0][2 * k] : 0.0;
    for (int i = 0; i < m; ++i) {
        const double g = (k > i && k < m) ? (k == m - 1 ? acc[0][2 * i + 1] : __ldcg(gram + static_cast<int64_t>(k) * ld + i)) : 0.0;
        if (k == i) hs = hk;
        __syncthreads();
        if (k > i) hk -= hs * g;
        __syncthreads();
    }
    if (k < m) h[k] = hk;
    if (k == 0) *rs.counter = 0u;
}

// w -= sum h_i v_i in index order, *out = ||w||. Walks the entries from the end, where pass 1 stopped and the
// basis is still in L2.
__global__ void __launch_bounds__(kThreads, 2) gs_update_kernel(int64_t words, const uint64_t* __restrict__ mask,
                                                                double* __restrict__ w, BasisList B, const double* h,
                                                                RedScratch rs, double* out)
{
    __shared__ double hs[kMaxAxpy];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, m = B.m;
    for (int i = threadIdx.x; i < m; i += kThreads) hs[i] = h[i];
    __syncthreads();
    double        acc    = 0.0;
    const int64_t chunks = (words + kGsPieces - 1) / kGsPieces;
    for (int64_t c = chunks - 1 - (static_cast<int64_t>(blockIdx.x) * kGsWarps + warp); c >= 0;
         c -= static_cast<int64_t>(kGsBlocks) * kGsWarps) {
        const int64_t first = c * kGsPieces, e = first * 64 + 2 * lane;
        double2       v[kGsPieces];
#pragma unroll
        for (int u = 0; u < kGsPieces; ++u)
            if (first + u < words) v[u] = *reinterpret_cast<const double2*>(w + e + 64 * u);
        for (int i = 0; i < m; i += 2) {
            const bool    two = i + 1 < m;
            const double* p0  = B.v[i] + e;
            const double* p1  = B.v[two ? i + 1 : i] + e;
            const double  h0 = hs[i], h1 = two ? hs[i + 1] : 0.0;
            double2       a0[kGsPieces], a1[kGsPieces];
#pragma unroll
            for (int u = 0; u < kGsPieces; ++u)
                if (first + u < words) {
                    a0[u] = *reinterpret_cast<const double2*>(p0 + 64 * u);
                    if (two) a1[u] = *reinterpret_cast<const double2*>(p1 + 64 * u);
                }
#pragma unroll
            for (int u = 0; u < kGsPieces; ++u)
                if (first + u < words) {
                    v[u].x = v[u].x - h0 * a0[u].x;
                    v[u].y = v[u].y - h0 * a0[u].y;
                    if (two) {
                        v[u].x = v[u].x - h1 * a1[u].x;
                        v[u].y = v[u].y - h1 * a1[u].y;
                    }
                }
        }
#pragma unroll
        for (int u = 0; u < kGsPieces; ++u)
            if (first + u < words) {
                *reinterpret_cast<double2*>(w + e + 64 * u) = v[u];
                const double2 q = masked(v[u], mask[first + u], lane);
                acc             = fma(q.y, q.y, fma(q.x, q.x, acc));
            }
    }
    block_finish(acc, rs, out, 1);
}

// CG update x += alpha p, r -= alpha ap with alpha = s_an / s_ad from device
// memory, then *out = ||r|| (owned). Skips the update when |s_ad| < DBL_MIN
// (pcg.hpp:119-124 returns there) and writes *out = -1 so the host can tell.
__global__ void __launch_bounds__(kThreads) cg_update_kernel(VecDesc L, double* __restrict__ x,
                                                              double* __restrict__ r, const double* __restrict__ p,
                                                              const double* __restrict__ ap, const double* s_an,
                                                              const double* s_ad, RedScratch rs, double* out)
{
    const double ad = *s_ad;
    if (fabs(ad) < DBL_MIN) {
        if (blockIdx.x == 0 && threadIdx.x == 0) *out = -1.0;
        return;
    }
    const double  alpha  = *s_an / ad;
    double        acc    = 0.0;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int s = 0; s < L.nseg; ++s) {
        const VecSeg S = L.seg[s];
        for (int c = 0; c < S.ncomp; ++c) {
            const int64_t o = S.offset + c * S.stride;
            for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < S.n; i += stride) {
                x[o + i]        = x[o + i] + alpha * p[o + i];
                const double rv = r[o + i] - alpha * ap[o + i];
                r[o + i]        = rv;
                if (S.owned[lat_of(i, S.rdiv)]) acc += rv * rv;
            }
        }
    }
    block_finish(acc, rs, out, 1);
}

// p = z + (s_num / s_den) p
__global__ void p_update_kernel(int64_t n, double* __restrict__ p, const double* __restrict__ z, const double* s_num,
                                const double* s_den)
{
    const double  beta   = *s_num / *s_den;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
        p[i] = z[i] + beta * p[i];
}

// v -= scale * (*s) on n entries
__global__ void sub_scalar_kernel(int64_t n, double* __restrict__ v, const double* s, double scale)
{
    const double  c      = scale * *s;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) v[i] -= c;
}

template <typename T>
__global__ void scale_recip_kernel(int64_t n, T* __restrict__ y, const T* __restrict__ x, const double* s)
{
    const T       f      = static_cast<T>(1.0 / *s);
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) y[i] = f * x[i];
}

// Bound by memory on the large levels and by the launch on the small ones, so the kernel takes what would be launches and
// passes of their own: FIRST starts a recurrence (d is not read), FROM_ZERO takes x = 0 and A x = 0 as known (neither is
// read), CLEAR leaves ax zeroed for the stored operators, which add into their output. With three memsets an
// apply, and a pass that wrote A x = 0, the level-6 mixed preconditioner took 3.52 ms instead of 3.16 and the level-4
// velocity solve 18.8 ms instead of 16.5.
// STREAM: the vectors that only this kernel touches (b, d, D^-1) pass with evict-first, so that x and A x, which the
// operator reads and writes around it, stay in L2. Taken where a step's five reads and two writes exceed 64 MB, that is
// from vectors of 9.6 MB on (five of them: 48 MB, with the operator's own data more than L2 keeps): with 16-byte accesses
// the level-6 mixed preconditioner went from 3.16 to 2.97 ms, and the level-4 velocity solve, whose vectors stay in L2, did
// not change.
template <typename T>
struct alignas(16) Pack {
    T v[16 / sizeof(T)];
};
template <bool STREAM, typename T>
__device__ __forceinline__ Pack<T> load_pack(const T* p)
{
    const float4* q = reinterpret_cast<const float4*>(p);
    const float4  t = STREAM ? __ldcs(q) : *q;
    Pack<T>       r;
    memcpy(&r, &t, 16);
    return r;
}
template <bool STREAM, typename T>
__device__ __forceinline__ void store_pack(T* p, const Pack<T>& r)
{
    float4 t;
    memcpy(&t, &r, 16);
    if (STREAM)
        __stcs(reinterpret_cast<float4*>(p), t);
    else
        *reinterpret_cast<float4*>(p) = t;
}

template <typename T, bool FIRST, bool FROM_ZERO, bool CLEAR, bool STREAM>
__global__ void cheb_kernel(int64_t n, T* x, T* d, const T* b, T* ax, const T* invd, T alpha, T beta)
{
    chain_enter();
    constexpr int kV     = 16 / sizeof(T);  // n and the vectors are multiples of 64 elements
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x * kV;
    for (int64_t i = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) * kV; i < n; i += stride) {
        const Pack<T> bp = load_pack<STREAM>(b + i), ip = load_pack<STREAM>(invd + i);
        Pack<T>       ap, dp, xp;
        if (!FROM_ZERO) ap = load_pack<false>(ax + i), xp = load_pack<false>(x + i);
        if (!FIRST) dp = load_pack<STREAM>(d + i);
#pragma unroll
        for (int k = 0; k < kV; ++k) {
            const T z  = (FROM_ZERO ? bp.v[k] : bp.v[k] - ap.v[k]) * ip.v[k];
            const T dn = FIRST ? alpha * z : alpha * z + beta * dp.v[k];
            dp.v[k]    = dn;
            xp.v[k]    = FROM_ZERO ? dn : xp.v[k] + dn;
            ap.v[k]    = T(0);
        }
        store_pack<STREAM>(d + i, dp);
        store_pack<false>(x + i, xp);
        if (CLEAR) store_pack<false>(ax + i, ap);
    }
}

template <typename T>
__global__ void mul_kernel(int64_t n, T* __restrict__ y, const T* __restrict__ a, const T* __restrict__ b, T c)
{
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
        y[i] = c * (a[i] * b[i]);
}

__global__ void multi_axpy_kernel(int64_t n, double* __restrict__ x, AxpyList L)
{
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        double acc = 0.0;
        for (int k = 0; k < L.m; ++k) acc = acc + L.y[k] * L.z[k][i];
        x[i] = x[i] + acc;
    }
}

__device__ __forceinline__ uint64_t splitmix64(uint64_t z)
{
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

template <typename T>
struct CompPtrs {
    T* p[4];
};

template <typename T>
__global__ void random_kernel(int64_t n, int ncomp, CompPtrs<T> v, int nr, const int32_t* __restrict__ canon_lat,
                              uint64_t seed)
{
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int c = 0; c < ncomp; ++c)
        for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
            const uint64_t lat = static_cast<uint64_t>(i / nr), r = static_cast<uint64_t>(i % nr);
            const uint64_t gid = (static_cast<uint64_t>(canon_lat[lat]) * nr + r) * ncomp + c;
            const uint64_t z   = splitmix64(seed + (gid + 1) * 0x9E3779B97F4A7C15ull);
            const double   u   = static_cast<double>(z >> 11) * (1.0 / 9007199254740992.0);
            v.p[c][i]          = static_cast<T>(2.0 * u - 1.0);
        }
}

template <typename T>
__global__ void nonfinite_kernel(int64_t n, const T* __restrict__ a, int* flag)
{
    bool          bad    = false;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
        if (!isfinite(static_cast<double>(a[i]))) bad = true;
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicExch(flag, 1);
}

// f32 -> f64 with a non-finite flag (the FGMRES NaN/Inf check of the
// preconditioner output, fgmres.hpp:191-210, folded into the conversion).
__global__ void widen_check_kernel(int64_t n, const float* __restrict__ in, double* __restrict__ out, int* flag)
{
    bool          bad    = false;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        const double v = static_cast<double>(in[i]);
        if (!isfinite(v)) bad = true;
        out[i] = v;
    }
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicExch(flag, 1);
}

// ---------------------------------------------------------------------------
// Coarsest-grid CG in one cluster launch.
// ---------------------------------------------------------------------------
__host__ __device__ constexpr int woff_c(int w, int n, int k)
{
    constexpr int t[2][6][3] = {{{0, 0, 0}, {1, 0, 0}, {0, 1, 0}, {0, 0, 1}, {1, 0, 1}, {0, 1, 1}},
                                {{1, 1, 0}, {0, 1, 0}, {1, 0, 0}, {1, 1, 1}, {0, 1, 1}, {1, 0, 1}}};
    return t[w][n][k];
}

// Cluster-wide barrier; release / acquire at cluster scope orders the global
// memory accesses of all threads of the cluster around it.
__device__ __forceinline__ void cluster_barrier()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ unsigned cluster_rank()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cluster_ncta()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}

constexpr int kPcgThreads = 1024;
constexpr int kPcgMaxCta  = 16;

// Sum of v over the cluster; every thread returns the same value (partials are
// summed in rank order).
__device__ double cluster_sum(double v, double* partials, int& buf, unsigned rank, unsigned ncta, double* red)
{
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int k = 0; k < kPcgThreads / 32; ++k) s += red[k];
        partials[buf * kPcgMaxCta + rank] = s;
    }
    cluster_barrier();
    double tot = 0.0;
    for (unsigned k = 0; k < ncta; ++k) tot += __ldcg(partials + buf * kPcgMaxCta + k);
    buf ^= 1;
    return tot;
}

// Per-CTA view of the coarsest level: this CTA's cells [c0, c0 + cnt), their
// node indices (int32, [w * 6 + n][local cell]) and their matrices (packed
// value-major, in shared memory when they fit, else the global array).
struct PcgView {
    int            c0, cnt, cpc;
    const int32_t* node;  // shared, [12][cpc]
    const double*  mb;    // matrices of local cell lc at mb[p * ms + lc]
    int64_t        ms;
};

__device__ __forceinline__ int pidx_rt(int a, int b)
{
    const int i = a < b ? a : b, j = a < b ? b : a;
    return i * (37 - i) / 2 + (j - i);
}

// dst (zero on entry) = A src with the interface sum; ends with a cluster barrier.
__device__ void pcg_matvec(const CoarsePcgArgs& A, const PcgView& V, const double* src, double* dst, unsigned g,
                           unsigned G)
{
    const int64_t S     = A.stride;
    const int     items = 36 * V.cnt;
    for (int it = threadIdx.x; it < items; it += blockDim.x) {
        const int lc   = it % V.cnt;
        const int rest = it / V.cnt;
        const int w    = rest & 1;
        const int a    = rest >> 1;
        double    acc  = 0.0;
#pragma unroll
        for (int b = 0; b < 18; ++b) {
            const int nb = b % 6, cb = b / 6;
            acc += V.mb[static_cast<int64_t>(w * 171 + pidx_rt(a, b)) * V.ms + lc] *
                   __ldcg(src + cb * S + V.node[(w * 6 + nb) * V.cpc + lc]);
        }
        const int na = a % 6, ca = a / 6;
        atomicAdd(dst + ca * S + V.node[(w * 6 + na) * V.cpc + lc], acc);
    }
    cluster_barrier();
    const int nr     = A.nr;
    const int iitems = A.num_classes * nr * 3;
    for (int it = static_cast<int>(g); it < iitems; it += static_cast<int>(G)) {
        const int r    = it % nr;
        const int rest = it / nr;
        const int c    = rest % 3;
        const int cls  = rest / 3;
        const int b0 = A.off[cls], b1 = A.off[cls + 1];
        double*   v  = dst + c * S;
        double    s  = 0.0;
        for (int m = b0; m < b1; ++m) s += __ldcg(v + static_cast<int64_t>(A.mem[m]) * nr + r);
        for (int m = b0; m < b1; ++m) v[static_cast<int64_t>(A.mem[m]) * nr + r] = s;
    }
    cluster_barrier();
}

__global__ void __launch_bounds__(kPcgThreads, 1) coarse_pcg_kernel(CoarsePcgArgs A)
{
    extern __shared__ __align__(16) unsigned char pcg_smem[];
    __shared__ double red[kPcgThreads / 32];
    const unsigned    rank = cluster_rank(), ncta = cluster_ncta();
    const unsigned    g = rank * kPcgThreads + threadIdx.x, G = ncta * kPcgThreads;
    const int         nl = A.nl, nr = A.nr;
    const int         nc = 10 * (nl - 1) * (nl - 1) * (nr - 1);

    PcgView V;
    V.cpc = A.cells_per_cta;
    V.c0  = static_cast<int>(rank) * V.cpc;
    V.cnt = nc - V.c0 < V.cpc ? nc - V.c0 : V.cpc;
    if (V.cnt < 0) V.cnt = 0;
    int32_t* node = reinterpret_cast<int32_t*>(pcg_smem);
    for (int i = threadIdx.x; i < 12 * V.cpc; i += blockDim.x) {
        const int lc = i % V.cpc, k = i / V.cpc;
        int32_t   v  = 0;
        if (lc < V.cnt) {
            const int cell = V.c0 + lc;
            const int r    = cell % (nr - 1);
            int       t    = cell / (nr - 1);
            const int y    = t % (nl - 1);
            t /= (nl - 1);
            const int x = t % (nl - 1), d = t / (nl - 1);
            const int w = k / 6, n = k % 6;
            v = static_cast<int32_t>(
                node_index(nl, nr, d, x + woff_c(w, n, 0), y + woff_c(w, n, 1), r + woff_c(w, n, 2)));
        }
        node[i] = v;
    }
    V.node = node;
    if (A.mats_in_smem) {
        double* ms = reinterpret_cast<double*>(pcg_smem + A.node_bytes);
        for (int i = threadIdx.x; i < 342 * V.cpc; i += blockDim.x) {
            const int lc = i % V.cpc, p = i / V.cpc;
            ms[i]        = lc < V.cnt ? A.mats[static_cast<int64_t>(p) * nc + V.c0 + lc] : 0.0;
        }
        V.mb = ms;
        V.ms = V.cpc;
    } else {
        V.mb = A.mats + V.c0;
        V.ms = nc;
    }
    __syncthreads();

    const int      n = static_cast<int>(A.n), n3 = 3 * n;
    const int64_t  S = A.stride;
    const uint32_t unr = static_cast<uint32_t>(nr);
    int            buf = 0;
    for (int i = static_cast<int>(g); i < n3; i += static_cast<int>(G)) {
        const int c = i / n, j = i - c * n;
        A.ap[c * S + j] = 0.0;
    }
    cluster_barrier();
    pcg_matvec(A, V, A.x, A.ap, g, G);
    double acc = 0.0;
    for (int i = static_cast<int>(g); i < n3; i += static_cast<int>(G)) {
        const int     c = i / n, j = i - c * n;
        const int64_t o = c * S + j;
        const double  rv = __ldcg(A.b + o) - __ldcg(A.ap + o);
        A.r[o]           = rv;
        A.p[o]           = rv;
        A.ap[o]          = 0.0;
        if (A.owned[static_cast<uint32_t>(j) / unr]) acc += rv * rv;
    }
    double       rr   = cluster_sum(acc, A.partials, buf, rank, ncta, red);
    const double init = sqrt(rr);
    double       res  = init;
    int          its  = 0;
    if (!(init < A.atol)) {
        double an = rr;
        for (int it = 1; it <= A.max_iter; ++it) {
            pcg_matvec(A, V, A.p, A.ap, g, G);
            acc = 0.0;
            for (int i = static_cast<int>(g); i < n3; i += static_cast<int>(G)) {
                const int     c = i / n, j = i - c * n;
                const int64_t o = c * S + j;
                if (A.owned[static_cast<uint32_t>(j) / unr]) acc += __ldcg(A.ap + o) * __ldcg(A.p + o);
            }
            const double ad = cluster_sum(acc, A.partials, buf, rank, ncta, red);
            if (fabs(ad) < DBL_MIN) break;
            const double alpha = an / ad;
            acc                = 0.0;
            for (int i = static_cast<int>(g); i < n3; i += static_cast<int>(G)) {
                const int     c = i / n, j = i - c * n;
                const int64_t o = c * S + j;
                A.x[o]          = __ldcg(A.x + o) + alpha * __ldcg(A.p + o);
                const double rv = __ldcg(A.r + o) - alpha * __ldcg(A.ap + o);
                A.r[o]          = rv;
                if (A.owned[static_cast<uint32_t>(j) / unr]) acc += rv * rv;
            }
            rr  = cluster_sum(acc, A.partials, buf, rank, ncta, red);
            res = sqrt(rr);
            its = it;
            if (res / init <= A.rtol || res < A.atol) break;
            const double bn = rr;
            if (fabs(an) < DBL_MIN) break;
            const double beta = bn / an;
            for (int i = static_cast<int>(g); i < n3; i += static_cast<int>(G)) {
                const int     c = i / n, j = i - c * n;
                const int64_t o = c * S + j;
                A.p[o]          = __ldcg(A.r + o) + beta * __ldcg(A.p + o);
                A.ap[o]         = 0.0;
            }
            cluster_barrier();
            an = bn;
        }
    }
    if (g == 0 && A.stats) {
        A.stats[0] = static_cast<double>(its);
        A.stats[1] = init;
        A.stats[2] = res;
    }
}

// ---------------------------------------------------------------------------
// Coarsest CG over assembled rows (levels of up to a few thousand nodes, e.g. level 2). The unknowns are the unique
// nodes, so there are no interface sums and no ownership masks; CTA k of the cluster owns a slice of them, with their
// rows as 3 x 3 blocks over at most m neighbours in shared memory (77 KB a CTA at level 2), and every CTA keeps full
// copies of p and r. An iteration is A p on the own rows (16 lanes a node), the cluster-wide <A p, p>, the own part of
// r sent to all CTAs together with its <r, r>, and p = r + beta p on the full copies: two cluster barriers, both sums in
// rank order, no atomics.
//
// Bound by latency (block and cluster barriers). Over element matrices, with partial vectors summed over distributed
// shared memory and interface sums, an iteration takes longer at every size: 14.2 us against 5.5 on level (2, 2) (lateral,
// radial). Where the rows do not fit they are read from L2 (A.rows_in_smem): level (2, 3) 22.7 -> 9.0 us, (2, 4)
// 28.7 -> 14.2, (3, 2) 30.1 -> 16.3. Levels whose vectors do not fit either keep the element matrices.
// ---------------------------------------------------------------------------
constexpr int kRowLanes = 16;

__device__ double cg_cluster_sum(double v, double* red, double* buf, cg::cluster_group& cluster)
{
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    const unsigned ncta = cluster.num_blocks();
    if (threadIdx.x < 32) {
        const double s = warp_sum(red[threadIdx.x]);
        if (threadIdx.x < ncta) cluster.map_shared_rank(buf, threadIdx.x)[cluster.block_rank()] = s;
    }
    cluster.sync();
    double s = 0.0;
    for (unsigned k = 0; k < ncta; ++k) s += buf[k];
    return s;
}

__global__ void __launch_bounds__(kPcgThreads, 1) coarse_cg_rows_kernel(CoarseCgArgs A)
{
    extern __shared__ __align__(16) unsigned char pcg_smem[];
    __shared__ double red[32];
    __shared__ double sums[2][kPcgMaxCta];
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = static_cast<int>(cluster.block_rank()), ncta = static_cast<int>(cluster.num_blocks());
    const int nu = A.nodes, m = A.neighbours, npc = (nu + ncta - 1) / ncta;
    const int u0 = rank * npc, cnt = max(min(npc, nu - u0), 0);
    double*   p   = reinterpret_cast<double*>(pcg_smem);  // [node][3], full
    double*   r   = p + 3 * nu;                           // full
    double*   x   = r + 3 * nu;                           // own
    double*   ap  = x + 3 * npc;                          // own
    double*   val = ap + 3 * npc;                         // own rows [node][m][3][3]
    int32_t*  nbr = reinterpret_cast<int32_t*>(A.rows_in_smem ? val + 9 * static_cast<size_t>(m) * npc : val);

    for (int i = threadIdx.x; i < 3 * nu; i += blockDim.x) p[i] = A.x[(i % 3) * A.stride + A.rep[i / 3]];
    for (int i = threadIdx.x; i < 3 * cnt; i += blockDim.x) x[i] = A.x[(i % 3) * A.stride + A.rep[u0 + i / 3]];
    for (int i = threadIdx.x; i < m * cnt; i += blockDim.x) nbr[i] = A.nbr[static_cast<int64_t>(u0) * m + i];
    const double* rows = A.values + static_cast<int64_t>(u0) * m * 9;
    if (A.rows_in_smem) {
        for (int i = threadIdx.x; i < 9 * m * cnt; i += blockDim.x) val[i] = rows[i];
        rows = val;
    }
    __syncthreads();

    const int lane = threadIdx.x & (kRowLanes - 1), group = threadIdx.x / kRowLanes, groups = kPcgThreads / kRowLanes;
    // ap = A p on the own rows; returns this thread's part of <A p, p>
    auto product = [&]() {
        double dot = 0.0;
        for (int first = group & ~1; first < cnt; first += groups) {  // both halves of a warp make the same trips
            const int u  = first + (group & 1);
            double    y0 = 0.0, y1 = 0.0, y2 = 0.0;
            if (u < cnt)
                for (int k = lane; k < m; k += kRowLanes) {
                    const double* v  = rows + (static_cast<int64_t>(u) * m + k) * 9;
                    const double* q  = p + 3 * nbr[u * m + k];
                    const double  q0 = q[0], q1 = q[1], q2 = q[2];
                    y0 = fma(v[2], q2, fma(v[1], q1, fma(v[0], q0, y0)));
                    y1 = fma(v[5], q2, fma(v[4], q1, fma(v[3], q0, y1)));
                    y2 = fma(v[8], q2, fma(v[7], q1, fma(v[6], q0, y2)));
                }
#pragma unroll
            for (int o = kRowLanes / 2; o > 0; o >>= 1) {
                y0 += __shfl_xor_sync(0xffffffffu, y0, o);
                y1 += __shfl_xor_sync(0xffffffffu, y1, o);
                y2 += __shfl_xor_sync(0xffffffffu, y2, o);
            }
            if (lane < 3 && u < cnt) {
                const double y = lane == 0 ? y0 : (lane == 1 ? y1 : y2);
                ap[3 * u + lane] = y;
                dot += y * p[3 * (u0 + u) + lane];
            }
        }
        __syncthreads();
        return dot;
    };
    // own part of r to every CTA
    auto send_r = [&](int i, double v) {
        for (int k = 0; k < ncta; ++k) cluster.map_shared_rank(r, k)[3 * u0 + i] = v;
    };

    (void)product();
    cluster.sync();  // every CTA has started: its shared memory may be written
    double acc = 0.0;
    for (int i = threadIdx.x; i < 3 * cnt; i += blockDim.x) {
        const double v = A.b[(i % 3) * A.stride + A.rep[u0 + i / 3]] - ap[i];
        acc += v * v;
        send_r(i, v);
    }
    double       rr   = cg_cluster_sum(acc, red, sums[1], cluster);
    const double init = sqrt(rr);
    double       res  = init;
    int          its  = 0;
    for (int i = threadIdx.x; i < 3 * nu; i += blockDim.x) p[i] = r[i];
    __syncthreads();
    if (!(init < A.atol)) {
        double an = rr;
        for (int it = 1; it <= A.max_iter; ++it) {
            const double ad = cg_cluster_sum(product(), red, sums[0], cluster);
            if (fabs(ad) < DBL_MIN) break;
            const double alpha = an / ad;
            acc                = 0.0;
            for (int i = threadIdx.x; i < 3 * cnt; i += blockDim.x) {
                x[i] += alpha * p[3 * u0 + i];
                const double v = r[3 * u0 + i] - alpha * ap[i];
                acc += v * v;
                send_r(i, v);
            }
            rr  = cg_cluster_sum(acc, red, sums[1], cluster);
            res = sqrt(rr);
            its = it;
            if (res / init <= A.rtol || res < A.atol) break;
            const double bn = rr;
            if (fabs(an) < DBL_MIN) break;
            const double beta = bn / an;
            for (int i = threadIdx.x; i < 3 * nu; i += blockDim.x) p[i] = r[i] + beta * p[i];
            __syncthreads();
            an = bn;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < A.n; i += blockDim.x) {  // every copy of the own nodes
        const int u = A.uid[i] - u0;
        if (u >= 0 && u < cnt)
            for (int c = 0; c < 3; ++c) A.x[c * A.stride + i] = x[3 * u + c];
    }
    if (rank == 0 && threadIdx.x == 0 && A.stats) {
        A.stats[0] = static_cast<double>(its);
        A.stats[1] = init;
        A.stats[2] = res;
    }
    cluster.sync();  // no CTA may leave while others still write to it
}

// Rows of coarse_cg_rows_kernel, one warp a node: the wedges around all copies of the node in ascending (cell, wedge),
// the distinct nodes in the order in which they come up, then one lane per matrix entry. Sums in wedge order, so the rows
// are reproducible. Set-up: on the host the same took 2.5 ms of a solver's construction on level 2.
constexpr int kRowWidth    = 21;  // 7 lateral x 3 radial
constexpr int kRowWedges   = 12;  // 6 lateral x 2 radial
constexpr int kAssembleThr = 128;

__global__ void __launch_bounds__(kAssembleThr) coarse_rows_kernel(int nl, int nr, int nodes, int m,
                                                                   const double* __restrict__ mats,
                                                                   const int32_t* __restrict__ copy_off,
                                                                   const int32_t* __restrict__ copies,
                                                                   const int32_t* __restrict__ uid, int32_t* nbr,
                                                                   double* values, int* flag)
{
    struct Row {
        int     wedges, width;
        int     at[kRowWedges];          // 18 cell + 9 w + i: cell, wedge, the node's index in it
        int8_t  slot[kRowWedges][6];     // neighbour of each node of the wedge
        int32_t node[kRowWidth];
    };
    __shared__ Row rows[kAssembleThr / 32];
    const int      lane = threadIdx.x & 31;
    const int      u    = (blockIdx.x * kAssembleThr + threadIdx.x) / 32;
    if (u >= nodes) return;
    Row&      R  = rows[threadIdx.x / 32];
    const int o = u / nr, r = u % nr, nc = 10 * (nl - 1) * (nl - 1) * (nr - 1);
    if (lane == 0) {
        int wedges = 0, width = 0;
        for (int k = copy_off[o]; k < copy_off[o + 1]; ++k) {
            const int c = copies[k], y = c % nl, x = (c / nl) % nl, d = c / (nl * nl);
            for (int q = 0; q < 8; ++q) {  // cells (x - 1, x) x (y - 1, y) x (r - 1, r), ascending
                const int xc = x - 1 + (q >> 2), yc = y - 1 + ((q >> 1) & 1), rc = r - 1 + (q & 1);
                if (xc < 0 || xc > nl - 2 || yc < 0 || yc > nl - 2 || rc < 0 || rc > nr - 2) continue;
                const int ab = (x - xc) + 2 * (y - yc), cell = ((d * (nl - 1) + xc) * (nl - 1) + yc) * (nr - 1) + rc;
                for (int w = 0; w < 2; ++w) {
                    const int q3 = w == 0 ? ab : 3 - ab;  // lateral index of the corner in wedge w
                    if (q3 > 2) continue;
                    if (wedges == kRowWedges) {
                        *flag = 1;
                        continue;
                    }
                    R.at[wedges] = 18 * cell + 9 * w + q3 + 3 * (r - rc);
                    for (int n = 0; n < 6; ++n) {
                        const int v = uid[node_index(nl, nr, d, xc + woff_c(w, n, 0), yc + woff_c(w, n, 1),
                                                     rc + woff_c(w, n, 2))];
                        int       j = 0;
                        while (j < width && R.node[j] != v) ++j;
                        if (j == width) {
                            if (width == m) {
                                *flag = 1;
                                j = 0;
                            } else {
                                R.node[width++] = v;
                            }
                        }
                        R.slot[wedges][n] = static_cast<int8_t>(j);
                    }
                    ++wedges;
                }
            }
        }
        R.wedges = wedges;
        R.width  = width;
    }
    __syncwarp();
    for (int k = lane; k < m; k += 32) nbr[static_cast<int64_t>(u) * m + k] = k < R.width ? R.node[k] : 0;
    for (int e = lane; e < 9 * m; e += 32) {
        const int j = e / 9, a = e % 9 / 3, b = e % 3;
        double    v = 0.0;
        for (int t = 0; t < R.wedges; ++t) {
            const int cell = R.at[t] / 18, w = R.at[t] % 18 / 9, i = R.at[t] % 9;
            for (int n = 0; n < 6; ++n)
                if (R.slot[t][n] == j) {
                    const int p = min(i + 6 * a, n + 6 * b), q = max(i + 6 * a, n + 6 * b);
                    v += mats[static_cast<int64_t>(w * 171 + p * (37 - p) / 2 + (q - p)) * nc + cell];
                }
        }
        values[static_cast<int64_t>(u) * 9 * m + e] = v;
    }
}

__global__ void inject_kernel(int nlc, int nrc, const double* __restrict__ fine, double* __restrict__ coarse,
                              int reciprocal)
{
    const int     nlf = 2 * nlc - 1, nrf = 2 * nrc - 1;
    const int64_t n   = 10ll * nlc * nlc * nrc;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int r = static_cast<int>(i % nrc);
        int64_t   t = i / nrc;
        const int y = static_cast<int>(t % nlc);
        t /= nlc;
        const int    x = static_cast<int>(t % nlc);
        const int    d = static_cast<int>(t / nlc);
        const double v = fine[node_index(nlf, nrf, d, 2 * x, 2 * y, 2 * r)];
        coarse[i]      = reciprocal ? 1.0 / v : v;
    }
}

__global__ void cell_average_kernel(int nlc, int nrc, const double* __restrict__ fine, double* __restrict__ coarse)
{
    const int     nlf = 2 * nlc - 1, nrf = 2 * nrc - 1;
    const int64_t n   = 10ll * (nlc - 1) * (nlc - 1) * (nrc - 1);
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int r = static_cast<int>(i % (nrc - 1));
        int64_t   t = i / (nrc - 1);
        const int y = static_cast<int>(t % (nlc - 1));
        t /= (nlc - 1);
        const int x = static_cast<int>(t % (nlc - 1));
        const int d = static_cast<int>(t / (nlc - 1));
        double    s = 0.0;
        for (int c = 0; c < 8; ++c)
            s += fine[node_index(nlf - 1, nrf - 1, d, 2 * x + (c & 1), 2 * y + ((c >> 1) & 1), 2 * r + (c >> 2))];
        coarse[i] = 0.125 * s;
    }
}

// Strong boundary treatment of a velocity right-hand side: Dirichlet rows
// zeroed, free-slip normal components removed (n = unit lateral coordinate).
__global__ void enforce_bcs_kernel(int nl, int nr, const double* __restrict__ coords, int bc_cmb, int bc_surf,
                                   CompPtrs<double> v)
{
    const int lat = blockIdx.x * blockDim.x + threadIdx.x;
    if (lat >= 10 * nl * nl) return;
    const double* c = coords + static_cast<int64_t>(lat) * 3;
    const double  m = sqrt(c[0] * c[0] + c[1] * c[1] + c[2] * c[2]);
    const double  n[3] = {c[0] / m, c[1] / m, c[2] / m};
    for (int side = 0; side < 2; ++side) {
        const int     bc = side == 0 ? bc_cmb : bc_surf;
        const int64_t id = static_cast<int64_t>(lat) * nr + (side == 0 ? 0 : nr - 1);
        if (bc == 1) {
            for (int k = 0; k < 3; ++k) v.p[k][id] = 0.0;
        } else if (bc == 2) {
            const double dn = n[0] * v.p[0][id] + n[1] * v.p[1][id] + n[2] * v.p[2][id];
            for (int k = 0; k < 3; ++k) v.p[k][id] -= dn * n[k];
        }
    }
}

inline int grid_for(int64_t n)
{
    int64_t b = (n + kThreads - 1) / kThreads;
    if (b > 148 * 16) b = 148 * 16;
    if (b < 1) b = 1;
    return static_cast<int>(b);
}
inline int launch_status(int kernels = 1)
{
    note_launch(kernels);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace

int solver_partials_size() { return kBlocks; }

template <typename T>
int vec_dot(const VecDesc& L, const T* a, const T* b, double* out_dev, RedScratch rs, bool take_sqrt, cudaStream_t st)
{
    vdot_kernel<T><<<kBlocks, kThreads, 0, st>>>(L, a, b, rs, out_dev, take_sqrt ? 1 : 0);
    return launch_status();
}
template int vec_dot<double>(const VecDesc&, const double*, const double*, double*, RedScratch, bool, cudaStream_t);
template int vec_dot<float>(const VecDesc&, const float*, const float*, double*, RedScratch, bool, cudaStream_t);

int owned_mask(const VecDesc& L, uint64_t* mask, cudaStream_t st)
{
    const int64_t words = L.total / 64;
    owned_mask_kernel<<<static_cast<unsigned>((words + 255) / 256), 256, 0, st>>>(L, mask, words);
    return launch_status();
}

int64_t gram_schmidt_partials(int max_basis) { return 2 * static_cast<int64_t>(max_basis) * kGsBlocks; }

int gram_schmidt(const VecDesc& L, const uint64_t* mask, double* w, const BasisList& B, double* gram, int ld, double* h,
                 double* norm, RedScratch rs, cudaStream_t st)
{
    if (B.m < 1 || B.m > kMaxAxpy || L.total % 64 != 0) return -1;
    const int64_t words = L.total / 64;
    gs_dots_kernel<<<kGsBlocks, kThreads, 0, st>>>(words, mask, w, B, rs, gram, ld, h);
    gs_update_kernel<<<kGsBlocks, kThreads, 0, st>>>(words, mask, w, B, h, rs, norm);
    return launch_status(2);
}

int cg_update(const VecDesc& L, double* x, double* r, const double* p, const double* ap, const double* s_an,
              const double* s_ad, double* out, RedScratch rs, cudaStream_t st)
{
    cg_update_kernel<<<kBlocks, kThreads, 0, st>>>(L, x, r, p, ap, s_an, s_ad, rs, out);
    return launch_status();
}

int sub_scalar(int64_t n, double* v, const double* s_dev, double scale, cudaStream_t st)
{
    sub_scalar_kernel<<<grid_for(n), kThreads, 0, st>>>(n, v, s_dev, scale);
    return launch_status();
}

int p_update(int64_t n, double* p, const double* z, const double* s_num, const double* s_den, cudaStream_t st)
{
    p_update_kernel<<<grid_for(n), kThreads, 0, st>>>(n, p, z, s_num, s_den);
    return launch_status();
}

template <typename T>
int scale_by_recip(int64_t n, T* y, const T* x, const double* s_dev, cudaStream_t st)
{
    scale_recip_kernel<T><<<grid_for(n), kThreads, 0, st>>>(n, y, x, s_dev);
    return launch_status();
}
template int scale_by_recip<double>(int64_t, double*, const double*, const double*, cudaStream_t);
template int scale_by_recip<float>(int64_t, float*, const float*, const double*, cudaStream_t);

template <typename T>
int cheb_step(int64_t n, T* x, T* d, const T* b, T* ax, const T* invdiag, T alpha, T beta, bool first, bool from_zero,
              bool clear, cudaStream_t st)
{
    if (n % 64 != 0) return -1;
    const auto launch = [&](auto kernel) {
        launch_chained(kernel, grid_for(n * static_cast<int64_t>(sizeof(T)) / 16), kThreads, 0, st, n, x, d, b, ax, invdiag,
                       alpha, beta);
    };
    const auto pick = [&](auto stream) {
        constexpr bool S = decltype(stream)::value;
        if (from_zero)
            launch(clear ? cheb_kernel<T, true, true, true, S> : cheb_kernel<T, true, true, false, S>);
        else if (first)
            launch(clear ? cheb_kernel<T, true, false, true, S> : cheb_kernel<T, true, false, false, S>);
        else
            launch(clear ? cheb_kernel<T, false, false, true, S> : cheb_kernel<T, false, false, false, S>);
    };
    if (7 * n * static_cast<int64_t>(sizeof(T)) > (int64_t(64) << 20))
        pick(std::true_type{});
    else
        pick(std::false_type{});
    return launch_status();
}
template int cheb_step<double>(int64_t, double*, double*, const double*, double*, const double*, double, double, bool,
                               bool, bool, cudaStream_t);
template int cheb_step<float>(int64_t, float*, float*, const float*, float*, const float*, float, float, bool, bool, bool,
                              cudaStream_t);

template <typename T>
int vec_mul(int64_t n, T* y, const T* a, const T* b, T c, cudaStream_t st)
{
    mul_kernel<T><<<grid_for(n), kThreads, 0, st>>>(n, y, a, b, c);
    return launch_status();
}
template int vec_mul<double>(int64_t, double*, const double*, const double*, double, cudaStream_t);
template int vec_mul<float>(int64_t, float*, const float*, const float*, float, cudaStream_t);

int multi_axpy(int64_t n, double* x, const AxpyList& list, cudaStream_t st)
{
    if (list.m < 0 || list.m > kMaxAxpy) return -1;
    if (list.m == 0) return 0;
    multi_axpy_kernel<<<grid_for(n), kThreads, 0, st>>>(n, x, list);
    return launch_status();
}

template <typename T>
int random_fill(int64_t n, int ncomp, T* const* comps, int nr, const int32_t* canon_lat, uint64_t seed,
                cudaStream_t st)
{
    if (ncomp < 1 || ncomp > 4) return -1;
    CompPtrs<T> v{};
    for (int c = 0; c < ncomp; ++c) v.p[c] = comps[c];
    random_kernel<T><<<grid_for(n), kThreads, 0, st>>>(n, ncomp, v, nr, canon_lat, seed);
    return launch_status();
}
template int random_fill<double>(int64_t, int, double* const*, int, const int32_t*, uint64_t, cudaStream_t);
template int random_fill<float>(int64_t, int, float* const*, int, const int32_t*, uint64_t, cudaStream_t);

template <typename T>
int flag_nonfinite(int64_t n, const T* a, int* flag_dev, cudaStream_t st)
{
    nonfinite_kernel<T><<<grid_for(n), kThreads, 0, st>>>(n, a, flag_dev);
    return launch_status();
}
template int flag_nonfinite<double>(int64_t, const double*, int*, cudaStream_t);
template int flag_nonfinite<float>(int64_t, const float*, int*, cudaStream_t);

int widen_check(int64_t n, const float* in, double* out, int* flag_dev, cudaStream_t st)
{
    widen_check_kernel<<<grid_for(n), kThreads, 0, st>>>(n, in, out, flag_dev);
    return launch_status();
}

namespace {
// cluster size (16 when the device allows non-portable clusters of this
// kernel with the given shared memory, else 8)
template <typename K>
int pcg_cluster_size(K kernel, size_t smem)
{
    int size = 8;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
        cudaLaunchConfig_t  cfg = {};
        cudaLaunchAttribute at[1];
        at[0].id               = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = kPcgMaxCta;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.gridDim            = dim3(kPcgMaxCta);
        cfg.blockDim           = dim3(kPcgThreads);
        cfg.dynamicSmemBytes   = smem;
        cfg.attrs              = at;
        cfg.numAttrs           = 1;
        int nclusters          = 0;
        if (cudaOccupancyMaxActiveClusters(&nclusters, kernel, &cfg) == cudaSuccess && nclusters > 0)
            size = kPcgMaxCta;
    }
    cudaGetLastError();
    return size;
}

constexpr size_t kPcgSmemLimit = 200 * 1024;

// Launch configuration of a coarsest level, decided once per level size and device (function attributes and
// occupancy queries stay out of launches, so the launch can be captured in a graph).
struct PcgConfig {
    int    cs = 0, cpc = 0, in_smem = 0;
    size_t node_bytes = 0, smem = 0;
};

int pcg_config(int nc, PcgConfig& out)
{
    static std::mutex                               mu;
    static std::map<std::pair<int, int>, PcgConfig> cache;
    std::lock_guard<std::mutex>                     lock(mu);
    int                                             dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return -2;
    const auto key = std::make_pair(dev, nc);
    auto       it  = cache.find(key);
    if (it != cache.end()) {
        out = it->second;
        return 0;
    }
    PcgConfig c;
    auto      layout = [&](int cs) {
        c.cs         = cs;
        c.cpc        = (nc + cs - 1) / cs;
        c.node_bytes = (static_cast<size_t>(48) * c.cpc + 15) / 16 * 16;
        c.smem       = c.node_bytes + static_cast<size_t>(342 * 8) * c.cpc;
        c.in_smem    = c.smem <= kPcgSmemLimit ? 1 : 0;
        if (!c.in_smem) c.smem = c.node_bytes;
    };
    layout(kPcgMaxCta);
    if (cudaFuncSetAttribute(coarse_pcg_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(kPcgSmemLimit)) != cudaSuccess) {
        cudaGetLastError();
        return -2;
    }
    if (pcg_cluster_size(coarse_pcg_kernel, c.smem) != kPcgMaxCta) layout(8);
    if (c.node_bytes > kPcgSmemLimit) return -1;
    cache[key] = c;
    out        = c;
    return 0;
}

// The same for the row kernel: cluster size, bytes, rows in shared memory or read from L2. cs = 0 where not even the
// vectors fit.
int rows_config(int nodes, int neighbours, PcgConfig& out)
{
    static std::mutex                                    mu;
    static std::map<std::tuple<int, int, int>, PcgConfig> cache;
    std::lock_guard<std::mutex>                          lock(mu);
    int                                                  dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return -2;
    const auto key = std::make_tuple(dev, nodes, neighbours);
    auto       it  = cache.find(key);
    if (it != cache.end()) {
        out = it->second;
        return 0;
    }
    PcgConfig c;
    auto      layout = [&](int cs) {
        const size_t npc  = static_cast<size_t>((nodes + cs - 1) / cs);
        const size_t vecs = sizeof(double) * (6 * static_cast<size_t>(nodes) + 6 * npc), list = sizeof(int32_t) * npc * neighbours;
        const size_t rows = sizeof(double) * 9 * npc * neighbours;
        c.in_smem         = vecs + list + rows <= kPcgSmemLimit ? 1 : 0;
        c.smem            = vecs + list + (c.in_smem ? rows : 0);
        c.cs              = c.smem <= kPcgSmemLimit ? cs : 0;
    };
    layout(kPcgMaxCta);
    if (c.cs != 0) {
        if (cudaFuncSetAttribute(coarse_cg_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(kPcgSmemLimit)) != cudaSuccess) {
            cudaGetLastError();
            return -2;
        }
        if (pcg_cluster_size(coarse_cg_rows_kernel, c.smem) != kPcgMaxCta) layout(8);
    }
    cache[key] = c;
    out        = c;
    return 0;
}

template <typename K, typename Args>
int launch_cluster(K kernel, const Args& args, const PcgConfig& c, cudaStream_t st)
{
    cudaLaunchConfig_t  cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id               = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = c.cs;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.gridDim            = dim3(c.cs);
    cfg.blockDim           = dim3(kPcgThreads);
    cfg.dynamicSmemBytes   = c.smem;
    cfg.stream             = st;
    cfg.attrs              = at;
    cfg.numAttrs           = 1;
    note_launch();
    if (cudaLaunchKernelEx(&cfg, kernel, args) != cudaSuccess) {
        cudaGetLastError();
        return -2;
    }
    return 0;
}
}  // namespace

int coarse_pcg_prepare(int nl, int nr)
{
    PcgConfig c;
    return pcg_config(10 * (nl - 1) * (nl - 1) * (nr - 1), c);
}

int coarse_pcg(const CoarsePcgArgs& args_in, cudaStream_t st)
{
    CoarsePcgArgs args = args_in;
    PcgConfig     c;
    const int     rc = pcg_config(10 * (args.nl - 1) * (args.nl - 1) * (args.nr - 1), c);
    if (rc != 0) return rc;
    args.cells_per_cta = c.cpc;
    args.node_bytes    = static_cast<int>(c.node_bytes);
    args.mats_in_smem  = c.in_smem;
    return launch_cluster(coarse_pcg_kernel, args, c, st);
}

bool coarse_cg_rows_fit(int nodes, int neighbours)
{
    PcgConfig c;
    return rows_config(nodes, neighbours, c) == 0 && c.cs != 0;
}

int coarse_cg_row_width(int nl, int nr) { return (nl > 2 ? 7 : 6) * std::min(nr, 3); }

int coarse_cg_rows_assemble(int nl, int nr, int nodes, int m, const double* mats, const int32_t* copy_off,
                            const int32_t* copies, const int32_t* uid, int32_t* nbr, double* values, int* flag,
                            cudaStream_t st)
{
    if (m < 1 || m > kRowWidth) return -1;
    coarse_rows_kernel<<<(nodes * 32 + kAssembleThr - 1) / kAssembleThr, kAssembleThr, 0, st>>>(
        nl, nr, nodes, m, mats, copy_off, copies, uid, nbr, values, flag);
    return launch_status();
}

int coarse_cg_rows(const CoarseCgArgs& args_in, cudaStream_t st)
{
    CoarseCgArgs args = args_in;
    PcgConfig    c;
    const int    rc = rows_config(args.nodes, args.neighbours, c);
    if (rc != 0) return rc;
    if (c.cs == 0) return -1;
    args.rows_in_smem = c.in_smem;
    return launch_cluster(coarse_cg_rows_kernel, args, c, st);
}

int coarse_pcg_partials_size() { return 2 * kPcgMaxCta; }

int enforce_velocity_bcs(int nl, int nr, const double* coords, int bc_cmb, int bc_surf, double* const* v,
                         cudaStream_t st)
{
    CompPtrs<double> p{};
    for (int k = 0; k < 3; ++k) p.p[k] = v[k];
    const int n = 10 * nl * nl;
    enforce_bcs_kernel<<<(n + 127) / 128, 128, 0, st>>>(nl, nr, coords, bc_cmb, bc_surf, p);
    return launch_status();
}

int coefficient_inject(int nlc, int nrc, const double* fine, double* coarse, bool reciprocal, cudaStream_t st)
{
    inject_kernel<<<grid_for(10ll * nlc * nlc * nrc), kThreads, 0, st>>>(nlc, nrc, fine, coarse, reciprocal ? 1 : 0);
    return launch_status();
}

int cell_coefficient_average(int nlc, int nrc, const double* fine, double* coarse, cudaStream_t st)
{
    cell_average_kernel<<<grid_for(10ll * nlc * nlc * nrc), kThreads, 0, st>>>(nlc, nrc, fine, coarse);
    return launch_status();
}

}  // namespace tn
