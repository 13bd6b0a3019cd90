// memLS NS linear solver on the device (flowsolver/src/memLS.f90).
//
// Layout: node-major vectors (dof, nNo) exactly as memLS's R(dof, nNo); block
// matrices split as DEPART does (memLS.f90:1612-1679) into mK (9, nnz),
// mG (3, nnz), mD (3, nnz), mL (nnz) and Gt (3, nnz).
//
// Two precisions share one implementation, templated on the matrix storage
// type M and the GMRES basis type B:
//   * FP64 (M = B = double): the plain path, same arithmetic as memLS.
//   * mixed (M = B = float): every inner Krylov matvec reads FP32 matrices
//     and the GMRES basis is FP32; FP64 is kept for the NSSOLVER outer
//     vectors and Gram system, every dot product / norm (FP64 accumulation),
//     the Givens rotations and back substitution, the CG recurrences, and a
//     final FP64 defect R - A x with iterative refinement.
//
// Kernels are HBM-bound: block SpMVs use four lanes per block row with four
// blocks per lane issued together; dot products and norms use a single-pass
// grid reduction whose last block sums the per-block partials in a fixed
// order (deterministic).  CGRAD runs as one persistent cooperative kernel per
// call: on the explicitly formed Schur operator (schur.cu) where the pattern
// allows, else on the two-product kernel below; GMRES as one per call, with
// its restarts, Givens rotations and back substitution, or, in the FP32-tangent
// mode, one per restart cycle.  The 2i x 2i Gram system (GE) and the outer
// iteration run on the host in FP64 on scalars copied back once per outer
// iteration.
//
// Modified Gram-Schmidt is fused: kernel j subtracts h(j-1) u_{j-1} from w and
// accumulates <w, u_j> in the same pass.
#include <cooperative_groups.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>

#include "common.cuh"
#include "gridred.cuh"
#include "memls.cuh"

namespace crimson {

// ---------------------------------------------------------------------------
// Small helpers
// ---------------------------------------------------------------------------
template <typename T>
struct V4;
template <>
struct V4<double> {
    using type = double4;
};
template <>
struct V4<float> {
    using type = float4;
};

__device__ __forceinline__ double4 ldg4(const double4* p) {
    const double2 lo = __ldg(reinterpret_cast<const double2*>(p));
    const double2 hi = __ldg(reinterpret_cast<const double2*>(p) + 1);
    return make_double4(lo.x, lo.y, hi.x, hi.y);
}
__device__ __forceinline__ float4 ldg4(const float4* p) { return __ldg(p); }
// Streaming (evict-first) loads for matrix streams that are read once per
// pass: they leave the L2 to the vectors and node records the same kernel
// gathers and re-reads (measured: the persistent CG 14% / 9% faster in
// FP32 / FP64 on the 4M-tet cylinder, the GMRES SpMV 8% in FP32).
__device__ __forceinline__ double4 ldcs4(const double4* p) {
    const double2 lo = __ldcs(reinterpret_cast<const double2*>(p));
    const double2 hi = __ldcs(reinterpret_cast<const double2*>(p) + 1);
    return make_double4(lo.x, lo.y, hi.x, hi.y);
}
__device__ __forceinline__ float4 ldcs4(const float4* p) { return __ldcs(p); }
template <typename T>
__device__ __forceinline__ typename V4<T>::type mk4(T a, T b, T c, T d);
template <>
__device__ __forceinline__ double4 mk4<double>(double a, double b, double c, double d) {
    return make_double4(a, b, c, d);
}
template <>
__device__ __forceinline__ float4 mk4<float>(float a, float b, float c, float d) {
    return make_float4(a, b, c, d);
}

// ---------------------------------------------------------------------------
// Reductions: partial sums per block -> last block sums them in block order.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void grid_reduce_finish(double bsum, double* part, unsigned int* ticket, double* out,
                                                   double* smem) {
    __shared__ bool am_last;
    if (threadIdx.x == 0) {
        part[blockIdx.x] = bsum;
        __threadfence();
        unsigned int t = atomicAdd(ticket, 1u);
        am_last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (am_last) {
        __threadfence();
        double s = 0.0;
        for (int b = threadIdx.x; b < gridDim.x; b += blockDim.x) s += ((volatile double*)part)[b];
        s = block_sum(s, smem);
        if (threadIdx.x == 0) {
            *out = s;
            *ticket = 0u;
        }
    }
}

static int red_grid(long long n) {
    int g = grid_for(n, 256, 8);
    return g > RedScratch::kMaxBlocks ? RedScratch::kMaxBlocks : g;
}

// out = <u, v> (FP64 accumulation)
template <typename U, typename V>
__global__ void k_dot(const U* __restrict__ u, const V* __restrict__ v, long long n, double* part,
                      unsigned int* ticket, double* out) {
    __shared__ double sm[32];
    double s = 0.0;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        s += (double)u[t] * (double)v[t];
    s = block_sum(s, sm);
    grid_reduce_finish(s, part, ticket, out, sm);
}

// MGS step: w -= (*hprev) * uprev (if uprev), then out = <w, uj>  (uj may be w -> squared norm)
template <typename B>
__global__ void k_mgs(B* w, const B* __restrict__ uprev, const double* __restrict__ hprev, const B* uj, long long n,
                      double* part, unsigned int* ticket, double* out) {
    __shared__ double sm[32];
    const double h = uprev ? *hprev : 0.0;
    double s = 0.0;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
         t += (long long)gridDim.x * blockDim.x) {
        double wv = (double)w[t];
        if (uprev) {
            wv = (double)(B)(wv - h * (double)uprev[t]);
            w[t] = (B)wv;
        }
        s += wv * (uj == w ? wv : (double)uj[t]);
    }
    s = block_sum(s, sm);
    grid_reduce_finish(s, part, ticket, out, sm);
}

// y = y + a*x
template <typename X, typename Y>
__global__ void k_axpy(double a, const X* __restrict__ x, Y* __restrict__ y, long long n) {
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        y[t] = (Y)((double)y[t] + a * (double)x[t]);
}

// y = x / d (d on device; the reference divides)
template <typename B>
__global__ void k_divide(const B* x, const double* __restrict__ dptr, B* y, long long n, int take_sqrt) {
    double d = *dptr;
    if (take_sqrt) d = sqrt(d);
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        y[t] = (B)((double)x[t] / d);
}

// z = x - y
template <typename A, typename Bt, typename C>
__global__ void k_sub(const A* x, const Bt* y, C* z, long long n) {
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        z[t] = (C)((double)x[t] - (double)y[t]);
}

// X += sum_j U_j y_j  (U_j at stride n), y on device
template <typename B>
__global__ void k_multi_axpy(double* __restrict__ X, const B* __restrict__ U, const double* __restrict__ yv, int m,
                             long long n) {
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        double xv = X[t];
        for (int j = 0; j < m; ++j) xv = xv + (double)U[(size_t)j * n + t] * yv[j];
        X[t] = xv;
    }
}

__global__ void k_scale(double a, double* __restrict__ x, long long n) {
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        x[t] = a * x[t];
}

template <typename T, typename S>
__global__ void k_convert(const S* __restrict__ in, T* __restrict__ out, long long n) {
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        out[t] = (T)in[t];
}

// ---------------------------------------------------------------------------
// Block SpMVs (SPARMULVV/VS/SV/SS, memLS.f90:2024-2236).
// Four lanes per block row; each lane handles blocks j = s + lane + 4k and
// issues kUnroll of them together (column index, matrix values, gathered
// vector entries), so 16 independent loads per row are in flight instead of
// one dependent col -> x chain.  Matrix data is read through the read-only
// path (__ldg); evict-first loads measured slower on this pattern.
// ---------------------------------------------------------------------------
constexpr int kLanes = 4;
constexpr int kUnroll = 4;

__device__ __forceinline__ double group_sum(double v) {
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v;
}

// Rows handled by this thread's lane group: r = r0 + threadIdx.x / kLanes,
// r0 block-uniform so every lane of a warp reaches the shuffles.
#define CR_ROW_LOOP(n)                                                                          \
    const int lane = threadIdx.x & (kLanes - 1);                                                \
    const long long ngrp = (long long)gridDim.x * (blockDim.x / kLanes);                        \
    for (long long r0 = (long long)blockIdx.x * (blockDim.x / kLanes); r0 < (n); r0 += ngrp) { \
        const long long r = r0 + threadIdx.x / kLanes;                                          \
        const bool rv = r < (n);

// Unrolled visit of the blocks of row r: j and c defined for the body; ok marks valid blocks.
#define CR_ROW_BLOCKS(rowptr, col, ...)                                              \
    if (rv) {                                                                         \
        const int rs_ = (rowptr)[r], re_ = (rowptr)[r + 1];                           \
        for (int b0_ = rs_ + lane; b0_ < re_; b0_ += kLanes * kUnroll) {              \
            int cj_[kUnroll];                                                         \
            _Pragma("unroll") for (int k_ = 0; k_ < kUnroll; ++k_) {                  \
                const int j_ = b0_ + k_ * kLanes;                                     \
                cj_[k_] = __ldg((col) + (j_ < re_ ? j_ : b0_));                       \
            }                                                                         \
            _Pragma("unroll") for (int k_ = 0; k_ < kUnroll; ++k_) {                  \
                const int j0_ = b0_ + k_ * kLanes;                                    \
                const bool ok = j0_ < re_;                                            \
                const size_t j = (size_t)(ok ? j0_ : b0_);                            \
                const int c = cj_[k_];                                                \
                __VA_ARGS__                                                           \
            }                                                                         \
        }                                                                             \
    }

// KU = K U, K (9, nnz), U/KU (3, n)
template <typename M, typename IN, typename OUT>
__global__ void __launch_bounds__(256) k_spmv_vv3(const int* __restrict__ rowptr, const int* __restrict__ col,
                                                  const M* __restrict__ K, const IN* __restrict__ U,
                                                  OUT* __restrict__ KU, int n) {
    CR_ROW_LOOP(n)
    double a0 = 0.0, a1 = 0.0, a2 = 0.0;
    CR_ROW_BLOCKS(rowptr, col, {
        const M* k = K + 9 * j;
        const IN* u = U + 3 * (size_t)c;
        const double u0 = (double)u[0], u1 = (double)u[1], u2 = (double)u[2];
        const double k0 = (double)__ldg(k + 0), k1 = (double)__ldg(k + 1), k2 = (double)__ldg(k + 2),
                     k3 = (double)__ldg(k + 3), k4 = (double)__ldg(k + 4), k5 = (double)__ldg(k + 5),
                     k6 = (double)__ldg(k + 6), k7 = (double)__ldg(k + 7), k8 = (double)__ldg(k + 8);
        if (ok) {
            a0 += k0 * u0 + k1 * u1 + k2 * u2;
            a1 += k3 * u0 + k4 * u1 + k5 * u2;
            a2 += k6 * u0 + k7 * u1 + k8 * u2;
        }
    })
    a0 = group_sum(a0);
    a1 = group_sum(a1);
    a2 = group_sum(a2);
    if (rv && lane == 0) {
        KU[3 * r + 0] = (OUT)a0;
        KU[3 * r + 1] = (OUT)a1;
        KU[3 * r + 2] = (OUT)a2;
    }
    }
}

// KU(i) = sum K(:,j).U(:,col)  (3 -> 1), or minuend(i) less it
template <typename M, typename IN, typename OUT>
__global__ void __launch_bounds__(256) k_spmv_vs3(const int* __restrict__ rowptr, const int* __restrict__ col,
                                                  const M* __restrict__ K, const IN* __restrict__ U,
                                                  OUT* __restrict__ KU, const double* __restrict__ minuend, int n) {
    CR_ROW_LOOP(n)
    double a = 0.0;
    CR_ROW_BLOCKS(rowptr, col, {
        const M* k = K + 3 * j;
        const IN* u = U + 3 * (size_t)c;
        const double t = (double)__ldg(k) * (double)u[0] + (double)__ldg(k + 1) * (double)u[1] +
                         (double)__ldg(k + 2) * (double)u[2];
        if (ok) a += t;
    })
    a = group_sum(a);
    if (rv && lane == 0) KU[r] = (OUT)(minuend ? minuend[r] - a : a);
    }
}

// KU(:,i) = sum K(:,j) U(col)  (1 -> 3); with rest, rest = minuend - KU
template <typename M, typename IN, typename OUT>
__global__ void __launch_bounds__(256) k_spmv_sv3(const int* __restrict__ rowptr, const int* __restrict__ col,
                                                  const M* __restrict__ K, const IN* __restrict__ U,
                                                  OUT* __restrict__ KU, const double* __restrict__ minuend,
                                                  double* __restrict__ rest, int n) {
    CR_ROW_LOOP(n)
    double a0 = 0.0, a1 = 0.0, a2 = 0.0;
    CR_ROW_BLOCKS(rowptr, col, {
        const M* k = K + 3 * j;
        const double u = (double)U[c];
        const double k0 = (double)__ldg(k), k1 = (double)__ldg(k + 1), k2 = (double)__ldg(k + 2);
        if (ok) {
            a0 += k0 * u;
            a1 += k1 * u;
            a2 += k2 * u;
        }
    })
    a0 = group_sum(a0);
    a1 = group_sum(a1);
    a2 = group_sum(a2);
    if (rv && lane == 0) {
        KU[3 * r + 0] = (OUT)a0;
        KU[3 * r + 1] = (OUT)a1;
        KU[3 * r + 2] = (OUT)a2;
        if (rest) {
            rest[3 * r + 0] = minuend[3 * r + 0] - a0;
            rest[3 * r + 1] = minuend[3 * r + 1] - a1;
            rest[3 * r + 2] = minuend[3 * r + 2] - a2;
        }
    }
    }
}

// KU = K U, scalar
template <typename M, typename IN, typename OUT>
__global__ void __launch_bounds__(256) k_spmv_ss(const int* __restrict__ rowptr, const int* __restrict__ col,
                                                 const M* __restrict__ K, const IN* __restrict__ U,
                                                 OUT* __restrict__ KU, int n) {
    CR_ROW_LOOP(n)
    double a = 0.0;
    CR_ROW_BLOCKS(rowptr, col, {
        const double t = (double)__ldg(K + j) * (double)U[c];
        if (ok) a += t;
    })
    a = group_sum(a);
    if (rv && lane == 0) KU[r] = (OUT)a;
    }
}

// (G^T v)(c) = sum over row c of G(:, trans j) . v(:, col j)   (transposed SPARMULVS)
template <typename M>
__global__ void __launch_bounds__(256) k_spmv_vs3_trans(const int* __restrict__ rowptr, const int* __restrict__ col,
                                                        const int* __restrict__ trans, const M* __restrict__ G,
                                                        const double* __restrict__ V, double* __restrict__ out, int n) {
    CR_ROW_LOOP(n)
    double acc = 0.0;
    CR_ROW_BLOCKS(rowptr, col, {
        const M* g = G + 3 * (size_t)trans[j];
        const double* v = V + 3 * (size_t)c;
        const double t = (double)g[0] * v[0] + (double)g[1] * v[1] + (double)g[2] * v[2];
        if (ok) acc += t;
    })
    acc = group_sum(acc);
    if (rv && lane == 0) out[r] = acc;
    }
}

// ---------------------------------------------------------------------------
// Sliced ELL copy of the pattern for the SpMVs inside the Krylov loops
// (GMRES's K products and the CG's G / {Gt, L} products).
// Rows are grouped in slices of 32 (one warp); a slice is stored column by
// column with width w = its longest row, so position of entry k of row r is
// sp[r / 32] + r % 32 + 32 k.  One thread per row: every load of column
// indices and matrix values is a fully coalesced 128-byte warp access, with
// no row-pointer -> column dependency; entries are summed in CSR order.
// Padding entries carry zero values and a valid column (the row itself;
// 0 for the rows past n of the last slice), so they add exactly +0.
// K is stored per component (structure of arrays, stride npad); the CG's
// operands as one 4-vector per entry: {G0, G1, G2, column} (one load gives
// the column and the values) and {Gt0, Gt1, Gt2, L}.  Converted once per NSSOLVER call,
// read ~10^3 times.
// ---------------------------------------------------------------------------
constexpr int kSlice = 32;
constexpr int kSellUnroll = 8;

// Visit the entries of row r, U at a time: pos (size_t) and c (int) defined
// for the body.
#define CR_SELL_ROW_U(U, sp, scol, r, ...)                                              \
    {                                                                                    \
        const int s_ = (r) >> 5;                                                         \
        const int p0_ = __ldg((sp) + s_);                                                \
        const int w_ = (__ldg((sp) + s_ + 1) - p0_) >> 5;                                \
        const int base_ = p0_ + ((r) & (kSlice - 1));                                    \
        for (int k0_ = 0; k0_ < w_; k0_ += (U)) {                                        \
            int cc_[(U)];                                                                \
            _Pragma("unroll") for (int u_ = 0; u_ < (U); ++u_) cc_[u_] =                 \
                (k0_ + u_ < w_) ? __ldg((scol) + base_ + kSlice * (k0_ + u_)) : 0;       \
            _Pragma("unroll") for (int u_ = 0; u_ < (U); ++u_) {                         \
                if (k0_ + u_ < w_) {                                                     \
                    const size_t pos = (size_t)base_ + (size_t)kSlice * (k0_ + u_);      \
                    const int c = cc_[u_];                                               \
                    __VA_ARGS__                                                          \
                }                                                                        \
            }                                                                            \
        }                                                                                \
    }
#define CR_SELL_ROW(sp, scol, r, ...) CR_SELL_ROW_U(kSellUnroll, sp, scol, r, __VA_ARGS__)
// Entries per stage of the CG's software-pipelined row loops, phases A (G P)
// and B: the matrix records of the next stage are loaded while the current
// stage's gathers are in flight.  Two stages are live, and across a barrier
// the first one, within the 64 registers of two 512-thread blocks per SM: FP32
// 4 and 3 (5 and 5 spill across the barriers; per iteration on 118k nodes
// 21.2 us against 22.0, and 4 and 4 21.6), FP64 2 and 2.
template <typename M>
struct CgStageA {
    static constexpr int value = sizeof(M) == 4 ? 4 : 2;
};
template <typename M>
struct CgStage {
    static constexpr int value = sizeof(M) == 4 ? 3 : 2;
};

// KU = K U on the sliced copy: K as {K0..K3} and {K4..K7} 4-vectors (npad
// each, one 16/32-byte load apiece) and K8 (npad); U / KU (3, n).
template <typename M, typename IN, typename OUT>
__global__ void __launch_bounds__(256) k_sell_vv3(const int* __restrict__ sp, const int* __restrict__ scol,
                                                  const M* __restrict__ Ks, long long npad,
                                                  const IN* __restrict__ U, OUT* __restrict__ KU, int n) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
        double a0 = 0.0, a1 = 0.0, a2 = 0.0;
        CR_SELL_ROW(sp, scol, r, {
            const IN* u = U + 3 * (size_t)c;
            const double u0 = (double)__ldg(u), u1 = (double)__ldg(u + 1), u2 = (double)__ldg(u + 2);
            const auto ka = ldcs4(reinterpret_cast<const typename V4<M>::type*>(Ks) + pos);
            const auto kb = ldcs4(reinterpret_cast<const typename V4<M>::type*>(Ks + 4 * npad) + pos);
            const double k0 = (double)ka.x, k1 = (double)ka.y, k2 = (double)ka.z, k3 = (double)ka.w,
                         k4 = (double)kb.x, k5 = (double)kb.y, k6 = (double)kb.z, k7 = (double)kb.w,
                         k8 = (double)__ldcs(Ks + 8 * npad + pos);
            a0 = a0 + k0 * u0 + k1 * u1 + k2 * u2;
            a1 = a1 + k3 * u0 + k4 * u1 + k5 * u2;
            a2 = a2 + k6 * u0 + k7 * u1 + k8 * u2;
        })
        KU[3 * (size_t)r + 0] = (OUT)a0;
        KU[3 * (size_t)r + 1] = (OUT)a1;
        KU[3 * (size_t)r + 2] = (OUT)a2;
    }
}

// Column index of every sliced position (pads: the row, or 0 past n).
__global__ void k_sell_cols(const int* __restrict__ rowptr, const int* __restrict__ col, const int* __restrict__ sp,
                            int n, int nrows_pad, int* __restrict__ scol) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < nrows_pad; r += gridDim.x * blockDim.x) {
        const int s = r >> 5;
        const int w = (sp[s + 1] - sp[s]) >> 5;
        const int base = sp[s] + (r & (kSlice - 1));
        const int rs = r < n ? rowptr[r] : 0;
        const int len = r < n ? rowptr[r + 1] - rs : 0;
        for (int k = 0; k < w; ++k) scol[base + kSlice * k] = k < len ? col[rs + k] : (r < n ? r : 0);
    }
}

// Largest |col - row| of a CSR pattern (atomicMax into *out).
__global__ void k_max_offset(const int* __restrict__ rowptr, const int* __restrict__ col, int n, int* out) {
    int m = 0;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x)
        for (int j = rowptr[r]; j < rowptr[r + 1]; ++j) m = max(m, abs(col[j] - r));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// Scaled split matrices (CSR, type M) -> sliced copies: K as two 4-vector
// arrays and one scalar array (npad each), and for the two-product CG (Gs not
// null) G (3, npad) per component, {Gt0, Gt1, Gt2, L} (npad).
template <typename M>
__global__ void k_to_sell(const int* __restrict__ rowptr, const int* __restrict__ sp, int n,
                          const double* __restrict__ mK, const double* __restrict__ mG, const double* __restrict__ Gt,
                          const double* __restrict__ mL, long long npad, M* __restrict__ Ks, M* __restrict__ Gs,
                          typename V4<M>::type* __restrict__ GLs) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
        const size_t base = (size_t)sp[r >> 5] + (r & (kSlice - 1));
        const int rs = rowptr[r], re = rowptr[r + 1];
        for (int j = rs; j < re; ++j) {
            const size_t pos = base + (size_t)kSlice * (j - rs);
            const size_t jj = (size_t)j;
            reinterpret_cast<typename V4<M>::type*>(Ks)[pos] =
                mk4<M>((M)mK[9 * jj], (M)mK[9 * jj + 1], (M)mK[9 * jj + 2], (M)mK[9 * jj + 3]);
            reinterpret_cast<typename V4<M>::type*>(Ks + 4 * npad)[pos] =
                mk4<M>((M)mK[9 * jj + 4], (M)mK[9 * jj + 5], (M)mK[9 * jj + 6], (M)mK[9 * jj + 7]);
            Ks[8 * npad + pos] = (M)mK[9 * jj + 8];
            if (!Gs) continue;
#pragma unroll
            for (int q = 0; q < 3; ++q) Gs[q * npad + pos] = (M)mG[3 * jj + q];
            GLs[pos] = mk4<M>((M)Gt[3 * jj], (M)Gt[3 * jj + 1], (M)Gt[3 * jj + 2], (M)mL[jj]);
        }
    }
}

// ---------------------------------------------------------------------------
// CGRAD as one persistent cooperative kernel (memLS.f90:367-430): on patterns
// that the explicit operator (schur.cu) excludes, and in the FP32-tangent mode.
//
// Per iteration three grid-wide barriers: (A) P = R + beta P formed on the
// fly while computing GP = G P, plus the coupled-face dots w_f . P; (B)
// SP = L P - Gt GP - sum_f coef_f (w_f . P) z_f and <P, SP>; (C) X += alpha P,
// R -= alpha SP, |R|^2.  The coupled-face (Sherman-Morrison) term of
// ADDBCMUL(PRE) is applied through the precomputed vectors w_f = G^T valM_f
// and z_f = Gt valM_f: Gt (GP + coef valM (valM . GP)) = Gt GP + coef (w.P) z
// -- exact.  Node records keep every gather to one aligned sector:
// recA = {R, P_prev} (16 B, FP64) read in phase A, recB = {GP, P} read in
// phase B, stored in the matrix type M (32 B FP64 / 16 B FP32: with FP32
// matrices the matvec operands are rounded to FP32 as the matrices are,
// while P itself stays FP64 for the updates); matrix entries G per
// component (three coalesced streams) and {Gt0, Gt1, Gt2, L}; the column
// indices block-resident in shared memory where they fit (CgCols).  Partial sums are written per block
// and summed in block order by every block after the barrier
// (deterministic, identical in all blocks).  Node records written by other
// blocks in an earlier phase are read with ordinary (L1-cached) loads: the
// grid barrier's acquire fence orders them after those writes, and the
// neighbour gathers of one block hit the same lines many times.  The matrix
// streams use evict-first loads (each value is read once per phase), so the
// node records and per-row vectors (~40 MB on the 4M-tet cylinder) stay in
// the 126 MB L2 from one phase to the next.  The loop
// is bounded by mItr.  X, R, P, SP, the recurrences and all dot products
// are FP64 in both precisions; M is the storage type of G, Gt, L and of
// the gathered copy of {GP, P}.
// ---------------------------------------------------------------------------
constexpr int kMaxCoupled = 8;
// 512-thread blocks, two per SM: half the blocks of 256-thread blocks at
// every grid barrier and block-order reduction (measured 2% per iteration).
constexpr int kCgThreads = 512;

template <typename M>
struct CgArgs {
    const int* sp;    // sliced pattern: slice offsets
    const int* scol;  // sliced pattern: columns (read when the columns are not block-resident)
    long long npad;
    int n;
    const M* G;                      // sliced G per component: G0 at [0, npad), G1, G2 (stride npad)
    const typename V4<M>::type* GL;  // sliced (npad) {Gt0, Gt1, Gt2, L}
    double* X;
    double2* recA;  // (n) {R, P of the previous iteration}
    typename V4<M>::type* recB;  // (n) {GP0, GP1, GP2, P} rounded to M: the gathered copy
    double* Pd;                  // (n) P in FP64 for the updates
    double* SP;
    int nface;
    const double* w;  // (nface, n)
    const double* z;  // (nface, n)
    double coef[kMaxCoupled];
    const double* rr;       // squared initial norm
    double relTol, absTol;
    int mItr;
    double* part;  // 3 regions of kCgPartStride * gridDim
    double* out;   // err, errO, i, suc, initial norm
};
constexpr int kCgPartStride = kMaxCoupled + 2;

__device__ __forceinline__ double sum_partials(const double* part, int k, double* sm) {
    double s = 0.0;
    for (int b = threadIdx.x; b < gridDim.x; b += blockDim.x) s += __ldcg(part + (size_t)b * kCgPartStride + k);
    return block_sum(s, sm);
}

// Column source of the CG row loops.  Block-resident (kRes): every block
// copies the columns of its own rows into shared memory once per launch, as
// 16-bit offsets col - row, and the iterations read no column index from
// HBM (4 B per entry and phase).  A warp's rows are whole slices (32 rows),
// so a warp's columns are the concatenation of its slices' column ranges in
// sliced order; entry k of a row sits at off + 32 k + lane, where off
// advances by the slice's length after each row.  Otherwise the columns are
// read from the sliced pattern.
template <bool kRes>
struct CgCols {
    const int* scol;
    const short* res;  // this warp's resident offsets (kRes)
    int off;           // offset of the current row's slice within res
    int lane;
    __device__ __forceinline__ int col(int r, int base, int k) const {
        if (kRes) return r + (int)res[off + kSlice * k + lane];
        return __ldg(scol + base + kSlice * k);
    }
    __device__ __forceinline__ void next_row(int w) {
        if (kRes) off += kSlice * w;
    }
};

// Fill this block's resident column offsets; returns this warp's base.
__device__ int cg_fill_cols(const int* __restrict__ sp, const int* __restrict__ scol, int n, short* res) {
    __shared__ int woff[kCgThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int s0 = (blockIdx.x * kCgThreads + wid * kSlice) / kSlice;
    const int sstride = gridDim.x * (kCgThreads / kSlice);
    const int nsl = (n + kSlice - 1) / kSlice;
    int tot = 0;
    for (int s = s0 + lane * sstride; s < nsl; s += 32 * sstride) tot += __ldg(sp + s + 1) - __ldg(sp + s);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
    if (lane == 0) woff[wid] = tot;
    __syncthreads();
    int base = 0;
    for (int q = 0; q < wid; ++q) base += woff[q];
    int off = base;
    for (int s = s0; s < nsl; s += sstride) {
        const int p0 = __ldg(sp + s), len = __ldg(sp + s + 1) - p0;
        const int row = s * kSlice + lane;  // position p0 + j belongs to row s*32 + j%32
        for (int j = lane; j < len; j += 32) res[off + j] = row < n ? (short)(__ldg(scol + p0 + j) - row) : (short)0;
        off += len;
    }
    __syncthreads();
    return base;
}

template <int NF, typename M, bool kRes>
__global__ void __launch_bounds__(kCgThreads, 2) k_cg_persistent(CgArgs<M> a) {
    namespace cgrp = cooperative_groups;
    cgrp::grid_group grid = cgrp::this_grid();
    extern __shared__ short cg_res[];
    __shared__ double sm[32];
    const int n = a.n;
    const long long npad = a.npad;
    double* partA = a.part;
    double* partB = a.part + (size_t)gridDim.x * kCgPartStride;
    double* partC = a.part + 2 * (size_t)gridDim.x * kCgPartStride;
    const int wbase = kRes ? cg_fill_cols(a.sp, a.scol, n, cg_res) : 0;
    constexpr int U = CgStage<M>::value;
    constexpr int UA = CgStageA<M>::value;
    const int r0 = blockIdx.x * blockDim.x + threadIdx.x, rstride = gridDim.x * blockDim.x;
    // A row's slice and the first stage of its matrix entries.  They are loaded
    // before the barrier that the row's gathers wait for: the matrix does not
    // change, and the loads' latency passes under the wait (per iteration 22.3 ->
    // 21.2 us on 118k nodes, 89.1 -> 86.1 on 695k).  19 us remain on the
    // smallest meshes: three barriers with their sums, two passes over a row.
    // Barriers that carry the sums (gridred.cuh) are slower here, 27 us: each of
    // the 296 blocks polls the packets of all.
    int w = 0, base = 0;
    M g0[UA], g1[UA], g2[UA];
    int cc[UA > U ? UA : U];
    typename V4<M>::type gl[U];
    const auto zero4 = mk4<M>(M(0), M(0), M(0), M(0));
    auto slice_of = [&](int r) {
        if (r >= n) return;
        const int p0 = __ldg(a.sp + (r >> 5));
        w = (__ldg(a.sp + (r >> 5) + 1) - p0) >> 5;
        base = p0 + (r & (kSlice - 1));
    };
    auto first_a = [&](int r) {
#pragma unroll
        for (int u = 0; u < UA; ++u) {
            const bool in = r < n && u < w;
            const size_t pos = (size_t)base + kSlice * u;
            g0[u] = in ? __ldcs(a.G + pos) : M(0);
            g1[u] = in ? __ldcs(a.G + npad + pos) : M(0);
            g2[u] = in ? __ldcs(a.G + 2 * npad + pos) : M(0);
            if (!kRes) cc[u] = in ? __ldg(a.scol + pos) : r;  // resident columns are read at use
        }
    };
    auto first_b = [&](int r) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool in = r < n && u < w;
            const size_t pos = (size_t)base + kSlice * u;
            gl[u] = in ? ldcs4(a.GL + pos) : zero4;
            if (!kRes) cc[u] = in ? __ldg(a.scol + pos) : r;
        }
    };
    slice_of(r0);
    first_a(r0);
    const double norm0 = sqrt(*a.rr);
    double err = norm0 * norm0, errO = err;
    double eps = fmax(a.absTol, a.relTol * norm0);
    eps = eps * eps;
    int suc = 0, i;
    for (i = 1; i <= a.mItr; ++i) {
        if (err < eps) {
            suc = 1;
            break;
        }
        const bool first = (i == 1);
        const double beta = first ? 0.0 : err / errO;
        errO = err;
        // ---- phase A: P = R + beta P_prev (on the fly), GP = G P, w_f . P ----
        double wp[NF > 0 ? NF : 1];
#pragma unroll
        for (int f = 0; f < (NF > 0 ? NF : 1); ++f) wp[f] = 0.0;
        CgCols<kRes> cs{a.scol, cg_res, wbase, (int)(threadIdx.x & 31)};
        for (int r = r0; r < n; r += rstride) {
            double a0 = 0.0, a1 = 0.0, a2 = 0.0;
            // stage: G values and columns of UA entries; the next stage is
            // loaded before this stage's gathers
            for (int k0 = 0; k0 < w; k0 += UA) {
                M n0[UA], n1[UA], n2[UA];
                int nc[UA];
#pragma unroll
                for (int u = 0; u < UA; ++u) {
                    const bool in = k0 + UA + u < w;
                    const size_t pos = (size_t)base + kSlice * (k0 + UA + u);
                    n0[u] = in ? __ldcs(a.G + pos) : M(0);
                    n1[u] = in ? __ldcs(a.G + npad + pos) : M(0);
                    n2[u] = in ? __ldcs(a.G + 2 * npad + pos) : M(0);
                    nc[u] = (!kRes && in) ? cs.col(r, base, k0 + UA + u) : r;
                }
#pragma unroll
                for (int u = 0; u < UA; ++u) {
                    if (k0 + u < w) {
                        const double2 rp = a.recA[kRes ? cs.col(r, base, k0 + u) : cc[u]];
                        const double pc = first ? rp.x : rp.x + beta * rp.y;
                        a0 = a0 + (double)g0[u] * pc;
                        a1 = a1 + (double)g1[u] * pc;
                        a2 = a2 + (double)g2[u] * pc;
                    }
                }
#pragma unroll
                for (int u = 0; u < UA; ++u) {
                    g0[u] = n0[u];
                    g1[u] = n1[u];
                    g2[u] = n2[u];
                    if (!kRes) cc[u] = nc[u];
                }
            }
            cs.next_row(w);
            if (r + rstride < n) {
                slice_of(r + rstride);
                first_a(r + rstride);
            }
            const double2 rr = a.recA[r];
            const double pr = first ? rr.x : rr.x + beta * rr.y;
            a.recB[r] = mk4<M>((M)a0, (M)a1, (M)a2, (M)pr);
            a.Pd[r] = pr;
#pragma unroll
            for (int f = 0; f < NF; ++f)
                if (f < a.nface) wp[f] += a.w[(size_t)f * n + r] * pr;
        }
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            if (f < a.nface) {
                double t = block_sum(wp[f], sm);
                if (threadIdx.x == 0) partA[(size_t)blockIdx.x * kCgPartStride + f] = t;
            }
        }
        slice_of(r0);
        first_b(r0);
        grid.sync();
        double cS[NF > 0 ? NF : 1];
#pragma unroll
        for (int f = 0; f < NF; ++f) cS[f] = f < a.nface ? a.coef[f] * sum_partials(partA, f, sm) : 0.0;
        // ---- phase B: SP = L P - Gt GP - sum_f cS_f z_f ; <P, SP> ----
        double dsum = 0.0;
        CgCols<kRes> cb{a.scol, cg_res, wbase, (int)(threadIdx.x & 31)};
        for (int r = r0; r < n; r += rstride) {
            double lp = 0.0, gg = 0.0;
            for (int k0 = 0; k0 < w; k0 += U) {
                int ccn[U];  // next stage
                typename V4<M>::type gln[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const bool in = k0 + U + u < w;
                    ccn[u] = (!kRes && in) ? cb.col(r, base, k0 + U + u) : r;
                    gln[u] = in ? ldcs4(a.GL + base + kSlice * (k0 + U + u)) : zero4;
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (k0 + u < w) {
                        const auto q = a.recB[kRes ? cb.col(r, base, k0 + u) : cc[u]];
                        lp = lp + (double)gl[u].w * (double)q.w;
                        gg = gg + (double)gl[u].x * (double)q.x + (double)gl[u].y * (double)q.y +
                             (double)gl[u].z * (double)q.z;
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (!kRes) cc[u] = ccn[u];
                    gl[u] = gln[u];
                }
            }
            cb.next_row(w);
            if (r + rstride < n) {
                slice_of(r + rstride);
                first_b(r + rstride);
            }
#pragma unroll
            for (int f = 0; f < NF; ++f)
                if (f < a.nface) gg += cS[f] * a.z[(size_t)f * n + r];
            const double v = lp - gg;
            a.SP[r] = v;
            dsum += a.Pd[r] * v;
        }
        dsum = block_sum(dsum, sm);
        if (threadIdx.x == 0) partB[(size_t)blockIdx.x * kCgPartStride] = dsum;
        grid.sync();
        const double alpha = errO / sum_partials(partB, 0, sm);
        // ---- phase C: X += alpha P, R -= alpha SP, |R|^2 ; recA = {R, P} ----
        double rs = 0.0;
        for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
             t += (long long)gridDim.x * blockDim.x) {
            const double pv = a.Pd[t];
            a.X[t] = a.X[t] + alpha * pv;
            const double rv = a.recA[t].x - alpha * a.SP[t];
            a.recA[t] = make_double2(rv, pv);
            rs += rv * rv;
        }
        rs = block_sum(rs, sm);
        if (threadIdx.x == 0) partC[(size_t)blockIdx.x * kCgPartStride] = rs;
        slice_of(r0);
        first_a(r0);
        grid.sync();
        const double e2 = sqrt(sum_partials(partC, 0, sm));
        err = e2 * e2;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.out[0] = err;
        a.out[1] = errO;
        a.out[2] = (double)i;
        a.out[3] = (double)suc;
        a.out[4] = norm0;
    }
}

// recA = {R, 0}
__global__ void k_cg_init(const double* __restrict__ R, double2* __restrict__ recA, int n) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) recA[t] = make_double2(R[t], 0.0);
}

// ext = valM scattered into a (3, n) vector
__global__ void k_face_ext(const int* __restrict__ glob, const double* __restrict__ valM, int fdof, int nsd, int nNoF,
                           double* __restrict__ ext) {
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < nNoF; a += gridDim.x * blockDim.x)
        for (int i = 0; i < nsd; ++i) ext[3 * (size_t)glob[a] + i] = valM[(size_t)fdof * a + i];
}

// ---------------------------------------------------------------------------
// ADDBCMUL pieces (memLS.f90:206-268): S = <valM, X> over face nodes; Y += S*coef*valM
// ---------------------------------------------------------------------------
template <typename V>
__global__ void k_face_dot(const int* __restrict__ glob, const double* __restrict__ valM, int fdof, int nsd,
                           int nNoF, const V* __restrict__ X, int dof, double* part, unsigned int* ticket,
                           double* out) {
    __shared__ double sm[32];
    double s = 0.0;
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < nNoF; a += gridDim.x * blockDim.x) {
        const int Ac = glob[a];
        for (int i = 0; i < nsd; ++i) s += valM[(size_t)fdof * a + i] * (double)X[(size_t)dof * Ac + i];
    }
    s = block_sum(s, sm);
    grid_reduce_finish(s, part, ticket, out, sm);
}

template <typename V>
__global__ void k_face_axpy(const int* __restrict__ glob, const double* __restrict__ valM, int fdof, int nsd,
                            int nNoF, const double* Sptr, double coef, V* __restrict__ Y, int dof) {
    const double S = coef * *Sptr;
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < nNoF; a += gridDim.x * blockDim.x) {
        const int Ac = glob[a];
        for (int i = 0; i < nsd; ++i)
            Y[(size_t)dof * Ac + i] = (V)((double)Y[(size_t)dof * Ac + i] + valM[(size_t)fdof * a + i] * S);
    }
}

// ---------------------------------------------------------------------------
// PRECOND (memLS.f90:1763-1943) pieces
// ---------------------------------------------------------------------------
// W from the diagonal blocks of Val (dof = 4, row-major 16 per block)
__global__ void k_w_from_val(double* __restrict__ Val, const int* __restrict__ diag, double* __restrict__ W, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double* v = Val + 16 * (size_t)diag[i];
        for (int d = 0; d < 4; ++d) {
            double w = v[5 * d];
            if (w == 0.0) {
                w = 1.0;
                v[5 * d] = 1.0;
            }
            W[4 * (size_t)i + d] = 1.0 / sqrt(fabs(w));
        }
    }
}

// Tangent block j as ElmGMR produced it: FP64 lhsK (9, nnz) / lhsP (4, nnz),
// or FP32 records of 16 floats (K(9), P(4), pads) when rec is not null.
struct TangentIn {
    const double* lhsK;
    const double* lhsP;
    const float* rec;
    __device__ __forceinline__ double K(size_t j, int t) const {
        return rec ? (double)rec[16 * j + t] : lhsK[9 * j + t];
    }
    __device__ __forceinline__ double P(size_t j, int t) const {
        return rec ? (double)rec[16 * j + 9 + t] : lhsP[4 * j + t];
    }
};

// W from lhsK / lhsP diagonals (fused SolFlow path; Val4 diagonal = K11,K22,K33,C)
__global__ void k_w_from_lhs(TangentIn T, const int* __restrict__ diag, double* __restrict__ W, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const size_t k = (size_t)diag[i];
        double w[4] = {T.K(k, 0), T.K(k, 4), T.K(k, 8), T.P(k, 3)};
        for (int d = 0; d < 4; ++d) {
            double v = w[d] == 0.0 ? 1.0 : w[d];
            W[4 * (size_t)i + d] = 1.0 / sqrt(fabs(v));
        }
    }
}

// W(1:i, glob) *= val  (Dirichlet faces)
__global__ void k_w_dirichlet(const int* __restrict__ glob, const double* __restrict__ val, int fdof, int ni, int nNoF,
                              double* __restrict__ W) {
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < nNoF; a += gridDim.x * blockDim.x) {
        const int Ac = glob[a];
        for (int i = 0; i < ni; ++i) W[4 * (size_t)Ac + i] = W[4 * (size_t)Ac + i] * val[(size_t)fdof * a + i];
    }
}

// Row then column scaling of Val (16 per block) + zero-diagonal fix + DEPART split
__global__ void k_scale_split_val(double* __restrict__ Val, const int* __restrict__ rowptr, const int* __restrict__ col,
                                  const int* __restrict__ diag, const double* __restrict__ W, int n,
                                  double* __restrict__ mK, double* __restrict__ mG, double* __restrict__ mD,
                                  double* __restrict__ mL) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
        const double* wr = W + 4 * (size_t)r;
        for (int j = rowptr[r]; j < rowptr[r + 1]; ++j) {
            const double* wc = W + 4 * (size_t)col[j];
            double* v = Val + 16 * (size_t)j;
            double t[16];
            for (int a = 0; a < 4; ++a)
                for (int b = 0; b < 4; ++b) t[4 * a + b] = (v[4 * a + b] * wr[a]) * wc[b];
            if (j == diag[r])
                for (int a = 0; a < 4; ++a)
                    if (t[5 * a] == 0.0) t[5 * a] = 1.0;
            for (int q = 0; q < 16; ++q) v[q] = t[q];
            double* k = mK + 9 * (size_t)j;
            k[0] = t[0]; k[1] = t[1]; k[2] = t[2];
            k[3] = t[4]; k[4] = t[5]; k[5] = t[6];
            k[6] = t[8]; k[7] = t[9]; k[8] = t[10];
            mG[3 * (size_t)j + 0] = t[3];
            mG[3 * (size_t)j + 1] = t[7];
            mG[3 * (size_t)j + 2] = t[11];
            mD[3 * (size_t)j + 0] = t[12];
            mD[3 * (size_t)j + 1] = t[13];
            mD[3 * (size_t)j + 2] = t[14];
            mL[j] = t[15];
        }
    }
}

// Gt(:, l) = -mG(:, trans(l))  (DEPART's transpose search, memLS.f90:1664-1675)
__global__ void k_gt(const double* __restrict__ mG, const int* __restrict__ trans, long long nnz, double* __restrict__ Gt) {
    for (long long l = (long long)blockIdx.x * blockDim.x + threadIdx.x; l < nnz; l += (long long)gridDim.x * blockDim.x) {
        const size_t j = (size_t)trans[l];
        Gt[3 * l + 0] = -mG[3 * j + 0];
        Gt[3 * l + 1] = -mG[3 * j + 1];
        Gt[3 * l + 2] = -mG[3 * j + 2];
    }
}

// Fused SolFlow pack + PRECOND scaling + DEPART from lhsK / lhsP:
//   Val4 rows 1-3 cols 1-3 = lhsK, col 4 rows 1-3 = -lhsP(1:3) of the
//   transposed block, row 4 cols 1-3 = lhsP(1:3), (4,4) = lhsP(4)
//   (solfar.f90:217-232), scaled by W(row) W(col) and split.
__global__ void k_scale_split_lhs(TangentIn T, const int* __restrict__ rowptr, const int* __restrict__ col,
                                  const int* __restrict__ diag, const int* __restrict__ trans,
                                  const double* __restrict__ W, int n, double* __restrict__ mK,
                                  double* __restrict__ mG, double* __restrict__ mD, double* __restrict__ mL) {
    // 16 lanes per row, one entry per lane: the block reads and writes of a
    // row are contiguous across the lanes
    const int sub = threadIdx.x & 15;
    const int ngroup = (gridDim.x * blockDim.x) >> 4;
    for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 4; r < n; r += ngroup) {
        const double* wr = W + 4 * (size_t)r;
        const int dg = diag[r];
        for (int j = rowptr[r] + sub; j < rowptr[r + 1]; j += 16) {
            const double* wc = W + 4 * (size_t)col[j];
            const size_t jj = (size_t)j, jt = (size_t)trans[j];
            const double Pj[4] = {T.P(jj, 0), T.P(jj, 1), T.P(jj, 2), T.P(jj, 3)};
            const double Pt[3] = {T.P(jt, 0), T.P(jt, 1), T.P(jt, 2)};
            double* k = mK + 9 * (size_t)j;
            for (int a = 0; a < 3; ++a)
                for (int b = 0; b < 3; ++b) {
                    double v = T.K(jj, 3 * a + b);
                    if (j == dg && a == b && v == 0.0) v = 1.0;
                    double t = (v * wr[a]) * wc[b];
                    if (j == dg && a == b && t == 0.0) t = 1.0;
                    k[3 * a + b] = t;
                }
            for (int a = 0; a < 3; ++a) mG[3 * (size_t)j + a] = (-Pt[a] * wr[a]) * wc[3];
            for (int b = 0; b < 3; ++b) mD[3 * (size_t)j + b] = (Pj[b] * wr[3]) * wc[b];
            double v = Pj[3];
            if (j == dg && v == 0.0) v = 1.0;
            double t = (v * wr[3]) * wc[3];
            if (j == dg && t == 0.0) t = 1.0;
            mL[j] = t;
        }
    }
}

// R = W*R  (node-major, dof 4), and R = R*W afterwards
__global__ void k_mul(double* __restrict__ R, const double* __restrict__ W, long long n) {
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        R[t] = W[t] * R[t];
}

// split (4, n) into (3, n) and (n), and merge back
__global__ void k_split4(const double* __restrict__ R, double* __restrict__ Rm, double* __restrict__ Rc, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        Rm[3 * (size_t)i + 0] = R[4 * (size_t)i + 0];
        Rm[3 * (size_t)i + 1] = R[4 * (size_t)i + 1];
        Rm[3 * (size_t)i + 2] = R[4 * (size_t)i + 2];
        Rc[i] = R[4 * (size_t)i + 3];
    }
}
__global__ void k_merge4(double* __restrict__ R, const double* __restrict__ Rm, const double* __restrict__ Rc, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        R[4 * (size_t)i + 0] = Rm[3 * (size_t)i + 0];
        R[4 * (size_t)i + 1] = Rm[3 * (size_t)i + 1];
        R[4 * (size_t)i + 2] = Rm[3 * (size_t)i + 2];
        R[4 * (size_t)i + 3] = Rc[i];
    }
}

// face%valM = face%val * W  (coupled faces)
__global__ void k_valm(const int* __restrict__ glob, const double* __restrict__ val, double* __restrict__ valM, int fdof,
                       int ni, int nNoF, const double* __restrict__ W) {
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < nNoF; a += gridDim.x * blockDim.x)
        for (int i = 0; i < ni; ++i)
            valM[(size_t)fdof * a + i] = val[(size_t)fdof * a + i] * W[4 * (size_t)glob[a] + i];
}

// Defect of the scaled NS system: D4 = R4 - [K u + G p ; D u + L p] given
// KU = K u (+ coupling), GP = G p, DU = D u, LP = L p (all FP64).
__global__ void k_defect4(const double* __restrict__ R4, const double* __restrict__ KU,
                          const double* __restrict__ GPm, const double* __restrict__ DU,
                          const double* __restrict__ LP, double* __restrict__ D4, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        for (int d = 0; d < 3; ++d)
            D4[4 * (size_t)i + d] = R4[4 * (size_t)i + d] - (KU[3 * (size_t)i + d] + GPm[3 * (size_t)i + d]);
        D4[4 * (size_t)i + 3] = R4[4 * (size_t)i + 3] - (DU[i] + LP[i]);
    }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
static double now_s() {
    return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

// device scalar slots
enum {
    kSlotDot = 0,
    kSlotNrm = 1,
    kSlotErr = 2,
    kSlotErrO = 3,
    kSlotDen = 4,
    kSlotFace = 8,      // up to 16 faces
    kSlotCg = 24,       // persistent CG outputs (5)
    kSlotGm = 32,       // persistent GMRES outputs (6), two calls
    kSlotH = 64,        // Hessenberg column (sD + 1)
    kSlotY = 64 + 512,  // back-substitution coefficients
    kSlotGram = 64 + 1024,
    kScalTotal = 64 + 1024 + 4096 + 1024
};

struct Ctx {
    crimson_lhs* L;
    cudaStream_t s;
    double* sc(int i) { return L->scal.p + i; }
    int sync_scal(int first, int count) {
        CR_CUDA(cudaMemcpyAsync(L->hscal + first, L->scal.p + first, sizeof(double) * count, cudaMemcpyDeviceToHost, s));
        CR_CUDA(cudaStreamSynchronize(s));
        return CRIMSON_OK;
    }
    template <typename U, typename V>
    void dot(const U* u, const V* v, long long n, int slot) {
        launch(k_dot<U, V>, red_grid(n), 256, 0, s, u, v, n, L->red.part.p, L->red.ticket.p, sc(slot));
    }
    int spmv_grid() const { return grid_for((long long)L->nNo * kLanes, 256, 8); }
    template <typename M, typename IN, typename OUT>
    void vv3(const M* K, const IN* U, OUT* KU) {
        launch(k_spmv_vv3<M, IN, OUT>, spmv_grid(), 256, 0, s, L->rowptr, L->col, K, U, KU, L->nNo);
    }
    template <typename M, typename IN, typename OUT>
    void vs3(const M* K, const IN* U, OUT* KU, const double* minuend = nullptr) {
        launch(k_spmv_vs3<M, IN, OUT>, spmv_grid(), 256, 0, s, L->rowptr, L->col, K, U, KU, minuend, L->nNo);
    }
    template <typename M, typename IN, typename OUT>
    void sv3(const M* K, const IN* U, OUT* KU, const double* minuend = nullptr, double* rest = nullptr) {
        launch(k_spmv_sv3<M, IN, OUT>, spmv_grid(), 256, 0, s, L->rowptr, L->col, K, U, KU, minuend, rest, L->nNo);
    }
    template <typename M, typename IN, typename OUT>
    void ss(const M* K, const IN* U, OUT* KU) {
        launch(k_spmv_ss<M, IN, OUT>, spmv_grid(), 256, 0, s, L->rowptr, L->col, K, U, KU, L->nNo);
    }
    template <typename M, typename IN, typename OUT>
    void vv3s(const M* Ks, const IN* U, OUT* KU) {
        launch(k_sell_vv3<M, IN, OUT>, grid_for(L->nNo, 256, 8), 256, 0, s, (const int*)L->sell_ptr.p,
               (const int*)L->sell_col.p, Ks, L->npad, U, KU, L->nNo);
    }
    bool any_coupled() const {
        for (auto& f : L->face)
            if (f.coupledFlag) return true;
        return false;
    }
    // ADDBCMUL on nsd-dof vectors: all face dots first (on X), then all updates of Y
    template <typename VX, typename VY>
    void addbcmul(int op, int dof, const VX* X, VY* Y) {
        int k = 0;
        for (auto& f : L->face) {
            if (f.coupledFlag) {
                int nsd = std::min(f.dof, dof);
                // a few nodes per thread: the face dot is a chain of gathers
                int g = (f.nNo + 4 * 128 - 1) / (4 * 128);
                g = std::max(1, std::min(g, (int)RedScratch::kMaxBlocks));
                launch(k_face_dot<VX>, g, 128, 0, s, f.glob.p, f.valM.p, f.dof, nsd, f.nNo, X, dof, L->red.part.p,
                       L->red.ticket.p, sc(kSlotFace + k));
            }
            ++k;
        }
        k = 0;
        for (auto& f : L->face) {
            if (f.coupledFlag) {
                int nsd = std::min(f.dof, dof);
                double coef = (op == 0) ? f.res : -f.res / (1.0 + f.res * f.nS);
                launch(k_face_axpy<VY>, grid_for(f.nNo, 256), 256, 0, s, f.glob.p, f.valM.p, f.dof, nsd, f.nNo,
                       (const double*)sc(kSlotFace + k), coef, Y, dof);
            }
            ++k;
        }
    }
};

// ---------------------------------------------------------------------------
// GMRES (memLS.f90:681-788) as one persistent cooperative kernel per call:
// restarts, Arnoldi iterations, Givens rotations, exit tests, back
// substitution and the update of X, without a host round trip.
//
// Per iteration: (P1) w = K u_{i-1} on the sliced K, with the coupled-face
// dots S0_f = valM_f . u_{i-1} and T_f = valM_f . w of ADDBCMUL; (MGS j) the
// face terms of ADDBCMUL (op 0, then op 1 with S1_f = T_f + sum_g coef0_g S0_g
// (valM_f . valM_g)) folded into the first pass, then w -= h_{j-1} u_{j-2} and
// h_j = <w, u_{j-1}>; (norm) w -= h_i u_{i-1} and |w|^2; every block applies
// the Givens rotations to the new Hessenberg column (identical arithmetic on
// identical sums, so the exit test agrees); u_i = w / h_{i+1}.
//
// Small and middle meshes are bound by the i + 3 grid barriers of an
// iteration.  Each of them carries its reduction (gridred.cuh), and only the
// last one, which publishes u_i to the neighbours' gathers, orders data.  Four
// lanes share a block row (a row's entries are four dependent load stages for
// one lane), lane c < 3 then owns component c: its w and the basis vector of
// the running pass stay in registers (kSlots values each), and the next
// pass's vector is loaded before the barrier that the pass waits for.  Meshes
// of more than 150,000 nodes (8 values per thread) are bound by the
// streams of K and the basis: one lane per row, w in memory (kSlots = 0).
// ---------------------------------------------------------------------------
// Threads of a block: 128 registers each for the register form, 64 for the
// streaming one.
constexpr int gm_threads(int slots) { return slots > 0 ? 512 : 1024; }
constexpr int kGmMaxSD = 64;
constexpr int kGmVals = 1 + 2 * kMaxCoupled;

template <typename M, typename B>
struct GmArgs {
    const int* sp;
    const int* scol;
    long long npad;
    int n;
    const M* Ks;          // sliced K: {K0..K3} (npad), {K4..K7} (npad), K8 (npad)
    B* u;                 // basis, vector k at u + k n3 (k = 0..sD)
    long long n3;
    int sD, mItr;
    double relTol, absTol;
    const double* R;      // right side (n3)
    double* X;            // solution (n3)
    int nface;            // coupled faces
    const int* fptr;      // (n + 1) entries of node r: fent[fptr[r] .. fptr[r + 1])
    const int* fent;      // entry ids grouped by node
    const int* fface;     // (entries) face of the entry
    const double* fval;   // (entries, 3) valM of the entry
    const double* gram;   // (nface, nface) valM_f . valM_g (diagonal: nS)
    double coef0[kMaxCoupled], coef1[kMaxCoupled];
    ulonglong2* pk;       // 2 regions of kGmVals packets per block
    unsigned long long epoch;
    double* out;          // iterations, suc (-1: a wait ran out), iNorm, fNorm, norm before the last cycle, nothing to do
};

__device__ __forceinline__ double quad_sum(double v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    return v;
}

// Entries k0, k0 + step, ... of row r of K times U.
template <int UN, typename M, typename IN>
__device__ __forceinline__ void gm_row(const int* __restrict__ sp, const int* __restrict__ scol,
                                       const M* __restrict__ Ks, long long npad, int r, int k0, int step, const IN* U,
                                       double a[3]) {
    const int p0 = __ldg(sp + (r >> 5));
    const int w = (__ldg(sp + (r >> 5) + 1) - p0) >> 5;
    const int base = p0 + (r & (kSlice - 1));
    for (int k = k0; k < w; k += step * UN) {
        int c[UN];
#pragma unroll
        for (int q = 0; q < UN; ++q) c[q] = k + step * q < w ? __ldg(scol + base + kSlice * (k + step * q)) : r;
#pragma unroll
        for (int q = 0; q < UN; ++q)
            if (k + step * q < w) {
                const size_t pos = (size_t)base + (size_t)kSlice * (k + step * q);
                const IN* u = U + 3 * (size_t)c[q];
                const double u0 = (double)u[0], u1 = (double)u[1], u2 = (double)u[2];
                const auto ka = ldcs4(reinterpret_cast<const typename V4<M>::type*>(Ks) + pos);
                const auto kb = ldcs4(reinterpret_cast<const typename V4<M>::type*>(Ks + 4 * npad) + pos);
                const double k8 = (double)__ldcs(Ks + 8 * npad + pos);
                a[0] = a[0] + (double)ka.x * u0 + (double)ka.y * u1 + (double)ka.z * u2;
                a[1] = a[1] + (double)ka.w * u0 + (double)kb.x * u1 + (double)kb.y * u2;
                a[2] = a[2] + (double)kb.z * u0 + (double)kb.w * u1 + k8 * u2;
            }
    }
}

template <typename M, typename B, int kSlots>
__global__ void __launch_bounds__(gm_threads(kSlots), 1) k_gmres(const __grid_constant__ GmArgs<M, B> a) {
    constexpr bool kReg = kSlots > 0;
    constexpr int NS = kReg ? kSlots : 1;
    extern __shared__ double gm_dyn[];
    __shared__ double red[32 * kGmVals], tot[kGmVals], cf[kMaxCoupled];
    __shared__ unsigned char fpend[32 * kMaxCoupled];
    __shared__ int sdone;
    __shared__ unsigned sown;
    const int sD = a.sD, ldh = sD + 1;
    double* const H = gm_dyn;                 // (sD + 1, sD) column-major, rotated
    double* const sc = H + (size_t)ldh * sD;  // rotations
    double* const sn = sc + sD;
    double* const err = sn + sD;              // (sD + 1)
    double* const yv = err + ldh;             // (sD)
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int n = a.n;
    const int tid0 = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
    // kReg: slot s of this thread is component q of row r0 + s rs; the
    // warp-uniform bound lets every lane reach the shuffles
    const int q = kReg ? (int)(threadIdx.x & 3) : 0, r0 = kReg ? tid0 >> 2 : tid0, rs = kReg ? nth >> 2 : nth;
    unsigned long long ep = a.epoch;
    bool fail = false;
    unsigned own = 0;
    auto reduce = [&](double v, bool data) {   // one value; returns the sum
        v = warp_sum(v);
        if (lane == 0) red[wid] = v;
        fail = grid_reduce(a.pk, kGmVals, red, 0, 0u, fpend, ++ep, data, tot, fail);
        return tot[0];
    };
    // which blocks hold nodes of which face
    if (a.nface > 0) {
        if (threadIdx.x == 0) sown = 0u;
        __syncthreads();
        unsigned m = 0;
        for (int r = r0; r < n; r += rs)
            for (int k = a.fptr[r]; k < a.fptr[r + 1]; ++k) m |= 1u << a.fface[a.fent[k]];
        m = __reduce_or_sync(0xffffffffu, m);
        if (lane == 0 && m) atomicOr(&sown, m);
        __syncthreads();
        own = sown;
        if (lane == 0) red[wid] = wid == 0 ? (double)own : 0.0;
        fail = grid_reduce(a.pk, kGmVals, red, 0, 0u, fpend, ++ep, false, tot, fail);
        const ulonglong2* pk = a.pk + (size_t)(ep & 1) * kGmVals * gridDim.x;
        for (int f = wid; f < a.nface; f += blockDim.x >> 5) {
            unsigned b = 0;
#pragma unroll
            for (int j = 0; j < kGrPolls; ++j)
                if (lane + 32 * j < (int)gridDim.x &&
                    (((unsigned)__longlong_as_double((long long)gr_load(pk + lane + 32 * j).x) >> f) & 1))
                    b |= 1u << j;
            fpend[32 * f + lane] = (unsigned char)b;
        }
        __syncthreads();
    }
    // face sums of value pairs (v0, v1): per-thread accumulation over the
    // entries of its rows, then one barrier.  body(fe, f, c, row, &x0, &x1)
    // adds an entry's component c.
    auto face_reduce = [&](auto&& body) {
        for (int f = 0; f < a.nface; ++f) {
            double x0 = 0.0, x1 = 0.0;
            if ((own >> f) & 1) {
                int s = 0;
                for (int r = r0; r < n; r += rs, ++s)
                    for (int k = a.fptr[r]; k < a.fptr[r + 1]; ++k) {
                        const int fe = a.fent[k];
                        if (a.fface[fe] == f) body(fe, r, s, x0, x1);
                    }
            }
            x0 = warp_sum(x0);
            x1 = warp_sum(x1);
            if (lane == 0) {
                red[32 * (1 + 2 * f) + wid] = x0;
                red[32 * (2 + 2 * f) + wid] = x1;
            }
        }
        if (lane == 0) red[wid] = 0.0;
        fail = grid_reduce(a.pk, kGmVals, red, a.nface, own, fpend, ++ep, false, tot, fail);
    };
    double w[NS];    // kReg: this thread's values of the running vector (rounded to B)
#pragma unroll
    for (int s = 0; s < NS; ++s) w[s] = 0.0;
    auto at = [&](int s) { return 3 * (size_t)(r0 + s * rs) + q; };                  // kReg: index of slot s
    auto has = [&](int s) { return q < 3 && r0 + s * rs < n; };
    B* wm = a.u;     // memory of the running vector (kSlots = 0)
    // component c of row r of the running vector (kReg: slot s)
    auto wval = [&](int r, int s, int c) {
        if (!kReg) return (double)wm[3 * (size_t)r + c];
        double v = 0.0;
#pragma unroll
        for (int z = 0; z < NS; ++z)
            if (z == s) v = w[z];
        return v;
    };
    // w += sum_f cf_f valM_f at the faces' nodes: each face's term rounded to B
    // (ADDBCMUL), or their sum (the closed form of its two passes)
    auto face_add = [&](bool each) {
        if (!own) return;
        int s = 0;
        for (int r = r0; r < n; r += rs, ++s) {
            const int k0 = a.fptr[r], k1 = a.fptr[r + 1];
            if (k1 == k0) continue;
            for (int c = kReg ? q : 0; c < (kReg ? min(q + 1, 3) : 3); ++c) {
                double v = wval(r, s, c), add = 0.0;
                for (int k = k0; k < k1; ++k) {
                    const int fe = a.fent[k];
                    const double x = a.fval[3 * (size_t)fe + c] * cf[a.fface[fe]];
                    if (each)
                        v = (double)(B)(v + x);
                    else
                        add += x;
                }
                if (!each) v = (double)(B)(v + add);
                if (kReg) {
#pragma unroll
                    for (int z = 0; z < NS; ++z)
                        if (z == s) w[z] = v;
                } else {
                    wm[3 * (size_t)r + c] = (B)v;
                }
            }
        }
    };
    // one component per lane (kReg) or all three: adds val . f over them
    auto dot3 = [&](int fe, auto&& f) {
        const double* v = a.fval + 3 * (size_t)fe;
        if (kReg) return q < 3 ? v[q] * f(q) : 0.0;
        return v[0] * f(0) + v[1] * f(1) + v[2] * f(2);
    };

    double eps = 0.0, iNorm = 0.0, fNorm = 0.0, dBase = 0.0;
    int itr = 0, suc = 0, idle = 0;
    for (int l = 1; l <= a.mItr && !fail; ++l) {
        // ---- u_0: the preconditioned residual, normalized ----
        wm = a.u;
        if (l == 1) {
            if (kReg) {
#pragma unroll
                for (int s = 0; s < NS; ++s) w[s] = has(s) ? (double)(B)a.R[at(s)] : 0.0;
            } else {
                for (int r = r0; r < n; r += rs)
                    for (int c = 0; c < 3; ++c) wm[3 * (size_t)r + c] = (B)a.R[3 * (size_t)r + c];
            }
        } else {
            ++itr;
            if (kReg) {
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    const int r = r0 + s * rs;
                    double x[3] = {0.0, 0.0, 0.0};
                    if (r < n) gm_row<4>(a.sp, a.scol, a.Ks, a.npad, r, q, 4, (const double*)a.X, x);
                    const double x0 = quad_sum(x[0]), x1 = quad_sum(x[1]), x2 = quad_sum(x[2]);
                    w[s] = has(s) ? (double)(B)(q == 0 ? x0 : (q == 1 ? x1 : x2)) : 0.0;
                }
            } else {
                for (int r = r0; r < n; r += rs) {
                    double x[3] = {0.0, 0.0, 0.0};
                    gm_row<4>(a.sp, a.scol, a.Ks, a.npad, r, 0, 1, (const double*)a.X, x);
                    for (int c = 0; c < 3; ++c) wm[3 * (size_t)r + c] = (B)x[c];
                }
            }
            if (a.nface > 0) {
                face_reduce([&](int fe, int r, int, double& x0, double&) {
                    x0 += dot3(fe, [&](int c) { return a.X[3 * (size_t)r + c]; });
                });
                if (threadIdx.x < (unsigned)a.nface) cf[threadIdx.x] = a.coef0[threadIdx.x] * tot[1 + 2 * threadIdx.x];
                __syncthreads();
                face_add(true);
            }
            if (kReg) {
#pragma unroll
                for (int s = 0; s < NS; ++s)
                    if (has(s)) w[s] = (double)(B)(a.R[at(s)] - w[s]);
            } else {
                for (int r = r0; r < n; r += rs)
                    for (int c = 0; c < 3; ++c) {
                        const size_t t = 3 * (size_t)r + c;
                        wm[t] = (B)(a.R[t] - (double)wm[t]);
                    }
            }
        }
        if (a.nface > 0) {
            face_reduce([&](int fe, int r, int s, double& x0, double&) {
                x0 += dot3(fe, [&](int c) { return wval(r, s, c); });
            });
            if (threadIdx.x < (unsigned)a.nface) cf[threadIdx.x] = a.coef1[threadIdx.x] * tot[1 + 2 * threadIdx.x];
            __syncthreads();
            face_add(true);
        }
        double d = 0.0;
        if (kReg) {
#pragma unroll
            for (int s = 0; s < NS; ++s) d += w[s] * w[s];
        } else {
            for (int r = r0; r < n; r += rs)
                for (int c = 0; c < 3; ++c) {
                    const double v = (double)wm[3 * (size_t)r + c];
                    d += v * v;
                }
        }
        const double e0 = sqrt(reduce(d, false));
        if (l == 1) {
            if (e0 <= a.absTol) {
                idle = 1;
                for (int r = r0; r < n; r += rs)
                    for (int c = kReg ? q : 0; c < (kReg ? min(q + 1, 3) : 3); ++c) a.X[3 * (size_t)r + c] = 0.0;
                break;
            }
            iNorm = fNorm = e0;
            eps = fmax(a.absTol, a.relTol * e0);
        }
        dBase = fNorm;
        if (threadIdx.x == 0) err[0] = e0;
        if (kReg) {
#pragma unroll
            for (int s = 0; s < NS; ++s)
                if (has(s)) a.u[at(s)] = (B)(w[s] / e0);
        } else {
            for (int r = r0; r < n; r += rs)
                for (int c = 0; c < 3; ++c) {
                    const size_t t = 3 * (size_t)r + c;
                    wm[t] = (B)((double)wm[t] / e0);
                }
        }
        reduce(0.0, true);
        int i;
        for (i = 1; i <= sD && !fail; ++i) {
            ++itr;
            // ---- P1: w = K u_{i-1} ----
            const B* uin = a.u + (size_t)(i - 1) * a.n3;
            wm = a.u + (size_t)i * a.n3;
            if (kReg) {
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    const int r = r0 + s * rs;
                    double x[3] = {0.0, 0.0, 0.0};
                    if (r < n) gm_row<4>(a.sp, a.scol, a.Ks, a.npad, r, q, 4, uin, x);
                    const double x0 = quad_sum(x[0]), x1 = quad_sum(x[1]), x2 = quad_sum(x[2]);
                    w[s] = has(s) ? (double)(B)(q == 0 ? x0 : (q == 1 ? x1 : x2)) : 0.0;
                }
            } else {
                for (int r = r0; r < n; r += rs) {
                    double x[3] = {0.0, 0.0, 0.0};
                    gm_row<4>(a.sp, a.scol, a.Ks, a.npad, r, 0, 1, uin, x);
                    for (int c = 0; c < 3; ++c) wm[3 * (size_t)r + c] = (B)x[c];
                }
            }
            B un[NS], up[NS];   // kReg: u_{j-1} of the pass, u_{j-2}
            if (kReg) {
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    un[s] = has(s) ? a.u[at(s)] : B(0);
                    up[s] = B(0);
                }
            }
            if (a.nface > 0) {
                face_reduce([&](int fe, int r, int s, double& x0, double& x1) {
                    x0 += dot3(fe, [&](int c) { return (double)uin[3 * (size_t)r + c]; });
                    x1 += dot3(fe, [&](int c) { return wval(r, s, c); });
                });
                if (threadIdx.x < (unsigned)a.nface) {
                    const int f = threadIdx.x;
                    double S1 = tot[2 + 2 * f];
                    for (int g = 0; g < a.nface; ++g) S1 += a.coef0[g] * tot[1 + 2 * g] * a.gram[f * a.nface + g];
                    cf[f] = a.coef0[f] * tot[1 + 2 * f] + a.coef1[f] * S1;
                }
                __syncthreads();
                face_add(false);
            }
            // ---- MGS passes j = 1..i, then the norm (j = i + 1) ----
            double* const hc = H + (size_t)(i - 1) * ldh;
            double hp = 0.0;
            for (int j = 1; j <= i + 1; ++j) {
                const bool last = j == i + 1;
                d = 0.0;
                if (kReg) {
#pragma unroll
                    for (int s = 0; s < NS; ++s) {
                        if (j > 1) w[s] = (double)(B)(w[s] - hp * (double)up[s]);
                        d += w[s] * (last ? w[s] : (double)un[s]);
                        up[s] = un[s];
                    }
                    if (j < i) {
                        const B* uj = a.u + (size_t)j * a.n3;
#pragma unroll
                        for (int s = 0; s < NS; ++s)
                            if (has(s)) un[s] = uj[at(s)];
                    }
                } else {
                    const B* uj = last ? wm : a.u + (size_t)(j - 1) * a.n3;
                    const B* uo = j > 1 ? a.u + (size_t)(j - 2) * a.n3 : wm;
                    for (int r = r0; r < n; r += rs)
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            const size_t t = 3 * (size_t)r + c;
                            double wv = (double)wm[t];
                            if (j > 1) {
                                wv = (double)(B)(wv - hp * (double)uo[t]);
                                wm[t] = (B)wv;
                            }
                            d += wv * (last ? wv : (double)__ldcs(uj + t));
                        }
                }
                hp = reduce(d, false);
                if (last) hp = sqrt(hp);
                if (threadIdx.x == 0) hc[j - 1] = hp;
            }
            // ---- Givens (memLS.f90:750-760), identical in every block ----
            if (threadIdx.x == 0) {
                double h0 = hc[0];
                for (int j = 1; j <= i - 1; ++j) {
                    const double h1 = hc[j];
                    hc[j - 1] = sc[j - 1] * h0 + sn[j - 1] * h1;
                    h0 = -sn[j - 1] * h0 + sc[j - 1] * h1;
                }
                const double t = sqrt(h0 * h0 + hc[i] * hc[i]);
                sc[i - 1] = h0 / t;
                sn[i - 1] = hc[i] / t;
                hc[i - 1] = t;
                hc[i] = 0.0;
                err[i] = -sn[i - 1] * err[i - 1];
                err[i - 1] = sc[i - 1] * err[i - 1];
                sdone = fabs(err[i]) < eps ? 1 : 0;
            }
            __syncthreads();
            if (sdone) suc = 1;
            if (sdone || i == sD) break;
            // ---- normalize ----
            if (kReg) {
#pragma unroll
                for (int s = 0; s < NS; ++s)
                    if (has(s)) a.u[(size_t)i * a.n3 + at(s)] = (B)(w[s] / hp);
            } else {
                for (int r = r0; r < n; r += rs)
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const size_t t = 3 * (size_t)r + c;
                        wm[t] = (B)((double)wm[t] / hp);
                    }
            }
            reduce(0.0, true);
        }
        if (fail) break;
        // ---- back substitution (one warp, columns from the last), X update ----
        fNorm = fabs(err[i]);
        if (wid == 0) {
            for (int k = lane; k < i; k += 32) yv[k] = err[k];
            __syncwarp();
            for (int j = i - 1; j >= 0; --j) {
                const double yj = yv[j] / H[(size_t)j * ldh + j];
                __syncwarp();
                if (lane == 0) yv[j] = yj;
                for (int k = lane; k < j; k += 32) yv[k] = yv[k] - H[(size_t)j * ldh + k] * yj;
                __syncwarp();
            }
        }
        __syncthreads();
        for (int r = r0; r < n; r += rs)
            for (int c = kReg ? q : 0; c < (kReg ? min(q + 1, 3) : 3); ++c) {
                const size_t t = 3 * (size_t)r + c;
                double xv = l == 1 ? 0.0 : a.X[t];
#pragma unroll 4
                for (int j = 0; j < i; ++j) xv = xv + (double)a.u[(size_t)j * a.n3 + t] * yv[j];
                a.X[t] = xv;
            }
        if (suc) break;
        if (l < a.mItr) reduce(0.0, true);   // the next cycle gathers X
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.out[0] = (double)itr;
        a.out[1] = fail ? -1.0 : (double)suc;
        a.out[2] = iNorm;
        a.out[3] = fNorm;
        a.out[4] = dBase;
        a.out[5] = (double)idle;
    }
}

// ---------------------------------------------------------------------------
// One restart cycle as a persistent kernel with cooperative_groups barriers,
// for the FP32-tangent mode (CRIMSON_MIXED_F32_TANGENT).  There the next
// nonlinear iteration rounds its tangent to FP32, which turns the 1e-11 by
// which any other order of summation moves a mixed solve (its basis is
// rounded to FP32 at every step) into 1e-8 of the time step's result; the
// mode keeps this kernel's order and with it its results.  Same iteration as
// k_gmres; restart residual, back substitution and X update on the host.
// ---------------------------------------------------------------------------
constexpr int kGmcThreads = 512;
constexpr int kGmPartStride = 2 * kMaxCoupled + 1;

template <typename M, typename B>
struct GmcArgs {
    const int* sp;
    const int* scol;
    long long npad;
    int n;
    const M* Ks;          // sliced K: {K0..K3} (npad), {K4..K7} (npad), K8 (npad)
    B* u;                 // basis, vector k at u + k n3 (k = 0..sD); u[0] normalized on entry
    long long n3;
    int sD;
    int nface;            // coupled faces
    const int* fptr;      // (n + 1) entries of node r: fent[fptr[r] .. fptr[r + 1])
    const int* fent;      // entry ids grouped by node
    const int* fface;     // (entries) face of the entry
    const double* fval;   // (entries, 3) valM of the entry
    const double* gram;   // (nface, nface) valM_f . valM_g (diagonal: nS)
    double coef0[kMaxCoupled], coef1[kMaxCoupled];
    double err0, eps;
    double* part;         // 2 regions of kGmPartStride * gridDim
    double* H;            // (sD + 1, sD) column-major, rotated (written by block 0)
    double* errv;         // (sD + 1)
    double* out;          // iterations done, suc
};

__device__ __forceinline__ double gm_sum(const double* part, int k, double* sm) {
    double s = 0.0;
    for (int b = threadIdx.x; b < gridDim.x; b += blockDim.x) s += __ldcg(part + (size_t)b * kGmPartStride + k);
    return block_sum(s, sm);
}

template <typename M, typename B, int NF>
__global__ void __launch_bounds__(kGmcThreads, 2) k_gmres_cycle(GmcArgs<M, B> a) {
    namespace cgrp = cooperative_groups;
    cgrp::grid_group grid = cgrp::this_grid();
    __shared__ double sm[32];
    __shared__ double sh[kGmMaxSD + 2];  // h_1 .. h_{i+1} of the current column
    __shared__ double sc[kGmMaxSD], ssn[kGmMaxSD], serr[kGmMaxSD + 1];
    __shared__ int sdone;
    const int n = a.n;
    const long long n3 = a.n3, npad = a.npad;
    const int tid0 = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
    if (threadIdx.x == 0) {
        serr[0] = a.err0;
        sdone = 0;
    }
    __syncthreads();
    int bar = 0;  // barrier counter: partial region = bar & 1
    auto region = [&]() { return a.part + (size_t)(bar & 1) * kGmPartStride * gridDim.x; };
    int i;
    for (i = 1; i <= a.sD; ++i) {
        const B* uin = a.u + (size_t)(i - 1) * n3;
        B* w = a.u + (size_t)i * n3;
        // ---- P1: w = K U(i-1); face dots S0_f (on U(i-1)) and T_f (on w) ----
        double s0[NF > 0 ? NF : 1], tf[NF > 0 ? NF : 1];
#pragma unroll
        for (int f = 0; f < (NF > 0 ? NF : 1); ++f) s0[f] = tf[f] = 0.0;
        for (int r = tid0; r < n; r += nth) {
            double a0 = 0.0, a1 = 0.0, a2 = 0.0;
            CR_SELL_ROW_U(4, a.sp, a.scol, r, {
                const B* uc = uin + 3 * (size_t)c;
                const double u0 = (double)uc[0], u1 = (double)uc[1], u2 = (double)uc[2];
                const auto ka = ldcs4(reinterpret_cast<const typename V4<M>::type*>(a.Ks) + pos);
                const auto kb = ldcs4(reinterpret_cast<const typename V4<M>::type*>(a.Ks + 4 * npad) + pos);
                const double k8 = (double)__ldcs(a.Ks + 8 * npad + pos);
                a0 = a0 + (double)ka.x * u0 + (double)ka.y * u1 + (double)ka.z * u2;
                a1 = a1 + (double)ka.w * u0 + (double)kb.x * u1 + (double)kb.y * u2;
                a2 = a2 + (double)kb.z * u0 + (double)kb.w * u1 + k8 * u2;
            })
            const B w0 = (B)a0, w1 = (B)a1, w2 = (B)a2;
            w[3 * (size_t)r + 0] = w0;
            w[3 * (size_t)r + 1] = w1;
            w[3 * (size_t)r + 2] = w2;
            if (NF > 0) {
                for (int k = a.fptr[r]; k < a.fptr[r + 1]; ++k) {
                    const int fe = a.fent[k];
                    const int f = a.fface[fe];
                    const double* v = a.fval + 3 * (size_t)fe;
                    const B* ur = uin + 3 * (size_t)r;
#pragma unroll
                    for (int q = 0; q < NF; ++q)
                        if (q == f) {
                            s0[q] += v[0] * (double)ur[0] + v[1] * (double)ur[1] + v[2] * (double)ur[2];
                            tf[q] += v[0] * (double)w0 + v[1] * (double)w1 + v[2] * (double)w2;
                        }
                }
            }
        }
        double cf[NF > 0 ? NF : 1];
        if (NF > 0) {
            double* pr = region();
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                if (f >= a.nface) break;
                const double x0 = block_sum(s0[f], sm), x1 = block_sum(tf[f], sm);
                if (threadIdx.x == 0) {
                    pr[(size_t)blockIdx.x * kGmPartStride + 2 * f] = x0;
                    pr[(size_t)blockIdx.x * kGmPartStride + 2 * f + 1] = x1;
                }
            }
        }
        grid.sync();
        if (NF > 0) {
            const double* pr = region();
            double S0[NF > 0 ? NF : 1], T[NF > 0 ? NF : 1];
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                S0[f] = T[f] = 0.0;
                if (f >= a.nface) continue;
                S0[f] = gm_sum(pr, 2 * f, sm);
                T[f] = gm_sum(pr, 2 * f + 1, sm);
            }
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                cf[f] = 0.0;
                if (f >= a.nface) continue;
                double S1 = T[f];
                for (int g = 0; g < a.nface; ++g) S1 += a.coef0[g] * S0[g] * a.gram[f * a.nface + g];
                cf[f] = a.coef0[f] * S0[f] + a.coef1[f] * S1;
            }
        }
        ++bar;
        // ---- MGS passes j = 1..i: h_j = <w, U(j-1)> after w -= h_{j-1} U(j-2) ----
        for (int j = 1; j <= i; ++j) {
            const B* uj = a.u + (size_t)(j - 1) * n3;
            const B* up = j >= 2 ? a.u + (size_t)(j - 2) * n3 : nullptr;
            const double hp = j >= 2 ? sh[j - 1] : 0.0;
            double d = 0.0;
            for (int r = tid0; r < n; r += nth) {
                int k0 = 0, k1 = 0;
                if (NF > 0 && j == 1) {
                    k0 = a.fptr[r];
                    k1 = a.fptr[r + 1];
                }
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const size_t t = 3 * (size_t)r + k;
                    double wv = (double)w[t];
                    if (j == 1) {
                        if (NF > 0 && k1 > k0) {
                            double add = 0.0;
                            for (int e = k0; e < k1; ++e) {
                                const int fe = a.fent[e];
                                const int f = a.fface[fe];
#pragma unroll
                                for (int q = 0; q < NF; ++q)
                                    if (q == f) add += a.fval[3 * (size_t)fe + k] * cf[q];
                            }
                            wv = (double)(B)(wv + add);
                            w[t] = (B)wv;
                        }
                    } else {
                        wv = (double)(B)(wv - hp * (double)up[t]);
                        w[t] = (B)wv;
                    }
                    d += wv * (double)__ldcs(uj + t);
                }
            }
            d = block_sum(d, sm);
            double* pr = region();
            if (threadIdx.x == 0) pr[(size_t)blockIdx.x * kGmPartStride] = d;
            grid.sync();
            const double hj = gm_sum(region(), 0, sm);
            if (threadIdx.x == 0) sh[j] = hj;
            ++bar;
            __syncthreads();
        }
        // ---- norm: w -= h_i U(i-1); |w|^2 ----
        {
            const double hp = sh[i];
            double d = 0.0;
            for (int r = tid0; r < n; r += nth) {
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const size_t t = 3 * (size_t)r + k;
                    const double wv = (double)(B)((double)w[t] - hp * (double)uin[t]);
                    w[t] = (B)wv;
                    d += wv * wv;
                }
            }
            d = block_sum(d, sm);
            double* pr = region();
            if (threadIdx.x == 0) pr[(size_t)blockIdx.x * kGmPartStride] = d;
            grid.sync();
            const double hn = gm_sum(region(), 0, sm);
            ++bar;
            // ---- Givens (memLS.f90:750-760), identical in every block ----
            if (threadIdx.x == 0) {
                double hc[kGmMaxSD + 1];
                for (int j = 1; j <= i; ++j) hc[j - 1] = sh[j];
                hc[i] = sqrt(hn);
                sh[i + 1] = hc[i];
                double tmp;
                for (int j = 1; j <= i - 1; ++j) {
                    tmp = sc[j - 1] * hc[j - 1] + ssn[j - 1] * hc[j];
                    hc[j] = -ssn[j - 1] * hc[j - 1] + sc[j - 1] * hc[j];
                    hc[j - 1] = tmp;
                }
                tmp = sqrt(hc[i - 1] * hc[i - 1] + hc[i] * hc[i]);
                sc[i - 1] = hc[i - 1] / tmp;
                ssn[i - 1] = hc[i] / tmp;
                hc[i - 1] = tmp;
                hc[i] = 0.0;
                serr[i] = -ssn[i - 1] * serr[i - 1];
                serr[i - 1] = sc[i - 1] * serr[i - 1];
                if (blockIdx.x == 0) {
                    for (int j = 0; j <= i; ++j) a.H[(size_t)(i - 1) * (a.sD + 1) + j] = hc[j];
                    a.errv[i - 1] = serr[i - 1];
                    a.errv[i] = serr[i];
                }
                sdone = fabs(serr[i]) < a.eps ? 1 : 0;
            }
            __syncthreads();
        }
        if (sdone) break;
        if (i == a.sD) break;
        // ---- normalize: U(i) = w / h_{i+1} ----
        {
            const double hn = sh[i + 1];
            for (long long t = tid0; t < n3; t += nth) w[t] = (B)((double)w[t] / hn);
            grid.sync();
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.out[0] = (double)(i > a.sD ? a.sD : i);
        a.out[1] = (double)sdone;
    }
}

// valM of the coupled faces gathered into (entries, 3): zero past nsd.
__global__ void k_gm_fval(const double* __restrict__ valM, int fdof, int nsd, int nNoF, double* __restrict__ out) {
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < nNoF; a += gridDim.x * blockDim.x)
        for (int k = 0; k < 3; ++k) out[3 * (size_t)a + k] = k < nsd ? valM[(size_t)fdof * a + k] : 0.0;
}

// Coupled-face map for the persistent cycle, rebuilt when the set of
// coupled faces changes: the entries (face node a of coupled face q, in face
// order) grouped by node (fptr / fent), the face of each entry, and the
// pairs of entries of different faces at one node (faces that share rim
// nodes), from which k_gm_gram forms the off-diagonal valM_f . valM_g.
static int gm_face_map(crimson_lhs* L, int* ok) {
    std::vector<int> cur;
    for (int k = 0; k < (int)L->face.size(); ++k)
        if (L->face[k].coupledFlag) cur.push_back(k);
    if (L->gm_map_ok >= 0 && cur == L->gm_faces) {
        *ok = L->gm_map_ok;
        return CRIMSON_OK;
    }
    L->gm_faces = cur;
    L->gm_map_ok = (int)cur.size() > kMaxCoupled ? 0 : -1;   // -1 until all of it is built
    *ok = 0;
    if (L->gm_map_ok == 0) return CRIMSON_OK;
    cudaStream_t s = L->stream;
    const int n = L->nNo;
    std::vector<int> node_of, fface;
    for (int q = 0; q < (int)cur.size(); ++q) {
        const MemlsFace& f = L->face[cur[q]];
        std::vector<int> g((size_t)f.nNo);
        CR_CUDA(cudaMemcpyAsync(g.data(), f.glob.p, sizeof(int) * g.size(), cudaMemcpyDeviceToHost, s));
        CR_CUDA(cudaStreamSynchronize(s));
        for (int a = 0; a < f.nNo; ++a) {
            if (g[a] < 0 || g[a] >= n) {
                L->gm_map_ok = 0;
                return CRIMSON_OK;
            }
            node_of.push_back(g[a]);
            fface.push_back(q);
        }
    }
    const int entries = (int)node_of.size();
    std::vector<int> fptr((size_t)n + 1, 0), fent((size_t)std::max(1, entries));
    for (int e = 0; e < entries; ++e) ++fptr[(size_t)node_of[e] + 1];
    for (int r = 0; r < n; ++r) fptr[(size_t)r + 1] += fptr[r];
    std::vector<int> fill(fptr.begin(), fptr.end() - 1);
    for (int e = 0; e < entries; ++e) fent[(size_t)fill[node_of[e]]++] = e;
    std::vector<int> pairs;  // (e1, e2) of different faces at one node
    for (int r = 0; r < n; ++r)
        for (int k1 = fptr[r]; k1 < fptr[(size_t)r + 1]; ++k1)
            for (int k2 = fptr[r]; k2 < fptr[(size_t)r + 1]; ++k2)
                if (k1 != k2 && fface[fent[k1]] != fface[fent[k2]]) {
                    pairs.push_back(fent[k1]);
                    pairs.push_back(fent[k2]);
                }
    CR_CHECK(L->gmFptr.upload(fptr.data(), fptr.size(), s));
    CR_CHECK(L->gmFent.upload(fent.data(), fent.size(), s));
    CR_CHECK(L->gmFface.alloc(std::max<size_t>(1, fface.size())));
    if (!fface.empty())
        CR_CUDA(cudaMemcpyAsync(L->gmFface.p, fface.data(), sizeof(int) * fface.size(), cudaMemcpyHostToDevice, s));
    L->gm_npairs = (int)pairs.size() / 2;
    CR_CHECK(L->gmPairs.alloc(std::max<size_t>(2, pairs.size())));
    if (!pairs.empty())
        CR_CUDA(cudaMemcpyAsync(L->gmPairs.p, pairs.data(), sizeof(int) * pairs.size(), cudaMemcpyHostToDevice, s));
    CR_CHECK(L->gmFval.alloc(3 * (size_t)std::max(1, entries)));
    CR_CHECK(L->gmGram.alloc((size_t)kMaxCoupled * kMaxCoupled));
    CR_CUDA(cudaStreamSynchronize(s));
    L->gm_map_ok = 1;
    *ok = 1;
    return CRIMSON_OK;
}

// valM_f . valM_g of the coupled faces: nS on the diagonal, the shared-node
// pairs off it (one thread, fixed order).
struct FaceNorms {
    double v[kMaxCoupled];
};
__global__ void k_gm_gram(const int* __restrict__ pairs, int npairs, const int* __restrict__ fface,
                          const double* __restrict__ fval, FaceNorms nS, int nface, double* __restrict__ gram) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    for (int f = 0; f < nface; ++f)
        for (int g = 0; g < nface; ++g) gram[f * nface + g] = f == g ? nS.v[f] : 0.0;
    for (int p = 0; p < npairs; ++p) {
        const int e1 = pairs[2 * p], e2 = pairs[2 * p + 1];
        const double* v1 = fval + 3 * (size_t)e1;
        const double* v2 = fval + 3 * (size_t)e2;
        gram[fface[e1] * nface + fface[e2]] += v1[0] * v2[0] + v1[1] * v2[1] + v1[2] * v2[2];
    }
}

// Coupled-face data of k_gmres for the NSSOLVER call: valM by entry and the
// faces' valM_f . valM_g.  *ok = 0 when the kernel does not apply (more than
// kMaxCoupled coupled faces).
static int gm_faces_prepare(crimson_lhs* L, int* ok) {
    CR_CHECK(gm_face_map(L, ok));
    if (!*ok) return CRIMSON_OK;
    cudaStream_t s = L->stream;
    FaceNorms nsv{};
    int off = 0;
    const int nface = (int)L->gm_faces.size();
    for (int q = 0; q < nface; ++q) {
        const MemlsFace& f = L->face[L->gm_faces[q]];
        launch(k_gm_fval, grid_for(f.nNo, 256), 256, 0, s, (const double*)f.valM.p, f.dof, std::min(f.dof, 3), f.nNo,
               L->gmFval.p + 3 * (size_t)off);
        nsv.v[q] = f.nS;
        off += f.nNo;
    }
    if (nface > 0)
        launch(k_gm_gram, 1, 32, 0, s, (const int*)L->gmPairs.p, L->gm_npairs, (const int*)L->gmFface.p,
               (const double*)L->gmFval.p, nsv, nface, L->gmGram.p);
    return CRIMSON_OK;
}

// Launches k_gmres for K X = R; the outcome goes to the scalar slots at slot
// (gmres_finish reads them after the stream has been waited for).
template <typename M, typename B>
static int gmres_launch(Ctx& C, const crimson_subls& ls, const M* Ks, const double* R, double* X, int slot) {
    crimson_lhs* L = C.L;
    cudaStream_t s = C.s;
    const int n = L->nNo;
    const int sms = std::min(sm_count(), kGrMaxBlocks);
    // Four lanes per row and at most 8 values per thread in registers; blocks
    // of 256 threads until every SM has one, then larger ones.  Larger meshes:
    // one lane per row.
    const long long quads = 4LL * n;
    const bool reg = quads <= 8LL * gm_threads(1) * sms;
    const int grid = (int)std::max(1LL, std::min<long long>(sms, (quads + 255) / 256));
    int threads = reg ? 256 : gm_threads(0);
    while (reg && threads < gm_threads(1) && (long long)grid * threads < quads) threads *= 2;
    const long long slots = reg ? (quads + (long long)grid * threads - 1) / ((long long)grid * threads) : 0;
    const void* fns[5] = {(const void*)k_gmres<M, B, 0>, (const void*)k_gmres<M, B, 1>, (const void*)k_gmres<M, B, 2>,
                          (const void*)k_gmres<M, B, 4>, (const void*)k_gmres<M, B, 8>};
    const void* kfn = fns[slots > 4 ? 4 : (slots > 2 ? 3 : (int)slots)];
    const size_t smem = sizeof(double) * ((size_t)(ls.sD + 1) * ls.sD + 4 * (size_t)ls.sD + 1);
    if (L->gmPk.n != 2 * (size_t)kGmVals * sms) {
        CR_CHECK(L->gmPk.alloc(2 * (size_t)kGmVals * sms));
        CR_CUDA(cudaMemsetAsync(L->gmPk.p, 0, sizeof(ulonglong2) * L->gmPk.n, s));
        L->gm_epoch = 0;
    }
    GmArgs<M, B> a;
    a.sp = L->sell_ptr.p;
    a.scol = L->sell_col.p;
    a.npad = L->npad;
    a.n = n;
    a.Ks = Ks;
    a.u = reinterpret_cast<B*>(L->basis.p);
    a.n3 = 3LL * n;
    a.sD = ls.sD;
    a.mItr = ls.mItr;
    a.relTol = ls.relTol;
    a.absTol = ls.absTol;
    a.R = R;
    a.X = X;
    a.nface = (int)L->gm_faces.size();
    a.fptr = L->gmFptr.p;
    a.fent = L->gmFent.p;
    a.fface = L->gmFface.p;
    a.fval = L->gmFval.p;
    a.gram = L->gmGram.p;
    for (int q = 0; q < kMaxCoupled; ++q) {
        a.coef0[q] = a.coef1[q] = 0.0;
        if (q < a.nface) {
            const MemlsFace& f = L->face[L->gm_faces[q]];
            a.coef0[q] = f.res;
            a.coef1[q] = -f.res / (1.0 + f.res * f.nS);
        }
    }
    a.pk = L->gmPk.p;
    a.epoch = L->gm_epoch;
    a.out = C.sc(slot);
    // barriers of a call: per cycle at most 6, per iteration at most sD + 3
    L->gm_epoch += 2 + (unsigned long long)std::max(ls.mItr, 0) * (6 + (unsigned long long)ls.sD * (ls.sD + 3));
    CR_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(double) * ((kGmMaxSD + 1) * kGmMaxSD + 4 * kGmMaxSD + 1))));
    void* kargs[] = {&a};
    note_launch();
    CR_CUDA(cudaLaunchCooperativeKernel(kfn, dim3(grid), dim3(threads), kargs, smem, s));
    return CRIMSON_OK;
}

// memLS's statistics of a k_gmres call from the slots it left (on the host).
static int gmres_finish(Ctx& C, crimson_subls& ls, int slot, double seconds) {
    const double* o = C.L->hscal + slot;
    ls.suc = 0;
    if (o[1] < 0.0) {
        set_last_error("GMRES: a wait of the persistent kernel ran out");
        return CRIMSON_ERR_CUDA;
    }
    if (o[5] != 0.0) {   // right side below the absolute tolerance
        ls.callD = 0.0;
        ls.dB = 0.0;
        return CRIMSON_OK;
    }
    ls.suc = (int)o[1];
    ls.itr += (int)o[0];
    ls.iNorm = o[2];
    ls.fNorm = o[3];
    ls.callD += seconds;
    ls.dB = 10.0 * std::log(o[3] / o[4]);
    return CRIMSON_OK;
}

// Runs one restart cycle on the device (k_gmres_cycle): U(0) normalized in
// the basis, err0 = its norm before normalizing.  Returns the iterations
// done, whether |err_i| < eps was reached, and the rotated Hessenberg
// columns / err values in the host arrays of gmres().  The caller has prepared
// the faces (gm_faces_prepare) and checked sD; *used = 0 when there is no
// cooperative fit.
template <typename M, typename B>
static int gmres_cycle(Ctx& C, crimson_subls& ls, const M* Ks, double err0, double eps, std::vector<double>& h,
                       std::vector<double>& err, int* iters, int* suc, int* used) {
    crimson_lhs* L = C.L;
    cudaStream_t s = C.s;
    const int sD = ls.sD;
    *used = 0;
    if (sD < 1 || sD > kGmMaxSD) return CRIMSON_OK;
    const int nface = (int)L->gm_faces.size();
    const void* fns[3] = {(const void*)k_gmres_cycle<M, B, 0>, (const void*)k_gmres_cycle<M, B, 1>,
                          (const void*)k_gmres_cycle<M, B, kMaxCoupled>};
    int& grid = L->gm_grid32;
    if (grid == 0) {
        int nb = 1 << 30;
        for (const void* f : fns) {
            int b = 0;
            CR_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, f, kGmcThreads, 0));
            nb = std::min(nb, b);
        }
        grid = nb >= 1 ? sm_count() * std::min(nb, 2) : -1;
    }
    if (grid < 1) return CRIMSON_OK;
    CR_CHECK(L->gmH.alloc((size_t)(kGmMaxSD + 1) * kGmMaxSD));
    CR_CHECK(L->gmErr.alloc(kGmMaxSD + 1));
    CR_CHECK(L->gmOut.alloc(2));
    CR_CHECK(L->gmPart.alloc(2 * (size_t)kGmPartStride * L->gm_grid32));
    GmcArgs<M, B> a;
    a.sp = L->sell_ptr.p;
    a.scol = L->sell_col.p;
    a.npad = L->npad;
    a.n = L->nNo;
    a.Ks = Ks;
    a.u = reinterpret_cast<B*>(L->basis.p);
    a.n3 = 3LL * L->nNo;
    a.sD = sD;
    a.nface = nface;
    a.fptr = L->gmFptr.p;
    a.fent = L->gmFent.p;
    a.fface = L->gmFface.p;
    a.fval = L->gmFval.p;
    a.gram = L->gmGram.p;
    for (int q = 0; q < kMaxCoupled; ++q) {
        a.coef0[q] = a.coef1[q] = 0.0;
        if (q < nface) {
            const MemlsFace& f = L->face[L->gm_faces[q]];
            a.coef0[q] = f.res;
            a.coef1[q] = -f.res / (1.0 + f.res * f.nS);
        }
    }
    a.err0 = err0;
    a.eps = eps;
    a.part = L->gmPart.p;
    a.H = L->gmH.p;
    a.errv = L->gmErr.p;
    a.out = L->gmOut.p;
    void* kargs[] = {&a};
    note_launch();
    const void* kfn = fns[nface == 0 ? 0 : (nface == 1 ? 1 : 2)];
    CR_CUDA(cudaLaunchCooperativeKernel(kfn, dim3(grid), dim3(kGmcThreads), kargs, 0, s));
    double out[2];
    CR_CUDA(cudaMemcpyAsync(out, L->gmOut.p, sizeof(out), cudaMemcpyDeviceToHost, s));
    CR_CUDA(cudaStreamSynchronize(s));
    const int it = (int)out[0];
    if (it < 1 || it > sD) return CRIMSON_ERR_STATE;
    CR_CUDA(cudaMemcpyAsync(h.data(), L->gmH.p, sizeof(double) * (size_t)(sD + 1) * it, cudaMemcpyDeviceToHost, s));
    CR_CUDA(cudaMemcpyAsync(err.data(), L->gmErr.p, sizeof(double) * (it + 1), cudaMemcpyDeviceToHost, s));
    CR_CUDA(cudaStreamSynchronize(s));
    CR_CUDA(cudaGetLastError());
    *iters = it;
    *suc = out[1] != 0.0 ? 1 : 0;
    *used = 1;
    return CRIMSON_OK;
}

// GMRES (memLS.f90:681-788) on dof = 3 with the restarts on the host: each
// cycle as one kernel (cycles: the FP32-tangent mode), or with one launch per
// step where no persistent kernel applies (more than kGmMaxSD Krylov vectors or
// kMaxCoupled coupled faces); K sliced in M, basis in B, R and X FP64; X may not alias R.
template <typename M, typename B>
static int gmres(Ctx& C, crimson_subls& ls, const M* Ks, const double* R, double* X, bool cycles) {
    crimson_lhs* L = C.L;
    cudaStream_t s = C.s;
    const int dof = 3;
    const long long n = (long long)dof * L->nNo;
    const int sD = ls.sD;
    B* u = reinterpret_cast<B*>(L->basis.p);
    auto U = [&](int k) { return u + (size_t)k * n; };
    std::vector<double> h((size_t)(sD + 1) * sD, 0.0), c(sD), sn(sD), err(sD + 1), y(sD);
    auto H = [&](int i, int j) -> double& { return h[(size_t)j * (sD + 1) + i]; };
    const double time = now_s();
    ls.suc = 0;
    CR_CUDA(cudaMemsetAsync(X, 0, sizeof(double) * n, s));
    double eps = 0.0;
    const bool coupled = C.any_coupled();
    int i = 0;
    for (int l = 1; l <= ls.mItr; ++l) {
        if (l == 1) {
            launch(k_convert<B, double>, grid_for(n, 256), 256, 0, s, R, U(0), n);
        } else {
            ls.itr = ls.itr + 1;
            C.vv3s(Ks, (const double*)X, U(0));
            C.addbcmul(0, dof, (const double*)X, U(0));
            launch(k_sub<double, B, B>, grid_for(n, 256), 256, 0, s, R, (const B*)U(0), U(0), n);
        }
        if (coupled) C.addbcmul(1, dof, (const B*)U(0), U(0));  // dots read X before any update: X may alias Y
        C.dot((const B*)U(0), (const B*)U(0), n, kSlotNrm);
        CR_CHECK(C.sync_scal(kSlotNrm, 1));
        err[0] = std::sqrt(L->hscal[kSlotNrm]);
        if (l == 1) {
            eps = err[0];
            if (eps <= ls.absTol) {
                ls.callD = 0.0;
                ls.dB = 0.0;
                return CRIMSON_OK;
            }
            ls.iNorm = eps;
            ls.fNorm = eps;
            eps = std::max(ls.absTol, ls.relTol * eps);
        }
        ls.dB = ls.fNorm;
        launch(k_divide<B>, grid_for(n, 256), 256, 0, s, (const B*)U(0), (const double*)C.sc(kSlotNrm), U(0), n, 1);
        int used = 0;
        if (cycles && std::is_same<M, float>::value) {
            int it = 0, ok = 0;
            CR_CHECK((gmres_cycle<float, float>(C, ls, (const float*)Ks, err[0], eps, h, err, &it, &ok, &used)));
            if (used) {
                ls.itr = ls.itr + it;
                i = it;
                if (ok) ls.suc = 1;
            }
        }
        for (i = used ? i : 1; !used && i <= sD; ++i) {
            ls.itr = ls.itr + 1;
            B* w = U(i);
            C.vv3s(Ks, (const B*)U(i - 1), w);
            C.addbcmul(0, dof, (const B*)U(i - 1), w);
            if (coupled) C.addbcmul(1, dof, (const B*)w, w);
            // fused modified Gram-Schmidt
            for (int j = 1; j <= i; ++j) {
                const B* uprev = (j == 1) ? nullptr : U(j - 2);
                launch(k_mgs<B>, red_grid(n), 256, 0, s, w, uprev, (const double*)C.sc(kSlotH + j - 2),
                       (const B*)U(j - 1), n, L->red.part.p, L->red.ticket.p, C.sc(kSlotH + j - 1));
            }
            launch(k_mgs<B>, red_grid(n), 256, 0, s, w, (const B*)U(i - 1), (const double*)C.sc(kSlotH + i - 1),
                   (const B*)w, n, L->red.part.p, L->red.ticket.p, C.sc(kSlotH + i));
            launch(k_divide<B>, grid_for(n, 256), 256, 0, s, (const B*)w, (const double*)C.sc(kSlotH + i), w, n, 1);
            CR_CHECK(C.sync_scal(kSlotH, i + 1));
            for (int j = 1; j <= i; ++j) H(j - 1, i - 1) = L->hscal[kSlotH + j - 1];
            H(i, i - 1) = std::sqrt(L->hscal[kSlotH + i]);
            double tmp;
            for (int j = 1; j <= i - 1; ++j) {
                tmp = c[j - 1] * H(j - 1, i - 1) + sn[j - 1] * H(j, i - 1);
                H(j, i - 1) = -sn[j - 1] * H(j - 1, i - 1) + c[j - 1] * H(j, i - 1);
                H(j - 1, i - 1) = tmp;
            }
            tmp = std::sqrt(H(i - 1, i - 1) * H(i - 1, i - 1) + H(i, i - 1) * H(i, i - 1));
            c[i - 1] = H(i - 1, i - 1) / tmp;
            sn[i - 1] = H(i, i - 1) / tmp;
            H(i - 1, i - 1) = tmp;
            H(i, i - 1) = 0.0;
            err[i] = -sn[i - 1] * err[i - 1];
            err[i - 1] = c[i - 1] * err[i - 1];
            if (std::fabs(err[i]) < eps) {
                ls.suc = 1;
                break;
            }
        }
        if (i > sD) i = sD;
        for (int j = 0; j < i; ++j) y[j] = err[j];
        for (int j = i; j >= 1; --j) {
            for (int k = j + 1; k <= i; ++k) y[j - 1] = y[j - 1] - H(j - 1, k - 1) * y[k - 1];
            y[j - 1] = y[j - 1] / H(j - 1, j - 1);
        }
        std::memcpy(L->hscal + kSlotY, y.data(), sizeof(double) * i);
        CR_CUDA(cudaMemcpyAsync(C.sc(kSlotY), L->hscal + kSlotY, sizeof(double) * i, cudaMemcpyHostToDevice, s));
        launch(k_multi_axpy<B>, grid_for(n, 256), 256, 0, s, X, (const B*)u, (const double*)C.sc(kSlotY), i, n);
        CR_CUDA(cudaStreamSynchronize(s));  // y staging buffer is reused
        ls.fNorm = std::fabs(err[i]);
        if (ls.suc) break;
    }
    ls.callD = now_s() - time + ls.callD;
    ls.dB = 10.0 * std::log(ls.fNorm / ls.dB);
    return CRIMSON_OK;
}

// Coupled-face vectors for the CG's ADDBCMUL(PRE) term: w_f = G^T valM_f and
// z_f = Gt valM_f, with the Sherman-Morrison coefficient -res/(1 + res nS).
// Built once per NSSOLVER call (valM, G, Gt are fixed during it).
template <typename M>
static int cg_faces(Ctx& C, const M* G, const M* Gt, int* nface, double* coef) {
    crimson_lhs* L = C.L;
    cudaStream_t s = C.s;
    const int n = L->nNo;
    int k = 0;
    for (auto& f : L->face) {
        if (!f.coupledFlag) continue;
        if (k >= kMaxCoupled) return CRIMSON_ERR_UNSUPPORTED;
        CR_CHECK(L->cgExt.alloc(3 * (size_t)n));
        CR_CHECK(L->cgW.alloc((size_t)kMaxCoupled * n));
        CR_CHECK(L->cgZ.alloc((size_t)kMaxCoupled * n));
        CR_CUDA(cudaMemsetAsync(L->cgExt.p, 0, sizeof(double) * 3 * (size_t)n, s));
        launch(k_face_ext, grid_for(f.nNo, 256), 256, 0, s, f.glob.p, f.valM.p, f.dof, std::min(f.dof, 3), f.nNo,
               L->cgExt.p);
        launch(k_spmv_vs3_trans<M>, C.spmv_grid(), 256, 0, s, L->rowptr, L->col, L->trans, G, (const double*)L->cgExt.p,
               L->cgW.p + (size_t)k * n, n);
        C.vs3(Gt, (const double*)L->cgExt.p, L->cgZ.p + (size_t)k * n);
        coef[k] = -f.res / (1.0 + f.res * f.nS);
        ++k;
    }
    *nface = k;
    CR_CUDA(cudaGetLastError());
    return CRIMSON_OK;
}

// Shared memory for block-resident CG columns (CgCols) on a grid of two
// blocks per SM: 0 when the pattern's column offsets exceed 16 bits; else
// 2 bytes per sliced entry of the fullest block.  Computed once per pattern.
static int cg_resident_bytes(crimson_lhs* L, size_t* bytes) {
    if (L->cg_res_bytes >= 0) {
        *bytes = (size_t)L->cg_res_bytes;
        return CRIMSON_OK;
    }
    cudaStream_t s = L->stream;
    const int n = L->nNo;
    int maxoff = 0;
    if (L->s2_state != 1) {   // an explicit operator's 2-ring offsets fit 16 bits, so these do
        CR_CHECK(L->cg_tmp.alloc(1));
        CR_CUDA(cudaMemsetAsync(L->cg_tmp.p, 0, sizeof(int), s));
        launch(k_max_offset, grid_for(n, 256), 256, 0, s, (const int*)L->rowptr, (const int*)L->col, n, L->cg_tmp.p);
        CR_CUDA(cudaMemcpyAsync(&maxoff, L->cg_tmp.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    }
    std::vector<int> sp((size_t)L->nslice + 1);
    CR_CUDA(cudaMemcpyAsync(sp.data(), L->sell_ptr.p, sizeof(int) * sp.size(), cudaMemcpyDeviceToHost, s));
    CR_CUDA(cudaStreamSynchronize(s));
    long long best = 0;
    if (maxoff <= 32767) {
        const int grid = 2 * sm_count();
        const int wpb = kCgThreads / kSlice;  // slices (warps) per block
        std::vector<long long> per((size_t)grid, 0);
        for (int q = 0; q < L->nslice; ++q) per[(size_t)((q / wpb) % grid)] += sp[q + 1] - sp[q];
        for (long long v : per) best = std::max(best, v);
        best = (2 * best + 15) / 16 * 16;
        if (best == 0) best = 16;
    }
    L->cg_res_bytes = best;
    *bytes = (size_t)best;
    return CRIMSON_OK;
}

// Half of an SM's 228 KB less the 1 KB the driver reserves per block: more
// never fits twice.
constexpr size_t kCgResidentMax = 113 * 1024;

// Launch form of the two-product CG kernel on this lhs (kernel family and
// grid), decided at the first CGRAD of a precision, whichever operator that
// takes: crimson_memls_cg_layout reports it.
template <typename M>
static int cg_layout(crimson_lhs* L, size_t* rbytes_out) {
    const void* kres[3] = {(const void*)k_cg_persistent<0, M, true>, (const void*)k_cg_persistent<1, M, true>,
                           (const void*)k_cg_persistent<kMaxCoupled, M, true>};
    const void* kglb[3] = {(const void*)k_cg_persistent<0, M, false>, (const void*)k_cg_persistent<1, M, false>,
                           (const void*)k_cg_persistent<kMaxCoupled, M, false>};
    int& grid = std::is_same<M, float>::value ? L->cg_grid32 : L->cg_grid;
    int& mode = std::is_same<M, float>::value ? L->cg_res32 : L->cg_res64;
    size_t rbytes = 0;
    CR_CHECK(cg_resident_bytes(L, &rbytes));
    if (grid == 0) {
        // block-resident columns when two blocks per SM fit with them; the
        // kernels' limit is the same for every lhs (a smaller one's own size
        // would make the launches of a larger one fail)
        mode = 0;
        if (rbytes > 0 && rbytes <= kCgResidentMax) {
            int ok = 1;
            for (const void* f : kres) {
                int nb = 0;
                if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCgResidentMax) !=
                        cudaSuccess ||
                    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, f, kCgThreads, rbytes) != cudaSuccess || nb < 2)
                    ok = 0;
            }
            (void)cudaGetLastError();  // a refused attribute only selects the other kernel
            mode = ok;
        }
        if (mode) {
            grid = 2 * sm_count();
        } else {
            int nb = 1 << 30;
            for (const void* f : kglb) {
                int b = 0;
                CR_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, f, kCgThreads, 0));
                nb = std::min(nb, b);
            }
            if (nb < 1) return CRIMSON_ERR_UNSUPPORTED;
            grid = sm_count() * std::min(nb, 8);
        }
    }
    *rbytes_out = rbytes;
    return CRIMSON_OK;
}

// CGRAD (memLS.f90:367-430) on the Schur-like operator L P - Gt G P; R in/out (n).
// use_s2: on the explicit operator (schur.cu), else with two products on
// Gs / GLs, the sliced G and {Gt, L} of this NSSOLVER call.  Launches only;
// the outcome goes to the slots kSlotCg (cgrad_finish).
template <typename M>
static int cgrad_launch(Ctx& C, const crimson_subls& ls, const M* Gs, const typename V4<M>::type* GLs, double* R,
                        int nface, const double* coef, bool use_s2) {
    crimson_lhs* L = C.L;
    cudaStream_t s = C.s;
    const int n = L->nNo;
    size_t rbytes = 0;
    CR_CHECK(cg_layout<M>(L, &rbytes));
    if (use_s2) {
        CR_CUDA(cudaEventRecord(L->ev0, s));
        CR_CHECK(cg_schur_launch<M>(L, R, nface, coef, ls.relTol, ls.absTol, ls.mItr, C.sc(kSlotCg)));
        CR_CUDA(cudaEventRecord(L->ev1, s));
        return CRIMSON_OK;
    }
    C.dot((const double*)R, (const double*)R, n, kSlotErr);
    const int grid = std::is_same<M, float>::value ? L->cg_grid32 : L->cg_grid;
    const int mode = std::is_same<M, float>::value ? L->cg_res32 : L->cg_res64;
    const int fi = nface == 0 ? 0 : (nface == 1 ? 1 : 2);
    const void* kfns[2][3] = {{(const void*)k_cg_persistent<0, M, false>, (const void*)k_cg_persistent<1, M, false>,
                               (const void*)k_cg_persistent<kMaxCoupled, M, false>},
                              {(const void*)k_cg_persistent<0, M, true>, (const void*)k_cg_persistent<1, M, true>,
                               (const void*)k_cg_persistent<kMaxCoupled, M, true>}};
    const void* kfn = kfns[mode ? 1 : 0][fi];
    const size_t dyn = mode ? rbytes : 0;
    (std::is_same<M, float>::value ? L->cg_form32 : L->cg_form64) =
        mode ? CRIMSON_CG_PRODUCTS_RESIDENT : CRIMSON_CG_PRODUCTS;
    CR_CHECK(L->cgPart.alloc(3 * (size_t)kCgPartStride * std::max(L->cg_grid, L->cg_grid32)));
    CR_CHECK(L->cgRecA.alloc(2 * (size_t)n));
    CR_CHECK(L->cgRecB.alloc(4 * (size_t)n));
    CR_CHECK(L->cgPd.alloc((size_t)n));
    CR_CHECK(L->cgX.alloc((size_t)n));
    CR_CHECK(L->cgSP.alloc((size_t)n));
    CR_CUDA(cudaMemsetAsync(L->cgX.p, 0, sizeof(double) * n, s));
    launch(k_cg_init, grid_for(n, 256), 256, 0, s, (const double*)R, reinterpret_cast<double2*>(L->cgRecA.p), n);
    CgArgs<M> a;
    a.sp = L->sell_ptr.p;
    a.scol = L->sell_col.p;
    a.npad = L->npad;
    a.n = n;
    a.G = Gs;
    a.GL = GLs;
    a.X = L->cgX.p;
    a.recA = reinterpret_cast<double2*>(L->cgRecA.p);
    a.recB = reinterpret_cast<typename V4<M>::type*>(L->cgRecB.p);
    a.Pd = L->cgPd.p;
    a.SP = L->cgSP.p;
    a.nface = nface;
    a.w = L->cgW.p;
    a.z = L->cgZ.p;
    for (int f = 0; f < kMaxCoupled; ++f) a.coef[f] = f < nface ? coef[f] : 0.0;
    a.rr = C.sc(kSlotErr);
    a.relTol = ls.relTol;
    a.absTol = ls.absTol;
    a.mItr = ls.mItr;
    a.part = L->cgPart.p;
    a.out = C.sc(kSlotCg);
    void* kargs[] = {&a};
    note_launch();
    CR_CUDA(cudaEventRecord(L->ev0, s));
    CR_CUDA(cudaLaunchCooperativeKernel(kfn, dim3(grid), dim3(kCgThreads), kargs, dyn, s));
    CR_CUDA(cudaEventRecord(L->ev1, s));
    CR_CUDA(cudaMemcpyAsync(R, L->cgX.p, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
    return CRIMSON_OK;
}

// memLS's statistics of the CGRAD call from the slots it left (on the host),
// after the stream has been waited for.
template <typename M>
static int cgrad_finish(Ctx& C, crimson_subls& ls) {
    crimson_lhs* L = C.L;
    const double err = L->hscal[kSlotCg + 0], errO = L->hscal[kSlotCg + 1];
    const int i = (int)L->hscal[kSlotCg + 2];
    if (L->hscal[kSlotCg + 3] < 0.0) {
        set_last_error("CGRAD: a wait of the persistent kernel ran out");
        return CRIMSON_ERR_CUDA;
    }
    ls.suc = (int)L->hscal[kSlotCg + 3];
    ls.iNorm = L->hscal[kSlotCg + 4];
    float ms = 0.f;
    CR_CUDA(cudaEventElapsedTime(&ms, L->ev0, L->ev1));
    auto& acc = std::is_same<M, float>::value ? L->cg_acc32 : L->cg_acc64;
    acc.ms += ms;
    acc.iters += i - 1;
    acc.launches += 1;
    if (L->s2_form_pending) {
        float fm = 0.f;
        CR_CUDA(cudaEventElapsedTime(&fm, L->s2_ev0, L->s2_ev1));
        L->s2_form_ms += fm;
        L->s2_forms += 1;
        L->s2_form_pending = false;
    }
    ls.fNorm = std::sqrt(err);
    ls.callD = 1e-3 * ms + ls.callD;
    ls.dB = 5.0 * std::log(err / errO);
    ls.itr = ls.itr + i - 1;
    return CRIMSON_OK;
}

// GE (memLS.f90:607-677), A column-major
static int ge_solve(int N, const double* A, double* B) {
    if (N == 2) {
        double pivot = A[0] * A[3] - A[1] * A[2];
        if (pivot == 0.0 || !std::isfinite(pivot)) return CRIMSON_ERR_SINGULAR;
        double saveEl = (B[0] * A[3] - B[1] * A[2]) / pivot;
        B[1] = (B[1] * A[0] - B[0] * A[1]) / pivot;
        B[0] = saveEl;
        return CRIMSON_OK;
    }
    std::vector<double> Cm((size_t)N * (N + 1));
    auto c = [&](int i, int j) -> double& { return Cm[(size_t)j * N + i]; };
    for (int j = 0; j < N; ++j)
        for (int i = 0; i < N; ++i) c(i, j) = A[(size_t)j * N + i];
    for (int i = 0; i < N; ++i) c(i, N) = B[i];
    for (int m = 0; m < N - 1; ++m) {
        int ipv = m;
        double pivot = std::fabs(c(m, m));
        for (int i = m + 1; i < N; ++i)
            if (std::fabs(c(i, m)) > pivot) {
                ipv = i;
                pivot = std::fabs(c(i, m));
            }
        if (pivot < 2.0 * 2.220446049250313e-16) return CRIMSON_ERR_SINGULAR;
        if (ipv != m)
            for (int j = m; j <= N; ++j) std::swap(c(m, j), c(ipv, j));
        for (int i = m + 1; i < N; ++i) {
            double saveEl = c(i, m) / c(m, m);
            c(i, m) = 0.0;
            for (int j = m + 1; j <= N; ++j) c(i, j) = c(i, j) - saveEl * c(m, j);
        }
    }
    for (int j = N - 1; j >= 0; --j) {
        for (int i = j + 1; i < N; ++i) c(j, N) = c(j, N) - c(j, i) * c(i, N);
        c(j, N) = c(j, N) / c(j, j);
    }
    for (int i = 0; i < N; ++i) B[i] = c(i, N);
    return CRIMSON_OK;
}

// ---------------------------------------------------------------------------
// NSSOLVER's least-squares system (memLS.f90:1540-1570): the products of the
// two newest columns A d (u part n3 values, p part n) with every column and
// with the right side.  Column c is MU + c n3 / MP + c n; pair (k, j) for
// k = c0, c0 + 1 and j <= k, and (k, right side).  One pass reads the two new
// columns, the right side and kGramCols older columns; per-block sums, then
// one warp per product sums the blocks in order.  (One reduction launch per
// product and part took 28 launches per outer iteration and re-read the new
// columns each time: 10 of 143 ms of a 452k-tet mixed time step.)
// ---------------------------------------------------------------------------
constexpr int kGramCols = 4;
constexpr int kGramSums = 5 + 2 * kGramCols;   // n.n, n.m, m.m, n.r, m.r, then n.o, m.o of every older column
constexpr int kGramThreads = 256;

__global__ void __launch_bounds__(kGramThreads) k_gram_part(const double* __restrict__ MU, const double* __restrict__ MP,
                                                            const double* __restrict__ Ru, const double* __restrict__ Rp,
                                                            long long n3, long long n, int c0, int o0, int no,
                                                            double* __restrict__ part) {
    __shared__ double red[kGramSums][kGramThreads / 32];
    double acc[kGramSums];
#pragma unroll
    for (int k = 0; k < kGramSums; ++k) acc[k] = 0.0;
    const long long tot = n3 + n;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < tot; t += (long long)gridDim.x * blockDim.x) {
        const bool u = t < n3;
        const double* base = u ? MU + t : MP + (t - n3);
        const size_t ld = (size_t)(u ? n3 : n);
        const double a = base[(size_t)c0 * ld], b = base[(size_t)(c0 + 1) * ld];
        double o[kGramCols];
#pragma unroll
        for (int k = 0; k < kGramCols; ++k) o[k] = k < no ? base[(size_t)(o0 + k) * ld] : 0.0;
        if (o0 == 0) {
            const double r = u ? Ru[t] : Rp[t - n3];
            acc[0] += a * a;
            acc[1] += a * b;
            acc[2] += b * b;
            acc[3] += a * r;
            acc[4] += b * r;
        }
#pragma unroll
        for (int k = 0; k < kGramCols; ++k) {
            acc[5 + 2 * k] += a * o[k];
            acc[6 + 2 * k] += b * o[k];
        }
    }
#pragma unroll
    for (int k = 0; k < kGramSums; ++k) {
        const double v = warp_sum(acc[k]);
        if ((threadIdx.x & 31) == 0) red[k][threadIdx.x >> 5] = v;
    }
    __syncthreads();
    if (threadIdx.x < kGramSums) {
        double v = 0.0;
        for (int w = 0; w < kGramThreads / 32; ++w) v += red[threadIdx.x][w];
        part[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = v;
    }
}

// out[k] = sum of the nblk block sums of product k, in order; one block per product
__global__ void __launch_bounds__(32) k_gram_sum(const double* __restrict__ part, int nblk, double* __restrict__ out) {
    double s = 0.0;
    for (int b = threadIdx.x; b < nblk; b += 32) s += part[(size_t)blockIdx.x * nblk + b];
    s = warp_sum(s);
    if (threadIdx.x == 0) out[blockIdx.x] = s;
}

// y = y0 + sum_j c_j x_j, columns x_j at stride ld * step, terms added in
// order (y0 may be null: 0); u and p parts in one launch
constexpr int kMaxCols = 44;
struct ColCoefs {
    double c[kMaxCols];
};
__global__ void __launch_bounds__(256) k_combine(const __grid_constant__ ColCoefs cf, int m, int step,
                                                 const double* __restrict__ Xu, const double* __restrict__ Xp,
                                                 const double* __restrict__ y0u, const double* __restrict__ y0p,
                                                 double* __restrict__ yu, double* __restrict__ yp, long long n3,
                                                 long long n) {
    const long long tot = (yu ? n3 : 0) + n;
    const long long nu = yu ? n3 : 0;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < tot; t += (long long)gridDim.x * blockDim.x) {
        const bool u = t < nu;
        const long long i = u ? t : t - nu;
        const double* x = u ? Xu + i : Xp + i;
        const size_t ld = (size_t)(u ? n3 : n) * step;
        const double* y0 = u ? y0u : y0p;
        double y = y0 ? y0[i] : 0.0;
        for (int j = 0; j < m; ++j) y = y + cf.c[j] * x[(size_t)j * ld];
        (u ? yu : yp)[i] = y;
    }
}

// Sliced matrix buffers of one precision (zeroed at allocation, so the
// padding entries stay zero: conversions only write real entries).
template <typename M>
static int sell_alloc(crimson_lhs* L, DBuf<M>& K, DBuf<M>& G, DBuf<M>& GL, bool two_product) {
    const size_t np = (size_t)L->npad + (size_t)kSlice * kSellUnroll;
    auto zeroed = [&](DBuf<M>& b, size_t n) {
        if (b.n == n) return CRIMSON_OK;
        CR_CHECK(b.alloc(n));
        CR_CUDA(cudaMemsetAsync(b.p, 0, sizeof(M) * n, L->stream));
        return CRIMSON_OK;
    };
    CR_CHECK(zeroed(K, 9 * np));
    if (two_product) {
        CR_CHECK(zeroed(G, 3 * np));
        CR_CHECK(zeroed(GL, 4 * np));
    }
    return CRIMSON_OK;
}
static int sell_mats(crimson_lhs* L, double** K, double** G, double4** GL, bool two_product) {
    CR_CHECK(sell_alloc(L, L->Ks64, L->Gs64, L->GLs64, two_product));
    *K = L->Ks64.p;
    *G = L->Gs64.p;
    *GL = reinterpret_cast<double4*>(L->GLs64.p);
    return CRIMSON_OK;
}
static int sell_mats(crimson_lhs* L, float** K, float** G, float4** GL, bool two_product) {
    CR_CHECK(sell_alloc(L, L->Ks32, L->Gs32, L->GLs32, two_product));
    *K = L->Ks32.p;
    *G = L->Gs32.p;
    *GL = reinterpret_cast<float4*>(L->GLs32.p);
    return CRIMSON_OK;
}

// Sliced pattern of a CSR pattern (rowptr, col on the device): slice widths
// from the row lengths (host), columns (device).  The column array carries
// kSlice * kSellUnroll zero entries past npad.  *npad_out is set last: 0 means
// not built.
int sell_build(const int* rowptr, const int* col, int n, cudaStream_t s, DBuf<int>& sell_ptr, DBuf<int>& sell_col,
               long long* npad_out, int* nslice_out) {
    std::vector<int> rp((size_t)n + 1);
    CR_CUDA(cudaMemcpyAsync(rp.data(), rowptr, sizeof(int) * (n + 1), cudaMemcpyDeviceToHost, s));
    CR_CUDA(cudaStreamSynchronize(s));
    const int ns = (n + kSlice - 1) / kSlice;
    std::vector<int> sp((size_t)ns + 1, 0);
    long long pos = 0;
    for (int q = 0; q < ns; ++q) {
        int w = 0;
        for (int r = q * kSlice; r < std::min(n, (q + 1) * kSlice); ++r) w = std::max(w, rp[r + 1] - rp[r]);
        sp[q] = (int)pos;
        pos += (long long)kSlice * w;
        if (pos + (long long)kSlice * kSellUnroll > 0x7fffffffLL) return CRIMSON_ERR_UNSUPPORTED;
    }
    sp[ns] = (int)pos;
    CR_CHECK(sell_ptr.upload(sp.data(), sp.size(), s));
    const size_t np = (size_t)pos + (size_t)kSlice * kSellUnroll;
    CR_CHECK(sell_col.alloc(np));
    CR_CUDA(cudaMemsetAsync(sell_col.p, 0, sizeof(int) * np, s));
    launch(k_sell_cols, grid_for((long long)ns * kSlice, 256), 256, 0, s, rowptr, col, (const int*)sell_ptr.p, n,
           ns * kSlice, sell_col.p);
    CR_CUDA(cudaStreamSynchronize(s));
    CR_CUDA(cudaGetLastError());
    *npad_out = pos;
    *nslice_out = ns;
    return CRIMSON_OK;
}

static int sell_pattern(crimson_lhs* L) {
    if (L->npad > 0) return CRIMSON_OK;
    CR_CHECK(sell_build(L->rowptr, L->col, L->nNo, L->stream, L->sell_ptr, L->sell_col, &L->npad, &L->nslice));
    return CRIMSON_OK;
}

// NSSOLVER (memLS.f90:1460-1759); R (4, nNo) FP64 in/out.  mK, mG, mD, mL,
// Gt: the scaled split matrices (FP64 CSR).  GMRES and CGRAD run on sliced
// copies in M (FP64, or FP32 for the mixed mode) with a type-B GMRES basis;
// every other product -- the A d of the search directions that enter the
// least-squares (Gram) problem, the Schur right side D u and the
// coupled-face vectors -- uses the FP64 matrices, so the Gram system, the
// residual estimate and the outer residuals are those of the FP64 operator.
template <typename M, typename B>
static int nssolver(crimson_lhs* L, crimson_ls* ls, const double* mK, const double* mG, const double* mD,
                    const double* mL, const double* Gt, double* R) {
    Ctx C{L, L->stream};
    cudaStream_t s = L->stream;
    const int nNo = L->nNo;
    const long long nv = 3LL * nNo;
    int iB = ls->RI.mItr;
    const int nB = 2 * iB;
    auto Ucol = [&](int k) { return L->U.p + (size_t)k * nv; };
    auto Pcol = [&](int k) { return L->P.p + (size_t)k * nNo; };
    auto MUc = [&](int k) { return L->MU.p + (size_t)k * nv; };
    auto MPc = [&](int k) { return L->MP.p + (size_t)k * nNo; };
    launch(k_split4, grid_for(nNo, 256), 256, 0, s, (const double*)R, L->Rmi.p, L->Rci.p, nNo);
    CR_CUDA(cudaMemcpyAsync(L->Rm.p, L->Rmi.p, sizeof(double) * nv, cudaMemcpyDeviceToDevice, s));
    CR_CUDA(cudaMemcpyAsync(L->Rc.p, L->Rci.p, sizeof(double) * nNo, cudaMemcpyDeviceToDevice, s));
    std::vector<double> A((size_t)nB * nB, 0.0), Bv(nB, 0.0), xB(nB, 0.0);
    auto Aa = [&](int i, int j) -> double& { return A[(size_t)j * nB + i]; };
    C.dot((const double*)L->Rm.p, (const double*)L->Rm.p, nv, 0);
    C.dot((const double*)L->Rc.p, (const double*)L->Rc.p, nNo, 1);
    CR_CHECK(C.sync_scal(0, 2));
    double nv1 = std::sqrt(L->hscal[0]), ns1 = std::sqrt(L->hscal[1]);
    double eps = std::sqrt(std::pow(nv1, 2.0) + std::pow(ns1, 2.0));
    if (!std::isfinite(eps)) {
        set_last_error("NSSOLVER: non-finite right-hand side");
        return CRIMSON_ERR_NONFINITE;
    }
    ls->RI.iNorm = eps;
    ls->RI.fNorm = eps;
    ls->CG.callD = 0.0;
    ls->GM.callD = 0.0;
    ls->CG.itr = 0;
    ls->GM.itr = 0;
    const double t0 = now_s();
    ls->RI.suc = 0;
    eps = std::max(ls->RI.absTol, ls->RI.relTol * eps);
    // BCPRE (memLS.f90:1683-1716): nS = |valM|^2 per coupled face, summed on
    // the host in the reference's node order (faces are small).
    {
        std::vector<std::vector<double>> vm(L->face.size());
        for (size_t k = 0; k < L->face.size(); ++k) {
            const MemlsFace& f = L->face[k];
            if (!f.coupledFlag) continue;
            vm[k].resize((size_t)f.dof * f.nNo);
            CR_CUDA(cudaMemcpyAsync(vm[k].data(), f.valM.p, sizeof(double) * vm[k].size(), cudaMemcpyDeviceToHost, s));
        }
        CR_CUDA(cudaStreamSynchronize(s));
        for (size_t k = 0; k < L->face.size(); ++k) {
            MemlsFace& f = L->face[k];
            if (!f.coupledFlag) continue;
            f.nS = 0.0;
            const int nsd = std::min(f.dof, 3);
            for (int a = 0; a < f.nNo; ++a)
                for (int i = 0; i < nsd; ++i) f.nS = f.nS + std::pow(vm[k][(size_t)f.dof * a + i], 2.0);
        }
    }
    int cg_nface = 0;
    double cg_coef[kMaxCoupled];
    CR_CHECK(cg_faces(C, mG, Gt, &cg_nface, cg_coef));
    M* Ks = nullptr;
    M* Gs = nullptr;
    typename V4<M>::type* GLs = nullptr;
    // the FP32-tangent mode keeps the summation orders of its results (k_gmres_cycle)
    const bool kept = ls->precision == CRIMSON_MIXED_F32_TANGENT;
    // CGRAD's operator: formed explicitly where the pattern allows (schur.cu)
    // and two products were not asked for; in the FP32-tangent mode only on request
    const bool want_s2 = !ls->two_products && (!kept || ls->schur);
    if (want_s2) CR_CHECK(schur_pattern(L));
    const bool use_s2 = want_s2 && L->s2_state == 1;
    if (ls->schur) L->s2_asked = true;
    if (use_s2) {
        CR_CHECK(schur_form<M>(L, mG, Gt, mL));
        if (cg_nface > 0) CR_CHECK(schur_faces(L, cg_nface));
    }
    CR_CHECK(sell_mats(L, &Ks, &Gs, &GLs, !use_s2));
    launch(k_to_sell<M>, grid_for(nNo, 256), 256, 0, s, L->rowptr, (const int*)L->sell_ptr.p, nNo, mK, mG, Gt, mL,
           L->npad, Ks, use_s2 ? nullptr : Gs, GLs);
    int gm_ok = 0;
    if (ls->GM.sD >= 1 && ls->GM.sD <= kGmMaxSD) CR_CHECK(gm_faces_prepare(L, &gm_ok));
    // One GMRES solve K X = R: k_gmres, whose statistics wait in slot g, or
    // the form driven by the host (which also sets X = 0 where no cycle may run)
    const bool gm_one = gm_ok && !kept && ls->GM.mItr >= 1;
    auto gmres_any = [&](const double* R_, double* X_, int g) -> int {
        if (!gm_one) return gmres<M, B>(C, ls->GM, (const M*)Ks, R_, X_, gm_ok != 0);
        CR_CUDA(cudaEventRecord(L->ev_gm[2 * g], s));
        CR_CHECK((gmres_launch<M, B>(C, ls->GM, (const M*)Ks, R_, X_, kSlotGm + 8 * g)));
        CR_CUDA(cudaEventRecord(L->ev_gm[2 * g + 1], s));
        return CRIMSON_OK;
    };
    auto gmres_stats = [&](int g) -> int {
        if (!gm_one) return CRIMSON_OK;
        float ms = 0.f;
        CR_CUDA(cudaEventElapsedTime(&ms, L->ev_gm[2 * g], L->ev_gm[2 * g + 1]));
        return gmres_finish(C, ls->GM, kSlotGm + 8 * g, 1e-3 * ms);
    };
    const int gram_grid = grid_for(4LL * nNo, kGramThreads, 4);
    CR_CHECK(L->gramPart.alloc((size_t)kGramSums * gram_grid));
    auto combine = [&](const ColCoefs& cf, int m, int step, const double* Xu, const double* Xp, const double* y0u,
                       const double* y0p, double* yu, double* yp) {
        launch(k_combine, grid_for((yu ? 4LL : 1LL) * nNo, 256), 256, 0, s, cf, m, step, Xu, Xp, y0u, y0p, yu, yp, nv,
               (long long)nNo);
    };
    int i, iBB = 0;
    for (i = 1; i <= ls->RI.mItr; ++i) {
        iB = 2 * i - 1;
        iBB = 2 * i;
        ls->RI.dB = ls->RI.fNorm;
        CR_CHECK(gmres_any(L->Rm.p, Ucol(i - 1), 0));
        C.vs3(mD, (const double*)Ucol(i - 1), Pcol(i - 1), (const double*)L->Rc.p);   // Rc - D u
        CR_CHECK(cgrad_launch<M>(C, ls->CG, (const M*)Gs, (const typename V4<M>::type*)GLs, Pcol(i - 1), cg_nface,
                                 cg_coef, use_s2));
        C.sv3(mG, (const double*)Pcol(i - 1), MUc(iB - 1), (const double*)L->Rm.p, MUc(iBB - 1));   // G p, Rm - G p
        CR_CHECK(gmres_any(MUc(iBB - 1), Ucol(i - 1), 1));
        if (std::is_same<M, double>::value)
            C.vv3s((const M*)Ks, (const double*)Ucol(i - 1), MUc(iBB - 1));  // the sliced copy is FP64
        else
            C.vv3(mK, (const double*)Ucol(i - 1), MUc(iBB - 1));
        C.addbcmul(0, 3, (const double*)Ucol(i - 1), MUc(iBB - 1));
        C.ss(mL, (const double*)Pcol(i - 1), MPc(iB - 1));
        C.vs3(mD, (const double*)Ucol(i - 1), MPc(iBB - 1));
        // Gram matrix entries for columns iB, iBB
        int nsum = 0;
        if (kept)
            for (int k = iB; k <= iBB; ++k) {
                auto both = [&](const double* u, const double* p) {
                    C.dot((const double*)u, (const double*)MUc(k - 1), nv, kSlotGram + nsum++);
                    C.dot((const double*)p, (const double*)MPc(k - 1), nNo, kSlotGram + nsum++);
                };
                for (int j = 1; j <= k; ++j) both(MUc(j - 1), MPc(j - 1));
                both(L->Rmi.p, L->Rci.p);
            }
        for (int o0 = 0; !kept && (o0 == 0 || o0 < iB - 1); o0 += kGramCols) {
            launch(k_gram_part, gram_grid, kGramThreads, 0, s, (const double*)L->MU.p, (const double*)L->MP.p,
                   (const double*)L->Rmi.p, (const double*)L->Rci.p, nv, (long long)nNo, iB - 1, o0,
                   std::min(kGramCols, iB - 1 - o0), L->gramPart.p);
            launch(k_gram_sum, kGramSums, 32, 0, s, (const double*)L->gramPart.p, gram_grid, C.sc(kSlotGram + nsum));
            nsum += kGramSums;
        }
        CR_CUDA(cudaMemcpyAsync(L->hscal + kSlotCg, L->scal.p + kSlotCg, sizeof(double) * (64 - kSlotCg),
                                cudaMemcpyDeviceToHost, s));
        CR_CHECK(C.sync_scal(kSlotGram, nsum));
        CR_CHECK(gmres_stats(0));
        CR_CHECK(cgrad_finish<M>(C, ls->CG));
        CR_CHECK(gmres_stats(1));
        const double* g = L->hscal + kSlotGram;
        if (kept) {
            for (int k = iB; k <= iBB; ++k) {
                for (int j = 1; j < k; ++j, g += 2) Aa(j - 1, k - 1) = Aa(k - 1, j - 1) = g[0] + g[1];
                Aa(k - 1, k - 1) = std::pow(std::sqrt(g[0]), 2.0) + std::pow(std::sqrt(g[1]), 2.0);
                Bv[k - 1] = g[2] + g[3];
                g += 4;
            }
        } else {
            Aa(iB - 1, iB - 1) = g[0];
            Aa(iB - 1, iBB - 1) = Aa(iBB - 1, iB - 1) = g[1];
            Aa(iBB - 1, iBB - 1) = g[2];
            Bv[iB - 1] = g[3];
            Bv[iBB - 1] = g[4];
            for (int j = 0; j < iB - 1; ++j) {
                const double* o = g + (size_t)(j / kGramCols) * kGramSums + 5 + 2 * (j % kGramCols);
                Aa(j, iB - 1) = Aa(iB - 1, j) = o[0];
                Aa(j, iBB - 1) = Aa(iBB - 1, j) = o[1];
            }
        }
        for (int t = 0; t < iBB; ++t) xB[t] = Bv[t];
        std::vector<double> Asub((size_t)iBB * iBB);
        for (int c = 0; c < iBB; ++c)
            for (int r = 0; r < iBB; ++r) Asub[(size_t)c * iBB + r] = Aa(r, c);
        CR_CHECK(ge_solve(iBB, Asub.data(), xB.data()));
        for (int t = 0; t < iBB; ++t)
            if (!std::isfinite(xB[t])) {
                set_last_error("NSSOLVER: non-finite least-squares coefficients");
                return CRIMSON_ERR_NONFINITE;
            }
        double sxb = 0.0;
        for (int t = 0; t < iBB; ++t) sxb = sxb + xB[t] * Bv[t];
        ls->RI.fNorm = std::sqrt(std::pow(ls->RI.iNorm, 2.0) - sxb);
        if (ls->RI.fNorm < eps) {
            ls->RI.suc = 1;
            break;
        }
        // Rm = Rmi - sum xB_j MU_j ; Rc = Rci - sum xB_j MP_j
        ColCoefs cf;
        for (int j = 0; j < iBB; ++j) cf.c[j] = -xB[j];
        combine(cf, iBB, 1, L->MU.p, L->MP.p, L->Rmi.p, L->Rci.p, L->Rm.p, L->Rc.p);
    }
    if (i > ls->RI.mItr) {
        ls->RI.itr = ls->RI.mItr;
    } else {
        ls->RI.itr = i;
        ColCoefs cf;
        for (int j = 0; j < iBB; ++j) cf.c[j] = -xB[j];
        combine(cf, iBB, 1, nullptr, L->MP.p, nullptr, L->Rci.p, nullptr, L->Rc.p);
    }
    C.dot((const double*)L->Rc.p, (const double*)L->Rc.p, nNo, 0);
    CR_CHECK(C.sync_scal(0, 1));
    ls->Resc = (int)std::lround(100.0 * std::pow(std::sqrt(L->hscal[0]) / ls->RI.fNorm, 2.0));
    ls->Resm = 100 - ls->Resc;
    // solution: Rmi = xB(2) U_1 + sum xB(2i) U_i ; Rci = xB(1) P_1 + sum xB(2i-1) P_i
    {
        ColCoefs cu, cp;
        for (i = 1; i <= ls->RI.itr; ++i) {
            cu.c[i - 1] = xB[2 * i - 1];
            cp.c[i - 1] = xB[2 * i - 2];
        }
        combine(cp, ls->RI.itr, 1, nullptr, L->P.p, nullptr, nullptr, nullptr, L->Rci.p);
        launch(k_combine, grid_for(nv, 256), 256, 0, s, cu, ls->RI.itr, 1, (const double*)nullptr, (const double*)L->U.p,
               (const double*)nullptr, (const double*)nullptr, (double*)nullptr, L->Rmi.p, 0LL, nv);
    }
    launch(k_merge4, grid_for(nNo, 256), 256, 0, s, R, (const double*)L->Rmi.p, (const double*)L->Rci.p, nNo);
    CR_CUDA(cudaStreamSynchronize(s));
    ls->RI.callD = now_s() - t0;
    ls->RI.dB = 10.0 * std::log(ls->RI.fNorm / ls->RI.dB);
    CR_CUDA(cudaGetLastError());
    return CRIMSON_OK;
}

static int lhs_work_alloc(crimson_lhs* L, const crimson_ls* ls) {
    const int nNo = L->nNo;
    const long long nnz = L->nnz;
    const int iB = ls->RI.mItr;
    const int sD = ls->GM.sD;
    if (sD + 1 > 512 || 8 * iB * iB + 64 > 4096 || iB > kMaxCols / 2) return CRIMSON_ERR_UNSUPPORTED;
    CR_CHECK(L->W.alloc(4 * (size_t)nNo));
    CR_CHECK(L->R.alloc(4 * (size_t)nNo));
    CR_CHECK(L->mK.alloc(9 * (size_t)nnz));
    CR_CHECK(L->mG.alloc(3 * (size_t)nnz));
    CR_CHECK(L->mD.alloc(3 * (size_t)nnz));
    CR_CHECK(L->mL.alloc((size_t)nnz));
    CR_CHECK(L->Rm.alloc(3 * (size_t)nNo));
    CR_CHECK(L->Rc.alloc((size_t)nNo));
    CR_CHECK(L->Rmi.alloc(3 * (size_t)nNo));
    CR_CHECK(L->Rci.alloc((size_t)nNo));
    CR_CHECK(L->U.alloc(3 * (size_t)nNo * iB));
    CR_CHECK(L->P.alloc((size_t)nNo * iB));
    CR_CHECK(L->MU.alloc(3 * (size_t)nNo * 2 * iB));
    CR_CHECK(L->MP.alloc((size_t)nNo * 2 * iB));
    CR_CHECK(L->basis.alloc(3 * (size_t)nNo * (sD + 1)));
    CR_CHECK(L->w3.alloc(3 * (size_t)nNo));
    CR_CHECK(sell_pattern(L));
    // each on its own: a call that failed part-way is made up for by the next
    CR_CHECK(L->scal.alloc(kScalTotal));
    if (!L->red.ticket.p) CR_CHECK(L->red.init());
    if (!L->hscal) CR_CUDA(cudaMallocHost(&L->hscal, sizeof(double) * kScalTotal));
    cudaEvent_t* const ev[] = {&L->ev0,       &L->ev1,       &L->ev_gm[0],  &L->ev_gm[1],
                               &L->ev_gm[2],  &L->ev_gm[3],  &L->s2_ev0,    &L->s2_ev1};
    for (cudaEvent_t* e : ev)
        if (!*e) CR_CUDA(cudaEventCreate(e));
    return CRIMSON_OK;
}

// memLS_SOLVE face flags (memLS.f90:1955-1986)
static void set_face_flags(crimson_lhs* L, const int* incL, const double* res) {
    for (int fa = 0; fa < L->nFaces; ++fa) {
        MemlsFace& f = L->face[fa];
        f.incFlag = !(incL && incL[fa] == 0);
        f.coupledFlag = false;
        if (!f.incFlag) continue;
        if (f.bGrp == CRIMSON_BC_TYPE_NEU && res && res[fa] != 0.0) {
            f.res = res[fa];
            f.coupledFlag = true;
        }
    }
}

// Dirichlet W scaling + valM of coupled faces (tail of PRECOND)
static int precond_faces(crimson_lhs* L, bool after_scale) {
    cudaStream_t s = L->stream;
    for (auto& f : L->face) {
        if (!f.created || f.nNo == 0) continue;
        if (!after_scale) {
            if (f.incFlag && f.bGrp == CRIMSON_BC_TYPE_DIR)
                launch(k_w_dirichlet, grid_for(f.nNo, 256), 256, 0, s, f.glob.p, f.val.p, f.dof, std::min(f.dof, 4),
                       f.nNo, L->W.p);
        } else if (f.coupledFlag) {
            launch(k_valm, grid_for(f.nNo, 256), 256, 0, s, f.glob.p, f.val.p, f.valM.p, f.dof, std::min(f.dof, 4),
                   f.nNo, L->W.p);
        }
    }
    CR_CUDA(cudaGetLastError());
    return CRIMSON_OK;
}

// One line per NS solve in the format of memLS's LOGFILE
// (flowsolver/src/memLS.f90:1720-1757), appended to ls->log_path when set:
// a header "gnNo nTasks nCoupledFaces" when the file is new, then the
// success code (100 RI + 10 GM + CG), RI / GM / CG iterations, the time
// split other / GM / CG in percent, the initial norm, the relative final
// norm, the wall time, Resm, Resc and dB.  The solve's time is the host's wall
// clock as in memLS; the shares of GM and CG are the device times of their
// kernels (the host does not wait for each), for GMRES driven by the host its
// wall clock.
static void log_solve(const crimson_lhs* L, const crimson_ls* ls) {
    if (ls->log_path.empty()) return;
    FILE* probe = std::fopen(ls->log_path.c_str(), "r");
    const bool exists = probe != nullptr;
    if (probe) std::fclose(probe);
    FILE* f = std::fopen(ls->log_path.c_str(), "a");
    if (!f) return;
    if (!exists) {
        int nc = 0;
        for (const auto& fc : L->face)
            if (fc.coupledFlag) ++nc;
        std::fprintf(f, "%12d%12d%12d\n", L->gnNo, 1, nc);
    }
    const int code = (ls->RI.suc ? 100 : 0) + (ls->GM.suc ? 10 : 0) + (ls->CG.suc ? 1 : 0);
    const double t = ls->RI.callD > 0.0 ? ls->RI.callD : 1.0;
    std::fprintf(f, "%4.3d%3d%4d%5d%4ld%4ld%4ld%9.2E%9.2E%9.2E%4d%4d%4ld\n", code, ls->RI.itr, ls->GM.itr,
                 ls->CG.itr, std::lround((ls->RI.callD - ls->GM.callD - ls->CG.callD) / t * 1e2),
                 std::lround(ls->GM.callD / t * 1e2), std::lround(ls->CG.callD / t * 1e2), ls->RI.iNorm,
                 ls->RI.iNorm != 0.0 ? ls->RI.fNorm / ls->RI.iNorm : 0.0, ls->RI.callD, ls->Resm, ls->Resc,
                 std::lround(ls->RI.dB));
    std::fclose(f);
}

static void copy_stats(const crimson_ls* ls, crimson_ls_stats* st) {
    if (!st) return;
    st->GM = ls->GM;
    st->CG = ls->CG;
    st->RI = ls->RI;
    st->LS_type = ls->LS_type;
    st->Resm = ls->Resm;
    st->Resc = ls->Resc;
}

// FP64 defect of the scaled system: D4 = R0 - A x (A with the coupled-face
// momentum term of ADDBCMUL(ADD)); returns |D4| and |R0|.
static int defect64(crimson_lhs* L, const double* R0, const double* x4, double* D4, double* nD, double* nR) {
    Ctx C{L, L->stream};
    cudaStream_t s = L->stream;
    const int n = L->nNo;
    // x split into xu (3, n) in Rmi and xp (n) in Rci; products into MU/MP slots 0
    launch(k_split4, grid_for(n, 256), 256, 0, s, x4, L->Rmi.p, L->Rci.p, n);
    double* KU = L->MU.p;
    double* GPm = L->MU.p + 3 * (size_t)n;
    double* DU = L->MP.p;
    double* LP = L->MP.p + (size_t)n;
    C.vv3((const double*)L->mK.p, (const double*)L->Rmi.p, KU);
    C.addbcmul(0, 3, (const double*)L->Rmi.p, KU);
    C.sv3((const double*)L->mG.p, (const double*)L->Rci.p, GPm);
    C.vs3((const double*)L->mD.p, (const double*)L->Rmi.p, DU);
    C.ss((const double*)L->mL.p, (const double*)L->Rci.p, LP);
    launch(k_defect4, grid_for(n, 256), 256, 0, s, R0, (const double*)KU, (const double*)GPm, (const double*)DU,
           (const double*)LP, D4, n);
    C.dot(D4, (const double*)D4, 4LL * n, 0);
    C.dot(R0, R0, 4LL * n, 1);
    CR_CHECK(C.sync_scal(0, 2));
    *nD = std::sqrt(L->hscal[0]);
    *nR = std::sqrt(L->hscal[1]);
    return CRIMSON_OK;
}

// NSSOLVER on the scaled system in L->R (in/out).  FP64: the reference's
// arithmetic.  Mixed: FP32 sliced copies of the scaled split matrices drive
// the Krylov matvecs (GMRES, CGRAD); every other product, in particular the
// A d of the search directions that enter the least-squares problem, uses
// the FP64 matrices, so a sweep's residual estimate is that of the FP64
// operator.  Each sweep solves A d = D, adds d to the FP64 solution and
// forms the FP64 defect D = R0 - A x, until |D| <= refine_tol |R0|
// (RI.relTol when refine_tol <= 0) or max_refine sweeps.  Every sweep's
// NSSOLVER stops at its own relative tolerances, so the sweeps reach a
// defect below what one NSSOLVER's estimate can resolve.  Iteration counts
// are summed over the sweeps.  has_gt: Gt is a separate matrix (host Val path),
// otherwise mD serves as Gt.
static int solve_scaled(crimson_lhs* L, crimson_ls* ls, bool has_gt) {
    cudaStream_t s = L->stream;
    const double* Gt64 = has_gt ? L->Gt.p : L->mD.p;
    if (ls->precision == CRIMSON_FP64)
        return nssolver<double, double>(L, ls, L->mK.p, L->mG.p, L->mD.p, L->mL.p, Gt64, L->R.p);
    const int n = L->nNo;
    CR_CHECK(L->R0.alloc(4 * (size_t)n));
    CR_CHECK(L->X4.alloc(4 * (size_t)n));
    CR_CUDA(cudaMemcpyAsync(L->R0.p, L->R.p, sizeof(double) * 4 * (size_t)n, cudaMemcpyDeviceToDevice, s));
    CR_CUDA(cudaMemsetAsync(L->X4.p, 0, sizeof(double) * 4 * (size_t)n, s));
    crimson_subls gm{}, cg{}, ri{};
    const double tol = ls->refine_tol > 0.0 ? ls->refine_tol : ls->RI.relTol;
    double rel = 1.0;
    L->refine_steps = 0;
    // Each sweep solves for the defect scaled to the norm of the original
    // right side, so the Krylov solvers' absolute tolerances and GE's
    // absolute pivot test see the same magnitudes in every sweep.  A later
    // sweep only has to bring the defect from nD to tol nR: its outer
    // relative tolerance is kRefineSafety * tol nR / nD (never tighter than
    // the first sweep's), so it stops after the reduction it needs.
    constexpr double kRefineSafety = 0.3;
    struct RelTolGuard {
        crimson_subls& ri;
        double v;
        ~RelTolGuard() { ri.relTol = v; }
    } guard{ls->RI, ls->RI.relTol};
    double sigma = 1.0;
    for (int ref = 0; ref < std::max(ls->max_refine, 1); ++ref) {
        CR_CHECK((nssolver<float, float>(L, ls, L->mK.p, L->mG.p, L->mD.p, L->mL.p, Gt64, L->R.p)));
        if (ref == 0) {
            gm = ls->GM;
            cg = ls->CG;
            ri = ls->RI;
        } else {
            gm.itr += ls->GM.itr;
            cg.itr += ls->CG.itr;
            ri.itr += ls->RI.itr;
            gm.callD += ls->GM.callD;
            cg.callD += ls->CG.callD;
            ri.callD += ls->RI.callD;
        }
        launch(k_axpy<double, double>, grid_for(4LL * n, 256), 256, 0, s, 1.0 / sigma, (const double*)L->R.p,
               L->X4.p, 4LL * n);
        double nD = 0.0, nR = 0.0;
        CR_CHECK(defect64(L, L->R0.p, L->X4.p, L->R.p, &nD, &nR));
        rel = nR > 0.0 ? nD / nR : 0.0;
        L->refine_steps = ref + 1;
        L->refine_rel = rel;
        if (!(rel > tol) || nD == 0.0) break;
        if (!std::isfinite(rel)) return CRIMSON_ERR_NONFINITE;
        sigma = nR / nD;
        launch(k_scale, grid_for(4LL * n, 256), 256, 0, s, sigma, L->R.p, 4LL * n);
        ls->RI.relTol = std::min(0.5, std::max(guard.v, kRefineSafety * tol / rel));
    }
    ls->RI.relTol = guard.v;
    ri.relTol = guard.v;
    ri.fNorm = rel * ri.iNorm;
    ri.suc = rel <= tol ? 1 : 0;
    ls->GM = gm;
    ls->CG = cg;
    ls->RI = ri;
    CR_CUDA(cudaMemcpyAsync(L->R.p, L->X4.p, sizeof(double) * 4 * (size_t)n, cudaMemcpyDeviceToDevice, s));
    return CRIMSON_OK;
}

int memls_solve_val(crimson_lhs* L, crimson_ls* ls, double* Ri, double* Val, const int* incL, const double* res,
                    crimson_ls_stats* st) {
    cudaStream_t s = L->stream;
    CR_CHECK(lhs_work_alloc(L, ls));
    CR_CHECK(L->Val.alloc(16 * (size_t)L->nnz));
    CR_CHECK(L->Gt.alloc(3 * (size_t)L->nnz));
    set_face_flags(L, incL, res);
    CR_CUDA(cudaMemcpyAsync(L->R.p, Ri, sizeof(double) * 4 * (size_t)L->nNo, cudaMemcpyHostToDevice, s));
    CR_CUDA(cudaMemcpyAsync(L->Val.p, Val, sizeof(double) * 16 * (size_t)L->nnz, cudaMemcpyHostToDevice, s));
    launch(k_w_from_val, grid_for(L->nNo, 256), 256, 0, s, L->Val.p, L->diag, L->W.p, L->nNo);
    CR_CHECK(precond_faces(L, false));
    launch(k_scale_split_val, grid_for(L->nNo, 128), 128, 0, s, L->Val.p, L->rowptr, L->col, L->diag,
           (const double*)L->W.p, L->nNo, L->mK.p, L->mG.p, L->mD.p, L->mL.p);
    launch(k_gt, grid_for(L->nnz, 256), 256, 0, s, (const double*)L->mG.p, L->trans, L->nnz, L->Gt.p);
    launch(k_mul, grid_for(4LL * L->nNo, 256), 256, 0, s, L->R.p, (const double*)L->W.p, 4LL * L->nNo);
    CR_CHECK(precond_faces(L, true));
    CR_CHECK(solve_scaled(L, ls, true));
    launch(k_mul, grid_for(4LL * L->nNo, 256), 256, 0, s, L->R.p, (const double*)L->W.p, 4LL * L->nNo);
    CR_CUDA(cudaMemcpyAsync(Ri, L->R.p, sizeof(double) * 4 * (size_t)L->nNo, cudaMemcpyDeviceToHost, s));
    CR_CUDA(cudaMemcpyAsync(Val, L->Val.p, sizeof(double) * 16 * (size_t)L->nnz, cudaMemcpyDeviceToHost, s));
    CR_CUDA(cudaStreamSynchronize(s));
    copy_stats(ls, st);
    log_solve(L, ls);
    return CRIMSON_OK;
}

// K_out(j) = K_in(trans(j))^T: the momentum blocks of the transposed system
__global__ void k_transpose_k(const double* __restrict__ Kin, const int* __restrict__ trans, long long nnz,
                              double* __restrict__ Kout) {
    for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < nnz; j += (long long)gridDim.x * blockDim.x) {
        const double* k = Kin + 9 * (size_t)trans[j];
        double* o = Kout + 9 * (size_t)j;
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) o[3 * a + b] = k[3 * b + a];
    }
}

// R(4, i) = -R(4, i)
__global__ void k_negate_p(double* __restrict__ R, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) R[4 * (size_t)i + 3] = -R[4 * (size_t)i + 3];
}

// transpose: solve with the transposed matrix.  Val4 = [K G; D L] built from
// lhsK / lhsP has G = -D^T (both come from lhsP(1:3)) and a symmetric L
// (the PSPG block is symmetrised per element), so
//   A^T = [K^T  -G; -D  L]  and  A^T [u; p] = [f; g]  <=>  [K^T G; D L] [u; -p] = [f; -g]:
// the same NS solve with the momentum blocks transposed and the pressure
// rows of the right side and of the solution negated.  The diagonal
// scaling, Dirichlet faces and the (symmetric) coupled-face terms carry over.
int memls_solve_lhs_device(crimson_lhs* L, crimson_ls* ls, const double* d_res, const double* d_lhsK,
                           const double* d_lhsP, const int* incL, const double* faceRes, double* d_sol,
                           crimson_ls_stats* st, bool transpose, const float* d_lhs32) {
    const TangentIn T{d_lhsK, d_lhsP, d_lhs32};
    cudaStream_t s = L->stream;
    CR_CHECK(lhs_work_alloc(L, ls));
    set_face_flags(L, incL, faceRes);
    CR_CUDA(cudaMemcpyAsync(L->R.p, d_res, sizeof(double) * 4 * (size_t)L->nNo, cudaMemcpyDeviceToDevice, s));
    launch(k_w_from_lhs, grid_for(L->nNo, 256), 256, 0, s, T, L->diag, L->W.p, L->nNo);
    CR_CHECK(precond_faces(L, false));
    launch(k_scale_split_lhs, grid_for(16LL * L->nNo, 128), 128, 0, s, T, L->rowptr, L->col, L->diag, L->trans,
           (const double*)L->W.p, L->nNo, L->mK.p, L->mG.p, L->mD.p, L->mL.p);
    launch(k_mul, grid_for(4LL * L->nNo, 256), 256, 0, s, L->R.p, (const double*)L->W.p, 4LL * L->nNo);
    CR_CHECK(precond_faces(L, true));
    if (transpose) {
        CR_CHECK(L->mKt.alloc(9 * (size_t)L->nnz));
        launch(k_transpose_k, grid_for(L->nnz, 256), 256, 0, s, (const double*)L->mK.p, L->trans, L->nnz, L->mKt.p);
        std::swap(L->mK, L->mKt);
        launch(k_negate_p, grid_for(L->nNo, 256), 256, 0, s, L->R.p, L->nNo);
    }
    // With Val4 built from lhsK/lhsP, Gt = -mG^T equals mD up to the order of
    // the two scaling products, so mD serves as Gt.
    CR_CHECK(solve_scaled(L, ls, false));
    if (transpose) launch(k_negate_p, grid_for(L->nNo, 256), 256, 0, s, L->R.p, L->nNo);
    launch(k_mul, grid_for(4LL * L->nNo, 256), 256, 0, s, L->R.p, (const double*)L->W.p, 4LL * L->nNo);
    CR_CUDA(cudaMemcpyAsync(d_sol, L->R.p, sizeof(double) * 4 * (size_t)L->nNo, cudaMemcpyDeviceToDevice, s));
    CR_CUDA(cudaStreamSynchronize(s));
    copy_stats(ls, st);
    log_solve(L, ls);
    return CRIMSON_OK;
}

// Diagnostics.  which: 0 = 3x3 block SpMV (K, sliced, FP64, as GMRES runs
// it), 1 = one CG iteration of the persistent FP64 CGRAD kernel (average over
// all launches so far, from CUDA events recorded around each launch),
// 2 = SPARMULSV (G), 3 = fused MGS step, 4 = one CG iteration of the
// FP32-matrix CGRAD kernel, 5 = 3x3 block SpMV with the sliced FP32 K,
// 6 = 3x3 block SpMV on the CSR FP64 K (four lanes per row).
int memls_kernel_time(crimson_lhs* L, int which, int reps, double* ms) {
    if (which == 1 || which == 4) {
        const auto& acc = which == 1 ? L->cg_acc64 : L->cg_acc32;
        if (acc.iters <= 0) return CRIMSON_ERR_STATE;
        *ms = acc.ms / (double)acc.iters;
        return CRIMSON_OK;
    }
    if (!L->mK.p || !L->basis.p || reps <= 0) return CRIMSON_ERR_STATE;
    if ((which == 5 && !L->Ks32.p) || (which == 0 && !L->Ks64.p)) return CRIMSON_ERR_STATE;
    cudaStream_t s = L->stream;
    Ctx C{L, s};
    const long long n3 = 3LL * L->nNo;
    cudaEvent_t e0, e1;
    CR_CUDA(cudaEventCreate(&e0));
    CR_CUDA(cudaEventCreate(&e1));
    auto run = [&]() {
        switch (which) {
            case 0: C.vv3s((const double*)L->Ks64.p, (const double*)L->basis.p, L->basis.p + n3); break;
            case 6: C.vv3((const double*)L->mK.p, (const double*)L->basis.p, L->basis.p + n3); break;
            case 2: C.sv3((const double*)L->mG.p, (const double*)L->P.p, L->w3.p); break;
            case 5: C.vv3s((const float*)L->Ks32.p, (const double*)L->basis.p, L->basis.p + n3); break;
            default:
                launch(k_mgs<double>, red_grid(n3), 256, 0, s, L->basis.p + 2 * n3, (const double*)L->basis.p,
                       (const double*)C.sc(kSlotH), (const double*)(L->basis.p + n3), n3, L->red.part.p,
                       L->red.ticket.p, C.sc(kSlotH + 1));
        }
    };
    for (int i = 0; i < 2; ++i) run();
    CR_CUDA(cudaEventRecord(e0, s));
    for (int i = 0; i < reps; ++i) run();
    CR_CUDA(cudaEventRecord(e1, s));
    CR_CUDA(cudaEventSynchronize(e1));
    float t = 0.f;
    CR_CUDA(cudaEventElapsedTime(&t, e0, e1));
    *ms = (double)t / reps;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    CR_CUDA(cudaGetLastError());
    return CRIMSON_OK;
}

}  // namespace crimson
