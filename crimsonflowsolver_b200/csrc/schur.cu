// Explicit Schur operator of memLS's CGRAD.
//
// memLS's CGRAD (flowsolver/src/memLS.f90:367-430) iterates on the
// continuity Schur complement without forming it: every iteration computes
// SP = L P - Gt (G P) - (coupled-face terms) as two sparse products.  Here
// S = L - Gt G is formed once per NSSOLVER call, in FP64 and in a fixed
// order, on the 2-ring pattern of the node graph, stored in FP64 or, for the
// mixed-precision solve, rounded once to FP32 with an FP64 correction of the
// own row's term that restores the row sum; an iteration is then one sparse
// product.  (The smooth modes are the ones the operator nearly annihilates
// and the rounding disturbs most: without the correction a mixed solve is up
// to 5e-10 from the FP64 one, with it 4e-11 in the median of 70 drawn
// systems; two products with rounded G, Gt, L and gathered {GP, P} 1.7e-10.)  Against the two products the stream per row is smaller
// (about 62 entries of 8 + 2 B against 14.7 blocks of 7 values: 620 / 823 B
// in FP64, 372 / 412 B in FP32), and an iteration has two grid-wide barriers
// instead of three.  (The two-product kernel stays for patterns that do not
// qualify: rows of more than kS2Cap entries, or column offsets past 16 bits
// -- a numbering without locality, where four times as many gathers would
// each cost a sector of their own.)
//
// Layout.  Rows in slices of 32 (one warp), a slice as wide as its longest
// row, cut into chunks of up to kS2Chunk columns.  A chunk is contiguous: its
// values column by column (32 rows each), then its int16 column offsets
// col - row: one bulk copy brings it into shared memory.
//
// CG kernel (persistent, one block per SM).  A block owns a contiguous range
// of slices.  Its warps take them in turn, so that at any time they gather
// from neighbouring rows and find them in the L1 (contiguous ranges per warp
// instead: 107 us against 97 per FP32 iteration on the 4M-tet cylinder); the
// slices left after the last full turn are split chunk by chunk, partial rows
// summed through shared memory in warp order.  Two forms:
//   * resident: where the block's chunks fit in shared memory (meshes up to
//     about 300,000 tets in FP64, 500,000 in FP32) they are loaded once per
//     call and no iteration touches the operator in memory again; bound by
//     the two barriers (1.2 and 2.0 us on 20 blocks, 2.6 and 3.9 on 148) and
//     one gather latency: 108k tets, 148 blocks, barrier stalls 28.6 per issue
//     of 38;
//   * streaming: every warp runs its chunks through a ring of two
//     shared-memory stages filled by cp.async.bulk, so the stream does not
//     stop at slice ends, barriers or iteration ends; bound by HBM, the
//     gathers' latency and the barriers together (2.1M tets: 46 us per FP64
//     iteration, 5.3 TB/s, DRAM 64% busy; 35 us FP32, 4.1 TB/s, 50%).
// Per iteration, before (two-product kernel) and now, B200: 4M-tet cylinder
// 118 / 80 us FP64, 74 / 57 FP32; 452k-tet bifurcation 24.6 / 16 FP32;
// 108k-tet cylinder 20 / 9.2 FP64; 1152 tets 15 / 5.5 FP64.
// S is formed in every NSSOLVER call, 2.2 ms on 4M tets: the time that 60 FP64
// or 130 FP32 iterations gain.  Solves at loose tolerances (0.4 / 0.01 / 0.2)
// take 111-290 there: whole steps 90 -> 71 ms FP64, 65 -> 58 mixed; 41-111 on
// 108k tets: 10 -> 5 ms and 8.9 -> 5.2.
//
// Iteration.  S P is kept by the recurrence S P = S R + beta S P_prev, so the
// product gathers only R (8 B per entry) and does not wait for P:
//   phase 1  SP = S R + beta SP, P = R + beta P, <P, SP>, w_f . P, z_f . P
//   barrier  alpha, and the coupled-face coefficients
//   phase 2  X += alpha P, R -= alpha (SP - sum_f coef_f (w_f . P) z_f), |R|^2
//   barrier  beta; orders R's new values before the next gathers
// The coupled-face term is exact: Gt (G P + c valM (valM . G P)) =
// Gt G P + c (w . P) z with w = G^T valM, z = Gt valM built once per NSSOLVER
// call; w and z vanish outside the faces' neighbourhoods, so a bit per slice
// says where they are read.
#include <algorithm>
#include <climits>
#include <vector>

#include "common.cuh"
#include "gridred.cuh"
#include "memls.cuh"

namespace crimson {

constexpr int kS2Cap = 256;        // 2-ring entries per row
constexpr int kS2Hash = 1024;      // slots of the pattern kernel's per-row set
constexpr int kS2Chunk = 8;        // columns of a chunk
constexpr int kS2FormWarps = 16;   // formation: rows in flight per block
constexpr int kS2CgWarps = 24;     // most warps of a CG block (80 registers a thread)
constexpr int kS2MaxFaces = 8;
constexpr int kS2Vals = 1 + 2 * kS2MaxFaces;   // reductions of one barrier

// Bytes of one column of a chunk (32 values and offsets).
template <typename M>
__host__ __device__ constexpr int s2_col_bytes() {
    return 32 * (int)(sizeof(M) + sizeof(short));
}

// Byte offset of entry e of a row (lane = row & 31) in the operator, and of
// its column offset; c0 = the slice's first column, w its width.
template <typename M>
__device__ __forceinline__ size_t s2_val_pos(int c0, int w, int e, int lane) {
    const int k0 = e & ~(kS2Chunk - 1), k = e - k0;
    constexpr int V = 16 / (int)sizeof(M);
    const size_t base = (size_t)(c0 + k0) * s2_col_bytes<M>();
    if (w - k0 >= kS2Chunk) return base + (size_t)((k / V) * 32 + lane) * 16 + (size_t)(k % V) * sizeof(M);
    return base + (size_t)(k * 32 + lane) * sizeof(M);
}
template <typename M>
__device__ __forceinline__ size_t s2_off_pos(int c0, int w, int e, int lane) {
    const int k0 = e & ~(kS2Chunk - 1), k = e - k0, kc = min(kS2Chunk, w - k0);
    const size_t base = (size_t)(c0 + k0) * s2_col_bytes<M>() + (size_t)kc * 32 * sizeof(M);
    if (kc == kS2Chunk) return base + (size_t)lane * 16 + (size_t)k * sizeof(short);
    return base + (size_t)(k * 32 + lane) * sizeof(short);
}

// ---------------------------------------------------------------------------
// Pattern: the sorted 2-ring of every row, one warp per row.  The distinct
// columns are collected in a shared-memory hash set and sorted by counting.
// Returns the row length (> kS2Cap: the row overflows).
// ---------------------------------------------------------------------------
__device__ int s2_ring2(const int* __restrict__ rowptr, const int* __restrict__ col, int r, int* set, int* list) {
    const int lane = threadIdx.x & 31;
    for (int q = lane; q < kS2Hash; q += 32) set[q] = -1;
    __syncwarp();
    const int rs = rowptr[r], re = rowptr[r + 1];
    int mine = 0;
    for (int t = rs; t < re; ++t) {
        const int k = col[t], ks = rowptr[k], ke = rowptr[k + 1];
        for (int u = ks + lane; u < ke; u += 32) {
            const int j = col[u];
            unsigned h = ((unsigned)j * 2654435761u) >> 22;   // kS2Hash slots
            for (int probe = 0; probe < kS2Hash; ++probe) {
                const int old = atomicCAS(set + h, -1, j);
                if (old == -1) ++mine;
                if (old == -1 || old == j) break;
                h = (h + 1) & (kS2Hash - 1);
            }
        }
        __syncwarp();
        // stop before the set can fill up: the row is over the cap anyway
        int tot = mine;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
        if (tot > kS2Cap) return tot;
    }
    int len = mine;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) len += __shfl_xor_sync(0xffffffffu, len, o);
    if (!list) return len;
    // compact, then place every column at the number of smaller ones
    int base = 0;
    for (int q0 = 0; q0 < kS2Hash; q0 += 32) {
        const int j = set[q0 + lane];
        const unsigned m = __ballot_sync(0xffffffffu, j >= 0);
        __syncwarp();
        if (j >= 0) set[base + __popc(m & ((1u << lane) - 1u))] = j;   // at or before q0 + lane
        base += __popc(m);
        __syncwarp();
    }
    for (int e = lane; e < len; e += 32) {
        const int j = set[e];
        int rank = 0;
        for (int q = 0; q < len; ++q) rank += set[q] < j ? 1 : 0;
        list[rank] = j;
    }
    __syncwarp();
    return len;
}

// Row lengths; stat[0] the longest, stat[1] the largest |col - row|.
__global__ void __launch_bounds__(256) k_s2_len(const int* __restrict__ rowptr, const int* __restrict__ col, int n,
                                                int* __restrict__ len, int* __restrict__ stat) {
    __shared__ int sets[8][kS2Hash];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int* set = sets[wid];
    int mlen = 0, moff = 0;
    for (int r = blockIdx.x * 8 + wid; r < n; r += gridDim.x * 8) {
        const int l = s2_ring2(rowptr, col, r, set, nullptr);
        if (lane == 0) len[r] = l;
        mlen = max(mlen, l);
        for (int q = lane; q < kS2Hash; q += 32)
            if (set[q] >= 0) moff = max(moff, abs(set[q] - r));
        __syncwarp();
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) moff = max(moff, __shfl_xor_sync(0xffffffffu, moff, o));
    if (lane == 0) {
        atomicMax(stat, mlen);
        atomicMax(stat + 1, moff);
    }
}

// Column offsets of every row into the operator's layout (pads: 0, the row
// itself; their values stay zero).  One warp per row, pad rows of the last
// slice included.
template <typename M>
__global__ void __launch_bounds__(256) k_s2_offsets(const int* __restrict__ rowptr, const int* __restrict__ col, int n,
                                                    int nrows_pad, const int* __restrict__ sc,
                                                    unsigned char* __restrict__ op) {
    __shared__ int sets[8][kS2Hash];
    __shared__ int lists[8][kS2Cap];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int r = blockIdx.x * 8 + wid; r < nrows_pad; r += gridDim.x * 8) {
        const int len = r < n ? s2_ring2(rowptr, col, r, sets[wid], lists[wid]) : 0;
        const int c0 = sc[r >> 5], w = sc[(r >> 5) + 1] - c0;
        for (int e = lane; e < w; e += 32)
            *reinterpret_cast<short*>(op + s2_off_pos<M>(c0, w, e, r & 31)) =
                e < len ? (short)(lists[wid][e] - r) : (short)0;
        __syncwarp();
    }
}

// Per lhs, once: row lengths, slices, chunks, the blocks' slice ranges.
// s2_state 1: usable, -1: the pattern does not qualify (0: not built; a call
// that fails leaves that).
static int s2_build(crimson_lhs* L) {
    cudaStream_t s = L->stream;
    const int n = L->nNo;
    L->s2_state = -1;   // unusable unless every step below succeeds
    CR_CHECK(L->s2_len.alloc((size_t)n));
    DBuf<int> stat;
    CR_CHECK(stat.alloc(2));
    CR_CUDA(cudaMemsetAsync(stat.p, 0, 2 * sizeof(int), s));
    launch(k_s2_len, grid_for(n, 8, 16), 256, 0, s, L->rowptr, L->col, n, L->s2_len.p, stat.p);
    std::vector<int> len((size_t)n);
    int hs[2] = {0, 0};
    CR_CUDA(cudaMemcpyAsync(hs, stat.p, sizeof(hs), cudaMemcpyDeviceToHost, s));
    CR_CUDA(cudaMemcpyAsync(len.data(), L->s2_len.p, sizeof(int) * (size_t)n, cudaMemcpyDeviceToHost, s));
    CR_CUDA(cudaStreamSynchronize(s));
    CR_CUDA(cudaGetLastError());
    if (hs[0] > kS2Cap || hs[1] > 32767) return CRIMSON_OK;
    const int ns = (n + 31) / 32;
    std::vector<int> sc((size_t)ns + 1, 0);
    std::vector<long long> cp((size_t)ns + 1, 0);   // chunks before each slice
    long long cols = 0, nnz2 = 0;
    for (int q = 0; q < ns; ++q) {
        int w = 1;
        for (int r = q * 32; r < std::min(n, (q + 1) * 32); ++r) {
            w = std::max(w, len[r]);
            nnz2 += len[r];
        }
        sc[q] = (int)cols;
        cols += w;
        cp[q + 1] = cp[q] + (w + kS2Chunk - 1) / kS2Chunk;
        if (32 * cols > (long long)INT_MAX) return CRIMSON_OK;
    }
    sc[ns] = (int)cols;
    // Blocks: one per SM, contiguous slice ranges with equal shares of the
    // work: chunks, and the per-row updates of a slice, which cost about as
    // much as one more chunk.  On small meshes fewer blocks, so that every
    // block has a chunk for each of four warps (fewer packets per barrier).
    const int sms = std::min(sm_count(), kGrMaxBlocks);
    const int grid = (int)std::max(1LL, std::min<long long>({(long long)sms, (long long)ns, (cp[ns] + 3) / 4}));
    std::vector<int2> blk((size_t)grid + 1);   // first slice, first chunk
    int q = 0;
    L->s2_max_rows = 0;
    int max_chunks = 0;
    for (int b = 0; b <= grid; ++b) {
        auto cost = [&](int sl) { return cp[sl] + sl; };
        const long long want = cost(ns) * b / grid;
        while (q < ns && cost(q) < want && (cost(q + 1) <= want || want - cost(q) > cost(q + 1) - want)) ++q;
        if (b == grid) q = ns;
        blk[b] = make_int2(q, (int)cp[q]);
        if (b > 0) {
            L->s2_max_rows = std::max(L->s2_max_rows, 32 * (blk[b].x - blk[b - 1].x));
            max_chunks = std::max(max_chunks, blk[b].y - blk[b - 1].y);
            L->s2_max_cols = std::max(L->s2_max_cols, sc[blk[b].x] - sc[blk[b - 1].x]);
        }
    }
    // Per warp its chunks in order.  A block's warps take its slices in turn,
    // so that at any time they work on neighbouring rows, whose gathers meet
    // in the L1; the slices left over after the last full turn are cut into
    // equal shares of chunks.
    L->s2_max_chunks = max_chunks;
    const int nw = std::min(kS2CgWarps, std::max(4, max_chunks));
    // chunk: first column, then slice << 6 | last << 5 | first << 4 | columns
    std::vector<uint2> desc;
    desc.reserve((size_t)cp[ns]);
    std::vector<int4> wl((size_t)grid * nw);   // begin, chunks, last warp that continues this one's last slice
    auto put = [&](int sl, int k) {
        const int w = sc[sl + 1] - sc[sl], k0 = k * kS2Chunk, kc = std::min(kS2Chunk, w - k0);
        desc.push_back(make_uint2((unsigned)(sc[sl] + k0), (unsigned)sl << 6 | (k0 + kc == w ? 32u : 0u) |
                                                               (k0 == 0 ? 16u : 0u) | (unsigned)kc));
    };
    for (int b = 0; b < grid; ++b) {
        const int s0 = blk[b].x, s1 = blk[b + 1].x;
        const int full = (s1 - s0) / nw * nw;
        const long long c0 = cp[s0 + full], tail = cp[s1] - c0;
        for (int w = 0; w < nw; ++w) {
            const int begin = (int)desc.size();
            for (int sl = s0 + w; sl < s0 + full; sl += nw)
                for (int k = 0; k < cp[sl + 1] - cp[sl]; ++k) put(sl, k);
            const long long t0 = tail * w / nw, t1 = tail * (w + 1) / nw;
            int sl = s0 + full;
            for (long long t = t0; t < t1; ++t) {
                while (cp[sl + 1] - c0 <= t) ++sl;
                put(sl, (int)(t - (cp[sl] - c0)));
            }
            int wlast = w;
            if (t1 > t0)   // sl is the slice of chunk t1 - 1
                while (wlast + 1 < nw && tail * (wlast + 1) / nw < cp[sl + 1] - c0) ++wlast;
            wl[(size_t)b * nw + w] = make_int4(begin, (int)desc.size() - begin, wlast, t1 > t0 ? 1 : 0);
        }
    }
    L->s2_warps = nw;
    CR_CHECK(L->s2_wl.upload(wl.data(), wl.size(), s));
    CR_CHECK(L->s2_sc.upload(sc.data(), sc.size(), s));
    CR_CHECK(L->s2_desc.upload(desc.data(), desc.size(), s));
    CR_CHECK(L->s2_blk.upload(blk.data(), blk.size(), s));
    CR_CHECK(L->s2_mask.alloc((size_t)ns + (size_t)grid));
    CR_CHECK(L->s2_pk.alloc(2 * (size_t)kS2Vals * grid));
    CR_CUDA(cudaMemsetAsync(L->s2_pk.p, 0, sizeof(ulonglong2) * L->s2_pk.n, s));
    CR_CUDA(cudaStreamSynchronize(s));
    L->s2_epoch = 0;
    L->s2_grid = grid;
    L->s2_nnz = nnz2;
    L->s2_npad = 32 * cols;
    L->s2_nslice = ns;
    L->s2_state = 1;
    return CRIMSON_OK;
}
int schur_pattern(crimson_lhs* L) {
    if (L->s2_state != 0) return CRIMSON_OK;
    const int rc = s2_build(L);
    if (rc != CRIMSON_OK) L->s2_state = 0;
    return rc;
}

// The operator's buffer in storage type M with its column offsets, on the
// first solve that uses it.
template <typename M>
static int s2_buffer(crimson_lhs* L, DBuf<unsigned char>& op) {
    const size_t bytes = (size_t)(L->s2_npad / 32) * s2_col_bytes<M>();
    if (op.p && op.n == bytes) return CRIMSON_OK;
    cudaStream_t s = L->stream;
    CR_CHECK(op.alloc(bytes));
    const int rows = 32 * L->s2_nslice;
    launch(k_s2_offsets<M>, grid_for(rows, 8, 16), 256, 0, s, L->rowptr, L->col, L->nNo, rows, (const int*)L->s2_sc.p,
           op.p);
    CR_CUDA(cudaGetLastError());
    return CRIMSON_OK;
}
static DBuf<unsigned char>& s2_op(crimson_lhs* L, const double*) { return L->s2_op64; }
static DBuf<unsigned char>& s2_op(crimson_lhs* L, const float*) { return L->s2_op32; }

// ---------------------------------------------------------------------------
// Values: S = L - Gt G in FP64, rounded to FP32 for M = float.  One warp per
// row; the row's 2-ring columns and FP64 accumulators sit in shared memory.
// Within a warp the lanes add distinct columns, and the contributions are
// added in a fixed order (L, then k in CSR order): deterministic.  16 rows
// (half a slice) per block pass, so the write-back fills whole sectors.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int s2_find(const int* cols, int len, int j) {
    int lo = 0, hi = len;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (cols[mid] < j)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

template <typename M>
__global__ void __launch_bounds__(32 * kS2FormWarps) k_s2_form(const int* __restrict__ rowptr, const int* __restrict__ col,
                                                              const double* __restrict__ mG,
                                                              const double* __restrict__ Gt,
                                                              const double* __restrict__ mL,
                                                              const int* __restrict__ len2, const int* __restrict__ sc,
                                                              int n, int nrows_pad, unsigned char* __restrict__ op,
                                                              double* __restrict__ rowfix) {
    extern __shared__ double s2_smem[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    // odd row stride: the write-back reads one column of 16 rows at a time
    double* a = s2_smem + wid * (kS2Cap + 1);
    int* cw = reinterpret_cast<int*>(s2_smem + kS2FormWarps * (kS2Cap + 1)) + wid * kS2Cap;
    __shared__ int lens[kS2FormWarps];
    for (int r0 = blockIdx.x * kS2FormWarps; r0 < nrows_pad; r0 += gridDim.x * kS2FormWarps) {
        const int r = r0 + wid;
        const int c0 = sc[r0 >> 5], w = sc[(r0 >> 5) + 1] - c0;
        const int len = r < n ? len2[r] : 0;
        for (int e = lane; e < len; e += 32) {
            cw[e] = r + (int)*reinterpret_cast<const short*>(op + s2_off_pos<M>(c0, w, e, r & 31));
            a[e] = 0.0;
        }
        if (lane == 0) lens[wid] = len;
        __syncwarp();
        if (r < n) {
            const int rs = rowptr[r], re = rowptr[r + 1];
            // every column met here is in the row's 2-ring; the guard only
            // keeps a malformed pattern from writing outside the row
            for (int t = rs + lane; t < re; t += 32) {
                const int j = col[t], q = s2_find(cw, len, j);
                if (q < len && cw[q] == j) a[q] += mL[t];
            }
            __syncwarp();
            for (int t = rs; t < re; ++t) {
                const int k = col[t];
                const double g0 = Gt[3 * (size_t)t], g1 = Gt[3 * (size_t)t + 1], g2 = Gt[3 * (size_t)t + 2];
                const int ks = rowptr[k], ke = rowptr[k + 1];
                for (int u = ks + lane; u < ke; u += 32) {
                    const double* gk = mG + 3 * (size_t)u;
                    const int j = col[u], q = s2_find(cw, len, j);
                    if (q < len && cw[q] == j) a[q] -= g0 * gk[0] + g1 * gk[1] + g2 * gk[2];
                }
                __syncwarp();
            }
            if (sizeof(M) == 4) {
                double d = 0.0;
                for (int e = lane; e < len; e += 32) d += a[e] - (double)(M)a[e];
                d = warp_sum(d);
                if (lane == 0) rowfix[r] = d;
            }
        }
        __syncthreads();
        for (int p = threadIdx.x; p < kS2FormWarps * w; p += blockDim.x) {
            const int row = p % kS2FormWarps, e = p / kS2FormWarps;
            *reinterpret_cast<M*>(op + s2_val_pos<M>(c0, w, e, (r0 + row) & 31)) =
                e < lens[row] ? (M)s2_smem[row * (kS2Cap + 1) + e] : M(0);
        }
        __syncthreads();
    }
}

template <typename M>
int schur_form(crimson_lhs* L, const double* mG, const double* Gt, const double* mL) {
    if (L->s2_state != 1) return CRIMSON_ERR_STATE;
    cudaStream_t s = L->stream;
    DBuf<unsigned char>& op = s2_op(L, (const M*)nullptr);
    CR_CHECK(s2_buffer<M>(L, op));
    if (sizeof(M) == 4) CR_CHECK(L->s2_rowfix.alloc((size_t)L->nNo));
    const size_t smem = kS2FormWarps * ((kS2Cap + 1) * sizeof(double) + kS2Cap * sizeof(int));
    CR_CUDA(cudaFuncSetAttribute(k_s2_form<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    CR_CUDA(cudaEventRecord(L->s2_ev0, s));
    const int rows = 32 * L->s2_nslice;
    launch(k_s2_form<M>, grid_for(rows, kS2FormWarps, 4), 32 * kS2FormWarps, smem, s, L->rowptr, L->col, mG, Gt, mL,
           (const int*)L->s2_len.p, (const int*)L->s2_sc.p, L->nNo, rows, op.p, L->s2_rowfix.p);
    CR_CUDA(cudaEventRecord(L->s2_ev1, s));
    CR_CUDA(cudaGetLastError());
    L->s2_form_pending = true;
    return CRIMSON_OK;
}
template int schur_form<double>(crimson_lhs*, const double*, const double*, const double*);
template int schur_form<float>(crimson_lhs*, const double*, const double*, const double*);

// Bit f of mask[slice]: w_f or z_f is not zero on some row of the slice.
__global__ void k_s2_mask(const double* __restrict__ w, const double* __restrict__ z, int nface, int n, int nslice,
                          unsigned* __restrict__ mask) {
    const int lane = threadIdx.x & 31;
    for (int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < nslice; s += (gridDim.x * blockDim.x) >> 5) {
        const int r = 32 * s + lane;
        unsigned m = 0;
        for (int f = 0; f < nface; ++f) {
            const bool nz = r < n && (w[(size_t)f * n + r] != 0.0 || z[(size_t)f * n + r] != 0.0);
            if (__any_sync(0xffffffffu, nz)) m |= 1u << f;
        }
        if (lane == 0) mask[s] = m;
    }
}

// The blocks' face bits: OR over their slices.
__global__ void k_s2_blkmask(const int2* __restrict__ blk, const unsigned* __restrict__ mask, int nblk,
                             unsigned* __restrict__ bmask) {
    for (int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < nblk; b += (gridDim.x * blockDim.x) >> 5) {
        unsigned m = 0;
        for (int s = blk[b].x + (threadIdx.x & 31); s < blk[b + 1].x; s += 32) m |= mask[s];
        m = __reduce_or_sync(0xffffffffu, m);
        if ((threadIdx.x & 31) == 0) bmask[b] = m;
    }
}

int schur_faces(crimson_lhs* L, int nface) {
    launch(k_s2_mask, grid_for(32LL * L->s2_nslice, 256), 256, 0, L->stream, (const double*)L->cgW.p,
           (const double*)L->cgZ.p, nface, L->nNo, L->s2_nslice, L->s2_mask.p);
    launch(k_s2_blkmask, grid_for(32LL * L->s2_grid, 256), 256, 0, L->stream, (const int2*)L->s2_blk.p,
           (const unsigned*)L->s2_mask.p, L->s2_grid, L->s2_mask.p + L->s2_nslice);
    CR_CUDA(cudaGetLastError());
    return CRIMSON_OK;
}

// ---------------------------------------------------------------------------
// CGRAD: one persistent cooperative launch per call.
// ---------------------------------------------------------------------------
struct CgS2Args {
    const unsigned char* op;
    const uint2* desc;
    const int4* wl;
    const int2* blk;
    const unsigned* mask;   // face bits of the slices, then of the blocks
    int nslice;
    const int* sc;           // first column of every slice
    int n, stages, nvec;     // nvec: vectors over the block's rows in shared memory
    int max_rows, max_cols;  // of a block
    int evict_first;         // the operator exceeds the L2: its lines go first
    const double* rowfix;    // (n) FP32 operator: what rounding took from the row sums
    double* rhs;             // in: right side; out: solution
    double* R;               // (2 n) the gathered residual, two alternating buffers
    double* Pg;              // (n) P, SP, X when they do not fit in shared memory
    double* SPg;
    double* Xg;
    int nface;
    const double* w;  // (nface, n)
    const double* z;  // (nface, n)
    double coef[kS2MaxFaces];
    double relTol, absTol;
    int mItr;
    ulonglong2* pk;   // 2 regions of kS2Vals packets per block
    unsigned long long epoch;
    double* out;      // err, errO, i, suc (-1: a wait ran out), initial norm
};

__device__ __forceinline__ unsigned s2_smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool s2_try_wait(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait for a stage's copy; without patience (a copy has timed out
// before) one try.
__device__ __forceinline__ bool s2_wait(unsigned bar, unsigned parity, bool patience) {
    if (s2_try_wait(bar, parity)) return true;
    if (!patience) return false;
    const long long t0 = clock64();
    while (clock64() - t0 < kGrWaitClocks)
        if (s2_try_wait(bar, parity)) return true;
    return false;
}

// One lane's share of a full chunk in shared memory.
template <typename M>
struct S2Lane;
template <>
struct S2Lane<double> {
    double x[kS2Chunk];
    __device__ __forceinline__ void load(const unsigned char* p) {
#pragma unroll
        for (int j = 0; j < kS2Chunk / 2; ++j) {
            const double2 q = *reinterpret_cast<const double2*>(p + 512 * j);
            x[2 * j] = q.x;
            x[2 * j + 1] = q.y;
        }
    }
};
template <>
struct S2Lane<float> {
    float x[kS2Chunk];
    __device__ __forceinline__ void load(const unsigned char* p) {
#pragma unroll
        for (int j = 0; j < kS2Chunk / 4; ++j) {
            const float4 q = *reinterpret_cast<const float4*>(p + 512 * j);
            x[4 * j] = q.x;
            x[4 * j + 1] = q.y;
            x[4 * j + 2] = q.z;
            x[4 * j + 3] = q.w;
        }
    }
};

// kRes: the block's chunks stay in shared memory (loaded once), else they
// stream through the warps' rings.
template <typename M, bool kRes>
__global__ void __launch_bounds__(32 * kS2CgWarps, 1) k_cg_schur(const __grid_constant__ CgS2Args a) {
    extern __shared__ __align__(128) unsigned char s2_dyn[];
    __shared__ double red[32 * kS2Vals], tot[kS2Vals];
    __shared__ unsigned char fpend[32 * kS2MaxFaces];
    // kept out of the registers of the inner loop: the places of P, SP, X and
    // of the staged w, z; |R|^2 now and before, eps, |R_0|, beta
    __shared__ double* vp[5];
    __shared__ double scal[5];
    constexpr int COL = s2_col_bytes<M>();
    constexpr int CB = kS2Chunk * COL;   // bytes of a stage
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int n = a.n, S = a.stages;
    const int2 b0 = a.blk[blockIdx.x], b1 = a.blk[blockIdx.x + 1];
    const int row0 = 32 * b0.x, nsl = b1.x - b0.x;
    const int4 wl = a.wl[blockIdx.x * nw + wid];   // this warp's chunks
    const int nck = wl.y;

    // shared memory: the chunks (all of the block's, or the warps' rings with
    // their mbarriers), partial rows of slices begun by an earlier warp, the
    // vectors, the face bits of the block's slices, descriptors
    const int c0 = a.sc[b0.x];
    const unsigned ring = kRes ? 0u : (unsigned)(wid * S * CB);
    const unsigned o_bars = kRes ? (unsigned)a.max_cols * COL : (unsigned)(nw * S * CB);
    const unsigned o_carry = o_bars + (kRes ? 0u : 8u * nw * S);
    const unsigned o_vec = o_carry + 256u * nw;
    const unsigned o_mask = o_vec + 8u * a.nvec * a.max_rows;
    const unsigned o_desc = o_mask + (unsigned)(a.max_rows / 8) + (a.max_rows / 8 & 4);
    unsigned long long* const bars = reinterpret_cast<unsigned long long*>(s2_dyn + o_bars) + wid * S;
    double* const carry = reinterpret_cast<double*>(s2_dyn + o_carry);
    unsigned* const mask = reinterpret_cast<unsigned*>(s2_dyn + o_mask);
    // ring: word 1 of the staged chunks' descriptors; kRes: the warp's descriptors
    unsigned* const sdesc =
        reinterpret_cast<unsigned*>(s2_dyn + o_desc) + (kRes ? 2 * (wl.x - a.wl[blockIdx.x * nw].x) : wid * S);
    const bool wz_local = kRes && a.nvec > 3;   // w_f, z_f of the block's rows in shared memory
    const size_t ldw = wz_local ? (size_t)a.max_rows : (size_t)n;
    if (threadIdx.x == 0) {
        double* vec = reinterpret_cast<double*>(s2_dyn + o_vec);
        vp[0] = a.nvec > 0 ? vec : a.Pg + row0;
        vp[1] = a.nvec > 0 ? vec + a.max_rows : a.SPg + row0;
        vp[2] = kRes ? vec + 2 * (size_t)a.max_rows : a.Xg + row0;
        vp[3] = wz_local ? vec + 3 * (size_t)a.max_rows : const_cast<double*>(a.w) + row0;
        vp[4] = wz_local ? vec + (3 + a.nface) * (size_t)a.max_rows : const_cast<double*>(a.z) + row0;
    }
    __syncthreads();

    int qi = wl.x;           // ring: list entry lane 0 issues next, and its descriptor
    uint2 dq = make_uint2(0u, 0u);
    auto issue = [&](int st) {   // lane 0
        unsigned long long policy;
        if (a.evict_first)
            asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
        else
            asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(policy));
        const unsigned bar = s2_smem_u32(bars + st), bytes = (dq.y & 15u) * COL;
        sdesc[st] = dq.y;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::
                "r"(s2_smem_u32(s2_dyn + ring + st * CB)), "l"(a.op + (size_t)dq.x * COL), "r"(bytes), "r"(bar), "l"(policy)
            : "memory");
        if (++qi == wl.x + nck) qi = wl.x;
        dq = a.desc[qi];
    };
    const int nload = kRes ? 0 : min(S, nck);
    if (kRes) {
        const size_t beg = (size_t)c0 * COL, bytes = (size_t)(a.sc[b1.x] - c0) * COL;
        for (size_t p = 16 * (size_t)threadIdx.x; p < bytes; p += 16 * (size_t)blockDim.x)
            *reinterpret_cast<uint4*>(s2_dyn + p) = *reinterpret_cast<const uint4*>(a.op + beg + p);
        for (int q = lane; q < nck; q += 32) reinterpret_cast<uint2*>(sdesc)[q] = a.desc[wl.x + q];
    } else if (lane == 0 && nck > 0) {
        for (int q = 0; q < S; ++q)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(s2_smem_u32(bars + q)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        dq = a.desc[qi];
        for (int st = 0; st < nload; ++st) issue(st);
    }
    unsigned cont = 0;   // warps whose partial rows complete this warp's last slice
    for (int w = wid + 1; w <= wl.z; ++w)
        if (a.wl[blockIdx.x * nw + w].w) cont |= 1u << w;
    const unsigned* bmask = a.mask + a.nslice;
    const unsigned own_faces = a.nface > 0 ? bmask[blockIdx.x] : 0u;
    for (int t = threadIdx.x; t < nsl; t += blockDim.x) mask[t] = a.nface > 0 ? a.mask[b0.x + t] : 0u;
    for (int f = wid; f < a.nface; f += nw) {
        unsigned m = gr_all_blocks();
#pragma unroll
        for (int j = 0; j < kGrPolls; ++j)
            if (((m >> j) & 1) && !((bmask[lane + 32 * j] >> f) & 1)) m &= ~(1u << j);
        fpend[32 * f + lane] = (unsigned char)m;
    }

    // ---- initial residual: |rhs|^2 over the block's rows; P = SP = X = 0 ----
    unsigned long long ep = a.epoch;
    double part = 0.0;
    for (int t = threadIdx.x; t < 32 * nsl; t += blockDim.x)
        if (row0 + t < n) {
            const double v = a.rhs[row0 + t];
            vp[0][t] = 0.0;
            vp[1][t] = 0.0;
            vp[2][t] = 0.0;
            a.R[row0 + t] = v;
            if (wz_local)
                for (int f = 0; f < a.nface; ++f) {
                    vp[3][f * ldw + t] = a.w[(size_t)f * n + row0 + t];
                    vp[4][f * ldw + t] = a.z[(size_t)f * n + row0 + t];
                }
            part += v * v;
        }
    part = warp_sum(part);
    if (lane == 0) red[wid] = part;
    bool fail = grid_reduce(a.pk, kS2Vals, red, 0, 0u, fpend, ++ep, true, tot, false);
    if (threadIdx.x == 0) {
        const double e = sqrt(tot[0]), eps = fmax(a.absTol, a.relTol * e);
        scal[0] = e * e;
        scal[1] = e;
        scal[2] = eps * eps;
        scal[3] = e;
        scal[4] = 0.0;
    }
    __syncthreads();

    int suc = 0, i;
    int gs = 0;              // ring: stage of the next chunk, its mbarrier phase
    unsigned parity = 0;
    bool ok = true;          // no copy of this warp timed out
    for (i = 1; i <= a.mItr && !fail; ++i) {
        if (scal[0] < scal[2]) {
            suc = 1;
            break;
        }
        // R alternates between two buffers: phase 2 writes the one that no
        // block has gathered from since the last barrier that ordered data
        const double* Rc = a.R + (size_t)((i - 1) & 1) * n;
        // ---- phase 1 ----
        double dps = 0.0;
        double acc0 = 0.0, acc1 = 0.0;
        bool owner = false, open = false;   // owner: this warp began the slice; open: it is not complete
        int slice = 0;
        // completes a slice: SP = S R + beta SP, P = R + beta P, <P, SP>
        auto finish = [&](double acc) {
            const int t = 32 * (slice - b0.x) + lane;
            if (row0 + t < n) {
                const double beta = scal[4], r = Rc[row0 + t];
                if (sizeof(M) == 4) acc = acc + a.rowfix[row0 + t] * r;
                const double sv = acc + beta * vp[1][t];
                const double pr = r + beta * vp[0][t];
                vp[1][t] = sv;
                vp[0][t] = pr;
                dps += pr * sv;
            }
        };
#pragma unroll 1
        for (int q = 0; q < nck; ++q) {
            unsigned d, p;
            if (kRes) {
                const uint2 e = reinterpret_cast<const uint2*>(sdesc)[q];
                d = e.y;
                p = (e.x - (unsigned)c0) * COL;
            } else {
                if (!s2_wait(s2_smem_u32(bars + gs), parity, ok)) ok = false;
                d = sdesc[gs];
                p = ring + gs * CB;
            }
            const int kc = (int)(d & 15u);
            slice = (int)(d >> 6);
            const double* Rr = Rc + min(32 * slice + lane, n - 1);
            if (d & 16u) owner = true;
            open = true;
            if (kc == kS2Chunk) {
                const uint4 o = *reinterpret_cast<const uint4*>(s2_dyn + p + kS2Chunk * 32 * sizeof(M) + 16 * lane);
                const unsigned w[4] = {o.x, o.y, o.z, o.w};
                double g[kS2Chunk];
#pragma unroll
                for (int u = 0; u < kS2Chunk; ++u) g[u] = Rr[u % 2 ? (int)w[u / 2] >> 16 : (int)(short)(w[u / 2] & 0xffffu)];
                S2Lane<M> c;
                c.load(s2_dyn + p + 16 * lane);
                if (!kRes) {
                    // the values are in registers: the stage takes the chunk one ring ahead
                    __syncwarp();
                    if (lane == 0) issue(gs);
                }
#pragma unroll
                for (int u = 0; u < kS2Chunk; u += 2) {
                    acc0 = acc0 + (double)c.x[u] * g[u];
                    acc1 = acc1 + (double)c.x[u + 1] * g[u + 1];
                }
            } else {
                const short* o = reinterpret_cast<const short*>(s2_dyn + p + kc * 32 * (int)sizeof(M)) + lane;
                const M* v = reinterpret_cast<const M*>(s2_dyn + p) + lane;
#pragma unroll 1
                for (int u = 0; u < kc; ++u) acc0 = acc0 + (double)v[32 * u] * Rr[(int)o[32 * u]];
                if (!kRes) {
                    __syncwarp();
                    if (lane == 0) issue(gs);
                }
            }
            if (!kRes && ++gs == nload) {
                gs = 0;
                parity ^= 1u;
            }
            if (d & 32u) {
                const double acc = acc0 + acc1;
                acc0 = acc1 = 0.0;
                if (owner)
                    finish(acc);
                else
                    carry[32 * wid + lane] = acc;
                owner = open = false;
            }
        }
        const double acc = acc0 + acc1;
        if (open && !owner) carry[32 * wid + lane] = acc;
        __syncthreads();
        if (open && owner) {
            double t = acc;
            for (unsigned m = cont; m; m &= m - 1) t = t + carry[32 * (__ffs(m) - 1) + lane];
            finish(t);
        }
        // coupled faces: w_f . P and z_f . P over the slices that touch them
        if (own_faces) {
            __syncthreads();
            for (unsigned m = own_faces; m; m &= m - 1) {
                const int f = __ffs(m) - 1;
                double wv = 0.0, zv = 0.0;
                for (int sl = wid; sl < nsl; sl += nw)
                    if ((mask[sl] >> f) & 1) {
                        const int t = 32 * sl + lane;
                        if (row0 + t < n) {
                            const double pr = vp[0][t];
                            wv += vp[3][f * ldw + t] * pr;
                            zv += vp[4][f * ldw + t] * pr;
                        }
                    }
                wv = warp_sum(wv);
                zv = warp_sum(zv);
                if (lane == 0) {
                    red[32 * (1 + 2 * f) + wid] = wv;
                    red[32 * (2 + 2 * f) + wid] = zv;
                }
            }
        }
        dps = warp_sum(dps);
        if (lane == 0) red[wid] = dps;
        fail = grid_reduce(a.pk, kS2Vals, red, a.nface, own_faces, fpend, ++ep, false, tot, !ok || fail);
        double den = tot[0];
        for (int f = 0; f < a.nface; ++f) den = den - a.coef[f] * tot[1 + 2 * f] * tot[2 + 2 * f];
        const double alpha = scal[0] / den;
        // ---- phase 2 ----
        double* Rw = a.R + (size_t)(i & 1) * n;
        double rs = 0.0;
        for (int sl = wid; sl < nsl; sl += nw) {
            const int t = 32 * sl + lane, r = row0 + t;
            if (r >= n) continue;
            double sv = vp[1][t];
            for (unsigned m = mask[sl]; m; m &= m - 1) {
                const int f = __ffs(m) - 1;
                sv = sv - a.coef[f] * tot[1 + 2 * f] * vp[4][f * ldw + t];
            }
            vp[2][t] = vp[2][t] + alpha * vp[0][t];
            const double rv = Rc[r] - alpha * sv;
            Rw[r] = rv;
            rs += rv * rv;
        }
        rs = warp_sum(rs);
        if (lane == 0) red[wid] = rs;
        fail = grid_reduce(a.pk, kS2Vals, red, 0, 0u, fpend, ++ep, true, tot, fail);
        if (threadIdx.x == 0) {
            const double e2 = sqrt(tot[0]), err = e2 * e2;
            scal[4] = err / scal[0];
            scal[1] = scal[0];
            scal[0] = err;
        }
        __syncthreads();
    }
    // the copies still under way, one per stage (also after a wait that ran out)
    for (int q = 0; q < nload; ++q) {
        s2_wait(s2_smem_u32(bars + gs), parity, true);
        if (++gs == nload) {
            gs = 0;
            parity ^= 1u;
        }
    }
    for (int t = threadIdx.x; t < 32 * nsl; t += blockDim.x)
        if (row0 + t < n) a.rhs[row0 + t] = vp[2][t];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.out[0] = scal[0];
        a.out[1] = scal[1];
        a.out[2] = (double)i;
        a.out[3] = fail ? -1.0 : (double)suc;
        a.out[4] = scal[3];
    }
}

// One CGRAD call: R (n) holds the right side and receives the solution; out
// (5 doubles, device) receives err, errO, the iteration index, the success
// flag and the initial norm.
template <typename M>
int cg_schur_launch(crimson_lhs* L, double* R, int nface, const double* coef, double relTol, double absTol, int mItr,
                    double* out) {
    if (L->s2_state != 1 || nface > kS2MaxFaces) return CRIMSON_ERR_STATE;
    cudaStream_t s = L->stream;
    const size_t n = (size_t)L->nNo;
    constexpr size_t kStatic = 8 * 1024;   // static shared memory (red, tot) and the driver's reserve
    const size_t budget = 227 * 1024 - kStatic;
    const int nw = L->s2_warps;
    const size_t cb = (size_t)kS2Chunk * s2_col_bytes<M>();
    const size_t vec1 = sizeof(double) * (size_t)L->s2_max_rows;
    const size_t fixed = sizeof(double) * 32 * (size_t)nw + sizeof(unsigned) * (size_t)(L->s2_max_rows / 32) + 16;
    const size_t own = (size_t)L->s2_max_cols * s2_col_bytes<M>() + sizeof(uint2) * (size_t)L->s2_max_chunks;
    // everything in shared memory, or a ring per warp
    const bool res = fixed + 3 * vec1 + own <= budget;
    // two stages per warp: more of them take the L1 from the gathers (4M-tet
    // cylinder, two / three stages: 80.7 / 85 us per FP64 iteration)
    constexpr int stages = 2;
    const size_t ring = (cb + sizeof(unsigned long long) + sizeof(unsigned)) * nw * stages;
    // vectors in shared memory.  Resident: P, SP, X and the faces' w and z.
    // Streaming: P and SP where that leaves at least 64 KB of L1 (4M-tet
    // cylinder, with / without: 56.6 / 58.1 us FP32, 82.3 / 80.7 us FP64,
    // where it would not).
    int nvec = res ? 3 + 2 * nface : 2;
    if (res && fixed + nvec * vec1 + own > budget) nvec = 3;
    if (!res && fixed + ring + 2 * vec1 > (size_t)160 * 1024) nvec = 0;
    const size_t smem = fixed + nvec * vec1 + (res ? own : ring);
    (sizeof(M) == 4 ? L->cg_form32 : L->cg_form64) = res ? CRIMSON_CG_SCHUR_RESIDENT : CRIMSON_CG_SCHUR;
    const void* kfn = res ? (const void*)k_cg_schur<M, true> : (const void*)k_cg_schur<M, false>;
    // the same value for every lhs: host threads that launch side by side set it alike
    CR_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)budget));
    CR_CHECK(L->s2_R.alloc(2 * n));
    if (nvec < 2) {
        CR_CHECK(L->cgPd.alloc(n));
        CR_CHECK(L->cgSP.alloc(n));
    }
    if (nvec < 3) CR_CHECK(L->cgX.alloc(n));
    CgS2Args a;
    a.op = s2_op(L, (const M*)nullptr).p;
    a.desc = L->s2_desc.p;
    a.wl = L->s2_wl.p;
    a.blk = L->s2_blk.p;
    a.mask = L->s2_mask.p;
    a.nslice = L->s2_nslice;
    a.n = L->nNo;
    a.sc = L->s2_sc.p;
    a.stages = stages;
    a.max_cols = L->s2_max_cols;
    a.nvec = nvec;
    a.max_rows = L->s2_max_rows;
    a.evict_first = s2_op(L, (const M*)nullptr).n > (size_t)80 << 20;
    a.rowfix = L->s2_rowfix.p;
    a.rhs = R;
    a.R = L->s2_R.p;
    a.Pg = L->cgPd.p;
    a.SPg = L->cgSP.p;
    a.Xg = L->cgX.p;
    a.nface = nface;
    a.w = L->cgW.p;
    a.z = L->cgZ.p;
    for (int f = 0; f < kS2MaxFaces; ++f) a.coef[f] = f < nface ? coef[f] : 0.0;
    a.relTol = relTol;
    a.absTol = absTol;
    a.mItr = mItr;
    a.pk = L->s2_pk.p;
    a.epoch = L->s2_epoch;
    a.out = out;
    L->s2_epoch += 2ull * (unsigned long long)std::max(mItr, 0) + 2;
    void* kargs[] = {&a};
    note_launch();
    CR_CUDA(cudaLaunchCooperativeKernel(kfn, dim3(L->s2_grid), dim3(32 * nw), kargs, smem, s));
    return CRIMSON_OK;
}
template int cg_schur_launch<double>(crimson_lhs*, double*, int, const double*, double, double, int, double*);
template int cg_schur_launch<float>(crimson_lhs*, double*, int, const double*, double, double, int, double*);

}  // namespace crimson
