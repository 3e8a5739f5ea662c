// The batched rank's rounds of 64 columns: the batch rule, for jobs of at most
// 1024 rows (jobs.cu has the schedules of 32-column rounds).
//
// Per round and job one CTA settles the job's next 64 columns:
//   - rr_block_kernel: the top-block inversion of the single-matrix elimination
//     (hme_panel.cuh) on the job's top rows.  A dense job's pivots are
//     practically always there, and no other row is touched in the panel.  The
//     trailing update is A22 -= A21 (B^-1 A12): rr_apply_kernel forms
//     B^-1 A12 in place, and A21 are the panel's columns as they stand, so the
//     update's left factor is read where it lies;
//   - rr_general_kernel, for the jobs that the block does not settle, and for
//     sparse ones (a job that failed the block stays here until its rows fill
//     up): the pivot search over the rows with a non-zero entry in the panel,
//     the row operations' effect on the identity kept in place, so the update's
//     left factor W comes out directly: the rows' A22 += W A12.  Up to 256 such
//     rows move to the top, behind the pivots, and the update covers no zero
//     rows; with more, rr_general_kernel<1024> takes 32 columns and a W of all
//     rows.
// Then the row moves, and one grouped split and limb GEMM (K <= 64) per modulus.
// Pivot rows' trailing blocks are final only for the update's sake: a rank needs
// no U, so the general kernel's pivot rows stay as they are.
//
// Against the schedules' rounds of 32 columns (a search over all rows in every
// panel, L11^-1, its product and an L21 gather): half the passes over the
// trailing blocks.  The rank phase of the 2000-job stream (half of it sparse,
// p = 65521 and 2^31 - 19, sides to 1024): 30 ms in rounds of 32 columns, 8.5 ms
// so (block kernel 1.2, listed rows 2.0, moves 0.6, products 0.9, splits and
// GEMMs 2.9 ms).  What bounds a round is the block's and the search's chain of
// 64 steps early on (several CTAs per SM hide it), and the GEMMs' passes over
// the trailing blocks.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <type_traits>
#include <vector>

#include "hme_elim.h"
#include "hme_grouped.h"
#include "hme_internal.h"
#include "hme_panel.cuh"
#include "hme_ptx.cuh"

namespace hme {
namespace {

// A modulus group: its jobs are [begin, end) of the job arrays; one grouped
// split + GEMM launch per round reads its tables.
struct RrGroup {
    uint32_t p, mont_qinv, mont_r2;
    uint64_t barrett;
    const CUtensorMap* tmA;  // stacked A planes of the group: {64, sum_m, L}
    const CUtensorMap* tmB;  // stacked B planes: {64, sum_n, L, L}
    uint8_t* planesA;
    uint8_t* planesB;
    uint64_t sum_m, sum_n;
    limb::EpiRed split_red;
    int bn;                  // grouped GEMM tile width
    int begin, end;
    int* tile_prob;          // per tile: the job (index within the group)
    int* block_job;          // per split block: the job (index within the group)
    int* totals;             // [0] tiles, [1] split blocks of the round
};

// How the panel code multiplies mod p.
__host__ __device__ constexpr int rr_arith(uint32_t p) {
    return p == 2 ? panel::kArithPow2 : p < (1u << 31) ? panel::kArithMont31 : panel::kArithMont32;
}

// The field F_p of a group as the panel code sees it.
__device__ __forceinline__ panel::Ring rr_ring(const RrGroup& G) {
    panel::Ring R;
    R.q = G.p;
    R.barrett = G.barrett;
    R.ell = G.p;
    R.k = 1;
    R.max_v = 0;
    R.mont_qinv = G.mont_qinv;
    R.mont_r2 = G.mont_r2;
    return R;
}

constexpr int kRrW = 64;
constexpr int kRrCompact = 256;
// Threads of the listed rows' kernel: a job of the stream has about 100 such rows, and a step is a barrier
// and a few updates per thread, so several CTAs per SM beat wide ones.  All rounds of the 2000-job stream:
// 256 threads 3.0 ms, 512 threads 2.0 to 2.2 ms, 1024 threads 2.35 ms (two or three CTAs of 512 per SM: the same).
constexpr int kRrThreads = 512;

struct RrJob {
    uint32_t* A;   // m x n, ld (device), destroyed
    uint64_t ld;
    int m, n, group;
    int r0, c0, active;
    int dense;            // the next round tries the top block
    int w, k, cnt, kind;  // the round: columns, pivots, listed rows, 1 top block / 2 listed rows moved / 3 all rows
    int a_row0, b_col0;   // the job's rows / columns in its group's stacked plane tensors
    uint32_t* F;          // B^-1 (64 x 64), or W: (cnt - k) x 64 of the listed rows, (m - r0 - k) x 32 of all
    int* rows;            // rows that move to r0, r0 + 1, ..
};

struct RrMove {
    uint32_t* A;
    uint64_t ld;
    int r0, count, ca, cb;  // rows[0 .. count) to r0 .., columns [ca, cb)
    const int* rows;
};
struct RrApply {
    uint32_t* A;  // the pivot rows' trailing block, 64 x cols
    uint64_t ld;
    int cols;     // 0: nothing
    const uint32_t* M;
    uint32_t p;
    uint64_t barrett;
};

// the round's job lists, and the jobs that go on
enum { kRrBlock = 0, kRrGeneral = 1, kRrTall = 2, kRrMove = 3, kRrSolve = 4, kRrLists = 5, kRrActive = 5, kRrCounters = 6 };

__global__ void rr_plan_kernel(RrJob* __restrict__ jobs, int nj, int* __restrict__ lists, int* __restrict__ counters) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < nj; j += gridDim.x * blockDim.x) {
        RrJob& J = jobs[j];
        J.k = 0;
        J.kind = 0;
        if (!J.active) continue;
        J.w = min(kRrW, J.n - J.c0);
        const int b = J.dense ? kRrBlock : kRrGeneral;
        lists[static_cast<size_t>(b) * nj + atomicAdd(&counters[b], 1)] = j;
    }
}

// The kernels with a panel take the jobs of one arithmetic and leave the others to their own launches.
template <int ARITH, int RS>
__global__ void __launch_bounds__(4 * RS) rr_block_kernel(RrJob* __restrict__ jobs, int nj, int* __restrict__ lists,
                                                          int* __restrict__ counters, const RrGroup* __restrict__ groups) {
    extern __shared__ __align__(16) uint32_t s_rr[];
    __shared__ int s_cols[panel::kMaxPanel], s_k, s_ok;
    const int njobs = counters[kRrBlock];
    for (int i = blockIdx.x; i < njobs; i += gridDim.x) {
        const int j = lists[i];
        RrJob& J = jobs[j];
        if (rr_arith(groups[J.group].p) != ARITH) continue;
        __syncthreads();  // the job before is done with the shared state
        panel::BlockArgs a;
        a.A = J.A;
        a.ld = J.ld;
        a.m = J.m;
        a.r0 = J.r0;
        a.c0 = J.c0;
        a.w = J.w;
        a.R = rr_ring(groups[J.group]);
        a.pivot_rows = J.rows;
        a.pivot_cols = s_cols;
        a.k_out = &s_k;
        a.ok = &s_ok;
        a.binv = J.F;
        a.diag = nullptr;
        const bool ok = panel::block_inverse<ARITH, RS>(a, s_rr);
        if (threadIdx.x == 0) {
            if (ok) {
                J.kind = 1;
                J.k = J.cnt = min(J.w, J.m - J.r0);
            } else {
                J.dense = 0;
                lists[static_cast<size_t>(kRrGeneral) * nj + atomicAdd(&counters[kRrGeneral], 1)] = j;
            }
        }
    }
}

// One CTA per job; MAXR = 256: 64 columns of up to 256 listed rows
// (more: the job goes to the tall list); MAXR = 1024: 32 columns of any rows.
template <int ARITH, int MAXR, int NT>
__global__ void __launch_bounds__(NT, NT == 1024 ? 1 : 2) rr_general_kernel(RrJob* __restrict__ jobs, int nj, int* __restrict__ lists,
                                                          int* __restrict__ counters, const RrGroup* __restrict__ groups) {
    using namespace panel;
    constexpr bool TALL = MAXR > kRrCompact;
    constexpr int NRW = MAXR / 32, NW = NT / 32;
    static_assert(NW >= NRW, "a warp for every 32 listed rows");
    constexpr int W = TALL ? 32 : kRrW;
    extern __shared__ __align__(16) uint32_t S[];  // [w][rs]
    __shared__ uint32_t s_x[2][MAXR];
    __shared__ int s_key[2][NRW], s_nz[2][NRW];
    __shared__ uint32_t s_inv;
    __shared__ int s_prow[W], s_colpiv[W], s_vac[W];
    __shared__ unsigned char s_isp[W];
    __shared__ int s_row[MAXR], s_step[MAXR], s_pos[MAXR];
    __shared__ unsigned s_mask[32];
    __shared__ int s_base[33];
    constexpr int kList = TALL ? kRrTall : kRrGeneral;
    constexpr int NONE = INT_MAX;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int njobs = counters[kList];
    for (int ji = blockIdx.x; ji < njobs; ji += gridDim.x) {
        const int jj = lists[static_cast<size_t>(kList) * nj + ji];
        RrJob& J = jobs[jj];
        if (rr_arith(groups[J.group].p) != ARITH) continue;
        __syncthreads();  // the job before is done with the shared state
        const int rows = J.m - J.r0, w = TALL ? min(W, J.w) : J.w;
        const uint32_t* P0 = J.A + static_cast<size_t>(J.r0) * J.ld + J.c0;
        const Ring R = rr_ring(groups[J.group]);
        // rows with a non-zero entry, in row order (rows <= 1024)
        for (int b = warp; b < 32; b += NW) {
            unsigned mine = 0;  // bit u: whether row 32 b + u has one
            for (int u = 0; u < 32 && 32 * b + u < rows; u += 4) {
                uint32_t x[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int r = 32 * b + u + e;
                    x[e] = 0;
                    if (r < rows)
                        for (int c = lane; c < w; c += 32) x[e] |= P0[static_cast<size_t>(r) * J.ld + c];
                }
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (__any_sync(0xffffffffu, x[e] != 0)) mine |= 1u << (u + e);
            }
            if (lane == 0) s_mask[b] = mine;
        }
        __syncthreads();
        if (warp == 0) {
            const int c = __popc(s_mask[lane]);
            int incl = c;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, off);
                if (lane >= off) incl += y;
            }
            s_base[lane] = incl - c;
            if (lane == 31) s_base[32] = incl;
        }
        __syncthreads();
        const int cnt = s_base[32];
        if (cnt > MAXR) {  // (MAXR = 256 only; the same in every thread)
            if (tid == 0) lists[static_cast<size_t>(kRrTall) * nj + atomicAdd(&counters[kRrTall], 1)] = jj;
            continue;
        }
        for (int b = warp; b < 32; b += NW)
            if ((s_mask[b] >> lane) & 1u) {
                const int at = s_base[b] + __popc(s_mask[b] & ((1u << lane) - 1u));
                s_row[at] = 32 * b + lane;
                s_step[at] = 0;
            }
        if (tid < W) s_colpiv[tid] = -1;
        __syncthreads();
        int rwn = 1;
        while (32 * rwn < cnt) rwn *= 2;
        const int G = NW / rwn, rs = 32 * rwn + 1;
#pragma unroll 4
        for (int r = warp; r < cnt; r += NW)
            for (int c = lane; c < w; c += 32) S[c * rs + r] = P0[static_cast<size_t>(s_row[r]) * J.ld + c];
        __syncthreads();
        const int rwi = warp & (rwn - 1), g = warp / rwn, li = 32 * rwi + lane;
        bool active = li < cnt;
        uint32_t* col = S + li;
        auto publish = [&](int c) {
            const uint32_t x = active ? col[c * rs] : 0u;
            const int key = __reduce_min_sync(0xffffffffu, x != 0 ? li : NONE);
            const unsigned nz = __ballot_sync(0xffffffffu, x != 0);
            s_x[c & 1][li] = x;
            if (lane == 0) {
                s_key[c & 1][rwi] = key;
                s_nz[c & 1][rwi] = __popc(nz);
            }
        };
        if (g == 0) publish(0);
        uint32_t scale = 1u;
        int k = 0;
        __syncthreads();
        for (int it = 0; it < w; ++it) {
            const int par = it & 1;
            int pk = NONE, nz = 0;
            for (int u = 0; u < rwn; ++u) {
                pk = min(pk, s_key[par][u]);
                nz += s_nz[par][u];
            }
            if (pk != NONE) {
                const uint32_t wt = s_x[par][pk];
                if (tid == 0) {
                    s_prow[k] = pk;
                    s_colpiv[it] = k;
                    s_step[pk] = k + 1;
                }
                if (li == pk) active = false;
                if (nz > 1) {
                    if (active) {
                        const uint32_t xn = ff_negate<ARITH>(s_x[par][li], R);
                        const uint32_t* pr = S + pk;
#pragma unroll 4
                        for (int j = g; j < w; j += G) {
                            const bool own = j == it;
                            const uint32_t y = own ? 0u : col[j * rs];
                            const uint32_t p = own ? scale : pr[j * rs];
                            col[j * rs] = ff_update<ARITH>(wt, y, xn, p, R);
                        }
                    }
                    scale = ARITH == kArithPow2 ? (scale * wt) & (R.q - 1u) : mont_mul(scale, wt, R.q, R.mont_qinv);
                }
                ++k;
            }
            if (it + 1 < w && ((it + 1) & (G - 1)) == g) publish(it + 1);
            __syncthreads();
        }
        if (tid == 0) {
            J.k = k;
            J.w = w;
            J.cnt = cnt;
            J.kind = TALL ? 3 : 2;
            // filled up: the block is worth trying again
            if (k == w && cnt == rows && rows > w) J.dense = 1;
        }
        if (k == 0 || J.c0 + w >= J.n || rows == k) continue;  // nothing to update
        if (tid < W) s_isp[tid] = 0;
        __syncthreads();
        if (tid == 0) s_inv = unit_inverse(scale, R);  // the rows below the pivots have the last scale
        // the listed rows' places: pivots in order; the others behind them (listed rows move), or where
        // they are but for those that a pivot row displaces (all rows)
        if constexpr (!TALL) {
            if (warp == 0) {
                int base = k;
                for (int r0 = 0; r0 < cnt; r0 += 32) {
                    const bool other = r0 + lane < cnt && s_step[r0 + lane] == 0;
                    const unsigned mask = __ballot_sync(0xffffffffu, other);
                    if (r0 + lane < cnt)
                        s_pos[r0 + lane] = other ? base + __popc(mask & ((1u << lane) - 1u)) : s_step[r0 + lane] - 1;
                    base += __popc(mask);
                }
            }
        } else {
            if (tid < k && s_row[s_prow[tid]] < k) s_isp[s_row[s_prow[tid]]] = 1;
            if (tid == 0) {
                int nv = 0;
                for (int t = 0; t < k; ++t)
                    if (s_row[s_prow[t]] >= k) s_vac[nv++] = s_row[s_prow[t]];
            }
            for (int i = tid; i < (rows - k) * W; i += NT) J.F[i] = 0u;
            __syncthreads();
            if (tid < cnt) {
                int pos = s_step[tid] ? s_step[tid] - 1 : s_row[tid];
                if (!s_step[tid] && pos < k) {
                    int rank = 0;
                    for (int i = 0; i < pos; ++i) rank += s_isp[i] ? 0 : 1;
                    pos = s_vac[rank];
                }
                s_pos[tid] = pos;
            }
        }
        __syncthreads();
        for (int r = warp; r < cnt; r += NW) {
            const int pos = s_pos[r];
            if (lane == 0 && pos < (TALL ? k : cnt)) J.rows[pos] = J.r0 + s_row[r];
            if (pos < k) continue;
            uint32_t* wd = J.F + static_cast<size_t>(pos - k) * W;
            const uint32_t sc = s_inv;
            for (int c = lane; c < w; c += 32) {
                const int t = s_colpiv[c];
                if (t >= 0) wd[t] = mod_mul(S[c * rs + r], sc, R.q, R.barrett);
            }
        }
    }
}

// gridDim.x CTAs per listed job, 32 columns at a time: rows[0 .. count) to r0 .. in columns [ca, cb), the
// rows they displace into their places (all reads before any write).
__global__ void __launch_bounds__(256) rr_moves_kernel(const RrMove* __restrict__ moves, const int* __restrict__ list,
                                                       const int* __restrict__ count) {
    extern __shared__ uint32_t s_mv[];  // [2 kRrCompact][32]
    __shared__ short s_src[2 * kRrCompact], s_dst[2 * kRrCompact];
    __shared__ unsigned char s_isp[kRrCompact];
    __shared__ int s_cnt[2][8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, njobs = *count;
    for (int i = blockIdx.y; i < njobs; i += gridDim.y) {
        const RrMove M = moves[list[i]];
        if (M.ca + static_cast<int>(blockIdx.x) * 32 >= M.cb) continue;
        __syncthreads();  // the job before is done with the shared state
        const int row = tid < M.count ? M.rows[tid] - M.r0 : tid;
        s_isp[tid] = 0;
        if (!__syncthreads_or(row != tid)) continue;  // all in place
        if (tid < M.count && row < M.count) s_isp[row] = 1;
        __syncthreads();
        const bool disp = tid < M.count && !s_isp[tid], vac = tid < M.count && row >= M.count;
        const unsigned md = __ballot_sync(0xffffffffu, disp), mv = __ballot_sync(0xffffffffu, vac);
        if (lane == 0) {
            s_cnt[0][warp] = __popc(md);
            s_cnt[1][warp] = __popc(mv);
        }
        __syncthreads();
        int nd = 0, d0 = 0, v0 = 0;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            nd += s_cnt[0][u];
            if (u < warp) {
                d0 += s_cnt[0][u];
                v0 += s_cnt[1][u];
            }
        }
        const unsigned below = (1u << lane) - 1u;
        if (tid < M.count) {
            s_src[tid] = static_cast<short>(row);
            s_dst[tid] = static_cast<short>(tid);
        }
        if (disp) s_src[M.count + d0 + __popc(md & below)] = static_cast<short>(tid);
        if (vac) s_dst[M.count + v0 + __popc(mv & below)] = static_cast<short>(row);
        __syncthreads();
        const int n = M.count + nd;
        uint32_t* A = M.A + static_cast<size_t>(M.r0) * M.ld;
        for (int c = M.ca + static_cast<int>(blockIdx.x) * 32 + lane; c - lane < M.cb; c += static_cast<int>(gridDim.x) * 32) {
            if (c < M.cb) {
#pragma unroll 4
                for (int u = warp; u < n; u += 8)
                    if (s_src[u] != s_dst[u]) s_mv[u * 32 + lane] = A[static_cast<size_t>(s_src[u]) * M.ld + c];
            }
            __syncthreads();
            if (c < M.cb) {
                for (int u = warp; u < n; u += 8)
                    if (s_src[u] != s_dst[u]) A[static_cast<size_t>(s_dst[u]) * M.ld + c] = s_mv[u * 32 + lane];
            }
            __syncthreads();
        }
    }
}

// A tile of rr_apply_kernel; MODE 0: p <= 2^16, 1: p < 2^31, 2: any p.
template <int MODE>
__device__ __forceinline__ void rr_apply_tile(const RrApply& J, const uint32_t (*s_M)[kRrW + 4], const uint32_t (*s_X)[33],
                                              uint32_t* src, bool in) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t acc[8] = {};
    uint32_t a0[8] = {}, a1[8] = {}, a2[8] = {};
#pragma unroll 2
    for (int s = 0; s < kRrW; s += 4) {
        const uint32_t x0 = s_X[s][lane], x1 = s_X[s + 1][lane], x2 = s_X[s + 2][lane], x3 = s_X[s + 3][lane];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const uint4 m = *reinterpret_cast<const uint4*>(&s_M[warp + 8 * e][s]);
            if constexpr (MODE == 0) {
                acc[e] += dot4(m.x, x0, m.y, x1, m.z, x2, m.w, x3);
            } else if constexpr (MODE == 1) {
                add96(a0[e], a1[e], a2[e], dot4(m.x, x0, m.y, x1, m.z, x2, m.w, x3));
            } else {
                mac96(a0[e], a1[e], a2[e], m.x, x0);
                mac96(a0[e], a1[e], a2[e], m.y, x1);
                mac96(a0[e], a1[e], a2[e], m.z, x2);
                mac96(a0[e], a1[e], a2[e], m.w, x3);
            }
        }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        uint64_t v = acc[e];
        if constexpr (MODE != 0) {
            const uint64_t h = reduce_u64((static_cast<uint64_t>(a2[e]) << 32) | a1[e], J.p, J.barrett);
            v = (h << 32) | a0[e];
        }
        if (in) src[static_cast<size_t>(warp + 8 * e) * J.ld] = reduce_u64(v, J.p, J.barrett);
    }
}

// A12 <- M A12 for the 64 pivot rows of the jobs settled by their top block:
// gridDim.x CTAs per listed job, 32 columns at a time, lane = column, eight rows per warp; each output is
// an exact dot product of 64 reduced once (64-bit sums for p <= 2^16, 64-bit
// sums of four products into 96 bits for p < 2^31, else 96-bit sums).
__global__ void __launch_bounds__(256, 3) rr_apply_kernel(const RrApply* __restrict__ jobs, const int* __restrict__ list,
                                                       const int* __restrict__ count) {
    __shared__ __align__(16) uint32_t s_M[kRrW][kRrW + 4];
    __shared__ uint32_t s_X[kRrW][33];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, njobs = *count;
    for (int i = blockIdx.y; i < njobs; i += gridDim.y) {
        const RrApply J = jobs[list[i]];
        if (static_cast<int>(blockIdx.x) * 32 >= J.cols) continue;
        __syncthreads();  // the job before is done with s_M
        {
            uint4 v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = reinterpret_cast<const uint4*>(J.M)[tid + 256 * e];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int at = 4 * (tid + 256 * e);
                *reinterpret_cast<uint4*>(&s_M[at >> 6][at & 63]) = v[e];
            }
        }
        for (int c0 = static_cast<int>(blockIdx.x) * 32; c0 < J.cols; c0 += static_cast<int>(gridDim.x) * 32) {
            const bool in = c0 + lane < J.cols;
            uint32_t* src = J.A + c0 + lane;
            uint32_t x[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] = in ? src[static_cast<size_t>(warp + 8 * e) * J.ld] : 0u;
            __syncthreads();  // the tile before is consumed
#pragma unroll
            for (int e = 0; e < 8; ++e) s_X[warp + 8 * e][lane] = x[e];
            __syncthreads();
            if (J.p > (1u << 31)) {
                rr_apply_tile<2>(J, s_M, s_X, src, in);
            } else if (J.p > (1u << 16)) {
                rr_apply_tile<1>(J, s_M, s_X, src, in);
            } else {
                rr_apply_tile<0>(J, s_M, s_X, src, in);
            }
        }
    }
}

// Each job's row moves, product, split and GEMM entries of the round, its tile
// and block counts, and its advance.
__global__ void rr_post_kernel(RrJob* __restrict__ jobs, int nj, RrMove* __restrict__ moves,
                               RrApply* __restrict__ applies, GroupedProblem* __restrict__ gprob,
                               GroupedSplitJob* __restrict__ gsplit, int* __restrict__ tiles, int* __restrict__ blocks,
                               const RrGroup* __restrict__ groups,
                               int* __restrict__ lists, int* __restrict__ counters) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < nj; j += gridDim.x * blockDim.x) {
        RrJob& J = jobs[j];
        RrMove& mv = moves[j];
        RrApply& ap = applies[j];
        tiles[j] = 0;
        blocks[j] = 0;
        if (!J.active) continue;
        const int k = J.k, c1 = J.c0 + J.w, ntrail = J.n - c1;
        const int below = J.kind == 2 ? J.cnt - k : J.m - J.r0 - k;  // rows that the update reaches
        if (k > 0 && ntrail > 0 && J.m - J.r0 > k) {
            mv.A = J.A;
            mv.ld = J.ld;
            mv.r0 = J.r0;
            mv.count = J.kind == 2 ? J.cnt : k;
            mv.ca = J.c0;
            mv.cb = J.n;
            mv.rows = J.rows;
            lists[static_cast<size_t>(kRrMove) * nj + atomicAdd(&counters[kRrMove], 1)] = j;
        }
        if (k > 0 && ntrail > 0 && below > 0) {
            const RrGroup& G = groups[J.group];
            uint32_t* A12 = J.A + static_cast<size_t>(J.r0) * J.ld + c1;
            if (J.kind == 1) {
                ap.A = A12;
                ap.ld = J.ld;
                ap.cols = ntrail;
                ap.M = J.F;
                lists[static_cast<size_t>(kRrSolve) * nj + atomicAdd(&counters[kRrSolve], 1)] = j;
                ap.p = G.p;
                ap.barrett = G.barrett;
            }
            GroupedProblem& gp = gprob[j];
            gp.tmA = G.tmA;
            gp.tmB = G.tmB;
            gp.C = J.A + static_cast<size_t>(J.r0 + k) * J.ld + c1;
            gp.ldc = J.ld;
            gp.M = below;
            gp.N = ntrail;
            gp.kblocks = 1;
            gp.op = J.kind == 1 ? HME_SUB : HME_ADD;
            gp.a_row0 = J.a_row0;
            gp.b_col0 = J.b_col0;
            tiles[j] = ((below + limb::kBM - 1) / limb::kBM) * ((ntrail + G.bn - 1) / G.bn);
            GroupedSplitJob& gs = gsplit[j];
            limb::SplitArgs& sa = gs.s;
            sa.A = J.kind == 1 ? J.A + static_cast<size_t>(J.r0 + k) * J.ld + J.c0 : J.F;
            sa.lda = J.kind == 1 ? J.ld : J.kind == 2 ? kRrW : 32;
            sa.B = A12;
            sa.ldb = J.ld;
            sa.M = below;
            sa.N = ntrail;
            sa.K = k;
            sa.Kp = kRrW;
            sa.red = G.split_red;
            sa.planesA = G.planesA + static_cast<size_t>(J.a_row0) * kRrW;
            sa.planesB = G.planesB + static_cast<size_t>(J.b_col0) * kRrW;
            sa.a_plane = G.sum_m * kRrW;
            sa.b_plane = G.sum_n * kRrW;
            sa.a_blocks = min(64, max(1, (below * (kRrW / 16) + 255) / 256));
            sa.b_blocks_k = 1;
            sa.a_vec = (reinterpret_cast<uintptr_t>(sa.A) & 15) == 0 && (sa.lda & 3) == 0;
            sa.skip = Skip{};
            gs.b_blocks = (ntrail + 31) / 32;
            blocks[j] = sa.a_blocks + gs.b_blocks;
        }
        J.r0 += k;
        J.c0 = c1;
        J.active = J.r0 < J.m && J.c0 < J.n;
        if (J.active) atomicAdd(&counters[kRrActive], 1);
    }
}

// Per group (one CTA each): exclusive prefix sums of the jobs' tile and block
// counts into the GEMM and split tables, and the totals.
__global__ void __launch_bounds__(1024) rr_scan_kernel(const RrGroup* __restrict__ groups,
                                                       const int* __restrict__ tiles,
                                                       const int* __restrict__ blocks,
                                                       GroupedProblem* __restrict__ gprob,
                                                       GroupedSplitJob* __restrict__ gsplit) {
    __shared__ int w_t[32], w_b[32];
    const RrGroup& G = groups[blockIdx.x];
    const int n = G.end - G.begin;
    const int per = (n + blockDim.x - 1) / blockDim.x;
    const int i0 = G.begin + static_cast<int>(threadIdx.x) * per;
    const int i1 = min(G.end, i0 + per);
    int st = 0, sb = 0;
    for (int i = i0; i < i1; ++i) {
        st += tiles[i];
        sb += blocks[i];
    }
    // exclusive scan of (st, sb) over the threads
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int it = st, ib = sb;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int yt = __shfl_up_sync(0xffffffffu, it, off), yb = __shfl_up_sync(0xffffffffu, ib, off);
        if (lane >= off) {
            it += yt;
            ib += yb;
        }
    }
    if (lane == 31) {
        w_t[warp] = it;
        w_b[warp] = ib;
    }
    __syncthreads();
    if (warp == 0) {
        int vt = lane < static_cast<int>(blockDim.x >> 5) ? w_t[lane] : 0;
        int vb = lane < static_cast<int>(blockDim.x >> 5) ? w_b[lane] : 0;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int yt = __shfl_up_sync(0xffffffffu, vt, off), yb = __shfl_up_sync(0xffffffffu, vb, off);
            if (lane >= off) {
                vt += yt;
                vb += yb;
            }
        }
        w_t[lane] = vt;  // inclusive prefix over warps
        w_b[lane] = vb;
    }
    __syncthreads();
    int bt = it - st + (warp > 0 ? w_t[warp - 1] : 0);
    int bb = ib - sb + (warp > 0 ? w_b[warp - 1] : 0);
    for (int i = i0; i < i1; ++i) {
        gprob[i].tile_begin = bt;
        gsplit[i].block_begin = bb;
        bt += tiles[i];
        bb += blocks[i];
    }
    if (threadIdx.x == blockDim.x - 1) {
        G.totals[0] = bt;
        G.totals[1] = bb;
    }
}

// The per-tile problem and per-block job indexes of every group: a warp per job.
__global__ void __launch_bounds__(256) rr_fill_kernel(const RrGroup* __restrict__ groups, const RrJob* __restrict__ jobs,
                                                      int nj, const int* __restrict__ tiles,
                                                      const int* __restrict__ blocks,
                                                      const GroupedProblem* __restrict__ gprob,
                                                      const GroupedSplitJob* __restrict__ gsplit) {
    const int lane = threadIdx.x & 31;
    for (int j = blockIdx.x * 8 + (threadIdx.x >> 5); j < nj; j += gridDim.x * 8) {
        const int nt = tiles[j], nb = blocks[j];
        if (nt == 0) continue;
        const RrGroup& G = groups[jobs[j].group];
        int* tp = G.tile_prob + gprob[j].tile_begin;
        int* bj = G.block_job + gsplit[j].block_begin;
        for (int t = lane; t < nt; t += 32) tp[t] = j - G.begin;
        for (int b = lane; b < nb; b += 32) bj[b] = j - G.begin;
    }
}

size_t a256(size_t x) { return (x + 255) / 256 * 256; }

size_t general_smem(int rows, int w) { return sizeof(uint32_t) * static_cast<size_t>(w) * (rows + 1); }

}  // namespace

bool batch_rank_rounds(hme_ctx* ctx, const std::vector<BatchMatrix>& mats, std::vector<int> order,
                       std::vector<int>& ranks) {
    // modulus groups: jobs sorted by modulus (stable)
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return mats[x].p < mats[y].p; });
    const int nj = static_cast<int>(order.size());
    std::vector<uint32_t> gmod;
    std::vector<int> gbegin;
    for (int i = 0; i < nj; ++i)
        if (i == 0 || mats[order[i]].p != mats[order[i - 1]].p) {
            gmod.push_back(mats[order[i]].p);
            gbegin.push_back(i);
        }
    const int ng = static_cast<int>(gmod.size());
    gbegin.push_back(nj);

    // ---- fixed layout: per-job state and buffers, per-group planes and tables
    std::vector<RrJob> jobs(nj);
    std::vector<RrGroup> groups(ng);
    std::vector<size_t> off(nj), g_planes(ng), g_tiles(ng, 0), g_blocks(ng, 0);
    size_t buf_bytes = 0, plane_bytes = 0;
    uint32_t max_n = 0;
    bool any_tall = false;
    for (int g = 0; g < ng; ++g) {
        const ModParams mp = make_mod(gmod[g]);
        const int L = static_cast<int>(mp.limbs), bn = grouped_bn_wide(L);
        uint64_t sm = 0, sn = 0;
        for (int i = gbegin[g]; i < gbegin[g + 1]; ++i) {
            const BatchMatrix& M = mats[order[i]];
            RrJob& J = jobs[i];
            J = RrJob{};
            J.A = M.A;
            J.ld = M.ld;
            J.m = static_cast<int>(M.m);
            J.n = static_cast<int>(M.n);
            J.group = g;
            J.active = J.dense = 1;
            J.a_row0 = static_cast<int>(sm);
            J.b_col0 = static_cast<int>(sn);
            sm += M.m;
            sn += M.n;
            off[i] = buf_bytes;
            // B^-1 or W, then the moved rows' list
            const size_t words = std::max<size_t>(static_cast<size_t>(std::min<uint32_t>(M.m, kRrCompact)) * kRrW,
                                                  M.m > kRrCompact ? static_cast<size_t>(M.m) * 32 : 0);
            buf_bytes += a256(sizeof(uint32_t) * words) + sizeof(int) * kRrCompact;
            any_tall = any_tall || M.m > kRrCompact;
            max_n = std::max(max_n, M.n);
            g_tiles[g] += static_cast<size_t>((M.m + limb::kBM - 1) / limb::kBM) * ((M.n + bn - 1) / bn);
            g_blocks[g] += 64 + (M.n + 31) / 32;
        }
        RrGroup& G = groups[g];
        G = RrGroup{};
        G.p = gmod[g];
        G.barrett = mp.barrett;
        uint32_t x = G.p;  // p^-1 mod 2^32 by Newton's iteration (x = p is right to 3 bits)
        for (int t = 0; t < 5; ++t) x *= 2u - G.p * x;
        G.mont_qinv = 0u - x;
        G.mont_r2 = static_cast<uint32_t>((static_cast<unsigned __int128>(1) << 64) % G.p);
        G.sum_m = sm;
        G.sum_n = sn;
        G.bn = bn;
        G.split_red = limb::make_split_red(mp);
        G.begin = gbegin[g];
        G.end = gbegin[g + 1];
        g_planes[g] = plane_bytes;
        plane_bytes += a256(static_cast<size_t>(L) * sm * kRrW) + a256(static_cast<size_t>(L) * L * sn * kRrW);
    }
    size_t tb = 0;
    auto take = [&](size_t bytes) {
        const size_t o = tb;
        tb += a256(bytes);
        return o;
    };
    const size_t o_jobs = take(sizeof(RrJob) * nj), o_moves = take(sizeof(RrMove) * nj);
    const size_t o_apply = take(sizeof(RrApply) * nj);
    const size_t o_gprob = take(sizeof(GroupedProblem) * nj), o_gsplit = take(sizeof(GroupedSplitJob) * nj);
    const size_t o_tiles = take(sizeof(int) * nj), o_blocks = take(sizeof(int) * nj);
    const size_t o_lists = take(sizeof(int) * kRrLists * static_cast<size_t>(nj));
    const size_t o_counters = take(sizeof(int) * kRrCounters);
    const size_t o_groups = take(sizeof(RrGroup) * ng), o_maps = take(sizeof(CUtensorMap) * 2 * ng);
    const size_t o_totals = take(sizeof(int) * 2 * ng);
    std::vector<size_t> o_tp(ng), o_bj(ng);
    for (int g = 0; g < ng; ++g) {
        o_tp[g] = take(sizeof(int) * g_tiles[g]);
        o_bj[g] = take(sizeof(int) * g_blocks[g]);
    }
    if (!ctx->ws.holds({{kSlotJobs1, tb}, {kSlotJobs4, buf_bytes}, {kSlotJobs0, plane_bytes}}, ctx->stream)) return false;
    uint8_t* tables = static_cast<uint8_t*>(ctx->ws.get(kSlotJobs1, tb));
    uint8_t* bufs = static_cast<uint8_t*>(ctx->ws.get(kSlotJobs4, buf_bytes));
    uint8_t* planes = static_cast<uint8_t*>(ctx->ws.get(kSlotJobs0, plane_bytes));
    RrJob* d_jobs = reinterpret_cast<RrJob*>(tables + o_jobs);
    RrMove* d_moves = reinterpret_cast<RrMove*>(tables + o_moves);
    RrApply* d_apply = reinterpret_cast<RrApply*>(tables + o_apply);
    GroupedProblem* d_gprob = reinterpret_cast<GroupedProblem*>(tables + o_gprob);
    GroupedSplitJob* d_gsplit = reinterpret_cast<GroupedSplitJob*>(tables + o_gsplit);
    int* d_tiles = reinterpret_cast<int*>(tables + o_tiles);
    int* d_blocks = reinterpret_cast<int*>(tables + o_blocks);
    int* d_lists = reinterpret_cast<int*>(tables + o_lists);
    int* d_counters = reinterpret_cast<int*>(tables + o_counters);
    RrGroup* d_groups = reinterpret_cast<RrGroup*>(tables + o_groups);
    CUtensorMap* d_maps = reinterpret_cast<CUtensorMap*>(tables + o_maps);
    int* d_totals = reinterpret_cast<int*>(tables + o_totals);
    for (int i = 0; i < nj; ++i) {
        const size_t end = i + 1 < nj ? off[i + 1] : buf_bytes;
        jobs[i].F = reinterpret_cast<uint32_t*>(bufs + off[i]);
        jobs[i].rows = reinterpret_cast<int*>(bufs + end - sizeof(int) * kRrCompact);
    }
    std::vector<CUtensorMap> maps(2 * static_cast<size_t>(ng));
    for (int g = 0; g < ng; ++g) {
        RrGroup& G = groups[g];
        const int L = static_cast<int>(make_mod(gmod[g]).limbs);
        G.planesA = planes + g_planes[g];
        G.planesB = G.planesA + a256(static_cast<size_t>(L) * G.sum_m * kRrW);
        {
            const cuuint64_t dims[3] = {kRrW, G.sum_m, static_cast<cuuint64_t>(L)};
            const cuuint64_t strides[2] = {kRrW, kRrW * G.sum_m};
            const cuuint32_t box[3] = {kRrW, limb::kBM, 1};
            encode_tma_u8_kb(&maps[2 * g], G.planesA, 3, dims, strides, box, kRrW);
        }
        {
            const cuuint64_t dims[4] = {kRrW, G.sum_n, static_cast<cuuint64_t>(L), static_cast<cuuint64_t>(L)};
            const cuuint64_t strides[3] = {kRrW, kRrW * G.sum_n, kRrW * G.sum_n * L};
            const cuuint32_t box[4] = {kRrW, static_cast<cuuint32_t>(G.bn), static_cast<cuuint32_t>(L), 1};
            encode_tma_u8_kb(&maps[2 * g + 1], G.planesB, 4, dims, strides, box, kRrW);
        }
        G.tmA = d_maps + 2 * g;
        G.tmB = d_maps + 2 * g + 1;
        G.tile_prob = reinterpret_cast<int*>(tables + o_tp[g]);
        G.block_job = reinterpret_cast<int*>(tables + o_bj[g]);
        G.totals = d_totals + 2 * g;
    }
    HME_CUDA(cudaMemcpyAsync(d_jobs, jobs.data(), sizeof(RrJob) * nj, cudaMemcpyHostToDevice, ctx->stream));
    HME_CUDA(cudaMemcpyAsync(d_groups, groups.data(), sizeof(RrGroup) * ng, cudaMemcpyHostToDevice, ctx->stream));
    HME_CUDA(cudaMemcpyAsync(d_maps, maps.data(), sizeof(CUtensorMap) * 2 * ng, cudaMemcpyHostToDevice, ctx->stream));

    // ---- launch shapes of a round (fixed)
    // A panel whose top 64 rows are singular (probability about 1 / p for a dense matrix) costs the job two
    // rounds over all rows: 32 spare rows below p = 1024, none above.
    const size_t gen_smem = general_smem(kRrCompact, kRrW), tall_smem = general_smem(1024, 32);
    const size_t move_smem = sizeof(uint32_t) * 2 * kRrCompact * 32;
    struct PanelKernels {
        decltype(&rr_block_kernel<panel::kArithPow2, 96>) block, general, tall;
        int rs;
        int grid_block, grid_general;
    };
    PanelKernels kern[3];
    int nkern = 0;
    auto add = [&](auto arith, uint32_t p_min) {
        constexpr int AR = decltype(arith)::value;
        PanelKernels& K = kern[nkern++];
        K.rs = p_min < 1024 ? 96 : 64;
        K.block = rr_block_kernel<AR, 96>;
        if constexpr (AR != panel::kArithPow2)
            if (K.rs == 64) K.block = rr_block_kernel<AR, 64>;
        K.general = rr_general_kernel<AR, kRrCompact, kRrThreads>;
        K.tall = rr_general_kernel<AR, 1024, 1024>;
        static OncePerDevice attr;
        attr.run([&](int) {
            HME_CUDA(cudaFuncSetAttribute(rr_general_kernel<AR, kRrCompact, kRrThreads>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(gen_smem)));
            HME_CUDA(cudaFuncSetAttribute(rr_general_kernel<AR, 1024, 1024>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(tall_smem)));
        });
        int occ_block = 1, occ_gen = 1;
        HME_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_block, K.block, 4 * K.rs,
                                                               panel::block_smem_bytes(K.rs, kRrW)));
        HME_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_gen, K.general, kRrThreads, gen_smem));
        K.grid_block = std::min(nj, ctx->num_sms * std::max(1, occ_block));
        K.grid_general = std::min(nj, ctx->num_sms * std::max(1, occ_gen));
    };
    for (int g = 0; g < ng; ++g) {  // (ascending: the first modulus of an arithmetic is its smallest)
        const int ar = rr_arith(gmod[g]);
        if (g > 0 && ar == rr_arith(gmod[g - 1])) continue;
        if (ar == panel::kArithPow2) add(std::integral_constant<int, panel::kArithPow2>{}, gmod[g]);
        else if (ar == panel::kArithMont31) add(std::integral_constant<int, panel::kArithMont31>{}, gmod[g]);
        else add(std::integral_constant<int, panel::kArithMont32>{}, gmod[g]);
    }
    static OncePerDevice attr;
    attr.run([&](int) {
        HME_CUDA(cudaFuncSetAttribute(rr_moves_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(move_smem)));
    });
    const int grid_tall = std::min(nj, ctx->num_sms);
    const int small_grid = std::min((nj + 255) / 256, ctx->num_sms * 8);
    const int fill_grid = std::min((nj + 7) / 8, ctx->num_sms * 8);
    const dim3 cols_grid(4, std::min(nj, ctx->num_sms * 2));
    auto round = [&]() {
        HME_CUDA(cudaMemsetAsync(d_counters, 0, sizeof(int) * kRrCounters, ctx->stream));
        HME_TIMED(ctx, "rank_plan", rr_plan_kernel<<<small_grid, 256, 0, ctx->stream>>>(d_jobs, nj, d_lists, d_counters));
        for (int i = 0; i < nkern; ++i) {
            const PanelKernels& K = kern[i];
            HME_TIMED(ctx, "rank_block", K.block<<<K.grid_block, 4 * K.rs, panel::block_smem_bytes(K.rs, kRrW), ctx->stream>>>(
                                             d_jobs, nj, d_lists, d_counters, d_groups));
        }
        for (int i = 0; i < nkern; ++i)
            HME_TIMED(ctx, "rank_general", kern[i].general<<<kern[i].grid_general, kRrThreads, gen_smem, ctx->stream>>>(
                                               d_jobs, nj, d_lists, d_counters, d_groups));
        for (int i = 0; any_tall && i < nkern; ++i)
            HME_TIMED(ctx, "rank_general", kern[i].tall<<<grid_tall, 1024, tall_smem, ctx->stream>>>(
                                               d_jobs, nj, d_lists, d_counters, d_groups));
        HME_TIMED(ctx, "rank_post", rr_post_kernel<<<small_grid, 256, 0, ctx->stream>>>(
                                        d_jobs, nj, d_moves, d_apply, d_gprob, d_gsplit, d_tiles, d_blocks, d_groups,
                                        d_lists, d_counters));
        HME_TIMED(ctx, "rank_post", rr_scan_kernel<<<ng, 1024, 0, ctx->stream>>>(d_groups, d_tiles, d_blocks, d_gprob,
                                                                                d_gsplit));
        HME_TIMED(ctx, "rank_post", rr_fill_kernel<<<fill_grid, 256, 0, ctx->stream>>>(d_groups, d_jobs, nj, d_tiles,
                                                                                      d_blocks, d_gprob, d_gsplit));
        HME_TIMED(ctx, "rank_moves", rr_moves_kernel<<<cols_grid, 256, move_smem, ctx->stream>>>(
                                         d_moves, d_lists + static_cast<size_t>(kRrMove) * nj, d_counters + kRrMove));
        HME_TIMED(ctx, "rank_apply", rr_apply_kernel<<<cols_grid, 256, 0, ctx->stream>>>(
                                         d_apply, d_lists + static_cast<size_t>(kRrSolve) * nj, d_counters + kRrSolve));
        for (int g = 0; g < ng; ++g) {
            const RrGroup& G = groups[g];
            grouped_launch_device_tables(ctx, make_mod(gmod[g]), kRrW, d_gsplit + G.begin, G.block_job, G.totals + 1,
                                         d_gprob + G.begin, G.tile_prob, G.totals);
        }
        HME_CUDA(cudaGetLastError());
    };
    for (int g = 0; g < ng; ++g) grouped_prepare_device_tables(make_mod(gmod[g]).limbs, kRrW);
    // A round takes 64 columns, or 32 of a job with more than 256 rows in the panel: the rounds that suffice
    // in the first case, then the others while the device reports active jobs.
    const int expect = static_cast<int>((max_n + kRrW - 1) / kRrW), most = static_cast<int>((max_n + 31) / 32);
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    struct GraphGuard {
        cudaGraph_t* g;
        cudaGraphExec_t* e;
        ~GraphGuard() {
            if (*e) cudaGraphExecDestroy(*e);
            if (*g) cudaGraphDestroy(*g);
        }
    } guard{&graph, &exec};
    if (!ctx->timer.on) {
        HME_CUDA(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
        try {
            round();
        } catch (...) {
            cudaStreamEndCapture(ctx->stream, &graph);
            throw;
        }
        HME_CUDA(cudaStreamEndCapture(ctx->stream, &graph));
        HME_CUDA(cudaGraphInstantiate(&exec, graph, 0));
    }
    for (int done = 0, active = 1; active != 0 && done < most;) {
        const int n = done == 0 ? expect : std::min(4, most - done);
        for (int r = 0; r < n; ++r) {
            if (exec) HME_CUDA(cudaGraphLaunch(exec, ctx->stream));
            else round();
        }
        done += n;
        HME_CUDA(cudaMemcpyAsync(&active, d_counters + kRrActive, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
        HME_CUDA(cudaStreamSynchronize(ctx->stream));
    }
    check_device_error(ctx);
    HME_CUDA(cudaMemcpy(jobs.data(), d_jobs, sizeof(RrJob) * nj, cudaMemcpyDeviceToHost));
    for (int i = 0; i < nj; ++i) ranks[order[i]] = jobs[i].r0;
    return true;
}

}  // namespace hme
