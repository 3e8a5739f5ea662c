// Device-resident elimination over F_p, p < 2^32 prime: RREF, rank, column
// rank profile, determinant (and, built on them, kernel basis, inverse, solve).
//
// Reference semantics: engine::elim::rref / column_rank_profile
// (src/ModArithmetic/DenseElim.h:153-169; Plu factor / trailing_update / to_rref
// DenseElim.cpp:323-560, rref :921).  RREF(A) is unique (leading 1, zero rows
// at the bottom) and its pivot columns are the column rank profile, so the pivot
// ROW choice cannot show in the output; this driver takes the reference's rule
// anyway (leftmost column with a non-zero in the Schur complement, topmost such
// row) because it is also the cheapest to find in parallel (a min over rows).
//
// Blocked right-looking LU, panels of `bw` columns:
//   1. the panel's pivots.  First the top-block path (panel_block_kernel): one
//      CTA eliminates the panel's top rows alone, which settles the panel when
//      they supply a unit for every column.  Then, where most of the panel's rows
//      are zero, panel_compact_kernel over the others, in one CTA.  Otherwise the
//      searching kernel: panel_cluster_kernel, the panel's active rows A[r0:m, c0:c0+bw) in the
//      shared memory of one thread-block cluster (up to 16 CTAs); per column
//      each CTA pushes its best (valuation, row) key and that row to every CTA
//      through distributed shared memory, one cluster barrier, a warp min of
//      the keys; fraction-free row updates, unit scales undone once per panel.
//      Panels too tall for one cluster take panel_factor_kernel: one
//      cooperative launch over all SMs with one bounded grid barrier per column.
//   2. move_pivot_rows_kernel: the pivot rows to rows r0 .. r0+k-1 in pivot
//      order, the rows they displace into their places (columns >= c0; columns
//      left of the panel of non-U rows hold dead multipliers).
//   3. the left factor W = [L^-1 - I; -X M] (panel_w_kernel): X the other rows'
//      entries at the pivot columns, M = B^-1 after the top block, L11^-1
//      (panel_linv_kernel) after a search; the compact kernel has written it.
//   4. [A12; A22] += W A12: one INT8-limb tcgen05 GEMM, K = k pivots; the top
//      rows become U12, the rest the Schur complement.
// A panel without a pivot asks whether anything is left below: a rank-deficient
// matrix stops there.
// Then RREF = U1^-1 U on the free columns only (the pivot columns of the RREF
// are the identity): every diagonal block of U1 is inverted in shared memory
// (one launch, tri_inv_kernel), many blocks are joined by pairs (pair_blocks_kernel), and the blocked backward substitution is two limb GEMMs per
// block (X_B = U_BB^-1 W_B, then W_above -= U_above,B X_B).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstring>
#include <exception>
#include <mutex>
#include <numeric>
#include <type_traits>
#include <vector>

#include "hme_elim.h"
#include "hme_grouped.h"
#include "hme_internal.h"
#include "hme_panel.cuh"
#include "hme_ptx.cuh"

namespace hme {
namespace {

using namespace panel;

constexpr int kPanelThreads = 256;
constexpr int kPanelWarps = kPanelThreads / 32;
constexpr int kPanelSmemMax = 160 * 1024;  // largest shared-memory row slice of the panel kernel
constexpr unsigned long long kNoKey = 0x7f7f7f7f7f7f7f7full;  // piv_slot sentinel (memset 0x7f)


// Pivot key of an entry: (valuation << 32 | row), or kNoKey when x is zero or
// its valuation exceeds the ring's max_v.
__device__ __forceinline__ unsigned long long pivot_key(uint32_t x, int row, const Ring& R) {
    if (x == 0) return kNoKey;
    const uint32_t v = R.k == 1 ? 0u : R.max_v == 0 ? (x % R.ell == 0 ? 1u : 0u) : valuation(x, R, R.max_v);
    if (v > R.max_v) return kNoKey;
    return (static_cast<unsigned long long>(v) << 32) | static_cast<unsigned>(row);
}

struct PanelArgs {
    uint32_t* A;
    uint64_t ld;
    int m;
    int c0, bw;  // panel columns [c0, c0 + bw)
    int r0;      // first active row
    Ring R;
    unsigned long long* piv_slot;  // [bw], kNoKey on entry: smallest (valuation, row) key per column
    uint32_t* cand;      // [2][grid][kMaxPanel]: candidate row values, by column parity
    int* pivot_rows;     // [bw] out
    int* pivot_cols;     // [bw] out
    int* k_out;          // out: pivots found
    unsigned* bar;       // [2]: arrival count, generation
    int* err;
    const int* skip;     // non-null and non-zero: the panel is settled already (top block, compact rows)
    int keep;            // pivotless columns left of a pivot are updated too (cluster kernel only)
};

// Bounded grid-wide barrier for a cooperative launch (all CTAs co-resident).
// Returns false on timeout or when another CTA already gave up.
__device__ bool grid_barrier(unsigned* bar, int* err, int* s_flag) {
    __syncthreads();
    if (threadIdx.x == 0) {
        volatile unsigned* vgen = bar + 1;
        volatile int* verr = err;
        const unsigned g = *vgen;
        __threadfence();
        const unsigned arrived = atomicAdd(bar, 1u);
        int ok = 1;
        if (arrived == gridDim.x - 1) {
            atomicExch(bar, 0u);
            __threadfence();
            atomicAdd(bar + 1, 1u);
        } else {
            const uint64_t t0 = global_timer_ns();
            uint32_t spin = 0;
            while (*vgen == g) {
                if ((++spin & 63u) == 0) {
                    if (*verr != 0) { ok = 0; break; }
                    if (global_timer_ns() - t0 > HME_WAIT_LIMIT_NS) {
                        atomicCAS(err, 0, DERR_GRID_BARRIER);
                        ok = 0;
                        break;
                    }
                }
            }
        }
        __threadfence();
        *s_flag = ok;
    }
    __syncthreads();
    return *s_flag != 0;
}

// One cooperative launch per panel.  With smem_rows, every CTA copies its
// slice of the panel (rpc rows x bw columns) into shared memory first and
// writes it back at the end, so the per-column work never leaves the SM; the
// global-memory mode (slices too large for shared memory) works in place.
__global__ void __launch_bounds__(kPanelThreads) panel_factor_kernel(const PanelArgs a, int smem_rows) {
    extern __shared__ uint32_t s_slice[];
    __shared__ uint32_t s_prow[kMaxPanel];
    __shared__ unsigned long long s_cand;
    __shared__ int s_flag;
    __shared__ unsigned long long s_piv;
    __shared__ uint32_t s_inv, s_div;

    // settled by the top-block path: the same in every CTA, before any grid barrier
    if (a.skip != nullptr && *a.skip != 0) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int active_rows = a.m - a.r0;
    const int rpc = (active_rows + gridDim.x - 1) / gridDim.x;
    const int row_begin = a.r0 + blockIdx.x * rpc;
    const int row_end = min(a.m, row_begin + rpc);
    const int cend = a.c0 + a.bw;
    const size_t cand_stride = static_cast<size_t>(gridDim.x) * kMaxPanel;

    // row i of the panel, indexed by absolute column c in [c0, cend)
    auto rowp = [&](int i) -> uint32_t* {
        return smem_rows ? s_slice + static_cast<size_t>(i - row_begin) * a.bw - a.c0
                         : a.A + static_cast<size_t>(i) * a.ld;
    };
    if (smem_rows) {
        for (int i = row_begin + warp; i < row_end; i += kPanelWarps) {
            const uint32_t* src = a.A + static_cast<size_t>(i) * a.ld;
            uint32_t* dst = rowp(i);
            for (int j = a.c0 + lane; j < cend; j += 32) dst[j] = src[j];
        }
    }
    // per-row multiplier of the current column, and per-row flag: the row
    // became a pivot row of this panel
    uint32_t* s_l = s_slice + (smem_rows ? static_cast<size_t>(rpc) * a.bw : 0);
    unsigned char* s_isp = reinterpret_cast<unsigned char*>(s_l + rpc);
    for (int i = threadIdx.x; i < rpc; i += blockDim.x) s_isp[i] = 0;
    __syncthreads();
    auto is_pivot_row = [&](int i) { return s_isp[i - row_begin] != 0; };

    // Publish this CTA's best pivot candidate for column c (smallest
    // (valuation, row) key, already in s_cand): the row's values of columns
    // [c, cend) into the parity slot, the key by atomicMin.
    auto publish_candidate = [&](int c) {
        __syncthreads();
        if (c < cend && s_cand != kNoKey) {
            const uint32_t* src = rowp(static_cast<int>(s_cand & 0xffffffffu));
            uint32_t* dst = a.cand + static_cast<size_t>(c & 1) * cand_stride + static_cast<size_t>(blockIdx.x) * kMaxPanel;
            for (int j = c + threadIdx.x; j < cend; j += blockDim.x) dst[j - a.c0] = src[j];
            __syncthreads();
            if (threadIdx.x == 0) {
                __threadfence();
                atomicMin(&a.piv_slot[c - a.c0], s_cand);
            }
        }
    };
    auto find_candidate = [&](int c) {
        if (threadIdx.x == 0) s_cand = kNoKey;
        __syncthreads();
        if (c < cend) {
            for (int i = row_begin + threadIdx.x; i < row_end; i += blockDim.x) {
                const unsigned long long key = pivot_key(rowp(i)[c], i, a.R);
                if (key != kNoKey && !is_pivot_row(i)) atomicMin(&s_cand, key);
            }
        }
        publish_candidate(c);
    };

    find_candidate(a.c0);
    int k = 0;
    bool ok = true;
    for (int c = a.c0; c < cend; ++c) {
        if (!grid_barrier(a.bar, a.err, &s_flag)) {
            ok = false;
            break;
        }
        if (threadIdx.x == 0) s_piv = *reinterpret_cast<volatile unsigned long long*>(&a.piv_slot[c - a.c0]);
        __syncthreads();
        const unsigned long long pkey = s_piv;
        if (pkey == kNoKey) {
            // column c is not a pivot column: every active row is zero there
            find_candidate(c + 1);
            continue;
        }
        const int prow = static_cast<int>(pkey & 0xffffffffu);
        const uint32_t pv = static_cast<uint32_t>(pkey >> 32);
        const int owner = (prow - a.r0) / rpc;
        const uint32_t* src = a.cand + static_cast<size_t>(c & 1) * cand_stride + static_cast<size_t>(owner) * kMaxPanel;
        for (int j = c + threadIdx.x; j < cend; j += blockDim.x)
            s_prow[j - a.c0] = *reinterpret_cast<const volatile uint32_t*>(&src[j - a.c0]);
        if (threadIdx.x == 0) {
            if (prow >= row_begin && prow < row_end) s_isp[prow - row_begin] = 1;
            if (blockIdx.x == 0) {
                a.pivot_rows[k] = prow;
                a.pivot_cols[k] = c;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            // pivot x = ell^v * u: multipliers are (x_i / ell^v) * u^-1
            const uint32_t x = s_prow[c - a.c0];
            const uint32_t div = a.R.pw[pv];
            s_div = div;
            s_inv = unit_inverse(x / div, a.R);
        }
        __syncthreads();
        const uint32_t inv = s_inv, div = s_div;
        ++k;
        // eliminate column c from this CTA's active rows in two phases:
        // (1) one thread per row: multiplier l = (x / ell^v) * u^-1, stored in
        //     the pivot column (packed L); (2) all threads over the (row,
        //     column > c) elements, l * pivot row subtracted; the elements of
        //     column c + 1 feed the next column's pivot candidate on the way.
        const int nloc = row_end - row_begin;
        if (threadIdx.x == 0) s_cand = kNoKey;
        for (int li = threadIdx.x; li < nloc; li += blockDim.x) {
            const int i = row_begin + li;
            uint32_t l = 0;
            if (i != prow && !is_pivot_row(i)) {
                uint32_t* row = rowp(i);
                const uint32_t x = row[c];
                if (x != 0) {
                    l = mod_mul(div == 1 ? x : x / div, inv, a.R.q, a.R.barrett);
                    row[c] = l;
                }
            }
            s_l[li] = l;
        }
        __syncthreads();
        const int width = cend - c - 1;
        if (width > 0) {
            const int total = nloc * width;
            for (int e = threadIdx.x; e < total; e += blockDim.x) {
                const int li = e / width, j = c + 1 + (e - li * width);
                const int i = row_begin + li;
                uint32_t* row = rowp(i);
                uint32_t y = row[j];
                const uint32_t l = s_l[li];
                if (l != 0) {
                    y = mod_sub(y, mod_mul(l, s_prow[j - a.c0], a.R.q, a.R.barrett), a.R.q);
                    row[j] = y;
                }
                if (j == c + 1 && i != prow && !is_pivot_row(i)) {
                    const unsigned long long key = pivot_key(y, i, a.R);
                    if (key != kNoKey) atomicMin(&s_cand, key);
                }
            }
        }
        publish_candidate(c + 1);
    }
    if (smem_rows) {
        __syncthreads();
        for (int i = row_begin + warp; i < row_end; i += kPanelWarps) {
            uint32_t* dst = a.A + static_cast<size_t>(i) * a.ld;
            const uint32_t* srow = rowp(i);
            for (int j = a.c0 + lane; j < cend; j += 32) dst[j] = srow[j];
        }
    }
    if (ok && blockIdx.x == 0 && threadIdx.x == 0) *a.k_out = k;
}

// ---- the panel on one thread-block cluster ---------------------------------------
// The same factorisation as panel_factor_kernel, for panels whose active rows
// fit the shared memory of one cluster (up to kClusterMax CTAs).  Each CTA
// keeps its slice of rows in shared memory, column-major, for the whole panel;
// the per-column exchange goes through distributed shared memory.
//
// Fraction-free row updates.  A column step needs no modular inverse: with the
// pivot x_p = ell^v * w (w a unit) every other active row becomes
//     row <- (w * row - (x_i / ell^v) * pivot_row) * rho          (mod q)
// with rho = 2^-32 in the Montgomery arithmetic of odd q (one reduction per
// element) and rho = 1 for q = 2^k (wraparound).  Every active row, pivot-free
// or not, is multiplied by the same unit w * rho, so after step t the active
// rows hold S_t times the values of the classical elimination, S_t = prod of
// (w_s rho) over s < t, and (x_i / ell^v) is stored as the raw multiplier.  The
// classical multiplier is (x_i / ell^v) * w_t^-1 and the classical pivot row
// t is its frozen raw row times S_t^-1; valuations (and zero / non-zero) do
// not change under unit scaling, so the pivot sequence is the classical one.
// After the last column every CTA computes the w_t^-1 in parallel and the
// prefix products S_t^-1, and rescales its rows once: the panel leaves the
// kernel as panel_factor_kernel leaves it (entry for entry over a field and for
// unit pivots; for pivots of valuation v > 0 the multiplier x / ell^v is only
// defined mod ell^(k-v), and the kernel's lift, consistent with the row
// updates it made, may differ from that kernel's by a multiple of ell^(k-v)).
// Like that kernel it updates only the columns right of each pivot.
//
// Per column:
//   1. every CTA pushes its best pivot key and that row's values (columns
//      [c, cend)) into a receive slot of every CTA of the cluster;
//   2. one hardware cluster barrier (release / acquire), reached once per
//      column by every thread of every CTA whatever the data;
//   3. every warp takes the smallest key of the slots (a warp min), and the
//      CTA updates its rows with the pivot row from its own receive slot.
// Receive slots are double-buffered by column parity: a CTA writes slot parity
// (it & 1) of column it only after passing barrier it - 1, when every CTA has
// finished column it - 2.  A cluster barrier before the first push makes sure
// every CTA of the cluster runs before any shared memory of it is written;
// after the last barrier no CTA touches another's shared memory.
constexpr int kClusterThreads = 1024;  // threads per CTA: 512 or 1024 (template NT)
constexpr int kClusterMax = 16;
constexpr int kClusterSmemMax = 200 * 1024;
constexpr int kClusterRowsMax = kClusterThreads;  // rows per CTA: at most one row per thread
constexpr int kKeyRowBits = 27;                   // 32-bit pivot key: valuation << 27 | row
constexpr uint32_t kKeyRowMask = (1u << kKeyRowBits) - 1u;

// column stride of the column-major slice: odd, so a warp storing one row's
// consecutive columns hits 32 different banks
__host__ __device__ constexpr int cluster_stride(int rows) { return rows | 1; }

__host__ __device__ constexpr size_t cluster_smem_bytes(int rows, int bw) {
    return sizeof(uint32_t) * static_cast<size_t>(cluster_stride(rows)) * bw + static_cast<size_t>(rows) + 16;
}

__device__ __forceinline__ void cluster_barrier_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ uint32_t pivot_key32(uint32_t x, int row, const Ring& R) {
    if (x == 0) return kNoKey32;
    const uint32_t v = R.k == 1 ? 0u : R.max_v == 0 ? (x % R.ell == 0 ? 1u : 0u) : valuation(x, R, R.max_v);
    if (v > R.max_v) return kNoKey32;
    return (v << kKeyRowBits) | static_cast<uint32_t>(row);
}

// The scale tables of a fraction-free factorization with k pivots, raw pivots
// s_w[0..k): s_inv[t] = w_t^-1 and s_sinv[t] = S_t^-1 = prod_{s<t} (w_s rho)^-1
// for t <= kMaxPanel (rho = 2^-32 for the Montgomery forms, else 1).  Called by
// every thread of the CTA; ends with a CTA barrier.
template <int ARITH>
__device__ void ff_scale_tables(int k, const uint32_t* s_w, uint32_t* s_inv, uint32_t* s_sinv, const Ring& R) {
    const int lane = threadIdx.x & 31;
    for (int t = threadIdx.x; t < k; t += blockDim.x) s_inv[t] = unit_inverse(s_w[t], R);
    __syncthreads();
    if (threadIdx.x < 32) {
        const uint32_t q = R.q;
        const uint64_t bm = R.barrett;
        const uint32_t one = 1u % q;
        // rho^-1 = 2^32 mod q (Montgomery) or 1
        const uint32_t rinv = ARITH == kArithPow2 ? one : mont_mul(R.mont_r2, 1u, q, R.mont_qinv);
        uint32_t f[kMaxPanel / 32];
        uint32_t run = one;
#pragma unroll
        for (int e = 0; e < kMaxPanel / 32; ++e) {
            const int t = lane * (kMaxPanel / 32) + e;
            f[e] = t < k ? mod_mul(s_inv[t], rinv, q, bm) : one;
            run = mod_mul(run, f[e], q, bm);
        }
        // inclusive scan of the lane products, then exclusive per element
        uint32_t incl = run;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl = mod_mul(incl, y, q, bm);
        }
        uint32_t ex = __shfl_up_sync(0xffffffffu, incl, 1);
        if (lane == 0) ex = one;
#pragma unroll
        for (int e = 0; e < kMaxPanel / 32; ++e) {
            s_sinv[lane * (kMaxPanel / 32) + e] = ex;
            ex = mod_mul(ex, f[e], q, bm);
        }
        if (lane == 31) s_sinv[kMaxPanel] = ex;
    }
    __syncthreads();
}

template <int ARITH, int NT>
__global__ void __launch_bounds__(NT, 1) panel_cluster_kernel(const PanelArgs a) {
    extern __shared__ __align__(16) uint32_t s_dyn[];
    __shared__ uint32_t r_key[2][kClusterMax];               // pushed keys, by parity and sender
    __shared__ uint32_t r_row[2][kClusterMax][kMaxPanel];     // pushed candidate rows (from column c)
    __shared__ uint32_t r_any[2][kClusterMax];                // pushed: the sender's active rows may have a pivot
    __shared__ uint32_t s_cand[2];                            // this CTA's best key, by parity
    __shared__ uint32_t s_w[kMaxPanel];                       // unit part of each step's raw pivot
    __shared__ uint32_t s_inv[kMaxPanel];                     // its inverse
    __shared__ uint32_t s_sinv[kMaxPanel + 1];                // S_t^-1
    __shared__ int s_colstep[kMaxPanel];                      // step t of pivot column c0 + j; else -1 - pivots left of it
    __shared__ int s_skip[kMaxPanel];                         // keep mode: the pivotless columns so far

    // settled by the top-block path: the same in every CTA, before any cluster barrier
    if (a.skip != nullptr && *a.skip != 0) return;
    const uint32_t crank = cluster_ctarank(), csize = cluster_nctarank();
    const int rows = a.m - a.r0;
    const int rpc = (rows + static_cast<int>(csize) - 1) / static_cast<int>(csize);
    const int row_begin = a.r0 + static_cast<int>(crank) * rpc;
    const int nloc = max(0, min(a.m, row_begin + rpc) - row_begin);
    if (rpc > NT) {  // the host never launches this; the test is the same in every CTA, before any barrier
        if (crank == 0 && threadIdx.x == 0) atomicCAS(a.err, 0, DERR_LAUNCH_SHAPE);
        return;
    }
    const int bw = a.bw, rs = cluster_stride(rpc);
    uint32_t* S = s_dyn;                                                           // [bw][rs]
    unsigned char* s_step = reinterpret_cast<unsigned char*>(S + static_cast<size_t>(bw) * rs);  // [rpc]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int nwarps = NT / 32;
    // thread -> (row li, phase sub): consecutive threads take consecutive rows,
    // so a warp reads one column of consecutive rows; g threads share a row
    int lg = 0;
    while ((1 << lg) < nloc) ++lg;
    const int nslots = 1 << lg, g = NT >> lg;
    const int li = tid & (nslots - 1), sub = tid >> lg;
    const bool has_row = li < nloc;

    for (int r = warp; r < nloc; r += nwarps) {
        const uint32_t* src = a.A + static_cast<size_t>(row_begin + r) * a.ld + a.c0;
        for (int j = lane; j < bw; j += 32) S[j * rs + r] = src[j];
    }
    for (int i = tid; i < rpc; i += NT) s_step[i] = 0;
    for (int j = tid; j < bw; j += NT) s_colstep[j] = -1;
    if (tid == 0) s_cand[0] = s_cand[1] = kNoKey32;
    __syncthreads();
    {
        uint32_t key = kNoKey32;
        if (has_row && sub == 0) key = pivot_key32(S[li], row_begin + li, a.R);
        key = __reduce_min_sync(0xffffffffu, key);
        if (lane == 0 && key != kNoKey32) atomicMin(&s_cand[0], key);
    }
    // every CTA of the cluster runs (its shared memory may be written) and s_cand[0] is complete
    cluster_barrier_all();

    const uint32_t rkey_addr = smem_u32(&r_key[0][0]);
    const uint32_t rrow_addr = smem_u32(&r_row[0][0][0]);
    const uint32_t rany_addr = smem_u32(&r_any[0][0]);
    int k = 0;
    int nskip = 0;  // pivotless columns so far (keep mode)
    int empty = 0;  // pivotless columns in a row; at the 2nd, 6th, 14th, .. the rest of the panel is looked over
    int look = 2;
    uint32_t any = 1;  // this CTA's active rows are not known to have no pivot in the rest of the panel
    int pend_col = -1;  // ring mode: multiplier x / ell^v stored after the column's CTA barrier
    uint32_t pend_xp = 0;
    for (int it = 0; it < bw; ++it) {
        const int par = it & 1;
        if (pend_col >= 0) {
            S[pend_col * rs + li] = pend_xp;
            pend_col = -1;
        }
        // (1) push this CTA's candidate for column c0 + it to every CTA (itself included)
        {
            const uint32_t mine = s_cand[par];
            if (warp < static_cast<int>(csize)) {
                const uint32_t d = static_cast<uint32_t>(warp);
                const uint32_t slot = par * kClusterMax + crank;
                if (lane == 0) {
                    st_dsmem_u32(dsmem_addr(rkey_addr + 4u * slot, d), mine);
                    st_dsmem_u32(dsmem_addr(rany_addr + 4u * slot, d), any);
                }
                if (mine != kNoKey32) {
                    const int lm = static_cast<int>(mine & kKeyRowMask) - row_begin;
                    const uint32_t dst = dsmem_addr(rrow_addr + 4u * slot * kMaxPanel, d);
                    for (int j = lane; j < bw - it; j += 32) st_dsmem_u32(dst + 4u * j, S[(it + j) * rs + lm]);
                    // keep mode: the row's entries of the pivotless columns behind them (they are left of it)
                    for (int j = lane; j < nskip; j += 32) st_dsmem_u32(dst + 4u * (bw - it + j), S[s_skip[j] * rs + lm]);
                }
            }
            if (tid == 0) s_cand[par ^ 1] = kNoKey32;  // collects column it + 1's candidate below
        }
        // (2) every push of this column lands before any CTA reads its slots
        cluster_barrier_all();
        // (3) the pivot: the smallest (valuation, row) key of the cluster
        const uint32_t kd = lane < static_cast<int>(csize) ? r_key[par][lane] : kNoKey32;
        const uint32_t pkey = __reduce_min_sync(0xffffffffu, kd);
        uint32_t key = kNoKey32;
        if (pkey == kNoKey32) {
            // no pivot in this column: every active row is unchanged; scan column it + 1
            if (!__any_sync(0xffffffffu, lane < static_cast<int>(csize) && r_any[par][lane] != 0)) {
                // no active row has a pivot from here on (the same verdict in every CTA)
                for (int j = it + tid; j < bw; j += NT) s_colstep[j] = -1 - k;
                break;
            }
            if (tid == 0) {
                s_colstep[it] = -1 - k;
                if (a.keep) s_skip[nskip] = it;  // read after this column's CTA barrier
            }
            if (a.keep) ++nskip;
            ++empty;
            if (it + 1 < bw && has_row && sub == 0 && s_step[li] == 0)
                key = pivot_key32(S[(it + 1) * rs + li], row_begin + li, a.R);
        } else {
            empty = 0;
            look = 2;
            const int owner = __ffs(__ballot_sync(0xffffffffu, kd == pkey)) - 1;
            const int prow = static_cast<int>(pkey & kKeyRowMask);
            const uint32_t v = pkey >> kKeyRowBits;
            const uint32_t* prv = r_row[par][owner];  // pivot row, column c0 + it at index 0
            const uint32_t w = div_pw(prv[0], v, a.R);
            const int oli = owner == static_cast<int>(crank) ? prow - row_begin : -1;
            if (tid == 0) {
                s_w[k] = w;
                s_colstep[it] = k;
                if (oli >= 0) s_step[oli] = static_cast<unsigned char>(k + 1);
                if (crank == 0) {
                    a.pivot_rows[k] = prow;
                    a.pivot_cols[k] = a.c0 + it;
                }
            }
            if (has_row && li != oli && s_step[li] == 0) {
                const uint32_t xp = div_pw(S[it * rs + li], v, a.R);
                const uint32_t xn = ff_negate<ARITH>(xp, a.R);
                int j = it + 1 + sub;
                uint32_t* sp = S + j * rs + li;
                const uint32_t* pp = prv + (j - it);
                const int sstep = g * rs;
                if (sub == 0 && j < bw) {  // column it + 1: the next column's candidate
                    const uint32_t y = ff_update<ARITH>(w, *sp, xn, *pp, a.R);
                    *sp = y;
                    key = pivot_key32(y, row_begin + li, a.R);
                    j += g;
                    sp += sstep;
                    pp += g;
                }
                for (; j + g < bw; j += 2 * g, sp += 2 * sstep, pp += 2 * g) {
                    const uint32_t y0 = ff_update<ARITH>(w, sp[0], xn, pp[0], a.R);
                    const uint32_t y1 = ff_update<ARITH>(w, sp[sstep], xn, pp[g], a.R);
                    sp[0] = y0;
                    sp[sstep] = y1;
                }
                if (j < bw) *sp = ff_update<ARITH>(w, *sp, xn, *pp, a.R);
                for (int u = sub; u < nskip; u += g) {
                    uint32_t* sk = S + s_skip[u] * rs + li;
                    *sk = ff_update<ARITH>(w, *sk, xn, prv[bw - it + u], a.R);
                }
                if (v != 0 && sub == 0) {
                    pend_col = it;
                    pend_xp = xp;
                }
            }
            ++k;
        }
        key = __reduce_min_sync(0xffffffffu, key);
        if (lane == 0 && key != kNoKey32) atomicMin(&s_cand[par ^ 1], key);
        if (empty == look) {  // the same in every thread of the cluster
            look = 2 * look + 2;
            // (entries that cannot be pivots stay so while there is none: over a ring with unit pivots
            // the rest of a level is seldom zero)
            bool x = false;
            if (has_row && s_step[li] == 0)
                for (int j = it + 1 + sub; j < bw; j += g) x |= pivot_key32(S[j * rs + li], 0, a.R) != kNoKey32;
            any = __syncthreads_or(x) ? 1u : 0u;
        } else {
            any = 1;
            __syncthreads();
        }
    }
    if (pend_col >= 0) S[pend_col * rs + li] = pend_xp;

    // ---- back to the classical values: w_t^-1 and S_t^-1 = prod_{s<t} w_s^-1 rho^-1
    ff_scale_tables<ARITH>(k, s_w, s_inv, s_sinv, a.R);
    if (has_row) {
        const int st = s_step[li];
        const int tau = st ? st - 1 : k;  // the step that froze this row's scale
        const uint32_t sc = s_sinv[tau];
        for (int j = sub; j < bw; j += g) {
            // a multiplier of step t < tau: times w_t^-1; any other entry was last
            // scaled by the step before min(tau, pivots left of column j)
            const int t = s_colstep[j];
            // (in keep mode pivotless columns take every step's scale)
            const uint32_t f = t >= 0 ? (t < tau ? s_inv[t] : sc) : s_sinv[a.keep ? tau : min(tau, -1 - t)];
            S[j * rs + li] = mod_mul(S[j * rs + li], f, a.R.q, a.R.barrett);
        }
    }
    __syncthreads();
    for (int r = warp; r < nloc; r += nwarps) {
        uint32_t* dst = a.A + static_cast<size_t>(row_begin + r) * a.ld + a.c0;
        for (int j = lane; j < bw; j += 32) dst[j] = S[j * rs + r];
    }
    if (crank == 0 && tid == 0) *a.k_out = k;
}

// ---- the top-block path -----------------------------------------------------------
// A panel's pivots can be taken from its top rows alone whenever they supply
// one for every column: a non-zero (over Z/ell^k a unit) entry of the Schur
// complement is a valid pivot of its column wherever it lies, and the column
// rank profile, the RREF and the Howell and Smith forms do not depend on the
// rows chosen.  So one CTA eliminates the top nbr x w block (nbr a little more
// than w where a column of a w-row block is likely to run out of units, so that
// even F_2 panels practically always succeed), picking the topmost unit of each
// column; with the nb = min(w, rows) pivot rows moved to the top, B the block
// of their panel columns, the rest of the elimination step is one product:
//   [A12; A22] += [B^-1 - I; -A21 B^-1] A12
// gives B^-1 A12 in the top rows (whose panel columns become the identity) and
// the Schur complement A22 - A21 B^-1 A12 below (nb = w whenever rows remain
// below).  When a column has no unit in the block, nothing is written and the
// searching kernel factors the panel.
// The padded size of an n x n triangular inverse: a power of two >= 8.
__host__ __device__ constexpr int tri_pad(int n) {
    int p = 8;
    while (p < n) p *= 2;
    return p;
}
__host__ __device__ constexpr int tri_stride(int p) { return p + 4; }  // rows 16-byte aligned
constexpr int tri_words(int p) { return p * tri_stride(p); }

// In place, X_i <- X_i^-1 mod q for `nmat` unit lower triangular P x P matrices
// in shared memory (P a power of two >= 8, matrix i at X + i * mstride, row
// stride tri_stride(P), zeros above the diagonal, identity padding).  8 x 8
// diagonal blocks by forward substitution (a thread per column), then doubling:
//   [A 0; C B]^-1 = [A^-1 0; -B^-1 (C A^-1) B^-1],
// every entry an exact 96-bit dot product reduced once, so the chain is
// 8 + 2 log2(P/8) dependent dot products instead of P elimination steps.
// tmp: nmat * P * P / 4 words.  Called by every thread of the CTA; ends with a
// barrier.
__device__ __forceinline__ uint32_t reduce96(uint32_t a0, uint32_t a1, uint32_t a2, uint32_t q, uint64_t barrett) {
    const uint32_t h = reduce_u64((static_cast<uint64_t>(a2) << 32) | a1, q, barrett);
    return reduce_u64((static_cast<uint64_t>(h) << 32) | a0, q, barrett);
}

__device__ void unit_lower_inverse(uint32_t* X, int P, int nmat, int mstride, uint32_t* tmp, uint32_t q,
                                   uint64_t barrett) {
    const int ls = tri_stride(P);
    for (int base = 0; base < nmat * P; base += blockDim.x) {
        const int idx = base + threadIdx.x;
        const bool valid = idx < nmat * P;
        const int mi = valid ? idx / P : 0, c = valid ? idx - mi * P : 0, cc = c & 7;
        uint32_t* M = X + mi * mstride + (c - cc) * (ls + 1);
        uint32_t x[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            uint32_t a0 = 0, a1 = 0, a2 = 0;
#pragma unroll
            for (int s = 0; s < r; ++s) mac96(a0, a1, a2, M[r * ls + s], x[s]);
            const uint32_t v = reduce96(a0, a1, a2, q, barrett);
            x[r] = r == cc ? 1u : v == 0 || r < cc ? 0u : q - v;
        }
        __syncwarp();  // the eight columns of a block belong to eight lanes of one warp: all have read it
#pragma unroll
        for (int r = 0; r < 8; ++r)
            if (valid && r >= cc) M[r * ls + cc] = x[r];
    }
    __syncthreads();
    for (int h = 8; h < P; h *= 2) {
        const int lh = __ffs(h) - 1, pairs = P >> (lh + 1);
        const int total = nmat * pairs * h * h;
        // tmp = C A^-1
        for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
            const int c = idx & (h - 1), r = (idx >> lh) & (h - 1), pr = idx >> (2 * lh);
            const int mi = pr / pairs, b0 = (pr - mi * pairs) * 2 * h;
            const uint32_t* Ai = X + mi * mstride + b0 * ls + b0;
            const uint32_t* Cr = Ai + (h + r) * ls;
            const uint32_t* Ac = Ai + c;
            uint32_t a0 = 0, a1 = 0, a2 = 0;
#pragma unroll 4
            for (int s = 0; s < h; ++s) mac96(a0, a1, a2, Cr[s], Ac[s * ls]);
            tmp[idx] = reduce96(a0, a1, a2, q, barrett);
        }
        __syncthreads();
        // C = -B^-1 tmp
        for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
            const int c = idx & (h - 1), r = (idx >> lh) & (h - 1), pr = idx >> (2 * lh);
            const int mi = pr / pairs, b0 = (pr - mi * pairs) * 2 * h;
            uint32_t* A0 = X + mi * mstride + b0 * ls + b0;
            const uint32_t* Bi = A0 + (h + r) * ls + h;
            const uint32_t* tp = tmp + (pr << (2 * lh)) + c;
            uint32_t a0 = 0, a1 = 0, a2 = 0;
#pragma unroll 4
            for (int s = 0; s < h; ++s) mac96(a0, a1, a2, Bi[s], tp[s << lh]);
            const uint32_t v = reduce96(a0, a1, a2, q, barrett);
            A0[(h + r) * ls + c] = v == 0 ? 0u : q - v;
        }
        __syncthreads();
    }
}

// Work may be queued behind a panel before its outcome is known: *fail takes the
// panel's number when the host must look at the panel (no pivot somewhere; with
// in_order, pivot rows that have to move); a panel launched after that does
// nothing.
struct BlockQueue {
    int* fail;
    int seq;
    int in_order;
    const int* err;   // the context's error word
    int* err_out;     // its value at the panel's end
};

template <int ARITH, int RS>
__global__ void __launch_bounds__(4 * RS) panel_block_kernel(const BlockArgs a, const BlockQueue q) {
    extern __shared__ __align__(16) uint32_t s_blk[];
    if (*q.fail != 0) return;
    bool look = !block_inverse<ARITH, RS>(a, s_blk);
    if (!look && q.in_order) {
        __syncthreads();  // the pivot rows are written
        const int t = threadIdx.x;
        look = __syncthreads_or(t < min(a.w, a.m - a.r0) && a.pivot_rows[t] != a.r0 + t);
    }
    if (threadIdx.x == 0) {
        if (look) *q.fail = q.seq;
        *q.err_out = *q.err;
    }
}

// ---- panels with few non-zero rows ----------------------------------------------------
// Sparse matrices (boundary-like blocks, U D V products close to diagonal) have
// panels in which most active rows are zero.  Zero rows never pivot and are
// never updated, so the search runs on the others alone: panel_rows_kernel
// lists them (and clears the update's left factor W), and when there are at
// most kCompactMost of them panel_compact_kernel factors them in one CTA, where
// a column costs one CTA barrier instead of the cluster's exchange.  It keeps
// every row operation's effect on the identity as well (in place: the pivot's
// column of a row holds that row's entry of the inverse of the operations), so W
// comes out directly, with no triangular inverse and no panel_w_kernel.
constexpr int kCompactRows = 256;
// More listed rows than two a column meet in most columns, and one CTA updates them
// all in every step: 26 panels of a banded 3000 x 2000 matrix mod 65521 (200 wide, 4
// entries a row) with up to 256 listed rows took 196 us each, against 104 us in
// the cluster search and 20 us for L11^-1 and W; the RREF 8.1 ms with up to 256
// rows, 6.35 ms with 128, 6.9 ms by searches alone.  An argument of the kernel: with
// the limit compiled in, its steps come out slower (a panel of the 2048 x 2048 U D V
// over Z/3^10 44 us against 37.5).
// Modulo powers of 2, where an update is two products without a reduction, all 256 pay:
// 2000 x 2000 mod 2 in 20 dense diagonal blocks 4.24 ms with 256 rows and 4.67 with 128.
constexpr int kCompactMost = 128, kCompactMostPow2 = 256;

struct CompactArgs {
    uint32_t* A;
    uint64_t ld;
    int m, r0, c0, w;
    Ring R;
    int most;         // listed rows to take, at most kCompactRows
    int* list;        // [kCompactRows] rows with a non-zero entry in the panel, in any order
    int* count;       // their number (counted on beyond the list); 0 between panels
    int after_block;  // the top block was tried before: nothing to do when it settled the panel
    int* ok;          // out: 2 when the panel was factored here, else 0 (left alone when the block settled it)
    int* pivot_rows;  // [w] out
    int* pivot_cols;  // [w] out
    int* k_out;       // out
    uint32_t* W;      // out: (m - r0) x w, row stride ldw, rows in their places after the pivot rows' moves
    int ldw;
};

__global__ void __launch_bounds__(256) panel_rows_kernel(const CompactArgs a) {
    if (a.after_block && *a.ok != 0) return;
    const int lane = threadIdx.x & 31, row = a.r0 + static_cast<int>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    if (row >= a.m) return;
    const uint32_t* src = a.A + static_cast<size_t>(row) * a.ld + a.c0;
    uint32_t* dst = a.W + static_cast<size_t>(row - a.r0) * a.ldw;
    uint32_t any = 0;
#pragma unroll
    for (int c = 0; c < kMaxPanel / 32; ++c)
        if (lane + 32 * c < a.w) {
            any |= src[lane + 32 * c];
            dst[lane + 32 * c] = 0u;
        }
    if (__any_sync(0xffffffffu, any != 0) && lane == 0) {
        const int at = atomicAdd(a.count, 1);
        if (at < kCompactRows) a.list[at] = row;
    }
}

__host__ __device__ constexpr size_t compact_smem_bytes(int w) {
    return sizeof(uint32_t) * static_cast<size_t>(w) * (kCompactRows + 1);
}

// One CTA of 32 warps.  The rows, in row order, sit in shared memory
// column-major, lanes over rows: rwn = 1, 2, 4 or 8 warps cover them and 32 /
// rwn groups of warps share the columns.  Pivot rule and fraction-free update
// are the cluster kernel's, but a step whose column has no other entry updates
// nothing (and no scale), and every column is updated, pivotless ones left of
// the pivot too, the pivot's own becoming the inverse's column.
// A 64-column panel of a 2048 x 2048 U D V over Z/2^16: 41 us and 2 us for the
// list, against 98 us for the cluster search and 21 us for L11^-1 and W.
template <int ARITH>
__global__ void __launch_bounds__(1024, 1) panel_compact_kernel(const CompactArgs a) {
    extern __shared__ __align__(16) uint32_t s_cmp[];
    __shared__ uint32_t s_x[2][kCompactRows];
    __shared__ uint32_t s_key[2][kCompactRows / 32];
    __shared__ int s_nz[2][kCompactRows / 32];
    __shared__ uint32_t s_S[kMaxPanel + 1], s_Sinv[kMaxPanel + 1];
    __shared__ int s_prow[kMaxPanel], s_pcol[kMaxPanel], s_colpiv[kMaxPanel];
    __shared__ int s_row[kCompactRows], s_step[kCompactRows];
    __shared__ int s_raw[kCompactRows];
    __shared__ unsigned char s_isp[kMaxPanel];
    __shared__ int s_vac[kMaxPanel];
    __shared__ int s_cnt;
    if (a.after_block && *a.ok != 0) return;
    const Ring& R = a.R;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, w = a.w;
    if (tid == 0) {
        s_cnt = *a.count;
        *a.count = 0;
    }
    __syncthreads();
    const int cnt = s_cnt;
    if (cnt > min(a.most, kCompactRows)) {
        if (tid == 0) *a.ok = 0;
        return;
    }
    // the list in row order (ranks by counting)
    if (tid < cnt) s_raw[tid] = a.list[tid];
    if (tid < kMaxPanel) s_colpiv[tid] = -1;
    __syncthreads();
    if (tid < cnt) {
        const int mine = s_raw[tid];
        int rank = 0;
        for (int u = 0; u < cnt; ++u) rank += s_raw[u] < mine ? 1 : 0;
        s_row[rank] = mine;
        s_step[tid] = 0;
    }
    __syncthreads();
    const int rwn = cnt <= 32 ? 1 : cnt <= 64 ? 2 : cnt <= 128 ? 4 : 8;
    const int G = 32 / rwn, rs = 32 * rwn + 1;
    uint32_t* S = s_cmp;  // [w][rs]
#pragma unroll 4
    for (int r = warp; r < cnt; r += 32) {
        const uint32_t* src = a.A + static_cast<size_t>(s_row[r]) * a.ld + a.c0;
#pragma unroll
        for (int c = 0; c < kMaxPanel / 32; ++c)
            if (lane + 32 * c < w) S[(lane + 32 * c) * rs + r] = src[lane + 32 * c];
    }
    __syncthreads();
    const int rwi = warp & (rwn - 1), g = warp / rwn, li = 32 * rwi + lane;
    bool active = li < cnt;  // in the list and not a pivot row yet
    uint32_t* col = S + li;
    // column c's entries, smallest (valuation, slot) and non-zeros of the active rows, for step c
    auto publish = [&](int c) {
        const uint32_t x = active ? col[c * rs] : 0u;
        uint32_t key = kNoKey32;
        if (x != 0) {
            const uint32_t v = R.k == 1 ? 0u : R.max_v == 0 ? (x % R.ell == 0 ? 1u : 0u) : valuation(x, R, R.max_v);
            if (v <= R.max_v) key = (v << 16) | static_cast<uint32_t>(li);
        }
        key = __reduce_min_sync(0xffffffffu, key);
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
        uint32_t pk = s_key[par][0];
        int nz = s_nz[par][0];
        for (int u = 1; u < rwn; ++u) {
            pk = min(pk, s_key[par][u]);
            nz += s_nz[par][u];
        }
        if (pk != kNoKey32) {
            const int prow = static_cast<int>(pk & 0xffffu);
            const uint32_t v = pk >> 16;
            const uint32_t wt = div_pw(s_x[par][prow], v, R);
            if (tid == 0) {
                s_S[k] = scale;
                s_prow[k] = prow;
                s_pcol[k] = it;
                s_colpiv[it] = k;
                s_step[prow] = k + 1;
            }
            if (li == prow) active = false;
            if (nz > 1) {
                if (active) {
                    const uint32_t xn = ff_negate<ARITH>(div_pw(s_x[par][li], v, R), R);
                    const uint32_t* pr = S + prow;
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
    // the rows' scales: row of pivot t by S_t, the others by the last
    if (tid == 0) s_S[k] = scale;
    __syncthreads();
    if (tid <= k) s_Sinv[tid] = unit_inverse(s_S[tid], R);
    // the rows' places after the moves (as move_pivot_rows_kernel makes them)
    if (tid < kMaxPanel) s_isp[tid] = 0;
    __syncthreads();
    if (tid < k && s_row[s_prow[tid]] - a.r0 < k) s_isp[s_row[s_prow[tid]] - a.r0] = 1;
    if (tid == 0) {
        int nv = 0;
        for (int t = 0; t < k; ++t)
            if (s_row[s_prow[t]] - a.r0 >= k) s_vac[nv++] = s_row[s_prow[t]] - a.r0;
    }
    __syncthreads();
    for (int r = warp; r < cnt; r += 32) {
        const int st = s_step[r], tau = st ? st - 1 : k;
        const uint32_t sc = s_Sinv[tau];
        int pos = st ? st - 1 : s_row[r] - a.r0;
        if (!st && pos < k) {
            int rank = 0;
            for (int i = lane; i < pos; i += 32) rank += s_isp[i] ? 0 : 1;
            pos = s_vac[__reduce_add_sync(0xffffffffu, rank)];
        }
        uint32_t* dst = a.A + static_cast<size_t>(s_row[r]) * a.ld + a.c0;
        uint32_t* wd = a.W + static_cast<size_t>(pos) * a.ldw;
        for (int j = lane; j < w; j += 32) {
            const uint32_t val = mod_mul(S[j * rs + r], sc, R.q, R.barrett);
            const int t = s_colpiv[j];
            const bool done = t >= 0 && t < tau;  // eliminated from this row: its entry is the inverse's
            dst[j] = done ? 0u : val;
            if (done) wd[t] = val;
        }
    }
    if (tid < k) {
        a.pivot_rows[tid] = s_row[s_prow[tid]];
        a.pivot_cols[tid] = a.c0 + s_pcol[tid];
    }
    if (tid == 0) {
        *a.k_out = k;
        *a.ok = 2;
    }
}

// Columns [c0, c0 + w) without pivots (pcols[0 .. k) has them) of rows [row0,
// row0 + rows) to columns dst, dst + 1, .. of the same rows: a warp per row.
__global__ void __launch_bounds__(256) append_cols_kernel(uint32_t* __restrict__ A, uint64_t ld, int row0, int rows,
                                                          int c0, int w, const int* __restrict__ pcols, int k,
                                                          int dst) {
    __shared__ int s_at[kMaxPanel];
    for (int j = threadIdx.x; j < w; j += 256) {
        int at = j;  // minus the pivot columns before it; -1 for a pivot column
        for (int t = 0; t < k; ++t) {
            const int c = pcols[t] - c0;
            if (c == j) at = INT_MIN / 2;
            else if (c < j) --at;
        }
        s_at[j] = at;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int i = static_cast<int>(blockIdx.x) * 8 + (threadIdx.x >> 5); i < rows; i += static_cast<int>(gridDim.x) * 8) {
        uint32_t* row = A + static_cast<size_t>(row0 + i) * ld;
        for (int j = lane; j < w; j += 32)
            if (s_at[j] >= 0) row[dst + s_at[j]] = row[c0 + j];
    }
}

// After a searched panel (its packed LU in place, the pivot rows moved to r0 ..
// r0 + k - 1): L11^-1 of the k pivot rows at the pivot columns, the factor the
// update takes in place of the top block's.
__global__ void __launch_bounds__(512) panel_linv_kernel(const uint32_t* __restrict__ A, uint64_t ld, int r0,
                                                         const int* __restrict__ pcols, int k, uint32_t q,
                                                         uint64_t barrett, uint32_t* __restrict__ linv) {
    extern __shared__ __align__(16) uint32_t s_li[];
    const int P = tri_pad(k), ls = tri_stride(P), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int s = lane; s < P; s += 32) {
        const int pc = s < k ? pcols[s] : 0;
#pragma unroll 8
        for (int t = warp; t < P; t += 16)
            s_li[t * ls + s] = t == s ? 1u : t < k && s < t ? A[static_cast<size_t>(r0 + t) * ld + pc] : 0u;
    }
    __syncthreads();
    unit_lower_inverse(s_li, P, 1, 0, s_li + tri_words(P), q, barrett);
    for (int idx = threadIdx.x; idx < k * k; idx += blockDim.x) {
        const int t = idx / k, s = idx - t * k;
        linv[idx] = s_li[t * ls + s];
    }
}
size_t linv_smem_bytes(int k) {
    const size_t p = tri_pad(k);
    return sizeof(uint32_t) * (tri_words(tri_pad(k)) + p * p / 4);
}

// The left factor of the fused update, W ((m - r0) x nb, row-major, ld nb):
// rows t < nb are M - I; a row x below becomes -x M, x = the row's entries at
// the pivot columns: untouched values and M = B^-1 after the top block,
// multipliers L21 and M = L11^-1 after a searched panel.  A warp takes four rows at
// once, lanes over output columns; each dot product runs exactly in a 96-bit
// carry chain (nb <= 128 products below 2^64) and is reduced once; SMALL: nb (q - 1)^2
// below 2^32, the sum in one word (a wide product takes the multiplier four times as
// long): 64 columns of 10515 x 8668 mod 13 12.8 -> 8.1 us a panel.
constexpr int kWRows = 32;
constexpr int kWRowsPerWarp = 4;

template <int WMAX, bool SMALL>
__global__ void __launch_bounds__(256) panel_w_kernel(const uint32_t* __restrict__ A, uint64_t ld, int r0, int m,
                                                      const int* __restrict__ pcols, int nb, const uint32_t* __restrict__ binv, uint32_t q,
                                                      uint64_t barrett, const Skip skip,
                                                      uint32_t* __restrict__ W) {
    if (skip.stands()) return;
    extern __shared__ __align__(16) uint32_t s_wk[];
    const int rb = r0 + static_cast<int>(blockIdx.x) * kWRows;  // first row of this CTA
    const int nr = min(kWRows, m - rb);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NW = 256 / 32;
    static_assert(NW * kWRowsPerWarp == kWRows, "one pass of the warps covers the CTA's rows");
    constexpr int CS = WMAX / 32;
    // the top rows: M - I
    for (int r = warp; r < nr; r += NW) {
        const int row = rb + r;
        if (row >= r0 + nb) break;
        for (int j = lane; j < nb; j += 32) {
            const size_t idx = static_cast<size_t>(row - r0) * nb + j;
            W[idx] = j == row - r0 ? mod_sub(binv[idx], 1u, q) : binv[idx];
        }
    }
    if (rb + nr <= r0 + nb) return;  // no row below the block in this CTA (uniform)
    uint32_t* Bi = s_wk;                                   // [nb][nb]
    const int xs = (nb + 3) & ~3;                          // row stride of Xr: whole 16-byte pieces
    uint32_t* Xr = s_wk + ((static_cast<size_t>(nb) * nb + 3) & ~size_t(3));  // [kWRows][xs]
    {
        // B^-1 in 16-byte pieces (its buffer is 16-byte aligned), four loads of a thread in flight
        const int n4 = (nb * nb) >> 2;
        const uint4* b4 = reinterpret_cast<const uint4*>(binv);
        uint4* d4 = reinterpret_cast<uint4*>(Bi);
        for (int base = 0; base < n4; base += 256 * 4) {
            uint4 v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int idx = base + tid + 256 * e;
                if (idx < n4) v[e] = b4[idx];
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int idx = base + tid + 256 * e;
                if (idx < n4) d4[idx] = v[e];
            }
        }
        for (int idx = 4 * n4 + tid; idx < nb * nb; idx += 256) Bi[idx] = binv[idx];
    }
    const int rl = warp * kWRowsPerWarp;  // this warp's rows: rl .. rl + 3 of the CTA
    {
        uint32_t v[kWRowsPerWarp][CS];
        int pc[CS];
#pragma unroll
        for (int c = 0; c < CS; ++c) pc[c] = lane + 32 * c < nb ? pcols[lane + 32 * c] : 0;
#pragma unroll
        for (int i = 0; i < kWRowsPerWarp; ++i) {
            const int row = rb + rl + i;
            const bool below = rl + i < nr && row >= r0 + nb;
            const uint32_t* src = A + static_cast<size_t>(below ? row : r0) * ld;
#pragma unroll
            for (int c = 0; c < CS; ++c) v[i][c] = below && lane + 32 * c < nb ? src[pc[c]] : 0u;
        }
#pragma unroll
        for (int i = 0; i < kWRowsPerWarp; ++i)
#pragma unroll
            for (int c = 0; c < CS; ++c) {
                const int j = lane + 32 * c;
                if (j < nb) Xr[(rl + i) * xs + j] = v[i][c];
            }
    }
    __syncthreads();
    uint32_t a0[kWRowsPerWarp][CS], a1[kWRowsPerWarp][CS], a2[kWRowsPerWarp][CS];
#pragma unroll
    for (int i = 0; i < kWRowsPerWarp; ++i)
#pragma unroll
        for (int c = 0; c < CS; ++c) a0[i][c] = a1[i][c] = a2[i][c] = 0;
    for (int t = 0; t < nb; ++t) {
        uint32_t bt[CS];
#pragma unroll
        for (int c = 0; c < CS; ++c) {
            const int j = lane + 32 * c;
            bt[c] = j < nb ? Bi[t * nb + j] : 0u;
        }
#pragma unroll
        for (int i = 0; i < kWRowsPerWarp; ++i) {
            const uint32_t x = Xr[(rl + i) * xs + t];
#pragma unroll
            for (int c = 0; c < CS; ++c) {
                if constexpr (SMALL) a0[i][c] += x * bt[c];
                else mac96(a0[i][c], a1[i][c], a2[i][c], x, bt[c]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < kWRowsPerWarp; ++i) {
        const int row = rb + rl + i;
        if (rl + i >= nr || row < r0 + nb) continue;
        uint32_t* dst = W + static_cast<size_t>(row - r0) * nb;
#pragma unroll
        for (int c = 0; c < CS; ++c) {
            const int j = lane + 32 * c;
            if (j < nb) {
                const uint64_t h =
                    SMALL ? 0u : reduce_u64((static_cast<uint64_t>(a2[i][c]) << 32) | a1[i][c], q, barrett);
                const uint32_t v = static_cast<uint32_t>(reduce_u64((h << 32) | a0[i][c], q, barrett));
                dst[j] = v == 0 ? 0u : q - v;
            }
        }
    }
}

// ---- the pivot rows to the top -------------------------------------------------------
// In columns [ca, cb): row r0 + t becomes the pivot row prow[t], t < k, and the
// rows this displaces fill the pivot rows' old places below r0 + k in order, so
// at most 2 k rows move however tall the matrix is (permuting every active row
// took 33 of the 74 ms of a 10515 x 8668 RREF mod 13).  The order of the other
// rows does not show in any result (the determinant's sign follows the same
// moves, row_moves_odd).  One CTA per 32 columns: all reads before any write.
constexpr int kMoveCols = 32;

__global__ void __launch_bounds__(256) move_pivot_rows_kernel(uint32_t* __restrict__ A, uint64_t ld, int r0, int k,
                                                              const int* __restrict__ prow, int ca, int cb,
                                                              const Skip skip) {
    if (skip.stands()) return;
    __shared__ uint32_t buf[2 * kMaxPanel][kMoveCols];
    __shared__ int s_src[2 * kMaxPanel], s_dst[2 * kMaxPanel];
    __shared__ unsigned char s_isp[kMaxPanel];
    __shared__ int s_cnt[2][kMaxPanel / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int pr = tid < k ? prow[tid] : -1;
    if (tid < kMaxPanel) s_isp[tid] = 0;
    __syncthreads();
    if (tid < k && pr - r0 < k) s_isp[pr - r0] = 1;
    __syncthreads();
    const bool disp = tid < k && !s_isp[tid], vac = tid < k && pr - r0 >= k;
    const unsigned md = __ballot_sync(0xffffffffu, disp), mv = __ballot_sync(0xffffffffu, vac);
    if (lane == 0 && warp < kMaxPanel / 32) {
        s_cnt[0][warp] = __popc(md);
        s_cnt[1][warp] = __popc(mv);
    }
    __syncthreads();
    int nd = 0, d0 = 0, v0 = 0;
#pragma unroll
    for (int u = 0; u < kMaxPanel / 32; ++u) {
        nd += s_cnt[0][u];
        if (u < warp) {
            d0 += s_cnt[0][u];
            v0 += s_cnt[1][u];
        }
    }
    const unsigned below = (1u << lane) - 1u;
    if (tid < k) {
        s_src[tid] = pr;
        s_dst[tid] = r0 + tid;
    }
    if (disp) s_src[k + d0 + __popc(md & below)] = r0 + tid;
    if (vac) s_dst[k + v0 + __popc(mv & below)] = pr;
    __syncthreads();
    const int n = k + nd, col = ca + static_cast<int>(blockIdx.x) * kMoveCols + lane;
    if (col < cb) {
#pragma unroll 4
        for (int u = warp; u < n; u += 8)
            if (s_src[u] != s_dst[u]) buf[u][lane] = A[static_cast<size_t>(s_src[u]) * ld + col];
    }
    __syncthreads();
    if (col < cb) {
        for (int u = warp; u < n; u += 8)
            if (s_src[u] != s_dst[u]) A[static_cast<size_t>(s_dst[u]) * ld + col] = buf[u][lane];
    }
}

// Whether those row moves are an odd permutation (host): n minus the number of
// cycles over the k top places and the places vacated below them.
bool row_moves_odd(const int* prow, int k, int r0) {
    std::vector<int> src(k), vac;
    std::vector<char> isp(k, 0);
    for (int t = 0; t < k; ++t) {
        const int p = prow[t] - r0;
        if (p < k) {
            isp[p] = 1;
            src[t] = p;
        } else {
            src[t] = k + static_cast<int>(vac.size());
            vac.push_back(p);
        }
    }
    for (int i = 0; i < k; ++i)
        if (!isp[i]) src.push_back(i);  // the displaced rows, in the vacated places' order
    const int n = static_cast<int>(src.size());
    std::vector<char> seen(n, 0);
    int cycles = 0;
    for (int i = 0; i < n; ++i) {
        if (seen[i]) continue;
        ++cycles;
        for (int j = i; !seen[j]; j = src[j]) seen[j] = 1;
    }
    return ((n - cycles) & 1) != 0;
}

// flags |= 1 when the rows x cols window has a non-zero entry, |= 2 when one can be
// a pivot.  A warp that has seen both leaves as one; one store per warp and row, and
// none of a bit that is set (every thread storing its own took 33 us on 1024 x 1024
// non-zero entries).
__global__ void __launch_bounds__(256) window_look_kernel(const uint32_t* __restrict__ A, uint64_t ld, int rows,
                                                          int cols, const Ring R, int* __restrict__ flags) {
    const int lane = threadIdx.x & 31;
    for (int i = blockIdx.x; i < rows; i += gridDim.x) {
        const int seen = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile int*>(flags), 0);
        if (seen == 3) return;
        int f = 0;
        for (int j = threadIdx.x; j < cols; j += blockDim.x) {
            const uint32_t x = A[static_cast<size_t>(i) * ld + j];
            if (x != 0) f |= pivot_key32(x, 0, R) != kNoKey32 ? 3 : 1;
        }
        f = __reduce_or_sync(0xffffffffu, f);
        if (lane == 0 && (f & ~seen) != 0) atomicOr(flags, f);
    }
}

// dst[i][t] = A[row0 + i][cols[t]]  (rows x k, ld k)
__global__ void gather_cols_kernel(const uint32_t* __restrict__ A, uint64_t ld, int row0, int rows,
                                   const int* __restrict__ cols, int k, uint32_t* __restrict__ dst) {
    const size_t total = static_cast<size_t>(rows) * k;
    for (size_t idx = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; idx < total;
         idx += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const int i = static_cast<int>(idx / k), t = static_cast<int>(idx % k);
        dst[idx] = A[static_cast<size_t>(row0 + i) * ld + cols[t]];
    }
}

// Inverses of the upper triangular diagonal blocks of U1, one CTA per block:
// block b covers rows [b*bb, b*bb + nb) and the pivot columns pcols[b*bb ..].
// U = D U' with U' unit upper; U'^T goes through unit_lower_inverse and U^-1 =
// U'^-1 D^-1 to out + b*bb*bb (nb x nb, row-major, ld nb).
__global__ void __launch_bounds__(1024) tri_inv_kernel(const uint32_t* __restrict__ A, uint64_t ld,
                                                       const int* __restrict__ pcols, int total, int bb, const Ring R,
                                                       uint32_t* __restrict__ out) {
    extern __shared__ __align__(16) uint32_t smem_ti[];
    __shared__ uint32_t dinv[kMaxPanel];
    const int i0 = blockIdx.x * bb, nb = min(bb, total - i0), P = tri_pad(nb), ls = tri_stride(P);
    uint32_t* X = smem_ti;
    for (int t = threadIdx.x; t < nb; t += blockDim.x)
        dinv[t] = unit_inverse(A[static_cast<size_t>(i0 + t) * ld + pcols[i0 + t]], R);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int s = lane; s < P; s += 32) {
        const int pc = s < nb ? pcols[i0 + s] : 0;
#pragma unroll 4
        for (int t = warp; t < P; t += 32) {  // U'[t][s] -> X[s][t]
            uint32_t v = t == s ? 1u : 0u;
            if (t < s && s < nb) v = mod_mul(A[static_cast<size_t>(i0 + t) * ld + pc], dinv[t], R.q, R.barrett);
            X[s * ls + t] = v;
        }
    }
    __syncthreads();
    unit_lower_inverse(X, P, 1, 0, smem_ti + tri_words(P), R.q, R.barrett);
    uint32_t* o = out + static_cast<size_t>(blockIdx.x) * bb * bb;
    for (int idx = threadIdx.x; idx < nb * nb; idx += blockDim.x) {
        const int i = idx / nb, j = idx - i * nb;
        o[idx] = mod_mul(X[j * ls + i], dinv[j], R.q, R.barrett);
    }
}

// Neighbouring diagonal blocks of U1 as one: [B1 U12; 0 B2]^-1 = [I1, -I1 U12 I2;
// 0, I2].  Each step of the substitution is four or five launches in a chain (about
// 25 us), so half as many steps pay for the two products of all pairs at once (about
// 25 us of kernels and two table uploads): RREF 4096 x 4096 of rank 3900 mod 2^31 - 19
// 4.84 ms with blocks of 128, 4.58 with pairs, 4.52 with pairs of pairs; 10515 x 8668
// mod 13 18.05, 17.18 and 16.83 ms.  Below kPairBlocks blocks a level costs what it
// saves, and one more would save four steps of the former.  This kernel lays out the
// pairs: V (its blocks' inverses, 0 elsewhere, ld = the pair's size) and U12.
constexpr int kPairBlocks = 8, kPairFrom = 256;  // pairs of blocks of 128 and 256

__global__ void __launch_bounds__(256) pair_blocks_kernel(const uint32_t* __restrict__ A, uint64_t ld,
                                                          const int* __restrict__ pcols, int rank, int bb,
                                                          const uint32_t* __restrict__ Uinv, uint32_t* __restrict__ V,
                                                          uint32_t* __restrict__ U12) {
    const int i0 = static_cast<int>(blockIdx.x) * 2 * bb, nb = min(2 * bb, rank - i0), n1 = min(bb, nb), n2 = nb - n1;
    const uint32_t* I1 = Uinv + static_cast<size_t>(2 * blockIdx.x) * bb * bb;
    const uint32_t* I2 = I1 + static_cast<size_t>(bb) * bb;
    uint32_t* v = V + static_cast<size_t>(blockIdx.x) * 4 * bb * bb;
    uint32_t* u = U12 + static_cast<size_t>(blockIdx.x) * bb * bb;
    for (int r = blockIdx.y; r < nb; r += gridDim.y)
        for (int c = threadIdx.x; c < nb; c += 256) {
            v[r * nb + c] = r < n1 ? (c < n1 ? I1[r * n1 + c] : 0u) : c < n1 ? 0u : I2[(r - n1) * n2 + c - n1];
            if (r < n1 && c >= n1) u[r * n2 + c - n1] = A[static_cast<size_t>(i0 + r) * ld + pcols[i0 + c]];
        }
}

// R (m x n, ld ldr): rows < rank: identity at the pivot columns, X at the free
// columns; rows >= rank: zero.
__global__ void assemble_rref_kernel(uint32_t* __restrict__ R, uint64_t ldr, int m, int n, int rank,
                                     const int* __restrict__ colmap, const uint32_t* __restrict__ X, int f) {
    // colmap[j] >= 0: pivot index of pivot column j; colmap[j] = -1 - t: free column number t
    const size_t total = static_cast<size_t>(m) * n;
    for (size_t idx = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; idx < total;
         idx += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const int i = static_cast<int>(idx / n), j = static_cast<int>(idx % n);
        uint32_t v = 0;
        if (i < rank) {
            const int cm = colmap[j];
            v = cm >= 0 ? (cm == i ? 1u : 0u) : X[static_cast<size_t>(i) * f + (-1 - cm)];
        }
        R[static_cast<size_t>(i) * ldr + j] = v;
    }
}

// diag[t] = A[t][pivots[t]]
__global__ void gather_diag_kernel(const uint32_t* __restrict__ A, uint64_t ld, const int* __restrict__ piv, int rank,
                                   uint32_t* __restrict__ diag) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < rank; t += gridDim.x * blockDim.x)
        diag[t] = A[static_cast<size_t>(t) * ld + piv[t]];
}

int grid_1d(size_t work, int sms) {
    return static_cast<int>(std::max<size_t>(1, std::min<size_t>((work + 255) / 256, static_cast<size_t>(sms) * 8)));
}

// Kernel attributes, once per device; the largest cluster the panel kernel can be
// launched with (0: none).
int setup_kernels(int device) {
    static OncePerDevice attr;
    // per device: the largest cluster the panel kernel can be launched with (0: none)
    static int cluster_caps[OncePerDevice::kMaxDevices] = {};
    attr.run([](int dev) {
        int& cluster_cap = cluster_caps[dev];
        cluster_cap = 0;
        HME_CUDA(cudaFuncSetAttribute(panel_factor_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPanelSmemMax));
        {
            const int bsm64 = static_cast<int>(block_smem_bytes(96, 64));
            for (const void* fn : {reinterpret_cast<const void*>(panel_block_kernel<kArithPow2, 64>),
                                   reinterpret_cast<const void*>(panel_block_kernel<kArithMont31, 64>),
                                   reinterpret_cast<const void*>(panel_block_kernel<kArithMont32, 64>),
                                   reinterpret_cast<const void*>(panel_block_kernel<kArithPow2, 96>),
                                   reinterpret_cast<const void*>(panel_block_kernel<kArithMont31, 96>),
                                   reinterpret_cast<const void*>(panel_block_kernel<kArithMont32, 96>),
                                   reinterpret_cast<const void*>(panel_block_kernel<kArithMont13, 96>)})
                HME_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bsm64));
            const int bsm128 = static_cast<int>(block_smem_bytes(128, kMaxPanel));
            for (const void* fn : {reinterpret_cast<const void*>(panel_block_kernel<kArithPow2, 128>),
                                   reinterpret_cast<const void*>(panel_block_kernel<kArithMont31, 128>),
                                   reinterpret_cast<const void*>(panel_block_kernel<kArithMont32, 128>),
                                   reinterpret_cast<const void*>(panel_block_kernel<kArithMont13, 128>)})
                HME_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bsm128));
            const int csm = static_cast<int>(compact_smem_bytes(kMaxPanel));
            for (const void* fn : {reinterpret_cast<const void*>(panel_compact_kernel<kArithPow2>),
                                   reinterpret_cast<const void*>(panel_compact_kernel<kArithMont31>),
                                   reinterpret_cast<const void*>(panel_compact_kernel<kArithMont32>)})
                HME_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, csm));
            HME_CUDA(cudaFuncSetAttribute(panel_linv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          static_cast<int>(linv_smem_bytes(kMaxPanel))));
            const int wsm = static_cast<int>(sizeof(uint32_t) * (kMaxPanel * kMaxPanel + kWRows * kMaxPanel));
            for (const void* fn : {reinterpret_cast<const void*>(panel_w_kernel<64, false>),
                                   reinterpret_cast<const void*>(panel_w_kernel<64, true>),
                                   reinterpret_cast<const void*>(panel_w_kernel<128, false>),
                                   reinterpret_cast<const void*>(panel_w_kernel<128, true>)})
                HME_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, wsm));
        }
        bool attrs_ok = true;
        for (const void* fn : {reinterpret_cast<const void*>(panel_cluster_kernel<kArithPow2, 512>),
                               reinterpret_cast<const void*>(panel_cluster_kernel<kArithMont31, 512>),
                               reinterpret_cast<const void*>(panel_cluster_kernel<kArithMont32, 512>),
                               reinterpret_cast<const void*>(panel_cluster_kernel<kArithPow2, 1024>),
                               reinterpret_cast<const void*>(panel_cluster_kernel<kArithMont31, 1024>),
                               reinterpret_cast<const void*>(panel_cluster_kernel<kArithMont32, 1024>)}) {
            attrs_ok = attrs_ok &&
                       cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kClusterSmemMax) ==
                           cudaSuccess &&
                       cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
        }
        if (attrs_ok) {
            for (int cs = kClusterMax; cs >= 1 && cluster_cap == 0; cs /= 2) {
                cudaLaunchConfig_t cfg{};
                cfg.gridDim = dim3(cs);
                cfg.blockDim = dim3(kClusterThreads);
                cfg.dynamicSmemBytes = kClusterSmemMax;
                cudaLaunchAttribute at[1];
                at[0].id = cudaLaunchAttributeClusterDimension;
                at[0].val.clusterDim.x = cs;
                at[0].val.clusterDim.y = 1;
                at[0].val.clusterDim.z = 1;
                cfg.attrs = at;
                cfg.numAttrs = 1;
                int n = 0;
                if (cudaOccupancyMaxActiveClusters(&n, panel_cluster_kernel<kArithMont31, 1024>, &cfg) == cudaSuccess &&
                    n >= 1)
                    cluster_cap = cs;
            }
        }
        cudaGetLastError();  // a refused query leaves no error behind
        HME_CUDA(cudaFuncSetAttribute(tri_inv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(linv_smem_bytes(kMaxPanel))));
    });
    return cluster_caps[device];
}

// The SMs and the skip word of the context's products while this lives, an
// exception's way out included: the word lies in the elimination's scratch, and a
// later product that read it would stand still or read freed memory.
class ProductSettings {
  public:
    ProductSettings(hme_ctx* ctx, int sm_cap, const Skip& skip) : ctx_(ctx) {
        ctx->gemm_sm_cap = sm_cap;
        ctx->gemm_skip = skip;
    }
    ~ProductSettings() {
        ctx_->gemm_sm_cap = 0;
        ctx_->gemm_skip = Skip{};
    }
    ProductSettings(const ProductSettings&) = delete;
    ProductSettings& operator=(const ProductSettings&) = delete;

  private:
    hme_ctx* ctx_;
};

// On an exception's way out of an elimination: the context's stream as the caller
// set it, and nothing of the elimination in flight on it or on the second stream
// (the caller may free the matrix, and the next elimination takes the same scratch).
class FailureDrain {
  public:
    explicit FailureDrain(hme_ctx* ctx) : ctx_(ctx), stream_(ctx->stream), exceptions_(std::uncaught_exceptions()) {}
    ~FailureDrain() {
        if (std::uncaught_exceptions() == exceptions_) return;
        ctx_->stream = stream_;
        cudaStreamSynchronize(ctx_->aux_stream);
        cudaStreamSynchronize(stream_);
        cudaGetLastError();
    }
    FailureDrain(const FailureDrain&) = delete;
    FailureDrain& operator=(const FailureDrain&) = delete;

  private:
    hme_ctx* ctx_;
    cudaStream_t stream_;
    int exceptions_;
};

int panel_width(const ElimOptions& opt) { return std::max(1, std::min<int>(opt.panel > 0 ? opt.panel : 64, kMaxPanel)); }

// The cluster that runs a panel of rows x w: it doubles (up to the largest the
// device runs) until each CTA holds at most rows_per_cta rows, and further while
// a slice does not fit; 0 when the panel needs the grid kernel.
int panel_cluster_size(int rows, int w, int cluster_cap, const ElimOptions& opt) {
    int cs = 0;
    if (opt.panel_kernel != 1 && cluster_cap > 0) {
        const size_t want = static_cast<size_t>(std::max(1, opt.rows_per_cta > 0 ? opt.rows_per_cta : 32));
        auto rpc_of = [&](int c) { return (static_cast<size_t>(rows) + c - 1) / c; };
        auto fits = [&](int c) {
            const size_t rpc = rpc_of(c);
            return rpc <= static_cast<size_t>(kClusterRowsMax) &&
                   cluster_smem_bytes(static_cast<int>(rpc), w) <= static_cast<size_t>(kClusterSmemMax);
        };
        int c = 1;
        while (c < cluster_cap && (rpc_of(c) > want || !fits(c))) c *= 2;
        if (fits(c)) cs = c;
    }
    return cs;
}

}  // namespace

bool elim_can_keep(hme_ctx* ctx, int m, const ElimOptions& opt) {
    return panel_cluster_size(m, panel_width(opt), setup_kernels(ctx->device), opt) > 0;
}

// ---------------------------------------------------------------------------------
ElimResult elim_device(hme_ctx* ctx, const ModParams& mp, uint32_t* A, size_t ld, int m, int n, bool want_rref,
                       uint32_t* R, size_t ldr, const ElimOptions& opt, const RingSpec* ring) {
    HME_REQUIRE(m >= 0 && n >= 0, "elim: negative shape");
    HME_REQUIRE(!(want_rref && ring && ring->k > 1), "elim: the RREF is a field-only object");
    HME_REQUIRE(!(ring && ring->keep_skipped) || (ring->max_v == 0 && ring->lu_cols == 0 && ld >= 2 * static_cast<size_t>(n)),
                "elim: keep_skipped needs unit pivots, all columns and room for n more");
    ElimResult res;
    res.sign_negative = false;
    if (m == 0 || n == 0) {
        if (want_rref && m > 0 && n > 0) HME_CUDA(cudaMemsetAsync(R, 0, 1, ctx->stream));
        return res;
    }
    const int bw = panel_width(opt);
    const uint32_t p = mp.p;
    // the ring: F_p by default, Z/ell^k with a pivot valuation bound when given
    Ring rg{};
    rg.q = p;
    rg.barrett = mp.barrett;
    rg.ell = ring ? ring->ell : p;
    rg.k = ring ? ring->k : 1;
    rg.max_v = ring ? ring->max_v : 0;
    {
        uint64_t pw = 1;
        for (uint32_t v = 0; v <= rg.k && v < 32; ++v) {
            rg.pw[v] = static_cast<uint32_t>(pw);
            pw *= rg.ell;
        }
        HME_REQUIRE(static_cast<uint64_t>(rg.pw[rg.k]) == p || rg.k == 1, "elim: modulus is not ell^k");
    }
    if (p & 1u) {
        uint32_t x = p;  // p^-1 mod 2^32 by Newton's iteration (x = p is right to 3 bits)
        for (int i = 0; i < 5; ++i) x *= 2u - p * x;
        rg.mont_qinv = 0u - x;
        rg.mont_r2 = static_cast<uint32_t>(((static_cast<unsigned __int128>(1) << 64)) % p);
    }
    const int lu_cols = ring && ring->lu_cols > 0 ? std::min(ring->lu_cols, n) : n;

    const int cluster_cap = setup_kernels(ctx->device);

    // device scratch: a ring of four sets, so that panels factored ahead on the second stream, and
    // queued before the host has seen the ones before them, never write the pivot lists that an
    // update still reads
    constexpr int kRing = 4;
    const int grid_cap = std::max(1, std::min(ctx->num_sms, opt.panel_ctas > 0 ? opt.panel_ctas : ctx->num_sms));
    struct Scratch {
        unsigned long long piv_slot[kMaxPanel];
        int pivot_rows[kMaxPanel];
        int pivot_cols[kMaxPanel];
        int k;
        int err;       // the device error word as of the panel's end
        int settled;   // 1: by the top block, 2: by the compact kernel, 0: by a searching kernel (or not yet)
        int count;     // rows listed for the compact kernel
        int fail;      // ring entry 0 only: queued work stands still (BlockQueue::fail)
        int list[kCompactRows];
        int rest;      // what the rest of the matrix holds (window_look_kernel)
        unsigned bar[2];
    };
    const size_t scratch_bytes = (sizeof(Scratch) + 255) / 256 * 256;
    const size_t cand_bytes = sizeof(uint32_t) * 2 * static_cast<size_t>(grid_cap) * kMaxPanel;
    const size_t uinv_bytes = sizeof(uint32_t) * kMaxPanel * kMaxPanel;  // the update's M
    uint8_t* base = static_cast<uint8_t*>(
        ctx->ws.get(kSlotElim0, kRing * (scratch_bytes + cand_bytes + uinv_bytes) + 256));
    // the update's left factor W at its largest, for panels in turn: the compact kernel writes its panel's
    // while the update before reads its own, and a panel is launched after the last update but one
    static_assert(kRing % 2 == 0, "neighbouring panels alternate between the two");
    const int ldw = std::min(bw, lu_cols);
    const size_t w_words = static_cast<size_t>(m) * ldw;
    uint32_t* d_W = static_cast<uint32_t*>(ctx->ws.get(kSlotElim2, 2 * sizeof(uint32_t) * w_words));
    Scratch* d_sb[kRing];
    uint32_t *d_candb[kRing], *d_uinvb[kRing], *d_Wb[kRing];
    for (int i = 0; i < kRing; ++i) {
        d_sb[i] = reinterpret_cast<Scratch*>(base + i * scratch_bytes);
        d_candb[i] = reinterpret_cast<uint32_t*>(base + kRing * scratch_bytes + i * cand_bytes);
        d_uinvb[i] = reinterpret_cast<uint32_t*>(base + kRing * (scratch_bytes + cand_bytes) + i * uinv_bytes);
        d_Wb[i] = d_W + (i & 1) * w_words;
        HME_CUDA(cudaMemsetAsync(d_sb[i]->bar, 0, sizeof(unsigned) * 2, ctx->stream));
        HME_CUDA(cudaMemsetAsync(&d_sb[i]->count, 0, 2 * sizeof(int), ctx->stream));  // count, fail
    }
    int* d_fail = &d_sb[0]->fail;
    // pinned copies of the scratch sets (the host reads a panel's pivots without waiting for
    // the other stream's work), the second stream and the events of the lookahead
    const size_t pinned_bytes = kRing * sizeof(Scratch);
    if (ctx->elim_pinned_bytes < pinned_bytes) {
        if (ctx->elim_pinned) {
            HME_CUDA(cudaDeviceSynchronize());
            HME_CUDA(cudaFreeHost(ctx->elim_pinned));
            ctx->elim_pinned = nullptr;
            ctx->elim_pinned_bytes = 0;
        }
        HME_CUDA(cudaMallocHost(&ctx->elim_pinned, pinned_bytes));
        ctx->elim_pinned_bytes = pinned_bytes;
    }
    Scratch* h_sb = static_cast<Scratch*>(ctx->elim_pinned);
    if (!ctx->aux_stream) {
        // the lookahead panel's stream at the highest priority: its cluster takes SMs as they free up
        int lo = 0, hi = 0;
        HME_CUDA(cudaDeviceGetStreamPriorityRange(&lo, &hi));
        HME_CUDA(cudaStreamCreateWithPriority(&ctx->aux_stream, cudaStreamNonBlocking, hi));
    }
    while (ctx->elim_ev.size() < 1 + 2 * kRing) {
        cudaEvent_t e;
        HME_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        ctx->elim_ev.push_back(e);
    }
    // ev_panel: the panel's kernels are done; ev_host: its results are in pinned memory
    const cudaEvent_t ev_next = ctx->elim_ev[0], *ev_panel = &ctx->elim_ev[1], *ev_host = &ctx->elim_ev[1 + kRing];
    const cudaStream_t s_main = ctx->stream, s_aux = ctx->aux_stream;
    const FailureDrain drain(ctx);
    // lookahead only where it can overlap: the cluster kernel (a few SMs), and not while the
    // per-kernel timer is on (its events assume one stream)
    const bool allow_lookahead = !opt.no_lookahead && !ctx->timer.on;

    // the cluster kernel when the active rows fit the shared memory of one cluster, else the grid kernel (0)
    auto cluster_size = [&](int rows, int w) { return panel_cluster_size(rows, w, cluster_cap, opt); };

    // the determinant's pivots of the panels that the top block settles (their diagonal in A is 1);
    // 0 where a searching kernel left the pivot in A
    uint32_t* d_blkdiag = nullptr;
    if (opt.want_diag) {
        d_blkdiag = static_cast<uint32_t*>(ctx->ws.get(kSlotElim4, sizeof(uint32_t) * (static_cast<size_t>(std::max(m, n)) + 16)));
        HME_CUDA(cudaMemsetAsync(d_blkdiag, 0, sizeof(uint32_t) * m, s_main));
    }
    // The panel's kernels in automatic mode: the top block, then the compact search of the non-zero
    // rows, then the search over all rows.  A failed attempt costs 10 us beside the search's 60 to 270,
    // so after one the next 3, then 7 panels pass over the top block (rank-deficient tails, sparse
    // matrices, rings whose columns run out of units), the next 3, 7, 15, then 31 over the compact rows
    // (dense matrices), and the count starts over with the next panel that it settles.  (A matrix that
    // fills up halfway is back on the top block after 7 panels at most: 2000 x 2000 mod 65521, 1000
    // columns of 4 entries and 1000 dense ones, 5.46 ms with pauses of up to 31 panels, 4.65 with 7.)
    // What is launched behind an attempt returns at once when the attempt settled the panel, so a
    // failure costs no round trip to the host; behind an attempt that is expected to succeed -- the kernel's last one did, or it is the
    // top block over a large field -- nothing is launched, and the host launches the rest if it must.
    const bool automatic = opt.panel_kernel == 0;
    struct Attempt {
        int most, rest = 0, pause = 3;
        bool sure = false;
        explicit Attempt(int longest_pause) : most(longest_pause) {}
        void settled() {
            pause = 3;
            sure = true;
        }
        void failed() {
            rest = pause;
            pause = std::min(most, 2 * pause + 1);
            sure = false;
        }
    } block(7), compact(31);
    block.sure = rg.k == 1 && p >= (1u << 20);
    const bool keep = ring && ring->keep_skipped;
    bool block_tried[kRing] = {}, compact_tried[kRing] = {}, search_run[kRing] = {};
    // a block over a large field finds its pivots in row order almost always: nothing is queued for moves
    const bool in_order = rg.k == 1 && p >= (1u << 20);
    // The panel [c0, c0 + w) of the active rows [r0, m) on `st`, from kernel `from` on (0 the top
    // block, 1 the compact rows, 2 the search).  Its pivots and the error word land in h_sb[par];
    // ev_panel[par] and ev_host[par] are recorded.  Returns the SMs that a GEMM beside the panel leaves free.
    int seq = 0, panel_seq[kRing] = {};  // numbers of the top-block attempts
    cudaStream_t panel_stream[kRing] = {s_main, s_main, s_main, s_main};
    auto launch_panel = [&](int c0, int w, int r0, int par, cudaStream_t st, int from) -> int {
        Scratch* d_s = d_sb[par];
        const cudaStream_t saved = ctx->stream;
        ctx->stream = st;  // HME_TIMED brackets the launch on the launching stream
        panel_stream[par] = st;
        PanelArgs pa{};
        pa.A = A;
        pa.ld = ld;
        pa.m = m;
        pa.c0 = c0;
        pa.bw = w;
        pa.r0 = r0;
        pa.R = rg;
        pa.piv_slot = d_s->piv_slot;
        pa.cand = d_candb[par];
        pa.pivot_rows = d_s->pivot_rows;
        pa.pivot_cols = d_s->pivot_cols;
        pa.k_out = &d_s->k;
        pa.bar = d_s->bar;
        pa.err = ctx->d_err;
        pa.keep = keep ? 1 : 0;
        const int rows = m - r0;
        int busy = 0;  // SMs the panel's kernels take
        bool more = true;  // the kernels after the ones launched so far may be needed
        const bool try_block = from == 0 && automatic && block.rest == 0;
        if (from == 0 && block.rest > 0) --block.rest;
        block_tried[par] = try_block;
        if (try_block) {
            BlockArgs ba{};
            ba.A = A;
            ba.ld = ld;
            ba.m = m;
            ba.r0 = r0;
            ba.c0 = c0;
            ba.w = w;
            ba.R = rg;
            ba.pivot_rows = d_s->pivot_rows;
            ba.pivot_cols = d_s->pivot_cols;
            ba.k_out = &d_s->k;
            ba.ok = &d_s->settled;
            ba.binv = d_uinvb[par];
            ba.diag = d_blkdiag;
            const BlockQueue bq{d_fail, ++seq, in_order ? 1 : 0, ctx->d_err, &d_s->err};
            panel_seq[par] = seq;
            // 64 row slots where a zero pivot is rare (chance about 64/p per panel), 32 spare rows over
            // smaller fields and rings
            const int rs = w > 64 ? 128 : rg.k == 1 && p >= (1u << 20) ? 64 : 96;
            const size_t bsm = block_smem_bytes(rs, w);
            auto launch_block = [&](auto kern) {
                HME_TIMED(ctx, "panel_block", kern<<<1, 4 * rs, bsm, st>>>(ba, bq));
            };
            if (rg.ell == 2) {
                if (rs == 64) launch_block(panel_block_kernel<kArithPow2, 64>);
                else if (rs == 96) launch_block(panel_block_kernel<kArithPow2, 96>);
                else launch_block(panel_block_kernel<kArithPow2, 128>);
            } else if (p < kMont13Max && rs != 64) {
                if (rs == 96) launch_block(panel_block_kernel<kArithMont13, 96>);
                else launch_block(panel_block_kernel<kArithMont13, 128>);
            } else if (p < (1u << 31)) {
                if (rs == 64) launch_block(panel_block_kernel<kArithMont31, 64>);
                else if (rs == 96) launch_block(panel_block_kernel<kArithMont31, 96>);
                else launch_block(panel_block_kernel<kArithMont31, 128>);
            } else {
                if (rs == 64) launch_block(panel_block_kernel<kArithMont32, 64>);
                else if (rs == 96) launch_block(panel_block_kernel<kArithMont32, 96>);
                else launch_block(panel_block_kernel<kArithMont32, 128>);
            }
            HME_CUDA(cudaGetLastError());
        }
        if (try_block) {
            more = !block.sure;
            busy = 1;
        }
        const bool try_compact = more && from <= 1 && automatic && compact.rest == 0;
        if (more && from <= 1 && compact.rest > 0) --compact.rest;
        compact_tried[par] = try_compact;
        if (try_compact) {
            CompactArgs ca{};
            ca.A = A;
            ca.ld = ld;
            ca.m = m;
            ca.r0 = r0;
            ca.c0 = c0;
            ca.w = w;
            ca.R = rg;
            ca.most = rg.ell == 2 ? kCompactMostPow2 : kCompactMost;
            ca.list = d_s->list;
            ca.count = &d_s->count;
            ca.after_block = try_block ? 1 : 0;
            ca.ok = &d_s->settled;
            ca.pivot_rows = d_s->pivot_rows;
            ca.pivot_cols = d_s->pivot_cols;
            ca.k_out = &d_s->k;
            ca.W = d_Wb[par];
            ca.ldw = ldw;
            HME_TIMED(ctx, "panel_rows", panel_rows_kernel<<<(rows + 7) / 8, 256, 0, st>>>(ca));
            auto launch_compact = [&](auto kern) {
                HME_TIMED(ctx, "panel_compact", kern<<<1, 1024, compact_smem_bytes(w), st>>>(ca));
            };
            if (rg.ell == 2) launch_compact(panel_compact_kernel<kArithPow2>);
            else if (p < (1u << 31)) launch_compact(panel_compact_kernel<kArithMont31>);
            else launch_compact(panel_compact_kernel<kArithMont32>);
            HME_CUDA(cudaGetLastError());
            more = !compact.sure;
            busy = 1;
        }
        const int cs = cluster_size(rows, w);
        HME_REQUIRE(opt.panel_kernel < 2 || cs > 0, "elim: the panel does not fit one cluster");
        HME_REQUIRE(!keep || cs > 0 || !more, "elim: the panel is too tall for the cluster kernel");
        search_run[par] = more;
        if (more) busy = cs;
        if (try_block || try_compact) pa.skip = &d_s->settled;
        if (!more) {
            // the host launches the panel's other kernels if the attempt fails
        } else if (cs > 0) {
            const int rpc = static_cast<int>((static_cast<size_t>(rows) + cs - 1) / cs);
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(cs);
            cfg.blockDim = dim3(kClusterThreads);
            cfg.dynamicSmemBytes = cluster_smem_bytes(rpc, w);
            cfg.stream = st;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = cs;
            at[0].val.clusterDim.y = 1;
            at[0].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            // q = 2^k: wraparound; odd q < 2^31: one Montgomery reduction per element; else two.
            // 512 threads per CTA while a CTA holds at most 512 rows (half the per-column
            // control work of 1024 threads), unless the panel-kernel setting asks for 1024
            const bool t512 = rpc <= 512 && opt.panel_kernel != 3;
            cfg.blockDim = dim3(t512 ? 512 : 1024);
            auto launch = [&](auto kern) {
                HME_TIMED(ctx, "panel_factor", HME_CUDA(cudaLaunchKernelEx(&cfg, kern, pa)));
            };
            if (rg.ell == 2) {
                if (t512) launch(panel_cluster_kernel<kArithPow2, 512>);
                else launch(panel_cluster_kernel<kArithPow2, 1024>);
            } else if (p < (1u << 31)) {
                if (t512) launch(panel_cluster_kernel<kArithMont31, 512>);
                else launch(panel_cluster_kernel<kArithMont31, 1024>);
            } else {
                if (t512) launch(panel_cluster_kernel<kArithMont32, 512>);
                else launch(panel_cluster_kernel<kArithMont32, 1024>);
            }
        } else {
            HME_CUDA(cudaMemsetAsync(d_s->piv_slot, 0x7f, sizeof(unsigned long long) * kMaxPanel, st));
            const int rpc_want = std::max(1, opt.rows_per_cta > 0 ? opt.rows_per_cta : 32);
            const int want_grid = std::max(1, std::min(grid_cap, (rows + rpc_want - 1) / rpc_want));
            const int rpc = (rows + want_grid - 1) / want_grid;
            const size_t slice_bytes = sizeof(uint32_t) * static_cast<size_t>(rpc) * w;
            const size_t extra = 5 * static_cast<size_t>(rpc) + 16;  // multipliers + pivot flags
            int smem_rows = slice_bytes + extra <= kPanelSmemMax ? 1 : 0;
            const size_t dyn = (smem_rows ? slice_bytes : 0) + extra;
            void* args[] = {&pa, &smem_rows};
            HME_TIMED(ctx, "panel_factor",
                      HME_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(panel_factor_kernel), want_grid,
                                                           kPanelThreads, args, dyn, st)));
        }
        HME_CUDA(cudaEventRecord(ev_panel[par], st));
        // the panel's error word next to its pivots (the block kernel has written it), then the pivots to
        // pinned memory
        if (try_compact || more)
            HME_CUDA(cudaMemcpyAsync(&d_s->err, ctx->d_err, sizeof(int), cudaMemcpyDeviceToDevice, st));
        HME_CUDA(cudaMemcpyAsync(&h_sb[par], d_s, sizeof(Scratch), cudaMemcpyDeviceToHost, st));
        HME_CUDA(cudaEventRecord(ev_host[par], st));
        ctx->stream = saved;
        return busy;
    };

    std::vector<int> pivots;
    pivots.reserve(std::min(m, n));
    // keep mode: the pivotless columns of the panels so far, appended right of the matrix, where the
    // later updates reach them
    int app = 0;
    auto append = [&](int c0, int w, int row0, int par, int k) {
        if (k == w || row0 >= m) return;
        HME_TIMED(ctx, "append_cols", append_cols_kernel<<<std::min((m - row0 + 7) / 8, 8 * ctx->num_sms), 256, 0, s_main>>>(
                                          A, ld, row0, m - row0, c0, w, d_sb[par]->pivot_cols, k, n + app));
        HME_CUDA(cudaGetLastError());
        app += w - k;
    };
    // One panel's update; `skip` where it is queued before the host knows the panel's outcome.
    struct Update {
        int c0, w, r0, k, par, by;
        bool moves;
        Skip skip;
        uint32_t* Wf = nullptr;
    };
    // columns [ca, cb): row moves (from c0 on), then [A12; A22] += W A12 on a tensor-core variant (it
    // reads A12 through its limb planes, so C may alias it)
    auto update = [&](Update& U, int ca, int cb, int sm_cap) {
        if (cb <= ca) return;
        if (U.moves) {
            HME_TIMED(ctx, "row_moves", move_pivot_rows_kernel<<<(cb - ca + kMoveCols - 1) / kMoveCols, 256, 0, s_main>>>(
                                            A, ld, U.r0, U.k, d_sb[U.par]->pivot_rows, ca, cb, U.skip));
            HME_CUDA(cudaGetLastError());
        }
        const int ua = std::max(ca, U.c0 + U.w), rows = m - U.r0, k = U.k;
        if (cb <= ua) return;
        if (!U.Wf && U.by == 2) U.Wf = d_Wb[U.par];
        if (!U.Wf) {
            uint32_t* mul = d_uinvb[U.par];
            const int* d_pcols = d_sb[U.par]->pivot_cols;
            if (U.by == 0) {
                HME_TIMED(ctx, "panel_linv", panel_linv_kernel<<<1, 512, linv_smem_bytes(k), s_main>>>(
                                                 A, ld, U.r0, d_pcols, k, p, mp.barrett, mul));
                HME_CUDA(cudaGetLastError());
            }
            U.Wf = d_Wb[U.par];
            const int g = (rows + kWRows - 1) / kWRows;
            const size_t wsm = sizeof(uint32_t) * (((static_cast<size_t>(k) * k + 3) & ~size_t(3)) +
                                                   static_cast<size_t>(kWRows) * ((k + 3) & ~3));
            const bool small = static_cast<double>(k) * (p - 1.0) * (p - 1.0) < 4294967296.0;
            auto kernel = k <= 64 ? (small ? panel_w_kernel<64, true> : panel_w_kernel<64, false>)
                                  : (small ? panel_w_kernel<128, true> : panel_w_kernel<128, false>);
            HME_TIMED(ctx, "panel_w", kernel<<<g, 256, wsm, s_main>>>(A, ld, U.r0, m, d_pcols, k, mul, p, mp.barrett,
                                                                     U.skip, U.Wf));
            HME_CUDA(cudaGetLastError());
        }
        const ProductSettings settings(ctx, sm_cap, U.skip);
        uint32_t* C12 = A + static_cast<size_t>(U.r0) * ld + ua;
        gemm_u32_variant(ctx, mp, rows, cb - ua, k, U.Wf, U.by == 2 ? ldw : k, C12, ld, C12, ld, HME_ADD,
                         gemm_default_variant(ctx, mp, rows, cb - ua));
    };
    int r0 = 0, c0 = 0, par = 0;
    int next_look = 0;  // panel count before which a pivotless panel does not look over the rest
    int look_gap = 1, panels = 0;
    auto next_of = [](int i) { return (i + 1) % kRing; };
    // lookahead only when the next panel runs on the cluster kernel (a few SMs beside the GEMM; the
    // cooperative grid kernel would wait for the whole device anyway)
    auto ahead = [&](int c1, int r1) {
        return allow_lookahead && c1 < lu_cols && r1 < m && cluster_size(m - r1, std::min(bw, lu_cols - c1)) > 0;
    };
    // LOOKAHEAD: the next panel's columns first; that panel is factored on the second stream while the
    // rest of this update runs here, the GEMM leaving the panel's SMs free; the main stream's later work
    // (the next panel's update) follows that panel
    auto update_ahead = [&](Update& U) {
        const int c1 = U.c0 + U.w, nw = std::min(bw, lu_cols - c1);
        update(U, U.c0, c1 + nw, 0);
        HME_CUDA(cudaEventRecord(ev_next, s_main));
        HME_CUDA(cudaStreamWaitEvent(s_aux, ev_next, 0));
        const int busy = launch_panel(c1, nw, U.r0 + U.k, next_of(U.par), s_aux, 0);
        update(U, c1 + nw, n + app, std::max(1, ctx->num_sms - busy));
        if (keep) append(U.c0, U.w, U.r0 + U.k, U.par, U.k);
        HME_CUDA(cudaStreamWaitEvent(s_main, ev_panel[next_of(U.par)], 0));
    };
    // the host's record of a panel with pivots: its columns, the sign of its row moves, the statistics (a
    // top block that looks for most of its pivots -- a field of fewer than 256 elements, a ring -- counts
    // as searched)
    auto record = [&](const Scratch& h, int row0, int by, bool moves) {
        if (by == 1 && rg.k == 1 && p >= 256) ++ctx->elim_block_panels;
        else ++ctx->elim_search_panels;
        ++panels;
        for (int t = 0; t < h.k; ++t) pivots.push_back(h.pivot_cols[t]);
        if (moves && row_moves_odd(h.pivot_rows, h.k, row0)) res.sign_negative = !res.sign_negative;
    };
    auto in_place = [](const Scratch& h, int row0) {
        for (int t = 0; t < h.k; ++t)
            if (h.pivot_rows[t] != row0 + t) return false;
        return true;
    };
    // Panels whose update, and the panel after them, were queued before the host knew their outcome, at
    // most two: where the top block is expected to settle the panel, the host only checks up on the panel
    // before, so that its round trip (about 20 us a panel) is off the chain.  A panel that turns out
    // otherwise raises the flag that everything queued behind it obeys, and the loop takes it up again.
    std::vector<Update> queued;
    bool launched = false;  // the panel at c0 was already factored ahead (on the second stream)
    while (true) {
        const bool more_panels = c0 < lu_cols && r0 < m;
        const int w = more_panels ? std::min(bw, lu_cols - c0) : 0;
        bool queue = false;
        if (more_panels) {
            if (!launched && queued.empty()) {
                launch_panel(c0, w, r0, par, s_main, 0);
                launched = true;
            }
            queue = launched && block_tried[par] && !compact_tried[par] && !search_run[par] && m - r0 > w &&
                    ahead(c0 + w, r0 + w);
            if (queue) {
                Update U{c0, w, r0, w, par, 1, !in_order, Skip{d_fail, panel_seq[par]}};
                update_ahead(U);
                queued.push_back(U);
                r0 += w;
                c0 += w;
                par = next_of(par);
            }
        }
        // check up on the queued panels: all but the newest, all when nothing more is queued
        bool undo = false;
        while (queued.size() > (queue ? 1u : 0u)) {
            const Update U = queued.front();
            HME_CUDA(cudaEventSynchronize(ev_host[U.par]));
            const Scratch& h = h_sb[U.par];
            if (h.err != 0) check_device_error(ctx);
            if (h.settled == 1 && (!in_order || in_place(h, U.r0))) {
                block.settled();
                record(h, U.r0, 1, !in_order && !in_place(h, U.r0));
                queued.erase(queued.begin());
                continue;
            }
            // stands still from this panel on: take it up again
            HME_CUDA(cudaStreamSynchronize(s_main));
            HME_CUDA(cudaStreamSynchronize(s_aux));
            HME_CUDA(cudaMemsetAsync(d_fail, 0, sizeof(int), s_main));
            c0 = U.c0;
            r0 = U.r0;
            par = U.par;
            launched = true;
            queued.clear();
            undo = true;
            break;
        }
        if (queue && !undo) continue;
        if (!(c0 < lu_cols && r0 < m)) break;
        const int wp = std::min(bw, lu_cols - c0);
        if (!launched) launch_panel(c0, wp, r0, par, s_main, 0);
        launched = false;
        HME_CUDA(cudaEventSynchronize(ev_host[par]));
        // what settled the panel: 1 the top block, 2 the compact rows, 0 the search
        int by = 0;
        for (;;) {
            by = block_tried[par] || compact_tried[par] ? h_sb[par].settled : 0;
            if (block_tried[par]) {
                by == 1 ? block.settled() : block.failed();
                HME_CUDA(cudaMemsetAsync(d_fail, 0, sizeof(int), s_main));  // nothing is queued behind it
            }
            if (compact_tried[par] && by != 1) by == 2 ? compact.settled() : compact.failed();
            if (by != 0 || search_run[par]) break;
            // an attempt that was expected to succeed did not (nothing was written): the panel's other
            // kernels, on its stream; the main stream's later work waits for them too
            launch_panel(c0, wp, r0, par, panel_stream[par], compact_tried[par] ? 2 : 1);
            if (panel_stream[par] != s_main) HME_CUDA(cudaStreamWaitEvent(s_main, ev_panel[par], 0));
            HME_CUDA(cudaEventSynchronize(ev_host[par]));
        }
        const Scratch& h_s = h_sb[par];
        if (h_s.err != 0) check_device_error(ctx);  // reports the timeout (and clears the word)
        const int k = h_s.k, c1 = c0 + wp;
        const bool moves = k > 0 && !in_place(h_s, r0);
        record(h_s, r0, by, moves);
        if (k == 0) {
            if (keep) append(c0, wp, r0, par, 0);
            c0 = c1;
            // no pivot in the panel: nothing moved, the next panel starts at r0 -- unless there is none in
            // the rest (one pass over it, against a panel's search each; after a pass that found one only
            // every 2nd, 4th, .. pivotless panel asks again).  Rows of Z/2^31 scaled by random powers of 2,
            // 1024 x 1024: Smith 35.3 ms asking whether the rest was zero, 7.6 ms asking for units.
            if (c1 < lu_cols && panels >= next_look) {
                int* d_rest = &d_sb[par]->rest;
                HME_CUDA(cudaMemsetAsync(d_rest, 0, sizeof(int), s_main));
                HME_TIMED(ctx, "rest_nonzero",
                          window_look_kernel<<<std::min(m - r0, 8 * ctx->num_sms), 256, 0, s_main>>>(
                              A + static_cast<size_t>(r0) * ld + c1, ld, m - r0, lu_cols - c1, rg, d_rest));
                HME_CUDA(cudaGetLastError());
                HME_CUDA(cudaMemcpyAsync(&h_sb[par].rest, d_rest, sizeof(int), cudaMemcpyDeviceToHost, s_main));
                HME_CUDA(cudaStreamSynchronize(s_main));
                if ((h_sb[par].rest & 2) == 0) {
                    if (keep && h_sb[par].rest != 0)  // its columns are left out too
                        for (int c = c1; c < n; c += kMaxPanel) append(c, std::min(kMaxPanel, n - c), r0, par, 0);
                    break;
                }
                next_look = panels + look_gap;
                look_gap *= 2;
            }
            continue;
        }
        Update U{c0, wp, r0, k, par, by, moves, Skip{}};
        if (ahead(c1, r0 + k)) {
            update_ahead(U);
            launched = true;
        } else {
            update(U, c0, n + app, 0);
            if (keep) append(c0, wp, r0 + k, par, k);
        }
        r0 += k;
        c0 = c1;
        par = next_of(par);
    }
    HME_CUDA(cudaStreamSynchronize(s_aux));
    res.rank = r0;
    res.pivots = pivots;
    res.appended = app;

    // determinant factors: the U diagonal
    if (opt.want_diag && res.rank > 0) {
        int* d_pv = static_cast<int*>(ctx->ws.get(kSlotElim3, sizeof(int) * (2 * static_cast<size_t>(n) + 16)));
        uint32_t* d_diag = reinterpret_cast<uint32_t*>(d_pv + n);
        HME_CUDA(cudaMemcpyAsync(d_pv, pivots.data(), sizeof(int) * res.rank, cudaMemcpyHostToDevice, ctx->stream));
        HME_TIMED(ctx, "gather_diag", gather_diag_kernel<<<grid_1d(res.rank, ctx->num_sms), 256, 0, ctx->stream>>>(
                                          A, ld, d_pv, res.rank, d_diag));
        HME_CUDA(cudaGetLastError());
        res.diag.resize(res.rank);
        HME_CUDA(cudaMemcpyAsync(res.diag.data(), d_diag, sizeof(uint32_t) * res.rank, cudaMemcpyDeviceToHost,
                                 ctx->stream));
        std::vector<uint32_t> blk(res.rank);
        HME_CUDA(cudaMemcpyAsync(blk.data(), d_blkdiag, sizeof(uint32_t) * res.rank, cudaMemcpyDeviceToHost,
                                 ctx->stream));
        HME_CUDA(cudaStreamSynchronize(ctx->stream));
        for (int t = 0; t < res.rank; ++t)
            if (blk[t] != 0) res.diag[t] = blk[t];
    }
    if (!want_rref) return res;

    // ---- RREF = U1^-1 U on the free columns ------------------------------------------
    const int rank = res.rank;
    const int f = n - rank;
    std::vector<int> colmap(n);
    std::vector<int> free_cols;
    {
        std::vector<char> isp(n, 0);
        for (int t = 0; t < rank; ++t) {
            isp[pivots[t]] = 1;
            colmap[pivots[t]] = t;
        }
        for (int j = 0; j < n; ++j)
            if (!isp[j]) {
                colmap[j] = -1 - static_cast<int>(free_cols.size());
                free_cols.push_back(j);
            }
    }
    int* d_cols = static_cast<int*>(ctx->ws.get(kSlotElim3, sizeof(int) * (2 * static_cast<size_t>(n) + 16)));
    int* d_piv = d_cols + n;  // pivots, then free columns at d_cols
    uint32_t* X = nullptr;
    if (rank > 0) {
        HME_CUDA(cudaMemcpyAsync(d_piv, pivots.data(), sizeof(int) * rank, cudaMemcpyHostToDevice, ctx->stream));
    }
    if (rank > 0 && f > 0) {
        HME_CUDA(cudaMemcpyAsync(d_cols, free_cols.data(), sizeof(int) * f, cudaMemcpyHostToDevice, ctx->stream));
        X = static_cast<uint32_t*>(ctx->ws.get(kSlotElim1, sizeof(uint32_t) * static_cast<size_t>(rank) * f));
        HME_TIMED(ctx, "gather_cols",
                  gather_cols_kernel<<<grid_1d(static_cast<size_t>(rank) * f, ctx->num_sms), 256, 0, ctx->stream>>>(
                      A, ld, 0, rank, d_cols, f, X));
        HME_CUDA(cudaGetLastError());
        int bb = std::max(16, std::min(opt.back_block > 0 ? opt.back_block : 128, 128));
        int nblk = (rank + bb - 1) / bb;
        // all diagonal blocks of U1 inverted at once, one CTA each
        // words of the blocks, then per level of pairs V, U12 and T
        const auto paired = [](int b, int blocks) { return b >= 128 && b <= kPairFrom && blocks >= kPairBlocks; };
        size_t words = static_cast<size_t>(nblk) * bb * bb;
        for (int b = bb, k = nblk; paired(b, k); b *= 2) {
            k = (k + 1) / 2;
            words += 6 * static_cast<size_t>(k) * b * b;
        }
        uint32_t* Uinv = static_cast<uint32_t*>(ctx->ws.get(kSlotElim5, sizeof(uint32_t) * words));
        {
            HME_TIMED(ctx, "tri_inv", tri_inv_kernel<<<nblk, 1024, linv_smem_bytes(std::min(bb, rank)), ctx->stream>>>(
                                          A, ld, d_piv, rank, bb, rg, Uinv));
            HME_CUDA(cudaGetLastError());
        }
        uint32_t* next = Uinv + static_cast<size_t>(nblk) * bb * bb;
        while (paired(bb, nblk)) {
            const int pairs = (nblk + 1) / 2;
            const size_t bsq = static_cast<size_t>(bb) * bb;
            uint32_t* V = next;
            uint32_t* U12 = V + 4 * bsq * pairs;
            uint32_t* T = U12 + bsq * pairs;
            next = T + bsq * pairs;
            HME_TIMED(ctx, "tri_inv", pair_blocks_kernel<<<dim3(pairs, 16), 256, 0, ctx->stream>>>(A, ld, d_piv, rank, bb,
                                                                                                  Uinv, V, U12));
            HME_CUDA(cudaGetLastError());
            std::vector<GemmJob> first, second;
            for (int j = 0; j < pairs; ++j) {
                const uint32_t nb = static_cast<uint32_t>(std::min(2 * bb, rank - 2 * j * bb)), n1 = std::min<uint32_t>(bb, nb);
                if (nb == n1) continue;
                GemmJob g;
                g.M = n1;
                g.N = g.K = nb - n1;
                g.A = U12 + bsq * j;
                g.B = Uinv + bsq * (2 * j + 1);
                g.C = T + bsq * j;
                g.lda = g.ldb = g.ldc = nb - n1;
                first.push_back(g);
                g.K = n1;
                g.A = Uinv + bsq * (2 * j);
                g.lda = n1;
                g.B = T + bsq * j;
                g.C = V + 4 * bsq * j + n1;
                g.ldc = nb;
                g.op = HME_SUB;
                second.push_back(g);
            }
            grouped_gemm_u32_device(ctx, mp, first);
            grouped_gemm_u32_device(ctx, mp, second);
            Uinv = V;
            bb *= 2;
            nblk = pairs;
        }
        // W (rank x f) in X's slot; the solution accumulates in Xs
        uint32_t* Xs = static_cast<uint32_t*>(ctx->ws.get(kSlotElim6, sizeof(uint32_t) * static_cast<size_t>(rank) * f));
        for (int blk = nblk - 1; blk >= 0; --blk) {
            const int i0 = blk * bb, nb = std::min(bb, rank - i0);
            // X_B = U_BB^-1 W_B
            gemm_u32_device(ctx, mp, nb, f, nb, Uinv + static_cast<size_t>(blk) * bb * bb, nb,
                            X + static_cast<size_t>(i0) * f, f, Xs + static_cast<size_t>(i0) * f, f, HME_SET);
            if (i0 > 0) {
                // W[0:i0] -= U1[0:i0, block pivots] * X_B
                uint32_t* Ub = static_cast<uint32_t*>(ctx->ws.get(kSlotElim2, sizeof(uint32_t) * static_cast<size_t>(i0) * nb));
                HME_TIMED(ctx, "gather_cols",
                          gather_cols_kernel<<<grid_1d(static_cast<size_t>(i0) * nb, ctx->num_sms), 256, 0, ctx->stream>>>(
                              A, ld, 0, i0, d_piv + i0, nb, Ub));
                HME_CUDA(cudaGetLastError());
                gemm_u32_device(ctx, mp, i0, f, nb, Ub, nb, Xs + static_cast<size_t>(i0) * f, f, X, f, HME_SUB);
            }
        }
        X = Xs;
    }
    int* d_colmap = static_cast<int*>(ctx->ws.get(kSlotElim4, sizeof(int) * (static_cast<size_t>(n) + 16)));
    HME_CUDA(cudaMemcpyAsync(d_colmap, colmap.data(), sizeof(int) * n, cudaMemcpyHostToDevice, ctx->stream));
    HME_TIMED(ctx, "assemble_rref",
              assemble_rref_kernel<<<grid_1d(static_cast<size_t>(m) * n, ctx->num_sms), 256, 0, ctx->stream>>>(
                  R, ldr, m, n, rank, d_colmap, X, std::max(f, 1)));
    HME_CUDA(cudaGetLastError());
    HME_CUDA(cudaStreamSynchronize(ctx->stream));
    return res;
}

}  // namespace hme
