// Howell and Smith forms over Z/ell^k (ell prime, ell^k < 2^32) on the device.
//
// Reference semantics (drjanosch42/hacs 0.2.1): the Howell form of rowspan(A),
// ENGINE_API.md Sec. 13.5 (elim::howell, DenseElim.h:239-249;
// ring2k::howell, Binary/Ring2k.h:960-969 = minimal-valuation echelon
// echelon_blocked :539-695 + howell_pass :853-954; ring3k::howell,
// Binary/Ring3k.h:101), and the Smith valuations sigma (ring2k::smith,
// Ring2k.h:702-845; ring3k::smith / smith_levels, Ring3k.cpp:615-843).  Both
// outputs are unique functions of the input, so the device result equals the
// reference's bit for bit whatever pivot rows the blocked elimination picks.
//
// Smith by valuation levels (the reference's algorithm): at level s, over
// Z/ell^(k-s), a unit-pivot LU of the r_s columns of the F_ell column rank profile
// (the blocked device LU, pivots of valuation 0) leaves a Schur complement that
// is 0 mod ell; r_s valuations equal s; the Schur complement divided by ell is
// the next level.
//
// Howell: the blocked device LU with minimal-valuation pivots gives echelon
// rows with the same row span; the Sec. 13.5 pass normalises all of them at
// once and inserts the non-zero closure rows one column at a time; the
// reduce-above runs in blocks of pivots, the floor quotients of the rows down
// to a block's last by one kernel and their application by one limb GEMM (mod
// ell^k).
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "hme_elim.h"
#include "hme_internal.h"
#include "hme_ptx.cuh"

namespace hme {
namespace {

constexpr int kHowellThreads = 1024;
constexpr int kReduceBlock = 64;
constexpr size_t kHowellLeadSmemMax = 192 * 1024;  // leading-column table of the Howell pass (48k rows)

struct RingK {
    uint32_t q, ell, k;
    uint64_t barrett;
    uint32_t pw[33];
};

RingK make_ring(uint32_t ell, uint32_t k) {
    RingK r{};
    r.ell = ell;
    r.k = k;
    uint64_t pw = 1;
    for (uint32_t v = 0; v <= k; ++v) {
        r.pw[v] = static_cast<uint32_t>(pw);
        pw *= ell;
    }
    r.q = r.pw[k];
    r.barrett = make_mod(r.q).barrett;
    return r;
}

__device__ __forceinline__ uint32_t pow_mod_d(uint32_t b, uint32_t e, uint32_t q, uint64_t barrett) {
    uint32_t r = 1 % q;
    while (e) {
        if (e & 1) r = mod_mul(r, b, q, barrett);
        b = mod_mul(b, b, q, barrett);
        e >>= 1;
    }
    return r;
}

// floor(2^64 / d) for 2 <= d < 2^32 (the Barrett constant of a small modulus)
__device__ __forceinline__ uint64_t make_barrett_d(uint32_t d) {
    const uint64_t q = ~0ull / d;  // floor((2^64 - 1) / d)
    return (q + 1) * d == 0 ? q + 1 : q;  // d divides 2^64 only for powers of two
}

__device__ __forceinline__ uint32_t val_k(uint32_t x, const RingK& R) {
    if (x == 0) return R.k;
    if (R.ell == 2) return min(static_cast<uint32_t>(__ffs(x) - 1), R.k);
    uint32_t v = 0;
    while (v < R.k && x % R.ell == 0) {
        x /= R.ell;
        ++v;
    }
    return v;
}

int grid_for(size_t work, int sms) {
    return static_cast<int>(std::max<size_t>(1, std::min<size_t>((work + 255) / 256, static_cast<size_t>(sms) * 8)));
}

// ---- small element-wise kernels --------------------------------------------------
__global__ void count_noncanonical_kernel(const uint32_t* __restrict__ A, uint64_t ld, int m, int n, uint32_t q,
                                          int* __restrict__ bad) {
    const size_t total = static_cast<size_t>(m) * n;
    for (size_t idx = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; idx < total;
         idx += static_cast<size_t>(gridDim.x) * blockDim.x)
        if (A[(idx / n) * ld + idx % n] >= q) atomicAdd(bad, 1);
}

// dst = src mod ell (compact m x n, ld dst_ld)
__global__ void mod_small_kernel(const uint32_t* __restrict__ src, uint64_t lds, int m, int n, uint32_t ell,
                                 uint32_t* __restrict__ dst, uint64_t ldd) {
    const size_t total = static_cast<size_t>(m) * n;
    for (size_t idx = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; idx < total;
         idx += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const int i = static_cast<int>(idx / n), j = static_cast<int>(idx % n);
        dst[static_cast<size_t>(i) * ldd + j] = src[static_cast<size_t>(i) * lds + j] % ell;
    }
}

// dst[i][j] = src[row0 + i][colmap[col0 + j]] / div  (exact division; div = 1 copies)
__global__ void gather_div_kernel(const uint32_t* __restrict__ src, uint64_t lds, int row0, int rows,
                                  const int* __restrict__ colmap, int col0, int cols, uint32_t div,
                                  uint32_t* __restrict__ dst, uint64_t ldd) {
    const size_t total = static_cast<size_t>(rows) * cols;
    for (size_t idx = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; idx < total;
         idx += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const int i = static_cast<int>(idx / cols), j = static_cast<int>(idx % cols);
        const uint32_t x = src[static_cast<size_t>(row0 + i) * lds + colmap[col0 + j]];
        dst[static_cast<size_t>(i) * ldd + j] = div == 1 ? x : x / div;
    }
}

// flags |= 1 when an entry is non-zero, |= 2 when one is a unit (not divisible by
// ell).  A warp leaves as one: its lanes may read the flags at different times, and
// the reduction below names all of them.
__global__ void __launch_bounds__(256) level_flags_kernel(const uint32_t* __restrict__ A, uint64_t ld, int m, int n,
                                                          uint32_t ell, int* __restrict__ flags) {
    for (int i = blockIdx.x; i < m; i += gridDim.x) {
        const int seen = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile int*>(flags), 0);
        if (seen == 3) return;
        int f = 0;
        for (int j = threadIdx.x; j < n; j += blockDim.x) {
            const uint32_t x = A[static_cast<size_t>(i) * ld + j];
            if (x != 0) f |= x % ell != 0 ? 3 : 1;
        }
        f = __reduce_or_sync(0xffffffffu, f);
        if ((threadIdx.x & 31) == 0 && (f & ~seen) != 0) atomicOr(flags, f);
    }
}

// dst[i][j] = src[row0 + i][col0 + j] / div (exact division; div = 1 copies), a row per CTA
__global__ void __launch_bounds__(256) copy_div_kernel(const uint32_t* __restrict__ src, uint64_t lds, int row0,
                                                       int rows, int col0, int cols, uint32_t div,
                                                       uint32_t* __restrict__ dst, uint64_t ldd) {
    for (int i = blockIdx.x; i < rows; i += gridDim.x) {
        const uint32_t* s = src + static_cast<size_t>(row0 + i) * lds + col0;
        for (int j = threadIdx.x; j < cols; j += blockDim.x)
            dst[static_cast<size_t>(i) * ldd + j] = div == 1 ? s[j] : s[j] / div;
    }
}

// The inverse of a unit u of Z/ell^k by Newton's iteration x <- x (2 - u x),
// which doubles the ell-adic precision per step: in 32-bit wraparound from
// x = u (right to 3 bits) for ell = 2; from the inverse mod ell,
// u^(ell - 2) mod ell, for odd ell (1 -> 2 -> 4 -> ... >= k digits).
__device__ __forceinline__ uint32_t ring_unit_inverse(uint32_t u, const RingK& R) {
    if (R.ell == 2) {
        uint32_t x = u;
        for (int i = 0; i < 5; ++i) x *= 2u - u * x;
        return R.k >= 32 ? x : (x & (R.q - 1u));
    }
    const uint32_t u0 = u % R.ell;
    uint32_t x = pow_mod_d(u0, R.ell - 2, R.ell, make_barrett_d(R.ell));
    for (uint32_t prec = 1; prec < R.k; prec *= 2) {
        const uint32_t ux = mod_mul(u % R.q, x, R.q, R.barrett);
        x = mod_mul(x, mod_sub(2u % R.q, ux, R.q), R.q, R.barrett);
    }
    return x;
}

// ---- the Sec. 13.5 pass ---------------------------------------------------------------
// The Howell form needs, for every pivot row P with pivot ell^v, v > 0, its
// closure ell^(k-v) P (zero in the pivot's column) reduced to zero by the rows
// below.  The form is unique, so the order is free: all echelon rows are
// normalised and their closures looked over at once (howell_rows_kernel); only
// the non-zero closures, and rows they displace, go through the sequential
// insertion (howell_insert_kernel).  Over a matrix whose closures vanish -- unit
// pivots, or rows with little right of their pivot -- nothing is sequential
// (the column-by-column pass took 5.1 ms for a 2048 x 2048 U D V over Z/2^16,
// 2.5 us a column).

// One CTA per echelon row i (pivot column pcol[i], an arbitrary unit times ell^v
// there): the stale multipliers left of the pivot to zero, the row scaled to
// lead with ell^v exactly; piv_id / piv_v of its column; lead[i] = the first
// non-zero column of its closure or n, counted in *nclose.
__global__ void __launch_bounds__(256) howell_rows_kernel(uint32_t* __restrict__ W, uint64_t ld, int n,
                                                          const int* __restrict__ pcol, const RingK R,
                                                          int* __restrict__ piv_id, int* __restrict__ piv_v,
                                                          int* __restrict__ lead, int* __restrict__ nclose) {
    __shared__ uint32_t s_ui;
    __shared__ int s_lead;
    const int i = blockIdx.x, c = pcol[i];
    uint32_t* P = W + static_cast<size_t>(i) * ld;
    const uint32_t x = P[c];
    const uint32_t v = val_k(x, R);
    if (threadIdx.x == 0) {
        s_ui = ring_unit_inverse(x / R.pw[v], R);
        s_lead = n;
    }
    __syncthreads();
    const uint32_t ui = s_ui, f = R.pw[R.k - v];
    int first = n;
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        const uint32_t y = j < c ? 0u : mod_mul(P[j], ui, R.q, R.barrett);
        P[j] = y;
        if (v > 0 && j > c && first == n && mod_mul(y, f, R.q, R.barrett) != 0) first = j;
    }
    if (first < n) atomicMin(&s_lead, first);
    __syncthreads();
    if (threadIdx.x == 0) {
        piv_id[c] = i;
        piv_v[c] = static_cast<int>(v);
        lead[i] = s_lead;
        if (s_lead < n) atomicAdd(nclose, 1);
    }
}

// The rows of the pass: echelon rows [0, r) in W, closures r, r + 1, .. in Z.
struct PassArgs {
    uint32_t* W;
    uint32_t* Z;
    uint64_t ld;
    int n, r, cap;   // cap: rows of the two stores together
    RingK R;
    int* piv_id;     // [n] row id of each column's pivot, -1 for none
    int* piv_v;      // [n]
    int* lead;       // [cap] work: leading column of every pending row, n for none (used when it does not fit shared memory)
    const int* first_lead;  // [r] from howell_rows_kernel
    int* closure;    // [r] the row id of an echelon row's closure, -1 where it is zero
    int* err;
    __device__ __forceinline__ uint32_t* row(int id) const {
        return id < r ? W + static_cast<size_t>(id) * ld : Z + static_cast<size_t>(id - r) * ld;
    }
};

// Stores the non-zero closures (ids r, r + 1, .. in echelon order; every CTA
// counts those before its row) and their leading columns.
__global__ void __launch_bounds__(256) howell_closures_kernel(const PassArgs a, const int* __restrict__ pcol,
                                                              int* __restrict__ lead_out) {
    const int i = blockIdx.x;
    const int z = a.first_lead[i];
    if (z >= a.n) {
        if (threadIdx.x == 0) a.closure[i] = -1;
        return;
    }
    int before = 0;
    for (int t = threadIdx.x; t < i; t += blockDim.x) before += a.first_lead[t] < a.n ? 1 : 0;
    __shared__ int s_before;
    if (threadIdx.x == 0) s_before = 0;
    __syncthreads();
    if (before) atomicAdd(&s_before, before);
    __syncthreads();
    const int id = a.r + s_before, c = pcol[i];
    const uint32_t f = a.R.pw[a.R.k - a.piv_v[c]];
    const uint32_t* P = a.row(i);
    uint32_t* Z = a.row(id);
    for (int j = threadIdx.x; j < a.n; j += blockDim.x) Z[j] = j > c ? mod_mul(P[j], f, a.R.q, a.R.barrett) : 0u;
    if (threadIdx.x == 0) {
        lead_out[s_before] = z;
        a.closure[i] = id;
    }
}

// The pending rows (the closures) inserted, one CTA.  Each round takes the
// smallest leading column c of a pending row; all of a column's rows are there
// when it comes up, so its pivot changes at most once: to the pending row of
// smallest valuation, if that is smaller than the pivot's.  Then the new
// pivot is normalised, its closure joins the pending rows, the old pivot row
// too, and every pending row of the column is reduced by the pivot, a warp
// each, which gives its next leading column.  The old pivot row's own closure
// leaves them, untouched so far (it starts right of the column): with the old
// pivot O = O' + ell^(w-v) P in terms of the new one, ell^(k-w) O = ell^(k-w) O' +
// ell^(k-v) P, a multiple of the reduced row and the new pivot's closure.  Kept, it
// would go on being reduced in every column: the whole call on a triangular 1024 x
// 1024 matrix over Z/2^31, random valuations on its diagonal, takes 39.7 ms with
// it and 17.6 without (30 ms with the column-by-column pass).
__global__ void __launch_bounds__(kHowellThreads) howell_insert_kernel(const PassArgs a, const int* __restrict__ lead0,
                                                                       int nclose, int smem_lead) {
    extern __shared__ int s_tab[];  // [cap] leading columns, when they fit
    __shared__ unsigned long long s_best;
    __shared__ int s_nel, s_c, s_nrows, s_zlead;
    __shared__ int s_el[kHowellThreads];
    __shared__ uint32_t s_ui;
    const RingK& R = a.R;
    int* lead = smem_lead ? s_tab : a.lead;
    const int none = a.n;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int i = threadIdx.x; i < a.cap; i += blockDim.x) lead[i] = i >= a.r && i < a.r + nclose ? lead0[i - a.r] : none;
    if (threadIdx.x == 0) {
        s_nrows = a.r + nclose;
        s_c = none;
    }
    __syncthreads();
    for (;;) {
        const int nrows = s_nrows;
        int c = none;
        for (int id = threadIdx.x; id < nrows; id += blockDim.x) c = min(c, lead[id]);
        c = __reduce_min_sync(0xffffffffu, c);
        if (lane == 0 && c < none) atomicMin(&s_c, c);
        if (threadIdx.x == 0) {
            s_best = ~0ull;
            s_nel = 0;
            s_zlead = none;
        }
        __syncthreads();
        c = s_c;
        if (c >= none) break;
        // the column's pending rows: the smallest (valuation, id) of all, a list of up to one CTA-size of them
        for (int id = threadIdx.x; id < nrows; id += blockDim.x) {
            if (lead[id] != c) continue;
            const uint32_t x = a.row(id)[c];
            atomicMin(&s_best, (static_cast<unsigned long long>(val_k(x, R)) << 32) | static_cast<unsigned>(id));
            const int slot = atomicAdd(&s_nel, 1);
            if (slot < kHowellThreads) s_el[slot] = id;
        }
        const int old = a.piv_id[c];
        const uint32_t old_v = old >= 0 ? static_cast<uint32_t>(a.piv_v[c]) : R.k;
        __syncthreads();
        const unsigned long long best = s_best;
        const bool change = static_cast<uint32_t>(best >> 32) < old_v;
        const int pid = change ? static_cast<int>(best & 0xffffffffu) : old;
        const uint32_t v = change ? static_cast<uint32_t>(best >> 32) : old_v;
        uint32_t* P = a.row(pid);
        int nel = min(s_nel, kHowellThreads);
        if (change) {
            if (threadIdx.x == 0) {
                s_ui = ring_unit_inverse(P[c] / R.pw[v], R);
                lead[pid] = none;
            }
            __syncthreads();
            const uint32_t ui = s_ui;
            for (int j = c + threadIdx.x; j < a.n; j += blockDim.x) P[j] = mod_mul(P[j], ui, R.q, R.barrett);
            __syncthreads();
            if (v > 0) {  // its closure
                if (nrows >= a.cap) {
                    if (threadIdx.x == 0) atomicCAS(a.err, 0, 64);  // store exhausted: cannot happen (one change per column)
                    return;
                }
                uint32_t* Z = a.row(nrows);
                const uint32_t f = R.pw[R.k - v];
                int first = none;
                for (int j = threadIdx.x; j < a.n; j += blockDim.x) {
                    const uint32_t z = j > c ? mod_mul(P[j], f, R.q, R.barrett) : 0u;
                    Z[j] = z;
                    if (z && first == none) first = j;
                }
                first = __reduce_min_sync(0xffffffffu, first);
                if (lane == 0 && first < none) atomicMin(&s_zlead, first);
            }
        }
        // R -= (R[c] / ell^v) P over columns [c, n): the listed rows and a displaced pivot
        for (int t = warp; t < nel + (change && old >= 0 ? 1 : 0); t += nw) {
            const int id = t < nel ? s_el[t] : old;
            if (id == pid) continue;
            uint32_t* Rw = a.row(id);
            const uint32_t f = Rw[c] / R.pw[v];
            __syncwarp();
            int first = none;
            for (int j = c + lane; j < a.n; j += 32) {
                const uint32_t y = mod_sub(Rw[j], mod_mul(f, P[j], R.q, R.barrett), R.q);
                Rw[j] = y;
                if (y != 0 && first == none) first = j;
            }
            first = __reduce_min_sync(0xffffffffu, first);
            if (lane == 0) lead[id] = first;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            if (change) {
                a.piv_id[c] = pid;
                a.piv_v[c] = static_cast<int>(v);
                // (an old pivot is an echelon row with its own column still: a column's pivot changes once)
                if (old >= 0 && a.closure[old] >= 0) lead[a.closure[old]] = none;
                if (s_zlead < none) {
                    lead[nrows] = s_zlead;
                    s_nrows = nrows + 1;
                }
            }
            s_c = none;
        }
        __syncthreads();
    }
}

// The pivots by column to lists: ids, columns, valuations and their number.
__global__ void __launch_bounds__(1024) howell_pivots_kernel(const int* __restrict__ piv_id,
                                                             const int* __restrict__ piv_v, int n,
                                                             int* __restrict__ ids, int* __restrict__ cols,
                                                             int* __restrict__ vals, int* __restrict__ count) {
    __shared__ int s_cnt[32], s_base;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_base = 0;
    __syncthreads();
    for (int c0 = 0; c0 < n; c0 += 1024) {
        const int c = c0 + threadIdx.x;
        const int id = c < n ? piv_id[c] : -1;
        const unsigned mask = __ballot_sync(0xffffffffu, id >= 0);
        if (lane == 0) s_cnt[warp] = __popc(mask);
        __syncthreads();
        int at = s_base + __popc(mask & ((1u << lane) - 1u)), all = s_base;
        for (int w = 0; w < 32; ++w) {
            if (w < warp) at += s_cnt[w];
            all += s_cnt[w];
        }
        if (id >= 0) {
            ids[at] = id;
            cols[at] = c;
            vals[at] = piv_v[c];
        }
        __syncthreads();
        if (threadIdx.x == 0) s_base = all;
        __syncthreads();
    }
    if (threadIdx.x == 0) *count = s_base;
}

// ---- blocked reduce-above --------------------------------------------------------------
// For the pivot block [t0, t0+b): Q[i][t] are the floor quotients of row i <
// t0 + b against the block's pivots applied in order (each quotient on the
// canonical residue after the previous ones; inside the block only by the
// pivots below the row), so that H[0 : t0+b] -= Q H[t0 : t0+b] reduces all of
// them at once.  A warp per row, two of the block's columns per lane: a pivot
// costs a shuffle and a compare where the quotient is 0.  (A thread per row with
// its 64 values in local memory and a separate triangle pass over the block:
// 36 + 28 us per block of a 2048 x 2048 form; this 7 us.)
__global__ void __launch_bounds__(256) reduce_quotients_kernel(const uint32_t* __restrict__ H, uint64_t ld, int t0,
                                                               int b, const int* __restrict__ pcol,
                                                               const int* __restrict__ pv, RingK R,
                                                               uint32_t* __restrict__ Q) {
    __shared__ uint32_t sB[kReduceBlock][kReduceBlock + 1];  // sB[t][t3] = H[t0+t][pcol[t0+t3]]
    __shared__ uint32_t sdiv[kReduceBlock];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int l0 = lane, l1 = lane + 32;
    const int pc0 = l0 < b ? pcol[t0 + l0] : 0, pc1 = l1 < b ? pcol[t0 + l1] : 0;
#pragma unroll 4
    for (int t = warp; t < b; t += 8) {
        const uint32_t* src = H + static_cast<size_t>(t0 + t) * ld;
        sB[t][l0] = l0 < b ? src[pc0] : 0u;
        sB[t][l1] = l1 < b ? src[pc1] : 0u;
    }
    for (int t = threadIdx.x; t < b; t += 256) sdiv[t] = R.pw[pv[t0 + t]];
    __syncthreads();
    const int i = static_cast<int>(blockIdx.x) * 8 + warp;
    if (i >= t0 + b) return;
    const uint32_t* src = H + static_cast<size_t>(i) * ld;
    uint32_t v0 = l0 < b ? src[pc0] : 0u, v1 = l1 < b ? src[pc1] : 0u;
    uint32_t q0 = 0, q1 = 0;
    for (int t = max(0, i - t0 + 1); t < b; ++t) {
        const uint32_t x = __shfl_sync(0xffffffffu, t < 32 ? v0 : v1, t & 31);
        const uint32_t d = sdiv[t];
        if (x < d) continue;  // the same in every lane
        const uint32_t qt = x / d;
        if (t < 32) q0 = lane == t ? qt : q0;
        else q1 = lane == t - 32 ? qt : q1;
        if (l0 > t) v0 = mod_sub(v0, mod_mul(qt, sB[t][l0], R.q, R.barrett), R.q);
        if (l1 > t) v1 = mod_sub(v1, mod_mul(qt, sB[t][l1], R.q, R.barrett), R.q);
    }
    uint32_t* dst = Q + static_cast<size_t>(i) * b;
    if (l0 < b) dst[l0] = q0;
    if (l1 < b) dst[l1] = q1;
}

// H[i] = row ids[i] of the pass's stores (h x n)
__global__ void gather_rows_by_id_kernel(const PassArgs a, const int* __restrict__ ids, int h, int n,
                                         uint32_t* __restrict__ H, uint64_t ldh) {
    const size_t total = static_cast<size_t>(h) * n;
    for (size_t idx = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; idx < total;
         idx += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const int i = static_cast<int>(idx / n), j = static_cast<int>(idx % n);
        H[static_cast<size_t>(i) * ldh + j] = a.row(ids[i])[j];
    }
}

size_t pad_ld(size_t cols) { return (cols + 15) / 16 * 16 + 16; }

void check_input(hme_ctx* ctx, const uint32_t* A, size_t ld, int m, int n, uint32_t q) {
    int* bad = static_cast<int*>(ctx->ws.get(kSlotElim6, 64));
    HME_CUDA(cudaMemsetAsync(bad, 0, sizeof(int), ctx->stream));
    HME_TIMED(ctx, "ring_check", count_noncanonical_kernel<<<grid_for(static_cast<size_t>(m) * n, ctx->num_sms), 256, 0,
                                                             ctx->stream>>>(A, ld, m, n, q, bad));
    int h = 0;
    HME_CUDA(cudaMemcpyAsync(&h, bad, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    HME_CUDA(cudaStreamSynchronize(ctx->stream));
    if (h) throw Error(HME_EINVAL, "input is not canonical mod ell^k (" + std::to_string(h) + " entries >= ell^k)");
}

}  // namespace

// ---- Smith valuations ------------------------------------------------------------------
// A level: the unit-pivot elimination over Z/ell^(k-s).  A column without a unit
// among the active rows is left out, and stays without one, since the rows that
// pivot later are 0 mod ell there too: so the pivots are the level's F_ell column
// rank profile, and the left-out columns of the remaining rows, updated to the
// end, are the Schur complement.  One elimination of the level matrix does it
// (keep_skipped); where its panels are too tall for that, the profile is found
// first by an elimination over F_ell, its columns move to the front, and the LU
// runs on them.  (Two eliminations per level: 16.2 ms for a 2048 x 2048 U D V over
// Z/3^10; one, with the compact panels: 6.8 ms.)
std::vector<uint32_t> smith_device(hme_ctx* ctx, uint32_t ell, uint32_t k, const uint32_t* A, size_t lda, int m,
                                   int n, const ElimOptions& opt) {
    std::vector<uint32_t> sigma;
    if (m == 0 || n == 0) return sigma;
    const RingK R0 = make_ring(ell, k);
    check_input(ctx, A, lda, m, n, R0.q);
    const bool keep = elim_can_keep(ctx, m, opt);
    // ping-pong buffers for the level matrices, padded leading dimension (with room for a level's
    // left-out columns)
    const size_t ld = pad_ld(keep ? 2 * static_cast<size_t>(n) : n);
    uint32_t* cur = static_cast<uint32_t*>(ctx->ws.get(kSlotRing0, sizeof(uint32_t) * static_cast<size_t>(m) * ld));
    uint32_t* nxt = static_cast<uint32_t*>(ctx->ws.get(kSlotRing1, sizeof(uint32_t) * static_cast<size_t>(m) * ld));
    uint32_t* tmp = keep ? nullptr
                         : static_cast<uint32_t*>(ctx->ws.get(kSlotRing2, sizeof(uint32_t) * static_cast<size_t>(m) * ld));
    int* d_map = static_cast<int*>(ctx->ws.get(kSlotRing3, sizeof(int) * (static_cast<size_t>(n) + 16)));
    int* d_flag = d_map + n;
    auto copy_div = [&](const uint32_t* src, size_t lds, int row0, int rows, int col0, int cols, uint32_t div,
                        uint32_t* dst) {
        HME_TIMED(ctx, "ring_gather", copy_div_kernel<<<std::min(rows, 16 * ctx->num_sms), 256, 0, ctx->stream>>>(
                                          src, lds, row0, rows, col0, cols, div, dst, ld));
        HME_CUDA(cudaGetLastError());
    };
    copy_div(A, lda, 0, m, 0, n, 1, cur);
    int rows = m, cols = n;
    for (uint32_t s = 0; s < k && rows > 0 && cols > 0; ++s) {
        const uint32_t kk = k - s;
        const RingK R = make_ring(ell, kk);
        // stop when the level matrix is zero: no further valuation < k; without a unit the level has
        // no invariant: divide by ell
        HME_CUDA(cudaMemsetAsync(d_flag, 0, sizeof(int), ctx->stream));
        HME_TIMED(ctx, "ring_nonzero", level_flags_kernel<<<std::min(rows, 8 * ctx->num_sms), 256, 0, ctx->stream>>>(
                                           cur, ld, rows, cols, ell, d_flag));
        int flags = 0;
        HME_CUDA(cudaMemcpyAsync(&flags, d_flag, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
        HME_CUDA(cudaStreamSynchronize(ctx->stream));
        if (flags == 0) break;
        if (flags == 1) {
            copy_div(cur, ld, 0, rows, 0, cols, ell, nxt);
            std::swap(cur, nxt);
            continue;
        }
        RingSpec rs;
        rs.ell = ell;
        rs.k = kk;
        rs.max_v = 0;
        if (keep) {
            rs.keep_skipped = true;
            const ElimResult lu = elim_device(ctx, make_mod(R.q), cur, ld, rows, cols, false, nullptr, 0, opt, &rs);
            for (int t = 0; t < lu.rank; ++t) sigma.push_back(s);
            const int nr = rows - lu.rank, nc = lu.appended;
            if (nr > 0 && nc > 0) copy_div(cur, ld, lu.rank, nr, cols, nc, ell, nxt);
            std::swap(cur, nxt);
            rows = nr;
            cols = nc;
            continue;
        }
        // (1) the F_ell column rank profile of the level matrix
        HME_TIMED(ctx, "ring_mod", mod_small_kernel<<<grid_for(static_cast<size_t>(rows) * cols, ctx->num_sms), 256, 0,
                                                      ctx->stream>>>(cur, ld, rows, cols, ell, tmp, ld));
        const ElimResult prof = elim_device(ctx, make_mod(ell), tmp, ld, rows, cols, false, nullptr, 0, opt);
        const int r = prof.rank;
        // (2) profile columns to the front, then the rest in order
        std::vector<int> cmap;
        cmap.reserve(cols);
        {
            std::vector<char> isp(cols, 0);
            for (int c : prof.pivots) {
                isp[c] = 1;
                cmap.push_back(c);
            }
            for (int c = 0; c < cols; ++c)
                if (!isp[c]) cmap.push_back(c);
        }
        HME_CUDA(cudaMemcpyAsync(d_map, cmap.data(), sizeof(int) * cols, cudaMemcpyHostToDevice, ctx->stream));
        HME_TIMED(ctx, "ring_gather", gather_div_kernel<<<grid_for(static_cast<size_t>(rows) * cols, ctx->num_sms), 256, 0,
                                                          ctx->stream>>>(cur, ld, 0, rows, d_map, 0, cols, 1, nxt, ld));
        // (3) unit-pivot LU of the first r columns over Z/ell^kk
        rs.lu_cols = r;
        const ElimResult lu = elim_device(ctx, make_mod(R.q), nxt, ld, rows, cols, false, nullptr, 0, opt, &rs);
        if (lu.rank != r)
            throw Error(HME_EINVAL, "smith: unit-pivot LU found " + std::to_string(lu.rank) + " pivots, expected " +
                                        std::to_string(r));
        for (int t = 0; t < r; ++t) sigma.push_back(s);
        // (4) the Schur complement divided by ell is the next level
        const int nr = rows - r, nc = cols - r;
        if (nr > 0 && nc > 0) copy_div(nxt, ld, r, nr, r, nc, ell, cur);
        rows = nr;
        cols = nc;
    }
    check_device_error(ctx);
    return sigma;
}

// ---- Howell form ----------------------------------------------------------------------
HowellOut howell_device(hme_ctx* ctx, uint32_t ell, uint32_t k, const uint32_t* A, size_t lda, int m, int n,
                        uint32_t* Hout, size_t ldout, const ElimOptions& opt) {
    HowellOut out;
    if (m == 0 || n == 0) return out;
    const RingK R = make_ring(ell, k);
    check_input(ctx, A, lda, m, n, R.q);
    const size_t ld = pad_ld(n);
    uint32_t* W = static_cast<uint32_t*>(ctx->ws.get(kSlotRing0, sizeof(uint32_t) * static_cast<size_t>(m) * ld));
    HME_TIMED(ctx, "ring_gather", copy_div_kernel<<<std::min(m, 16 * ctx->num_sms), 256, 0, ctx->stream>>>(
                                      A, lda, 0, m, 0, n, 1, W, ld));
    HME_CUDA(cudaGetLastError());
    // (1) minimal-valuation echelon (same row span)
    RingSpec rs;
    rs.ell = ell;
    rs.k = k;
    rs.max_v = k - 1;
    rs.lu_cols = n;
    ElimOptions o = opt;
    const ElimResult lu = elim_device(ctx, make_mod(R.q), W, ld, m, n, false, nullptr, 0, o, &rs);
    const int r = lu.rank;
    if (r == 0) return out;
    // (2) the Sec. 13.5 pass
    int* d_idx = static_cast<int*>(ctx->ws.get(kSlotRing2, sizeof(int) * (8 * static_cast<size_t>(n) + 64)));
    int* d_pid = d_idx;
    int* d_pcol = d_idx + n;
    int* d_pv = d_idx + 2 * n;
    int* d_piv_id = d_idx + 3 * n;   // by column
    int* d_piv_v = d_idx + 4 * n;
    int* d_lead = d_idx + 5 * n;     // of the echelon rows' closures
    int* d_lead0 = d_idx + 6 * n;    // of the non-zero closures, in order
    int* d_closure = d_idx + 7 * n;  // the echelon rows' closures' ids
    int* d_cnt = d_idx + 8 * n;      // non-zero closures, pivots
    HME_CUDA(cudaMemcpyAsync(d_pcol, lu.pivots.data(), sizeof(int) * r, cudaMemcpyHostToDevice, ctx->stream));
    HME_CUDA(cudaMemsetAsync(d_piv_id, 0xff, sizeof(int) * n, ctx->stream));
    HME_CUDA(cudaMemsetAsync(d_cnt, 0, 2 * sizeof(int), ctx->stream));
    HME_TIMED(ctx, "howell_rows", howell_rows_kernel<<<r, 256, 0, ctx->stream>>>(W, ld, n, d_pcol, R, d_piv_id, d_piv_v,
                                                                                d_lead, d_cnt));
    HME_CUDA(cudaGetLastError());
    int nclose = 0;
    HME_CUDA(cudaMemcpyAsync(&nclose, d_cnt, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    HME_CUDA(cudaStreamSynchronize(ctx->stream));
    PassArgs pa{};
    pa.W = W;
    pa.ld = ld;
    pa.n = n;
    pa.r = r;
    pa.R = R;
    pa.piv_id = d_piv_id;
    pa.piv_v = d_piv_v;
    pa.first_lead = d_lead;
    pa.closure = d_closure;
    pa.err = ctx->d_err;
    if (nclose > 0) {
        // the closures and, per column, at most one more of a new pivot; the leading columns beside them
        const size_t zrows = static_cast<size_t>(nclose) + n;
        pa.cap = r + static_cast<int>(zrows);
        const size_t lead_bytes = sizeof(int) * static_cast<size_t>(pa.cap);
        pa.Z = static_cast<uint32_t*>(ctx->ws.get(kSlotRing1, sizeof(uint32_t) * zrows * ld + lead_bytes));
        pa.lead = reinterpret_cast<int*>(pa.Z + zrows * ld);
        HME_TIMED(ctx, "howell_pass", howell_closures_kernel<<<r, 256, 0, ctx->stream>>>(pa, d_pcol, d_lead0));
        HME_CUDA(cudaGetLastError());
        const int in_smem = lead_bytes <= kHowellLeadSmemMax ? 1 : 0;
        static OncePerDevice attr;
        attr.run([](int) {
            HME_CUDA(cudaFuncSetAttribute(howell_insert_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          static_cast<int>(kHowellLeadSmemMax)));
        });
        HME_TIMED(ctx, "howell_pass", howell_insert_kernel<<<1, kHowellThreads, in_smem ? lead_bytes : 0, ctx->stream>>>(
                                          pa, d_lead0, nclose, in_smem));
        HME_CUDA(cudaGetLastError());
    }
    HME_TIMED(ctx, "howell_rows", howell_pivots_kernel<<<1, 1024, 0, ctx->stream>>>(d_piv_id, d_piv_v, n, d_pid, d_pcol,
                                                                                  d_pv, d_cnt + 1));
    HME_CUDA(cudaGetLastError());
    int h = 0;
    HME_CUDA(cudaMemcpyAsync(&h, d_cnt + 1, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    check_device_error(ctx);
    out.pivots.resize(h);
    out.pivot_v.resize(h);
    if (h == 0) return out;
    HME_CUDA(cudaMemcpyAsync(out.pivots.data(), d_pcol, sizeof(int) * h, cudaMemcpyDeviceToHost, ctx->stream));
    HME_CUDA(cudaMemcpyAsync(out.pivot_v.data(), d_pv, sizeof(int) * h, cudaMemcpyDeviceToHost, ctx->stream));
    // (3) H = the pivot rows in pivot order, then the blocked reduce-above
    const size_t ldh = ld;
    uint32_t* H = static_cast<uint32_t*>(ctx->ws.get(kSlotRing4, sizeof(uint32_t) * static_cast<size_t>(h) * ldh));
    HME_TIMED(ctx, "ring_gather", gather_rows_by_id_kernel<<<grid_for(static_cast<size_t>(h) * n, ctx->num_sms), 256, 0,
                                                             ctx->stream>>>(pa, d_pid, h, n, H, ldh));
    HME_CUDA(cudaStreamSynchronize(ctx->stream));
    uint32_t* Q = static_cast<uint32_t*>(ctx->ws.get(kSlotRing5, sizeof(uint32_t) * static_cast<size_t>(h) * kReduceBlock));
    const ModParams mq = make_mod(R.q);
    for (int t0 = 0; t0 < h; t0 += kReduceBlock) {
        const int b = std::min(kReduceBlock, h - t0);
        const int c0 = out.pivots[t0];
        if (t0 + b == 1) continue;
        HME_TIMED(ctx, "reduce_quot", reduce_quotients_kernel<<<(t0 + b + 7) / 8, 256, 0, ctx->stream>>>(
                                          H, ldh, t0, b, d_pcol, d_pv, R, Q));
        HME_CUDA(cudaGetLastError());
        // on a tensor-core variant: the block's own rows are among the reduced ones (C aliases B, which
        // is read through its limb planes)
        gemm_u32_variant(ctx, mq, t0 + b, n - c0, b, Q, b, H + static_cast<size_t>(t0) * ldh + c0, ldh, H + c0, ldh,
                         HME_SUB, gemm_default_variant(ctx, mq, t0 + b, n - c0));
    }
    check_device_error(ctx);
    // straight to the caller's rows (a host copy of the form in between cost 9 of 18 ms at 2048 x 2048)
    HME_CUDA(cudaMemcpy2DAsync(Hout, sizeof(uint32_t) * ldout, H, sizeof(uint32_t) * ldh, sizeof(uint32_t) * n, h,
                               cudaMemcpyDeviceToHost, ctx->stream));
    HME_CUDA(cudaStreamSynchronize(ctx->stream));
    return out;
}

}  // namespace hme

// ---- C ABI ---------------------------------------------------------------------------------
using namespace hme;

namespace {
void check_ring(uint32_t ell, uint32_t k) {
    HME_REQUIRE(k >= 1, "ring: k must be >= 1");
    HME_REQUIRE(ell >= 2 && is_prime_u32(ell), "ring: ell must be a prime");
    uint64_t q = 1;
    for (uint32_t i = 0; i < k; ++i) {
        q *= ell;
        HME_REQUIRE(q < (1ull << 32), "ring: ell^k must be < 2^32");
    }
}
}  // namespace

extern "C" {

int hme_howell_u32(hme_ctx* ctx, uint32_t ell, uint32_t k, uint32_t m, uint32_t n, const uint32_t* A, size_t lda,
                   uint32_t* H, size_t ldh, uint32_t* pivots, uint32_t* pivot_v, uint32_t* h) {
    return guard([&] {
        HME_REQUIRE(ctx && h, "null argument");
        check_ring(ell, k);
        bind(ctx);
        *h = 0;
        if (m == 0 || n == 0) return;
        HME_REQUIRE(A && lda >= n && H && ldh >= n && pivots && pivot_v, "bad buffers");
        uint32_t* d = static_cast<uint32_t*>(ctx->ws.get(kSlotStageA, sizeof(uint32_t) * static_cast<size_t>(m) * n));
        HME_CUDA(cudaMemcpy2DAsync(d, sizeof(uint32_t) * n, A, sizeof(uint32_t) * lda, sizeof(uint32_t) * n, m,
                                   cudaMemcpyHostToDevice, ctx->stream));
        const HowellOut r = howell_device(ctx, ell, k, d, n, m, n, H, ldh, ctx->elim);
        const uint32_t hh = static_cast<uint32_t>(r.pivots.size());
        for (uint32_t i = 0; i < hh; ++i) {
            pivots[i] = r.pivots[i];
            pivot_v[i] = r.pivot_v[i];
        }
        *h = hh;
    });
}

int hme_smith_u32(hme_ctx* ctx, uint32_t ell, uint32_t k, uint32_t m, uint32_t n, const uint32_t* A, size_t lda,
                  uint32_t* sigma, uint32_t* count) {
    return guard([&] {
        HME_REQUIRE(ctx && count, "null argument");
        check_ring(ell, k);
        bind(ctx);
        *count = 0;
        if (m == 0 || n == 0) return;
        HME_REQUIRE(A && lda >= n && sigma, "bad buffers");
        uint32_t* d = static_cast<uint32_t*>(ctx->ws.get(kSlotStageA, sizeof(uint32_t) * static_cast<size_t>(m) * n));
        HME_CUDA(cudaMemcpy2DAsync(d, sizeof(uint32_t) * n, A, sizeof(uint32_t) * lda, sizeof(uint32_t) * n, m,
                                   cudaMemcpyHostToDevice, ctx->stream));
        const std::vector<uint32_t> s = smith_device(ctx, ell, k, d, n, m, n, ctx->elim);
        for (size_t i = 0; i < s.size(); ++i) sigma[i] = s[i];
        *count = static_cast<uint32_t>(s.size());
    });
}

}  // extern "C"
