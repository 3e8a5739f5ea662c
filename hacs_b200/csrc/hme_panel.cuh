// Panel arithmetic and the top-block inversion, shared by the single-matrix
// elimination (elim.cu) and the batched ranks (rank_rounds.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "hme_mod.h"
#include "hme_ptx.cuh"

namespace hme {
namespace panel {

constexpr int kMaxPanel = 128;
constexpr uint32_t kNoKey32 = 0xffffffffu;

// Inverse of a unit u of Z/q, q = ell^k, without divisions on the slow path:
//   ell = 2: Newton's iteration x <- x (2 - u x) in native 32-bit wraparound
//            (each step doubles the correct low bits), then reduced mod 2^k;
//   k > 1:   the inverse mod ell (binary extended gcd) lifted by the same
//            iteration mod q (Hensel), doubling the ell-adic precision;
//   k = 1:   the binary extended gcd mod the odd prime q.
__device__ __forceinline__ uint32_t inv_binary_xgcd(uint32_t u, uint32_t q) {
    // invariant: x1 * u == a (mod q), x2 * u == b (mod q), q odd.  Bounded:
    // each pass shrinks a + b by at least one bit position or a subtraction,
    // so 128 passes cover 32-bit operands; a non-unit (gcd > 1) returns 0.
    if (u == 0) return 0;
    uint32_t a = u, b = q, x1 = 1, x2 = 0;
    for (int guard_it = 0; a != 1 && b != 1; ++guard_it) {
        if (a == 0 || b == 0 || guard_it > 128) return 0;
        while ((a & 1) == 0) {
            a >>= 1;
            x1 = (x1 & 1) ? static_cast<uint32_t>((static_cast<uint64_t>(x1) + q) >> 1) : x1 >> 1;
        }
        while ((b & 1) == 0) {
            b >>= 1;
            x2 = (x2 & 1) ? static_cast<uint32_t>((static_cast<uint64_t>(x2) + q) >> 1) : x2 >> 1;
        }
        if (a >= b) {
            a -= b;
            x1 = x1 >= x2 ? x1 - x2 : static_cast<uint32_t>(static_cast<uint64_t>(x1) + q - x2);
        } else {
            b -= a;
            x2 = x2 >= x1 ? x2 - x1 : static_cast<uint32_t>(static_cast<uint64_t>(x2) + q - x1);
        }
    }
    return a == 1 ? x1 : x2;
}

// The ring Z/q, q = ell^k (k = 1: the field F_ell), as the elimination sees it.
struct Ring {
    uint32_t q;          // modulus
    uint64_t barrett;    // floor(2^64 / q)
    uint32_t ell, k;
    uint32_t max_v;      // pivots of valuation <= max_v only (0: unit pivots)
    uint32_t mont_qinv;  // q odd: -q^-1 mod 2^32 (Montgomery reduction)
    uint32_t mont_r2;    // q odd: 2^64 mod q
    uint32_t pw[32];     // ell^0 .. ell^k
};

// Montgomery product x * y * 2^-32 mod q for odd q < 2^32 and x, y < q: the
// sum T + m q may carry out of 64 bits when q > 2^31, so the carry is kept.
__device__ __forceinline__ uint32_t mont_mul(uint32_t x, uint32_t y, uint32_t q, uint32_t qinv) {
    const uint64_t t = static_cast<uint64_t>(x) * y;
    const uint32_t mq = static_cast<uint32_t>(t) * qinv;
    const uint64_t u = t + static_cast<uint64_t>(mq) * q;
    const uint64_t r = (u >> 32) + (u < t ? (1ull << 32) : 0ull);  // < 2q
    return static_cast<uint32_t>(r >= q ? r - q : r);
}

// The same for odd q < 2^31: no carry out of 64 bits.
__device__ __forceinline__ uint32_t mont_mul31(uint32_t x, uint32_t y, uint32_t q, uint32_t qinv) {
    const uint64_t t = static_cast<uint64_t>(x) * y;
    const uint32_t mq = static_cast<uint32_t>(t) * qinv;
    const uint32_t r = static_cast<uint32_t>((t + static_cast<uint64_t>(mq) * q) >> 32);
    return min(r, r - q);
}

// u^(q-2) mod q (Fermat) for an odd prime q, two bits of the exponent at a time
// in the Montgomery domain: about 3/2 log2 q dependent products.
template <bool BELOW31>
__device__ __forceinline__ uint32_t inv_fermat_as(uint32_t u, const Ring& R) {
    const uint32_t q = R.q, qi = R.mont_qinv;
    auto mul = [&](uint32_t x, uint32_t y) { return BELOW31 ? mont_mul31(x, y, q, qi) : mont_mul(x, y, q, qi); };
    const uint32_t u1 = mul(u, R.mont_r2);  // u * 2^32 mod q
    const uint32_t u2 = mul(u1, u1), u3 = mul(u2, u1);
    const uint32_t e = q - 2;  // >= 1
    int b = (31 - __clz(e)) & ~1;
    uint32_t d = (e >> b) & 3u;
    uint32_t r = d == 1 ? u1 : d == 2 ? u2 : u3;
    for (b -= 2; b >= 0; b -= 2) {
        r = mul(r, r);
        r = mul(r, r);
        d = (e >> b) & 3u;
        if (d) r = mul(r, d == 1 ? u1 : d == 2 ? u2 : u3);
    }
    return mul(r, 1u);  // out of the Montgomery domain
}
__device__ __forceinline__ uint32_t inv_fermat(uint32_t u, const Ring& R) {
    return R.q < (1u << 31) ? inv_fermat_as<true>(u, R) : inv_fermat_as<false>(u, R);
}

__device__ __forceinline__ uint32_t unit_inverse(uint32_t u, const Ring& R) {
    if (R.k == 1 && R.ell != 2) return inv_fermat(u % R.q, R);
    if (R.ell == 2) {
        uint32_t x = u;  // correct to 3 bits for odd u
        for (int i = 0; i < 5; ++i) x *= 2u - u * x;
        return R.k >= 32 ? x : (x & (R.q - 1));
    }
    if (R.k == 1) return inv_binary_xgcd(u % R.q, R.q);
    uint32_t x = inv_binary_xgcd(u % R.ell, R.ell);  // inverse mod ell
    for (uint32_t prec = 1; prec < R.k; prec *= 2) {
        const uint32_t ux = mod_mul(u, x, R.q, R.barrett);
        x = mod_mul(x, mod_sub(2u % R.q, ux, R.q), R.q, R.barrett);
    }
    return x;
}

// ell-adic valuation of x != 0, capped at cap + 1 (enough to reject a candidate).
__device__ __forceinline__ uint32_t valuation(uint32_t x, const Ring& R, uint32_t cap) {
    if (R.ell == 2) return min(static_cast<uint32_t>(__ffs(x) - 1), cap + 1);
    uint32_t v = 0;
    while (v <= cap && x % R.ell == 0) {
        x /= R.ell;
        ++v;
    }
    return v;
}

// kArithMont13: q < 2^13, where two products, or a sub-panel's seventeen, sum in
// one 32-bit word.
enum : int { kArithPow2 = 0, kArithMont31 = 1, kArithMont32 = 2, kArithMont13 = 3 };
constexpr uint32_t kMont13Max = 1u << 13;

// x / ell^v for x divisible by ell^v
__device__ __forceinline__ uint32_t div_pw(uint32_t x, uint32_t v, const Ring& R) {
    return v == 0 ? x : R.ell == 2 ? x >> v : x / R.pw[v];
}

// The negated multiplier as the row update wants it.
template <int ARITH>
__device__ __forceinline__ uint32_t ff_negate(uint32_t xp, const Ring& R) {
    if constexpr (ARITH == kArithPow2) return 0u - xp;
    else return xp == 0 ? 0u : R.q - xp;
}

// (w * y + xn * pr) * rho mod q, xn the negated multiplier (ff_negate)
template <int ARITH>
__device__ __forceinline__ uint32_t ff_update(uint32_t w, uint32_t y, uint32_t xn, uint32_t pr, const Ring& R) {
    if constexpr (ARITH == kArithPow2) {
        return (w * y + xn * pr) & (R.q - 1u);
    } else if constexpr (ARITH == kArithMont13) {
        const uint32_t t = w * y + xn * pr;  // < 2^27: the low words of t + m q cancel, with a carry unless t = 0
        const uint32_t r = __umulhi(t * R.mont_qinv, R.q) + (t != 0 ? 1u : 0u);
        return min(r, r - R.q);
    } else if constexpr (ARITH == kArithMont31) {
        // q < 2^31: both products < 2^62, t < 2^63, t + m q < 2^64
        const uint64_t t = static_cast<uint64_t>(w) * y + static_cast<uint64_t>(xn) * pr;
        const uint32_t mq = static_cast<uint32_t>(t) * R.mont_qinv;
        const uint32_t r = static_cast<uint32_t>((t + static_cast<uint64_t>(mq) * R.q) >> 32);
        return r >= R.q ? r - R.q : r;
    } else {
        return mod_add(mont_mul(w, y, R.q, R.mont_qinv), mont_mul(xn, pr, R.q, R.mont_qinv), R.q);
    }
}

struct BlockArgs {
    uint32_t* A;
    uint64_t ld;
    int m, r0, c0, w;
    Ring R;
    int* pivot_rows;  // [w] out
    int* pivot_cols;  // [w] out
    int* k_out;       // out
    int* ok;          // out: 1 when the top block settled the panel, else 0
    uint32_t* binv;   // out: B^-1 (nb x nb, row-major)
    uint32_t* diag;   // out when non-null: the classical pivots, at r0 ..
};

constexpr int kSubCols = 16;  // columns of a sub-panel

// Row stride of the block in words: whole 16-byte pieces, an odd number of
// them, so that eight lanes reading the same piece of eight rows hit 32 banks.
__host__ __device__ constexpr int block_stride(int w) {
    return (((w + 3) / 4) & 1) ? (w + 3) / 4 * 4 : (w + 3) / 4 * 4 + 4;
}
__host__ __device__ constexpr size_t block_smem_bytes(int rs, int w) {
    return sizeof(uint32_t) * static_cast<size_t>(rs + kSubCols) * block_stride(w);
}

// (w y + xn pr) rho on the four words of a piece
template <int ARITH>
__device__ __forceinline__ uint4 ff_update4(uint32_t w, uint4 y, uint32_t xn, uint4 pr, const Ring& R) {
    return make_uint4(ff_update<ARITH>(w, y.x, xn, pr.x, R), ff_update<ARITH>(w, y.y, xn, pr.y, R),
                      ff_update<ARITH>(w, y.z, xn, pr.z, R), ff_update<ARITH>(w, y.w, xn, pr.w, R));
}
// A sum of at most 17 products below q^2, reduced: two Montgomery steps (the
// sum times rho^2) for odd q, the truncation for q = 2^k.  The first step
// leaves at most 9.5 q + 1, the second at most q.
template <int ARITH>
__device__ __forceinline__ uint32_t ff_reduce96(uint32_t a0, uint32_t a1, uint32_t a2, const Ring& R) {
    if constexpr (ARITH == kArithPow2) {
        return a0 & (R.q - 1u);
    } else {
        uint32_t m = a0 * R.mont_qinv;
        // (a2:a1:a0 + m q) / 2^32: the low words cancel, with a carry unless both are zero
        uint64_t v = (static_cast<uint64_t>(a2) << 32 | a1) + __umulhi(m, R.q) + (a0 != 0 ? 1u : 0u);
        m = static_cast<uint32_t>(v) * R.mont_qinv;
        v = (v >> 32) + __umulhi(m, R.q) + (static_cast<uint32_t>(v) != 0 ? 1u : 0u);
        return static_cast<uint32_t>(v >= R.q ? v - R.q : v);
    }
}

// x y rho (x y for q = 2^k)
template <int ARITH>
__device__ __forceinline__ uint32_t ff_mul(uint32_t x, uint32_t y, const Ring& R) {
    if constexpr (ARITH == kArithPow2) return (x * y) & (R.q - 1u);
    else if constexpr (ARITH == kArithMont32) return mont_mul(x, y, R.q, R.mont_qinv);
    else return mont_mul31(x, y, R.q, R.mont_qinv);
}
// x y rho^2 (x y for q = 2^k)
template <int ARITH>
__device__ __forceinline__ uint32_t ff_scale2(uint32_t x, uint32_t y, const Ring& R) {
    if constexpr (ARITH == kArithPow2) return (x * y) & (R.q - 1u);
    else return ff_mul<ARITH>(ff_mul<ARITH>(x, y, R), 1u, R);
}

// One CTA of 4 RS threads, RS row slots: blocked in-place Gauss-Jordan
// inversion of the block with the pivot search, in sub-panels of 16 columns.
// The block sits in shared memory row-major; lanes over rows, four thread
// groups over 16-byte pieces of the rows.
//
// Steps of a sub-panel touch its 16 columns only (a piece per thread, kept in
// registers): step t takes the topmost unpivoted row with a unit in column t
// and updates every other row, pivoted or not, fraction-free as in the cluster
// kernel: row <- (w row - x pivot row) rho; one CTA barrier per step (column
// t + 1's entries and candidates leave step t through s_x and s_cand).  Column t
// then holds the column of the inverse that belongs to the pivot row: before
// the step that column is S_t (the rows' common scale, S_0 = 1, S_t+1 = S_t w_t
// rho) in the pivot row and 0 elsewhere.  After n steps pivot row t holds S_n /
// (S_t rho) times its row of the sub-panel's inverse.  With V the scale of the
// block before the sub-panel (V_0 = 1, V <- V S_n rho^2), the pivot rows take a
// product by S_t V rho; C (rows x 16) is then S_n times the left factor of the
// sub-panel's update (V S_n times it in the pivot rows, whose block carries a
// V^-1), and the other columns take
//   y <- (S_n y [row not a pivot of this sub-panel] + sum_t C_t P_t) rho^2
// with the pivot rows' values P from before the sub-panel: 16 products per
// entry reduced once instead of 16 reduced updates.  The sub-panel's own
// columns, columns of the inverse, are multiplied by V rho^2.  At the end every entry is V times its value: one modular inverse for
// the whole block.
//
// Bound by the chain of w steps and by the multiplier (a reduced update is
// three wide products).  A 64-column panel mod 2^31 - 19: 43 + 20 us as one
// CTA's LU and row solves over the GPU, 49 us as 64 whole-row steps, 35 us so
// (cycles: 16 steps of a sub-panel 9700, its update 6000, four times, while every warp
// kept the running scale in step; the inverse
// and the write 10300 before one warp inverted, two exponent bits at a time, and the
// write took Montgomery products);
// mod 13 (96 slots) 46 us with the wide products of kArithMont31 and 40 us with
// kArithMont13, where the cluster search of 10515 rows took 200 to 270.
template <int ARITH, int RS>
__device__ bool block_inverse(const BlockArgs& a, uint32_t* s_blk) {
    __shared__ uint32_t s_w[kMaxPanel], s_S[kMaxPanel + 1], s_V[kMaxPanel / kSubCols + 2];  // the last word: the scale's inverse
    __shared__ uint32_t s_x[2][RS];  // the rows' entries in the step's column, by parity
    __shared__ int s_prow[kMaxPanel];
    __shared__ int s_cand[2][RS / 32];
    constexpr int NT = 4 * RS, NW = NT / 32;
    constexpr int WC = RS == 128 ? 4 : 2;  // panels of up to 128 or 64 columns: 32 WC
    const int w = a.w, rows = a.m - a.r0, nb = min(w, rows), nbr = min(RS, rows);
    const Ring& R = a.R;
    const int ls = block_stride(w), nq = (w + 3) / 4;
    uint32_t* T = s_blk;             // [RS][ls]
    uint32_t* P = s_blk + RS * ls;   // [16][ls]: a sub-panel's pivot rows before it
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int li = tid % RS, g = tid / RS, wg = warp % (RS / 32);
    {
        // the block's rows, all of a thread's loads in flight at once
        uint32_t v[RS / NW][WC];
#pragma unroll
        for (int i = 0; i < RS / NW; ++i) {
            const int r = warp + NW * i;
            const uint32_t* src = a.A + static_cast<size_t>(a.r0 + min(r, nbr - 1)) * a.ld + a.c0;
#pragma unroll
            for (int c = 0; c < WC; ++c) v[i][c] = lane + 32 * c < w ? src[lane + 32 * c] : 0u;
        }
#pragma unroll
        for (int i = 0; i < RS / NW; ++i)
#pragma unroll
            for (int c = 0; c < WC; ++c)
                if (lane + 32 * c < 4 * nq) T[(warp + NW * i) * ls + lane + 32 * c] = v[i][c];
    }
    __syncthreads();
    auto is_unit = [&](uint32_t x) { return x != 0 && (R.k == 1 || x % R.ell != 0); };
    const bool in = li < nbr;
    bool pivoted = !in;
    uint32_t* row = T + li * ls;
    uint32_t V = 1u;
    for (int cs = 0, sub = 0; cs < nb; cs += kSubCols, ++sub) {
        const int ns = min(kSubCols, nb - cs);  // steps of this sub-panel
        const int q0 = cs >> 2, q1 = (cs + ns + 3) >> 2;  // its pieces
        const int qg = q0 + g;                  // this thread's piece of it
        const bool live = qg < q1;
        uint4 y = live ? *reinterpret_cast<const uint4*>(row + 4 * qg) : make_uint4(0, 0, 0, 0);
        if (g == 0) {
            s_x[0][li] = y.x;
            const unsigned mask = __ballot_sync(0xffffffffu, !pivoted && is_unit(y.x));
            if (lane == 0) s_cand[0][wg] = mask ? 32 * wg + __ffs(mask) - 1 : RS;
        }
        if (tid == 0) s_S[cs] = 1u;
        int mine = -1;  // the step of this sub-panel whose pivot is this thread's row
        __syncthreads();
        // step 4 u + C; false when its column has no unit in the block (the same in every thread)
        auto step = [&](auto cc, int u) -> bool {
            constexpr int C = decltype(cc)::value;
            constexpr int par = C & 1;
            const int t = cs + 4 * u + C;
            int prow = s_cand[par][0];
#pragma unroll
            for (int v = 1; v < RS / 32; ++v) prow = min(prow, s_cand[par][v]);
            if (prow == RS) return false;
            uint4 p4 = *reinterpret_cast<const uint4*>(T + prow * ls + 4 * min(qg, nq - 1));
            const uint32_t wt = s_x[par][prow], S = s_S[t];
            const uint32_t xn = ff_negate<ARITH>(s_x[par][li], R);
            if (tid == 0) {
                s_w[t] = wt;
                s_prow[t] = prow;
            }
            const bool is_pivot = li == prow;
            if (is_pivot) {
                pivoted = true;
                mine = 4 * u + C;
            }
            if (u == g) {  // column t: 0 in the other rows, S in the pivot row (nobody reads that word in this step)
                (C == 0 ? p4.x : C == 1 ? p4.y : C == 2 ? p4.z : p4.w) = S;
                (C == 0 ? y.x : C == 1 ? y.y : C == 2 ? y.z : y.w) = is_pivot ? S : 0u;
            }
            const uint4 z = ff_update4<ARITH>(wt, y, xn, p4, R);
            if (!is_pivot) y = z;
            if (live) *reinterpret_cast<uint4*>(row + 4 * qg) = y;
            if ((C == 3 ? u + 1 : u) == g) {  // the group of column t + 1
                const uint32_t next = C == 0 ? y.y : C == 1 ? y.z : C == 2 ? y.w : y.x;
                s_x[par ^ 1][li] = next;
                const unsigned mask = __ballot_sync(0xffffffffu, !pivoted && is_unit(next));
                if (lane == 0) s_cand[par ^ 1][wg] = mask ? 32 * wg + __ffs(mask) - 1 : RS;
            }
            if (warp == 0) {
                const uint32_t Sn = ff_mul<ARITH>(S, wt, R);
                if (lane == 0) s_S[t + 1] = Sn;
            }
            __syncthreads();
            return true;
        };
        bool ok = true;
        for (int u = 0; ok && 4 * u < ns; ++u) {
            ok = step(std::integral_constant<int, 0>{}, u);
            if (ok && 4 * u + 1 < ns) ok = step(std::integral_constant<int, 1>{}, u);
            if (ok && 4 * u + 2 < ns) ok = step(std::integral_constant<int, 2>{}, u);
            if (ok && 4 * u + 3 < ns) ok = step(std::integral_constant<int, 3>{}, u);
        }
        if (!ok) {
            if (tid == 0) *a.ok = 0;
            return false;
        }
        const uint32_t S = s_S[cs + ns];
        if (tid == 0) s_V[sub] = V;
        // C of the pivot rows to the common scale, and the pivot rows' other pieces aside
        if (mine >= 0) {
            const uint32_t f = mod_mul(s_S[cs + mine], V, R.q, R.barrett);
            if (live) {
                auto sc = [&](uint32_t x) { return ff_mul<ARITH>(x, f, R); };
                y = make_uint4(sc(y.x), sc(y.y), sc(y.z), sc(y.w));
                *reinterpret_cast<uint4*>(row + 4 * qg) = y;
            }
            for (int q = g; q < nq; q += 4)
                if (q < q0 || q >= q1)
                    *reinterpret_cast<uint4*>(P + mine * ls + 4 * q) = *reinterpret_cast<const uint4*>(row + 4 * q);
        }
        __syncthreads();
        uint32_t c[kSubCols];
#pragma unroll
        for (int i = 0; i < kSubCols / 4; ++i) {
            const uint4 v = 4 * i < ns ? *reinterpret_cast<const uint4*>(row + cs + 4 * i) : make_uint4(0, 0, 0, 0);
            c[4 * i] = v.x;
            c[4 * i + 1] = 4 * i + 1 < ns ? v.y : 0u;
            c[4 * i + 2] = 4 * i + 2 < ns ? v.z : 0u;
            c[4 * i + 3] = 4 * i + 3 < ns ? v.w : 0u;
        }
        __syncthreads();  // the sub-panel's own columns change below
        if (in) {
            if (live) {
                // (columns of the last piece beyond the pivots, where the block has fewer rows than
                // columns, have that scale already)
                const int left = cs + ns - 4 * qg;
                y = make_uint4(ff_scale2<ARITH>(y.x, V, R), ff_scale2<ARITH>(y.y, left > 1 ? V : 1u, R),
                               ff_scale2<ARITH>(y.z, left > 2 ? V : 1u, R), ff_scale2<ARITH>(y.w, left > 3 ? V : 1u, R));
                *reinterpret_cast<uint4*>(row + 4 * qg) = y;
            }
            const uint32_t sy = mine >= 0 ? 0u : S;
            for (int q = g; q < nq; q += 4) {
                if (q >= q0 && q < q1) continue;
                uint4 v = *reinterpret_cast<const uint4*>(row + 4 * q);
                uint32_t* vw = reinterpret_cast<uint32_t*>(&v);
                uint32_t a0[4], a1[4], a2[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const uint64_t t = static_cast<uint64_t>(sy) * vw[e];
                    a0[e] = static_cast<uint32_t>(t);
                    a1[e] = ARITH == kArithMont13 ? 0u : static_cast<uint32_t>(t >> 32);
                    a2[e] = 0;
                }
                const uint32_t* pq = P + 4 * q;
#pragma unroll
                for (int i = 0; i < kSubCols; i += 4) {
                    if (i >= ns) break;
                    uint4 p[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) p[e] = *reinterpret_cast<const uint4*>(pq + min(i + e, ns - 1) * ls);
                    if constexpr (ARITH == kArithMont32) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            mac96(a0[0], a1[0], a2[0], c[i + e], p[e].x);
                            mac96(a0[1], a1[1], a2[1], c[i + e], p[e].y);
                            mac96(a0[2], a1[2], a2[2], c[i + e], p[e].z);
                            mac96(a0[3], a1[3], a2[3], c[i + e], p[e].w);
                        }
                    } else if constexpr (ARITH == kArithPow2 || ARITH == kArithMont13) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            a0[0] += c[i + e] * p[e].x;
                            a0[1] += c[i + e] * p[e].y;
                            a0[2] += c[i + e] * p[e].z;
                            a0[3] += c[i + e] * p[e].w;
                        }
                    } else {
                        add96(a0[0], a1[0], a2[0], dot4(c[i], p[0].x, c[i + 1], p[1].x, c[i + 2], p[2].x, c[i + 3], p[3].x));
                        add96(a0[1], a1[1], a2[1], dot4(c[i], p[0].y, c[i + 1], p[1].y, c[i + 2], p[2].y, c[i + 3], p[3].y));
                        add96(a0[2], a1[2], a2[2], dot4(c[i], p[0].z, c[i + 1], p[1].z, c[i + 2], p[2].z, c[i + 3], p[3].z));
                        add96(a0[3], a1[3], a2[3], dot4(c[i], p[0].w, c[i + 1], p[1].w, c[i + 2], p[2].w, c[i + 3], p[3].w));
                    }
                }
                v = make_uint4(ff_reduce96<ARITH>(a0[0], a1[0], a2[0], R), ff_reduce96<ARITH>(a0[1], a1[1], a2[1], R),
                               ff_reduce96<ARITH>(a0[2], a1[2], a2[2], R), ff_reduce96<ARITH>(a0[3], a1[3], a2[3], R));
                *reinterpret_cast<uint4*>(row + 4 * q) = v;
            }
        }
        V = ff_scale2<ARITH>(V, S, R);
        __syncthreads();
    }
    // one warp inverts the scale (the chain's latency; all of them would queue at the multiplier), times
    // 2^32 for the Montgomery products below
    if (warp == 0) {
        const uint32_t vinv = unit_inverse(V, R);
        if (lane == 0) s_V[kMaxPanel / kSubCols + 1] = ARITH == kArithPow2 ? vinv : ff_mul<ARITH>(vinv, R.mont_r2, R);
    }
    __syncthreads();
    const uint32_t vinv = s_V[kMaxPanel / kSubCols + 1];
#pragma unroll 4
    for (int t = warp; t < nb; t += NW) {
        const int pl = s_prow[t];
        uint32_t* dst = a.A + static_cast<size_t>(a.r0 + pl) * a.ld + a.c0;
#pragma unroll
        for (int c = 0; c < WC; ++c) {
            const int j = lane + 32 * c;
            if (j >= w) break;
            const uint32_t v = ff_mul<ARITH>(T[pl * ls + j], vinv, R);
            if (j < nb) a.binv[t * nb + j] = v;
            dst[j] = j >= nb ? v : j == t ? 1u : 0u;
        }
    }
    if (tid < nb) {
        a.pivot_rows[tid] = a.r0 + s_prow[tid];
        a.pivot_cols[tid] = a.c0 + tid;
        // the classical pivots, for the determinant: w_t / (S_t V)
        if (a.diag) {
            const uint32_t s = mod_mul(s_S[tid], s_V[tid / kSubCols], R.q, R.barrett);
            a.diag[a.r0 + tid] = mod_mul(s_w[tid], unit_inverse(s, R), R.q, R.barrett);
        }
    }
    if (tid == 0) {
        *a.k_out = nb;
        *a.ok = 1;
    }
    return true;
}

}  // namespace panel
}  // namespace hme
