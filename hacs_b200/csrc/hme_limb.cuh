// Shared pieces of the INT8-limb GEMM kernels (limb_gemm.cu, grouped_gemm.cu):
// tile configuration, and the limb-split device routines.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/hme.h"
#include "hme_internal.h"
#include "hme_mod.h"
#include "hme_ptx.cuh"

namespace hme {
namespace limb {

constexpr int kBM = 128;     // UMMA M (rows of C per tile, one TMEM lane each)
constexpr int kBK = 128;     // bytes of K per pipeline stage: one 128-byte swizzle row
// Epilogue warps of L limbs: four per TMEM lane quarter (they take its
// 16-column chunks in turn); two for L = 2 and 3, where four leave too few
// registers for the chunk ahead.  Adding an 8192 x 8192 x 64 product to C, 8 / 16
// warps: L = 1 157 / 131 us, L = 2 130 / 144, L = 3 164 / 205, L = 4 154 / 144.
constexpr int epi_warps(int L) { return L == 2 || L == 3 ? 8 : 16; }
constexpr int gemm_threads(int L) { return 64 + 32 * epi_warps(L); }  // + the TMA warp and the MMA warp

// KB: bytes of K per pipeline stage = the width of one swizzle row (128, 64 or
// 32; products whose K fits a narrower row stream no zero padding).
template <int L, int BN, int KB = kBK>
struct Cfg {
    static_assert(KB == 128 || KB == 64 || KB == 32, "k-block of 128, 64 or 32 bytes");
    static constexpr int UN = L * BN;  // UMMA N: L accumulators of BN columns
    static_assert(UN % 16 == 0 && UN >= 16 && UN <= 256, "UMMA N must be a multiple of 16 in [16, 256]");
    static_assert(BN % 16 == 0, "the epilogue drains 16 columns at a time");
    static constexpr int A_BYTES = kBM * KB;
    static constexpr int B_BYTES = UN * KB;
    static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
    static constexpr int STAGES = (196608 / STAGE_BYTES) < 12 ? (196608 / STAGE_BYTES) : 12;
    static constexpr int ACC_STRIDE = UN <= 32 ? 32 : UN <= 64 ? 64 : UN <= 128 ? 128 : 256;
    static constexpr int TMEM_COLS = 2 * ACC_STRIDE;
    static constexpr int BAR_BYTES = 256;
    static constexpr int EPI_BYTES = epi_warps(L) * 32 * 16 * 4;  // per-warp 32 x 16 staging chunk (swizzled)
    static constexpr uint32_t IDESC = idesc_u8(kBM, UN);
    static_assert((2 * STAGES + 5) * 8 + 8 <= BAR_BYTES, "barrier area too small");
    // the one-k-block pipeline (short_tiles): L limb blocks of B stay in shared
    // memory while the CTA walks down a column of tiles; A streams through a ring
    static constexpr int B_TILE_BYTES = L * B_BYTES;
    static constexpr int B_BUFS = 2 * B_TILE_BYTES <= 131072 ? 2 : 1;
    static constexpr int A_SLOTS = ((196608 - B_BUFS * B_TILE_BYTES) / A_BYTES) < 10
                                       ? ((196608 - B_BUFS * B_TILE_BYTES) / A_BYTES) : 10;
    static_assert(A_SLOTS >= L, "the A ring holds at least one tile");
    static_assert((2 * A_SLOTS + 2 * B_BUFS + 5) * 8 + 8 <= BAR_BYTES, "barrier area too small");
    // operand blocks of either pipeline, then the barriers and the epilogue's stages
    static constexpr int LONG_BYTES = STAGES * STAGE_BYTES;
    static constexpr int SHORT_BYTES = B_BUFS * B_TILE_BYTES + A_SLOTS * A_BYTES;
    static constexpr int SMEM = (LONG_BYTES > SHORT_BYTES ? LONG_BYTES : SHORT_BYTES) + 1024 + BAR_BYTES + EPI_BYTES;
    static_assert(SMEM <= 232448, "more shared memory than a CTA can have");
};

// ---- the epilogue: accumulators -> residues -> C ----------------------------------
// One output is s = sum_j 256^j D_j (< 2^56) reduced mod p and combined with C.
// With K at most a few hundred (the trailing updates of the eliminations and of
// the job stream) a tile's MMAs take less time than its epilogue, so the GEMM
// is bound by the epilogue's instruction count and by the latency of reading C.
// Two things keep it short:
//  - the reduction takes one 32-bit multiply-high: hi = s >> sh1 (32 bits),
//    q = (hi * M >> 32) >> sh2 with M = floor(2^(31+b)/p), b the bit length of
//    p, sh1 the bits of s's bound beyond 32, sh2 = b - 1 - sh1.  q is at most
//    floor(s/p) and misses it by less than 2^sh1/p + 2^-(31+b) s <= 2^(sh1+2-b)
//    before the floor, so with sh1 <= b - 2 the rest s - q p is below 2p, and
//    with p < 2^31 it fits a word and one unsigned min(r, r - p) finishes it.
//    p = 0 (the wraparound mode) has M = 0: the truncation to 32 bits.  Every
//    other modulus has sh1 <= b - 1 (a limb's sums stay below 2^31, and 256^(L-1)
//    < p): the rest, below 3p, in 64 bits and two corrections (with
//    a 64-bit Barrett step, six wide products, 3000 x 3000 x 256 mod 2^32 - 17
//    takes 48 us, 45 so);
//  - C moves in 16-byte pieces where its rows are 16-byte aligned, and a
//    chunk's old values are loaded one chunk ahead of their use.
// Per output 73 -> 33 instructions for four limbs.  Adding an 8192 x 8192 x 64
// product to C (82 us of C at the copy rate; with short_tiles below, the limb
// split included): p = 13 244 -> 133 us, 65521 256 -> 132, 2^24 - 3 293 -> 167,
// 2^31 - 19 293 -> 144, 2^32 - 5 294 -> 197.
struct EpiRed {
    uint32_t p;
    uint32_t M;
    int sh1, sh2;
    int fast;
};

// The constants for sums up to `bound` (below 2^64) mod p.
inline EpiRed make_epi_bound(const ModParams& mp, unsigned __int128 bound) {
    EpiRed r{};
    r.p = mp.p;
    if (mp.p == 0) {
        r.fast = 1;
        return r;
    }
    int sb = 0;
    while (sb < 128 && (bound >> sb) != 0) ++sb;
    int b = 0;
    while (b < 32 && (mp.p >> b) != 0) ++b;
    r.sh1 = sb > 32 ? sb - 32 : 0;
    r.sh2 = b - 1 - r.sh1;
    HME_REQUIRE(r.sh2 >= 0, "gemm: sums too large for the reduction");
    const unsigned __int128 m = (static_cast<unsigned __int128>(1) << (31 + b)) / mp.p;
    r.M = m >> 32 ? 0xffffffffu : static_cast<uint32_t>(m);
    r.fast = mp.p < (1u << 31) && r.sh1 <= b - 2 ? 1 : 0;
    return r;
}
// The constants for 256 v of the limb split, v below 256^limbs.
inline EpiRed make_split_red(const ModParams& mp) {
    return make_epi_bound(mp, static_cast<unsigned __int128>(256) << (8 * mp.limbs));
}
// The constants for products whose K (per launch) is at most kc.
inline EpiRed make_epi(const ModParams& mp, uint64_t kc) {
    unsigned __int128 bound = 0;
    for (uint32_t j = 0; j < mp.limbs; ++j)
        bound += (static_cast<unsigned __int128>(mp.limbs) * 255u * 255u * kc) << (8 * j);
    return make_epi_bound(mp, bound);
}

template <bool FAST>
__device__ __forceinline__ uint32_t epi_reduce_u64(uint64_t s, const EpiRed& r) {
    const uint32_t lo = static_cast<uint32_t>(s);
    const uint32_t hi = __funnelshift_r(lo, static_cast<uint32_t>(s >> 32), r.sh1);
    const uint32_t q = __umulhi(hi, r.M) >> r.sh2;
    if constexpr (FAST) {
        const uint32_t x = lo - q * r.p;
        return min(x, x - r.p);
    } else {
        const uint64_t x = s - static_cast<uint64_t>(q) * r.p;
        const uint32_t xl = static_cast<uint32_t>(x);
        const uint32_t y = (x >> 32) != 0 || xl >= r.p ? xl - r.p : xl;
        return min(y, y - r.p);  // p >= 2^31: y < p already, and y - p wraps above it
    }
}

template <int L, bool FAST>
__device__ __forceinline__ uint32_t epi_reduce(uint32_t v0, uint32_t v1, uint32_t v2, uint32_t v3, const EpiRed& r) {
    uint64_t s = v0;
    if (L > 1) s += static_cast<uint64_t>(v1) * 256u;
    if (L > 2) s += static_cast<uint64_t>(v2) * 65536u;
    if (L > 3) s += static_cast<uint64_t>(v3) * 16777216u;
    return epi_reduce_u64<FAST>(s, r);
}

// How C and the reduced value combine, one form for the three ops: with old = 0
// for Set, old + (x ^ flip) + bias is old + x, or old + p - x for Sub, below 2p.
struct EpiOp {
    uint32_t flip, bias;
    bool set;
};
__device__ __forceinline__ EpiOp epi_op(int op, const EpiRed& r) {
    return op == HME_SUB ? EpiOp{0xffffffffu, r.p + 1u, false} : EpiOp{0u, 0u, op == HME_SET};
}

template <bool FAST>
__device__ __forceinline__ uint32_t epi_combine(uint32_t old, uint32_t x, const EpiOp& o, const EpiRed& r) {
    if constexpr (FAST) {  // p < 2^31 (or 0: wraparound): the unsigned min picks the canonical one
        const uint32_t t = old + (x ^ o.flip) + o.bias;
        return min(t, t - r.p);
    } else {
        if (o.set) return x;
        return o.flip ? mod_sub(old, x, r.p) : mod_add(old, x, r.p);
    }
}

// One warp's share of a tile's drain: rows row0 .. row0 + 31 (its TMEM lane
// quarter), every (warps of the quarter)-th 16-column chunk from chunk `grp` on.  A thread
// reads its row's accumulators, reduces them and hands them through the warp's
// swizzled 32 x 16 stage (16-byte piece c of row r at c ^ (r >> 1 & 3): no bank
// conflict either way), so that C is read and written along rows: 8 rows x 64
// bytes per warp instruction (VEC: C and ldc 16-byte aligned), else 2 rows x 64
// bytes of single words.  Values of C are loaded one chunk ahead; the first
// chunk's before the accumulator is waited for.
struct EpiTile {
    uint32_t* C;
    uint64_t ldc;
    int M, N, row0, col0, op;
};

struct EpiOld {
    uint32_t v[16];
};

__device__ __forceinline__ bool epi_vec(const uint32_t* C, uint64_t ldc) {
    return ((reinterpret_cast<uintptr_t>(C) & 15) | (ldc & 3)) == 0;
}

// The thread's first word of a chunk in C; opaque, so that the addresses of a
// chunk's loads are not kept in registers for its stores.
__device__ __forceinline__ uint32_t* epi_ptr(const EpiTile& t, int row, int col) {
    uint32_t* p = t.C + static_cast<size_t>(row) * t.ldc + col;
    asm volatile("" : "+l"(p));
    return p;
}

__device__ __forceinline__ void epi_load_old(const EpiTile& t, int c0, bool vec, int lane, EpiOld& o) {
    if (t.op == HME_SET) {
#pragma unroll
        for (int u = 0; u < 16; ++u) o.v[u] = 0u;
        return;
    }
    if (vec) {
        const int col = t.col0 + c0 + 4 * (lane & 3), row = t.row0 + (lane >> 2), left = t.N - col;
        const uint32_t* p = epi_ptr(t, row, col);
        const size_t step = 8 * t.ldc;
#pragma unroll
        for (int u = 0; u < 4; ++u, p += step) {
            uint4 x = make_uint4(0, 0, 0, 0);
            if (row + 8 * u < t.M && left > 0) {
                if (left >= 4) {
                    x = *reinterpret_cast<const uint4*>(p);
                } else {
                    x.x = p[0];
                    if (left > 1) x.y = p[1];
                    if (left > 2) x.z = p[2];
                }
            }
            o.v[4 * u] = x.x; o.v[4 * u + 1] = x.y; o.v[4 * u + 2] = x.z; o.v[4 * u + 3] = x.w;
        }
    } else {
        const int col = t.col0 + c0 + (lane & 15), row = t.row0 + (lane >> 4);
        const int rows = col < t.N ? t.M - row : 0;
        const uint32_t* p = epi_ptr(t, row, col);
        const size_t step = 2 * t.ldc;
#pragma unroll
        for (int u = 0; u < 16; ++u, p += step) o.v[u] = 2 * u < rows ? *p : 0u;
    }
}

template <int L, bool FAST>
__device__ __forceinline__ void epi_chunk(const EpiTile& t, int c0, bool vec, int lane, uint32_t (&v)[L][16],
                                          const EpiOld& o, uint32_t* stage, const EpiRed& r) {
    const int wsw = (lane >> 1) & 3;
    const EpiOp eo = epi_op(t.op, r);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        uint32_t x[4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
            x[e] = epi_reduce<L, FAST>(v[0][4 * c + e], v[L > 1 ? 1 : 0][4 * c + e], v[L > 2 ? 2 : 0][4 * c + e],
                                       v[L > 3 ? 3 : 0][4 * c + e], r);
        *reinterpret_cast<uint4*>(stage + 16 * lane + 4 * (c ^ wsw)) = make_uint4(x[0], x[1], x[2], x[3]);
    }
    __syncwarp();
    if (vec) {
        const int cg = lane & 3, r0 = lane >> 2, col = t.col0 + c0 + 4 * cg, row = t.row0 + r0, left = t.N - col;
        uint32_t* p = epi_ptr(t, row, col);
        const size_t step = 8 * t.ldc;
#pragma unroll
        for (int u = 0; u < 4; ++u, p += step) {
            const uint4 s = *reinterpret_cast<const uint4*>(stage + 16 * (r0 + 8 * u) + 4 * (cg ^ ((r0 >> 1) & 3)));
            uint4 x;
            x.x = epi_combine<FAST>(o.v[4 * u], s.x, eo, r);
            x.y = epi_combine<FAST>(o.v[4 * u + 1], s.y, eo, r);
            x.z = epi_combine<FAST>(o.v[4 * u + 2], s.z, eo, r);
            x.w = epi_combine<FAST>(o.v[4 * u + 3], s.w, eo, r);
            if (row + 8 * u < t.M && left > 0) {
                if (left >= 4) {
                    *reinterpret_cast<uint4*>(p) = x;
                } else {
                    p[0] = x.x;
                    if (left > 1) p[1] = x.y;
                    if (left > 2) p[2] = x.z;
                }
            }
        }
    } else {
        const int cc = lane & 15, r0 = lane >> 4, col = t.col0 + c0 + cc, row = t.row0 + r0;
        const int rows = col < t.N ? t.M - row : 0;
        uint32_t* p = epi_ptr(t, row, col);
        const size_t step = 2 * t.ldc;
#pragma unroll
        for (int u = 0; u < 16; ++u, p += step) {
            const uint32_t s = stage[16 * (r0 + 2 * u) + 4 * ((cc >> 2) ^ (u & 3)) + (cc & 3)];
            if (2 * u < rows) *p = epi_combine<FAST>(o.v[u], s, eo, r);
        }
    }
    __syncwarp();
}

// Drains one accumulator (taddr: its first column, in this warp's lane
// quarter).  `o` holds the first chunk's old values (epi_load_old).  The
// accumulator is released (mbar_arrive on acc_empty) as soon as the last chunk
// has left tensor memory.
template <int L, int BN, bool FAST>
__device__ __forceinline__ void epi_drain(const EpiTile& t, uint32_t taddr, int grp, bool vec, int lane, EpiOld& o,
                                          uint32_t* stage, uint64_t* acc_empty, const EpiRed& r) {
    constexpr int STEP = 16 * (epi_warps(L) / 4);
    if (16 * grp >= BN) {  // no chunk for this warp
        mbar_arrive(acc_empty);
        return;
    }
#pragma unroll 1
    for (int c0 = 16 * grp; c0 < BN; c0 += STEP) {
        uint32_t v[L][16];
#pragma unroll
        for (int j = 0; j < L; ++j) tmem_ld16(taddr + j * BN + c0, v[j]);
        const bool last = c0 + STEP >= BN;
        EpiOld nxt;
        if (L <= 2 && !last) epi_load_old(t, c0 + STEP, vec, lane, nxt);
        tmem_wait_ld();
        if (last) {
            tc_fence_before();
            mbar_arrive(acc_empty);
        }
        epi_chunk<L, FAST>(t, c0, vec, lane, v, o, stage, r);
        if (!last) {
            if (L <= 2) {
#pragma unroll
                for (int u = 0; u < 16; ++u) o.v[u] = nxt.v[u];
            } else {  // four accumulators leave no registers for a second set
                epi_load_old(t, c0 + STEP, vec, lane, o);
            }
        }
    }
}

// ---- the GEMM pipelines ------------------------------------------------------------
// Warp 0 issues the TMA loads, warp 1 owns tensor memory and issues the MMAs,
// the other warps drain the double-buffered accumulators into C.  `Src` gives
// the tiles: tile(t) -> TileRef, and total() of them.
struct TileRef {
    const CUtensorMap* tmA;
    const CUtensorMap* tmB;
    int a_row, b_col;       // first plane row of the A tile / of the B tile
    int k_begin, kblocks;   // k-blocks of KB bytes from byte k_begin on
    uint32_t* C;
    uint64_t ldc;
    int M, N, row0, col0, op;
    int b_key;              // equal for tiles that share their B tile
};

// Time-bounded wait that ignores the abort flag: used while tearing down, to
// let in-flight copies and MMAs land before shared / tensor memory is released.
__device__ __forceinline__ void drain_wait(uint64_t* bar, uint32_t parity, int* err) {
    int never = 0;
    mbar_wait(bar, parity, &never, err, DERR_WAIT_DRAIN);
}

// The epilogue warps' loop over the tiles first, first + step, .. < end.
template <int L, int BN, int KB, class Src>
__device__ __forceinline__ void epilogue_tiles(const Src& src, int first, int end, int step, int warp, int lane,
                                               uint32_t tmem_base, uint32_t* epi_stage, uint64_t* acc_full,
                                               uint64_t* acc_empty, volatile int* abort_flag, const EpiRed& red,
                                               int* err) {
    using CF = Cfg<L, BN, KB>;
    const int q = warp & 3;  // the TMEM lane quarter this warp may read
    const int grp = (warp - 2) >> 2;  // its place among the lane quarter's warps
    const uint32_t lane_base = static_cast<uint32_t>(q * 32) << 16;
    uint32_t* stage = epi_stage + (warp - 2) * 32 * 16;
    // Add / Sub read C: each lane prefetches its row of a tile into L2 one tile
    // ahead, so the HBM reads of the next tile overlap this tile's drain
    auto prefetch_tile = [&](int t) {
        if (t >= end || grp != 0) return;
        const TileRef r = src.tile(t);
        if (r.op == HME_SET) return;
        const int row = r.row0 + q * 32 + lane;
        if (row < r.M) prefetch_l2_span(r.C + static_cast<size_t>(row) * r.ldc + r.col0, min(BN, r.N - r.col0));
    };
    prefetch_tile(first);
    int lt = 0;
    for (int tile = first; tile < end; tile += step, ++lt) {
        prefetch_tile(tile + step);
        const int a = lt & 1;
        const TileRef r = src.tile(tile);
        const EpiTile t{r.C, r.ldc, r.M, r.N, r.row0 + q * 32, r.col0, r.op};
        const bool vec = epi_vec(r.C, r.ldc);
        EpiOld old;
        epi_load_old(t, 16 * grp, vec, lane, old);
        if (!mbar_wait(&acc_full[a], (lt >> 1) & 1, abort_flag, err, DERR_WAIT_ACCUM)) break;
        tc_fence_after();
        const uint32_t taddr = tmem_base + lane_base + a * CF::ACC_STRIDE;
        if (red.fast) epi_drain<L, BN, true>(t, taddr, grp, vec, lane, old, stage, &acc_empty[a], red);
        else epi_drain<L, BN, false>(t, taddr, grp, vec, lane, old, stage, &acc_empty[a], red);
    }
}

// An epilogue of a pipeline: what the epilogue warps do with the accumulators.
template <int L, int BN, int KB>
struct ResidueEpilogue {  // residues mod p into C
    const EpiRed& red;
    template <class Src>
    __device__ __forceinline__ void run(const Src& src, int first, int end, int step, int warp, int lane,
                                        uint32_t tmem_base, uint32_t* epi_stage, uint64_t* acc_full,
                                        uint64_t* acc_empty, volatile int* abort_flag, int* err) const {
        epilogue_tiles<L, BN, KB>(src, first, end, step, warp, lane, tmem_base, epi_stage, acc_full, acc_empty,
                                  abort_flag, red, err);
    }
};

// Products of several k-blocks: A and B blocks stream through one ring, tiles
// are taken with the stride of the grid.
template <int L, int BN, int KB, class Src, class Epi>
__device__ __forceinline__ void long_tiles(const Src& src, const Epi& epi, int* err) {
    using CF = Cfg<L, BN, KB>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sA = smem;
    uint8_t* sB = smem + CF::STAGES * CF::A_BYTES;
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + CF::STAGES * CF::STAGE_BYTES);
    uint64_t* empty = full + CF::STAGES;
    uint64_t* acc_full = empty + CF::STAGES;
    uint64_t* acc_empty = acc_full + 2;
    uint64_t* drain = acc_empty + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    uint32_t* epi_stage = reinterpret_cast<uint32_t*>(smem + CF::STAGES * CF::STAGE_BYTES + CF::BAR_BYTES);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < CF::STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&acc_full[a], 1);
            mbar_init(&acc_empty[a], 32 * epi_warps(L));
        }
        mbar_init(drain, 1);
        *abort_flag = 0;
        fence_mbar_init();
        fence_proxy_async_smem();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, CF::TMEM_COLS);
        tmem_relinquish();
    }
    src.prefetch_maps();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // the set-up above overlaps the tail of the limb split when this grid is a
    // programmatic dependent of it; the planes are read only after this point
    grid_dep_wait();
    const int total_tiles = src.total();

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (lane == 0) {
            int it = 0;
            bool ok = true;
            for (int tile = blockIdx.x; ok && tile < total_tiles; tile += gridDim.x) {
                const TileRef r = src.tile(tile);
                for (int i = 0; ok && i < L; ++i) {
                    for (int kb = 0; kb < r.kblocks; ++kb, ++it) {
                        const int s = it % CF::STAGES;
                        const uint32_t ph = (it / CF::STAGES) & 1;
                        if (!mbar_wait(&empty[s], ph ^ 1, abort_flag, err, DERR_WAIT_EMPTY)) {
                            ok = false;
                            break;
                        }
                        mbar_arrive_expect_tx(&full[s], CF::STAGE_BYTES);
                        const int kx = r.k_begin + kb * KB;
                        tma_load_3d(sA + s * CF::A_BYTES, r.tmA, &full[s], kx, r.a_row, i);
                        tma_load_4d(sB + s * CF::B_BYTES, r.tmB, &full[s], kx, r.b_col, 0, i);
                    }
                }
            }
            if (!ok) {
                // let every copy issued into shared memory land before the CTA exits
                for (int t = max(0, it - CF::STAGES); t < it; ++t)
                    drain_wait(&full[t % CF::STAGES], (t / CF::STAGES) & 1, err);
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        if (lane == 0) {
            int it = 0, lt = 0;
            bool ok = true, issued_any = false;
            for (int tile = blockIdx.x; ok && tile < total_tiles; tile += gridDim.x, ++lt) {
                const int kblocks = src.kblocks(tile);
                const int a = lt & 1;
                const uint32_t aph = (lt >> 1) & 1;
                if (!mbar_wait(&acc_empty[a], aph ^ 1, abort_flag, err, DERR_WAIT_ACCUM_FREE)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t d = tmem_base + a * CF::ACC_STRIDE;
                for (int i = 0; ok && i < L; ++i) {
                    for (int kb = 0; kb < kblocks; ++kb, ++it) {
                        const int s = it % CF::STAGES;
                        const uint32_t ph = (it / CF::STAGES) & 1;
                        if (!mbar_wait(&full[s], ph, abort_flag, err, DERR_WAIT_FULL)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        const uint64_t adesc = smem_desc_kmajor<KB>(smem_u32(sA + s * CF::A_BYTES));
                        const uint64_t bdesc = smem_desc_kmajor<KB>(smem_u32(sB + s * CF::B_BYTES));
#pragma unroll
                        for (int kk = 0; kk < KB / 32; ++kk) {
                            // +32 bytes along K inside the swizzle atom = +2 in the 16-byte address field
                            mma_u8(d, adesc + 2 * kk, bdesc + 2 * kk, CF::IDESC, (i | kb | kk) != 0);
                        }
                        issued_any = true;
                        mma_commit(&empty[s]);
                    }
                }
                if (ok) mma_commit(&acc_full[a]);
            }
            if (!ok && issued_any) {
                mma_commit(drain);
                drain_wait(drain, 0, err);
            }
        }
    } else {
        epi.run(src, blockIdx.x, total_tiles, gridDim.x, warp, lane, tmem_base, epi_stage, acc_full, acc_empty,
                abort_flag, err);
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, CF::TMEM_COLS);
    }
}

// Products of one k-block (K <= KB: the eliminations' trailing updates, the
// job stream's rounds).  Streamed like the long ones, a 128 x 64 tile of four
// limbs would read 96 KB of planes per 32 KB of C, and the update would be
// bound by the L2 -> SM traffic (4096 x 4096 x 64 mod 2^31 - 19: 200 MB of
// planes beside 134 MB of C).  So a CTA takes a contiguous run of tiles, in an
// order that walks down the columns, keeps the B tile (all L limb blocks) in
// shared memory while it lasts, and streams only A (a third of the bytes).
template <int L, int BN, int KB, class Src>
__device__ __forceinline__ void short_tiles(const Src& src, const EpiRed& red, int* err) {
    using CF = Cfg<L, BN, KB>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sB = smem;                                    // [B_BUFS][L][B_BYTES]
    uint8_t* sA = smem + CF::B_BUFS * CF::B_TILE_BYTES;    // [A_SLOTS][A_BYTES]
    uint64_t* fullA = reinterpret_cast<uint64_t*>(sA + CF::A_SLOTS * CF::A_BYTES);
    uint64_t* emptyA = fullA + CF::A_SLOTS;
    uint64_t* fullB = emptyA + CF::A_SLOTS;
    uint64_t* emptyB = fullB + CF::B_BUFS;
    uint64_t* acc_full = emptyB + CF::B_BUFS;
    uint64_t* acc_empty = acc_full + 2;
    uint64_t* drain = acc_empty + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    uint32_t* epi_stage = reinterpret_cast<uint32_t*>(sA + CF::A_SLOTS * CF::A_BYTES + CF::BAR_BYTES);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < CF::A_SLOTS; ++s) {
            mbar_init(&fullA[s], 1);
            mbar_init(&emptyA[s], 1);
        }
        for (int s = 0; s < CF::B_BUFS; ++s) {
            mbar_init(&fullB[s], 1);
            mbar_init(&emptyB[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&acc_full[a], 1);
            mbar_init(&acc_empty[a], 32 * epi_warps(L));
        }
        mbar_init(drain, 1);
        *abort_flag = 0;
        fence_mbar_init();
        fence_proxy_async_smem();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, CF::TMEM_COLS);
        tmem_relinquish();
    }
    src.prefetch_maps();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    grid_dep_wait();  // the planes (and device tables) are read only after this point
    const long long total = src.total();
    const int first = static_cast<int>(total * blockIdx.x / gridDim.x);
    const int end = static_cast<int>(total * (blockIdx.x + 1) / gridDim.x);

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (lane == 0) {
            int it = 0, nb = 0, key = -1;
            bool ok = true;
            for (int tile = first; ok && tile < end; ++tile) {
                const TileRef r = src.tile(tile);
                if (nb == 0 || r.b_key != key) {
                    key = r.b_key;
                    const int b = nb % CF::B_BUFS;
                    if (!mbar_wait(&emptyB[b], ((nb / CF::B_BUFS) & 1) ^ 1, abort_flag, err, DERR_WAIT_EMPTY)) {
                        ok = false;
                        break;
                    }
                    mbar_arrive_expect_tx(&fullB[b], CF::B_TILE_BYTES);
#pragma unroll
                    for (int i = 0; i < L; ++i)
                        tma_load_4d(sB + b * CF::B_TILE_BYTES + i * CF::B_BYTES, r.tmB, &fullB[b], r.k_begin, r.b_col,
                                    0, i);
                    ++nb;
                }
                for (int i = 0; i < L; ++i, ++it) {
                    const int s = it % CF::A_SLOTS;
                    if (!mbar_wait(&emptyA[s], ((it / CF::A_SLOTS) & 1) ^ 1, abort_flag, err, DERR_WAIT_EMPTY)) {
                        ok = false;
                        break;
                    }
                    mbar_arrive_expect_tx(&fullA[s], CF::A_BYTES);
                    tma_load_3d(sA + s * CF::A_BYTES, r.tmA, &fullA[s], r.k_begin, r.a_row, i);
                }
            }
            if (!ok) {
                // let every copy issued into shared memory land before the CTA exits
                for (int t = max(0, it - CF::A_SLOTS); t < it; ++t)
                    drain_wait(&fullA[t % CF::A_SLOTS], (t / CF::A_SLOTS) & 1, err);
                for (int t = max(0, nb - CF::B_BUFS); t < nb; ++t)
                    drain_wait(&fullB[t % CF::B_BUFS], (t / CF::B_BUFS) & 1, err);
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        if (lane == 0) {
            int it = 0, lt = 0, nb = 0, key = -1;
            bool ok = true, issued_any = false;
            for (int tile = first; ok && tile < end; ++tile, ++lt) {
                const int bk = src.b_key(tile);
                if (nb == 0 || bk != key) {
                    // the B tile before this one is free once the MMAs issued so far are done
                    if (nb > 0) mma_commit(&emptyB[(nb - 1) % CF::B_BUFS]);
                    key = bk;
                    if (!mbar_wait(&fullB[nb % CF::B_BUFS], (nb / CF::B_BUFS) & 1, abort_flag, err, DERR_WAIT_FULL)) {
                        ok = false;
                        break;
                    }
                    ++nb;
                }
                const int b = (nb - 1) % CF::B_BUFS;
                const int a = lt & 1;
                if (!mbar_wait(&acc_empty[a], ((lt >> 1) & 1) ^ 1, abort_flag, err, DERR_WAIT_ACCUM_FREE)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t d = tmem_base + a * CF::ACC_STRIDE;
                for (int i = 0; i < L; ++i, ++it) {
                    const int s = it % CF::A_SLOTS;
                    if (!mbar_wait(&fullA[s], (it / CF::A_SLOTS) & 1, abort_flag, err, DERR_WAIT_FULL)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint64_t adesc = smem_desc_kmajor<KB>(smem_u32(sA + s * CF::A_BYTES));
                    const uint64_t bdesc =
                        smem_desc_kmajor<KB>(smem_u32(sB + b * CF::B_TILE_BYTES + i * CF::B_BYTES));
#pragma unroll
                    for (int kk = 0; kk < KB / 32; ++kk)
                        mma_u8(d, adesc + 2 * kk, bdesc + 2 * kk, CF::IDESC, (i | kk) != 0);
                    issued_any = true;
                    mma_commit(&emptyA[s]);
                }
                if (ok) mma_commit(&acc_full[a]);
            }
            if (!ok && issued_any) {
                mma_commit(drain);
                drain_wait(drain, 0, err);
            }
        }
    } else {
        epilogue_tiles<L, BN, KB>(src, first, end, 1, warp, lane, tmem_base, epi_stage, acc_full, acc_empty,
                                  abort_flag, red, err);
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, CF::TMEM_COLS);
    }
}

// ---- limb split (one launch for both operands) ------------------------------------
// Blocks [0, a_blocks): A planes[i][m][k] = byte i of A[m][k], 16 k per thread
// (four 16-byte loads when A rows are 16-byte aligned).  Blocks [a_blocks, ..):
// B planes[i][j][n][k] = byte j of (256^i * B[k][n] mod p), B transposed to
// K-major through shared memory, 64 k x 32 n per block, 8 k per thread.
// k in [K, Kp) is written as zero in both.
struct SplitArgs {
    const uint32_t* A;
    uint64_t lda;
    const uint32_t* B;
    uint64_t ldb;
    int M, N, K, Kp;
    EpiRed red;          // make_split_red
    uint8_t* planesA;
    uint8_t* planesB;
    int a_blocks;        // blocks of the A part
    int b_blocks_k;      // B part: blocks along k (64 k each)
    bool a_vec;          // A rows 16-byte aligned: vector loads
    uint64_t a_plane;    // bytes between A limb planes (0: M * Kp)
    uint64_t b_plane;    // bytes between B limb planes (0: N * Kp)
    Skip skip;
};

// idx / kch, in 32 bits where the operand's pieces can be counted in them
__device__ __forceinline__ int split_row(size_t idx, size_t total, int kch) {
    return total >> 32 ? static_cast<int>(idx / kch)
                       : static_cast<int>(static_cast<uint32_t>(idx) / static_cast<uint32_t>(kch));
}

// Rows that are not 16-byte aligned go four words a thread, so that a warp's loads
// and stores cover consecutive words (16 a thread would load with a stride of 64
// bytes); figures at split_b_tile.  The index is divided in 32 bits: with a 64-bit
// division per four words the 65521 half of 2000 uneven jobs took 726 us, 610 so.
template <int L>
__device__ __forceinline__ void split_a_words(const SplitArgs& s, int block) {
    const int kch = s.Kp >> 2;
    const size_t total = static_cast<size_t>(s.M) * kch;
    const size_t plane = s.a_plane ? s.a_plane : static_cast<size_t>(s.M) * s.Kp;
    const size_t step = static_cast<size_t>(s.a_blocks) * blockDim.x;
    for (size_t i0 = static_cast<size_t>(block) * blockDim.x + threadIdx.x; i0 < total; i0 += 4 * step) {
        uint32_t x[4][4];
        uint8_t* dst[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const size_t idx = i0 + u * step, at = min(idx, total - 1);
            const int row = split_row(at, total, kch);
            const int k0 = static_cast<int>(at - static_cast<size_t>(row) * kch) << 2;
            const uint32_t* src = s.A + static_cast<size_t>(row) * s.lda + k0;
            dst[u] = s.planesA + static_cast<size_t>(row) * s.Kp + k0;
#pragma unroll
            for (int e = 0; e < 4; ++e) x[u][e] = idx < total && k0 + e < s.K ? __ldg(src + e) : 0u;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (i0 + u * step >= total) break;
#pragma unroll
            for (int j = 0; j < L; ++j) {
                uint32_t w = 0;
#pragma unroll
                for (int e = 0; e < 4; ++e) w |= ((x[u][e] >> (8 * j)) & 0xffu) << (8 * e);
                *reinterpret_cast<uint32_t*>(dst[u] + j * plane) = w;
            }
        }
    }
}

template <int L>
__device__ __forceinline__ void split_a_part(const SplitArgs& s, int block) {
    if (!s.a_vec) {
        split_a_words<L>(s, block);
        return;
    }
    const int kch = s.Kp >> 4;
    const size_t total = static_cast<size_t>(s.M) * kch;
    const size_t plane = s.a_plane ? s.a_plane : static_cast<size_t>(s.M) * s.Kp;
    for (size_t idx = static_cast<size_t>(block) * blockDim.x + threadIdx.x; idx < total;
         idx += static_cast<size_t>(s.a_blocks) * blockDim.x) {
        const int row = split_row(idx, total, kch);
        const int k0 = static_cast<int>(idx - static_cast<size_t>(row) * kch) << 4;
        const uint32_t* src = s.A + static_cast<size_t>(row) * s.lda + k0;
        uint32_t x[16];
        if (k0 + 16 <= s.K) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint4 v = __ldg(reinterpret_cast<const uint4*>(src) + q);
                x[4 * q] = v.x; x[4 * q + 1] = v.y; x[4 * q + 2] = v.z; x[4 * q + 3] = v.w;
            }
        } else {
#pragma unroll
            for (int e = 0; e < 16; ++e) x[e] = (k0 + e < s.K) ? __ldg(src + e) : 0u;
        }
        uint8_t* dst = s.planesA + static_cast<size_t>(row) * s.Kp + k0;
#pragma unroll
        for (int j = 0; j < L; ++j) {
            uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
            for (int e = 0; e < 16; ++e) w[e >> 2] |= ((x[e] >> (8 * j)) & 0xffu) << (8 * (e & 3));
            *reinterpret_cast<uint4*>(dst + j * plane) = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
}

// Bound by the writes of the L^2 planes as long as 256 v mod p is cheap: one
// 32-bit multiply-high (epi_reduce_u64) where a 64-bit Barrett step took six wide
// products.
// Both parts, mod 2^31 - 19, 1677 x 771 x 1419 (unaligned rows): 13.6 -> 9.5 us;
// mod 65521, 1024^3 5.1 -> 4.1 us, 8192^3 191 -> 175 us (144 at the copy rate).
template <int L, bool FAST>
__device__ __forceinline__ void split_b_tile(const SplitArgs& s, int block, uint32_t (*tile)[33]) {
    const int k0 = (block % s.b_blocks_k) * 64, n0 = (block / s.b_blocks_k) * 32;
    // all eight loads of a thread in flight before the first shared-memory store
    // (blockDim.x == 256: 8 x 256 = the 64 x 32 tile)
    uint32_t v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int t = threadIdx.x + 256 * q;
        const int k = k0 + (t >> 5), n = n0 + (t & 31);
        v[q] = (k < s.K && n < s.N) ? __ldg(s.B + static_cast<size_t>(k) * s.ldb + n) : 0u;
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int t = threadIdx.x + 256 * q;
        tile[t >> 5][t & 31] = v[q];
    }
    __syncthreads();
    const int nn = threadIdx.x >> 3, kc = threadIdx.x & 7;
    const int n = n0 + nn, kb = k0 + kc * 8;
    if (n >= s.N || kb >= s.Kp) return;
    uint32_t out[L][L][2];
#pragma unroll
    for (int i = 0; i < L; ++i)
#pragma unroll
        for (int j = 0; j < L; ++j) out[i][j][0] = out[i][j][1] = 0;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        uint32_t v = tile[kc * 8 + e][nn];
#pragma unroll
        for (int i = 0; i < L; ++i) {
            if (i) v = epi_reduce_u64<FAST>(static_cast<uint64_t>(v) << 8, s.red);
#pragma unroll
            for (int j = 0; j < L; ++j) out[i][j][e >> 2] |= ((v >> (8 * j)) & 0xffu) << (8 * (e & 3));
        }
    }
    const size_t plane = s.b_plane ? s.b_plane : static_cast<size_t>(s.N) * s.Kp;
#pragma unroll
    for (int i = 0; i < L; ++i)
#pragma unroll
        for (int j = 0; j < L; ++j)
            *reinterpret_cast<uint2*>(s.planesB + (i * L + j) * plane + static_cast<size_t>(n) * s.Kp + kb) =
                make_uint2(out[i][j][0], out[i][j][1]);
}

template <int L>
__device__ __forceinline__ void split_b_part(const SplitArgs& s, int block, uint32_t (*tile)[33]) {
    if (s.red.fast) split_b_tile<L, true>(s, block, tile);
    else split_b_tile<L, false>(s, block, tile);
}

}  // namespace limb

// Host: encode a tiled uint8 TMA descriptor (limb planes) with the swizzle matching a k-block of kb bytes (128,
// 64 or 32).
void encode_tma_u8_kb(CUtensorMap* map, void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides,
                      const cuuint32_t* box, int kb);

}  // namespace hme
