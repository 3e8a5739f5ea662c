// The mod-p GEMM for u64 residues (any modulus 2 <= p < 2^64): C op= A*B mod p.
//
// Reference semantics: engine::kernels::gemm<uint64_t> / engine::cuda::gemm
// <uint64_t> (src/ModArithmetic/Kernels.h:178-185; src/Cuda/cuda_kernels.cu
// :151-163 and the u64 tiles :365-381): the exact sum of k products, reduced
// to the canonical residue, combined by Set / Add / Sub.  The reference's u64
// regime multiplies in Montgomery form (odd p < 2^63) or with a wide mulmod
// (otherwise), one reduction per product, on CUDA cores.
//
// Method (residue number system over 8-bit moduli).  With canonical inputs the
// exact integer X = sum_k a_ik b_kj lies in [0, k (p-1)^2].  Take the first t of
// the pairwise coprime moduli 256, 255, 253, 251, 247, 241, .. whose product M
// exceeds 4 k (p-1)^2.  Then:
//   1. A_t = A mod m_t, B_t = (M/m_t)^-1 B mod m_t, one byte per entry, written
//      directly as the K-major planes that the tensor cores read (one launch for
//      both operands and all t);
//   2. Y_t = A_t B_t mod m_t: t one-limb products in one launch (tcgen05 kind::i8,
//      a tile of every modulus in one queue), reduced and stored as bytes;
//   3. the CRT, element by element: X = sum_t Y_t M/m_t - w M with w = sum_t
//      Y_t / m_t - X/M, and since X/M < 1/4, w is the nearest integer to sum_t Y_t
//      F_t / 2^15 with F_t = 2^15 / m_t rounded to a byte (off by less than
//      0.09).  So X mod p = (sum_t Y_t (M/m_t mod p) + w (p - M mod p)) mod p, the
//      sums by byte dot products (dp4a) over the bytes of the constants.
// One product of p^2 bits costs about 2 log2 p / 7.8 one-limb products: 18 mod
// 2^61 - 1, where 9 primes below 2^16 cost 36 limb products and 12 launches, and
// 10 mod 2^31 - 19 (u32 entries, rns_gemm_u32_device), where the four-limb
// product costs 16.  2048^3 mod 2^61 - 1: 476 -> 248 us (split 66, products 120 at
// 2.6 POPS of int8, CRT 44; the split is bound by its integer arithmetic).
// Moduli below 2^32 with u64 entries narrow to u32 and the u32 GEMM computes the
// product mod p directly.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "hme_internal.h"
#include "hme_limb.cuh"
#include "hme_ptx.cuh"

namespace hme {
namespace {

using namespace limb;

// Pairwise coprime (255 = 3 5 17, 253 = 11 23, 247 = 13 19, 217 = 7 31, the others
// but 256 prime); all 22 give 170 bits, k (p-1)^2 needs at most 161.  Each is
// above 128, so that 2^15 / m fits a byte.
constexpr int kMaxRns = 22;
constexpr int kRnsGroups = (kMaxRns + 3) / 4;
constexpr uint32_t kModuli[kMaxRns] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223,
                                       217, 211, 199, 197, 193, 191, 181, 179, 173, 167, 163};

// The moduli's and p's constants, passed by value.
struct RnsPlan {
    int t;
    uint32_t m[kMaxRns];
    uint32_t mi20[kMaxRns];     // floor(2^20 / m_t)
    uint32_t red[kMaxRns];      // floor(2^(31+b) / m_t) to 32 bits, b the bit length of m_t
    int sh[kMaxRns];            // b - 1
    uint32_t ea[kMaxRns][2];    // bytes 256^i mod m_t, i = 0..7
    uint32_t eb[kMaxRns][2];    // bytes (M / m_t)^-1 256^i mod m_t
    uint32_t f[kRnsGroups];     // bytes 2^15 / m_t rounded, four moduli per word
    uint32_t w[kRnsGroups][8];  // word (g, j): byte j of W_t = (M / m_t) mod p (times 2^64 mod p when mont), four moduli
    uint32_t nlo, nhi;          // (p - M mod p) mod p (times 2^64 mod p when mont): low and high 32 bits
    uint64_t p;
    uint64_t ninv;              // -p^-1 mod 2^64 (mont)
    EpiRed red32;               // p < 2^32: the reduction of the last sum
    int mont;
};

// x mod m from the byte dot products s = sum_i x_i e_i < 8 255^2 < 2^19: the
// quotient estimate is floor(s / m) or one less.
__device__ __forceinline__ uint32_t res_byte(uint32_t s, uint32_t m, uint32_t mi20) {
    const uint32_t r = s - ((s * mi20) >> 20) * m;
    return min(r, r - m);
}
__device__ __forceinline__ uint32_t byte_dot(uint32_t x, uint32_t e0, uint32_t) { return __dp4a(x, e0, 0u); }
__device__ __forceinline__ uint32_t byte_dot(uint64_t x, uint32_t e0, uint32_t e1) {
    return __dp4a(static_cast<uint32_t>(x >> 32), e1, __dp4a(static_cast<uint32_t>(x), e0, 0u));
}

using u128 = unsigned __int128;

// (hi 2^64 + lo) 2^-64 mod p for hi 2^64 + lo < p 2^64, p odd and < 2^63
__device__ __forceinline__ uint64_t redc(uint64_t lo, uint64_t hi, uint64_t p, uint64_t ninv) {
    const uint64_t m = lo * ninv;
    const uint64_t ml = m * p, mh = __umul64hi(m, p);
    const uint64_t c = (lo + ml) < lo ? 1u : 0u;  // lo + m p == 0 mod 2^64
    const uint64_t r = hi + mh + c;
    return r >= p ? r - p : r;
}

__device__ __forceinline__ uint64_t add_mod64(uint64_t a, uint64_t b, uint64_t p) {
    const uint64_t s = a + b;
    return (s < a || s >= p) ? s - p : s;
}
__device__ __forceinline__ uint64_t sub_mod64(uint64_t a, uint64_t b, uint64_t p) {
    return a >= b ? a - b : a + (p - b);
}
__device__ __forceinline__ uint64_t combine64(uint64_t old, uint64_t v, int op, uint64_t p) {
    return op == HME_SET ? v : op == HME_ADD ? add_mod64(old, v, p) : sub_mod64(old, v, p);
}

// Both operands' planes in one launch.  Blocks [0, a_blocks): plane t of A, [m][Kp],
// 16 k per thread, one 16-byte store per plane.  The rest: plane t of B, [n][Kp]
// (transposed through shared memory, 64 k x 32 n per block, 8 k per thread).
// Zero for k in [K, Kp).  Bound by the writes (t bytes per entry against the
// 4 or 8 read) and the residues' arithmetic in equal parts.
template <class T>
__global__ void __launch_bounds__(256) rns_split_kernel(const T* __restrict__ A, uint64_t lda, const T* __restrict__ B,
                                                        uint64_t ldb, uint32_t m, uint32_t n, uint32_t k, uint32_t Kp,
                                                        uint8_t* __restrict__ pa, uint8_t* __restrict__ pb,
                                                        uint32_t a_blocks, const __grid_constant__ RnsPlan P) {
    __shared__ T tile[64][33];
    grid_dep_launch();  // the GEMM that follows may start its set-up
    if (blockIdx.x < a_blocks) {
        const uint32_t kch = Kp >> 4;
        const size_t total = static_cast<size_t>(m) * kch, plane = static_cast<size_t>(m) * Kp;
        for (size_t idx = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; idx < total;
             idx += static_cast<size_t>(a_blocks) * blockDim.x) {
            const uint32_t row = static_cast<uint32_t>(idx / kch);
            const uint32_t k0 = static_cast<uint32_t>(idx - static_cast<size_t>(row) * kch) << 4;
            const T* src = A + row * lda + k0;
            T x[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) x[e] = k0 + e < k ? src[e] : T(0);
            uint8_t* dst = pa + static_cast<size_t>(row) * Kp + k0;
            for (int t = 0; t < P.t; ++t, dst += plane) {
                const uint32_t e0 = P.ea[t][0], e1 = P.ea[t][1], md = P.m[t], mi = P.mi20[t];
                uint32_t w[4];
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    w[g] = 0;
#pragma unroll
                    for (int e = 0; e < 4; ++e) w[g] |= res_byte(byte_dot(x[4 * g + e], e0, e1), md, mi) << (8 * e);
                }
                *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
            }
        }
    } else {
        const uint32_t bk = (Kp + 63) / 64, blk = blockIdx.x - a_blocks;
        const uint32_t k0 = (blk % bk) * 64, n0 = (blk / bk) * 32;
        T v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const uint32_t t = threadIdx.x + 256 * q, kk = k0 + (t >> 5), c = n0 + (t & 31);
            v[q] = (kk < k && c < n) ? B[kk * ldb + c] : T(0);
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const uint32_t t = threadIdx.x + 256 * q;
            tile[t >> 5][t & 31] = v[q];
        }
        __syncthreads();
        const uint32_t nn = threadIdx.x >> 3, kc = threadIdx.x & 7;
        const uint32_t col = n0 + nn, kb = k0 + kc * 8;
        if (col >= n || kb >= Kp) return;
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = tile[kc * 8 + e][nn];
        uint8_t* dst = pb + static_cast<size_t>(col) * Kp + kb;
        const size_t plane = static_cast<size_t>(n) * Kp;
        for (int t = 0; t < P.t; ++t, dst += plane) {
            const uint32_t e0 = P.eb[t][0], e1 = P.eb[t][1], md = P.m[t], mi = P.mi20[t];
            uint32_t w[2];
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                w[g] = 0;
#pragma unroll
                for (int e = 0; e < 4; ++e) w[g] |= res_byte(byte_dot(v[4 * g + e], e0, e1), md, mi) << (8 * e);
            }
            *reinterpret_cast<uint2*>(dst) = make_uint2(w[0], w[1]);
        }
    }
}

// The products of all moduli: tiles of modulus 0 first, then 1, .., each in the
// grouped raster of the limb GEMM.  The planes of one operand are one tensor of
// t m (t n) rows; a tile that runs past its plane reads the next plane's rows,
// which only reach accumulator rows and columns that are not stored.
template <int BN>
struct RnsTiles {
    const CUtensorMap* tmA;
    const CUtensorMap* tmB;
    int M, N, t, k_begin, kblocks_, tiles_m, tiles_n;

    __device__ __forceinline__ int total() const { return t * tiles_m * tiles_n; }
    __device__ __forceinline__ int kblocks(int) const { return kblocks_; }
    __device__ __forceinline__ void prefetch_maps() const {
        if (threadIdx.x == 0) {
            prefetch_tmap(tmA);
            prefetch_tmap(tmB);
        }
    }
    __device__ __forceinline__ void place(int tile, int& md, int& tm, int& tn) const {
        const int per = tiles_m * tiles_n;
        md = tile / per;
        const int local = tile - md * per;
        const int per_group = 16 * tiles_n, grp = local / per_group, first_m = 16 * grp;
        const int gm = min(tiles_m - first_m, 16), in = local - grp * per_group;
        tm = first_m + in % gm;
        tn = in / gm;
    }
    __device__ __forceinline__ TileRef tile(int i) const {
        int md, tm, tn;
        place(i, md, tm, tn);
        TileRef r{};
        r.tmA = tmA;
        r.tmB = tmB;
        r.a_row = md * M + tm * kBM;
        r.b_col = md * N + tn * BN;
        r.k_begin = k_begin;
        r.kblocks = kblocks_;
        return r;
    }
};

// Accumulators to bytes mod m_t: 32 columns of its row per thread and step, one
// multiply-high per entry, two 16-byte stores; rows of the output planes are
// Np bytes, a multiple of 32.
template <int BN, int KB>
struct RnsEpilogue {
    uint8_t* Y;
    int Np, add;
    const RnsPlan& P;

    template <class Src>
    __device__ __forceinline__ void run(const Src& src, int first, int end, int step, int warp, int lane,
                                        uint32_t tmem_base, uint32_t*, uint64_t* acc_full, uint64_t* acc_empty,
                                        volatile int* abort_flag, int* err) const {
        using CF = Cfg<1, BN, KB>;
        constexpr int STEP = 32 * (epi_warps(1) / 4);
        const int q = warp & 3, grp = (warp - 2) >> 2;
        const uint32_t lane_base = static_cast<uint32_t>(q * 32) << 16;
        int lt = 0;
        for (int tile = first; tile < end; tile += step, ++lt) {
            const int a = lt & 1;
            int md, tm, tn;
            src.place(tile, md, tm, tn);
            const uint32_t m = P.m[md], rd = P.red[md];
            const int sh = P.sh[md], row = tm * kBM + q * 32 + lane;
            uint8_t* dst = Y + (static_cast<size_t>(md) * src.M + row) * Np + tn * BN;
            if (!mbar_wait(&acc_full[a], (lt >> 1) & 1, abort_flag, err, DERR_WAIT_ACCUM)) break;
            tc_fence_after();
            const uint32_t taddr = tmem_base + lane_base + a * CF::ACC_STRIDE;
            if (32 * grp >= BN) mbar_arrive(&acc_empty[a]);
#pragma unroll 1
            for (int c0 = 32 * grp; c0 < BN; c0 += STEP) {
                uint32_t v[2][16];
                tmem_ld16(taddr + c0, v[0]);
                tmem_ld16(taddr + c0 + 16, v[1]);
                tmem_wait_ld();
                if (c0 + STEP >= BN) {
                    tc_fence_before();
                    mbar_arrive(&acc_empty[a]);
                }
                const bool live = row < src.M && tn * BN + c0 < Np;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t w[4];
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        w[g] = 0;
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const uint32_t s = v[h][4 * g + e];
                            const uint32_t x = s - (__umulhi(s, rd) >> sh) * m;
                            w[g] |= min(x, x - m) << (8 * e);
                        }
                    }
                    if (live) {
                        uint4* out = reinterpret_cast<uint4*>(dst + c0 + 16 * h);
                        if (add) {  // a later chunk of K
                            const uint4 o = *out;
                            const uint32_t ow[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
                            for (int g = 0; g < 4; ++g) {
                                uint32_t z = 0;
#pragma unroll
                                for (int e = 0; e < 4; ++e) {
                                    const uint32_t x = ((w[g] >> (8 * e)) & 0xffu) + ((ow[g] >> (8 * e)) & 0xffu);
                                    z |= min(x, x - m) << (8 * e);
                                }
                                w[g] = z;
                            }
                        }
                        *out = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                }
            }
        }
    }
};

template <int BN, int KB>
__global__ void __launch_bounds__(gemm_threads(1), 1)
    rns_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, int M, int N,
                    int k_begin, int kblocks, uint8_t* Y, int Np, int add, int* err,
                    const __grid_constant__ RnsPlan P) {
    long_tiles<1, BN, KB>(
        RnsTiles<BN>{&tmA, &tmB, M, N, P.t, k_begin, kblocks, (M + kBM - 1) / kBM, (N + BN - 1) / BN},
        RnsEpilogue<BN, KB>{Y, Np, add, P}, err);
}

// C[r][c] op= CRT(Y_.[r][c]) mod p, four columns per thread: the Y of four moduli
// and four columns come as four words, transposed by byte permutes, so that
// each constant's byte j takes one dp4a per four moduli.
template <class T>
__global__ void __launch_bounds__(256) rns_crt_kernel(const uint8_t* __restrict__ Y, uint32_t rows, uint32_t cols,
                                                      uint32_t Np, T* __restrict__ C, uint64_t ldc, int op,
                                                      const __grid_constant__ RnsPlan P) {
    constexpr int NJ = sizeof(T);
    const size_t plane = static_cast<size_t>(rows) * Np;
    const uint32_t quads = (cols + 3) / 4;
    const size_t total = static_cast<size_t>(rows) * quads;
    for (size_t idx = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; idx < total;
         idx += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const uint32_t r = static_cast<uint32_t>(idx / quads), c = 4 * static_cast<uint32_t>(idx - static_cast<size_t>(r) * quads);
        const uint8_t* src = Y + static_cast<size_t>(r) * Np + c;
        uint32_t s[4][NJ] = {}, wf[4] = {};
        for (int t0 = 0, g = 0; t0 < P.t; t0 += 4, ++g) {
            uint32_t y[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
                y[e] = t0 + e < P.t ? *reinterpret_cast<const uint32_t*>(src + (t0 + e) * plane) : 0u;
            const uint32_t l01 = __byte_perm(y[0], y[1], 0x5140), h01 = __byte_perm(y[0], y[1], 0x7362);
            const uint32_t l23 = __byte_perm(y[2], y[3], 0x5140), h23 = __byte_perm(y[2], y[3], 0x7362);
            const uint32_t z[4] = {__byte_perm(l01, l23, 0x5410), __byte_perm(l01, l23, 0x7632),
                                   __byte_perm(h01, h23, 0x5410), __byte_perm(h01, h23, 0x7632)};
            const uint32_t f = P.f[g];
#pragma unroll
            for (int u = 0; u < 4; ++u) wf[u] = __dp4a(z[u], f, wf[u]);
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const uint32_t wj = P.w[g][j];
#pragma unroll
                for (int u = 0; u < 4; ++u) s[u][j] = __dp4a(z[u], wj, s[u][j]);
            }
        }
        T* cp = C + r * ldc + c;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (c + u >= cols) break;
            const uint32_t w = (wf[u] + (1u << 14)) >> 15;
            // sums below 22 255^2 < 2^21 per byte place, so each half stays below 2^47
            uint64_t s0 = static_cast<uint64_t>(w) * P.nlo;
#pragma unroll
            for (int j = 0; j < 4; ++j) s0 += static_cast<uint64_t>(s[u][j]) << (8 * j);
            if constexpr (NJ == 8) {
                uint64_t s1 = static_cast<uint64_t>(w) * P.nhi;
#pragma unroll
                for (int j = 4; j < 8; ++j) s1 += static_cast<uint64_t>(s[u][j]) << (8 * (j - 4));
                const uint64_t lo = s0 + (s1 << 32);
                const uint64_t hi = (s1 >> 32) + (lo < s0 ? 1u : 0u);
                const uint64_t v = P.mont ? redc(lo, hi, P.p, P.ninv)
                                          : static_cast<uint64_t>(((static_cast<u128>(hi) << 64) | lo) % P.p);
                cp[u] = combine64(op == HME_SET ? 0u : cp[u], v, op, P.p);
            } else {
                const uint32_t p = static_cast<uint32_t>(P.p);
                const uint32_t v = P.red32.fast ? epi_reduce_u64<true>(s0, P.red32) : epi_reduce_u64<false>(s0, P.red32);
                cp[u] = op == HME_SET ? v : op == HME_ADD ? mod_add(cp[u], v, p) : mod_sub(cp[u], v, p);
            }
        }
    }
}

// u64 -> u32 (entries below p < 2^32)
__global__ void __launch_bounds__(256) narrow_kernel(const uint64_t* __restrict__ X, uint64_t ldx, uint32_t rows,
                                                     uint32_t cols, uint32_t* __restrict__ out) {
    for (uint32_t r = blockIdx.y; r < rows; r += gridDim.y)
        for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < cols; c += gridDim.x * blockDim.x)
            out[static_cast<size_t>(r) * cols + c] = static_cast<uint32_t>(X[r * ldx + c]);
}
// C[r][c] op= R[r][c]  mod p
__global__ void __launch_bounds__(256) widen_kernel(const uint32_t* __restrict__ R, uint32_t rows, uint32_t cols,
                                                    uint64_t* __restrict__ C, uint64_t ldc, int op, uint64_t p) {
    for (uint32_t r = blockIdx.y; r < rows; r += gridDim.y)
        for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < cols; c += gridDim.x * blockDim.x) {
            uint64_t* cp = C + r * ldc + c;
            *cp = combine64(op == HME_SET ? 0u : *cp, R[static_cast<size_t>(r) * cols + c], op, p);
        }
}
__global__ void zero64_kernel(uint64_t* C, uint64_t ldc, uint32_t rows, uint32_t cols) {
    for (uint32_t r = blockIdx.y; r < rows; r += gridDim.y)
        for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < cols; c += gridDim.x * blockDim.x)
            C[r * ldc + c] = 0;
}

dim3 grid2d(uint32_t rows, uint32_t cols, int sms) {
    const uint32_t gx = std::min<uint32_t>((cols + 255) / 256, 64);
    const uint32_t gy = std::max<uint32_t>(1, std::min<uint32_t>(rows, static_cast<uint32_t>(sms) * 16 / gx + 1));
    return dim3(gx, std::min<uint32_t>(gy, 65535));
}

uint64_t mulmod_host(uint64_t a, uint64_t b, uint64_t p) { return static_cast<uint64_t>(static_cast<u128>(a) * b % p); }
// The plan for modulus p and inner dimension k, entries of `bytes` bytes.
RnsPlan make_plan(uint64_t p, uint32_t k, int bytes) {
    RnsPlan P{};
    // bits needed: M > 4 k (p-1)^2, with one bit of margin on the double-precision logs
    const double need = std::log2(static_cast<double>(std::max<uint32_t>(k, 1))) +
                        2.0 * std::log2(static_cast<double>(p - 1)) + 3.0;
    double have = 0;
    while (have <= need) {
        HME_REQUIRE(P.t < kMaxRns, "gemm_u64: inner dimension too large for the residue system");
        P.m[P.t] = kModuli[P.t];
        have += std::log2(static_cast<double>(kModuli[P.t++]));
    }
    P.p = p;
    P.mont = bytes == 8 && (p & 1) && p < (uint64_t(1) << 63);
    // the last sum: 22 products of bytes per byte place and w N
    if (bytes == 4)
        P.red32 = make_epi_bound(make_mod(static_cast<uint32_t>(p)),
                                 (static_cast<unsigned __int128>(kMaxRns) * 255 * 255 * 0x01010101u) +
                                     (static_cast<unsigned __int128>(kMaxRns) << 32));
    const uint64_t r64 = P.mont ? static_cast<uint64_t>((static_cast<u128>(1) << 64) % p) : 1;  // 2^64 mod p
    uint64_t m_mod_p = 1;
    for (int t = 0; t < P.t; ++t) m_mod_p = mulmod_host(m_mod_p, P.m[t], p);
    for (int t = 0; t < P.t; ++t) {
        const uint32_t m = P.m[t];
        uint64_t mt_p = 1 % p;  // (M / m_t) mod p
        uint32_t mt_m = 1;      // (M / m_t) mod m_t
        for (int s = 0; s < P.t; ++s)
            if (s != t) {
                mt_p = mulmod_host(mt_p, P.m[s], p);
                mt_m = mt_m * P.m[s] % m;
            }
        uint32_t inv = 1;
        while (inv * mt_m % m != 1) ++inv;  // m <= 256
        int b = 0;
        while ((m >> b) != 0) ++b;
        P.mi20[t] = (1u << 20) / m;
        P.red[t] = static_cast<uint32_t>(std::min<uint64_t>(0xffffffffull, (uint64_t(1) << (31 + b)) / m));
        P.sh[t] = b - 1;
        uint32_t e = 1;
        for (int i = 0; i < 8; ++i, e = e * 256 % m) {
            P.ea[t][i / 4] |= (e % m) << (8 * (i % 4));
            P.eb[t][i / 4] |= (e * inv % m) << (8 * (i % 4));
        }
        P.f[t / 4] |= ((2u * 32768u + m) / (2u * m)) << (8 * (t % 4));
        const uint64_t w = P.mont ? mulmod_host(mt_p, r64, p) : mt_p;
        for (int j = 0; j < 8; ++j) P.w[t / 4][j] |= static_cast<uint32_t>((w >> (8 * j)) & 0xffu) << (8 * (t % 4));
    }
    const uint64_t neg = m_mod_p ? p - m_mod_p : 0;
    const uint64_t nm = P.mont ? mulmod_host(neg, r64, p) : neg;
    P.nlo = static_cast<uint32_t>(nm);
    P.nhi = static_cast<uint32_t>(nm >> 32);
    if (P.mont) {
        uint64_t inv = p;  // Newton: p inv == 1 mod 2^64
        for (int i = 0; i < 6; ++i) inv *= 2 - p * inv;
        P.ninv = 0 - inv;
    }
    return P;
}

// The largest first row of a plane: TMA coordinates are signed 32-bit numbers, and the stacked planes of one
// launch put row r of plane t at t m + r.
constexpr uint32_t kMaxPlaneRows = (1u << 31) - 256;

// One launch over moduli [t0, t0 + moduli) and a chunk of K after another.
template <int BN, int KB>
void launch_rns_run(hme_ctx* ctx, uint32_t m, uint32_t n, uint32_t k, int Kp, uint8_t* pa, uint8_t* pb, uint8_t* Y,
                    int Np, const RnsPlan& plan, int t0, int moduli) {
    using CF = Cfg<1, BN, KB>;
    RnsPlan P = plan;  // the run's moduli first
    P.t = moduli;
    for (int t = 0; t < moduli; ++t) {
        P.m[t] = plan.m[t0 + t];
        P.red[t] = plan.red[t0 + t];
        P.sh[t] = plan.sh[t0 + t];
    }
    pa += static_cast<size_t>(t0) * m * Kp;
    pb += static_cast<size_t>(t0) * n * Kp;
    Y += static_cast<size_t>(t0) * m * Np;
    CUtensorMap tmA, tmB;
    {
        const cuuint64_t dims[3] = {static_cast<cuuint64_t>(Kp), static_cast<cuuint64_t>(m) * P.t, 1};
        const cuuint64_t strides[2] = {static_cast<cuuint64_t>(Kp), static_cast<cuuint64_t>(Kp) * m * P.t};
        const cuuint32_t box[3] = {KB, kBM, 1};
        encode_tma_u8_kb(&tmA, pa, 3, dims, strides, box, KB);
    }
    {
        const cuuint64_t dims[4] = {static_cast<cuuint64_t>(Kp), static_cast<cuuint64_t>(n) * P.t, 1, 1};
        const cuuint64_t strides[3] = {static_cast<cuuint64_t>(Kp), static_cast<cuuint64_t>(Kp) * n * P.t,
                                       static_cast<cuuint64_t>(Kp) * n * P.t};
        const cuuint32_t box[4] = {KB, BN, 1, 1};
        encode_tma_u8_kb(&tmB, pb, 4, dims, strides, box, KB);
    }
    const size_t tiles = static_cast<size_t>(P.t) * ((m + kBM - 1) / kBM) * ((n + BN - 1) / BN);
    HME_REQUIRE(tiles < (size_t(1) << 31), "gemm_u64: too many tiles");
    const int sms = ctx->gemm_sm_cap > 0 ? std::min(ctx->gemm_sm_cap, ctx->num_sms) : ctx->num_sms;
    const uint32_t chunk = limb_k_chunk(1);
    for (uint32_t k0 = 0; k0 < k; k0 += chunk) {
        const uint32_t kc = std::min(chunk, k - k0);
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(static_cast<unsigned>(std::min<size_t>(tiles, sms)));
        cfg.blockDim = dim3(gemm_threads(1));
        cfg.dynamicSmemBytes = CF::SMEM;
        cfg.stream = ctx->stream;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = t0 == 0 && k0 == 0 && !ctx->timer.on ? 1 : 0;
        HME_TIMED(ctx, "limb_gemm",
                  HME_CUDA(cudaLaunchKernelEx(&cfg, rns_gemm_kernel<BN, KB>, tmA, tmB, static_cast<int>(m),
                                              static_cast<int>(n), static_cast<int>(k0),
                                              static_cast<int>((kc + KB - 1) / KB), Y, Np, k0 == 0 ? 0 : 1, ctx->d_err,
                                              P)));
    }
}

template <int BN, int KB>
void launch_rns_gemm(hme_ctx* ctx, uint32_t m, uint32_t n, uint32_t k, int Kp, uint8_t* pa, uint8_t* pb, uint8_t* Y,
                     int Np, const RnsPlan& P) {
    static OncePerDevice attr;
    attr.run([](int) {
        HME_CUDA(cudaFuncSetAttribute(rns_gemm_kernel<BN, KB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      Cfg<1, BN, KB>::SMEM));
    });
    // all moduli in one launch, unless their planes' rows pass the coordinates (8 x 200 000 000 mod 2^40 - 87)
    const int run = static_cast<int>(std::min<uint32_t>(P.t, kMaxPlaneRows / std::max(m, n)));
    for (int t0 = 0; t0 < P.t; t0 += run)
        launch_rns_run<BN, KB>(ctx, m, n, k, Kp, pa, pb, Y, Np, P, t0, std::min(run, P.t - t0));
}

// C op= A*B mod p over the residue system; pa, pb, Y: the planes' buffers.
template <class T>
void rns_gemm(hme_ctx* ctx, const RnsPlan& P, uint32_t m, uint32_t n, uint32_t k, const T* A, size_t lda, const T* B,
              size_t ldb, T* C, size_t ldc, int op, uint8_t* pa, uint8_t* pb, uint8_t* Y) {
    const int Kp = limb_kp(k), Np = static_cast<int>((n + 31) / 32 * 32), sms = ctx->num_sms;
    const uint32_t ga = static_cast<uint32_t>(std::min<size_t>((static_cast<size_t>(m) * (Kp / 16) + 255) / 256, sms * 16ull));
    const uint32_t gb = static_cast<uint32_t>((Kp + 63) / 64) * ((n + 31) / 32);
    HME_TIMED(ctx, "rns_split", rns_split_kernel<T><<<ga + gb, 256, 0, ctx->stream>>>(A, lda, B, ldb, m, n, k, Kp, pa, pb,
                                                                                      ga, P));
    HME_CUDA(cudaGetLastError());
    auto gemm = [&](auto bn, auto kb) {
        launch_rns_gemm<decltype(bn)::value, decltype(kb)::value>(ctx, m, n, k, Kp, pa, pb, Y, Np, P);
    };
    using std::integral_constant;
    auto by_k = [&](auto bn) {
        if (k <= 32) gemm(bn, integral_constant<int, 32>{});
        else if (k <= 64) gemm(bn, integral_constant<int, 64>{});
        else gemm(bn, integral_constant<int, 128>{});
    };
    if (n > 128) by_k(integral_constant<int, 256>{});
    else by_k(integral_constant<int, 128>{});
    const size_t quads = static_cast<size_t>(m) * ((n + 3) / 4);
    HME_TIMED(ctx, "rns_crt", rns_crt_kernel<T><<<static_cast<unsigned>(std::min<size_t>((quads + 255) / 256, sms * 16ull)), 256, 0,
                                                  ctx->stream>>>(Y, m, n, Np, C, ldc, op, P));
    HME_CUDA(cudaGetLastError());
}

size_t align256(size_t x) { return (x + 255) / 256 * 256; }

// C op= A*B mod p, device pointers, on ctx->stream.
void gemm_u64_device(hme_ctx* ctx, uint64_t p, uint32_t m, uint32_t n, uint32_t k, const uint64_t* A, size_t lda,
                     const uint64_t* B, size_t ldb, uint64_t* C, size_t ldc, int op) {
    HME_REQUIRE(p >= 2, "gemm_u64: modulus must be >= 2");
    HME_REQUIRE(op == HME_SET || op == HME_ADD || op == HME_SUB, "gemm_u64: op must be HME_SET, HME_ADD or HME_SUB");
    if (m == 0 || n == 0) return;
    HME_REQUIRE(C && ldc >= n, "gemm_u64: bad C");
    if (k == 0) {
        if (op == HME_SET) {
            HME_TIMED(ctx, "zero64", zero64_kernel<<<grid2d(m, n, ctx->num_sms), 256, 0, ctx->stream>>>(C, ldc, m, n));
            HME_CUDA(cudaGetLastError());
        }
        return;
    }
    HME_REQUIRE(A && B && lda >= k && ldb >= n, "gemm_u64: bad A / B");
    HME_REQUIRE(std::max({m, n, k}) <= kMaxPlaneRows, "gemm_u64: dimension too large");
    const int sms = ctx->num_sms;
    if (p < (uint64_t(1) << 32)) {
        uint32_t* a32 = static_cast<uint32_t*>(ctx->ws.get(kSlotRns0, 4ull * m * k));
        uint32_t* b32 = static_cast<uint32_t*>(ctx->ws.get(kSlotRns1, 4ull * k * n));
        uint32_t* c32 = static_cast<uint32_t*>(ctx->ws.get(kSlotRns2, 4ull * m * n));
        HME_TIMED(ctx, "narrow", narrow_kernel<<<grid2d(m, k, sms), 256, 0, ctx->stream>>>(A, lda, m, k, a32));
        HME_TIMED(ctx, "narrow", narrow_kernel<<<grid2d(k, n, sms), 256, 0, ctx->stream>>>(B, ldb, k, n, b32));
        HME_CUDA(cudaGetLastError());
        gemm_u32_device(ctx, make_mod(static_cast<uint32_t>(p)), m, n, k, a32, k, b32, n, c32, n, HME_SET);
        HME_TIMED(ctx, "widen", widen_kernel<<<grid2d(m, n, sms), 256, 0, ctx->stream>>>(c32, m, n, C, ldc, op, p));
        HME_CUDA(cudaGetLastError());
        return;
    }
    const RnsPlan P = make_plan(p, k, 8);
    const int Kp = limb_kp(k);
    uint8_t* pa = static_cast<uint8_t*>(ctx->ws.get(kSlotRns0, static_cast<size_t>(P.t) * m * Kp));
    uint8_t* pb = static_cast<uint8_t*>(ctx->ws.get(kSlotRns1, static_cast<size_t>(P.t) * n * Kp));
    uint8_t* Y = static_cast<uint8_t*>(ctx->ws.get(kSlotRns2, static_cast<size_t>(P.t) * m * ((n + 31) / 32 * 32)));
    rns_gemm(ctx, P, m, n, k, A, lda, B, ldb, C, ldc, op, pa, pb, Y);
}

}  // namespace

// Whether a u32 product over the residue system beats the limb product: the
// four-limb one costs 16 products of 2 m n k int8 operations, this one t = 8 to 11
// and more in its split and CRT.  Both sides' times in us, fitted to measured
// ones (p = 2^31 - 19, limbs / residue system): 64 x 64 x 8192 83 / 36, 300 x 300
// x 8000 95 / 52, 2048^3 128 / 121, 4096^3 829 / 664, 1024^3 26 / 38, 4096 x 4096
// x 1024 220 / 264, 1677 x 771 x 1419 52 / 53.
bool rns_gemm_u32_pays(const ModParams& mp, uint32_t m, uint32_t n, uint32_t k, int sms) {
    if (mp.limbs < 4) return false;  // 9 moduli against 9 limb products below 2^24
    const double mk = static_cast<double>(m) * k, kn = static_cast<double>(k) * n, mn = static_cast<double>(m) * n;
    const double kb = (k + 127) / 128, tm = (m + kBM - 1) / kBM;
    const double bits = std::log2(static_cast<double>(k)) + 2 * std::log2(static_cast<double>(mp.p)) + 3;
    const double t = std::ceil(bits / 7.93);
    const bool narrow = 4 * tm * ((n + 63) / 64) < 3.0 * sms;
    const double lt = tm * ((n + (narrow ? 31 : 63)) / (narrow ? 32 : 64)), rt = t * tm * ((n + 255) / 256);
    const double limb = 6 + (8 * mk + 20 * kn) / 4.5e6 + std::ceil(lt / sms) * (4 * kb * (narrow ? 0.27 : 0.38) + 2);
    const double rns = 14 + (mk + kn) * t * 3.5e-7 + std::ceil(rt / sms) * (kb * 0.38 + 1.5) + mn * t * 4.0e-7;
    return rns < 0.95 * limb;
}

// C op= A*B mod p, u32 entries, p < 2^32, device pointers, on ctx->stream; false, with nothing done, when its
// planes (up to twice the limb product's) cannot be had.
bool rns_gemm_u32_device(hme_ctx* ctx, const ModParams& mp, uint32_t m, uint32_t n, uint32_t k, const uint32_t* A,
                         size_t lda, const uint32_t* B, size_t ldb, uint32_t* C, size_t ldc, int op) {
    const RnsPlan P = make_plan(mp.p, k, 4);
    const int Kp = limb_kp(k);
    const size_t pbytes = align256(static_cast<size_t>(P.t) * n * Kp);
    const size_t need_a = static_cast<size_t>(P.t) * m * Kp;
    const size_t need_b = pbytes + static_cast<size_t>(P.t) * m * ((n + 31) / 32 * 32);
    if (!ctx->ws.holds({{kSlotPlanesA, need_a}, {kSlotPlanesB, need_b}}, ctx->stream)) return false;
    uint8_t* pa = static_cast<uint8_t*>(ctx->ws.get(kSlotPlanesA, need_a));
    uint8_t* pb = static_cast<uint8_t*>(ctx->ws.get(kSlotPlanesB, need_b));
    rns_gemm(ctx, P, m, n, k, A, lda, B, ldb, C, ldc, op, pa, pb, pb + pbytes);
    return true;
}

}  // namespace hme

using namespace hme;

extern "C" {

int hme_gemm_u64_dev(hme_ctx* ctx, uint64_t p, uint32_t m, uint32_t n, uint32_t k, const uint64_t* A, size_t lda,
                     const uint64_t* B, size_t ldb, uint64_t* C, size_t ldc, int op) {
    return guard([&] {
        HME_REQUIRE(ctx != nullptr, "null context");
        bind(ctx);
        gemm_u64_device(ctx, p, m, n, k, A, lda, B, ldb, C, ldc, op);
    });
}

int hme_gemm_u64(hme_ctx* ctx, uint64_t p, uint32_t m, uint32_t n, uint32_t k, const uint64_t* A, size_t lda,
                 const uint64_t* B, size_t ldb, uint64_t* C, size_t ldc, int op) {
    return guard([&] {
        HME_REQUIRE(ctx != nullptr, "null context");
        HME_REQUIRE(op == HME_SET || op == HME_ADD || op == HME_SUB, "gemm_u64: op must be HME_SET, HME_ADD or HME_SUB");
        if (m == 0 || n == 0) return;
        HME_REQUIRE(C && ldc >= n && (k == 0 || (A && B && lda >= k && ldb >= n)), "gemm_u64: bad buffers");
        bind(ctx);
        uint64_t* dA = k ? static_cast<uint64_t*>(ctx->ws.get(kSlotStageA, 8ull * m * k)) : nullptr;
        uint64_t* dB = k ? static_cast<uint64_t*>(ctx->ws.get(kSlotStageB, 8ull * k * n)) : nullptr;
        uint64_t* dC = static_cast<uint64_t*>(ctx->ws.get(kSlotStageC, 8ull * m * n));
        if (k) {
            HME_CUDA(copy_rows_async(dA, 8ull * k, A, 8 * lda, 8ull * k, m, cudaMemcpyHostToDevice, ctx->stream));
            HME_CUDA(copy_rows_async(dB, 8ull * n, B, 8 * ldb, 8ull * n, k, cudaMemcpyHostToDevice, ctx->stream));
        }
        if (op != HME_SET)
            HME_CUDA(copy_rows_async(dC, 8ull * n, C, 8 * ldc, 8ull * n, m, cudaMemcpyHostToDevice, ctx->stream));
        gemm_u64_device(ctx, p, m, n, k, dA, k, dB, n, dC, n, op);
        if (op == HME_SET || k)
            HME_CUDA(copy_rows_async(C, 8 * ldc, dC, 8ull * n, 8ull * n, m, cudaMemcpyDeviceToHost, ctx->stream));
        HME_CUDA(cudaStreamSynchronize(ctx->stream));
        check_device_error(ctx);
    });
}

}  // extern "C"
