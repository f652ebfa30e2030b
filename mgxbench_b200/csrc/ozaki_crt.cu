// ozaki_crt.cu -- FP64-accurate GEMM on the INT8 tensor cores by Ozaki scheme II (the CRT form;
// Ozaki, Uchino & Imamura 2025, "Ozaki Scheme II: A GEMM-oriented emulation of floating-point
// matrix multiplication using an integer modular technique").
//
// Where the slice form (ozaki.cu) multiplies s digit slices pairwise (s(s+1)/2 INT8 products),
// this form scales each row of A and column of B by a power of two to integers, takes them modulo
// q pairwise-coprime moduli p_l <= 256, multiplies the residues (one INT8 product per modulus)
// and rebuilds the integer product by the Chinese remainder theorem.  q = 15 moduli give FP64
// accuracy at K = 16384, against 36 products for 8 slices.
//
//   moduli   the first q of 256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211,
//            199, 197, 193; P = p_1 ... p_q, L = bit length of P; alpha = (L-3)/2, beta = L-3-alpha.
//   scale    row i of A: e = frexp exponent of max|a_ik|, c_k = max(1, ceil(|a_ik| 2^(22-e))) for
//            a_ik != 0, S = sum c_k^2 (an integer sum, so the result does not depend on the
//            order), u = (bitlen(S-1)+1)/2, sigma_i = alpha - e + 22 - u; then 2^sigma_i ||a_i||
//            <= 2^alpha.  Columns of B likewise (tau_j, beta).  By Cauchy-Schwarz the exact
//            product C'_ij of A' = rint(2^sigma A) and B' = rint(B 2^tau) is below P/4.
//   residues A' mod p_l as int8 (symmetric; [-128, 127] for 256), B' likewise.
//   products R_l = (A'_l B'_l) mod p_l in [0, p_l), exact in int32 while K <= 130816.
//   CRT      w_l = (P/p_l) ((P/p_l)^-1 mod p_l) in three 40-bit chunks; s_t = sum_l w_t,l R_l is
//            exact in FP64; Q = rint((s1 + s2 2^-40) / P~); d_t = s_t - Q P_t (exact);
//            C_ij = fma(fma(d1, 2^40, d2), 2^40, d3) 2^(E3 - sigma_i - tau_j).
//
// Kernels:
//   crt_row_scale   sigma per row of A (one block per row, integer sum of squares)
//   crt_col_max / crt_col_sumsq   tau per column of B (integer atomics; the last block of a column
//                   group takes the scales)
//   crt_split_a     residues of A as swizzled K-major 256-row slabs [modulus][tile][K block]
//   crt_split_b     residues of B^T, same layout (thread per column, coalesced reads)
//   crt_gemm        persistent tcgen05 kernel over (modulus, 256 x 256 tile) work items:
//       warp 0      producer: one bulk copy per operand per stage (KPACK K blocks); at each new
//                   work item it waits (at most 20 us) until every CTA has started its item, so
//                   the CTAs that share an operand tile read it within microseconds of each
//                   other and mostly from L2 (DRAM reads at N = 16384: 118 -> 48 GB per launch)
//       warp 1      TMEM owner and MMA issuer: two M=128 N=256 K=32 kind::i8 MMAs per K block
//                   (rows 0-127 and 128-255), int32 accumulators in all 512 TMEM columns, each
//                   handed over on its own
//       warps 2-17  epilogue (16 warps, four per TMEM lane quarter, 64 columns each): both
//                   accumulators in turn: tcgen05.ld, release, exact reduction mod p_l (biased
//                   Barrett), one byte per output
//   crt_combine     CRT recombination of the q residue planes, scaling, (C +) store
// All waits are bounded (mgx_common.cuh); TMEM is always released before the CTA exits.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>

#include "crt_pairs.h"
#include "mgx_common.cuh"

namespace mgx {
namespace crt {

constexpr int MAXQ = 16;
constexpr int MINQ = 8;
constexpr int KMAX = 130816;           // 4088 K blocks: k * 128 * 128 < 2^31
constexpr int TILE = 256;              // output tile TILE x TILE, operand slabs TILE rows
constexpr int KB = 32;                 // bytes of K per MMA
constexpr int SLAB = TILE * KB;        // 8 KiB: one operand, one K block
// K blocks per pipeline stage.  Shorter stages cost more than the deeper ring gives: pairs, K = N =
// 16384, 51.4 ms with 4 stages of 4 K blocks, 55.9 with 8 of 2, 67.0 with 16 of 1.
constexpr int KPACK = 4;
constexpr int EPI_WARPS = 16;          // four per TMEM lane quarter, 64 columns of either accumulator each
constexpr int THREADS = (2 + EPI_WARPS) * 32;
constexpr int NONFINITE = 0x7fffffff;
constexpr int OUT_TILE_BYTES = TILE * TILE;   // one residue byte per output
constexpr int RASTER = 16;             // tile rows that sweep the columns together

__constant__ int c_moduli[MAXQ] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193};
static const int h_moduli[MAXQ] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193};

// The same as compile-time constants: unrolled code takes them as immediates.
__host__ __device__ constexpr uint32_t modulus(int l)
{
    constexpr uint32_t p[MAXQ] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193};
    return p[l];
}

// Host-computed constants of one modulus set.
struct Consts {
    int q, L, alpha, beta;
    int E3;                // L - 120 + 60
    // CRT recombination, scaled by powers of two (see crt_combine)
    double w[MAXQ][3];     // CRT weights in 40-bit chunks, 2^974
    double pc[3];          // P in 40-bit chunks, 2^-60
    double inv_phat;       // 2^60 / (P / 2^(L-40))
    uint32_t barrett[MAXQ];  // ceil(2^32 / p_l)
};

// ---------------------------------------------------------------- shared numerics
__host__ __device__ __forceinline__ int frexp_exp_bits(unsigned long long absbits)
{
    if (absbits == 0) return 0;
    const int biased = (int)(absbits >> 52);
    if (biased != 0) return biased - 1022;
    const unsigned long long mant = absbits & ((1ull << 52) - 1);
#ifdef __CUDA_ARCH__
    return -1022 - (__clzll((long long)mant) - 12);
#else
    return -1022 - (__builtin_clzll(mant) - 12);
#endif
}

__device__ __forceinline__ double pow2i(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }

__device__ __forceinline__ double scale2(double x, int e)
{
    if (e >= -1022 && e <= 1023) return __dmul_rn(x, pow2i(e));
    const int e1 = e / 2, e2 = e - e1;
    return __dmul_rn(__dmul_rn(x, pow2i(e1)), pow2i(e2));
}

// 2^e as f1 f2, the factors scale2 multiplies by (f2 = 1 when one factor is enough).
__device__ __forceinline__ void scale_factors(int e, double &f1, double &f2)
{
    if (e >= -1022 && e <= 1023) {
        f1 = pow2i(e);
        f2 = 1.0;
    } else {
        const int e1 = e / 2;
        f1 = pow2i(e1);
        f2 = pow2i(e - e1);
    }
}

// ceil(|x| 2^(22-e))^2 for x != 0 (at least 1), 0 for x == 0, with 2^(22-e) = f1 f2 as
// scale_factors gives it (the same products as scale2).  |x| < 2^e, so the ceiling is an integer
// in [1, 2^22]: its low 32 bits come from 2^52 + c, and the square is one 32 x 32 -> 64 multiply.
__device__ __forceinline__ unsigned long long sq_term(double x, double f1, double f2)
{
    const double ax = fabs(x);
    if (ax == 0.0) return 0ull;
    double c = ceil(__dmul_rn(__dmul_rn(ax, f1), f2));
    if (c < 1.0) c = 1.0;
    const uint32_t ci = (uint32_t)__double2loint(__dadd_rn(c, 4503599627370496.0));
    return (unsigned long long)ci * ci;
}

// Scale exponent from the exponent of the maximum and the integer sum of squares.
__device__ __forceinline__ int sigma_of(unsigned long long mx, unsigned long long S, int target)
{
    if (mx == 0) return 0;
    const int e = frexp_exp_bits(mx);
    const int bl = (S - 1) ? 64 - __clzll((long long)(S - 1)) : 0;
    return target - e + 22 - (bl + 1) / 2;
}

// ---------------------------------------------------------------- scale kernels
// What the column passes add to and count with, zeroed before them: by the row pass of the same
// split, or by crt_zero.
struct ColStats {
    unsigned long long *max, *sum;  // per column
    unsigned int *arrived;          // per group of 256 columns: blocks of crt_col_sumsq that are done
    int n;
};

__device__ __forceinline__ void zero_stats(const ColStats &z, long long i, long long step)
{
    for (; i < z.n; i += step) {
        z.max[i] = 0ull;
        z.sum[i] = 0ull;
        if (i % 256 == 0) z.arrived[i / 256] = 0u;
    }
}

__global__ void __launch_bounds__(256) crt_zero(const ColStats z)
{
    pdl_wait();
    pdl_trigger();
    zero_stats(z, blockIdx.x * 256 + threadIdx.x, gridDim.x * 256ll);
}

// Maximum over a warp of non-negative doubles' bit patterns, as far as the scale needs it: the high
// words' maximum, and the low words' only where no high word is set (the exponent of a value with a
// non-zero high word does not depend on its low word, nor do the zero and non-finite tests).
__device__ __forceinline__ unsigned long long warp_max_bits(unsigned long long v)
{
    const uint32_t hi = __reduce_max_sync(0xffffffffu, (uint32_t)(v >> 32));
    if (hi != 0) return (unsigned long long)hi << 32;
    return __reduce_max_sync(0xffffffffu, (uint32_t)v);
}

// One block of T threads per row: the row's maximum, then its integer sum of squares.
// KEEP > 0: rows of at most KEEP x T elements, held in registers, so A is read once and the loads of a
// row are all in flight together.  Longer rows (KEEP = 0, 512 threads): the second pass finds
// the row in L2 (at 4 blocks per SM, 592 rows, 77 MB at k = 16384, are in flight, against L2's 126 MB),
// so A is read from DRAM once there too.  With 512 threads and two passes for every row, 2501 rows of
// 3001 took 25 us, mostly waiting on a few short loads per thread; now 16.
template <int T, int KEEP>
__global__ void __launch_bounds__(T) crt_row_scale(const double *__restrict__ A, int m, int k, int lda, int target,
                                                   int *__restrict__ sg, const ColStats z, int *status)
{
    __shared__ unsigned long long red[T / 32], sum[T / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row = blockIdx.x;
    pdl_wait();
    pdl_trigger();
    zero_stats(z, (long long)blockIdx.x * T + threadIdx.x, (long long)gridDim.x * T);
    const double *r = A + (size_t)row * lda;
    unsigned long long mx = 0;
    double v[KEEP > 0 ? KEEP : 1];
    if constexpr (KEEP > 0) {
#pragma unroll
        for (int u = 0; u < KEEP; ++u) {
            const int kk = threadIdx.x + u * T;
            v[u] = kk < k ? __ldg(r + kk) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < KEEP; ++u) {
            const unsigned long long b = (unsigned long long)__double_as_longlong(v[u]) & 0x7fffffffffffffffull;
            mx = b > mx ? b : mx;
        }
    } else {
        for (int kk = threadIdx.x; kk < k; kk += T) {
            const unsigned long long b = (unsigned long long)__double_as_longlong(__ldg(r + kk)) & 0x7fffffffffffffffull;
            mx = b > mx ? b : mx;
        }
    }
    mx = warp_max_bits(mx);
    if (lane == 0) red[warp] = mx;
    __syncthreads();
    mx = warp_max_bits(lane < T / 32 ? red[lane] : 0ull);
    if (mx >= 0x7ff0000000000000ull) {
        if (threadIdx.x == 0) {
            sg[row] = NONFINITE;
            record_status(status, kDevNonFinite);
        }
        return;
    }
    const int e = frexp_exp_bits(mx);
    double f1, f2;
    scale_factors(22 - e, f1, f2);
    unsigned long long S = 0;  // an exact integer sum: the order of its terms does not matter
    if (mx != 0) {
        if constexpr (KEEP > 0) {
#pragma unroll
            for (int u = 0; u < KEEP; ++u) S += sq_term(v[u], f1, f2);
        } else {
            int kk = threadIdx.x;
            for (; kk + 3 * T < k; kk += 4 * T) {
                double w[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) w[u] = __ldg(r + kk + u * T);
#pragma unroll
                for (int u = 0; u < 4; ++u) S += sq_term(w[u], f1, f2);
            }
            for (; kk < k; kk += T) S += sq_term(__ldg(r + kk), f1, f2);
        }
    }
    for (int o = 16; o > 0; o >>= 1) S += __shfl_xor_sync(0xffffffffu, S, o);
    if (lane == 0) sum[warp] = S;
    __syncthreads();
    if (warp == 0) {
        S = lane < T / 32 ? sum[lane] : 0ull;
        for (int o = T / 64; o > 0; o >>= 1) S += __shfl_xor_sync(0xffffffffu, S, o);
        if (lane == 0) sg[row] = sigma_of(mx, S, target);
    }
}

// grid (ceil(n/256), ychunks); each thread scans a run of rows of one column, 8 loads in flight.
// It reads B before it waits for the kernel before it, the residues of A or the clearing of colmax: that
// kernel writes nothing of B, and this one only starts once all its blocks have seen their own
// predecessors complete.  So the scan fills the end of the residue pass: whole products at 1024^3 62.3
// -> 58.3 us, 512^3 34.4 -> 31.8, 1.3% at 2501 x 1999 x 3001 (323 us in all).  The residue passes loading
// their values before the wait gained nothing more.
__global__ void __launch_bounds__(256) crt_col_max(const double *__restrict__ B, int k, int n, int ldb,
                                                   unsigned long long *colmax)
{
    const int j = blockIdx.x * 256 + threadIdx.x;
    if (j >= n) return;
    const int rows_per = (k + gridDim.y - 1) / gridDim.y;
    const int r0 = blockIdx.y * rows_per;
    const int r1 = min(k, r0 + rows_per);
    unsigned long long mx = 0;
    const unsigned long long *b = reinterpret_cast<const unsigned long long *>(B) + j;
    int r = r0;
    for (; r + 8 <= r1; r += 8) {
        unsigned long long v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = __ldg(b + (size_t)(r + u) * ldb) & 0x7fffffffffffffffull;
#pragma unroll
        for (int u = 0; u < 8; ++u) mx = v[u] > mx ? v[u] : mx;
    }
    for (; r < r1; ++r) {
        const unsigned long long v = __ldg(b + (size_t)r * ldb) & 0x7fffffffffffffffull;
        mx = v > mx ? v : mx;
    }
    pdl_wait();
    pdl_trigger();
    if (mx) atomicMax(colmax + j, mx);
}

// The same grid: sums of squares, then tau, taken by the last block of each column group to arrive.
__global__ void __launch_bounds__(256) crt_col_sumsq(const double *__restrict__ B, int k, int n, int ldb,
                                                     const ColStats z, int target, int *__restrict__ tu, int *status)
{
    __shared__ bool last;
    pdl_wait();
    pdl_trigger();
    const int j = blockIdx.x * 256 + threadIdx.x;
    const unsigned long long mx = j < n ? z.max[j] : 0ull;
    if (mx != 0 && mx < 0x7ff0000000000000ull) {
        const int e = frexp_exp_bits(mx);
        double f1, f2;
        scale_factors(22 - e, f1, f2);
        const int rows_per = (k + gridDim.y - 1) / gridDim.y;
        const int r0 = blockIdx.y * rows_per;
        const int r1 = min(k, r0 + rows_per);
        unsigned long long S = 0;  // an exact integer sum: the order of its terms does not matter
        int r = r0;
        for (; r + 8 <= r1; r += 8) {
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = __ldg(B + (size_t)(r + u) * ldb + j);
#pragma unroll
            for (int u = 0; u < 8; ++u) S += sq_term(v[u], f1, f2);
        }
        for (; r < r1; ++r) S += sq_term(__ldg(B + (size_t)r * ldb + j), f1, f2);
        if (S) atomicAdd(z.sum + j, S);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(z.arrived + blockIdx.x, 1u) == gridDim.y - 1;
    __syncthreads();
    if (!last || j >= n) return;
    __threadfence();
    if (mx >= 0x7ff0000000000000ull) {
        tu[j] = NONFINITE;
        record_status(status, kDevNonFinite);
    } else {
        tu[j] = sigma_of(mx, __ldcg(z.sum + j), target);
    }
}

// ---------------------------------------------------------------- residue kernels
// Residues of one value: x = rint(v 2^sg) (|x| < 2^63) is split exactly into xh 2^32 + xl with
// xh = rint(x 2^-32), |xl| <= 2^31, by adding 1.5 * 2^52: a double 1.5 * 2^52 + z with |z| < 2^51 is
// rounded to an integer by the add itself (nearest, ties to even, as rint) and holds z mod 2^32
// in its low word.  Two moduli p, p' share the FP64 part, their product pp <= 65280:
//   Y = fma(xh, 2^32 mod pp, xl + 1.5 * 2^52)      exact; Y = 1.5 * 2^52 + y, |y| < 2^48, y = x (mod pp)
//   t = fma(Y, 1/pp, magic)    low word off + rint(y / pp + d), |d| <= 1/2: the magic's rounding
//   u = lo(Y) - pp lo(t)       the bits of the float M + z, z = x (mod pp), |z| <= pp + 4, where off
//                              puts M's bits there (pp off = -bits(M) mod 2^32)
// and each residue follows in FP32, r = z - p rint(z / p) in [-(p-1)/2, (p-1)/2] for odd p, +-128 for
// 256, from q = fma(u, 1/p, 1.5 * 2^23 - rint(M/p)) and the low byte of u - p lo(q).  M in [2^23, 2^24)
// is a multiple of 256 (so it does not touch the low byte) for which M (1/p) with the rounded 1/p
// lies within 1.5 * 2^-10 of an integer for both moduli; z / p is never within 1 / (2p) of a
// half-integer for odd p.  The pairs are those for which such an M exists.  tests/test_crt_residues.py
// checks every z of every pair, and the first stage against exact integers.
// Bound by issue slots: 3.5 instructions per residue, one of them FP64 (two slots of that pipe), and
// 0.75 to pack the bytes.  With three FP64 operations and an integer one per modulus, rint and floor
// conversions and a finiteness test per value, the pass over B took 34 us at 3001 x 1999 with the FP64
// pipe 62% busy; now 31 us, with four blocks per SM instead of three.  Whole products: 2048 x 2048 x
// 16384 1.327 -> 1.300 ms, 4096^3 1.122 -> 1.108.
// The kernels split 8 values first (split32) and then run each pair over all 8 (all_residues).
constexpr double kRound = 6755399441055744.0;            // 1.5 * 2^52
constexpr double kRoundF = 12582912.0;                   // 1.5 * 2^23

struct ModulusPair {
    int a, b, M;   // indices of the moduli
};
struct PairSet {
    ModulusPair pair[MAXQ / 2];
    int single;    // the modulus left over where q is odd, else -1
};
constexpr PairSet kPairs[MAXQ - MINQ + 1] = {
    /*  8 */ {{{0, 3, 8481792}, {1, 5, 14687744}, {2, 6, 15112448}, {4, 7, 14733056}}, -1},
    /*  9 */ {{{0, 2, 16666880}, {1, 5, 14687744}, {4, 8, 14480128}, {6, 7, 14255872}}, 3},
    /* 10 */ {{{0, 3, 8481792}, {1, 5, 14687744}, {2, 6, 15112448}, {4, 9, 13784576}, {7, 8, 13659392}}, -1},
    /* 11 */ {{{0, 3, 8481792}, {1, 5, 14687744}, {2, 6, 15112448}, {4, 8, 14480128}, {7, 10, 14792704}}, 9},
    /* 12 */ {{{0, 9, 16690176}, {1, 5, 14687744}, {2, 4, 15112448}, {3, 10, 13879296}, {6, 7, 14255872}, {8, 11, 12721408}}, -1},
    /* 13 */ {{{0, 3, 8481792}, {1, 5, 14687744}, {2, 12, 16602112}, {4, 11, 13721344}, {6, 8, 14011136}, {7, 10, 14792704}}, 9},
    /* 14 */ {{{0, 9, 16690176}, {1, 5, 14687744}, {2, 12, 16602112}, {3, 13, 12786944}, {4, 8, 14480128}, {6, 11, 13276928}, {7, 10, 14792704}}, -1},
    /* 15 */ {{{0, 3, 8481792}, {1, 5, 14687744}, {2, 12, 16602112}, {4, 11, 13721344}, {6, 7, 14255872}, {8, 13, 11666176}, {10, 14, 14221824}}, 9},
    /* 16 */ {{{0, 9, 16690176}, {1, 5, 14687744}, {2, 12, 16602112}, {3, 15, 12401408}, {4, 7, 14733056}, {6, 8, 14011136}, {10, 14, 14221824}, {11, 13, 11054848}}, -1}};

// off with pp off = -bits(M) (mod 2^32); bits(M) is a multiple of 256, which covers an even pp.
constexpr uint32_t pair_offset(uint32_t pp, int M)
{
    const uint32_t bits = 0x4B000000u + (uint32_t)(M - (1 << 23));
    const bool even = pp % 2 == 0;
    const uint32_t odd = even ? pp / 256 : pp, target = 0u - (even ? bits / 256 : bits);
    uint32_t inv = odd;  // Newton's iteration for odd^-1 mod 2^32
    for (int i = 0; i < 5; ++i) inv *= 2u - odd * inv;
    return target * inv & (even ? 0xffffffu : 0xffffffffu);
}

// x = rint(v 2^sg) as xh 2^32 + xl; returns xh and xl + kRound.
__device__ __forceinline__ void split32(double v, double f1, double f2, double &xh, double &xr)
{
    const double x = __dmul_rn(__dmul_rn(v, f1), f2);
    xh = __dsub_rn(__fma_rn(x, 2.3283064365386963e-10, kRound), kRound);  // rint(x * 2^-32)
    xr = __dadd_rn(__fma_rn(-xh, 4294967296.0, x), kRound);
}

// Low bytes of w[0..7], w[0] in the lowest byte.
__device__ __forceinline__ uint2 pack8(const uint32_t (&w)[8])
{
    auto pack4 = [](uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
        return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
    };
    return make_uint2(pack4(w[0], w[1], w[2], w[3]), pack4(w[4], w[5], w[6], w[7]));
}

// All Q moduli's residue bytes of xh/xr[0..7], element j in byte j, given to put(l, bytes).
template <int Q, int I = 0, typename Put>
__device__ __forceinline__ void all_residues(const double (&xh)[8], const double (&xr)[8], const Put &put)
{
    constexpr PairSet set = kPairs[Q - MINQ];
    uint32_t w0[8], w1[8];
    if constexpr (I < Q / 2) {
        constexpr int a = set.pair[I].a, b = set.pair[I].b, M = set.pair[I].M;
        constexpr uint32_t p0 = modulus(a), p1 = modulus(b), pp = p0 * p1;
        constexpr double c = (double)((1ull << 32) % pp), ip = 1.0 / (double)pp;
        constexpr double magic = kRound + (double)pair_offset(pp, M) - (double)(long long)(kRound * ip + 0.5);
        constexpr float ip0 = 1.0f / (float)p0, ip1 = 1.0f / (float)p1;
        constexpr float c0 = (float)(kRoundF - (double)(long long)((double)M * (double)ip0 + 0.5));
        constexpr float c1 = (float)(kRoundF - (double)(long long)((double)M * (double)ip1 + 0.5));
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const double Y = __fma_rn(xh[j], c, xr[j]);
            const double t = __fma_rn(Y, ip, magic);
            const uint32_t u = (uint32_t)__double2loint(Y) + (uint32_t)__double2loint(t) * (0u - pp);
            w0[j] = u + __float_as_uint(__fmaf_rn(__uint_as_float(u), ip0, c0)) * (0u - p0);
            w1[j] = u + __float_as_uint(__fmaf_rn(__uint_as_float(u), ip1, c1)) * (0u - p1);
        }
        put(a, pack8(w0));
        put(b, pack8(w1));
        all_residues<Q, I + 1>(xh, xr, put);
    } else if constexpr (set.single >= 0) {
        constexpr uint32_t p0 = modulus(set.single);
        constexpr double c = (double)((1ull << 32) % p0), ip = 1.0 / (double)p0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const double Y = __fma_rn(xh[j], c, xr[j]);
            const double t = __fma_rn(__dsub_rn(Y, kRound), ip, kRound);  // rint(y / p): the residue is exact
            w0[j] = (uint32_t)__double2loint(Y) + (uint32_t)__double2loint(t) * (0u - p0);
        }
        put(set.single, pack8(w0));
    }
}

// Slab layout: byte (row r, k byte c) of K block kb of 256-row tile t of modulus l sits at
// l * mod_stride + (t * kblocks + kb) * 8192 + r * 32 + (c ^ (((r >> 2) & 1) << 4)) -- the
// 32-byte swizzled K-major image the MMA reads, so a stage is one contiguous bulk copy.
__device__ __forceinline__ size_t slab_offset(int tile, int kb, int kblocks, int r, int c)
{
    return ((size_t)tile * kblocks + kb) * (size_t)SLAB + (size_t)r * 32 + (c ^ (((r >> 2) & 1) << 4));
}

// Block: 64 rows of A x one 32-wide K block; warp w takes rows 8w..8w+7.  The rows are read whole
// (32 consecutive doubles per load, whatever A's pitch) into a warp-private tile of 8 x 256 bytes
// and handed on as lane -> row (lane / 4) and 8 consecutive k (lane % 4), so four lanes write the 32
// residue bytes of a row, one 8-byte store each per modulus.  The 16-byte pieces of each lane's
// 64 bytes are rotated so that the 16-byte reads are free of bank conflicts.
template <int Q>
__global__ void __launch_bounds__(256, 4) crt_split_a(const double *__restrict__ A, int m, int k, int lda, int kblocks,
                                                      const int *__restrict__ sg, uint8_t *__restrict__ ra,
                                                      size_t mod_stride)
{
    __shared__ __align__(16) double tile[8][8][32];
    pdl_wait();
    pdl_trigger();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int kb = blockIdx.y, row0 = blockIdx.x * 64 + warp * 8, r = lane >> 2, kq = lane & 3, row = row0 + r;
    {
        const int kk = kb * 32 + lane;
        const double *src = A + (size_t)row0 * lda + kk;
        double v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = (row0 + i < m && kk < k) ? __ldg(src + (size_t)i * lda) : 0.0;
        // 16-byte piece c = 4 q + j of row i goes to place 4 q + (j + q / 2 + 2 (i & 1)) % 4
        const int q = lane >> 3, j = (lane >> 1) & 3;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            tile[warp][i][(4 * q + ((j + (q >> 1) + 2 * (i & 1)) & 3)) * 2 + (lane & 1)] = v[i];
    }
    // the residues of a row that is not finite do not matter: its results are NaN
    int s = (row < m) ? sg[row] : 0;
    if (s == NONFINITE) s = 0;
    double f1, f2;
    scale_factors(s, f1, f2);
    __syncwarp();
    double xh[8], xr[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const double2 v = *reinterpret_cast<const double2 *>(&tile[warp][r][(4 * kq + ((j + (kq >> 1) + 2 * (r & 1)) & 3)) * 2]);
        split32(v.x, f1, f2, xh[2 * j], xr[2 * j]);
        split32(v.y, f1, f2, xh[2 * j + 1], xr[2 * j + 1]);
    }
    uint8_t *dst = ra + slab_offset(row / TILE, kb, kblocks, row % TILE, kq * 8);
    all_residues<Q>(xh, xr, [&](int l, uint2 b) { *reinterpret_cast<uint2 *>(dst + (size_t)l * mod_stride) = b; });
}

// Block: 64 consecutive columns of B x one 32-wide K block.  Warp w takes 32 of the columns
// (lane = column, so every load is one coalesced 256-byte row segment) and K quarter w % 4
// (8 consecutive k).  The 8 residue bytes of each (column, quarter) go to their swizzled place
// in a shared-memory copy of the block's slab rows; the 64 rows x 32 bytes of each modulus are
// one contiguous 2 KiB run of the slab (column j of B is row j % 256 of slab tile j / 256),
// written out with 16-byte stores.
template <int Q>
__global__ void __launch_bounds__(256, 4) crt_split_b(const double *__restrict__ B, int k, int n, int ldb, int kblocks,
                                                      const int *__restrict__ tu, uint8_t *__restrict__ rb,
                                                      size_t mod_stride)
{
    __shared__ __align__(16) unsigned char st[Q][64 * 32];
    pdl_wait();
    pdl_trigger();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kb = blockIdx.y, kq = warp & 3;
    const int rl = (warp >> 2) * 32 + lane;          // row of the block's 64
    const int col = blockIdx.x * 64 + rl;
    int s = (col < n) ? tu[col] : 0;
    if (s == NONFINITE) s = 0;   // as for A's rows
    const double *bcol = B + (col < n ? col : 0);
    double f1, f2;
    scale_factors(s, f1, f2);
    double xh[8], xr[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int kk = kb * 32 + kq * 8 + j;
        const double v = (col < n && kk < k) ? __ldg(bcol + (size_t)kk * ldb) : 0.0;
        split32(v, f1, f2, xh[j], xr[j]);
    }
    const int soff = rl * 32 + ((kq * 8) ^ (((rl >> 2) & 1) << 4));
    all_residues<Q>(xh, xr, [&](int l, uint2 b) { *reinterpret_cast<uint2 *>(&st[l][soff]) = b; });
    __syncthreads();
    const int c0 = blockIdx.x * 64;
    unsigned char *dst = rb + ((size_t)(c0 / TILE) * kblocks + kb) * (size_t)SLAB + (size_t)(c0 % TILE) * 32;
    for (int idx = threadIdx.x; idx < Q * 128; idx += 256) {
        const int l = idx >> 7, o = (idx & 127) * 16;
        *reinterpret_cast<uint4 *>(dst + (size_t)l * mod_stride + o) = *reinterpret_cast<const uint4 *>(&st[l][o]);
    }
}

// ---------------------------------------------------------------- tcgen05 helpers
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tc_commit(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tc_mma_i8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// K-major operand tile (rows 32 bytes apart) with the 32-byte swizzle: groups of 8 rows 256 B
// apart (SBO), LBO unused (1), descriptor version 1, layout type 6.
__device__ __forceinline__ uint64_t sw32_desc(uint32_t smem_addr)
{
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr >> 4) & 0x3FFF);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(256 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)6 << 61;
    return d;
}

// kind::i8 instruction descriptor: D s32, A s8, B s8, both K-major, M = 128, N = 256.
constexpr uint32_t IDESC_S8_128x256 = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(256 >> 3) << 17) |
                                      ((uint32_t)(128 >> 4) << 24);
// The same for a pair of CTAs, M = 256: 128 rows of each.
constexpr uint32_t IDESC_S8_256x256 = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(256 >> 3) << 17) |
                                      ((uint32_t)(256 >> 4) << 24);

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// g mod p in [0, p) for any int32 g: Barrett with M = ceil(2^32 / p) on |g| gives floor(|g|/p)
// or one more (the error of M is below 2^31 / 2^32), corrected by one add; then the sign.
// Checked exhaustively over all int32 for every modulus of the set.
__device__ __forceinline__ uint32_t mod_p(int32_t g, uint32_t p, uint32_t M)
{
    const uint32_t a = g < 0 ? 0u - (uint32_t)g : (uint32_t)g;
    const uint32_t qq = __umulhi(a, M);
    int32_t r = (int32_t)(a - qq * p);
    if (r < 0) r += (int32_t)p;
    return (g >= 0 || r == 0) ? (uint32_t)r : p - (uint32_t)r;
}

// g mod p, or that minus p, for an accumulator of K <= KMAX int8 x int8 products (|g| <= 2^14 K <
// 2^31 - 2^22): a = g + bias with bias = p floor(2^31 / p) lies in (0, 2^32) and a = g (mod p).
// Barrett with M = ceil(2^32 / p) gives q = floor(a / p) or one more.
__device__ __forceinline__ uint32_t mod_p_acc(uint32_t g, uint32_t p, uint32_t M, uint32_t bias)
{
    const uint32_t a = g + bias;
    return a - __umulhi(a, M) * p;
}

// Four residues in [0, p) in the bytes of a word; pp: p in both halves.  The last step, the unsigned min
// of r and r + p, fits 16 bits (r is in [-p, p), p <= 256), so one instruction takes two.  The epilogue's
// instructions bound how soon the second accumulator is free (3,400 cycles a half): against one value at a
// time, 8192 x 8192 x 1024 1.426 -> 1.404 ms, 1333 x 2011 x 1777 144.4 -> 142.8 us, 4096^3 1084 -> 1075.
__device__ __forceinline__ uint32_t mod_p_acc4(const uint32_t *g, uint32_t p, uint32_t pp, uint32_t M, uint32_t bias)
{
    uint32_t a = __byte_perm(mod_p_acc(g[0], p, M, bias), mod_p_acc(g[1], p, M, bias), 0x5410);
    uint32_t b = __byte_perm(mod_p_acc(g[2], p, M, bias), mod_p_acc(g[3], p, M, bias), 0x5410);
    a = __viaddmin_u16x2(a, pp, a);
    b = __viaddmin_u16x2(b, pp, b);
    return __byte_perm(a, b, 0x6420);
}

struct GemmParams {
    const uint8_t *ra, *rb;   // residue slabs [modulus][tile][K block][256 x 32 B], at the block's first tile
    uint8_t *rc;              // output residues [modulus][tile row][tile column][64 KiB], at the block's first tile
    size_t a_slabs, b_slabs, rc_mod;       // slabs of a modulus, bytes of its residue plane
    CUtensorMap ma, mb;                    // pairs: the slabs of A and B as {256 words, 8, slabs}
    int tiles_m, tiles_n;     // tiles of this block of the product
    int rc_tile_ld;           // tiles per row of the residue planes (the whole product's)
    int kblocks, q;
    int ksplit;               // K slices per (modulus, tile): 1, or the split-K form's count
    int kb_split;             // K blocks per slice
    size_t rc_slice;          // bytes between the residue planes of consecutive K slices
    int *status;
    unsigned int *sync;       // this launch's arrival counter (zeroed before the launch), or nullptr
    uint32_t barrett[MAXQ];
    uint32_t bias[MAXQ];      // p floor(2^31 / p), for mod_p_acc
};

// Shared memory of a CTA.  Alone: whole A and B slabs, 3 stages of 64 KiB.  As one of a pair: its own A
// slabs and half of the pair's B slabs, 4 stages of 48 KiB.
template <bool PAIR>
struct Ring {
    static constexpr int B_SLAB = PAIR ? SLAB / 2 : SLAB;
    static constexpr int STAGE_BYTES = KPACK * (SLAB + B_SLAB);
    static constexpr int STAGES = PAIR ? 4 : 3;
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
};

// Work item w: modulus w / (tiles), then groups of RASTER tile rows sweeping the columns
// together (the group's rows of A stay in L2 while each column tile of B is read once per group).
// tm: tile row, or pair of tile rows.
template <bool PAIR>
__device__ __forceinline__ void item_of(const GemmParams &p, int w, int &l, int &tm, int &tn, int &ks)
{
    constexpr int GROUP = PAIR ? RASTER / 2 : RASTER;
    ks = w % p.ksplit;       // K slice (consecutive items: the same tile's slices)
    w /= p.ksplit;
    const int rows = PAIR ? (p.tiles_m + 1) / 2 : p.tiles_m;
    const int per = rows * p.tiles_n;
    l = w / per;
    const int t = w - l * per;
    const int per_group = GROUP * p.tiles_n;
    const int g = t / per_group, r = t % per_group;
    const int first = g * GROUP;
    const int gsize = min(rows - first, GROUP);
    tm = first + r % gsize;
    tn = r / gsize;
}

// ---------------------------------------------------------------- CTA pairs
__device__ __forceinline__ void cluster_sync()
{
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Arrives on the barrier at `bar`'s offset in CTA `rank` of the cluster.
__device__ __forceinline__ void mbar_arrive_remote(uint64_t *bar, uint32_t rank)
{
    asm volatile(
        "{\n\t.reg .b32 a;\n\t"
        "mapa.shared::cluster.u32 a, %0, %1;\n\t"
        "mbarrier.arrive.shared::cluster.b64 _, [a];\n\t}" ::"r"(smem_u32(bar)),
        "r"(rank)
        : "memory");
}

// TMA box of this CTA, from this GPU's own memory into this CTA's shared memory, which completes on the
// barrier at `bar`'s offset in the first CTA of the pair (bit 24 of the address is the CTA's rank).
__device__ __forceinline__ void pair_load(void *dst, const CUtensorMap *map, int row, int slab, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 "
        "[%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(0), "r"(row), "r"(slab), "r"(smem_u32(bar) & 0xFEFFFFFFu)
        : "memory");
}

// Commit of the issuer's MMAs to a barrier (of both CTAs of a pair).
template <bool PAIR>
__device__ __forceinline__ void commit(uint64_t *bar)
{
    if (PAIR)
        asm volatile(
            "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                smem_u32(bar)),
            "h"((uint16_t)3)
            : "memory");
    else
        tc_commit(bar);
}

template <bool PAIR>
__device__ __forceinline__ void mma_i8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t accumulate)
{
    if (PAIR)
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
            "l"(adesc), "l"(bdesc), "r"(IDESC_S8_256x256), "r"(accumulate)
            : "memory");
    else
        tc_mma_i8(tmem_d, adesc, bdesc, IDESC_S8_128x256, accumulate);
}

// PAIR: two CTAs of a cluster work on two tile rows of one tile column.  Each copies its own A and half
// of the B slabs, and the first CTA issues tcgen05 cta_group::2 MMAs (M = 256) that read both CTAs'
// shared memory, so a CTA takes 12 KiB per K block from L2 instead of 16, reads half of B from its
// shared memory, and a fourth stage fits.  The copies are TMA boxes because only those can complete on
// the other CTA's barrier: the second CTA's bytes count on the first one's, and nothing relays them
// (a relaying warp costs 1.5% at 4096, 15% if it releases at cluster scope).  At the power limit the
// chip trades the saved energy for clock and utilisation -- residue products alone, 15 moduli, run
// back to back at 1 kW: 2927 -> 2997 TOP/s at N = 16384 (tensor pipe busy 89% -> 92%), 2713 -> 2814 at
// 4096, 2185 -> 2311 at 2048.
template <bool PAIR>
__global__ void __launch_bounds__(THREADS, 1) crt_gemm(const __grid_constant__ GemmParams p)
{
    using G = Ring<PAIR>;
    constexpr int STAGES = G::STAGES, STAGE_BYTES = G::STAGE_BYTES, B_SLAB = G::B_SLAB;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                                            ~uintptr_t(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + STAGES * STAGE_BYTES);
    uint64_t *empty = full + STAGES;
    uint64_t *acc_full = empty + STAGES;   // one per accumulator (tile rows 0-127, 128-255)
    uint64_t *acc_empty = acc_full + 2;
    uint64_t *drain = acc_empty + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drain + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int items = p.q * (PAIR ? (p.tiles_m + 1) / 2 : p.tiles_m) * p.tiles_n * p.ksplit;
    const int rank = PAIR ? (int)(blockIdx.x & 1) : 0;
    const int first = PAIR ? blockIdx.x >> 1 : blockIdx.x, step = PAIR ? gridDim.x >> 1 : gridDim.x;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int h = 0; h < 2; ++h) {
            mbar_init(&acc_full[h], 1);
            mbar_init(&acc_empty[h], PAIR ? 2 * EPI_WARPS : EPI_WARPS);
        }
        mbar_init(drain, 1);
        fence_barrier_init();
    }
    if (warp == 1) {
        if (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                         "r"(512)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                         "r"(512)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync();  // both CTAs' barriers and TMEM are set up
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();  // the set-up above overlaps the end of the previous kernel
    pdl_trigger();

    if (warp == 0) {
        // ------------------------------------------------------------ bulk-copy producer
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            int armed[STAGES];
            for (int s = 0; s < STAGES; ++s) armed[s] = -1;
            bool ok = true;
            for (int w = first; w < items && ok; w += step) {
                int l, tm, tn, ks;
                item_of<PAIR>(p, w, l, tm, tn, ks);
                const int kb_begin = ks * p.kb_split, kb_end = min(p.kblocks, kb_begin + p.kb_split);
                // Soft lockstep: CTAs that share an operand tile read it from L2 only while they
                // stay within a few microseconds of each other, so every producer waits at each
                // new item until all CTAs have started theirs -- or 20 us, then goes on anyway.
                // Nothing depends on it for correctness, so it cannot deadlock (two launches that
                // share the GPU just wait out the 20 us).
                if (p.sync) {
                    atomicAdd(p.sync, 1u);
                    const unsigned int target =
                        (unsigned int)(min((long long)(w / step + 1) * step, (long long)items) * (PAIR ? 2 : 1));
                    const unsigned long long t0 = global_ns();
                    while (*reinterpret_cast<volatile unsigned int *>(p.sync) < target &&
                           global_ns() - t0 < 20000ull)
                        __nanosleep(64);
                }
                // (the second half of an odd last pair loads the last tile row again and stores nothing)
                const int row = PAIR ? min(2 * tm + rank, p.tiles_m - 1) : tm;
                const size_t sa0 = (size_t)l * p.a_slabs + (size_t)row * p.kblocks;
                const size_t sb0 = (size_t)l * p.b_slabs + (size_t)tn * p.kblocks;
                for (int kb0 = kb_begin; kb0 < kb_end; kb0 += KPACK) {
                    if (!mbar_wait_bounded(&empty[stage], phase ^ 1u, p.status, kDevTimeoutEmpty)) {
                        ok = false;
                        break;
                    }
                    const int nkb = min(KPACK, kb_end - kb0);
                    unsigned char *sa = smem + stage * STAGE_BYTES, *sb = sa + KPACK * SLAB;
                    if (PAIR) {
                        // Whole boxes, also where the K range ends inside one.  Both CTAs' copies arrive on
                        // the first CTA's barrier, which expects the bytes of both.
                        if (rank == 0) {
                            mbar_arrive_expect_tx(&full[stage], 2u * STAGE_BYTES);
                            armed[stage] = (int)phase;
                        }
                        pair_load(sa, &p.ma, 0, (int)(sa0 + kb0), &full[stage]);
                        pair_load(sb, &p.mb, 4 * rank, (int)(sb0 + kb0), &full[stage]);
                    } else {
                        const uint32_t bytes = (uint32_t)(nkb * SLAB);
                        mbar_arrive_expect_tx(&full[stage], 2u * bytes);
                        armed[stage] = (int)phase;
                        bulk_load(sa, p.ra + (sa0 + kb0) * SLAB, bytes, &full[stage]);
                        bulk_load(sb, p.rb + (sb0 + kb0) * SLAB, bytes, &full[stage]);
                    }
                    if (++stage == STAGES) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
            }
            for (int s = 0; s < STAGES; ++s)
                if (armed[s] >= 0) mbar_wait_bounded(&full[s], (uint32_t)armed[s], p.status, kDevTimeoutFull);
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        // The epilogue releases accumulator 0 as soon as it has read it and accumulator 1 half a drain
        // later.  Until then the issuer runs ahead with accumulator 0's MMAs over the stages that are
        // in shared memory, then catches up with accumulator 1's.  From there on the two MMAs of a K block
        // follow each other: they share its B tile, and issuing a stage's four MMAs of one
        // accumulator before the other's costs power (16384^3: 54.3 ms against 51.7).  Against one
        // hand-over of both accumulators after the whole drain (5,000 idle of 33,800 cycles per item at
        // K = 3008): 8192 x 8192 x 1024 1.60 -> 1.49 ms, 4096^3 1.14 -> 1.12, 16384^3 51.2 -> 50.8.
        if (lane == 0 && rank == 0) {
            int stage = 0;
            uint32_t phase = 0, acc_phase = 0;
            bool ok = true;
            const uint32_t smem_base = smem_u32(smem);
            for (int w = first; w < items && ok; w += step) {
                const int kb_begin = (w % p.ksplit) * p.kb_split, kb_end = min(p.kblocks, kb_begin + p.kb_split);
                // MMAs over the stage at `st` that starts at K block kb, of accumulators h0 .. h1
                auto issue = [&](int st, int kb, bool lo, bool hi) {
                    const int nkb = min(KPACK, kb_end - kb);
                    const uint32_t sa = smem_base + st * STAGE_BYTES;
                    const uint64_t a0 = sw32_desc(sa), b0 = sw32_desc(sa + KPACK * SLAB);
#pragma unroll
                    for (int j = 0; j < KPACK; ++j) {
                        if (j < nkb) {
                            const uint32_t acc = (kb + j > kb_begin) ? 1u : 0u;
                            const uint64_t bj = b0 + (uint64_t)((j * B_SLAB) >> 4);
                            if (lo) mma_i8<PAIR>(tmem_base, a0 + (uint64_t)((j * SLAB) >> 4), bj, acc);
                            if (hi) mma_i8<PAIR>(tmem_base + 256, a0 + (uint64_t)((j * SLAB + SLAB / 2) >> 4), bj, acc);
                        }
                    }
                };
                auto next = [&](int &st, uint32_t &ph) {
                    if (++st == STAGES) {
                        st = 0;
                        ph ^= 1u;
                    }
                };
                auto wait_stage = [&](int st, uint32_t ph) {
                    const bool got = mbar_wait_bounded(&full[st], ph, p.status, kDevTimeoutFull);
                    tc_fence_after();
                    return got;
                };
                if (!mbar_wait_bounded(&acc_empty[0], acc_phase ^ 1u, p.status, kDevTimeoutAcc)) break;
                tc_fence_after();
                int kb0 = kb_begin, ahead = 0, st = stage;
                uint32_t ph = phase;
                while (ok && ahead < STAGES && kb0 < kb_end &&
                       !mbar_try_wait(&acc_empty[1], acc_phase ^ 1u)) {
                    ok = wait_stage(st, ph);
                    if (!ok) break;
                    issue(st, kb0, true, false);
                    kb0 += KPACK;
                    ++ahead;
                    next(st, ph);
                }
                if (ok) ok = mbar_wait_bounded(&acc_empty[1], acc_phase ^ 1u, p.status, kDevTimeoutAcc);
                if (!ok) break;
                acc_phase ^= 1u;
                tc_fence_after();
                for (int i = 0; i < ahead; ++i) {
                    issue(stage, kb_begin + i * KPACK, false, true);
                    commit<PAIR>(&empty[stage]);  // frees the stage once these MMAs have read it
                    next(stage, phase);
                }
                for (; kb0 < kb_end; kb0 += KPACK) {
                    ok = wait_stage(stage, phase);
                    if (!ok) break;
                    if (kb0 + KPACK < kb_end) {
                        issue(stage, kb0, true, true);
                    } else {  // accumulator 0 is done first, and drains while the other's MMAs run
                        issue(stage, kb0, true, false);
                        commit<PAIR>(&acc_full[0]);
                        issue(stage, kb0, false, true);
                    }
                    commit<PAIR>(&empty[stage]);
                    next(stage, phase);
                }
                if (ok) {
                    if (kb_begin + ahead * KPACK >= kb_end) commit<PAIR>(&acc_full[0]);  // all of it ran ahead
                    commit<PAIR>(&acc_full[1]);
                }
            }
            // Drain: all MMAs this thread issued have finished before TMEM is released.
            commit<PAIR>(drain);
            mbar_wait_bounded(drain, 0, p.status, kDevTimeoutAcc);
        }
    } else {
        // ------------------------------------------------------------ epilogue (warps 2..)
        const int qd = warp & 3;         // TMEM lane quarter this warp may access
        const int c0 = (warp - 2) >> 2 << 1;  // first of its two 32-column chunks
        uint32_t acc_phase = 0;
        bool ok = true;
        for (int w = first; w < items && ok; w += step) {
            int l, tm, tn, ks;
            item_of<PAIR>(p, w, l, tm, tn, ks);
            const int row = PAIR ? 2 * tm + rank : tm;
            const uint32_t pm = (uint32_t)c_moduli[l], M = p.barrett[l], bias = p.bias[l], pm2 = pm * 0x10001u;
            uint8_t *dst = p.rc + (size_t)ks * p.rc_slice + (size_t)l * p.rc_mod +
                           ((size_t)row * p.rc_tile_ld + tn) * OUT_TILE_BYTES + (size_t)(qd * 32) * 256 + lane * 8;
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
                bool got = true;
                if (lane == 0) got = mbar_wait_sleepy(&acc_full[h], acc_phase, p.status, kDevTimeoutAcc);
                got = __shfl_sync(0xffffffffu, got ? 1 : 0, 0) != 0;
                if (!got) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t tbase = tmem_base + ((uint32_t)(32 * qd) << 16) + h * 256;
                uint32_t r[2][32];
                tmem_ld32(tbase + c0 * 32, r[0]);
                tmem_ld32(tbase + (c0 + 1) * 32, r[1]);
                tmem_wait_ld();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if (PAIR && rank == 1)
                        mbar_arrive_remote(&acc_empty[h], 0);
                    else
                        mbar_arrive(&acc_empty[h]);
                }
                if (PAIR && row >= p.tiles_m) continue;
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    uint32_t pk[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) pk[j] = mod_p_acc4(&r[b][4 * j], pm, pm2, M, bias);
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        *reinterpret_cast<uint2 *>(dst + (size_t)h * (128 * 256) + (size_t)(4 * (c0 + b) + u) * 256) =
                            make_uint2(pk[2 * u], pk[2 * u + 1]);
                }
            }
            acc_phase ^= 1u;
        }
    }

    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    __syncwarp();
    if (PAIR) cluster_sync();  // neither CTA leaves while the other may still reach its memory
    if (warp == 1) {
        if (PAIR)
            asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
        else
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
    }
}

// ---------------------------------------------------------------- CRT recombination
// Product residues of one 256 x 256 tile are stored [h][quarter][8-column chunk][lane][8 B]: the
// epilogue warp of TMEM lane quarter `quarter` and accumulator h writes 256 contiguous bytes per
// chunk.  One warp here takes one (tile, h, quarter, chunk): lane = row within the quarter,
// 8 columns.  Where C's rows are 32-byte aligned a lane stores its own 64 bytes, two whole sectors.
// Elsewhere these would be partial sectors, so the block's 8 warps, which hold 64 consecutive columns
// of the same 32 rows, pass through shared memory and write 512-byte row pieces (2501 x 1999: 41 us
// by 8-byte stores, 33 staged; 2496 x 2000: 33 staged, 29 by 32-byte stores).
// beta_one: C (+)= result.
//
// Bound by the FP64 pipe, three multiply-adds per residue.  A residue byte R becomes an FP64 operand
// by one byte permute: as byte 1 of the high word it is the subnormal R 2^-1034, and the weights
// carry 2^974, so the sums come out as s 2^-60, exact as before (no bit is lost: they are multiples
// of 2^-60 below 2^-8).  P's chunks and the exponents carry the same 2^60, which no rounding sees.
// Before, an add turned 2^52 + R into R, every scale factor was built and range-checked per element,
// and rint was a conversion: 152 instructions per output, 39-41 us there and 424 us at 8192 x 8192 (347
// now: 1.54 GB of residues and C, 4.4 TB/s).
constexpr int kCombineShift = 60;
constexpr int COMBINE_LD = 66;  // doubles of a staged row: 16-byte stores of 8 lanes hit every bank once

struct CombineParams {
    const uint8_t *rc;        // the block's first tile of the residue planes
    size_t rc_mod;
    int ksplit;               // K slices whose residues are added mod p first (1: none)
    size_t rc_slice;          // bytes between the residue planes of consecutive K slices
    double *C;                // the block's first element of C
    int m, n, ldc, tiles_n, rc_tile_ld, beta_one, vec_store;
    const int *sg, *tu;
    Consts K;
};

// SPLITK: the residue planes of p.ksplit K slices are added modulo p first (a separate
// instantiation with a larger register budget, so the whole-K kernel keeps its own).
template <int Q, bool SPLITK>
__global__ void __launch_bounds__(256, SPLITK ? 2 : 3) crt_combine(const __grid_constant__ CombineParams p)
{
    const int lane = threadIdx.x & 31;
    __shared__ __align__(16) double out[32][COMBINE_LD];
    pdl_wait();
    pdl_trigger();
    const int warp = threadIdx.x >> 5;
    const long long unit = (long long)blockIdx.x * 8 + warp;
    const int c = (int)(unit & 31), qd = (int)((unit >> 5) & 3), h = (int)((unit >> 7) & 1);
    const long long tile = unit >> 8;
    const int tm = (int)(tile / p.tiles_n), tn = (int)(tile % p.tiles_n);
    const int row0 = tm * TILE + h * 128 + qd * 32, row = row0 + lane;
    const int col0 = tn * TILE + c * 8;
    if (row0 >= p.m || tn * TILE + (c & ~7) * 8 >= p.n) return;  // the whole block is outside
    const uint8_t *src = p.rc + ((size_t)tm * p.rc_tile_ld + tn) * OUT_TILE_BYTES +
                         (size_t)((h * 4 + qd) * 32 + c) * 256 + lane * 8;
    uint2 res[Q];
#pragma unroll
    for (int l = 0; l < Q; ++l) res[l] = __ldg(reinterpret_cast<const uint2 *>(src + (size_t)l * p.rc_mod));
    const int srow = row < p.m ? p.sg[row] : 0;
    int e[8];  // the outputs' exponents
    bool plain = srow != NONFINITE;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int scol = p.tu[min(col0 + j, p.n - 1)];
        plain = plain && scol != NONFINITE;
        e[j] = p.K.E3 - srow - scol;
    }
    if (SPLITK) {
        // the slices' residues (each < p) add modulo p
#pragma unroll
        for (int l = 0; l < Q; ++l) {
            uint32_t r[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) r[j] = ((j < 4 ? res[l].x : res[l].y) >> (8 * (j & 3))) & 255u;
            for (int t = 1; t < p.ksplit; ++t) {
                const uint2 u = __ldg(reinterpret_cast<const uint2 *>(src + (size_t)t * p.rc_slice + (size_t)l * p.rc_mod));
#pragma unroll
                for (int j = 0; j < 8; ++j) r[j] += ((j < 4 ? u.x : u.y) >> (8 * (j & 3))) & 255u;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) r[j] = mod_p((int32_t)r[j], (uint32_t)c_moduli[l], p.K.barrett[l]);
            res[l] = make_uint2(r[0] | r[1] << 8 | r[2] << 16 | r[3] << 24, r[4] | r[5] << 8 | r[6] << 16 | r[7] << 24);
        }
    }
    // plain: every scale is finite and every exponent within one normal factor (as a rule)
#pragma unroll
    for (int j = 0; j < 8; ++j) plain = plain && e[j] >= -1022 && e[j] <= 1023;
    plain = __all_sync(0xffffffffu, plain);
#pragma unroll
    for (int j0 = 0; j0 < 8; j0 += 4) {
        double s1[4], s2[4], s3[4], v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) s1[j] = s2[j] = s3[j] = 0.0;
#pragma unroll
        for (int l = 0; l < Q; ++l) {
            const uint32_t word = j0 == 0 ? res[l].x : res[l].y;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const double r = __hiloint2double((int)__byte_perm(word, 0u, 0x4404 | (j << 4)), 0);  // R 2^-1034
                s1[j] = __fma_rn(p.K.w[l][0], r, s1[j]);
                s2[j] = __fma_rn(p.K.w[l][1], r, s2[j]);
                s3[j] = __fma_rn(p.K.w[l][2], r, s3[j]);
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const double q = __dmul_rn(__fma_rn(s2[j], 0x1p-40, s1[j]), p.K.inv_phat);
            const double Qd = __dsub_rn(__dadd_rn(q, kRound), kRound);  // rint(q), |q| < 2^12
            const double d1 = __fma_rn(-Qd, p.K.pc[0], s1[j]);
            const double d2 = __fma_rn(-Qd, p.K.pc[1], s2[j]);
            const double d3 = __fma_rn(-Qd, p.K.pc[2], s3[j]);
            const double cc = __fma_rn(__fma_rn(d1, 0x1p40, d2), 0x1p40, d3);
            if (plain) {
                v[j] = __dmul_rn(cc, __hiloint2double((e[j0 + j] + 1023) << 20, 0));
            } else {
                const int scol = p.tu[min(col0 + j0 + j, p.n - 1)];
                v[j] = (srow == NONFINITE || scol == NONFINITE) ? __longlong_as_double(0x7ff8000000000000ll)
                                                                : scale2(cc, e[j0 + j]);
            }
        }
        if (p.vec_store == 4) {
            const int col = col0 + j0;
            double *dst = p.C + (size_t)row * p.ldc + col;
            if (row >= p.m) continue;
            if (col + 3 < p.n) {
                if (p.beta_one) {
                    double o[4];
                    asm volatile("ld.global.v4.f64 {%0,%1,%2,%3}, [%4];"
                                 : "=d"(o[0]), "=d"(o[1]), "=d"(o[2]), "=d"(o[3])
                                 : "l"(dst));
#pragma unroll
                    for (int u = 0; u < 4; ++u) v[u] = __dadd_rn(o[u], v[u]);
                }
                asm volatile("st.global.v4.f64 [%0], {%1,%2,%3,%4};" ::"l"(dst), "d"(v[0]), "d"(v[1]), "d"(v[2]),
                             "d"(v[3])
                             : "memory");
            } else {
#pragma unroll
                for (int u = 0; u < 3; ++u)
                    if (col + u < p.n) dst[u] = p.beta_one ? __dadd_rn(dst[u], v[u]) : v[u];
            }
            continue;
        }
        double2 *o = reinterpret_cast<double2 *>(&out[lane][warp * 8 + j0]);
        o[0] = make_double2(v[0], v[1]);
        o[1] = make_double2(v[2], v[3]);
    }
    if (p.vec_store == 4) return;
    __syncthreads();
    // warp w writes rows 4 w ..: 64 columns each
    const int cbase = tn * TILE + (c & ~7) * 8;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = warp * 4 + i;
        if (row0 + r >= p.m) break;
        double *crow = p.C + (size_t)(row0 + r) * p.ldc + cbase;
        if (p.vec_store) {
            const int cc = 2 * lane;
            const double2 v = *reinterpret_cast<const double2 *>(&out[r][cc]);
            if (cbase + cc + 1 < p.n) {
                double2 *dst = reinterpret_cast<double2 *>(crow + cc);
                const double2 o = p.beta_one ? *dst : make_double2(0.0, 0.0);
                *dst = p.beta_one ? make_double2(__dadd_rn(o.x, v.x), __dadd_rn(o.y, v.y)) : v;
            } else if (cbase + cc < p.n) {
                crow[cc] = p.beta_one ? __dadd_rn(crow[cc], v.x) : v.x;
            }
        } else {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int cc = lane + 32 * u;
                if (cbase + cc < p.n) crow[cc] = p.beta_one ? __dadd_rn(crow[cc], out[r][cc]) : out[r][cc];
            }
        }
    }
}

// ---------------------------------------------------------------- host constants
static void chunks40(unsigned __int128 v, int L, double out[3])
{
    for (int t = 0; t < 3; ++t) {
        const int e = L - 40 * (t + 1);
        unsigned __int128 c;
        if (e >= 0) {
            c = v >> e;
            v -= c << e;
        } else {
            c = v << (-e);
            v = 0;
        }
        out[t] = (double)(uint64_t)c;
    }
}

static bool make_consts(int q, Consts &K)
{
    if (q < MINQ || q > MAXQ) return false;
    memset(&K, 0, sizeof K);
    unsigned __int128 P = 1;
    for (int l = 0; l < q; ++l) P *= (unsigned)h_moduli[l];
    int L = 0;
    for (unsigned __int128 t = P; t; t >>= 1) ++L;
    K.q = q;
    K.L = L;
    K.alpha = (L - 3) / 2;
    K.beta = L - 3 - K.alpha;
    K.E3 = L - 120 + kCombineShift;
    for (int l = 0; l < q; ++l) {
        const unsigned p = (unsigned)h_moduli[l];
        const unsigned __int128 M = P / p;
        const unsigned mm = (unsigned)(M % p);
        unsigned inv = 1;
        while ((mm * inv) % p != 1) ++inv;
        chunks40(M * inv, L, K.w[l]);
        for (double &c : K.w[l]) c = ldexp(c, 1034 - kCombineShift);
        K.barrett[l] = (uint32_t)(0xffffffffull / p + 1);
    }
    chunks40(P, L, K.pc);
    K.inv_phat = ldexp(1.0 / fma(K.pc[1], 0x1p-40, K.pc[0]), kCombineShift);
    for (double &c : K.pc) c = ldexp(c, -kCombineShift);
    return true;
}

}  // namespace crt
}  // namespace mgx

using namespace mgx;

namespace {

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

struct CrtLayout {
    size_t ra, rb, rc, sg, tu, colmax, colsum, sync, arrived, total;
    size_t ra_mod, rb_mod, rc_mod;
    int kblocks, tiles_m, tiles_n;
    int ksplit, kb_split;   // K slices (1: whole K) and K blocks per slice
};

// Workspace of one K range of at most KMAX: residue slabs of A and B^T (rows rounded up to 256,
// K to 32), the residue planes of the product, the scale exponents and the column sums.
// With ksplit > 1 (the split-K form, k <= KMAX) the 32-wide K blocks are cut into slices of
// ceil(kblocks / ksplit) blocks, and the product residues get one set of planes per slice.
CrtLayout crt_layout(int m, int n, int k, int q, int ksplit = 1)
{
    CrtLayout L;
    int kc = k < crt::KMAX ? k : crt::KMAX;
    L.kblocks = (kc + 31) / 32;
    if (L.kblocks == 0) L.kblocks = 1;
    if (ksplit < 1) ksplit = 1;
    if (ksplit > L.kblocks) ksplit = L.kblocks;
    L.kb_split = (L.kblocks + ksplit - 1) / ksplit;
    L.ksplit = (L.kblocks + L.kb_split - 1) / L.kb_split;
    L.tiles_m = (m + crt::TILE - 1) / crt::TILE;
    L.tiles_n = (n + crt::TILE - 1) / crt::TILE;
    L.ra_mod = (size_t)L.tiles_m * L.kblocks * crt::SLAB;
    L.rb_mod = (size_t)L.tiles_n * L.kblocks * crt::SLAB;
    L.rc_mod = (size_t)L.tiles_m * L.tiles_n * crt::OUT_TILE_BYTES;
    size_t off = 0;
    L.ra = off;
    off = align256(off + (size_t)q * L.ra_mod);
    L.rb = off;
    off = align256(off + (size_t)q * L.rb_mod);
    L.rc = off;
    off = align256(off + (size_t)q * L.rc_mod * L.ksplit);
    L.sg = off;
    off = align256(off + sizeof(int) * (size_t)m);
    L.tu = off;
    off = align256(off + sizeof(int) * (size_t)n);
    L.colmax = off;
    off = align256(off + sizeof(unsigned long long) * (size_t)n);
    L.colsum = off;
    off = align256(off + sizeof(unsigned long long) * (size_t)n);
    L.sync = off;                       // arrival counters of the products launches (two slots)
    off = align256(off + 2 * sizeof(unsigned int));
    L.arrived = off;                    // per column group: blocks that are done with its sums
    off = align256(off + sizeof(unsigned int) * (size_t)((n + 255) / 256));
    L.total = off;
    return L;
}

template <template <int> class F, typename... Args>
int dispatch_q(int q, Args... args)
{
    switch (q) {
    case 8: return F<8>::run(args...);
    case 9: return F<9>::run(args...);
    case 10: return F<10>::run(args...);
    case 11: return F<11>::run(args...);
    case 12: return F<12>::run(args...);
    case 13: return F<13>::run(args...);
    case 14: return F<14>::run(args...);
    case 15: return F<15>::run(args...);
    case 16: return F<16>::run(args...);
    default:
        mgx_set_last_message("mgx_gemm_ozaki_crt: %d moduli is outside 8..16", q);
        return MGX_E_INVALID;
    }
}

template <int Q>
struct SplitA {
    static int run(const double *A, int m, int k, int lda, const CrtLayout &L, const int *sg, uint8_t *ra,
                   cudaStream_t stream)
    {
        const int tiles = (m + crt::TILE - 1) / crt::TILE;
        MGX_HOST_CHECK(mgx_launch_dependent(crt::crt_split_a<Q>, dim3(tiles * 4, L.kblocks), 256, 0, stream, A, m, k, lda,
                                            L.kblocks, sg, ra, L.ra_mod));
        return MGX_SUCCESS;
    }
};

template <int Q>
struct SplitB {
    static int run(const double *B, int n, int k, int ldb, const CrtLayout &L, const int *tu, uint8_t *rb,
                   cudaStream_t stream)
    {
        const int tiles = (n + crt::TILE - 1) / crt::TILE;
        MGX_HOST_CHECK(mgx_launch_dependent(crt::crt_split_b<Q>, dim3(tiles * 4, L.kblocks), 256, 0, stream, B, k, n, ldb,
                                            L.kblocks, tu, rb, L.rb_mod));
        return MGX_SUCCESS;
    }
};

template <int Q>
struct Combine {
    static int run(const crt::CombineParams &cp, long long blocks, cudaStream_t stream)
    {
        MGX_HOST_CHECK(mgx_launch_dependent(cp.ksplit > 1 ? crt::crt_combine<Q, true> : crt::crt_combine<Q, false>,
                                            dim3((unsigned)blocks), 256, 0, stream, cp));
        return MGX_SUCCESS;
    }
};

crt::ColStats col_stats(unsigned char *ws, const CrtLayout &L, int c0, int n)
{
    crt::ColStats z;
    z.max = reinterpret_cast<unsigned long long *>(ws + L.colmax) + c0;
    z.sum = reinterpret_cast<unsigned long long *>(ws + L.colsum) + c0;
    z.arrived = reinterpret_cast<unsigned int *>(ws + L.arrived) + c0 / 256;
    z.n = n;
    return z;
}

// Scale exponents and residues of rows [r0, r0 + m) of A (m x k, k <= KMAX; r0 a multiple of
// 256) into the whole-problem workspace.  `zero`: column statistics for the row pass to clear.
int crt_split_a_impl(const double *A, int m, int k, int lda, int r0, const crt::Consts &K, unsigned char *ws,
                     const CrtLayout &L, cudaStream_t stream, const crt::ColStats &zero = crt::ColStats{})
{
    if (m <= 0) return MGX_SUCCESS;
    int *status = mgx_device_status_ptr();
    int *sg = reinterpret_cast<int *>(ws + L.sg) + r0;
    uint8_t *ra = ws + L.ra + (size_t)(r0 / crt::TILE) * L.kblocks * crt::SLAB;
    // the fewest threads that hold a row in 16 registers each
    auto scale = [&](auto kernel, int threads) {
        return mgx_launch_dependent(kernel, dim3((unsigned)m), dim3(threads), 0, stream, A, m, k, lda, K.alpha, sg, zero,
                                    status);
    };
    MGX_HOST_CHECK(k <= 1024   ? scale(crt::crt_row_scale<64, 16>, 64)
                   : k <= 2048 ? scale(crt::crt_row_scale<128, 16>, 128)
                   : k <= 4096 ? scale(crt::crt_row_scale<256, 16>, 256)
                   : k <= 8192 ? scale(crt::crt_row_scale<512, 16>, 512)
                               : scale(crt::crt_row_scale<512, 0>, 512));
    return dispatch_q<SplitA>(K.q, A, m, k, lda, L, (const int *)sg, ra, stream);
}

// The same for columns [c0, c0 + n) of B (k x n).  `zeroed`: their statistics are clear.
int crt_split_b_impl(const double *B, int n, int k, int ldb, int c0, const crt::Consts &K, unsigned char *ws,
                     const CrtLayout &L, cudaStream_t stream, bool zeroed = false)
{
    if (n <= 0) return MGX_SUCCESS;
    int *status = mgx_device_status_ptr();
    int *tu = reinterpret_cast<int *>(ws + L.tu) + c0;
    const crt::ColStats z = col_stats(ws, L, c0, n);
    uint8_t *rb = ws + L.rb + (size_t)(c0 / crt::TILE) * L.kblocks * crt::SLAB;
    const int groups = (n + 255) / 256;
    if (!zeroed)
        MGX_HOST_CHECK(mgx_launch_dependent(crt::crt_zero, dim3((unsigned)(groups < 64 ? groups : 64)), 256, 0, stream, z));
    const int sms = mgx_sm_count();
    int ych = (sms * 8) / groups;
    if (ych > (k + 63) / 64) ych = (k + 63) / 64;
    if (ych < 1) ych = 1;
    const dim3 grid((unsigned)groups, (unsigned)ych);
    MGX_HOST_CHECK(mgx_launch_dependent(crt::crt_col_max, grid, 256, 0, stream, B, k, n, ldb, z.max));
    MGX_HOST_CHECK(mgx_launch_dependent(crt::crt_col_sumsq, grid, 256, 0, stream, B, k, n, ldb, z, K.beta, tu, status));
    return dispatch_q<SplitB>(K.q, B, n, k, ldb, L, (const int *)tu, rb, stream);
}

int crt_split_impl(const double *A, const double *B, int m, int n, int k, int lda, int ldb, const crt::Consts &K,
                   unsigned char *ws, const CrtLayout &L, cudaStream_t stream)
{
    int rc = crt_split_a_impl(A, m, k, lda, 0, K, ws, L, stream, col_stats(ws, L, 0, n));
    if (rc == MGX_SUCCESS) rc = crt_split_b_impl(B, n, k, ldb, 0, K, ws, L, stream, true);
    return rc;
}

// A block of the product inside a whole-problem workspace: rows [r0, r0 + m) and columns
// [c0, c0 + n), r0 and c0 multiples of 256.
struct CrtView {
    const uint8_t *ra, *rb;
    size_t a_slab0, b_slab0;  // slabs before ra, rb in the workspace
    uint8_t *rc;
    const int *sg, *tu;
    int m, n, tiles_m, tiles_n;
};

CrtView crt_view(const CrtLayout &L, unsigned char *ws, int r0, int c0, int m, int n)
{
    CrtView v;
    const int tm0 = r0 / crt::TILE, tn0 = c0 / crt::TILE;
    v.ra = ws + L.ra + (size_t)tm0 * L.kblocks * crt::SLAB;
    v.rb = ws + L.rb + (size_t)tn0 * L.kblocks * crt::SLAB;
    v.a_slab0 = (size_t)tm0 * L.kblocks;
    v.b_slab0 = (size_t)tn0 * L.kblocks;
    v.rc = ws + L.rc + ((size_t)tm0 * L.tiles_n + tn0) * crt::OUT_TILE_BYTES;
    v.sg = reinterpret_cast<const int *>(ws + L.sg) + r0;
    v.tu = reinterpret_cast<const int *>(ws + L.tu) + c0;
    v.m = m;
    v.n = n;
    v.tiles_m = (m + crt::TILE - 1) / crt::TILE;
    v.tiles_n = (n + crt::TILE - 1) / crt::TILE;
    return v;
}

// Pairs of CTAs that the current context's SMs hold at once: one per two SMs on a whole B200, fewer where a
// partition has SMs without a partner.  More clusters than that would start only when others have ended, and
// every item of those would wait out the lockstep's limit for them.  Asked once per context (its id is
// never used again); without an id, each time.  0 (CTAs alone) where it cannot be told.
int crt_pair_slots()
{
    struct Known {
        unsigned long long ctx;
        int clusters;
    };
    static std::mutex mu;
    static Known known[64];
    static int count = 0;
    const unsigned long long ctx = mgx_context_id();
    if (ctx != 0) {
        std::lock_guard<std::mutex> lk(mu);
        for (int i = 0; i < count; ++i)
            if (known[i].ctx == ctx) return known[i].clusters;
    }
    constexpr int smem = crt::Ring<true>::SMEM_BYTES;
    const int most = mgx_sm_count() / 2;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2u * (unsigned)(most > 0 ? most : 1));
    cfg.blockDim = dim3(crt::THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int active = 0;
    if (cudaFuncSetAttribute(crt::crt_gemm<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&active, crt::crt_gemm<true>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    if (ctx != 0) {
        std::lock_guard<std::mutex> lk(mu);
        if (count < 64) known[count++] = Known{ctx, active};
    }
    return active;
}

// Residue products of a block on the tensor cores (one persistent launch).
int crt_products_impl(const crt::Consts &K, const CrtLayout &L, const CrtView &v, cudaStream_t stream,
                      unsigned int *sync = nullptr)
{
    crt::GemmParams p;
    memset(&p, 0, sizeof p);
    p.ra = v.ra;
    p.rb = v.rb;
    p.rc = v.rc;
    p.a_slabs = L.ra_mod / crt::SLAB;
    p.b_slabs = L.rb_mod / crt::SLAB;
    p.rc_mod = L.rc_mod;
    p.tiles_m = v.tiles_m;
    p.tiles_n = v.tiles_n;
    p.rc_tile_ld = L.tiles_n;
    p.kblocks = L.kblocks;
    p.q = K.q;
    p.ksplit = L.ksplit;
    p.kb_split = L.kb_split;
    p.rc_slice = (size_t)K.q * L.rc_mod;
    p.status = mgx_device_status_ptr();
    for (int l = 0; l < crt::MAXQ; ++l) {
        p.barrett[l] = K.barrett[l];
        p.bias[l] = (uint32_t)crt::h_moduli[l] * (0x80000000u / (uint32_t)crt::h_moduli[l]);
    }
    const long long items = (long long)K.q * v.tiles_m * v.tiles_n * L.ksplit;
    if (items <= 0) return MGX_SUCCESS;
    if (items > 0x7fffffffll) {
        mgx_set_last_message("mgx_gemm_ozaki_crt: product too large (%lld work items)", items);
        return MGX_E_UNSUPPORTED;
    }
    const int sms = mgx_sm_count();
    const int grid = (long long)sms < items ? sms : (int)items;
    // The lockstep pays over many items (8192 x 8192 x 1024, 104 per CTA: 1.57 ms with it, 1.60 without;
    // 3000 x 3000 x 16384, 15: 2.46, 2.59).  Over few, its counter's memset, which also keeps the products
    // from being a dependent launch, costs more: 1024^3, 2 per CTA: 68 us with it, 63 without; 2501 x
    // 1999 x 3001, 8: 344, 340.
    if (sync && items >= 10ll * grid) {
        MGX_HOST_CHECK(cudaMemsetAsync(sync, 0, sizeof(unsigned int), stream));
        p.sync = sync;
    }
    const long long pairs = (long long)K.q * ((v.tiles_m + 1) / 2) * v.tiles_n * L.ksplit;
    int slots = crt::pairs_to_launch(items, pairs, sms, sms / 2);
    if (slots > 0) slots = crt::pairs_to_launch(items, pairs, sms, crt_pair_slots());
    if (slots > 0) {
        int rc = mgx_encode_tmap_3d(&p.ma, CU_TENSOR_MAP_DATA_TYPE_INT32, 4, v.ra, 256, 8, K.q * p.a_slabs - v.a_slab0,
                                    1024, crt::SLAB, 256, 8, crt::KPACK, CU_TENSOR_MAP_SWIZZLE_NONE);
        if (rc == MGX_SUCCESS)
            rc = mgx_encode_tmap_3d(&p.mb, CU_TENSOR_MAP_DATA_TYPE_INT32, 4, v.rb, 256, 8,
                                    K.q * p.b_slabs - v.b_slab0, 1024, crt::SLAB, 256, 4, crt::KPACK,
                                    CU_TENSOR_MAP_SWIZZLE_NONE);
        if (rc != MGX_SUCCESS) return rc;
        constexpr int smem = crt::Ring<true>::SMEM_BYTES;
        MGX_HOST_CHECK(cudaFuncSetAttribute(crt::crt_gemm<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        MGX_HOST_CHECK(mgx_launch_dependent_cluster(crt::crt_gemm<true>, dim3(2u * (unsigned)slots), crt::THREADS, smem,
                                                    stream, 2, p));
        return MGX_SUCCESS;
    }
    constexpr int smem = crt::Ring<false>::SMEM_BYTES;
    MGX_HOST_CHECK(cudaFuncSetAttribute(crt::crt_gemm<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    MGX_HOST_CHECK(mgx_launch_dependent(crt::crt_gemm<false>, dim3((unsigned)grid), crt::THREADS, smem, stream, p));
    return MGX_SUCCESS;
}

// CRT recombination of a block into C (the block's first element; leading dimension ldc).
int crt_combine_impl(double *C, int ldc, int beta_one, const crt::Consts &K, const CrtLayout &L, const CrtView &v,
                     cudaStream_t stream)
{
    crt::CombineParams cp;
    memset(&cp, 0, sizeof cp);
    cp.rc = v.rc;
    cp.rc_mod = L.rc_mod;
    cp.ksplit = L.ksplit;
    cp.rc_slice = (size_t)K.q * L.rc_mod;
    cp.C = C;
    cp.m = v.m;
    cp.n = v.n;
    cp.ldc = ldc;
    cp.tiles_n = v.tiles_n;
    cp.rc_tile_ld = L.tiles_n;
    cp.beta_one = beta_one;
    // doubles that C's rows are aligned to: 4, 2 or (0) one
    cp.vec_store = (ldc % 4 == 0 && (reinterpret_cast<uintptr_t>(C) & 31) == 0)   ? 4
                   : (ldc % 2 == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0) ? 2
                                                                                  : 0;
    cp.sg = v.sg;
    cp.tu = v.tu;
    cp.K = K;
    const long long blocks = (long long)v.tiles_m * v.tiles_n * 32;
    if (blocks <= 0) return MGX_SUCCESS;
    return dispatch_q<Combine>(K.q, cp, blocks, stream);
}

int crt_multiply_impl(double *C, int m, int n, int ldc, int beta_one, const crt::Consts &K, unsigned char *ws,
                      const CrtLayout &L, cudaStream_t stream)
{
    const CrtView v = crt_view(L, ws, 0, 0, m, n);
    int rc = crt_products_impl(K, L, v, stream, reinterpret_cast<unsigned int *>(ws + L.sync));
    if (rc == MGX_SUCCESS) rc = crt_combine_impl(C, ldc, beta_one, K, L, v, stream);
    return rc;
}

}  // namespace

extern "C" MGX_API size_t mgx_crt_workspace_size(int m, int n, int k, int moduli)
{
    if (m < 0 || n < 0 || k < 0 || moduli < crt::MINQ || moduli > crt::MAXQ) return 0;
    return crt_layout(m, n, k, moduli).total;
}

extern "C" MGX_API int mgx_crt_kmax(void) { return crt::KMAX; }

int mgx_crt_run(const double *A, const double *B, double *C, int m, int n, int k, int lda, int ldb, int ldc,
                int beta_one, int moduli, void *workspace, size_t workspace_bytes, cudaStream_t stream)
{
    crt::Consts K;
    if (m < 0 || n < 0 || k < 0 || !crt::make_consts(moduli, K) || (m > 0 && n > 0 && (!C || ldc < n)) ||
        (m > 0 && n > 0 && k > 0 && (!A || !B || lda < k || ldb < n))) {
        mgx_set_last_message("mgx_gemm_ozaki_crt: invalid arguments m=%d n=%d k=%d moduli=%d (8..16)", m, n, k, moduli);
        return MGX_E_INVALID;
    }
    if (m == 0 || n == 0) return MGX_SUCCESS;
    if (k == 0) {
        if (beta_one) return MGX_SUCCESS;
        MGX_HOST_CHECK(cudaMemset2DAsync(C, (size_t)ldc * sizeof(double), 0, (size_t)n * sizeof(double), m, stream));
        return MGX_SUCCESS;
    }
    const CrtLayout L = crt_layout(m, n, k, moduli);
    if (!workspace || workspace_bytes < L.total || (reinterpret_cast<uintptr_t>(workspace) & 255)) {
        mgx_set_last_message("mgx_gemm_ozaki_crt: workspace needs %zu bytes, 256-byte aligned (got %zu)", L.total,
                             workspace_bytes);
        return MGX_E_WORKSPACE;
    }
    unsigned char *ws = static_cast<unsigned char *>(workspace);
    for (int k0 = 0; k0 < k; k0 += crt::KMAX) {
        const int kc = (k - k0 < crt::KMAX) ? k - k0 : crt::KMAX;
        int rc = crt_split_impl(A + k0, B + (size_t)k0 * ldb, m, n, kc, lda, ldb, K, ws, L, stream);
        if (rc != MGX_SUCCESS) return rc;
        rc = crt_multiply_impl(C, m, n, ldc, (k0 > 0) ? 1 : beta_one, K, ws, L, stream);
        if (rc != MGX_SUCCESS) return rc;
    }
    return MGX_SUCCESS;
}

static int crt_phase_check(int m, int n, int k, int moduli, const void *workspace, size_t workspace_bytes,
                           const char *who, crt::Consts &K, CrtLayout &L)
{
    if (m < 0 || n < 0 || k < 0 || k > crt::KMAX || !crt::make_consts(moduli, K)) {
        mgx_set_last_message("%s: invalid arguments m=%d n=%d k=%d (<= %d) moduli=%d (8..16)", who, m, n, k, crt::KMAX,
                             moduli);
        return MGX_E_INVALID;
    }
    L = crt_layout(m, n, k, moduli);
    if (!workspace || workspace_bytes < L.total || (reinterpret_cast<uintptr_t>(workspace) & 255)) {
        mgx_set_last_message("%s: workspace needs %zu bytes, 256-byte aligned (got %zu)", who, L.total, workspace_bytes);
        return MGX_E_WORKSPACE;
    }
    return MGX_SUCCESS;
}

extern "C" MGX_API int mgx_crt_split(const double *A, const double *B, int m, int n, int k, int lda, int ldb,
                                     int moduli, void *workspace, size_t workspace_bytes, void *stream)
{
    crt::Consts K;
    CrtLayout L;
    int rc = crt_phase_check(m, n, k, moduli, workspace, workspace_bytes, "mgx_crt_split", K, L);
    if (rc != MGX_SUCCESS) return rc;
    if ((m > 0 && k > 0 && (!A || lda < k)) || (n > 0 && k > 0 && (!B || ldb < n))) {
        mgx_set_last_message("mgx_crt_split: invalid operand pointers or leading dimensions");
        return MGX_E_INVALID;
    }
    if (m == 0 || n == 0 || k == 0) return MGX_SUCCESS;
    return crt_split_impl(A, B, m, n, k, lda, ldb, K, static_cast<unsigned char *>(workspace), L, (cudaStream_t)stream);
}

extern "C" MGX_API int mgx_crt_products(int m, int n, int k, int moduli, void *workspace, size_t workspace_bytes,
                                        void *stream)
{
    crt::Consts K;
    CrtLayout L;
    int rc = crt_phase_check(m, n, k, moduli, workspace, workspace_bytes, "mgx_crt_products", K, L);
    if (rc != MGX_SUCCESS) return rc;
    if (m == 0 || n == 0 || k == 0) return MGX_SUCCESS;
    unsigned char *ws = static_cast<unsigned char *>(workspace);
    return crt_products_impl(K, L, crt_view(L, ws, 0, 0, m, n), (cudaStream_t)stream,
                             reinterpret_cast<unsigned int *>(ws + L.sync));
}

extern "C" MGX_API int mgx_crt_combine(double *C, int m, int n, int k, int ldc, int beta_one, int moduli,
                                       void *workspace, size_t workspace_bytes, void *stream)
{
    crt::Consts K;
    CrtLayout L;
    int rc = crt_phase_check(m, n, k, moduli, workspace, workspace_bytes, "mgx_crt_combine", K, L);
    if (rc != MGX_SUCCESS) return rc;
    if (m > 0 && n > 0 && (!C || ldc < n)) {
        mgx_set_last_message("mgx_crt_combine: invalid C or ldc");
        return MGX_E_INVALID;
    }
    if (m == 0 || n == 0) return MGX_SUCCESS;
    if (k == 0) {
        if (beta_one) return MGX_SUCCESS;
        MGX_HOST_CHECK(cudaMemset2DAsync(C, (size_t)ldc * sizeof(double), 0, (size_t)n * sizeof(double), m,
                                         (cudaStream_t)stream));
        return MGX_SUCCESS;
    }
    unsigned char *ws = static_cast<unsigned char *>(workspace);
    return crt_combine_impl(C, ldc, beta_one ? 1 : 0, K, L, crt_view(L, ws, 0, 0, m, n), (cudaStream_t)stream);
}

// Hooks for the host-buffer schedule (mgx_gemm_host in ozaki.cu): a workspace for the whole
// M x N x K product (K <= KMAX), panels prepared as they arrive and blocks computed from them.
size_t mgx_crt_host_ws_bytes(int M, int N, int K, int q) { return crt_layout(M, N, K, q).total; }

int mgx_crt_host_rows(const double *A, int m, int lda, int r0, int M, int N, int K, int q, unsigned char *ws,
                      cudaStream_t stream)
{
    crt::Consts C;
    if (!crt::make_consts(q, C)) return MGX_E_INVALID;
    return crt_split_a_impl(A, m, K, lda, r0, C, ws, crt_layout(M, N, K, q), stream);
}

int mgx_crt_host_cols(const double *B, int n, int ldb, int c0, int M, int N, int K, int q, unsigned char *ws,
                      cudaStream_t stream)
{
    crt::Consts C;
    if (!crt::make_consts(q, C)) return MGX_E_INVALID;
    return crt_split_b_impl(B, n, K, ldb, c0, C, ws, crt_layout(M, N, K, q), stream);
}

int mgx_crt_host_block(double *Cb, int ldc, int r0, int c0, int m, int n, int M, int N, int K, int q,
                       unsigned char *ws, cudaStream_t stream, int slot)
{
    crt::Consts C;
    if (!crt::make_consts(q, C)) return MGX_E_INVALID;
    const CrtLayout L = crt_layout(M, N, K, q);
    const CrtView v = crt_view(L, ws, r0, c0, m, n);
    int rc = crt_products_impl(C, L, v, stream, reinterpret_cast<unsigned int *>(ws + L.sync) + (slot & 1));
    if (rc == MGX_SUCCESS) rc = crt_combine_impl(Cb, ldc, 0, C, L, v, stream);
    return rc;
}

extern "C" MGX_API size_t mgx_crt_splitk_workspace_size(int m, int n, int k, int moduli, int ksplit)
{
    if (m < 0 || n < 0 || k < 0 || moduli < crt::MINQ || moduli > crt::MAXQ || ksplit < 1 || k > crt::KMAX) return 0;
    return crt_layout(m, n, k, moduli, ksplit).total;
}

extern "C" MGX_API int mgx_gemm_ozaki_crt_splitk(const double *A, const double *B, double *C, int m, int n, int k,
                                                 int lda, int ldb, int ldc, int beta_one, int moduli, int ksplit,
                                                 void *workspace, size_t workspace_bytes, void *stream)
{
    crt::Consts K;
    if (m < 0 || n < 0 || k < 0 || ksplit < 1 || !crt::make_consts(moduli, K) || (m > 0 && n > 0 && (!C || ldc < n)) ||
        (m > 0 && n > 0 && k > 0 && (!A || !B || lda < k || ldb < n))) {
        mgx_set_last_message("mgx_gemm_ozaki_crt_splitk: invalid arguments m=%d n=%d k=%d moduli=%d ksplit=%d", m, n, k,
                             moduli, ksplit);
        return MGX_E_INVALID;
    }
    if (k > crt::KMAX) {
        mgx_set_last_message("mgx_gemm_ozaki_crt_splitk: k = %d is above one int32 residue accumulation (%d)", k,
                             crt::KMAX);
        return MGX_E_UNSUPPORTED;
    }
    if (ksplit == 1 || m == 0 || n == 0 || k == 0)
        return mgx_crt_run(A, B, C, m, n, k, lda, ldb, ldc, beta_one ? 1 : 0, moduli, workspace, workspace_bytes,
                           (cudaStream_t)stream);
    const CrtLayout L = crt_layout(m, n, k, moduli, ksplit);
    if (!workspace || workspace_bytes < L.total || (reinterpret_cast<uintptr_t>(workspace) & 255)) {
        mgx_set_last_message("mgx_gemm_ozaki_crt_splitk: workspace needs %zu bytes, 256-byte aligned (got %zu)", L.total,
                             workspace_bytes);
        return MGX_E_WORKSPACE;
    }
    unsigned char *ws = static_cast<unsigned char *>(workspace);
    cudaStream_t st = (cudaStream_t)stream;
    int rc = crt_split_impl(A, B, m, n, k, lda, ldb, K, ws, L, st);
    if (rc == MGX_SUCCESS) rc = crt_multiply_impl(C, m, n, ldc, beta_one ? 1 : 0, K, ws, L, st);
    return rc;
}

extern "C" MGX_API int mgx_gemm_ozaki_crt(const double *A, const double *B, double *C, int m, int n, int k, int lda,
                                          int ldb, int ldc, int beta_one, int moduli, void *workspace,
                                          size_t workspace_bytes, void *stream)
{
    return mgx_crt_run(A, B, C, m, n, k, lda, ldb, ldc, beta_one ? 1 : 0, moduli, workspace, workspace_bytes,
                       (cudaStream_t)stream);
}

// A-priori modulus count.  With alpha + beta = L - 3 bits shared by the two operands, the
// rounding of A' and B' to integers leaves a normwise error close to sqrt(k / 6) 2^(-(L-3)/2)
// (each entry is rounded to within 1/2, the scale puts row and column norms at 2^alpha, 2^beta);
// measured on the oracle it stays within 2x of that, floored near 5e-17 by the FP64 result.
// Returns the smallest q in 8..16 whose prediction, times 2 and a 1.25 safety factor, meets
// `target`, else 16.
extern "C" MGX_API int mgx_crt_choose_moduli(int k, double target)
{
    if (!(target > 0.0)) target = 1e-15;
    const double kk = k > 1 ? (double)k : 1.0;
    double lp = 0.0;
    for (int q = 1; q <= crt::MAXQ; ++q) {
        lp += log2((double)crt::h_moduli[q - 1]);
        if (q < crt::MINQ) continue;
        const int L = (int)floor(lp) + 1;
        double e = 2.0 * sqrt(kk / 6.0) * exp2(-0.5 * (L - 3));
        if (e < 5e-17) e = 5e-17;
        if (e * 1.25 <= target) return q;
    }
    return crt::MAXQ;
}
