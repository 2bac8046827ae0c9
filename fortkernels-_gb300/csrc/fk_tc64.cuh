// fk_tc64.cuh -- the FP64 band x G contraction on the tensor cores
// (tcgen05): error-free digit products (the Ozaki scheme: K. Ozaki, T. Ogita,
// S. Oishi, S. Rump, Numer. Algorithms 59, 2012) with the fused weighted row
// reduction of fk_gemm.cuh.
//
//   S[m][n] = sum_k A[m][k] * B[n][k]          (complex FP64)
//   P[slot][m][g] = sum_n w(m, n) * S[m][n]    (FP64 partials, fixed order)
//
// Why.  GB300's FP64 pipe (DMMA included) does ~1.2 TFLOP/s; its tensor cores
// do ~1950 TFLOP/s of FP16 products with FP32 accumulation, and sums of integer
// products are exact there while they stay below 2^24.  So every row of an
// operand (per k-slice) is scaled by the power of two that puts its largest
// magnitude into [2^59, 2^60), rounded to a 60-bit integer, and cut into seven
// signed 9-bit digits (values -256..255, exact in FP16; the leading one within
// +-64).  Digit products of the same weight, class c = i + j, share one
// accumulator:
//   S = 2^(Ea + Eb - 46) * sum_{c = 0..6} C_c * 2^(-9 c),  C_c = sum_{i+j=c} sum_k a_i[k] b_j[k]
// (re and im products together).  Classes 0..4 are drained every 32 k-values,
// where |C_c| <= 64 * (2 * 2^14 + 3 * 2^16) < 2^24: every one of these sums is
// exact, and they are added exactly as 64-bit integers.  Classes 5 and 6 weigh
// 2^-45 and 2^-54 and accumulate over the whole k-slice in FP32; classes 7 and
// above are left out.
//
// Error.  Unlike an FP64 dot product's it is relative to the rows' largest
// magnitudes, not to the terms: the classes left out amount to 2^-57.2 sqrt(2 K)
// 2^(Ea + Eb) (rms over a slice of K k-values, measured against exact sums for
// uniform, normal, graded and outlying values; at most 2^-55.7).  On rows of one
// scale that is 2^-55 of |S|, below the rounding of an FP64 sum; on a row with an
// outlier over a zero of the other operand, or on rows graded in opposite
// directions, it can be more than all of S.  So the epilogue keeps, per row and
// weighted sum, the largest term |w| |S| of all columns and slices (rowmax) and
// per unit the largest |w| 2^(Ea + Eb) (bound), both as powers of two, and the
// DMMA kernel of fk_gemm.cuh, launched behind, redoes the tiles (64 rows of a unit)
// where the error exceeds 2^-48 of rowmax in some row (Plan::excess, d64::redo_mask): at
// most 3e-15 of the row's largest term, per column and slice, stays.  The guard costs
// 0.3-1% of a call (512 x 32768 x 20 402 -> 404 us, FF 512 x 4096 x 512 x 15 3.70 -> 3.73 ms,
// the half sum's two contractions at 678 x 1792 x 7 280 -> 286 us).  A row with an infinity, a
// NaN or magnitudes beyond 2^+-400 sets a flag: the contraction then does
// nothing and the DMMA kernel fills all of the partial sums.
//
// One unit is a 256-row x 64-column tile over one k-slice, on a CTA pair
// (tcgen05 cta_group::2, M = 256, N = 128: D = [S_re | S_im]); per 32 k-values
// it issues 28 digit pairs x 4 MMAs of 64 cycles each = 7168 cycles, which
// bound it.  N = 128 is the narrowest MMA at full rate (measured 64 cycles; N =
// 64 takes 43-48, bound by the operand reads of shared memory), and a class then
// takes 128 of the 512 accumulator columns: two buffers rotate through classes
// 0..4 and two hold classes 5 and 6.  Operands arrive digit by digit (A 16 KB
// and half of B 8 KB per CTA) into nine slots and a stage's digit pairs run in
// an order that spreads the classes' drains and the slots' reuse over the stage
// (PAIRS, below).
// Measured (GB300): the contraction of GPP 512 x 2 x 32768 x 20 takes 0.17 ms
// (DMMA 7.85 ms), FF's planes at 512 x 4096 x 512 x 15 take 3.28 ms (DMMA 222 ms;
// the A planes over the bands that read them only).  A call's errors against 64-bit
// references are of the DMMA path's size, on some shapes lower and on some higher (FF
// 512 x 4096 x 512 x 15 1.9e-15 against 4.8e-15, 40 x 640 x 48 x 6 2.6e-15 against
// 8.4e-16, GPP 512 x 32768 x 20 3.0e-15 against 2.6e-15): what is left there is the
// order of the weighted sums, not the digits.
#pragma once
#include <algorithm>
#include <cmath>

#include <cuda_fp16.h>

#include "fk_gemm.cuh"
#include "fk_internal.h"
#include "fk_tc.cuh"
#include "fk_tc_contract.cuh"

namespace fk {
namespace tc64 {

constexpr int ND = 7;                 // digits per value
constexpr int NROT = 5;               // classes 0..4 drained per stage
constexpr int BM = 256, BN = 64;      // tile of a CTA pair (128 rows per CTA)
constexpr int BK = 32;                // complex k-values per stage
constexpr int SLOTS = 9;              // digit slots of the operand ring
constexpr uint32_t A_DIG = 2u * 128 * 64;    // one digit of one CTA's A rows: [re][im][128 rows][64 B]
constexpr uint32_t B_DIG = 2u * 64 * 64;     // one digit of one CTA's half of B
constexpr uint32_t B_IMG = 3u * 64 * 64;     // the same in the image: [im][re][-im][64 rows][64 B]
constexpr uint32_t SLOT_BYTES = A_DIG + B_DIG;
constexpr int THREADS = 384;          // warp 0 MMA (odd CTA: relay), warp 1 copies, warps 4..11 epilogue
constexpr int EPI_WARPS = 8;
constexpr size_t SMEM = (size_t)SLOTS * SLOT_BYTES + 1024 + 512;
constexpr int MAXK = 8192;            // k-values per slice at most: the 64-bit sums and the slice's conversion
constexpr long long DRAIN_LIMIT = 4000000000LL;
constexpr int MAXPL = 64;             // planes of one launch

// Planes (batches) of one launch, each over its own range of 256-row tiles.
struct PlaneTab {
    int n;
    int n2;  // the planes before n2 also get the sums weighted by W2 (FF)
    int u0[MAXPL + 1], mt0[MAXPL], MT[MAXPL];
};

struct Args {
    const uint8_t* A;    // [128-row tile][kstage][digit][re, im][128][64 B]
    const uint8_t* B;    // [plane][nt][kstage][digit][im, re, -im][64][64 B]
    const int* ea;       // [slice][M] exponent of each A row's slice
    const int* eb;       // [plane][slice][N]
    const double2 *W1, *W2;  // epilogue weights [column or igp][M]; W2: FF's second sum (planes before tab.n2)
    double2* P;          // [plane][slice][nt][re/im half][M][G]
    int M, N, NT, KS, kst_unit, kstages, G;
    const int* skip;     // nonzero: a row cannot be represented, do nothing
    unsigned* rowmax;    // [plane][G][M] largest term of each sum (guard_term; zero at entry)
    unsigned* bound;     // [plane][slice][nt][G][M] largest |w| 2^(Ea + Eb) of a unit (zero at entry)
    int re_only;         // only the real parts of the sums are used (real-valued GPP)
    int* err;
    long long wait_limit;
    PlaneTab tab;
};

// ------------------------------------------------------------- conversion
struct SplitArgs {
    const double2 *src, *src2;  // batches from n1 on read their planes from src2
    int n1;
    long ld, plane_stride;
    const int* planes;   // plane index of each batch (nullptr: identity)
    const int* rowmap;   // image row -> source row (nullptr: identity)
    int rows, K, KS, kst_unit, kstages, tiles;  // tiles: row tiles per plane in the image
    uint8_t* img;
    int* exps;           // [plane][slice][rows]
    int* flag;
    int* err;
    long long wait_limit;
};

__device__ __forceinline__ unsigned long long abs_bits(double v) {
    return (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
}
// The guard's powers of two, in few integer instructions and registers: the biased exponent of
// a double (0 .. 2046), of the larger part of a weight, and one word per sum that holds two
// maxima, |w| |S| in its low half and |w| 2^Eb in its high half.  Zeros need no case of
// their own: a zero weight or sum counts as 2^-1023 on both sides of the comparison, a row of
// zeros has the exponent ZERO_ROW, far below that.
constexpr int ZERO_ROW = -2600, GUARD_EB = 3000;
__device__ __forceinline__ unsigned exponent_of(double s) { return ((unsigned)__double2hiint(s) << 1) >> 21; }
__device__ __forceinline__ unsigned exponent_of(double2 w) {
    return max((unsigned)__double2hiint(w.x) << 1, (unsigned)__double2hiint(w.y) << 1) >> 21;
}
__device__ __forceinline__ unsigned guard_pair(double s, int eb) {
    return ((unsigned)(eb + GUARD_EB) << 16) + exponent_of(s);
}
__device__ __forceinline__ unsigned guard_max(unsigned g, unsigned pair, double2 w) {
    return __vmaxu2(g, pair + exponent_of(w) * 0x10001u);
}
// Both maxima on one scale (the second times 2^Ea), as words that are positive for every sum (0: none).
__device__ __forceinline__ unsigned guard_term(unsigned g) { return (g & 0xffffu) + 4096u; }
__device__ __forceinline__ unsigned guard_bound(unsigned g, int ea) {
    return g >> 16 ? (unsigned)max(1, (int)(g >> 16) - GUARD_EB + 1023 + ea + 4096) : 0u;
}
// x as an integer multiple of 2^(E - 59), E = emax - 1023 (|result| <= 2^60),
// plus 256 in every digit position: digit d (0 the leading one) is then the
// 9-bit field at 54 - 9 d minus 256.
__device__ __forceinline__ unsigned long long biased_fixed(double x, int emax) {
    constexpr unsigned long long BIAS = 256ull * 0x0040201008040201ull;  // sum of 256 * 2^(9 i), i = 0..6
    const unsigned long long b = abs_bits(x);
    const int e = (int)(b >> 52);
    unsigned long long m = (b & 0xfffffffffffffull) | (e ? 0x10000000000000ull : 0ull);
    const int sh = 7 - (emax - max(e, 1));
    if (sh >= 0) m <<= sh;
    else m = sh < -60 ? 0ull : (m + (1ull << (-sh - 1))) >> (-sh);
    return __double_as_longlong(x) < 0 ? BIAS - m : BIAS + m;
}
// digits d of two values as an FP16 pair
__device__ __forceinline__ uint32_t digit_pair(unsigned long long u0, unsigned long long u1, int d) {
    const uint32_t f = ((uint32_t)(u0 >> (54 - 9 * d)) & 511u) | (((uint32_t)(u1 >> (54 - 9 * d)) & 511u) << 16);
    const uint32_t biased = f | 0x64006400u;  // 1024 + field
    const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&biased), __half2half2(__ushort_as_half(0x6500)));  // - 1280
    return *reinterpret_cast<const uint32_t*>(&h);
}

// The digits of 8 values k .. k+7 of image row `row`: one 16-byte swizzle chunk per
// digit and part (tile: the row tile's image).
template <bool BSIDE>
__device__ __forceinline__ void store_digits(uint8_t* tile, int row, int k, const double2 (&v)[8], int emax) {
    constexpr int R = BSIDE ? BN : 128;
    unsigned long long ur[8], ui[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        ur[j] = biased_fixed(v[j].x, emax);
        ui[j] = biased_fixed(v[j].y, emax);
    }
    uint8_t* st = tile + (long)(k / BK) * (ND * (BSIDE ? B_IMG : A_DIG)) + tc::sw64_offset(row % R, k % BK);
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        uint4 re, im;
        re.x = digit_pair(ur[0], ur[1], d); re.y = digit_pair(ur[2], ur[3], d);
        re.z = digit_pair(ur[4], ur[5], d); re.w = digit_pair(ur[6], ur[7], d);
        im.x = digit_pair(ui[0], ui[1], d); im.y = digit_pair(ui[2], ui[3], d);
        im.z = digit_pair(ui[4], ui[5], d); im.w = digit_pair(ui[6], ui[7], d);
        if (BSIDE) {
            uint8_t* q = st + (long)d * B_IMG;
            *(uint4*)q = im;
            *(uint4*)(q + 4096) = re;
            *(uint4*)(q + 8192) = make_uint4(im.x ^ 0x80008000u, im.y ^ 0x80008000u, im.z ^ 0x80008000u, im.w ^ 0x80008000u);
        } else {
            uint8_t* q = st + (long)d * A_DIG;
            *(uint4*)q = re;
            *(uint4*)(q + 8192) = im;
        }
    }
}

// One block per (k-slice, row, plane): the slice's largest magnitude, then its
// digits.  Memory-bound: reads 16 and writes 28 (A) or 42 (B, with -im) bytes per
// complex value.  SMEM: the slice (at most SMEM_K k-values) comes to shared memory
// by bulk copies, several blocks per SM overlapping theirs with the others' digits,
// and a thread reads its 8 values in an order rotated by its lane
// (tcx::smem_chunk8); longer slices are read twice from global memory.
constexpr int SMEM_K = 4096;
template <bool BSIDE, bool SMEM_ROW>
__global__ void __launch_bounds__(256) split_kernel(SplitArgs s) {
    extern __shared__ __align__(16) uint8_t smem_row[];
    const double2* rowbuf = (const double2*)smem_row;
    const int ks = blockIdx.x, batch = blockIdx.z;
    const int plane = s.planes ? s.planes[batch] : batch;
    const int kst0 = ks * s.kst_unit, kst1 = min(s.kstages, kst0 + s.kst_unit);
    const int k0 = kst0 * BK, k1 = min(s.K, kst1 * BK), nk = k1 - k0;
    __shared__ unsigned long long wm[8];
    __shared__ __align__(8) uint64_t bar;
    __shared__ int ok;
    if (SMEM_ROW && threadIdx.x == 0) {
        tc::mbar_init(&bar, 1);
        tc::fence_barrier_init();
    }
    uint32_t ph = 0;
    for (int row = blockIdx.y; row < s.rows; row += gridDim.y, ph ^= 1) {
        const double2* src = (batch < s.n1 ? s.src : s.src2) + (long)plane * s.plane_stride + (long)(s.rowmap ? s.rowmap[row] : row) * s.ld + k0;
        if (SMEM_ROW) {
            __syncthreads();  // the previous row was read
            if (threadIdx.x == 0) {
                const uint32_t bytes = (uint32_t)nk * 16u;
                tc::mbar_arrive_expect_tx(&bar, bytes);
                for (uint32_t o = 0; o < bytes; o += 16384u)
                    tc::bulk_g2s(smem_row + o, (const uint8_t*)src + o, min(16384u, bytes - o), &bar);
                ok = tc::mbar_wait(&bar, ph, s.wait_limit) ? 1 : 0;
                if (!ok) {  // the block exits only after its copy has landed
                    atomicOr(s.err, 0x200);
                    tc::mbar_wait(&bar, ph, DRAIN_LIMIT);
                }
            }
            __syncthreads();
            if (!ok) return;
        }
        unsigned long long mx = 0;
        for (int k = threadIdx.x; k < nk; k += blockDim.x) {
            const double2 v = SMEM_ROW ? rowbuf[k] : src[k];
            mx = max(mx, max(abs_bits(v.x), abs_bits(v.y)));
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, off));
        __syncthreads();  // wm of the previous row was read
        if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = mx;
        __syncthreads();
        mx = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) mx = max(mx, wm[w]);
        const int emax = (int)(mx >> 52);
        const bool bad = mx != 0 && (emax < 1023 - 400 || emax > 1023 + 400);  // infinities and NaN too
        if (threadIdx.x == 0) {
            s.exps[((long)batch * s.KS + ks) * s.rows + row] = mx ? emax - 1023 : ZERO_ROW;
            if (bad) atomicOr(s.flag, 1);
        }
        uint8_t* tile = s.img + ((long)batch * s.tiles + row / (BSIDE ? BN : 128)) * s.kstages *
                                    (long)(ND * (BSIDE ? B_IMG : A_DIG));
        for (int c = 8 * threadIdx.x; c < (kst1 - kst0) * BK; c += 8 * blockDim.x) {
            double2 v[8];
            if (SMEM_ROW) {
                tcx::smem_chunk8(rowbuf, c, nk, v);
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = c + j < nk ? src[c + j] : make_double2(0.0, 0.0);
            }
            store_digits<BSIDE>(tile, row, k0 + c, v, emax);
        }
    }
}

// Epilogue weights in FP64, [h][M]: W1 = wscale * vcoul[igp] * conj(aqsm[row][acol]), W2 = conj(aqsm) (or null);
// row = rowmap[m] or m0 + m.  Also clears the guard's nzero words (a memset of its own took 2 us).
static __global__ void weights_kernel(int M, int m0, int ncols, const double2* aqsm, long ldm, const double* vcoul,
                                      const int* igp, const int* acol, double wscale, double2* W1, double2* W2,
                                      const int* rowmap, unsigned* zero, long nzero) {
    const long stride = (long)gridDim.x * gridDim.y * blockDim.x;
    for (long i = ((long)blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x; i < nzero; i += stride) zero[i] = 0;
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    for (int h = blockIdx.y; h < ncols; h += gridDim.y) {
        const int g = igp[h];
        double2 w1 = make_double2(0.0, 0.0), w2 = w1;
        if (g >= 0) {
            const double2 am = aqsm[(long)(rowmap ? rowmap[m] : m0 + m) * ldm + acol[h]];
            w2 = cconj(am);
            w1 = cscale(w2, wscale * vcoul[g]);
        }
        W1[(long)h * M + m] = w1;
        if (W2) W2[(long)h * M + m] = w2;
    }
}

// ------------------------------------------------------------ contraction
// The order of a stage's 28 digit pairs (i, j), each four MMAs (256 cycles):
//   06 60 | 04 40 13 31 22 | 15 | 03 30 12 21 | 51 05 | 02 20 11 | 50 24 42 | 01 10 | 14 41 33 23 32 | 00
// The drained classes 4, 3, 2, 1, 0 end at pairs 7, 12, 17, 22 and 28, about a
// fifth of the stage apart, with the pairs of classes 5 and 6 between them: the
// epilogue takes ~1400 cycles per class, and class after class from 0 to 6 (or
// 6 to 0) left the tensor cores waiting for it (11-12 thousand cycles per stage
// instead of 7168).  Digits become free after pairs 2 (6), 18 (5), 24 (4, 1),
// 27 (3, 2) and 28 (0), at least nine pairs (2300 cycles) before the next
// stage's digit in the same slot is taken.
// The issuing warp's own time counts: it issues an MMA in ~13-18 cycles and ~20
// of them queue up, but a loop that reads the pair from a table, with its waits
// and votes, took ~500 cycles per pair (13.8 thousand per stage), so the pairs are
// unrolled with compile-time digits.
// Entry: i | j << 3 | accumulator << 6 (0: a rotating one, 2, 3: classes 5, 6) |
// first pair of its class << 8 | last pair of a drained class << 9 | first use of
// digit i << 10, of j << 11 | last use of digit i << 12, of j << 13.
constexpr uint32_t pair_at(int n) {
    constexpr uint16_t PAIRS[28] = {
        0x0df0, 0x10c6, 0x0920, 0x0004, 0x0c19, 0x000b, 0x0612,
        0x08e9, 0x0118, 0x0003, 0x0011, 0x020a, 0x00cd, 0x01a8,
        0x0110, 0x0002, 0x0209, 0x1085, 0x00e2, 0x00d4, 0x0108,
        0x0201, 0x00a1, 0x308c, 0x00db, 0x009a, 0x3093, 0x1300};
    return PAIRS[n];
}

// The slots of a stage's digits.  The next stage loads its digits in the order
// 0 6 4 1 3 2 5 into the two spare slots, then the slots of this stage's digits
// 6, 5, 4, 1, 3; the slots of digits 2 and 0 are the next spares.  Every role
// walks the same sequence.  `ph` holds, per slot, the parity of its next use.
struct Ring {
    unsigned long long map = 0x876543210ull;  // four bits per entry: digits 0..6, spares
    uint32_t ph = 0;
    __device__ __forceinline__ int slot(int i) const { return (int)(map >> (4 * i)) & 15; }
    __device__ __forceinline__ uint32_t parity(int s) const { return (ph >> s) & 1u; }
    static __device__ __forceinline__ int load_order(int k) { return (int)(0x5231460u >> (4 * k)) & 15; }
    __device__ __forceinline__ void next() {
#pragma unroll
        for (int i = 0; i < ND; ++i) ph ^= 1u << slot(i);
        auto at = [&](int i) { return (map >> (4 * i)) & 15ull; };
        map = at(7) | at(5) << 4 | at(1) << 8 | at(4) << 12 | at(6) << 16 | at(3) << 20 | at(8) << 24 | at(2) << 28 |
              at(0) << 32;
    }
};

// The four MMAs of a digit pair: k-steps 0 and 1 of A_re x [B_re | B_im] and of
// A_im x [-B_im | B_re] (im tiles 8 KB (A) and 4 KB (B) behind re).  alo, blo: low
// words of the digits' descriptors, hi their common high word.
__device__ __forceinline__ void mma_digits(uint32_t d, uint32_t alo, uint32_t blo, uint32_t hi, uint32_t idesc,
                                           uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p, q;\n .reg .b32 x, y;\n .reg .b64 a, b;\n"
        " setp.ne.b32 p, %5, 0;\n setp.eq.u32 q, 0, 0;\n"
        " mov.b64 a, {%1, %3};\n mov.b64 b, {%2, %3};\n"
        " tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %4, p;\n"
        " add.u32 x, %1, 512;\n add.u32 y, %2, 256;\n mov.b64 a, {x, %3};\n mov.b64 b, {y, %3};\n"
        " tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %4, q;\n"
        " add.u32 x, %1, 2;\n add.u32 y, %2, 2;\n mov.b64 a, {x, %3};\n mov.b64 b, {y, %3};\n"
        " tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %4, q;\n"
        " add.u32 x, %1, 514;\n add.u32 y, %2, 258;\n mov.b64 a, {x, %3};\n mov.b64 b, {y, %3};\n"
        " tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %4, q;\n}\n" ::"r"(d),
        "r"(alo), "r"(blo), "r"(hi), "r"(idesc), "r"(accumulate)
        : "memory");
}

// (h + f) * 2^ex to the nearest double, h a 64-bit integer, |f| < 2^30 (integer
// instructions: the FP64 pipe takes 64 cycles per warp instruction).
__device__ __forceinline__ double fixed_to_double(long long h, float f, int ex) {
    const float fi = rintf(f);
    h += (long long)__float2int_rn(fi);
    // eight more bits below the unit while they fit
    const bool room = (unsigned long long)(h + (1ll << 53)) < (1ull << 54);
    if (room) {
        h = h * 256 + (long long)__float2int_rn((f - fi) * 256.f);
        ex -= 8;
    }
    const unsigned long long a = (unsigned long long)(h < 0 ? -h : h);
    if (a == 0) return 0.0;
    const int lz = __clzll((long long)a);
    const unsigned long long n = a << lz;  // leading one at bit 63
    unsigned long long q = (n >> 11) + ((n >> 10) & 1ull);  // 53 bits, rounded to nearest
    // exponent of bit 63 is 63 - lz + ex; a carry out of the 53 bits adds one to the exponent field
    const unsigned long long bits = ((unsigned long long)(1023 + 63 - lz + ex - 1) << 52) + q;
    return __longlong_as_double((long long)(bits | (h < 0 ? 0x8000000000000000ull : 0ull)));
}

// A unit's part of the guard for sum c of row m: its largest term (the maximum over units and
// halves does not depend on their order) and its bound (the same in both halves).
__device__ __forceinline__ void guard(const Args& t, int pl, int ks, int nt, int c, int m, int half, unsigned g, int ea) {
    if (half == 0 || !t.re_only) atomicMax(&t.rowmax[((long)pl * t.G + c) * t.M + m], guard_term(g));
    if (half == 0) t.bound[((((long)pl * t.KS + ks) * t.NT + nt) * t.G + c) * t.M + m] = guard_bound(g, ea);
}

template <int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1) contract_kernel(const __grid_constant__ Args t) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* base = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = (uint64_t*)(base + SLOTS * SLOT_BYTES);
    uint64_t* full = bars;                 // [SLOTS] the slot's copies have landed (even CTA: in both)
    uint64_t* empty = bars + SLOTS;        // [SLOTS] the slot's MMAs are done
    uint64_t* accFull = bars + 2 * SLOTS;  // [4]
    uint64_t* accEmpty = accFull + 4;      // [4]
    uint64_t* done = accEmpty + 4;
    uint32_t* tslot = (uint32_t*)(done + 1);
    __shared__ int s_abort_flag;
    volatile int& s_abort = s_abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = tc::cluster_rank();
    const int pid = (int)(blockIdx.x >> 1), npairs = (int)(gridDim.x >> 1);
    if (*t.skip) return;  // the same in every CTA: written by earlier launches only

    if (tid == 0) {
        for (int s = 0; s < SLOTS; ++s) {
            tc::mbar_init(&full[s], rank == 0 ? 2 : 1);  // its copies, and the relay of the odd CTA's
            tc::mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 4; ++b) {
            tc::mbar_init(&accFull[b], 1);
            tc::mbar_init(&accEmpty[b], 2 * EPI_WARPS);
        }
        tc::mbar_init(done, 1);
        tc::fence_barrier_init();
        s_abort = 0;
    }
    if (warp == 0) {
        tc::tmem_alloc_pair(tslot, 512);
        tc::tmem_relinquish_pair();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::cluster_sync();
    tc::tc_fence_after();
    const uint32_t tmem = *tslot;
    const int units = t.tab.u0[t.tab.n];
    const long long lim = t.wait_limit;
    auto fail = [&](int code) {
        atomicOr(t.err, code);
        s_abort = 1;
    };
    // unit -> plane, this pair's 256-row tile, n-tile, k-slice and its stages
    struct Unit {
        int pl, mt, nt, ks, nst;
    };
    auto unit_of = [&](int u, int& pl) {
        while (u >= t.tab.u0[pl + 1]) ++pl;
        Unit x;
        x.pl = pl;
        int r = u - t.tab.u0[pl];
        x.mt = t.tab.mt0[pl] + r % t.tab.MT[pl];
        r /= t.tab.MT[pl];
        x.nt = r % t.NT;
        x.ks = r / t.NT;
        x.nst = min(t.kstages, (x.ks + 1) * t.kst_unit) - x.ks * t.kst_unit;
        return x;
    };

    // 384 threads at 168 registers (64512) are split 128 x 72 + 256 x 216 (64512)
    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    if (warp == 0) {
        if (rank == 1 && lane == 0) {
            // ---------------------------------------------------- relay (odd CTA)
            Ring ring;
            int pl = 0;
            bool ok = true;
            for (int u = pid; u < units && ok; u += npairs) {
                const Unit x = unit_of(u, pl);
                for (int st = 0; st < x.nst && ok; ++st, ring.next())
                    for (int k = 0; k < ND; ++k) {
                        const int s = ring.slot(Ring::load_order(k));
                        if (!tc::mbar_wait(&full[s], ring.parity(s), lim) || s_abort) {
                            fail(2);
                            ok = false;
                            break;
                        }
                        tc::mbar_arrive_peer(&full[s], 0);
                    }
            }
        } else if (rank == 0) {
            // ---------------------------------------------------------------- MMA (all lanes; one issues)
            const bool issue = tc::elect_one();
            const uint32_t idesc = tc::idesc_f16(BM, 2 * BN);
            // descriptors differ in the address field (low word) only
            const uint64_t d0 = tc::sdesc_sw64(tc::smem_u32(base));
            const uint32_t dhi = (uint32_t)(d0 >> 32), dlo = (uint32_t)d0;
            Ring ring;
            uint32_t rc = 0, uc = 0;  // rotating classes issued, units
            int pl = 0;
            bool ok = true;
            for (int u = pid; u < units && ok; u += npairs, ++uc) {
                const Unit x = unit_of(u, pl);
                for (int st = 0; st < x.nst && ok; ++st, ring.next()) {
                    uint32_t lo[ND];  // low words of the digits' A descriptors
#pragma unroll
                    for (int i = 0; i < ND; ++i) lo[i] = dlo + (uint32_t)ring.slot(i) * (SLOT_BYTES >> 4);
                    auto landed = [&](int i) {
                        const int s = ring.slot(i);
                        return tc::mbar_wait_cluster(&full[s], ring.parity(s), lim);
                    };
#pragma unroll
                    for (int n = 0; n < 28; ++n) {
                        constexpr uint32_t ROT = 0xC0, FIRST = 0x100, LAST = 0x200, TAKE = 0xC00;
                        const uint32_t e = pair_at(n);  // compile-time: the loop is unrolled
                        const int i = e & 7, j = (e >> 3) & 7;
                        const bool rot = !(e & ROT);
                        const uint32_t buf = rot ? (rc & 1u) : (e >> 6) & 3u;
                        if (e & (TAKE | FIRST)) {
                            bool ready = (!(e & 0x400) || landed(i)) && (!(e & 0x800) || landed(j));
                            if ((e & FIRST) && (rot || st == 0))
                                ready = tc::mbar_wait_cluster(&accEmpty[buf], (rot ? (rc >> 1) & 1u : uc & 1u) ^ 1u, lim) && ready;
                            if (!tc::warp_all(ready)) {
                                fail((e & TAKE) ? 2 : 1);
                                ok = false;
                                break;
                            }
                            tc::tc_fence_after();
                        }
                        if (issue) {
                            mma_digits(tmem + buf * 128u, lo[i], lo[j] + (A_DIG >> 4), dhi, idesc,
                                       ((e & FIRST) && (rot || st == 0)) ? 0u : 1u);
                            if (e & LAST) tc::mma_commit_pair(&accFull[buf], 3);
                            if (e & 0x1000) tc::mma_commit_pair(&empty[ring.slot(i)], 3);
                            if (e & 0x2000) tc::mma_commit_pair(&empty[ring.slot(j)], 3);
                        }
                        if (e & LAST) ++rc;
                    }
                }
                if (ok && issue) {
                    tc::mma_commit_pair(&accFull[2], 3);
                    tc::mma_commit_pair(&accFull[3], 3);
                }
            }
            // every issued MMA has completed before TMEM and the operands are released
            if (issue) tc::mma_commit_pair(done, 1);
            if (!tc::mbar_wait(done, 0, DRAIN_LIMIT)) fail(4);
        }
    } else if (warp == 1) {
        // -------------------------------------------------------------- copies
        if (lane == 0) {
            Ring ring;
            int pl = 0;
            uint32_t used = 0, last = 0;  // slots copied into, and the parity of each one's last copy
            bool ok = true;
            for (int u = pid; u < units && ok; u += npairs) {
                const Unit x = unit_of(u, pl);
                const long kst0 = (long)x.ks * t.kst_unit;
                const uint8_t* a = t.A + ((long)(2 * x.mt + (int)rank) * t.kstages + kst0) * (long)(ND * A_DIG);
                const uint8_t* b = t.B + (((long)x.pl * t.NT + x.nt) * t.kstages + kst0) * (long)(ND * B_IMG) +
                                   (rank == 0 ? 4096 : 0);  // even CTA: [re; -im], odd: [im; re]
                for (int st = 0; st < x.nst && ok; ++st, ring.next(), a += ND * A_DIG, b += ND * B_IMG)
                    for (int k = 0; k < ND; ++k) {
                        const int i = Ring::load_order(k), s = ring.slot(i);
                        if (!tc::mbar_wait(&empty[s], ring.parity(s) ^ 1u, lim) || s_abort) {
                            fail(8);
                            ok = false;
                            break;
                        }
                        uint8_t* dst = base + s * SLOT_BYTES;
                        tc::mbar_arrive_expect_tx(&full[s], SLOT_BYTES);
                        tc::bulk_g2s(dst, a + i * A_DIG, A_DIG, &full[s]);
                        tc::bulk_g2s(dst + A_DIG, b + i * B_IMG, B_DIG, &full[s]);
                        used |= 1u << s;
                        last = (last & ~(1u << s)) | ring.parity(s) << s;
                    }
            }
            // every copy this thread started lands before the CTA exits
            bool drained = true;
            for (int s = 0; s < SLOTS; ++s)
                if (used >> s & 1u) drained = drained && tc::mbar_wait(&full[s], last >> s & 1u, DRAIN_LIMIT);
            if (!drained) fail(128);
        }
    }
    } else {
        // ------------------------------------------------------------ epilogue
        asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
        // warp = (lane quarter, half): rows q4*32 + lane, columns of S_re (half 0) or S_im (half 1)
        const int q4 = warp & 3, half = (warp - 4) >> 2;
        const uint32_t tl = tmem + ((uint32_t)(q4 * 32) << 16) + (uint32_t)(half * BN);
        uint32_t rc = 0, uc = 0;
        int pl = 0;
        bool ok = true;
        for (int u = pid; u < units && ok; u += npairs, ++uc) {
            const Unit x = unit_of(u, pl);
            long long H[BN];
#pragma unroll
            for (int j = 0; j < BN; ++j) H[j] = 0;
            auto wait_full = [&](uint32_t buf, uint32_t par) {
                if (!tc::warp_all(tc::mbar_wait(&accFull[buf], par, lim) && !s_abort)) {
                    fail(16);
                    return false;
                }
                tc::tc_fence_after();
                return true;
            };
            auto release = [&](uint32_t buf) {
                tc::tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if (rank == 1) tc::mbar_arrive_peer(&accEmpty[buf], 0);
                    else tc::mbar_arrive(&accEmpty[buf]);
                }
            };
            for (int st = 0; st < x.nst && ok; ++st) {
#pragma unroll
                for (int c = NROT - 1; c >= 0; --c, ++rc) {
                    const uint32_t buf = rc & 1u;
                    if (!wait_full(buf, (rc >> 1) & 1u)) {
                        ok = false;
                        break;
                    }
                    // the second half's load is in flight while the first half is added
                    float v[2][32];
                    auto load = [&](int h) {
                        tc::tmem_ld16(tl + buf * 128u + 32 * h, *(float(*)[16]) & v[h][0]);
                        tc::tmem_ld16(tl + buf * 128u + 32 * h + 16, *(float(*)[16]) & v[h][16]);
                    };
                    auto add = [&](int h) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) asm volatile("" : "+f"(v[h][j]));  // not before its wait
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            H[32 * h + j] += (long long)__float2int_rn(v[h][j]) * (1ll << (36 - 9 * c));
                    };
                    load(0);
                    tc::tmem_ld_wait();
                    load(1);
                    add(0);
                    tc::tmem_ld_wait();
                    release(buf);
                    add(1);
                }
            }
            if (!ok || !wait_full(2, uc & 1u) || !wait_full(3, uc & 1u)) {
                ok = false;
                break;
            }
            // classes 5 and 6, then the weighted row sums
            const int m = x.mt * BM + (int)rank * 128 + q4 * 32 + lane, mc = min(m, t.M - 1);
            const int ea = t.ea[(long)x.ks * t.M + mc];
            const int* ebp = t.eb + ((long)x.pl * t.KS + x.ks) * t.N + x.nt * BN;
            const int n0 = x.nt * BN, ncol = min(BN, t.N - n0);
            const bool both = EPI == EPI_FF && x.pl < t.tab.n2;
            double2 g[3] = {make_double2(0.0, 0.0), make_double2(0.0, 0.0), make_double2(0.0, 0.0)};
            unsigned gm[3] = {0u, 0u, 0u};  // the guard's maxima of each sum
            // GPP: eight columns per turn of a rolled loop, H moving down by eight, and g[k] the sum
            // of class (t0 + k) % 3 of the columns.  Unrolled over the 64 columns the code runs once
            // per unit and its bound was fetching it: 64 x 777 x 7 220 -> 217 us, 512 x 32768 x 20
            // 409 -> 400 us.  FF (twice the arithmetic per column) stays unrolled: rolled, 40 x 640 x
            // 48 x 6 took 130 us instead of 127.
            constexpr int TURN = EPI == EPI_FF ? BN : 8;
#pragma unroll 1
            for (int t0 = 0; t0 < BN; t0 += TURN) {
#pragma unroll
                for (int q = 0; q < TURN; q += 8) {
                    const int j0 = t0 + q;
                    float c5[8], c6[8];
                    tc::tmem_ld8(tl + 256u + j0, c5);
                    tc::tmem_ld8(tl + 384u + j0, c6);
                    tc::tmem_ld_wait();
                    if (j0 + 8 >= BN) {
                        release(2);
                        release(3);
                    }
#pragma unroll
                    for (int jb = 0; jb < 8; jb += 4) {
                        if (EPI != EPI_FF && j0 + jb >= ncol) continue;  // warp-uniform
                        double2 w1[4], w2[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const int col = min(j0 + jb + j, ncol - 1), n = n0 + col, h = EPI == EPI_GPP ? n / 3 : n;
                            w1[j] = t.W1[(long)h * t.M + mc];
                            if (EPI == EPI_FF) w2[j] = both ? t.W2[(long)h * t.M + mc] : make_double2(0.0, 0.0);
                        }
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            if (j0 + jb + j >= ncol) continue;  // warp-uniform
                            const double s = fixed_to_double(
                                H[q + jb + j], fmaf(c6[jb + j], 0x1p-18f, c5[jb + j] * 0x1p-9f), ea + ebp[j0 + jb + j] - 46);
                            // half 0: w * s, half 1: w * (i s)
                            const int gi = EPI == EPI_GPP ? (jb + j) % 3 : 0;
                            const double sr = half ? -s : s;
                            const unsigned pair = guard_pair(s, ebp[j0 + jb + j]);
                            gm[gi] = guard_max(gm[gi], pair, w1[j]);
                            g[gi].x = fma(half ? w1[j].y : w1[j].x, sr, g[gi].x);
                            g[gi].y = fma(half ? w1[j].x : w1[j].y, s, g[gi].y);
                            if (EPI == EPI_FF && both) {
                                gm[1] = guard_max(gm[1], pair, w2[j]);
                                g[1].x = fma(half ? w2[j].y : w2[j].x, sr, g[1].x);
                                g[1].y = fma(half ? w2[j].x : w2[j].y, s, g[1].y);
                            }
                        }
                    }
                }
#pragma unroll
                for (int j = 0; j + TURN < BN; ++j) H[j] = H[j + TURN];
                if (EPI == EPI_GPP) {  // (t0 + 8) % 3 = (t0 + 2) % 3
                    auto turn = [](auto(&v)[3]) {
                        const auto v0 = v[0], v1 = v[1];
                        v[0] = v[2];
                        v[1] = v0;
                        v[2] = v1;
                    };
                    turn(g);
                    turn(gm);
                }
            }
            if (EPI == EPI_GPP) {  // back to class k % 3 (64 % 3 = 1)
                auto back = [](auto(&v)[3]) {
                    const auto v2 = v[2];
                    v[2] = v[1];
                    v[1] = v[0];
                    v[0] = v2;
                };
                back(g);
                back(gm);
            }
            if (m < t.M) {
                double2* out = t.P + ((((long)x.pl * t.KS + x.ks) * t.NT + x.nt) * 2 + half) * (long)t.M * t.G + (long)m * t.G;
                if (EPI == EPI_GPP) {
                    // column n0 + j is of frequency (n0 + j) % 3
                    const int r = n0 % 3;
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        out[(q + r) % 3] = g[q];
                        guard(t, x.pl, x.ks, x.nt, (q + r) % 3, m, half, gm[q], ea);
                    }
                } else {
                    for (int q = 0; q < t.G; ++q) {
                        out[q] = q == 0 ? g[0] : g[1];
                        guard(t, x.pl, x.ks, x.nt, q, m, half, q == 0 ? gm[0] : gm[1], ea);
                    }
                }
            }
        }
    }

    tc::tc_fence_before();
    __syncthreads();
    tc::cluster_sync();  // neither CTA releases its operands or TMEM before both are done
    if (warp == 0) {
        __syncwarp();
        tc::tmem_dealloc_pair(tmem, 512);
    }
}

// ------------------------------------------------------------------- plan
constexpr size_t GUARD_HEAD = 256;  // the flag of rows that cannot be represented, in front of the guard's words
struct Plan {
    int MT, NT, KS, kst_unit, kstages;
    size_t bytesA, bytesB, bytesEa, bytesEb;  // images and exponents (B: of one plane)
    size_t slots() const { return (size_t)KS * NT * 2; }  // partial slots per plane
    // the guard's words (Bufs::guard) of `planes` planes of G sums over M rows
    size_t guard_bytes(int M, int G, int planes) const {
        return GUARD_HEAD + (size_t)planes * G * M * (1 + (size_t)KS * NT) * sizeof(unsigned);
    }
    // A tile is redone where bound exceeds rowmax by more than this power of two: the error
    // 2^-57.2 sqrt(2 K) 2^bound then exceeds 2^-48 2^rowmax.  (The synthetic inputs of this
    // package, all branches: at most 2^3 sqrt(2 K), 2^5 for a single column of 32 k-values;
    // the limit is 2^9.)
    int excess() const { return (int)std::floor(9.0 - 0.5 * std::log2(2.0 * kst_unit * BK)); }
};

// The k-split: the fewest pair-cycles over whole waves, a unit costing ~8700
// cycles per stage and `sums` for its weighted sums (measured on GB300: ~50000 for one
// sum per column, ~90000 with FF's second one; see the epilogue's FP64 instructions).
// row_tiles: the launch's row tiles over all planes (0: every plane has all of
// them).  KS == 0: no split fits (callers keep the DMMA kernel).
inline Plan make_plan(int M, int N, int K, int planes, int pairs, long row_tiles = 0, double sums = 50000.0) {
    Plan p{};
    p.MT = ceil_div(std::max(M, 1), BM);
    p.NT = ceil_div(std::max(N, 1), BN);
    p.kstages = ceil_div(K, BK);
    const long tiles = (row_tiles > 0 ? row_tiles : (long)p.MT * std::max(planes, 1)) * p.NT;
    double best = 1e300;
    for (int ks = 1; ks <= std::min(p.kstages, 512); ++ks) {
        const int ku = ceil_div(p.kstages, ks);
        if (ku * BK > MAXK || ceil_div(p.kstages, ku) != ks) continue;
        if (2l * p.NT * ks * std::max(planes, 1) > 65535) continue;  // the DMMA kernel's grid
        const long waves = (tiles * ks + pairs - 1) / pairs;
        const double cost = (double)waves * (ku * 8700.0 + sums);
        if (cost < best * 0.999) {
            best = cost;
            p.KS = ks;
            p.kst_unit = ku;
        }
    }
    p.bytesA = (size_t)2 * p.MT * p.kstages * ND * A_DIG;
    p.bytesB = (size_t)p.NT * p.kstages * ND * B_IMG;
    p.bytesEa = (size_t)p.KS * std::max(M, 1) * sizeof(int);
    p.bytesEb = (size_t)p.KS * std::max(N, 1) * sizeof(int);
    return p;
}

// Workspace of one contraction: images, exponents, weights.
struct Bufs {
    uint8_t *A, *B;
    int *ea, *eb;
    double2 *W1, *W2;
    uint8_t* guard;       // [flag][rowmax of `planes` planes][bound]
    size_t guard_bytes;
    int planes;           // planes the guard covers
    int* flag() const { return (int*)guard; }
    unsigned* rowmax() const { return (unsigned*)(guard + GUARD_HEAD); }
};

template <bool BSIDE>
inline void launch_split(Ctx& c, const SplitArgs& s, int batches) {
    const int nk = s.kst_unit * BK;
    const dim3 grid(s.KS, std::min(s.rows, 65535), batches);
    const int threads = nk > 1024 ? 256 : 128;
    if (nk <= SMEM_K) {
        auto k = split_kernel<BSIDE, true>;
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_K * 16);
        // the SM's memory split as the GPP prep asks for it, so that blocks of both share an SM
        cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        k<<<grid, threads, nk * 16, c.stream>>>(s);
    } else {
        split_kernel<BSIDE, false><<<grid, threads, 0, c.stream>>>(s);
    }
    ++c.launches;
}

// The digits of a.A's rows m0 .. m0+M-1 (or rowmap[0 .. M)) and the flag's reset.
inline cudaError_t enqueue_a(Ctx& c, const ContractArgs& a, const Plan& p, const Bufs& b) {
    const cudaError_t e = cudaMemsetAsync(b.flag(), 0, sizeof(int), c.stream);
    if (e != cudaSuccess) return e;
    SplitArgs s{a.rowmap ? a.A : a.A + (long)a.m0 * a.lda, nullptr, 1, a.lda, 0, nullptr, a.rowmap, a.M, a.K, p.KS, p.kst_unit,
                p.kstages, 2 * p.MT, b.A, b.ea, b.flag(), c.errword, c.wait_limit};
    launch_split<false>(c, s, 1);
    return cudaSuccess;  // (launch errors: the caller's check behind its last launch)
}

// The digits of a.batches planes (at most MAXPL) of a.B, the contraction over the row tiles of `tab` and the
// DMMA kernel for rows that cannot be represented and tiles the digits are too coarse for.  The
// launch's first plane is plane0 of the guard's; re_only as in Args.
template <int EPI>
inline void enqueue(Ctx& c, ContractArgs a, const Plan& p, const Bufs& b, const PlaneTab& tab, int plane0 = 0,
                    bool re_only = false) {
    SplitArgs s{(const double2*)a.B, (const double2*)a.B2, a.B2 ? a.batches1 : a.batches, a.ldb, a.bstride, a.batch_plane, nullptr, a.N, a.K, p.KS, p.kst_unit, p.kstages,
                p.NT, b.B, b.eb, b.flag(), c.errword, c.wait_limit};
    launch_split<true>(c, s, a.batches);
    const long rows = (long)a.G * a.M;  // guard words per plane: rowmax, and bound of one unit column
    unsigned* rowmax = b.rowmax() + plane0 * rows;
    unsigned* bound = b.rowmax() + b.planes * rows + plane0 * rows * p.KS * p.NT;
    Args t{b.A, b.B, b.ea, b.eb, b.W1, b.W2, a.P, a.M, a.N, p.NT, p.KS, p.kst_unit, p.kstages, a.G,
           b.flag(), rowmax, bound, re_only ? 1 : 0, c.errword, c.wait_limit, tab};
    auto k = contract_kernel<EPI>;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
    kernel_begin(c);
    k<<<2 * std::min(tab.u0[tab.n], c.sms / 2), THREADS, SMEM, c.stream>>>(t);
    kernel_end(c);
    a.nt_tiles = 2 * p.NT;
    a.KS = p.KS;
    a.kchunk = p.kst_unit * BK;
    auto f = d64::contract_kernel<EPI>;
    cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)d64::SMEM);
    const int tiles = ceil_div(a.M, d64::BM) * a.nt_tiles * a.KS * a.batches;
    f<<<std::min(tiles, 2 * c.sms), d64::THREADS, d64::SMEM, c.stream>>>(a, d64::Redo{b.flag(), rowmax, bound, p.excess()});
    c.launches += 2;
}

// The weights, and the guard's reset: ahead of each contraction, or of a call's launches over its planes.
inline void enqueue_weights(Ctx& c, const ContractArgs& a, int ncols, const Bufs& b, bool second) {
    weights_kernel<<<dim3(ceil_div(a.M, 128), std::min(ncols, 65535)), 128, 0, c.stream>>>(
        a.M, a.m0, ncols, a.aqsm, a.ldm, a.vcoul, a.igp, a.acol, a.wscale, b.W1, second ? b.W2 : nullptr, a.rowmap,
        b.rowmax(), (long)((b.guard_bytes - GUARD_HEAD) / sizeof(unsigned)));
    ++c.launches;
}

inline PlaneTab one_plane(const Plan& p) {
    PlaneTab t{};
    t.n = 1;
    t.u0[1] = p.MT * p.NT * p.KS;
    t.MT[0] = p.MT;
    return t;
}

}  // namespace tc64
}  // namespace fk
