/*
 * Split-precision (Ozaki-style) form of the FMM GEMM on the sm_103a tensor
 * cores, with BF16 slices (base-256 digits, tcgen05 kind::f16) or FP8-E4M3
 * slices (base-32 digits, kind::f8f6f4). db below is the digit width: 8 or 5.
 *
 * Per product r of the (flattened) FMM algorithm:
 *
 *   1. exps:   row exponents E_i of S_r = sum_q U[q,r] A_q and column
 *              exponents F_j of T_r = sum_q V[q,r] B_q, from the bound
 *              |S_r[i,:]| <= sum_q |U[q,r]| * max|A_q[i,:]|, evaluated in FP64
 *              in the same order as the sums themselves (so the bound holds
 *              for the rounded sums too). The per-sub-block row/column maxima
 *              are computed once per call (amax/bmax kernels). These
 *              power-of-two scales are per row of S_r and per column of T_r
 *              for both formats: a scale that varied along k would give each
 *              k block's products a different weight and end the exact
 *              integer accumulation over k.
 *   2. pack:   the fused multi-operand pack (plugin/ref_kernels/
 *              bli_packm_fmm_ref.c:89-147): S_r (T_r) is formed in FP64 in
 *              sub-block order with zero fill, then split there into `s`
 *              balanced base-2^db digits d_1..d_s:
 *                  S[i,p] ~= 2^(E_i + 1 - db*s) * sum_t d_t[i,p] 2^(db(s-t))
 *              using integer arithmetic on the FP64 bit pattern. BF16 digits
 *              are integers in [-128, 128] (at most 8 significant bits), FP8
 *              digits integers in [-16, 16] (at most 4): exact either way.
 *              Digits are written K-major ("slices" [t][row][k]).
 *   3. gemm:   tcgen05.mma (FP32 accumulation in TMEM) over the slice pairs
 *              (t,u) with t+u = g for the levels g = 2..s+1. A digit product
 *              is an integer of magnitude <= 2^14 (BF16) or 2^8 (FP8), so a
 *              chunk of 16 stage rows (1024 BF16 or 2048 FP8 terms) sums to an
 *              integer of magnitude <= 2^24 that FP32 holds exactly; the
 *              epilogue warps drain each chunk from TMEM (double-buffered, so
 *              the tensor core keeps running), convert it exactly to int32 and
 *              add it to the level sum L_g. The level sums make up a 64-bit
 *              fixed-point value Z in units of level G (BF16: G = 6, or 7
 *              when k_pad <= 128; FP8: G = min(s + 1, 10); the finest units
 *              that keep Z inside int64), written to global memory digit by
 *              digit as the levels finish (ZPlanes):
 *                  Z = sum_{g<=G} L_g * 2^(db(G-g)) + sum_{g>G} round(L_g / 2^(db(g-G)))
 *              and M_r[i,j] ~= 2^(E_i + F_j + 2 - db*G) * Z is formed in FP64
 *              and added with alpha*W[p,r] into every C sub-block p (the
 *              multi-C epilogue, plugin/ref_kernels/bli_gemm_fmm_ref.c:99-120).
 *
 * FP64 is only used for the packing sums, the bounds, the int64 -> FP64
 * conversion and the C updates; the digit split, the level sums and Z are
 * exact integer arithmetic, so the result is deterministic and reproducible
 * bit for bit by a CPU restatement.
 *
 * Limits: k_e = ceil(k/k~) <= 16384 per call (level sums stay inside int32
 * and Z inside int64); slices 2..8 (BF16) or 2..12 (FP8); finite inputs.
 *
 * Execution. Two persistent GEMM kernels: split_gemm_kernel (one CTA per SM,
 * 128 x 256 tiles) and split_gemm_pair_kernel (clusters of two CTAs, 256 x 256
 * tiles, tcgen05.mma cta_group::2), used from m_e = 1024; both draw their
 * (problem, product, tile) work items dynamically from a counter, so the
 * items in flight stay contiguous. A single call packs, multiplies and
 * updates C per product group; when the workspace holds all products it runs
 * them as two groups, the second group's packs and the first group's C
 * updates on pool streams beside the other group's GEMM, and a group's GEMM
 * as launches of about 24 rounds of items. The host-buffer call overlaps the
 * copies with the work (A in row halves and B in column chunks chased by
 * their packs, the GEMM in up to 2 x 4 blocks of tiles that start on a part of
 * each operand, each block's C sent and read back with its C updates), unless
 * the operands are small. A classical call runs three kernels: prep_kernel
 * (maxima, exponents and digits), the GEMM, with the tiles of a small grid cut
 * into work units, and the C updates. Batched calls run waves of up
 * to 80 problems, one GEMM launch per tile kind per wave, waves alternating
 * between two workspace halves so a wave's packs overlap the previous wave.
 * Every path gives the same bits for a problem.
 */
#include "fmm_internal.h"
#include "sm103_ptx.cuh"

#include <cuda.h>
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <chrono>
#include <atomic>
#include <cstring>
#include <deque>
#include <mutex>
#include <type_traits>
#include <utility>
#include <vector>

namespace {

constexpr int kTileM = 128;
constexpr int kTileN = 256;             /* N = 256: 128 clocks per MMA hide the accumulator dependency */
constexpr int kBK = 64;                 /* BF16 k elements per stage (128 bytes; 128 FP8 elements) */
constexpr int kStages = 4;
constexpr int kChunkKB = 16;            /* k-blocks per exact FP32 chunk: 1024 terms, |sum| <= 2^24 */
constexpr int kEpiWarps = 16;          /* four per TMEM lane quarter */
constexpr int kEpiCols = kTileN / 4;    /* columns per epilogue thread */
constexpr int kGemmThreads = 64 + 32 * kEpiWarps;  /* TMA warp, MMA warp, epilogue warps */
constexpr uint32_t kATileBytes = kTileM * kBK * 2;  /* 16 KB */
constexpr uint32_t kBTileBytes = kTileN * kBK * 2;  /* 32 KB */
constexpr uint32_t kStageBytes = kATileBytes + kBTileBytes;
constexpr int kTmemCols = 512;          /* 2 x 256 accumulator columns */
constexpr int kMaxKe = 16384;
constexpr int kRasterGroup = 12;        /* tile rows per raster band */
constexpr size_t kGemmSmem = (size_t)kStages * kStageBytes + 1024 + 256;

__host__ __device__ __forceinline__ int64_t round_up(int64_t x, int64_t m) { return (x + m - 1) / m * m; }

/* ------------------------------------------------------------ digits ---- */

/* E with 2^(E-1) <= b < 2^E for finite b > 0; 0 for b == 0. */
__device__ __forceinline__ int exp_above(double b)
{
    const uint64_t bits = (uint64_t)__double_as_longlong(b) & 0x7fffffffffffffffull;
    if (bits == 0) return 0;
    const int bexp = (int)(bits >> 52);
    if (bexp > 0) return bexp - 1022;
    return -1010 - __clzll((long long)bits);
}

/* Balanced base-2^DB digits of x relative to 2^E (|x| < 2^E): X =
 * round(x * 2^(DB*s-E-1)) (ties away from zero), |X| <= 2^(DB*s-1), split as
 * d[s-1], ..., d[1] in [-2^(DB-1), 2^(DB-1)) from the bottom and d[0] in
 * [-2^(DB-1), 2^(DB-1)]. DB = 8 (BF16 slices): every digit has at most 8
 * significant bits; DB = 5 (FP8-E4M3 slices): every digit is an integer of
 * magnitude at most 16, at most 4 significant bits. Both are exact.
 * The same digits in one step: Y = X + sum_{j < S-1} 2^(DB-1) * 2^(DB*j).
 * Adding 2^(DB-1) at every lower digit position turns the balanced digits
 * into plain DB-bit fields, so the low S-1 fields of Y are d[S-1] + 2^(DB-1),
 * ..., d[1] + 2^(DB-1) and floor(Y / 2^(DB(S-1))) is d[0]: the balanced
 * digits above, without a digit loop. Y is kept modulo 2^64 (its low fields
 * are exact); d[0] is (X >> DB(S-1)) plus the carry out of the low fields,
 * which stays exact for the 64-bit X of the largest S. */
struct Digits {
    int64_t X;
    uint64_t Y;
};

template <int S, int DB>
__host__ __device__ constexpr uint64_t digit_offset()
{
    uint64_t off = 0;
    for (int j = 0; j < S - 1; ++j) off |= (uint64_t)1 << (DB * j + DB - 1);
    return off;
}

template <int S, int DB>
__device__ __forceinline__ Digits split_offset_any(double x, int E)
{
    const uint32_t hi = (uint32_t)__double2hiint(x);
    const int bexp = (int)(hi >> 20) & 0x7ff;
    /* |x| = mant * 2^ex; a subnormal has exponent field 1 without the implicit bit */
    const int ex = (bexp > 1 ? bexp : 1) - 1075;
    const uint64_t mant = ((uint64_t)((hi & 0x000fffffu) | (bexp ? 0x00100000u : 0u)) << 32) | (uint32_t)__double2loint(x);
    /* round(mant * 2^sh), ties away: ((mant >> (r - 1)) + 1) >> 1 with r = -sh.
     * PTX shifts by 64 and more give 0, as the rounding does there. For a
     * normal |x| < 2^E sh is at most DB*S - 54: left shifts are rare. */
    const int sh = ex + DB * S - E - 1;
    uint64_t t;
    asm("shr.u64 %0, %1, %2;" : "=l"(t) : "l"(mant), "r"((uint32_t)(-sh - 1)));
    uint64_t u = (t + 1) >> 1;
    if (sh >= 0) u = mant << sh;
    const int64_t neg = (int64_t)(int32_t)hi >> 31;   /* 0 or -1 */
    const int64_t X = ((int64_t)u ^ neg) - neg;
    return Digits{X, (uint64_t)X + digit_offset<S, DB>()};
}

/* split_offset_any for N elements of one line, in about half the integer
 * instructions (which bound the packs): with t = mant >> (r - 1), OFF =
 * digit_offset and s = 0 or -1 for the sign, Y = X + OFF is
 * ((t ^ s) + 2 OFF + 1) >> 1 for either sign (-floor(a / 2) =
 * floor((1 - a) / 2)), so rounding, negation and offset are one 64-bit
 * addition (a batch's classical problems: 785 -> 739 us of digits in all). Where
 * r - 1 could be negative (down to -7: |x| < 2^E, DB*S > 53) the mantissa is
 * shifted up by 10 first; not by more, so that its top bit stays below bit 63
 * and a shift held at 63 leaves 0. Needs Y and its extra bit inside 64 bits
 * (DB*S <= 60) and no left shift: E >= DB*S - 1074 (lines below that hold
 * subnormal numbers only). */
template <int S, int DB, int N>
__device__ __forceinline__ void split_offsets(const double (&x)[N], int E, Digits (&Y)[N])
{
    constexpr bool kTop = DB * S > 53;
    if (DB * S > 60 || E < DB * S - 1074) {
#pragma unroll
        for (int i = 0; i < N; ++i) Y[i] = split_offset_any<S, DB>(x[i], E);
        return;
    }
    const int K = E + 1075 - DB * S + (kTop ? 10 : 0);   /* r - 1 = K - max(exponent field, 1) */
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const uint32_t hi = (uint32_t)__double2hiint(x[i]);
        const int bexp = (int)(hi >> 20) & 0x7ff;
        uint64_t mant = ((uint64_t)((hi & 0x000fffffu) | ((uint32_t)min(bexp, 1) << 20)) << 32) |
                        (uint32_t)__double2loint(x[i]);
        if (kTop) mant <<= 10;
        const uint64_t t = mant >> min(K - max(bexp, 1), 63);
        const uint64_t neg = (uint64_t)((int64_t)(int32_t)hi >> 31);
        Y[i].X = 0;   /* not needed below 64 digit bits */
        Y[i].Y = (uint64_t)((int64_t)((t ^ neg) + (2 * digit_offset<S, DB>() + 1)) >> 1);
    }
}

/* digit t (0 = most significant) of a BF16 split as an exact float. A lower
 * digit is byte S-1-t of Y minus 128: the byte is placed in the mantissa of
 * 2^23 (one byte permute) and 2^23 + 128 is subtracted, both exact. The top
 * digit goes through the same 2^23-offset conversion from its integer value.
 * With t a compile-time constant after unrolling, the field choice folds away. */
template <int S>
__device__ __forceinline__ float digit_f(const Digits& g, int t)
{
    constexpr int sh = 8 * (S - 1);
    constexpr uint64_t kOff = digit_offset<S, 8>();
    constexpr uint64_t kMask = (1ull << sh) - 1;
    if (t == 0) {
        const int d = S < 8 ? (int)((int64_t)g.Y >> sh)
                            : (int)(g.X >> sh) + (int)((((uint64_t)g.X & kMask) + kOff) >> sh);
        return __int_as_float(0x4B400000 + d) - 12582912.0f;   /* exact for |d| < 2^22 */
    }
    const int fi = S - 1 - t;
    const uint32_t w = fi < 4 ? (uint32_t)g.Y : (uint32_t)(g.Y >> 32);
    return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540u + (unsigned)(fi & 3))) - 8388736.0f;
}

/* two floats that are exact in BF16 (at most 8 significant bits) as a packed
 * bf16x2 word, first value in the low half: their upper 16 bits */
__device__ __forceinline__ uint32_t pack_bf16x2_exact(float lo, float hi)
{
    return __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632u);
}

/* the FP8-E4M3 pair of the FP16 pair h - base, exact for integers of magnitude <= 16 */
__device__ __forceinline__ uint32_t e4m3x2_of(uint32_t h, uint32_t base)
{
    unsigned short r;
    asm("{\n\t.reg .b32 d;\n\tsub.rn.f16x2 d, %1, %2;\n\tcvt.rn.satfinite.e4m3x2.f16x2 %0, d;\n\t}"
        : "=h"(r) : "r"(h), "r"(base));
    return (uint32_t)r;
}

/* FP8 digits of N elements, put(slice, words of four elements each). A 5-bit
 * field f of Y becomes f - 16 in E4M3 through FP16 pairs of two elements: f in
 * the mantissa of 1024 (bits 0..4) or, without a shift, of 32 (bits 5..9), the
 * offset subtracted, both exact. Three fields of two elements travel in one
 * word. Bound by the integer pipe (shifts, masks, conversions), of which this
 * takes two thirds of one FP32 number per field: packs of 322 x1 at 4097 x 3001
 * x 5000, 10 slices, 214 and 248 -> 196 and 219 us. */
template <int S, int N, class Put>
__device__ __forceinline__ void fp8_digits(const Digits (&Y)[N], Put put)
{
    uint32_t p[N / 2], w[N / 4];
    auto emit = [&](int tt, uint32_t mask, uint32_t one, uint32_t base) {
#pragma unroll
        for (int q = 0; q < N / 4; ++q)
            w[q] = e4m3x2_of((p[2 * q] & mask) | one, base) | (e4m3x2_of((p[2 * q + 1] & mask) | one, base) << 16);
        put(tt, w);
    };
    /* the top digit in [-16, 16]: as the bits of the FP16 number 1040 + d */
#pragma unroll
    for (int x = 0; x < N / 2; ++x)
        p[x] = __byte_perm((uint32_t)((int64_t)Y[2 * x].Y >> (5 * (S - 1))) + 0x6410u,
                           (uint32_t)((int64_t)Y[2 * x + 1].Y >> (5 * (S - 1))) + 0x6410u, 0x5410u);
    emit(0, 0xffffffffu, 0u, 0x64106410u);
#pragma unroll
    for (int f = 0; f < S - 1; f += 3) {
#pragma unroll
        for (int x = 0; x < N / 2; ++x)
            p[x] = __byte_perm((uint32_t)(Y[2 * x].Y >> (5 * f)), (uint32_t)(Y[2 * x + 1].Y >> (5 * f)), 0x5410u);
        emit(S - 1 - f, 0x001f001fu, 0x64006400u, 0x64106410u);                       /* 1024 + f - 1040 */
        if (f + 1 < S - 1) emit(S - 2 - f, 0x03e003e0u, 0x50005000u, 0x52005200u);    /* 32 + f - 48 */
        if (f + 2 < S - 1) {
#pragma unroll
            for (int x = 0; x < N / 2; ++x) p[x] >>= 5;
            emit(S - 3 - f, 0x03e003e0u, 0x50005000u, 0x52005200u);
        }
    }
}

/* Writes the S digit slices of 8 consecutive k elements: slice tt of the
 * element at (slice-0) element offset off lands at off + tt * slice_stride
 * of a BF16 (DB = 8, 16 bytes per slice) or FP8-E4M3 (DB = 5, 8 bytes per
 * slice) array. */
template <int S, int DB>
__device__ __forceinline__ void store_digits8(uint8_t* __restrict__ base, int64_t off, int64_t slice_stride,
                                              const Digits (&Y)[8])
{
    if constexpr (DB == 8) {
#pragma unroll
        for (int tt = 0; tt < S; ++tt) {
            uint32_t w[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) w[h] = pack_bf16x2_exact(digit_f<S>(Y[2 * h], tt), digit_f<S>(Y[2 * h + 1], tt));
            *(uint4*)(base + 2 * (off + (int64_t)tt * slice_stride)) = make_uint4(w[0], w[1], w[2], w[3]);
        }
    } else {
        fp8_digits<S>(Y, [&](int tt, const uint32_t (&w)[2]) {
            *(uint2*)(base + off + (int64_t)tt * slice_stride) = make_uint2(w[0], w[1]);
        });
    }
}

/* store_digits8 for 4 consecutive k elements (8 or 4 bytes per slice) */
template <int S, int DB>
__device__ __forceinline__ void store_digits4(uint8_t* __restrict__ base, int64_t off, int64_t slice_stride,
                                              const Digits (&Y)[4])
{
    if constexpr (DB == 8) {
#pragma unroll
        for (int tt = 0; tt < S; ++tt) {
            uint32_t w[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) w[h] = pack_bf16x2_exact(digit_f<S>(Y[2 * h], tt), digit_f<S>(Y[2 * h + 1], tt));
            *(uint2*)(base + 2 * (off + (int64_t)tt * slice_stride)) = make_uint2(w[0], w[1]);
        }
    } else {
        fp8_digits<S>(Y, [&](int tt, const uint32_t (&w)[1]) {
            *(uint32_t*)(base + off + (int64_t)tt * slice_stride) = w[0];
        });
    }
}

/* v * 2^e, in at most two exact power-of-two multiplications. */
__device__ __forceinline__ double scale2(double v, int e)
{
    if (e > 1000) {
        v *= __longlong_as_double((long long)(1000 + 1023) << 52);
        e -= 1000;
    } else if (e < -1000) {
        v *= __longlong_as_double((long long)(-1000 + 1023) << 52);
        e += 1000;
    }
    return v * __longlong_as_double((long long)(e + 1023) << 52);
}

/* ------------------------------------------------- table access -------- */

struct Tab {
    int mt, kt, nt, R;
    const int* u_off; const int* v_off; const int* w_off;
    const int* u_ent; const int* v_ent; const int* w_ent;
    const int* wp_off; const int* wp_ent;
};

__host__ __device__ __forceinline__ Tab tab_view(const int* tab)
{
    Tab t;
    t.mt = tab[0]; t.kt = tab[1]; t.nt = tab[2]; t.R = tab[3];
    t.u_off = tab + FMM_ALG_HDR;
    t.v_off = t.u_off + (t.R + 1);
    t.w_off = t.v_off + (t.R + 1);
    t.u_ent = t.w_off + (t.R + 1);
    t.v_ent = t.u_ent + 2 * t.u_off[t.R];
    t.w_ent = t.v_ent + 2 * t.v_off[t.R];
    t.wp_off = t.w_ent + 2 * t.w_off[t.R];
    t.wp_ent = t.wp_off + (t.mt * t.nt + 1);
    return t;
}

/* ----------------------------------------------------- max kernels ----- */

/* amax[b*m + i] = max over the columns of k-block b of |A[i, :]| (as the bit
 * pattern of a non-negative double, which orders like the value). */
__device__ __forceinline__ void amax_body(const double* __restrict__ A, int64_t lda, int64_t m, int64_t k, int kt,
                                          unsigned long long* __restrict__ amax, int cols_per_block, int64_t bx,
                                          int by, int64_t bz, int64_t i_first = 0, int64_t i_end = -1)
{
    const int64_t i = i_first + bx * (int64_t)blockDim.x + threadIdx.x;
    const int b = by;
    if (i >= (i_end < 0 ? m : i_end)) return;
    int64_t co, cl;
    fmm_part_geom(k, kt, b, &co, &cl);
    const int64_t c0 = bz * cols_per_block;
    if (c0 >= cl) return;
    const int64_t c1 = cl < c0 + cols_per_block ? cl : c0 + cols_per_block;
    const double* col = A + i + (co + c0) * lda;
    const int nc = (int)(c1 - c0);
    unsigned long long mx = 0;
    int c = 0;
    for (; c + 8 <= nc; c += 8) {   /* eight independent loads in flight */
        unsigned long long v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
            v[u] = (unsigned long long)__double_as_longlong(__ldg(col + (int64_t)(c + u) * lda)) &
                   0x7fffffffffffffffull;
#pragma unroll
        for (int u = 0; u < 8; ++u) mx = v[u] > mx ? v[u] : mx;
    }
    for (; c < nc; ++c) {
        const unsigned long long v =
            (unsigned long long)__double_as_longlong(__ldg(col + (int64_t)c * lda)) & 0x7fffffffffffffffull;
        mx = v > mx ? v : mx;
    }
    atomicMax(&amax[(int64_t)b * m + i], mx);
}

/* the rows [i_first, i_end) of A */
__global__ void amax_kernel(const double* __restrict__ A, int64_t lda, int64_t m, int64_t k,
                            int kt, unsigned long long* __restrict__ amax, int cols_per_block, int64_t i_first,
                            int64_t i_end)
{
    amax_body(A, lda, m, k, kt, amax, cols_per_block, blockIdx.x, blockIdx.y, blockIdx.z, i_first, i_end);
}

/* bmax[b*n + j] = max over the rows of k-block b of |B[:, j]| for the columns
 * j in [c0, c1); one warp per (j, b). */
__device__ __forceinline__ void bmax_body(const double* __restrict__ B, int64_t ldb, int64_t k, int64_t n, int kt,
                                          unsigned long long* __restrict__ bmax, int64_t c0, int64_t c1, int64_t bx)
{
    const int64_t w = (bx * (int64_t)blockDim.x + threadIdx.x) / 32;
    const int lane = threadIdx.x % 32;
    const int64_t nc = c1 - c0;
    if (w >= nc * kt) return;
    const int64_t j = c0 + w % nc;
    const int b = (int)(w / nc);
    int64_t ro, rl;
    fmm_part_geom(k, kt, b, &ro, &rl);
    unsigned long long mx = 0;
    for (int64_t p = lane; p < rl; p += 32) {
        const unsigned long long v =
            (unsigned long long)__double_as_longlong(B[ro + p + j * ldb]) & 0x7fffffffffffffffull;
        mx = v > mx ? v : mx;
    }
#pragma unroll
    for (int o = 16; o > 0; o /= 2) {
        const unsigned long long y = __shfl_xor_sync(0xffffffffu, mx, o);
        mx = y > mx ? y : mx;
    }
    if (lane == 0) bmax[(int64_t)b * n + j] = mx;
}

__global__ void bmax_kernel(const double* __restrict__ B, int64_t ldb, int64_t k, int64_t n,
                            int kt, unsigned long long* __restrict__ bmax, int64_t c0, int64_t c1)
{
    bmax_body(B, ldb, k, n, kt, bmax, c0, c1, blockIdx.x);
}

/* Row exponents of S_r (index < m_pad) and column exponents of T_r (index
 * m_pad + j) for the products r = r0 + blockIdx.y of a group, into
 * e_row[q][m_pad] and f_col[q][n_pad]; a launch covers the indices
 * [first, end), so the row side (needs only amax) and the column side (needs
 * only bmax) can run on different streams. */
__device__ __forceinline__ void exps_body(const int* __restrict__ tab, int r0, int64_t m, int64_t n, int64_t k,
                                          int64_t m_pad, int64_t n_pad, const unsigned long long* __restrict__ amax,
                                          const unsigned long long* __restrict__ bmax, int* __restrict__ e_row,
                                          int* __restrict__ f_col, int64_t first, int64_t end, int64_t bx, int by)
{
    const Tab t = tab_view(tab);
    const int r = r0 + by;
    e_row += (int64_t)by * m_pad;
    f_col += (int64_t)by * n_pad;
    const int64_t me = (m + t.mt - 1) / t.mt, ne = (n + t.nt - 1) / t.nt;
    const int64_t idx = first + bx * (int64_t)blockDim.x + threadIdx.x;
    if (idx >= end) return;
    if (idx < m_pad) {
        const int64_t i = idx;
        double bnd = 0.0;
        bool first = true;
        if (i < me) {
            for (int e = t.u_off[r]; e < t.u_off[r + 1]; ++e) {
                const int part = t.u_ent[2 * e];
                const double c = fabs((double)t.u_ent[2 * e + 1]);
                int64_t ro, rl;
                fmm_part_geom(m, t.mt, part / t.kt, &ro, &rl);
                if (i >= rl) continue;
                const double mx = __longlong_as_double((long long)amax[(int64_t)(part % t.kt) * m + ro + i]);
                bnd = first ? c * mx : fma(c, mx, bnd);
                first = false;
            }
        }
        e_row[i] = exp_above(bnd);
    } else if (idx < m_pad + n_pad) {
        const int64_t j = idx - m_pad;
        double bnd = 0.0;
        bool first = true;
        if (j < ne) {
            for (int e = t.v_off[r]; e < t.v_off[r + 1]; ++e) {
                const int part = t.v_ent[2 * e];
                const double c = fabs((double)t.v_ent[2 * e + 1]);
                int64_t co, cl;
                fmm_part_geom(n, t.nt, part % t.nt, &co, &cl);
                if (j >= cl) continue;
                const double mx = __longlong_as_double((long long)bmax[(int64_t)(part / t.nt) * n + co + j]);
                bnd = first ? c * mx : fma(c, mx, bnd);
                first = false;
            }
        }
        f_col[j] = exp_above(bnd);
    }
    (void)k;
}

__global__ void exps_kernel(const int* __restrict__ tab, int r0, int64_t m, int64_t n, int64_t k,
                            int64_t m_pad, int64_t n_pad,
                            const unsigned long long* __restrict__ amax,
                            const unsigned long long* __restrict__ bmax,
                            int* __restrict__ e_row, int* __restrict__ f_col, int64_t first, int64_t end)
{
    exps_body(tab, r0, m, n, k, m_pad, n_pad, amax, bmax, e_row, f_col, first, end, blockIdx.x, blockIdx.y);
}

/* ----------------------------------------------------- pack kernels ---- */

constexpr int kPackMaxEnt = 256;

/* one sub-block term of a packing sum: base pointer, extent, coefficient as
 * a double and its kind (0: +1, 1: -1, 2: other), so the per-element code
 * does no conversion and no FP64 compare */
struct PEnt {
    const double* base;
    double coef;
    int rows, cols;
    int kind;
    int pad;
};

__device__ __forceinline__ PEnt make_pent(const double* base, int64_t rows, int64_t cols, int c)
{
    PEnt x;
    x.base = base;
    x.coef = (double)c;
    x.rows = (int)rows;
    x.cols = (int)cols;
    x.kind = c == 1 ? 0 : (c == -1 ? 1 : 2);
    x.pad = 0;
    return x;
}

/* first term of a packing sum over a thread's values: s[t] = c * s[t],
 * exact like the FP64 product; sign flips for c = +-1 keep it off the FP64
 * pipe, and the branch (uniform over the CTA) is taken once for all values */
template <int N>
__device__ __forceinline__ void scale_first(const PEnt& x, double (&s)[N])
{
    if (x.kind == 1) {
#pragma unroll
        for (int t = 0; t < N; ++t)
            s[t] = __longlong_as_double(__double_as_longlong(s[t]) ^ (long long)0x8000000000000000ull);
    } else if (x.kind == 2) {
#pragma unroll
        for (int t = 0; t < N; ++t) s[t] = x.coef * s[t];
    }
}

/* A side, all products r0 .. r0+np-1 of a group in one launch: CTA (q, tile)
 * forms the tile of ROWS rows x 64 k of S_r, r = r0 + q, and writes its digits
 * row-major (K-major) into slices sa[q][t][m_pad][k_pad]. The product index
 * runs fastest in the block order, so the products at one tile position run
 * together and read their shared A sub-block tiles through L2 once. ROWS = 64
 * (256 threads); ROWS = 32 (128 threads, 25 KB of shared memory, at most 64
 * registers) where the packs run beside a GEMM (split_overlap), small enough
 * for an SM with a resident GEMM CTA. */
template <int S, int DB, int ROWS>
__device__ __forceinline__ void pack_a_body(const int* __restrict__ tab, int r0, int np, const double* __restrict__ A,
                                            int64_t lda, int64_t m, int64_t k, int64_t m_pad, int64_t k_pad,
                                            const int* __restrict__ e_row, uint8_t* __restrict__ sa, int64_t bx,
                                            int64_t by, int64_t i_first = 0)
{
    __shared__ double Sf[64][ROWS + 1];
    __shared__ PEnt ent[kPackMaxEnt];
    const Tab t = tab_view(tab);
    const int64_t me = (m + t.mt - 1) / t.mt, ke = (k + t.kt - 1) / t.kt;
    const int q = (int)(bx % np);
    const int r = r0 + q;
    const int64_t i0 = i_first + (bx / np) * ROWS, p0 = by * 64;
    e_row += (int64_t)q * m_pad;
    const int64_t slice0 = (int64_t)q * S * m_pad * k_pad;   /* element offset of this product */
    const int eb = t.u_off[r], ne_ = t.u_off[r + 1] - eb;
    for (int e = threadIdx.x; e < ne_; e += blockDim.x) {
        const int part = t.u_ent[2 * (eb + e)];
        int64_t ro, rl, co, cl;
        fmm_part_geom(m, t.mt, part / t.kt, &ro, &rl);
        fmm_part_geom(k, t.kt, part % t.kt, &co, &cl);
        ent[e] = make_pent(A + ro + co * lda, rl, cl, t.u_ent[2 * (eb + e) + 1]);
    }
    __syncthreads();
    /* 16 elements per thread in two halves of 8: each term's 8 loads go out
     * together, and the first term's coefficient (uniform over the CTA) is
     * applied once after them */
    const int li = threadIdx.x % ROWS, kq = threadIdx.x / ROWS;   /* row, k offset 0..3 */
    const int64_t gi = i0 + li;
    const bool row_ok = ne_ > 0 && gi < me;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        double v8[8];
#pragma unroll
        for (int y = 0; y < 8; ++y) v8[y] = 0.0;
        if (row_ok) {
            /* term e + 1's loads go out before term e's FMAs; per term, one
             * row test and one k limit, then a pointer step of 4 columns per
             * element (no per-element index arithmetic) */
            const int64_t st4 = 4 * lda;
            auto load8 = [&](const PEnt& x, double (&d)[8]) {
                const bool rok = gi < x.rows;
                const int64_t kl = (ke < x.cols ? ke : x.cols) - (p0 + kq + 32 * h);   /* valid while 4y < kl */
                const double* pt = x.base + gi + (p0 + kq + 32 * h) * lda;
#pragma unroll
                for (int y = 0; y < 8; ++y) {
                    d[y] = (rok && 4 * y < kl) ? __ldg(pt) : 0.0;
                    pt += st4;
                }
            };
            double nx[8];
            load8(ent[0], v8);
            if (ne_ > 1) load8(ent[1], nx);
            scale_first(ent[0], v8);
            for (int e = 1; e < ne_; ++e) {
                double cur[8];
#pragma unroll
                for (int y = 0; y < 8; ++y) cur[y] = nx[y];
                if (e + 1 < ne_) load8(ent[e + 1], nx);
                const double c = ent[e].coef;
#pragma unroll
                for (int y = 0; y < 8; ++y) v8[y] = fma(c, cur[y], v8[y]);
            }
        }
#pragma unroll
        for (int y = 0; y < 8; ++y) Sf[kq + 4 * (8 * h + y)][li] = v8[y];
    }
    __syncthreads();
    /* thread -> (row, 8 consecutive k): 4 rows x 128 bytes per warp store */
    const int kg = threadIdx.x % 8;
    for (int rr = threadIdx.x / 8; rr < ROWS; rr += ROWS / 2) {
        const int64_t gi = i0 + rr;
        const int E = e_row[gi];
        double x8[8];
#pragma unroll
        for (int x = 0; x < 8; ++x) x8[x] = Sf[kg * 8 + x][rr];
        Digits Y[8];
        split_offsets<S, DB>(x8, E, Y);
        store_digits8<S, DB>(sa, slice0 + gi * k_pad + p0 + kg * 8, m_pad * k_pad, Y);
    }
}

template <int S, int DB, int ROWS>
__global__ void __launch_bounds__(ROWS * 4, ROWS == 64 ? 4 : 8)
pack_a_kernel(const int* __restrict__ tab, int r0, int np, const double* __restrict__ A, int64_t lda,
              int64_t m, int64_t k, int64_t m_pad, int64_t k_pad,
              const int* __restrict__ e_row, uint8_t* __restrict__ sa, int64_t i_first)
{
    pack_a_body<S, DB, ROWS>(tab, r0, np, A, lda, m, k, m_pad, k_pad, e_row, sa, blockIdx.x, blockIdx.y, i_first);
}

/* B side, all products of a group: CTA (q, tile) forms the tile of COLS
 * columns x 64 k of T_r, r = r0 + q (column j of T_r is contiguous in k
 * already), and writes its digits into slices sb[q][t][n_pad][k_pad];
 * product index fastest, as on the A side. COLS = 32 (256 threads), or 16
 * (128 threads, at most 64 registers) beside a GEMM. Eight lanes
 * read 64 contiguous bytes of a column per load (a load that gives each lane
 * eight consecutive k touches 16 lines and is bound by L1) and exchange the
 * sums through shared memory: 222 x2 at 4096, 6 slices, 339 -> 277 us. */
template <int S, int DB, int COLS>
__device__ __forceinline__ void pack_b_body(const int* __restrict__ tab, int r0, int np, const double* __restrict__ B,
                                            int64_t ldb, int64_t k, int64_t n, int64_t n_pad, int64_t k_pad,
                                            const int* __restrict__ f_col, uint8_t* __restrict__ sb, int64_t j_first,
                                            int64_t bx, int64_t by)
{
    __shared__ PEnt ent[kPackMaxEnt];
    __shared__ double Tf[COLS][72];   /* element k at k + k / 8: no bank conflicts either way */
    const Tab t = tab_view(tab);
    const int64_t ne = (n + t.nt - 1) / t.nt, ke = (k + t.kt - 1) / t.kt;
    const int q = (int)(bx % np);
    const int r = r0 + q;
    f_col += (int64_t)q * n_pad;
    const int64_t slice0 = (int64_t)q * S * n_pad * k_pad;
    const int eb = t.v_off[r], ne_ = t.v_off[r + 1] - eb;
    for (int e = threadIdx.x; e < ne_; e += blockDim.x) {
        const int part = t.v_ent[2 * (eb + e)];
        int64_t ro, rl, co, cl;
        fmm_part_geom(k, t.kt, part / t.nt, &ro, &rl);
        fmm_part_geom(n, t.nt, part % t.nt, &co, &cl);
        ent[e] = make_pent(B + ro + co * ldb, rl, cl, t.v_ent[2 * (eb + e) + 1]);
    }
    __syncthreads();
    const int kg = threadIdx.x % 8;
    const int64_t gj = j_first + (bx / np) * COLS + threadIdx.x / 8;
    const int64_t p0 = by * 64;
    double v8[8];   /* k = p0 + kg + 8 y: a column's eight lanes read 64 bytes side by side */
#pragma unroll
    for (int x = 0; x < 8; ++x) v8[x] = 0.0;
    if (ne_ > 0 && gj < ne) {
        /* term e + 1's loads go out before term e's FMAs; per term, one
         * column test and one k limit, then 8 values at fixed offsets from
         * one pointer */
        auto load8 = [&](const PEnt& x, double (&d)[8]) {
            const int64_t kl = (ke < x.rows ? ke : x.rows) - (p0 + kg);   /* valid while 8y < kl */
            const bool cok = gj < x.cols;
            const double* pt = x.base + gj * ldb + p0 + kg;
#pragma unroll
            for (int y = 0; y < 8; ++y) d[y] = (cok && 8 * y < kl) ? __ldg(pt + 8 * y) : 0.0;
        };
        double nx[8];
        load8(ent[0], v8);
        if (ne_ > 1) load8(ent[1], nx);
        scale_first(ent[0], v8);
        for (int e = 1; e < ne_; ++e) {
            double cur[8];
#pragma unroll
            for (int y = 0; y < 8; ++y) cur[y] = nx[y];
            if (e + 1 < ne_) load8(ent[e + 1], nx);
            const double c = ent[e].coef;
#pragma unroll
            for (int y = 0; y < 8; ++y) v8[y] = fma(c, cur[y], v8[y]);
        }
    }
    /* to eight consecutive k per lane, within the column's lanes */
    double* mine = Tf[threadIdx.x / 8];
#pragma unroll
    for (int y = 0; y < 8; ++y) mine[kg + 9 * y] = v8[y];
    __syncwarp();
#pragma unroll
    for (int x = 0; x < 8; ++x) v8[x] = mine[9 * kg + x];
    const int F = f_col[gj];
    Digits Y[8];
    split_offsets<S, DB>(v8, F, Y);
    store_digits8<S, DB>(sb, slice0 + gj * k_pad + p0 + kg * 8, n_pad * k_pad, Y);
}

template <int S, int DB, int COLS>
__global__ void __launch_bounds__(COLS * 8, COLS == 32 ? 4 : 8)
pack_b_kernel(const int* __restrict__ tab, int r0, int np, const double* __restrict__ B, int64_t ldb,
              int64_t k, int64_t n, int64_t n_pad, int64_t k_pad,
              const int* __restrict__ f_col, uint8_t* __restrict__ sb, int64_t j_first)
{
    pack_b_body<S, DB, COLS>(tab, r0, np, B, ldb, k, n, n_pad, k_pad, f_col, sb, j_first, blockIdx.x, blockIdx.y);
}

/* a call of f(integral_constant S, integral_constant DB) for a slice count and format */
template <class F>
auto with_slices(int fmt, int s, F f)
{
#define FMM_CASE(S_, DB_) return f(std::integral_constant<int, S_>(), std::integral_constant<int, DB_>())
    if (fmt == 0) {
        switch (s) {
        case 2: FMM_CASE(2, 8);
        case 3: FMM_CASE(3, 8);
        case 4: FMM_CASE(4, 8);
        case 5: FMM_CASE(5, 8);
        case 6: FMM_CASE(6, 8);
        case 7: FMM_CASE(7, 8);
        default: FMM_CASE(8, 8);
        }
    }
    switch (s) {
    case 2: FMM_CASE(2, 5);
    case 3: FMM_CASE(3, 5);
    case 4: FMM_CASE(4, 5);
    case 5: FMM_CASE(5, 5);
    case 6: FMM_CASE(6, 5);
    case 7: FMM_CASE(7, 5);
    case 8: FMM_CASE(8, 5);
    case 9: FMM_CASE(9, 5);
    case 10: FMM_CASE(10, 5);
    case 11: FMM_CASE(11, 5);
    default: FMM_CASE(12, 5);
    }
#undef FMM_CASE
}

/* Which packs a launch_packs call issues: both sides, or one side only; the
 * A side over the S_r rows [ia0, ia1) (multiples of 64, or ia1 = m_pad), the
 * B side over the T_r columns [jb0, jb1) (multiples of 32, or jb1 = n_pad). */
struct PackSel {
    bool a = true, b = true;
    int64_t ia0 = 0, ia1 = -1;
    int64_t jb0 = 0, jb1 = -1;
    bool small = false;   /* the 128-thread tiles that fit beside a resident GEMM CTA */
};

template <int S, int DB>
void launch_packs_t(const int* tab, int r, int np, const double* A, int64_t lda, const double* B, int64_t ldb,
                    int64_t m, int64_t n, int64_t k, int64_t m_pad, int64_t n_pad, int64_t k_pad,
                    const int* e_row, const int* f_col, uint8_t* sa, uint8_t* sb, cudaStream_t st,
                    cudaStream_t st_b, const PackSel& sel)
{
    const int64_t i1 = sel.ia1 < 0 ? m_pad : sel.ia1;
    const int rows = sel.small ? 32 : 64;
    const dim3 ka((unsigned)(np * ((i1 - sel.ia0 + rows - 1) / rows)), (unsigned)(k_pad / 64));
    if (sel.a && i1 > sel.ia0 && sel.small)
        pack_a_kernel<S, DB, 32><<<ka, 128, 0, st>>>(tab, r, np, A, lda, m, k, m_pad, k_pad, e_row, sa, sel.ia0);
    else if (sel.a && i1 > sel.ia0)
        pack_a_kernel<S, DB, 64><<<ka, 256, 0, st>>>(tab, r, np, A, lda, m, k, m_pad, k_pad, e_row, sa, sel.ia0);
    const int64_t j1 = sel.jb1 < 0 ? n_pad : sel.jb1;
    if (!sel.b || j1 <= sel.jb0) return;
    const int cols = sel.small ? 16 : 32;
    const dim3 kb((unsigned)(np * ((j1 - sel.jb0 + cols - 1) / cols)), (unsigned)(k_pad / 64));
    if (sel.small)
        pack_b_kernel<S, DB, 16><<<kb, 128, 0, st_b>>>(tab, r, np, B, ldb, k, n, n_pad, k_pad, f_col, sb, sel.jb0);
    else
        pack_b_kernel<S, DB, 32><<<kb, 256, 0, st_b>>>(tab, r, np, B, ldb, k, n, n_pad, k_pad, f_col, sb, sel.jb0);
}

/* digit slices of the products r .. r+np-1 (exponents already in place);
 * fmt 0: BF16 (s = 2..8), fmt 1: FP8-E4M3 (s = 2..12); the B side on st_b */
void launch_packs(int fmt, int s, const int* tab, int r, int np, const double* A, int64_t lda, const double* B,
                  int64_t ldb, int64_t m, int64_t n, int64_t k, int64_t m_pad, int64_t n_pad,
                  int64_t k_pad, const int* e_row, const int* f_col, uint8_t* sa, uint8_t* sb,
                  cudaStream_t st, cudaStream_t st_b, const PackSel& sel = PackSel())
{
    with_slices(fmt, s, [&](auto S, auto DB) {
        launch_packs_t<S(), DB()>(tab, r, np, A, lda, B, ldb, m, n, k, m_pad, n_pad, k_pad, e_row, f_col, sa, sb, st,
                                  st_b, sel);
    });
}

/* ------------------------------- classical: maxima, exponents, digits ---- */

/* The classical GEMM's whole operand side in one launch: a cluster of CTAs
 * owns 16 rows of A (or 16 columns of B), each CTA a k chunk. Every CTA takes
 * its chunk's maxima, the cluster combines them through distributed shared
 * memory, and the CTA reads its chunk again (from L2 mostly) and splits the
 * digits. The same exponents and digits as the general path's maxima,
 * exponents and packs (one term of coefficient 1), which takes seven launches.
 * Bound by latency (loads in flight) and instruction issue: 8192 x 8192 of both
 * operands, 6 slices, 560 us (4.8 TB/s of the 2.7 GB it cannot do without);
 * 575 us with split_offset_any, 690 us with 64-bit maxima as well, 680 us
 * through cp.async tiles. */
constexpr int kPrepLines = 16, kPrepK = 128, kPrepThreads = 256;
constexpr int kPrepPitch = kPrepK + kPrepK / 16 + 1;   /* one pad per 16 k, odd row pitch: no bank conflicts either way */

struct PrepShared {
    double tile[2][kPrepLines * kPrepPitch];
    uint2 part[kPrepThreads / kPrepLines][kPrepLines];   /* (OR of low words, maximum of high words) */
    uint2 mx[kPrepLines];                                /* this CTA's, read by the cluster */
};

/* lines [l0, l0 + 16) of A (rows) or B (columns), k chunk `rank` of `nrank` */
template <int S, int DB, bool A_SIDE>
__device__ __forceinline__ void prep_body(PrepShared& sh, const double* __restrict__ X, int64_t ld, int64_t lines,
                                          int64_t k, int64_t l_pad, int64_t k_pad, int* __restrict__ ex,
                                          uint8_t* __restrict__ out, int64_t l0, int rank, int nrank)
{
    namespace cgr = cooperative_groups;
    const int tid = threadIdx.x;
    const int64_t chunk = ((k_pad + nrank - 1) / nrank + kPrepK - 1) / kPrepK * kPrepK;
    const int64_t p0 = rank * chunk, p1 = p0 + chunk < k_pad ? p0 + chunk : k_pad;
    const int64_t pe = p1 < k ? p1 : k;   /* the chunk's k with data */
    const int tiles = p1 > p0 ? (int)((p1 - p0 + kPrepK - 1) / kPrepK) : 0;
    /* a thread's eight elements of a 16 x 128 tile, lanes along the operand's
     * contiguous direction: A one line, every 16th k; B one k, every 2nd line */
    const int line = A_SIDE ? tid % kPrepLines : tid / kPrepK;
    const int kq = A_SIDE ? tid / kPrepLines : tid % kPrepK;
    const int lines_left = (int)(lines - l0 < kPrepLines ? lines - l0 : kPrepLines) - line;
    const double* x0 = A_SIDE ? X + (l0 + line) + (p0 + kq) * ld : X + (p0 + kq) + (l0 + line) * ld;
    const int64_t ystep = (A_SIDE ? 16 : 2) * ld, tstep = A_SIDE ? kPrepK * ld : kPrepK;
    const int k_left = pe > p0 ? (int)(pe - p0) - kq : -kq;   /* this thread's k from the chunk's start */
    auto load = [&](int t, double (&v)[8]) {                  /* tile t of the chunk */
        const double* q = x0 + t * tstep;
        const int kl = k_left - t * kPrepK;
        const int lim = A_SIDE ? (lines_left > 0 ? kl : 0) : (kl > 0 ? lines_left : 0);
#pragma unroll
        for (int y = 0; y < 8; ++y) v[y] = (A_SIDE ? 16 : 2) * y < lim ? __ldg(q + y * ystep) : 0.0;
    };
    /* What the exponent needs of a line's largest |x|: its high word, and where
     * that is 0 (below 2^-1042) the leading bit of the low words. A side: one
     * line per thread, B side: eight. */
    constexpr int NL = A_SIDE ? 1 : 8;
    uint32_t mh[NL], ml[NL];
#pragma unroll
    for (int y = 0; y < NL; ++y) mh[y] = ml[y] = 0;
    auto take = [&](const double (&v)[8]) {
#pragma unroll
        for (int y = 0; y < 8; ++y) {
            const int z = A_SIDE ? 0 : y;
            mh[z] = max(mh[z], (uint32_t)__double2hiint(v[y]) & 0x7fffffffu);
            ml[z] |= (uint32_t)__double2loint(v[y]);
        }
    };
    double v[8];
    {
        double w[8];
        for (int t = 0; t < tiles; t += 2) {   /* sixteen loads in flight */
            load(t, v);
            load(t + 1, w);
            take(v);
            take(w);
        }
    }
    if (A_SIDE) {
        sh.part[tid / kPrepLines][tid % kPrepLines] = make_uint2(ml[0], mh[0]);
    } else {
#pragma unroll
        for (int y = 0; y < NL; ++y) {
            const uint32_t h = __reduce_max_sync(0xffffffffu, mh[y]), l = __reduce_or_sync(0xffffffffu, ml[y]);
            /* line = tid / 128 + 2 y; the four warps of a line each leave one maximum */
            if (tid % 32 == 0) sh.part[tid / 32 % 4][line + 2 * y] = make_uint2(l, h);
        }
    }
    __syncthreads();
    if (tid < kPrepLines) {
        uint2 m = make_uint2(0, 0);
        for (int q = 0; q < (A_SIDE ? kPrepThreads / kPrepLines : 4); ++q) {
            m.x |= sh.part[q][tid].x;
            m.y = max(m.y, sh.part[q][tid].y);
        }
        sh.mx[tid] = m;
    }
    if (nrank > 1) {
        cgr::cluster_group cl = cgr::this_cluster();
        cl.sync();
        uint2 m = make_uint2(0, 0);
        if (tid < kPrepLines)
            for (int q = 0; q < nrank; ++q) {
                const uint2 z = *cl.map_shared_rank(&sh.mx[tid], q);
                m.x |= z.x;
                m.y = max(m.y, z.y);
            }
        cl.sync();   /* every CTA has read the others' maxima */
        if (tid < kPrepLines) sh.mx[tid] = m;
    }
    if (tiles > 0) load(0, v);
    __syncthreads();
    /* exponent of the line's maximum (exp_above: normal numbers by the exponent
     * field, subnormal ones by the leading bit) */
    auto exponent = [&](int x) {
        const uint2 m = sh.mx[x];
        return exp_above(__hiloint2double((int)m.y, (int)(m.y ? 0u : m.x)));
    };
    if (rank == 0 && tid < kPrepLines) ex[l0 + tid] = exponent(tid);
    /* digits: a warp takes lines w and w + 8, four consecutive k per lane:
     * 256-byte stores per line and slice */
    const int rl = tid / 32, k4 = tid % 32 * 4;
    const int E0 = exponent(rl), E1 = exponent(rl + 8);
    const int64_t off = (l0 + rl) * k_pad + p0 + k4;
    const int pos = rl * kPrepPitch + k4 + k4 / 16;
    for (int t = 0; t < tiles; ++t) {
        double* tile = sh.tile[t & 1];   /* the other one may still be read */
#pragma unroll
        for (int y = 0; y < 8; ++y) {
            const int li = A_SIDE ? line : line + 2 * y, kk = A_SIDE ? kq + 16 * y : kq;
            tile[li * kPrepPitch + kk + kk / 16] = v[y];
        }
        __syncthreads();
        if (t + 1 < tiles) load(t + 1, v);   /* in flight under this tile's digits */
        if (p0 + t * kPrepK + k4 < p1) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                double x4[4];
#pragma unroll
                for (int x = 0; x < 4; ++x) x4[x] = tile[pos + h * 8 * kPrepPitch + x];
                Digits Y[4];
                split_offsets<S, DB>(x4, h ? E1 : E0, Y);
                store_digits4<S, DB>(out, off + h * 8 * k_pad + (int64_t)t * kPrepK, l_pad * k_pad, Y);
            }
        }
    }
}

template <int S, int DB>
__global__ void __launch_bounds__(kPrepThreads, 3)   /* four per SM would spill */
prep_kernel(const double* __restrict__ A, int64_t lda, const double* __restrict__ B, int64_t ldb, int64_t m,
            int64_t n, int64_t k, int64_t m_pad, int64_t n_pad, int64_t k_pad, int* __restrict__ e_row,
            int* __restrict__ f_col, uint8_t* __restrict__ sa, uint8_t* __restrict__ sb,
            unsigned int* __restrict__ sched, int nrank)
{
    __shared__ PrepShared sh;
    sm103::grid_launch_dependents();
    const int64_t c = blockIdx.x / (unsigned)nrank, ca = m_pad / kPrepLines;
    const int rank = (int)(blockIdx.x % (unsigned)nrank);
    if (blockIdx.x == 0 && threadIdx.x == 0) *sched = 0;   /* the GEMM's work-item counter */
    if (c < ca)
        prep_body<S, DB, true>(sh, A, lda, m, k, m_pad, k_pad, e_row, sa, c * kPrepLines, rank, nrank);
    else
        prep_body<S, DB, false>(sh, B, ldb, n, k, n_pad, k_pad, f_col, sb, (c - ca) * kPrepLines, rank, nrank);
}

/* ------------------------------------------------------ GEMM kernel ---- */

/* (double)z * 2^e for |z| < 2^62 in integer arithmetic (round to nearest
 * even, then exponent offset), identical to the FP64 conversion and
 * power-of-two scaling whenever the result is a normal number; other cases
 * take the FP64 route. Keeps the per-element FP64 work to the C updates. */
/* the FP64 route for results outside the normal range, kept out of line so
 * the common path carries no FP64 instruction */
__device__ __noinline__ double i64_to_double_scaled_slow(int64_t z, int e)
{
    return scale2((double)z, e);
}

__device__ __forceinline__ double i64_to_double_scaled(int64_t z, int e)
{
    if (z == 0) return 0.0;
    const uint64_t sign = z < 0 ? 0x8000000000000000ull : 0ull;
    uint64_t u = z < 0 ? (uint64_t)(-z) : (uint64_t)z;
    int p = 63 - __clzll((long long)u);
    uint64_t m;
    if (p <= 52) {
        m = u << (52 - p);
    } else {
        const int sh = p - 52;
        m = u >> sh;
        const uint64_t rem = u & ((1ull << sh) - 1), half = 1ull << (sh - 1);
        if (rem > half || (rem == half && (m & 1))) {
            ++m;
            if (m == (1ull << 53)) { m >>= 1; ++p; }
        }
    }
    const int be = p + 1023 + e;
    if (be < 1 || be > 2046) return i64_to_double_scaled_slow(z, e);
    return __longlong_as_double((long long)(sign | ((uint64_t)be << 52) | (m & 0x000fffffffffffffull)));
}

/* One problem of a GEMM launch: the digit slices of a product group of one
 * FMM GEMM and where its level accumulators go. */
struct GemmProblem {
    CUtensorMap tmA;      /* A slices [product][s][m_pad][k_pad], box 64 x 128 */
    CUtensorMap tmB;      /* B slices [product][s][n_pad][k_pad], box 64 x 256 */
    uint8_t* Z;           /* [product] Z planes (ZPlanes) */
    int s;                /* slices */
    int zlevel;           /* G: the level whose unit Z counts in */
    int zmin;             /* lowest level with a digit plane (ZPlanes) */
    int znd;              /* digit planes */
    int zrow0;            /* first Z row of the launch's tile row 0 */
    int nunits, unit_kb;  /* work units per tile, k blocks per unit at most; nunits 0: whole tiles (UnitSpan) */
    int nkb;              /* k_pad / kbe */
    int kbe;              /* k elements per 128-byte stage row: 64 (BF16) or 128 (FP8) */
    int db;               /* digit bits: 8 (BF16) or 5 (FP8-E4M3) */
    int fmt;              /* 0: BF16 slices, kind::f16; 1: FP8-E4M3 slices, kind::f8f6f4 */
    int m_pad, n_pad;     /* rows per slice in the A / B slice arrays */
    int tiles_m, tiles_n; /* per product */
    int item_begin;       /* first work item of this problem in the launch */
};

/* problems per GEMM launch: the table travels as a kernel parameter, whose
 * space is 32764 bytes (a GemmProblem is 384 bytes with its two 128-byte
 * aligned tensor maps) */
constexpr int kMaxLaunchProblems = 80;

/* Everything a launch needs, passed by value (tensor maps included), so a
 * launch copies nothing to the device and can be captured in a graph. Single
 * calls launch kernels of their own with room for one problem: 32 KB of
 * parameters cost a launch several microseconds. */
template <int N>
struct GemmLaunchOf {
    int nprob;
    int nitems;           /* sum over problems of products * tiles */
    int* err;
    unsigned int* sched;  /* next work item, zero at launch */
    GemmProblem prob[N];
};
using GemmLaunch = GemmLaunchOf<kMaxLaunchProblems>;
using GemmLaunch1 = GemmLaunchOf<1>;
static_assert(sizeof(GemmLaunch) <= 32764, "GemmLaunch must fit the kernel parameter space");

__host__ __device__ __forceinline__ int level_pairs(int g, int s)
{
    return (g - 1 < s ? g - 1 : s) - (g - s > 1 ? g - s : 1) + 1;
}

/* A tile's k blocks of all slice pairs as work units, for a product grid too
 * small to give every SM a tile: a unit is part of one level, its k blocks
 * [q0, q1) in the producer's order, at most unit_kb of them. Each unit leaves
 * its sums as one int32 plane ([n_pad/4][m_pad] int4, below); the C
 * update adds a level's planes (an exact integer sum) before it rounds and
 * combines the levels, so Z is the same value. */
struct UnitSpan {
    int g, q0, q1;
};

__host__ __device__ __forceinline__ int level_units(int g, int s, int nkb, int unit_kb)
{
    return (level_pairs(g, s) * nkb + unit_kb - 1) / unit_kb;
}

__host__ __device__ __forceinline__ UnitSpan unit_span(int s, int nkb, int unit_kb, int u)
{
    for (int g = s + 1; g > 2; --g) {
        const int cnt = level_units(g, s, nkb, unit_kb);
        if (u < cnt) {
            const int lk = level_pairs(g, s) * nkb, len = (lk + cnt - 1) / cnt;
            return UnitSpan{g, u * len, u * len + len < lk ? u * len + len : lk};
        }
        u -= cnt;
    }
    const int cnt = level_units(2, s, nkb, unit_kb), len = (nkb + cnt - 1) / cnt;
    return UnitSpan{2, u * len, u * len + len < nkb ? u * len + len : nkb};
}

/* the k blocks [q0, q1) of level g that an item runs: all of every level, or its unit's */
__device__ __forceinline__ UnitSpan level_span(const GemmProblem& P, const UnitSpan& u, int g)
{
    return P.nunits ? u : UnitSpan{g, 0, level_pairs(g, P.s) * P.nkb};
}

/* Work item b -> problem, product and tile: problems in order, products in
 * order within a problem, then a grouped raster of kRasterGroup tile rows so
 * the CTAs resident together share slice panels in L2. */
struct Item {
    int p, r, tile_m, tile_n, unit;
};

template <class GL>
__device__ __forceinline__ Item decode_item(const GL& L, int b, int raster = kRasterGroup)
{
    int p = 0, hi = L.nprob - 1;        /* last problem with item_begin <= b */
    while (p < hi) {
        const int mid = (p + hi + 1) / 2;
        if (L.prob[mid].item_begin <= b) p = mid; else hi = mid - 1;
    }
    const GemmProblem& P = L.prob[p];
    const int local = b - P.item_begin;
    const int per_prod = P.tiles_m * P.tiles_n;
    Item it;
    it.p = p;
    it.r = local / per_prod;
    it.unit = 0;
    if (P.nunits) {   /* one product: the tiles of unit 0, then of unit 1, ... */
        it.unit = it.r;
        it.r = 0;
    }
    const int id = local % per_prod;
    const int per_group = raster * P.tiles_n;
    const int grp = id / per_group, first_m = grp * raster;
    const int gm = min(P.tiles_m - first_m, raster);
    const int in_grp = id % per_group;
    it.tile_m = first_m + in_grp % gm;
    it.tile_n = in_grp / gm;
    return it;
}

constexpr int kSchedSlots = 4;
/* readers of each ring slot: the even CTA's MMA thread, every epilogue warp of
 * both CTAs, the odd CTA's producer */
constexpr int kSchedConsumers = 1 + 2 * kEpiWarps + 1;

/* Consumer side of the pair kernel's work-item ring: the even CTA's producer
 * takes items from a global counter and writes each into slot `slot` of both
 * CTAs' rings; a consumer waits for the slot, reads it and reports it read on
 * the even CTA's sempty barrier (release at cluster scope: the read is done
 * before the slot can be written again). */
struct ItemRing {
    uint32_t base;   /* shared-memory address of sfull[0]; sempty and sitem follow */
    int slot;
    uint32_t ph;

    __device__ __forceinline__ uint32_t full_at() const { return base + 8u * (uint32_t)slot; }
    __device__ __forceinline__ uint32_t empty_at() const { return base + 8u * (uint32_t)(kSchedSlots + slot); }
    __device__ __forceinline__ uint32_t item_at() const { return base + 16u * kSchedSlots + 4u * (uint32_t)slot; }
    __device__ __forceinline__ void next()
    {
        if (++slot == kSchedSlots) { slot = 0; ph ^= 1; }
    }
    __device__ __forceinline__ bool take(int* b, volatile int* abort_flag, int* err, int code)
    {
        if (!sm103::mbar_wait_acq_cluster_u32(full_at(), ph, abort_flag, err, code)) return false;
        *b = (int)sm103::ld_shared_u32(item_at());
        sm103::mbar_arrive_release_cluster(sm103::mapa(empty_at(), 0));
        next();
        return true;
    }
    /* lane 0 of a warp takes the slot and hands the item to the other lanes */
    __device__ __forceinline__ bool take_warp(int* b, int lane, volatile int* abort_flag, int* err, int code)
    {
        int got = 0, v = 0;
        if (lane == 0) {
            got = take(&v, abort_flag, err, code) ? 1 : 0;
        } else {
            next();
        }
        got = __shfl_sync(0xffffffffu, got, 0);
        *b = __shfl_sync(0xffffffffu, v, 0);
        return got != 0;
    }
};

/* How Z = sum_{g<=G} L_g 2^(db(G-g)) + sum_{g>G} round(L_g / 2^(db(g-G))) is
 * stored: the GEMM runs the levels from the least significant one down to
 * g = 2, and at the end of a level g <= G its low db bits are final (every
 * later level is a multiple of 2^db units of it), so they go to that level's
 * digit plane and the rest of the sum carries into level g - 1 in the same
 * 32-bit register; what is left after g = 2 is the high plane:
 *
 *     Z = (... (hi << db | d[zmin]) << db | ... | d[gtop]) << db(G - gtop),
 *     gtop = min(s + 1, G).
 *
 * Levels above G carry their rounded value (shifted up to the next level's
 * unit, so it is rounded exactly once). Every sum stays inside int32: a carry
 * is at most 2^-5 of the sum it comes from. zmin = 3; 4 in the FP8 format
 * (|2^5 L_2 + L_3 + carry| <= 2^27 + 2^23 + 2^20) and for BF16 when G = 7
 * (k_pad <= 128: 2^29 + 2^22 + 2^16), where levels 3 and 2 share the high
 * plane. Z takes at most 8 bytes per element in the BF16 format, 11 in FP8.
 *
 * Layout of one product, by groups of four columns: for each group m_pad x
 * int4 (high plane, a row's four columns side by side), then per digit plane
 * (zmin first) m_pad x 4 bytes. An epilogue thread owns one row, so a warp
 * stores whole 512- and 128-byte lines, each byte once, with plain stores.
 * Adding each level into an int64 Z with red.global.add.u64 instead moved
 * 6 x 8 bytes per element through the L2 atomic units (6 slices); the GEMM of
 * 222 x1 at 3000 x 2500 x 2049 took 455 us that way and takes 402 us now, of
 * a 300 x 700 x 450 classical problem 93 and 71 us. */
struct ZPlanes {
    int zmin, nd;
    __host__ __device__ static ZPlanes of(int s, int G, int fmt)
    {
        ZPlanes z;
        z.zmin = fmt != 0 || G == 7 ? 4 : 3;
        const int gtop = s + 1 < G ? s + 1 : G;
        z.nd = gtop >= z.zmin ? gtop - z.zmin + 1 : 0;
        return z;
    }
};

/* bytes of one 4-column group of Z */
__host__ __device__ __forceinline__ int64_t z_group_bytes(int64_t m_pad, int nd) { return m_pad * 4 * (4 + nd); }

/* the same index, in a way the compiler cannot carry loads across: the
 * epilogue's 64 sums leave no room to keep a problem's fields in registers
 * for a whole item, so they are read from the launch parameter where they are
 * used */
__device__ __forceinline__ int opaque(int x)
{
    asm volatile("" : "+r"(x));
    return x;
}

/* Drains one work item from the accumulator into Z (one epilogue warp: 32
 * TMEM lanes, kEpiCols columns from tmem address `tl`, one row per thread):
 * every chunk of every level, levels s+1 .. 2. zh is the address of Z row zi
 * in the high plane of the thread's first column group. `arrive(buf)` reports
 * a TMEM buffer read. */
template <class GL, class Arrive>
__device__ __forceinline__ bool drain_item(const GL& L, int p, uint8_t* zh, int zi, uint32_t tl, uint64_t* accf,
                                           int& buf, uint32_t& aph, int lane, volatile int* abort_flag, int code,
                                           Arrive arrive)
{
    int lsum[kEpiCols];
#pragma unroll
    for (int x = 0; x < kEpiCols; ++x) lsum[x] = 0;
    for (int g = L.prob[p].s + 1; g >= 2; --g) {
        int left, mul;
        {
            const GemmProblem& P = L.prob[opaque(p)];
            left = (level_pairs(g, P.s) * P.nkb + kChunkKB - 1) / kChunkKB;   /* chunks */
            mul = g == 2 && P.zmin == 4 ? 1 << P.db : 1;                      /* levels 3 and 2 in one register */
        }
        for (; left > 0; --left) {
            if (!sm103::mbar_wait(&accf[buf], aph, abort_flag, L.err, code)) return false;
            sm103::tc_fence_after();
#pragma unroll
            for (int h = 0; h < kEpiCols / 8; ++h) {
                uint32_t v[8];
                SM103_TMEM_LD_X8(tl + buf * kTileN + h * 8, v);
                sm103::tmem_wait_ld();
#pragma unroll
                for (int x = 0; x < 8; ++x)
                    lsum[h * 8 + x] += __float2int_rn(__uint_as_float(v[x])) * mul;   /* exact: integer, |v| <= 2^24 */
            }
            sm103::tc_fence_before();
            __syncwarp();
            if (lane == 0) arrive(buf);
            buf ^= 1;
            if (buf == 0) aph ^= 1;
        }
        const GemmProblem& P = L.prob[opaque(p)];
        const int G = P.zlevel, db = P.db, zmin = P.zmin, m_pad = P.m_pad;
        /* the GEMM never reads Z back: its lines leave L2 before the slices' */
        uint64_t pol;
        asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
        if (g > G) {
            /* round to units of G (ties up), back up to the next level's unit */
            const int sh = db * (g - G), up = g - 1 > G ? sh - db : 0;
#pragma unroll
            for (int x = 0; x < kEpiCols; ++x) lsum[x] = (((lsum[x] >> (sh - 1)) + 1) >> 1) << up;
        } else if (g >= zmin) {
            const uint64_t gstep = (uint64_t)z_group_bytes(m_pad, P.znd);
            const uint32_t dmask = db == 8 ? 0xffffffffu : 0x1f1f1f1fu;
            uint8_t* q = zh + ((int64_t)m_pad * 4 * (4 + g - zmin) - (int64_t)zi * 12);
#pragma unroll
            for (int x = 0; x < kEpiCols; x += 4) {
                const uint32_t w01 = __byte_perm((uint32_t)lsum[x], (uint32_t)lsum[x + 1], 0x0040u);
                const uint32_t w23 = __byte_perm((uint32_t)lsum[x + 2], (uint32_t)lsum[x + 3], 0x0040u);
                const uint32_t w = __byte_perm(w01, w23, 0x5410u) & dmask;
                asm volatile("st.global.L2::cache_hint.u32 [%0], %1, %3;\n\tadd.u64 %0, %0, %2;"
                             : "+l"(q) : "r"(w), "l"(gstep), "l"(pol) : "memory");
#pragma unroll
                for (int y = 0; y < 4; ++y) lsum[x + y] >>= db;
            }
        } else if (g == 2) {
            const uint64_t gstep = (uint64_t)z_group_bytes(m_pad, P.znd);
            uint8_t* q = zh;
#pragma unroll
            for (int x = 0; x < kEpiCols; x += 4) {
                asm volatile("st.global.L2::cache_hint.v4.u32 [%0], {%1, %2, %3, %4}, %6;\n\tadd.u64 %0, %0, %5;"
                             : "+l"(q) : "r"(lsum[x]), "r"(lsum[x + 1]), "r"(lsum[x + 2]), "r"(lsum[x + 3]),
                               "l"(gstep), "l"(pol) : "memory");
            }
        }
    }
    return true;
}

/* drain_item for a work unit: its chunks' sums, stored as they are. zp: the
 * thread's row in the unit's plane of its first column group. */
template <class GL, class Arrive>
__device__ __forceinline__ bool drain_unit(const GL& L, int4* zp, int64_t gstep, int nkb_unit, uint32_t tl,
                                           uint64_t* accf, int& buf, uint32_t& aph, int lane,
                                           volatile int* abort_flag, int code, Arrive arrive)
{
    int lsum[kEpiCols];
#pragma unroll
    for (int x = 0; x < kEpiCols; ++x) lsum[x] = 0;
    for (int left = (nkb_unit + kChunkKB - 1) / kChunkKB; left > 0; --left) {
        if (!sm103::mbar_wait(&accf[buf], aph, abort_flag, L.err, code)) return false;
        sm103::tc_fence_after();
#pragma unroll
        for (int h = 0; h < kEpiCols / 8; ++h) {
            uint32_t v[8];
            SM103_TMEM_LD_X8(tl + buf * kTileN + h * 8, v);
            sm103::tmem_wait_ld();
#pragma unroll
            for (int x = 0; x < 8; ++x) lsum[h * 8 + x] += __float2int_rn(__uint_as_float(v[x]));
        }
        sm103::tc_fence_before();
        __syncwarp();
        if (lane == 0) arrive(buf);
        buf ^= 1;
        if (buf == 0) aph ^= 1;
    }
#pragma unroll
    for (int x = 0; x < kEpiCols; x += 4) {
        *zp = make_int4(lsum[x], lsum[x + 1], lsum[x + 2], lsum[x + 3]);
        zp += gstep;
    }
    return true;
}

/* Persistent GEMM over a list of work items (problem, product of its group,
 * 128 x 256 output tile), drawn dynamically: the producer takes the next item
 * from L.sched and passes it to the other roles through a CTA-local item
 * ring, so the CTAs' items in flight stay contiguous. One CTA per
 * SM: warp 0 issues the TMA loads of the digit-slice tiles, warp 1 the
 * tcgen05.mma (M=128, N=256, K=16 BF16 or K=32 FP8 per the item's problem:
 * 128 clocks per MMA hide the accumulator dependency), warps 2..17 drain
 * each exact chunk (16 stage rows: 1024 BF16 or 2048 FP8 terms) from the
 * double-buffered TMEM accumulator into int32 level sums and write the
 * digits of Z that a finished level settles (drain_item). The pipeline, TMEM
 * allocation and barrier phases run on across items, so one item's last
 * stores overlap the next item's first MMAs. */
template <class GL>
__global__ void __launch_bounds__(kGemmThreads, 1)
split_gemm_kernel(const __grid_constant__ GL L)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* sA = smem;
    uint8_t* sB = smem + kStages * kATileBytes;
    uint64_t* full = (uint64_t*)(smem + kStages * kStageBytes);
    uint64_t* empty = full + kStages;
    uint64_t* accf = empty + kStages;
    uint64_t* acce = accf + 2;
    uint64_t* drain = acce + 2;
    uint64_t* sfull = drain + 1;                  /* item ring: slot written */
    uint64_t* sempty = sfull + kSchedSlots;       /* item ring: slot read by every consumer */
    int* sitem = (int*)(sempty + kSchedSlots);
    uint32_t* tmem_slot = (uint32_t*)(sitem + kSchedSlots);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;

    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) { sm103::mbar_init(&full[i], 1); sm103::mbar_init(&empty[i], 1); }
        for (int i = 0; i < 2; ++i) { sm103::mbar_init(&accf[i], 1); sm103::mbar_init(&acce[i], kEpiWarps); }
        sm103::mbar_init(drain, 1);
        for (int i = 0; i < kSchedSlots; ++i) {
            sm103::mbar_init(&sfull[i], 1);
            sm103::mbar_init(&sempty[i], 1 + kEpiWarps);   /* the MMA thread and every epilogue warp */
        }
        *abort_flag = 0;
        sm103::fence_mbar_init();
    }
    if (warp == 1) { sm103::tmem_alloc(tmem_slot, kTmemCols); sm103::tmem_relinquish(); }
    sm103::tc_fence_before();
    __syncthreads();
    sm103::tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    sm103::grid_launch_dependents();
    sm103::grid_wait();   /* the slices, L.sched and (a reused) Z are the launches' before this one */
    if (warp == 0) {
        /* ---------------- TMA producer ---------------- */
        if (lane == 0) {
            int st = 0;
            uint32_t ph = 0;
            uint32_t armed = 0;  /* stages armed in the current pass (bit mask) */
            bool ok = true;
            int last_p = -1;
            ItemRing ring{sm103::smem_u32(sfull), 0, 0};
            for (;;) {
                /* the producer takes the next item from L.sched and publishes it */
                if (!sm103::mbar_wait_acq_cluster_u32(ring.empty_at(), ring.ph ^ 1, abort_flag, L.err, 7)) {
                    ok = false;
                    break;
                }
                int b = (int)atomicAdd(L.sched, 1u);
                if (b >= L.nitems) b = -1;
                sitem[ring.slot] = b;
                sm103::mbar_arrive(&sfull[ring.slot]);
                ring.next();
                if (b < 0) break;
                const Item it = decode_item(L, b);
                const GemmProblem& P = L.prob[it.p];
                if (it.p != last_p) { sm103::prefetch_tmap(&P.tmA); sm103::prefetch_tmap(&P.tmB); last_p = it.p; }
                const int s = P.s, nkb = P.nkb;
                const int arow = it.r * s * P.m_pad + it.tile_m * kTileM;
                const int brow = it.r * s * P.n_pad + it.tile_n * kTileN;
                /* Pair order: levels from s+1 down to 2 (ZPlanes), t ascending
                 * in odd levels and descending in even ones, so the last pair
                 * of a level and the first of the next share a slice
                 * ((4,1)->(3,1), (1,3)->(1,2), ...), and k runs
                 * forward and backward on alternate pairs, so a shared slice's
                 * most recently loaded blocks are read again first, while they
                 * are still in L2. The MMA side only counts stages; every
                 * chunk sum is exact in any order. (An L2 prefetch of the boxes
                 * eight stages ahead measured 3x slower, with 7x the DRAM
                 * reads.) */
                const UnitSpan us = P.nunits ? unit_span(s, nkb, P.unit_kb, it.unit) : UnitSpan{0, 0, 0};
                const int g_hi = P.nunits ? us.g : s + 1, g_lo = P.nunits ? us.g : 2;
                int pi = 0;
                for (int g = g_hi; g >= g_lo && ok; --g) {
                    const int tlo = max(1, g - s), thi = min(s, g - 1);
                    const UnitSpan sp = level_span(P, us, g);
                    int x = sp.q0 / nkb, y = sp.q0 - x * nkb;
                    for (int q = sp.q0; q < sp.q1; ++q) {
                        const int t = (g & 1) ? tlo + x : thi - x;
                        const int u = g - t;
                        const int kb = ((pi + x) & 1) ? nkb - 1 - y : y;
                        if (!sm103::mbar_wait(&empty[st], ph ^ 1, abort_flag, L.err, 1)) { ok = false; break; }
                        sm103::mbar_arrive_expect_tx(&full[st], kStageBytes);
                        sm103::tma_load_2d(sA + st * kATileBytes, &P.tmA, &full[st], kb * P.kbe,
                                           arow + (t - 1) * P.m_pad);
                        sm103::tma_load_2d(sB + st * kBTileBytes, &P.tmB, &full[st], kb * P.kbe,
                                           brow + (u - 1) * P.n_pad);
                        armed |= 1u << st;
                        if (++st == kStages) { st = 0; ph ^= 1; armed = 0; }
                        if (++y == nkb) { y = 0; ++x; }
                    }
                    pi += thi - tlo + 1;
                }
            }
            if (!ok) {
                /* let every load already issued land before the CTA exits */
                for (int i = 0; i < kStages; ++i) {
                    const uint32_t par = (armed >> i) & 1u ? ph : ph ^ 1;
                    uint64_t t0 = sm103::globaltimer();
                    while (!sm103::mbar_try_wait(&full[i], par) &&
                           sm103::globaltimer() - t0 < sm103::kWaitLimitNs) {}
                }
            }
        }
    } else if (warp == 1) {
        /* ---------------- MMA issuer ---------------- */
        if (lane == 0) {
            constexpr uint32_t idesc16 = sm103::idesc_bf16_f32(kTileM, kTileN);
            constexpr uint32_t idesc8 = sm103::idesc_e4m3_f32(kTileM, kTileN);
            int st = 0, buf = 0;
            uint32_t ph = 0, aph = 0;
            bool ok = true;
            ItemRing ring{sm103::smem_u32(sfull), 0, 0};
            for (;;) {
                int b;
                if (!ring.take(&b, abort_flag, L.err, 8)) { ok = false; break; }
                if (b < 0) break;
                const Item it = decode_item(L, b);
                const GemmProblem& P = L.prob[it.p];
                const int fmt = P.fmt;
                const UnitSpan us = P.nunits ? unit_span(P.s, P.nkb, P.unit_kb, it.unit) : UnitSpan{0, 0, 0};
                const int g_hi = P.nunits ? us.g : P.s + 1, g_lo = P.nunits ? us.g : 2;
                for (int g = g_hi; g >= g_lo && ok; --g) {
                    const UnitSpan sp = level_span(P, us, g);
                    const int level_kb = sp.q1 - sp.q0;
                    for (int jl = 0; jl < level_kb; ) {
                        if (jl % kChunkKB == 0) {
                            if (!sm103::mbar_wait(&acce[buf], aph ^ 1, abort_flag, L.err, 2)) { ok = false; break; }
                            sm103::tc_fence_after();
                        }
                        if (!sm103::mbar_wait(&full[st], ph, abort_flag, L.err, 3)) { ok = false; break; }
                        sm103::tc_fence_after();
                        const uint32_t a0 = sm103::smem_u32(sA + st * kATileBytes);
                        const uint32_t b0 = sm103::smem_u32(sB + st * kBTileBytes);
                        /* four MMAs per 128-byte stage row: K = 16 BF16 or 32 FP8
                         * elements each, 32 bytes apart */
                        if (fmt) {
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk)
                                sm103::mma_f8(tmem + buf * kTileN, sm103::smem_desc_sw128(a0 + kk * 32),
                                              sm103::smem_desc_sw128(b0 + kk * 32), idesc8,
                                              (jl % kChunkKB != 0 || kk != 0) ? 1u : 0u);
                        } else {
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk)
                                sm103::mma_bf16(tmem + buf * kTileN, sm103::smem_desc_sw128(a0 + kk * 32),
                                                sm103::smem_desc_sw128(b0 + kk * 32), idesc16,
                                                (jl % kChunkKB != 0 || kk != 0) ? 1u : 0u);
                        }
                        sm103::mma_commit(&empty[st]);
                        if (++st == kStages) { st = 0; ph ^= 1; }
                        ++jl;
                        if (jl % kChunkKB == 0 || jl == level_kb) {
                            sm103::mma_commit(&accf[buf]);
                            buf ^= 1;
                            if (buf == 0) aph ^= 1;
                        }
                    }
                }
            }
            /* all issued MMAs complete before TMEM is released */
            sm103::mma_commit(drain);
            uint64_t t0 = sm103::globaltimer();
            while (!sm103::mbar_try_wait(drain, 0) && sm103::globaltimer() - t0 < sm103::kWaitLimitNs) {}
        }
    } else {
        /* ---------------- epilogue warps ---------------- */
        const int quarter = warp % 4;                  /* TMEM lane quarter this warp may access */
        const int colbase = ((warp - 2) / 4) * kEpiCols;
        const int row = quarter * 32 + lane;
        const uint32_t tl = tmem + ((uint32_t)(quarter * 32) << 16);
        int buf = 0;
        uint32_t aph = 0;
        ItemRing ring{sm103::smem_u32(sfull), 0, 0};
        for (;;) {
            int b;
            if (!ring.take_warp(&b, lane, abort_flag, L.err, 9)) break;
            if (b < 0) break;
            const Item it = decode_item(L, b);
            const GemmProblem& P = L.prob[it.p];
            const int zi = P.zrow0 + it.tile_m * kTileM + row;
            if (P.nunits) {
                const UnitSpan us = unit_span(P.s, P.nkb, P.unit_kb, it.unit);
                int4* zp = (int4*)P.Z + ((int64_t)it.unit * P.n_pad + it.tile_n * kTileN + colbase) / 4 * P.m_pad + zi;
                if (!drain_unit(L, zp, P.m_pad, us.q1 - us.q0, tl + colbase, accf, buf, aph, lane, abort_flag, 4,
                                [&](int q) { sm103::mbar_arrive(&acce[q]); }))
                    break;
                continue;
            }
            uint8_t* z0 = P.Z + ((int64_t)it.r * P.n_pad + it.tile_n * kTileN + colbase) / 4 *
                                    z_group_bytes(P.m_pad, P.znd);
            if (!drain_item(L, it.p, z0 + (int64_t)zi * 16, zi, tl + colbase, accf, buf, aph, lane, abort_flag, 4,
                            [&](int q) { sm103::mbar_arrive(&acce[q]); }))
                break;
        }
    }
    sm103::tc_fence_before();
    __syncthreads();
    sm103::tc_fence_after();
    if (warp == 1) sm103::tmem_dealloc(tmem, kTmemCols);
}

/* ---------------------------------------------------- CTA-pair GEMM ---- */

constexpr int kPairTileM = 256;                       /* rows of a pair tile (128 per CTA) */
constexpr int kPairMinRows = 1024;                    /* m_e from which single calls use pair tiles */
constexpr int kPairStages = 6;
constexpr int kPairRasterGroup = 6;                   /* pair-tile rows per raster band (1536 rows) */
std::atomic<int> g_pair_rows{kPairMinRows};           /* m_e from which GEMMs take pair tiles (host) */
constexpr uint32_t kPairHalfBytes = 128 * kBK * 2;    /* 16 KB: 128 rows of one 128-byte stage row */
constexpr uint32_t kPairStageBytes = 2 * kPairHalfBytes;
constexpr size_t kPairSmem = (size_t)kPairStages * kPairStageBytes + 1024 + 512;



/* The same GEMM as split_gemm_kernel with CTA pairs (clusters of two), with
 * work items drawn dynamically: the even CTA's producer takes the next item
 * from L.sched (atomicAdd) and writes it into both CTAs' item rings; every
 * other role reads the ring, so the clusters' items in flight stay
 * contiguous and share operand panels in L2 (a static round robin lets them
 * drift apart). A work item is a 256 x 256 tile of a product; each CTA loads its 128 rows of the A
 * slice tile and its 128-column half of the B slice tile (32 KB per stage
 * instead of 48 KB, so the L2 feeds each SM a third less per MMA and the
 * six-stage ring looks 50% further ahead), and the even CTA issues
 * tcgen05.mma cta_group::2 (M=256, N=256) into both CTAs' TMEM. Both CTAs'
 * stage loads complete on the even CTA's barrier (TMA cta_group::2); the MMA
 * commits arrive on both CTAs' stage and accumulator barriers; each CTA's epilogue drains its own 128 rows exactly
 * as in split_gemm_kernel and reports the buffer free to the even CTA. All
 * waits are bounded; the two cluster barriers (after barrier set-up, before
 * TMEM release) are reached by every thread of both CTAs. */
template <class GL>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGemmThreads, 1)
split_gemm_pair_kernel(const __grid_constant__ GL L)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* sA = smem;
    uint8_t* sB = smem + kPairStages * kPairHalfBytes;
    uint64_t* full = (uint64_t*)(smem + kPairStages * kPairStageBytes);
    uint64_t* empty = full + kPairStages;
    uint64_t* accf = empty + kPairStages;
    uint64_t* acce = accf + 2;
    uint64_t* drain = acce + 2;
    uint64_t* sfull = drain + 1;                  /* item ring: slot written */
    uint64_t* sempty = sfull + kSchedSlots;       /* item ring: slot read by every consumer (even CTA) */
    int* sitem = (int*)(sempty + kSchedSlots);
    uint32_t* tmem_slot = (uint32_t*)(sitem + kSchedSlots);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const uint32_t rank = sm103::cluster_ctarank();

    if (threadIdx.x == 0) {
        for (int i = 0; i < kPairStages; ++i) {
            sm103::mbar_init(&full[i], 1);
            sm103::mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) { sm103::mbar_init(&accf[i], 1); sm103::mbar_init(&acce[i], 2 * kEpiWarps); }
        sm103::mbar_init(drain, 1);
        for (int i = 0; i < kSchedSlots; ++i) {
            sm103::mbar_init(&sfull[i], 1);
            sm103::mbar_init(&sempty[i], kSchedConsumers);
        }
        *abort_flag = 0;
        sm103::fence_mbar_init();
    }
    if (warp == 1) { sm103::tmem_alloc_pair(tmem_slot, kTmemCols); sm103::tmem_relinquish_pair(); }
    sm103::tc_fence_before();
    sm103::cluster_sync();   /* both CTAs' barriers exist before any remote arrive */
    sm103::tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        /* ---------------- TMA producer (both CTAs) ---------------- */
        if (lane == 0) {
            int st = 0;
            uint32_t ph = 0;
            uint32_t armed = 0;
            bool ok = true;
            int last_p = -1;
            ItemRing ring{sm103::smem_u32(sfull), 0, 0};
            for (;;) {
                int b;
                if (rank == 0) {
                    /* the even producer takes the next item and publishes it
                     * to both CTAs' rings */
                    if (!sm103::mbar_wait_acq_cluster_u32(ring.empty_at(), ring.ph ^ 1, abort_flag, L.err, 17)) {
                        ok = false;
                        break;
                    }
                    b = (int)atomicAdd(L.sched, 1u);
                    if (b >= L.nitems) b = -1;
                    sitem[ring.slot] = b;
                    sm103::st_shared_cluster_u32(sm103::mapa(sm103::smem_u32(&sitem[ring.slot]), 1), (uint32_t)b);
                    sm103::mbar_arrive(&sfull[ring.slot]);
                    sm103::mbar_arrive_release_cluster(sm103::mapa(sm103::smem_u32(&sfull[ring.slot]), 1));
                    ring.next();
                } else if (!ring.take(&b, abort_flag, L.err, 18)) {
                    ok = false;
                    break;
                }
                if (b < 0) break;
                const Item it = decode_item(L, b, kPairRasterGroup);
                const GemmProblem& P = L.prob[it.p];
                if (it.p != last_p) { sm103::prefetch_tmap(&P.tmA); sm103::prefetch_tmap(&P.tmB); last_p = it.p; }
                const int s = P.s, nkb = P.nkb;
                const int arow = it.r * s * P.m_pad + it.tile_m * kPairTileM + 128 * (int)rank;
                const int brow = it.r * s * P.n_pad + it.tile_n * kTileN + 128 * (int)rank;
                int pi = 0;   /* the single-CTA kernel's pair order */
                for (int g = s + 1; g >= 2 && ok; --g) {
                    const int tlo = max(1, g - s), thi = min(s, g - 1);
                    for (int x = 0; x <= thi - tlo && ok; ++x, ++pi) {
                        const int t = (g & 1) ? tlo + x : thi - x;
                        const int u = g - t;
                        for (int y = 0; y < nkb; ++y) {
                            const int kb = (pi & 1) ? nkb - 1 - y : y;
                            if (!sm103::mbar_wait(&empty[st], ph ^ 1, abort_flag, L.err, 11)) { ok = false; break; }
                            /* both CTAs' loads complete on the even CTA's full[st]; the
                             * even CTA expects the bytes of both */
                            if (rank == 0) sm103::mbar_arrive_expect_tx(&full[st], 2 * kPairStageBytes);
                            const uint32_t fb = sm103::mapa(sm103::smem_u32(&full[st]), 0);
                            sm103::tma_load_2d_pair(sA + st * kPairHalfBytes, &P.tmA, fb, kb * P.kbe,
                                                    arow + (t - 1) * P.m_pad);
                            sm103::tma_load_2d_pair(sB + st * kPairHalfBytes, &P.tmB, fb, kb * P.kbe,
                                                    brow + (u - 1) * P.n_pad);
                            armed |= 1u << st;
                            if (++st == kPairStages) { st = 0; ph ^= 1; armed = 0; }
                        }
                    }
                }
            }
            if (!ok && rank == 0) {
                for (int i = 0; i < kPairStages; ++i) {
                    const uint32_t par = (armed >> i) & 1u ? ph : ph ^ 1;
                    uint64_t t0 = sm103::globaltimer();
                    while (!sm103::mbar_try_wait(&full[i], par) &&
                           sm103::globaltimer() - t0 < sm103::kWaitLimitNs) {}
                }
            }
            (void)armed;
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            /* ---------------- even CTA: MMA issuer ---------------- */
            constexpr uint32_t idesc16 = sm103::idesc_bf16_f32(kPairTileM, kTileN);
            constexpr uint32_t idesc8 = sm103::idesc_e4m3_f32(kPairTileM, kTileN);
            int st = 0, buf = 0;
            uint32_t ph = 0, aph = 0;
            bool ok = true;
            ItemRing ring{sm103::smem_u32(sfull), 0, 0};
            for (;;) {
                int b;
                if (!ring.take(&b, abort_flag, L.err, 19)) { ok = false; break; }
                if (b < 0) break;
                const Item it = decode_item(L, b, kPairRasterGroup);
                const int s = L.prob[it.p].s, nkb = L.prob[it.p].nkb, fmt = L.prob[it.p].fmt;
                for (int g = s + 1; g >= 2 && ok; --g) {
                    const int level_kb = level_pairs(g, s) * nkb;
                    for (int jl = 0; jl < level_kb && ok; ) {
                        if (jl % kChunkKB == 0) {
                            if (!sm103::mbar_wait(&acce[buf], aph ^ 1, abort_flag, L.err, 13)) { ok = false; break; }
                            sm103::tc_fence_after();
                        }
                        if (!sm103::mbar_wait(&full[st], ph, abort_flag, L.err, 14)) { ok = false; break; }
                        sm103::tc_fence_after();
                        const uint32_t a0 = sm103::smem_u32(sA + st * kPairHalfBytes);
                        const uint32_t b0 = sm103::smem_u32(sB + st * kPairHalfBytes);
                        if (fmt) {
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk)
                                sm103::mma_f8_pair(tmem + buf * kTileN, sm103::smem_desc_sw128(a0 + kk * 32),
                                                   sm103::smem_desc_sw128(b0 + kk * 32), idesc8,
                                                   (jl % kChunkKB != 0 || kk != 0) ? 1u : 0u);
                        } else {
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk)
                                sm103::mma_bf16_pair(tmem + buf * kTileN, sm103::smem_desc_sw128(a0 + kk * 32),
                                                     sm103::smem_desc_sw128(b0 + kk * 32), idesc16,
                                                     (jl % kChunkKB != 0 || kk != 0) ? 1u : 0u);
                        }
                        sm103::mma_commit_pair(&empty[st]);
                        if (++st == kPairStages) { st = 0; ph ^= 1; }
                        ++jl;
                        if (jl % kChunkKB == 0 || jl == level_kb) {
                            sm103::mma_commit_pair(&accf[buf]);
                            buf ^= 1;
                            if (buf == 0) aph ^= 1;
                        }
                    }
                }
            }
            /* all issued MMAs complete before either CTA releases TMEM */
            sm103::mma_commit_pair(drain);
            uint64_t t0 = sm103::globaltimer();
            while (!sm103::mbar_try_wait(drain, 0) && sm103::globaltimer() - t0 < sm103::kWaitLimitNs) {}
        }
    } else {
        /* ---------------- epilogue warps (both CTAs) ---------------- */
        const int quarter = warp % 4;
        const int colbase = ((warp - 2) / 4) * kEpiCols;
        const int row = quarter * 32 + lane;
        const uint32_t tl = tmem + ((uint32_t)(quarter * 32) << 16);
        const uint32_t acce0 = sm103::mapa(sm103::smem_u32(acce), 0);
        int buf = 0;
        uint32_t aph = 0;
        ItemRing ring{sm103::smem_u32(sfull), 0, 0};
        for (;;) {
            int b;
            if (!ring.take_warp(&b, lane, abort_flag, L.err, 20)) break;
            if (b < 0) break;
            const Item it = decode_item(L, b, kPairRasterGroup);
            const GemmProblem& P = L.prob[it.p];
            const int zi = P.zrow0 + it.tile_m * kPairTileM + 128 * (int)rank + row;
            uint8_t* z0 = P.Z + ((int64_t)it.r * P.n_pad + it.tile_n * kTileN + colbase) / 4 *
                                    z_group_bytes(P.m_pad, P.znd);
            if (!drain_item(L, it.p, z0 + (int64_t)zi * 16, zi, tl + colbase, accf, buf, aph, lane, abort_flag, 16,
                            [&](int q) { sm103::mbar_arrive_cluster(acce0 + q * 8); }))
                break;
        }
    }
    sm103::tc_fence_before();
    __syncthreads();
    sm103::cluster_sync();   /* no remote arrive or MMA still targets either CTA */
    sm103::tc_fence_after();
    if (warp == 1) sm103::tmem_dealloc_pair(tmem, kTmemCols);
}

/* Multi-C epilogue for a group of products [r0, r0 + nprod): one thread per
 * (C sub-block p = blockIdx.y, element (i, j) of p) adds alpha*W[p,r] *
 * M_r[i,j] for the group's products in increasing order, with M_r[i,j] =
 * 2^(E_i + F_j + 2 - db*G) * Z_r[i,j] = 2^(ebase + E_i + F_j) * Z_r[i,j]
 * converted in integer arithmetic
 * (plugin/ref_kernels/bli_gemm_fmm_ref.c:99-120, once per group instead of
 * once per product). */
constexpr int kScatterMaxEnt = 1024;

/* Z of a product group as the C updates read it (see ZPlanes) */
struct ZView {
    const uint8_t* base;
    int64_t prod;     /* bytes per product */
    int64_t group;    /* bytes per 4-column group */
    int m_pad, n_pad;
    int nd;           /* digit planes */
    int ebase;        /* exponent of Z's unit relative to 2^(E_i + F_j) */
};

constexpr int kScatterCols = 4;   /* columns per thread: one column group of Z */

/* The 5-bit digits of two columns in the 16-bit halves of x[p], plane zmin + p,
 * absent ones zero: three digits of both columns to a word, then each
 * column's Z from its high word. Digit by digit in 64 bits the conversion took
 * twice the instructions and bounded the C updates per sub-block (the ALU pipe
 * 75% busy): 333 x2 at 3101 x 2244 x 73, 5 slices, 1590 us a call, 1400 now. */
struct Fp8Pair {
    uint32_t a, b, c;

    __device__ __forceinline__ explicit Fp8Pair(const uint32_t (&x)[7])
        : a((x[0] * 32 + x[1]) * 32 + x[2]), b((x[3] * 32 + x[4]) * 32 + x[5]), c(x[6])
    {
    }
    /* column u: hi * 32^7 + its seven digits, down to the nd that there are */
    __device__ __forceinline__ int64_t value(int hi, int u, int nd) const
    {
        const uint32_t d0 = u ? a >> 16 : a & 0xffffu, d1 = u ? b >> 16 : b & 0xffffu, d2 = u ? c >> 16 : c & 0xffffu;
        const uint32_t low = d0 * (1u << 20) + d1 * 32 + d2, high = (uint32_t)hi * 8 + (d0 >> 12);
        return (int64_t)(((uint64_t)high << 32) | low) >> (5 * (7 - nd));
    }
};

/* One row of a column group of one product: the loads (one int4, nd words, the
 * exponents), then the four Z values. FMT 0: at most four byte digits below
 * the high word, absent ones zero (Z counts in units of level G whatever the
 * slice count); FMT 1: nd = G - 3 five-bit digits. */
template <int FMT>
struct ZRow {
    static constexpr int NP = FMT ? 7 : 4;
    int4 hi;
    int4 f;
    int e;
    uint32_t w[NP];

    __device__ __forceinline__ void load(const ZView& v, const int* __restrict__ e_row, const int* __restrict__ f_col,
                                         int q, int i, int j)
    {
        const uint8_t* g = v.base + q * v.prod + (int64_t)(j >> 2) * v.group;
        hi = *(const int4*)(g + (int64_t)i * 16);
        const uint8_t* d = g + ((int64_t)v.m_pad * 16 + (int64_t)i * 4);
#pragma unroll
        for (int p = 0; p < NP; ++p) w[p] = p < v.nd ? *(const uint32_t*)(d + (int64_t)p * v.m_pad * 4) : 0u;
        e = e_row[(int64_t)q * v.m_pad + i];
        f = *(const int4*)(f_col + (int64_t)q * v.n_pad + j);
    }
    /* M[i, j + u] = 2^(ebase + E_i + F_j) * Z */
    __device__ __forceinline__ void values(const ZView& v, double (&M)[kScatterCols]) const
    {
        const int h[4] = {hi.x, hi.y, hi.z, hi.w}, fc[4] = {f.x, f.y, f.z, f.w};
        const int er = e + v.ebase;
        if (FMT == 0) {
            /* the four words' bytes, transposed: digit 0 on top */
            const uint32_t a0 = __byte_perm(w[1], w[0], 0x5140u), a1 = __byte_perm(w[1], w[0], 0x7362u);
            const uint32_t b0 = __byte_perm(w[3], w[2], 0x5140u), b1 = __byte_perm(w[3], w[2], 0x7362u);
            const uint32_t lo[4] = {__byte_perm(b0, a0, 0x5410u), __byte_perm(b0, a0, 0x7632u),
                                    __byte_perm(b1, a1, 0x5410u), __byte_perm(b1, a1, 0x7632u)};
#pragma unroll
            for (int u = 0; u < 4; ++u)
                M[u] = i64_to_double_scaled((int64_t)(((uint64_t)(uint32_t)h[u] << 32) | lo[u]), er + fc[u]);
        } else {
            uint32_t x[7], y[7];   /* columns 0 and 2, 1 and 3 */
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                x[p] = __byte_perm(w[p], 0u, 0x4240u);
                y[p] = __byte_perm(w[p], 0u, 0x4341u);
            }
            const Fp8Pair even(x), odd(y);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                M[u] = i64_to_double_scaled((u & 1 ? odd : even).value(h[u], u >> 1, v.nd), er + fc[u]);
        }
    }
};

/* ZRow for two columns of a group (j even) */
template <int FMT>
struct ZPair {
    static constexpr int NP = FMT ? 7 : 4;
    int2 hi, f;
    int e;
    uint32_t w[NP];

    __device__ __forceinline__ void load(const ZView& v, const int* __restrict__ e_row, const int* __restrict__ f_col,
                                         int q, int i, int j)
    {
        const uint8_t* g = v.base + q * v.prod + (int64_t)(j >> 2) * v.group;
        hi = *(const int2*)(g + (int64_t)i * 16 + (j & 2) * 4);
        const uint8_t* d = g + ((int64_t)v.m_pad * 16 + (int64_t)i * 4 + (j & 2));
#pragma unroll
        for (int p = 0; p < NP; ++p) w[p] = p < v.nd ? *(const uint16_t*)(d + (int64_t)p * v.m_pad * 4) : 0u;
        e = e_row[(int64_t)q * v.m_pad + i];
        f = *(const int2*)(f_col + (int64_t)q * v.n_pad + j);
    }
    __device__ __forceinline__ void values(const ZView& v, double (&M)[2]) const
    {
        const int h[2] = {hi.x, hi.y}, fc[2] = {f.x, f.y};
        const int er = e + v.ebase;
        if (FMT == 0) {
            const uint32_t a = __byte_perm(w[0], w[1], 0x5410u), b = __byte_perm(w[2], w[3], 0x5410u);
            const uint32_t lo[2] = {__byte_perm(a, b, 0x0246u), __byte_perm(a, b, 0x1357u)};
#pragma unroll
            for (int u = 0; u < 2; ++u)
                M[u] = i64_to_double_scaled((int64_t)(((uint64_t)(uint32_t)h[u] << 32) | lo[u]), er + fc[u]);
        } else {
            uint32_t x[7];
#pragma unroll
            for (int p = 0; p < NP; ++p) x[p] = __byte_perm(w[p], 0u, 0x4140u);
            const Fp8Pair both(x);
#pragma unroll
            for (int u = 0; u < 2; ++u) M[u] = i64_to_double_scaled(both.value(h[u], u, v.nd), er + fc[u]);
        }
    }
};

/* beta*c of the C update, as scale_c_kernel forms it */
__device__ __forceinline__ double beta_c(double beta, const double* c)
{
    if (beta == 1.0) return *c;
    return beta == 0.0 ? 0.0 : beta * *c;
}

/* C updates of one C sub-block p: tiles of tr rows (a power of two, 8 to 128) x
 * 512 / tr columns, a thread a row of a 4-column group. Where scatter_all_better
 * says so. One thread gathers the sub-block's entries for each tile, which
 * bounds narrow product grids: with 128 rows x 4 columns on 8 rows, 444 x2 on an
 * 8 x 600 grid takes 8.5 ms a call instead of 5.2. */
constexpr int kScatterThreads = 128;

struct ScatterEntries {
    double lam[kScatterMaxEnt];
    int prod[kScatterMaxEnt];
    int n;
};

/* tile bx of sub-block p; WIDE: tr is 128, so a block's columns are the same for all its threads (3% of the kernel) */
template <int FMT, bool WIDE>
__device__ __forceinline__ void scatter_part_body(ScatterEntries& sh, const int* __restrict__ tab, int r0, int nprod,
                                                  int64_t m, int64_t n, double alpha, double beta, const ZView& Z,
                                                  const int* __restrict__ e_row, const int* __restrict__ f_col,
                                                  double* __restrict__ C, int64_t ldc, int tr, int p, uint32_t bx)
{
    const Tab t = tab_view(tab);
    int ro, rl, co, cl;
    fmm_part_geom32((int)m, t.mt, p / t.nt, &ro, &rl);
    fmm_part_geom32((int)n, t.nt, p % t.nt, &co, &cl);
    if (rl <= 0 || cl <= 0) return;   /* empty sub-block (dimension smaller than its split) */
    /* this part's entries that fall in the group, in product order */
    if (threadIdx.x == 0) {
        int q = 0;
        for (int e = t.wp_off[p]; e < t.wp_off[p + 1] && q < kScatterMaxEnt; ++e) {
            const int r = t.wp_ent[2 * e] - r0;
            if (r < 0) continue;
            if (r >= nprod) break;
            sh.prod[q] = r;
            sh.lam[q] = alpha * (double)t.wp_ent[2 * e + 1];
            ++q;
        }
        sh.n = q;
    }
    __syncthreads();
    const int ne = sh.n;
    const int TR = WIDE ? kScatterThreads : tr;
    const uint32_t me = (uint32_t)((m + t.mt - 1) / t.mt), tiles_i = (me + TR - 1) / TR;
    const int i = (int)(bx % tiles_i * TR) + (int)(WIDE ? threadIdx.x : threadIdx.x % TR);
    const int j = (int)(WIDE ? bx / tiles_i : bx / tiles_i * (kScatterThreads / TR) + threadIdx.x / TR) * 4;
    if ((ne == 0 && beta == 1.0) || i >= rl || j >= cl) return;
    double* cp = C + ro + i + (int64_t)(co + j) * ldc;
    double c[kScatterCols];
#pragma unroll
    for (int u = 0; u < 4; ++u) c[u] = j + u < cl ? beta_c(beta, cp + u * ldc) : 0.0;
    ZRow<FMT> z;
    if (ne > 0) z.load(Z, e_row, f_col, sh.prod[0], i, j);
    for (int q = 0; q < ne; ++q) {
        double M[kScatterCols];
        z.values(Z, M);
        if (q + 1 < ne) z.load(Z, e_row, f_col, sh.prod[q + 1], i, j);   /* in flight under this product's updates */
#pragma unroll
        for (int u = 0; u < 4; ++u) c[u] = fma(sh.lam[q], M[u], c[u]);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
        if (j + u < cl) cp[u * ldc] = c[u];
}

/* grid: tiles x sub-blocks */
template <int FMT, bool WIDE>
__global__ void __launch_bounds__(kScatterThreads)
scatter_kernel(const int* __restrict__ tab, int r0, int nprod, int64_t m, int64_t n, double alpha, double beta,
               const ZView Z, const int* __restrict__ e_row, const int* __restrict__ f_col, double* __restrict__ C,
               int64_t ldc, int tr)
{
    __shared__ ScatterEntries sh;
    scatter_part_body<FMT, WIDE>(sh, tab, r0, nprod, m, n, alpha, beta, Z, e_row, f_col, C, ldc, tr, (int)blockIdx.y,
                           blockIdx.x);
}

/* Multi-C epilogue, element-major: a thread takes a row of a 4-column group, or
 * of half of one, of the product grid (rows [i_lo, i_lo + i_rows), all m_e rows
 * when i_rows is 0; columns [c0, c1)) and updates those elements of every C
 * sub-block p, so each product's Z_r is read (whole words) and converted once
 * and shared by all sub-blocks it feeds. The sub-blocks' running values live
 * in shared memory (cs[p][pair][thread], two columns each); for every
 * sub-block the updates still come in increasing product order, so the result
 * is identical to scatter_kernel's. Used when the sub-block count and the
 * group's W entries fit the shared-memory budget.
 *
 * Bound by the FP64 pipe (2 FMA/clk/SM) once an algorithm has several
 * sub-blocks, if four independent chains per thread and enough threads feed it
 * (222 x1 at 3000 x 2500: 66 us, 107 us with one element per thread; its 12
 * FMAs per element of the product grid take 37 us of the pipe). Shared memory
 * limits the threads, so above 6 sub-blocks a thread takes two columns (222
 * x2 at 4096, 16 sub-blocks: 326 us, 416 with four; 333 x1: 260 and 270), up
 * to that four, which read fewer and wider words (222 x1: 73 us with two). The
 * classical case is bound by HBM instead (8 bytes of Z, 16 of C per element). */
constexpr int kScatterAllSmem = 32 * 1024;   /* cs[] budget: P * threads * columns * 8 */
constexpr int kScatterAllMaxSmem = 96 * 1024;

/* scatter_all_body for one sub-block fed by one product (the classical split GEMM): no shared memory, the C
 * values in registers; HBM-bound (Z and C). l: alpha times W. Tiles of blockDim.x rows x 4 columns. */
template <int FMT>
__device__ __forceinline__ void scatter_one_body(int64_t n, double l, double beta, const ZView& Z,
                                                 const int* __restrict__ e_row, const int* __restrict__ f_col,
                                                 double* __restrict__ C, int64_t ldc, int c0, int c1, uint32_t vb,
                                                 uint32_t vg, uint32_t i_lo, uint32_t rows)
{
    const int T = (int)blockDim.x, jl = min((int)n, c1);
    const uint32_t tiles_i = (rows + T - 1) / T, tiles = tiles_i * (uint32_t)((c1 + 3) / 4 - c0 / 4);
    for (uint32_t x = vb; x < tiles; x += vg) {
        const int i = (int)(i_lo + x % tiles_i * T) + (int)threadIdx.x, j = (int)(c0 / 4 + x / tiles_i) * 4;
        if (i >= (int)(i_lo + rows)) continue;
        ZRow<FMT> z;
        z.load(Z, e_row, f_col, 0, i, j);
        double* cp = C + i + (int64_t)j * ldc;
        double c[kScatterCols], M[kScatterCols];
#pragma unroll
        for (int u = 0; u < 4; ++u) c[u] = j + u >= c0 && j + u < jl ? beta_c(beta, cp + u * ldc) : 0.0;
        z.values(Z, M);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (j + u >= c0 && j + u < jl) cp[u * ldc] = fma(l, M[u], c[u]);
    }
}

/* vb, vg: the block's index among the vg blocks that share the element range */
template <int FMT, int NC>
__device__ __forceinline__ void scatter_all_body(const int* __restrict__ tab, int r0, int nprod, int64_t m, int64_t n,
                                                 double alpha, double beta, const ZView& Z,
                                                 const int* __restrict__ e_row, const int* __restrict__ f_col,
                                                 double* __restrict__ C, int64_t ldc, int c0, int c1, uint32_t vb,
                                                 uint32_t vg, uint32_t i_lo = 0, uint32_t i_rows = 0)
{
    extern __shared__ __align__(16) double sm_all[];
    const Tab t = tab_view(tab);
    const int P = t.mt * t.nt, T = (int)blockDim.x, tid = (int)threadIdx.x;
    const int eb = t.w_off[r0], E = t.w_off[r0 + nprod] - eb;
    const uint32_t me = (uint32_t)((m + t.mt - 1) / t.mt);
    const uint32_t rows = i_rows ? i_rows : me;
    if (P == 1 && E == 1 && nprod == 1) {
        scatter_one_body<FMT>(n, alpha * (double)t.w_ent[2 * eb + 1], beta, Z, e_row, f_col, C, ldc, c0, c1, vb, vg, i_lo,
                              rows);
        return;
    }
    const int TR = T * NC / 4;                                            /* rows per tile */
    const uint32_t tiles_i = (rows + TR - 1) / TR;
    const uint32_t tiles = tiles_i * (uint32_t)((c1 + 3) / 4 - c0 / 4);   /* row tiles fastest */
    constexpr int NH = NC / 2;           /* column pairs of a thread */
    double2* cs = (double2*)sm_all;      /* [P][NH][T] */
    double* lam = sm_all + P * T * NC;   /* [E] */
    int* pidx = (int*)(lam + E);         /* [E] */
    int* off = pidx + E;                 /* [nprod + 1] */
    int4* geo = (int4*)(cs + P * NH * T + (E * 12 + (nprod + 1) * 4 + 15) / 16);   /* [P]: ro, rl, co, cl */
    for (int x = tid; x < E; x += T) {
        pidx[x] = t.w_ent[2 * (eb + x)];
        lam[x] = alpha * (double)t.w_ent[2 * (eb + x) + 1];
    }
    for (int x = tid; x <= nprod; x += T) off[x] = t.w_off[r0 + x] - eb;
    for (int p = tid; p < P; p += T) {
        int4 g;
        fmm_part_geom32((int)m, t.mt, p / t.nt, &g.x, &g.y);
        fmm_part_geom32((int)n, t.nt, p % t.nt, &g.z, &g.w);
        geo[p] = g;
    }
    __syncthreads();
    const int tr = tid % TR, th = tid / TR * NC;     /* row of the tile, first of the thread's columns */
    for (uint32_t x = vb; x < tiles; x += vg) {
        const int i = (int)(i_lo + x % tiles_i * TR) + tr, j = (int)(c0 / 4 + x / tiles_i) * 4 + th;
        if (i >= (int)(i_lo + rows)) continue;
        std::conditional_t<NC == 4, ZRow<FMT>, ZPair<FMT>> z;
        z.load(Z, e_row, f_col, 0, i, j);
        /* elements outside a smaller sub-block or the column range are
         * carried along as zeros and not stored */
        for (int p = 0; p < P; ++p) {
            const int4 g = geo[p];
            const int jl = i < g.y ? min(g.w, c1) : 0;
            const double* cp = C + g.x + i + (int64_t)(g.z + j) * ldc;
            double c[NC];
#pragma unroll
            for (int u = 0; u < NC; ++u) c[u] = j + u >= c0 && j + u < jl ? beta_c(beta, cp + u * ldc) : 0.0;
#pragma unroll
            for (int h = 0; h < NH; ++h) cs[(p * NH + h) * T + tid] = make_double2(c[2 * h], c[2 * h + 1]);
        }
        for (int q = 0; q < nprod; ++q) {
            double M[NC];
            z.values(Z, M);
            if (q + 1 < nprod) z.load(Z, e_row, f_col, q + 1, i, j);   /* in flight under this product's updates */
            /* four values at a time, one sub-block's or two's (a product's are
             * distinct): their loads and FMAs are under way together */
            const int e = off[q + 1];
            for (int y = off[q]; y < e; y += 4 / NC) {
                const bool two = NC == 4 || y + 1 < e;
                double2* c = cs + pidx[y] * NH * T + tid;
                double2* d = NC == 4 ? c + T : cs + pidx[two ? y + 1 : y] * T + tid;
                const double l = lam[y], l2 = NC == 4 ? l : (two ? lam[y + 1] : 0.0);
                double2 a = *c, b = *d;
                a.x = fma(l, M[0], a.x);
                a.y = fma(l, M[1], a.y);
                if (two) {
                    b.x = fma(l2, M[NC - 2], b.x);
                    b.y = fma(l2, M[NC - 1], b.y);
                }
                *c = a;
                if (two) *d = b;
            }
        }
        for (int p = 0; p < P; ++p) {
            const int4 g = geo[p];
            const int jl = i < g.y ? min(g.w, c1) : 0;
            double* cp = C + g.x + i + (int64_t)(g.z + j) * ldc;
            double2 a[NH];
#pragma unroll
            for (int h = 0; h < NH; ++h) a[h] = cs[(p * NH + h) * T + tid];
#pragma unroll
            for (int h = 0; h < NH; ++h) {
                if (j + 2 * h >= c0 && j + 2 * h < jl) cp[2 * h * ldc] = a[h].x;
                if (j + 2 * h + 1 >= c0 && j + 2 * h + 1 < jl) cp[(2 * h + 1) * ldc] = a[h].y;
            }
        }
    }
}

/* columns per thread of the element-major C update of P sub-blocks: see above */
__host__ __device__ __forceinline__ int scatter_cols(int P) { return P <= 6 ? 4 : 2; }

/* its dynamic shared memory: the values of T threads, E entries and nprod offsets of the group, the sub-blocks' places */
size_t scatter_all_smem(int P, int T, int E, int nprod)
{
    return (size_t)P * T * scatter_cols(P) * 8 + ((size_t)E * 12 + (size_t)(nprod + 1) * 4 + 15) / 16 * 16 + (size_t)P * 16;
}

template <int FMT, int NC>
__global__ void __launch_bounds__(256, FMT == 0 ? 0 : NC == 4 ? 3 : 4)
scatter_all_kernel(const int* __restrict__ tab, int r0, int nprod, int64_t m, int64_t n, double alpha, double beta,
                   const ZView Z, const int* __restrict__ e_row, const int* __restrict__ f_col,
                   double* __restrict__ C, int64_t ldc, int c0, int c1, uint32_t i_lo, uint32_t i_rows)
{
    scatter_all_body<FMT, NC>(tab, r0, nprod, m, n, alpha, beta, Z, e_row, f_col, C, ldc, c0, c1, blockIdx.x, gridDim.x,
                              i_lo, i_rows);
}


/* C update of a classical GEMM whose tiles ran as work units: a thread takes
 * a row of a column group, adds each level's planes, rounds and combines the
 * levels into Z and updates C as scatter_all_kernel does. Blocks of 32 rows x
 * 16 columns; reads nunits x 4 bytes per element, mostly from L2. */
__global__ void __launch_bounds__(128)
scatter_units_kernel(int m, int n, double alpha, double beta, const int4* __restrict__ Zp, int m_pad, int n_pad, int s,
                     int nkb, int unit_kb, int nunits, int G, int db, int ebase, const int* __restrict__ e_row,
                     const int* __restrict__ f_col, double* __restrict__ C, int64_t ldc)
{
    const int i = (int)blockIdx.x * 32 + (int)threadIdx.x % 32, j = ((int)blockIdx.y * 4 + (int)threadIdx.x / 32) * 4;
    sm103::grid_wait();
    if (i >= m || j >= n) return;
    double* cp = C + i + (int64_t)j * ldc;
    double c[kScatterCols];
#pragma unroll
    for (int u = 0; u < 4; ++u) c[u] = j + u < n ? beta_c(beta, cp + u * ldc) : 0.0;
    const int er = e_row[i] + ebase;
    const int4 f = *(const int4*)(f_col + j);
    const int fc[4] = {f.x, f.y, f.z, f.w};
    const int4* q = Zp + (int64_t)(j / 4) * m_pad + i;
    const int64_t plane = (int64_t)n_pad / 4 * m_pad;
    int64_t z[kScatterCols] = {0, 0, 0, 0};
    int l[kScatterCols] = {0, 0, 0, 0};
    int g = s + 1, left = level_units(g, s, nkb, unit_kb);
    constexpr int U = 8;   /* planes in flight */
    for (int p0 = 0; p0 < nunits; p0 += U) {
        int4 v[U];
#pragma unroll
        for (int x = 0; x < U; ++x)
            if (p0 + x < nunits) v[x] = q[(p0 + x) * plane];
#pragma unroll
        for (int x = 0; x < U; ++x) {
            if (p0 + x >= nunits) break;
            l[0] += v[x].x;
            l[1] += v[x].y;
            l[2] += v[x].z;
            l[3] += v[x].w;
            if (--left > 0) continue;
#pragma unroll
            for (int u = 0; u < 4; ++u) {   /* the level is complete */
                if (g > G)
                    z[u] += ((l[u] >> (db * (g - G) - 1)) + 1) >> 1;
                else
                    z[u] += (int64_t)((uint64_t)(int64_t)l[u] << (db * (G - g)));
                l[u] = 0;
            }
            --g;
            left = level_units(g, s, nkb, unit_kb);
        }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
        if (j + u < n) cp[u * ldc] = fma(alpha, i64_to_double_scaled(z[u], er + fc[u]), c[u]);
}

/* ------------------------------------- batched waves: side work per wave ---- */

/* A wave of a batch runs each side kernel (C scaling and maxima zeroing,
 * maxima, exponents, packs, C updates) as one launch over all its problems
 * instead of one launch per problem: the problems travel by value in a table
 * (like the GEMM's), each owns a contiguous range of the launch's blocks, and
 * a block finds its problem by binary search and runs the same per-block code
 * (the *_body functions) the single-problem kernels run, so the results are
 * the single calls' bits. */
struct WaveProb {
    const int* tab;
    const double* A;
    const double* B;
    double* C;
    unsigned long long* amax;
    unsigned long long* bmax;
    int* e_row;
    int* f_col;
    uint8_t* sa;
    uint8_t* sb;
    ZView Z;
    int64_t lda, ldb, ldc, m, n, k, m_pad, n_pad, k_pad;
    int64_t b0;   /* the problem's first block in this launch */
    int64_t nb;   /* its blocks */
    int64_t gx;   /* blocks along the first coordinate of its per-problem grid */
    double alpha, beta;
    int R, kt, fmt, tr;   /* tr: rows of a tile of the C updates by sub-block */
};
struct WaveLaunch {
    int nprob;
    WaveProb p[kMaxLaunchProblems];
};
static_assert(sizeof(WaveLaunch) <= 32764, "WaveLaunch must fit the kernel parameter space");

__device__ __forceinline__ int wave_find(const WaveLaunch& W, int64_t b)
{
    int lo = 0, hi = W.nprob - 1;   /* last problem with b0 <= b */
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (W.p[mid].b0 <= b) lo = mid; else hi = mid - 1;
    }
    return lo;
}

/* the maxima arrays zeroed, grid-stride over each problem's range */
__global__ void __launch_bounds__(256) wave_prep_kernel(const __grid_constant__ WaveLaunch W)
{
    const WaveProb& P = W.p[wave_find(W, blockIdx.x)];
    const int64_t vb = blockIdx.x - P.b0;
    const int64_t za = (int64_t)P.kt * P.m, zb = (int64_t)P.kt * P.n;
    for (int64_t x = vb * blockDim.x + threadIdx.x; x < za + zb; x += P.nb * (int64_t)blockDim.x) {
        if (x < za)
            P.amax[x] = 0;
        else
            P.bmax[x - za] = 0;
    }
}

/* row maxima of A (gx blocks: 256 rows x one k part x 256 columns) then column maxima of B */
__global__ void __launch_bounds__(256) wave_maxima_kernel(const __grid_constant__ WaveLaunch W)
{
    const WaveProb& P = W.p[wave_find(W, blockIdx.x)];
    const int64_t vb = blockIdx.x - P.b0;
    if (vb < P.gx) {
        const int64_t rb = (P.m + 255) / 256;
        amax_body(P.A, P.lda, P.m, P.k, P.kt, P.amax, 256, vb % rb, (int)((vb / rb) % P.kt), vb / rb / P.kt);
    } else {
        bmax_body(P.B, P.ldb, P.k, P.n, P.kt, P.bmax, 0, P.n, vb - P.gx);
    }
}

__global__ void __launch_bounds__(256) wave_exps_kernel(const __grid_constant__ WaveLaunch W)
{
    const WaveProb& P = W.p[wave_find(W, blockIdx.x)];
    const int64_t vb = blockIdx.x - P.b0;
    exps_body(P.tab, 0, P.m, P.n, P.k, P.m_pad, P.n_pad, P.amax, P.bmax, P.e_row, P.f_col, 0, P.m_pad + P.n_pad,
              vb % P.gx, (int)(vb / P.gx));
}

template <int S, int DB>
__global__ void __launch_bounds__(256, 4) wave_pack_a_kernel(const __grid_constant__ WaveLaunch W)
{
    const WaveProb& P = W.p[wave_find(W, blockIdx.x)];
    const int64_t vb = blockIdx.x - P.b0;
    pack_a_body<S, DB, 64>(P.tab, 0, P.R, P.A, P.lda, P.m, P.k, P.m_pad, P.k_pad, P.e_row, P.sa, vb % P.gx,
                             vb / P.gx);
}

template <int S, int DB>
__global__ void __launch_bounds__(256, 4) wave_pack_b_kernel(const __grid_constant__ WaveLaunch W)
{
    const WaveProb& P = W.p[wave_find(W, blockIdx.x)];
    const int64_t vb = blockIdx.x - P.b0;
    pack_b_body<S, DB, 32>(P.tab, 0, P.R, P.B, P.ldb, P.k, P.n, P.n_pad, P.k_pad, P.f_col, P.sb, 0, vb % P.gx,
                             vb / P.gx);
}

/* the classical problems' maxima, exponents and digits (prep_kernel), clusters of nrank CTAs */
template <int S, int DB>
__global__ void __launch_bounds__(kPrepThreads, 3) wave_classical_kernel(const __grid_constant__ WaveLaunch W, int nrank)
{
    __shared__ PrepShared sh;
    const WaveProb& P = W.p[wave_find(W, blockIdx.x)];
    const int64_t c = (blockIdx.x - P.b0) / nrank, ca = P.m_pad / kPrepLines;
    const int rank = (int)(blockIdx.x % (unsigned)nrank);
    if (c < ca)
        prep_body<S, DB, true>(sh, P.A, P.lda, P.m, P.k, P.m_pad, P.k_pad, P.e_row, P.sa, c * kPrepLines, rank, nrank);
    else
        prep_body<S, DB, false>(sh, P.B, P.ldb, P.n, P.k, P.n_pad, P.k_pad, P.f_col, P.sb, (c - ca) * kPrepLines, rank,
                                nrank);
}

/* the C updates of the classical problems of a wave */
__global__ void __launch_bounds__(256, 4) wave_scatter_one_kernel(const __grid_constant__ WaveLaunch W)
{
    const WaveProb& P = W.p[wave_find(W, blockIdx.x)];
    const uint32_t vb = (uint32_t)(blockIdx.x - P.b0), vg = (uint32_t)P.nb;
    if (P.fmt)
        scatter_one_body<1>(P.n, P.alpha, P.beta, P.Z, P.e_row, P.f_col, P.C, P.ldc, 0, (int)P.n, vb, vg, 0, (uint32_t)P.m);
    else
        scatter_one_body<0>(P.n, P.alpha, P.beta, P.Z, P.e_row, P.f_col, P.C, P.ldc, 0, (int)P.n, vb, vg, 0, (uint32_t)P.m);
}

/* the others', in the element-major form */
__global__ void __launch_bounds__(256, 4) wave_scatter_kernel(const __grid_constant__ WaveLaunch W)
{
    const WaveProb& P = W.p[wave_find(W, blockIdx.x)];
    const uint32_t vb = (uint32_t)(blockIdx.x - P.b0), vg = (uint32_t)P.nb;
    const int nt = P.tab[2], c1 = (int)((P.n + nt - 1) / nt);
    auto go = [&](auto F, auto N) {
        scatter_all_body<decltype(F)::value, decltype(N)::value>(P.tab, 0, P.R, P.m, P.n, P.alpha, P.beta, P.Z,
                                                                 P.e_row, P.f_col, P.C, P.ldc, 0, c1, vb, vg);
    };
    constexpr std::integral_constant<int, 0> bf16{};
    constexpr std::integral_constant<int, 1> fp8{};
    constexpr std::integral_constant<int, 2> pair{};
    constexpr std::integral_constant<int, 4> row{};
    if (scatter_cols(P.tab[0] * nt) == 4) {
        if (P.fmt) go(fp8, row); else go(bf16, row);
    } else {
        if (P.fmt) go(fp8, pair); else go(bf16, pair);
    }
}

/* the rest, by sub-block: gx tiles for each */
__global__ void __launch_bounds__(kScatterThreads, 8) wave_scatter_part_kernel(const __grid_constant__ WaveLaunch W)
{
    __shared__ ScatterEntries sh;
    const WaveProb& P = W.p[wave_find(W, blockIdx.x)];
    const int64_t vb = blockIdx.x - P.b0;
    const int p = (int)(vb / P.gx);
    const uint32_t bx = (uint32_t)(vb % P.gx);
    if (P.fmt)
        scatter_part_body<1, false>(sh, P.tab, 0, P.R, P.m, P.n, P.alpha, P.beta, P.Z, P.e_row, P.f_col, P.C, P.ldc, P.tr, p, bx);
    else
        scatter_part_body<0, false>(sh, P.tab, 0, P.R, P.m, P.n, P.alpha, P.beta, P.Z, P.e_row, P.f_col, P.C, P.ldc, P.tr, p, bx);
}

/* --------------------------------------------------------- host -------- */

PFN_cuTensorMapEncodeTiled_v12000 get_encode_fn()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, []() {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
    });
    return fn;
}

/* 2-D map over slices[rows_total][k_pad] of BF16 (fmt 0) or FP8-E4M3 bytes
 * (fmt 1): boxes one 128-byte row of k (64 or 128 elements) by box_rows rows,
 * 128-byte swizzle. */
int make_slice_map(CUtensorMap* map, const void* base, int64_t k_pad, int64_t rows_total, int box_rows, int fmt)
{
    PFN_cuTensorMapEncodeTiled_v12000 enc = get_encode_fn();
    if (!enc) return FMM_ERR_CUDA;
    const int esz = fmt ? 1 : 2;                         /* FP8-E4M3 bytes or BF16 */
    cuuint64_t dims[2] = {(cuuint64_t)k_pad, (cuuint64_t)rows_total};
    cuuint64_t strides[1] = {(cuuint64_t)(k_pad * esz)};
    cuuint32_t box[2] = {(cuuint32_t)(128 / esz), (cuuint32_t)box_rows};   /* 128-byte rows */
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(map, fmt ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                     const_cast<void*>(base), dims, strides, box,
                     estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? FMM_OK : FMM_ERR_CUDA;
}

/* Products are processed in groups: all products of a group are packed, then
 * one GEMM launch covers every (product, tile) work item of the group, then
 * one scatter pass updates C. The group size is the largest that keeps the
 * per-group workspace (slices + Z) under kGroupBudget. */
constexpr size_t kGroupBudget = (size_t)32 << 30;

/* SMs of the GPU that the rules below were measured on (launches ask the device for its own) */
constexpr int64_t kSms = 152;

struct Dims {
    int64_t me, ne, ke, m_pad, n_pad, k_pad;
};

/* k elements per 128-byte stage row of a slice format */
inline int kbe_of(int fmt) { return fmt ? 128 : kBK; }

Dims dims_of(const AlgView& alg, int64_t m, int64_t n, int64_t k, int fmt = 0)
{
    Dims d;
    d.me = (m + alg.mt - 1) / alg.mt;
    d.ne = (n + alg.nt - 1) / alg.nt;
    d.ke = (k + alg.kt - 1) / alg.kt;
    /* rows padded to the 256-row pair tiles once m_e >= 1024 (at most 25%
     * padding there); any multiple of 128 also serves the single-CTA kernel */
    d.m_pad = round_up(std::max<int64_t>(d.me, 1), d.me >= kPairMinRows ? kPairTileM : kTileM);
    d.n_pad = round_up(std::max<int64_t>(d.ne, 1), kTileN);
    d.k_pad = round_up(std::max<int64_t>(d.ke, 1), kbe_of(fmt));
    return d;
}

/* G, the level whose unit Z counts in: BF16 6, or 7 when k_pad <= 128 (the
 * finest unit keeping Z inside int64); FP8 s + 1 up to 10 (exact for s <= 9) */
int zlevel_of(const Dims& d, int s, int fmt)
{
    if (fmt) return std::min(s + 1, 10);
    return d.k_pad <= 128 ? 7 : 6;
}

/* bytes of one product's Z planes */
size_t z_bytes(const Dims& d, int s, int fmt)
{
    return (size_t)d.n_pad / 4 * (size_t)z_group_bytes(d.m_pad, ZPlanes::of(s, zlevel_of(d, s, fmt), fmt).nd);
}

size_t per_product_bytes(const Dims& d, int s, int fmt)
{
    return (fmt ? 1 : 2) * (size_t)s * (size_t)(d.m_pad + d.n_pad) * (size_t)d.k_pad + z_bytes(d, s, fmt) +
           4 * (size_t)(d.m_pad + d.n_pad) + 1024;
}

int group_size(const AlgView& alg, const Dims& d, int s, size_t budget, int fmt)
{
    const size_t per = per_product_bytes(d, s, fmt);
    size_t g = budget / per;
    if (g < 1) g = 1;
    if (g > (size_t)alg.R) g = (size_t)alg.R;
    /* tensor-map row coordinates are 32-bit */
    while (g > 1 && (int64_t)g * s * std::max(d.m_pad, d.n_pad) > 0x7fffffffLL) --g;
    return (int)g;
}

struct WsLayout {
    size_t amax, bmax, sched, erow, fcol, sa, sb, z, total;
    int group;
};

WsLayout ws_layout_g(const AlgView& alg, const Dims& d, int64_t m, int64_t n, int s, int G, int fmt)
{
    const size_t esz = fmt ? 1 : 2;
    WsLayout L;
    size_t off = 0;
    auto take = [&](size_t bytes) { size_t o = off; off += (bytes + 255) / 256 * 256; return o; };
    L.group = G;
    L.amax = take(sizeof(unsigned long long) * (size_t)alg.kt * (size_t)m);
    L.bmax = take(sizeof(unsigned long long) * (size_t)alg.kt * (size_t)n);
    L.sched = take(2 * sizeof(unsigned int));   /* work-item counters of GEMM launches in flight together */
    L.erow = take(sizeof(int) * (size_t)G * (size_t)d.m_pad);
    L.fcol = take(sizeof(int) * (size_t)G * (size_t)d.n_pad);
    L.sa = take(esz * (size_t)G * s * (size_t)d.m_pad * (size_t)d.k_pad);
    L.sb = take(esz * (size_t)G * s * (size_t)d.n_pad * (size_t)d.k_pad);
    L.z = take((size_t)G * z_bytes(d, s, fmt));
    L.total = off;
    return L;
}

/* Layout for the largest product group whose whole workspace fits in
 * `budget` bytes (at least one product). */
WsLayout ws_layout(const AlgView& alg, int64_t m, int64_t n, int64_t k, int s, size_t budget = kGroupBudget,
                   int fmt = 0)
{
    const Dims d = dims_of(alg, m, n, k, fmt);
    int G = group_size(alg, d, s, budget, fmt);
    WsLayout L = ws_layout_g(alg, d, m, n, s, G, fmt);
    while (G > 1 && L.total > budget) L = ws_layout_g(alg, d, m, n, s, --G, fmt);
    return L;
}

/* Work units of a classical GEMM (UnitSpan), for a product grid whose tiles
 * leave SMs idle: the units per tile that the model below finds cheapest, none
 * when whole tiles do as well (planes of at most kUnitBytes). A k block costs about 760 clocks on the single-SM kernel and 640 on
 * CTA pairs, a unit or tile 3000 beside them, the extra planes the C update
 * reads about one clock per 2000 bytes. 300 x 700 x 450, 6 slices: 9 tiles of
 * 168 k blocks, 71 us; as 9 x 17 units 14 us. */
constexpr size_t kUnitBytes = (size_t)128 << 20;

struct UnitPlan {
    int nunits = 0, unit_kb = 0;
    size_t bytes = 0;
};

UnitPlan unit_plan(const Dims& d, int s, int fmt, bool pair)
{
    constexpr int64_t sms = kSms;
    constexpr double kb_single = 760, kb_pair = 640, per_unit = 3000, bytes_per_clk = 2000;
    const int64_t tiles = d.m_pad / kTileM * (d.n_pad / kTileN);
    const int nkb = (int)(d.k_pad / kbe_of(fmt));
    UnitPlan best;
    if (tiles >= sms) return best;
    const size_t plane = 4 * (size_t)d.m_pad * (size_t)d.n_pad;
    const double all = (double)nkb * s * (s + 1) / 2;
    double least = all * kb_single + per_unit;   /* one round of whole tiles */
    if (pair) least = (double)((tiles / 2 + sms / 2 - 1) / (sms / 2)) * (all * kb_pair + per_unit);
    least *= 0.9;
    for (int parts = 2; parts <= 64; ++parts) {
        const int T = std::max(2, (int)((all + parts - 1) / parts));
        int nu = 0, longest = 0;
        for (int g = s + 1; g >= 2; --g) {
            const int cnt = level_units(g, s, nkb, T), lk = level_pairs(g, s) * nkb;
            nu += cnt;
            longest = std::max(longest, (lk + cnt - 1) / cnt);
        }
        if (nu * plane > kUnitBytes) continue;
        const double t = (double)((tiles * nu + sms - 1) / sms) * (longest * kb_single + per_unit) +
                         (double)(nu - 2) * (double)plane / bytes_per_clk;
        if (t < least) {
            least = t;
            best.nunits = nu;
            best.unit_kb = T;
            best.bytes = (size_t)nu * plane;
        }
    }
    return best;
}

/* opt-in event timing of the GEMM launches */
std::mutex g_timing_mu;
bool g_timing = false;
std::vector<std::pair<cudaEvent_t, cudaEvent_t>> g_pending, g_pool;
uint64_t g_timed_products = 0;

void timing_mark(cudaStream_t st, bool before)
{
    static thread_local std::pair<cudaEvent_t, cudaEvent_t> cur;
    std::lock_guard<std::mutex> lk(g_timing_mu);
    if (before) {
        if (g_pool.empty()) {
            cudaEvent_t a, b;
            cudaEventCreate(&a);
            cudaEventCreate(&b);
            g_pool.push_back({a, b});
        }
        cur = g_pool.back();
        g_pool.pop_back();
        cudaEventRecord(cur.first, st);
    } else {
        cudaEventRecord(cur.second, st);
        g_pending.push_back(cur);
    }
}

}  // namespace

extern "C" int fmm_gpu_set_split_pair_rows(int min_rows)
{
    return g_pair_rows.exchange(std::max(min_rows, kPairMinRows));
}

extern "C" void fmm_gpu_set_kernel_timing(int enable)
{
    std::lock_guard<std::mutex> lk(g_timing_mu);
    g_timing = enable != 0;
}

extern "C" int fmm_gpu_read_kernel_timing(double* total_ms, uint64_t* launches, uint64_t* products)
{
    std::lock_guard<std::mutex> lk(g_timing_mu);
    double sum = 0.0;
    int rc = FMM_OK;
    for (auto& pr : g_pending) {
        float ms = 0.f;
        if (cudaEventSynchronize(pr.second) != cudaSuccess ||
            cudaEventElapsedTime(&ms, pr.first, pr.second) != cudaSuccess)
            rc = FMM_ERR_CUDA;
        sum += ms;
        g_pool.push_back(pr);
    }
    if (launches) *launches = g_pending.size();
    if (products) *products = g_timed_products;
    if (total_ms) *total_ms = sum;
    g_pending.clear();
    g_timed_products = 0;
    return rc;
}

size_t fmm_split_ws_bytes(const AlgView& alg, int64_t m, int64_t n, int64_t k, int slices, int fmt)
{
    const WsLayout L = ws_layout(alg, m, n, k, slices, kGroupBudget, fmt);
    if (L.group < alg.R) return L.total;
    /* room for the two overlapping product groups when they fit the budget */
    const Dims d = dims_of(alg, m, n, k, fmt);
    const int G1 = (alg.R + 1) / 2;
    if (alg.R < 2) return L.total;
    const WsLayout L1 = ws_layout_g(alg, d, m, n, slices, G1, fmt);
    const size_t two = L1.total + (L1.total - L1.erow);
    return two <= kGroupBudget ? std::max(L.total, two) : L.total;
}

/* the same with room for a classical problem's work units (whichever way the
 * pair threshold stands at the call) */
size_t fmm_split_full_ws_bytes(const AlgView& alg, int64_t m, int64_t n, int64_t k, int slices, int fmt)
{
    const size_t b = fmm_split_ws_bytes(alg, m, n, k, slices, fmt);
    if (m == 0 || n == 0 || k == 0 || alg.R != 1 || alg.mt != 1 || alg.kt != 1 || alg.nt != 1) return b;
    const Dims d = dims_of(alg, m, n, k, fmt);
    return b + std::max(unit_plan(d, slices, fmt, false).bytes, unit_plan(d, slices, fmt, true).bytes);
}

/* One split-form GEMM problem being executed: its algorithm, geometry,
 * operands and the part of the workspace it uses. */
struct SplitJob {
    AlgView alg;
    Dims d;
    int64_t m, n, k;
    double alpha, beta;
    const double* A;
    int64_t lda;
    const double* B;
    int64_t ldb;
    double* C;
    int64_t ldc;
    int s;
    int fmt;       /* 0: BF16 slices, 1: FP8-E4M3 slices */
    bool trivial;  /* nothing beyond C := beta*C */
    bool classical; /* one product of coefficient 1: prep_kernel forms its operands */
    WsLayout L;
    uint8_t* w;
    uint8_t* z;    /* the group's Z planes; null: outside the workspace (job_bind) */
};

static int job_init(SplitJob& j, const AlgView& alg, int64_t m, int64_t n, int64_t k, double alpha,
                    const double* A, int64_t lda, const double* B, int64_t ldb, double beta, double* C,
                    int64_t ldc, int s, int fmt = 0)
{
    if (fmt != 0 && fmt != 1) return FMM_ERR_ARG;
    if (s < 2 || s > (fmt ? 12 : 8)) return FMM_ERR_ARG;
    j.fmt = fmt;
    j.alg = alg;
    j.m = m; j.n = n; j.k = k;
    j.alpha = alpha; j.beta = beta;
    j.A = A; j.lda = lda; j.B = B; j.ldb = ldb; j.C = C; j.ldc = ldc;
    j.s = s;
    j.w = j.z = nullptr;
    j.trivial = m == 0 || n == 0 || k == 0 || alpha == 0.0;
    j.classical = fmm_plain_classical(alg);
    if (j.trivial) return FMM_OK;
    if (alg.max_nnz_u > kPackMaxEnt || alg.max_nnz_v > kPackMaxEnt) return FMM_ERR_UNSUPPORTED;
    if (m > 0x7fffffffLL || n > 0x7fffffffLL) return FMM_ERR_UNSUPPORTED;
    j.d = dims_of(alg, m, n, k, fmt);
    if (j.d.ke > kMaxKe) return FMM_ERR_UNSUPPORTED;
    if (j.d.me * j.d.ne > 0xffffffffLL) return FMM_ERR_UNSUPPORTED;
    /* the scatter keeps one C part's W entries of a group in shared memory */
    const Tab ht = tab_view(alg.htab);
    for (int p = 0; p < alg.mt * alg.nt; ++p)
        if (ht.wp_off[p + 1] - ht.wp_off[p] > kScatterMaxEnt) return FMM_ERR_UNSUPPORTED;
    return FMM_OK;
}

/* Workspace of the job for a product group within `budget` bytes. The least
 * accepted holds one product with 8 bytes of Z per element; FP8 Z planes of 7
 * slices and more need 9 to 11, and where they do not fit j.z stays null. */
static int job_bind(SplitJob& j, void* ws, size_t ws_bytes, size_t budget)
{
    if (j.trivial) return FMM_OK;
    j.L = ws_layout(j.alg, j.m, j.n, j.k, j.s, budget, j.fmt);
    if ((int64_t)j.L.group * j.s * std::max(j.d.m_pad, j.d.n_pad) > 0x7fffffffLL) return FMM_ERR_UNSUPPORTED;
    const size_t least = j.L.group > 1 ? j.L.total
                                       : std::min(j.L.total, j.L.z + 8 * (size_t)j.d.m_pad * (size_t)j.d.n_pad);
    if (ws == nullptr || ws_bytes < least) return FMM_ERR_WORKSPACE;
    if (((uintptr_t)ws & 255) != 0) return FMM_ERR_ARG;
    j.w = (uint8_t*)ws;
    j.z = ws_bytes < j.L.total ? nullptr : j.w + j.L.z;
    return FMM_OK;
}

/* workspace of the job for a group of exactly G products */
static int job_bind_group(SplitJob& j, void* ws, size_t ws_bytes, int G)
{
    if (j.trivial) return FMM_OK;
    j.L = ws_layout_g(j.alg, j.d, j.m, j.n, j.s, G, j.fmt);
    if ((int64_t)j.L.group * j.s * std::max(j.d.m_pad, j.d.n_pad) > 0x7fffffffLL) return FMM_ERR_UNSUPPORTED;
    if (ws == nullptr || ws_bytes < j.L.total) return FMM_ERR_WORKSPACE;
    if (((uintptr_t)ws & 255) != 0) return FMM_ERR_ARG;
    j.w = (uint8_t*)ws;
    j.z = j.w + j.L.z;
    return FMM_OK;
}

/* Side streams: in a batch wave, the per-problem work (maxima, exponents,
 * packs, scatter) of different problems, so their small kernels overlap
 * instead of queueing behind each other on the caller's stream; in a single
 * call, the B-side maxima and pack beside the A-side ones. Created once per
 * device; forked from and joined back to the caller's stream with events,
 * which a stream capture follows. One call at a time uses a pool (g_side_use). */
/* Timeline of the last host-buffer call (fmm_gpu_set_host_timeline): device
 * times, from the first copy's start, of A on the device, B on the device,
 * the first GEMM launch's start, the last GEMM launch's end, C's last column
 * chunk back on the host; plus the call's host wall time. A call without
 * overlapped schedule has the start and end of its whole device part for the
 * GEMM's. */
constexpr int kTimelinePoints = 5;
std::atomic<bool> g_timeline{false};
std::mutex g_timeline_mu;
double g_timeline_ms[kTimelinePoints + 1] = {0, 0, 0, 0, 0, 0};

constexpr int kWaveStreams = 8;                  /* batched waves: pack streams, then scatter streams */
constexpr int kSideStreams = 2 * kWaveStreams;

struct SidePool {
    int device;
    cudaStream_t s[kSideStreams];
    cudaEvent_t fork;
    cudaEvent_t join[kSideStreams];
    cudaEvent_t wave_pk[2][kWaveStreams];   /* a workspace half's packs done */
    cudaEvent_t wave_gm[2];                 /* a workspace half's GEMM done */
    cudaEvent_t wave_sc[2][kWaveStreams];   /* a workspace half's C updates done */
    cudaEvent_t gate[3];   /* host-buffer calls: A, B and C on the device */
    cudaEvent_t chunk[32]; /* host-buffer calls: B chunks in (0..7), C chunks out (8..31) */
    cudaEvent_t blk[16];   /* host-buffer calls, blocked schedule: A halves up, A halves and B parts packed, GEMM blocks done */
    cudaEvent_t tl[kTimelinePoints + 1];  /* host-buffer calls: the call's timeline (timing events) */
    cudaStream_t hi;       /* greatest priority: GEMMs that side work runs beside */
    cudaStream_t top[3];   /* greatest priority: side work that runs between GEMMs (host-buffer calls) */
};

std::mutex g_side_mu, g_side_use;
std::vector<SidePool*> g_side;

SidePool* side_pool()
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    std::lock_guard<std::mutex> lk(g_side_mu);
    for (SidePool* p : g_side)
        if (p->device == dev) return p;
    SidePool* p = new SidePool;
    p->device = dev;
    int least = 0, greatest = 0;
    cudaDeviceGetStreamPriorityRange(&least, &greatest);
    bool ok = cudaEventCreateWithFlags(&p->fork, cudaEventDisableTiming) == cudaSuccess &&
              cudaStreamCreateWithPriority(&p->hi, cudaStreamNonBlocking, greatest) == cudaSuccess;
    for (int i = 0; i < 3 && ok; ++i)
        ok = cudaStreamCreateWithPriority(&p->top[i], cudaStreamNonBlocking, greatest) == cudaSuccess;
    for (int i = 0; i < 3 && ok; ++i) ok = cudaEventCreateWithFlags(&p->gate[i], cudaEventDisableTiming) == cudaSuccess;
    for (int i = 0; i <= kTimelinePoints && ok; ++i) ok = cudaEventCreate(&p->tl[i]) == cudaSuccess;
    for (int i = 0; i < 32 && ok; ++i) ok = cudaEventCreateWithFlags(&p->chunk[i], cudaEventDisableTiming) == cudaSuccess;
    for (int i = 0; i < 16 && ok; ++i) ok = cudaEventCreateWithFlags(&p->blk[i], cudaEventDisableTiming) == cudaSuccess;
    for (int h = 0; h < 2 && ok; ++h) {
        ok = cudaEventCreateWithFlags(&p->wave_gm[h], cudaEventDisableTiming) == cudaSuccess;
        for (int i = 0; i < kWaveStreams && ok; ++i)
            ok = cudaEventCreateWithFlags(&p->wave_pk[h][i], cudaEventDisableTiming) == cudaSuccess &&
                 cudaEventCreateWithFlags(&p->wave_sc[h][i], cudaEventDisableTiming) == cudaSuccess;
    }
    for (int i = 0; i < kSideStreams && ok; ++i)
        ok = cudaStreamCreateWithFlags(&p->s[i], cudaStreamNonBlocking) == cudaSuccess &&
             cudaEventCreateWithFlags(&p->join[i], cudaEventDisableTiming) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        return nullptr;   /* the batch then runs on the caller's stream alone */
    }
    g_side.push_back(p);
    return p;
}

int side_fork(SidePool* p, cudaStream_t st)
{
    if (!p) return FMM_OK;
    if (cudaEventRecord(p->fork, st) != cudaSuccess) return FMM_ERR_CUDA;
    for (int i = 0; i < kSideStreams; ++i)
        if (cudaStreamWaitEvent(p->s[i], p->fork, 0) != cudaSuccess) return FMM_ERR_CUDA;
    return FMM_OK;
}

int side_join(SidePool* p, cudaStream_t st)
{
    if (!p) return FMM_OK;
    for (int i = 0; i < kSideStreams; ++i)
        if (cudaEventRecord(p->join[i], p->s[i]) != cudaSuccess || cudaStreamWaitEvent(st, p->join[i], 0) != cudaSuccess)
            return FMM_ERR_CUDA;
    return FMM_OK;
}

/* one side stream (s[0]) beside the caller's stream */
int side_fork1(SidePool* p, cudaStream_t st)
{
    if (cudaEventRecord(p->fork, st) != cudaSuccess) return FMM_ERR_CUDA;
    return cudaStreamWaitEvent(p->s[0], p->fork, 0) == cudaSuccess ? FMM_OK : FMM_ERR_CUDA;
}

int side_join1(SidePool* p, cudaStream_t st)
{
    if (cudaEventRecord(p->join[0], p->s[0]) != cudaSuccess) return FMM_ERR_CUDA;
    return cudaStreamWaitEvent(st, p->join[0], 0) == cudaSuccess ? FMM_OK : FMM_ERR_CUDA;
}

/* per-sub-block row maxima of A (amax) */
static int job_maxima_a(SplitJob& j, cudaStream_t st)
{
    unsigned long long* amax = (unsigned long long*)(j.w + j.L.amax);
    if (cudaMemsetAsync(amax, 0, sizeof(unsigned long long) * (size_t)j.alg.kt * (size_t)j.m, st) != cudaSuccess)
        return FMM_ERR_CUDA;
    /* columns per block: 256, halved (down to 32) while the grid has fewer
     * than 8 blocks per SM, so short-and-wide A still fills the GPU */
    const int64_t rows_blocks = (j.m + 255) / 256 * j.alg.kt;
    int cpb = 256;
    while (cpb > 32 && rows_blocks * ((j.d.ke + cpb - 1) / cpb) < 8 * kSms) cpb /= 2;
    dim3 grid((unsigned)((j.m + 255) / 256), (unsigned)j.alg.kt, (unsigned)((j.d.ke + cpb - 1) / cpb));
    amax_kernel<<<grid, 256, 0, st>>>(j.A, j.lda, j.m, j.k, j.alg.kt, amax, cpb, 0, j.m);
    fmm_count_launch(1);
    return FMM_OK;
}

/* per-sub-block column maxima of B (bmax) for the B columns [c0, c1) */
static void job_maxima_b(SplitJob& j, cudaStream_t st, int64_t c0 = 0, int64_t c1 = -1)
{
    if (c1 < 0) c1 = j.n;
    if (c1 <= c0) return;
    unsigned long long* bmax = (unsigned long long*)(j.w + j.L.bmax);
    const int64_t warps = (c1 - c0) * j.alg.kt;
    bmax_kernel<<<(unsigned)((warps * 32 + 255) / 256), 256, 0, st>>>(j.B, j.ldb, j.k, j.n, j.alg.kt, bmax, c0,
                                                                      c1);
    fmm_count_launch(1);
}

/* the per-sub-block row/column maxima of A and B; with a
 * side pool the B maxima run on its stream s[0], which job_pack joins back */
static int job_prologue(SplitJob& j, cudaStream_t st, SidePool* sp = nullptr)
{
    int rc;
    if (j.trivial) return fmm_scale_c(j.m, j.n, j.beta, j.C, j.ldc, st);   /* else beta goes with the C updates */
    if ((rc = job_maxima_a(j, st)) != FMM_OK) return rc;
    if (sp && (rc = side_fork1(sp, st)) != FMM_OK) return rc;
    job_maxima_b(j, sp ? sp->s[0] : st);
    return FMM_OK;
}

/* exponents and digit slices of products [r0, r0 + np); np never exceeds
 * the group the job's workspace was laid out for */
static int job_pack(SplitJob& j, int r0, int np, cudaStream_t st, SidePool* sp = nullptr, bool small = false)
{
    if (np > j.L.group) return FMM_ERR_WORKSPACE;
    const Dims& d = j.d;
    unsigned long long* amax = (unsigned long long*)(j.w + j.L.amax);
    unsigned long long* bmax = (unsigned long long*)(j.w + j.L.bmax);
    int* e_row = (int*)(j.w + j.L.erow);
    int* f_col = (int*)(j.w + j.L.fcol);
    uint8_t* sa = j.w + j.L.sa;
    uint8_t* sb = j.w + j.L.sb;
    if (np <= 0) return FMM_OK;
    /* one launch per kernel for the whole group (grid y holds the product of
     * the exponent pass; the pack grids' x extent np * tiles stays far below
     * 2^31 since np * s * max(m_pad, n_pad) < 2^31) */
    /* A side (row exponents, A slices) on st; B side (column exponents, B
     * slices) on the side stream, after the B maxima queued there */
    cudaStream_t stb = sp ? sp->s[0] : st;
    exps_kernel<<<dim3((unsigned)((d.m_pad + 255) / 256), (unsigned)np), 256, 0, st>>>(
        j.alg.tab, r0, j.m, j.n, j.k, d.m_pad, d.n_pad, amax, bmax, e_row, f_col, 0, d.m_pad);
    int rc;
    if (sp && (rc = side_fork1(sp, st)) != FMM_OK) return rc;
    exps_kernel<<<dim3((unsigned)((d.n_pad + 255) / 256), (unsigned)np), 256, 0, stb>>>(
        j.alg.tab, r0, j.m, j.n, j.k, d.m_pad, d.n_pad, amax, bmax, e_row, f_col, d.m_pad, d.m_pad + d.n_pad);
    PackSel sel;
    sel.small = small;
    launch_packs(j.fmt, j.s, j.alg.tab, r0, np, j.A, j.lda, j.B, j.ldb, j.m, j.n, j.k, d.m_pad, d.n_pad, d.k_pad, e_row,
                 f_col, sa, sb, st, stb, sel);
    if (sp && (rc = side_join1(sp, st)) != FMM_OK) return rc;
    fmm_count_launch(4);
    return FMM_OK;
}

/* The two sides of job_pack separately, for a caller that receives B in
 * column chunks: the A side (row exponents, A slices) and the B side over
 * the T_r columns [j0, j1) (multiples of 32, or j1 = n_pad). */
static void job_pack_a(SplitJob& j, int r0, int np, cudaStream_t st)
{
    const Dims& d = j.d;
    exps_kernel<<<dim3((unsigned)((d.m_pad + 255) / 256), (unsigned)np), 256, 0, st>>>(
        j.alg.tab, r0, j.m, j.n, j.k, d.m_pad, d.n_pad, (unsigned long long*)(j.w + j.L.amax),
        (unsigned long long*)(j.w + j.L.bmax), (int*)(j.w + j.L.erow), (int*)(j.w + j.L.fcol), 0, d.m_pad);
    PackSel sel;
    sel.b = false;
    launch_packs(j.fmt, j.s, j.alg.tab, r0, np, j.A, j.lda, j.B, j.ldb, j.m, j.n, j.k, d.m_pad, d.n_pad, d.k_pad,
                 (int*)(j.w + j.L.erow), (int*)(j.w + j.L.fcol), j.w + j.L.sa, j.w + j.L.sb, st, st, sel);
    fmm_count_launch(2);
}

static void job_pack_b_cols(SplitJob& j, int r0, int np, int64_t j0, int64_t j1, cudaStream_t st)
{
    const Dims& d = j.d;
    if (j1 <= j0) return;
    exps_kernel<<<dim3((unsigned)((j1 - j0 + 255) / 256), (unsigned)np), 256, 0, st>>>(
        j.alg.tab, r0, j.m, j.n, j.k, d.m_pad, d.n_pad, (unsigned long long*)(j.w + j.L.amax),
        (unsigned long long*)(j.w + j.L.bmax), (int*)(j.w + j.L.erow), (int*)(j.w + j.L.fcol), d.m_pad + j0,
        d.m_pad + j1);
    PackSel sel;
    sel.a = false;
    sel.jb0 = j0;
    sel.jb1 = j1;
    launch_packs(j.fmt, j.s, j.alg.tab, r0, np, j.A, j.lda, j.B, j.ldb, j.m, j.n, j.k, d.m_pad, d.n_pad, d.k_pad,
                 (int*)(j.w + j.L.erow), (int*)(j.w + j.L.fcol), j.w + j.L.sa, j.w + j.L.sb, st, st, sel);
    fmm_count_launch(2);
}

/* per-sub-block row maxima of A (amax, zeroed beforehand) for the
 * product-grid rows [a, b): the A rows ro_p + [a, b) of every row part p */
static void job_maxima_a_rows(SplitJob& j, cudaStream_t st, int64_t a, int64_t b)
{
    unsigned long long* amax = (unsigned long long*)(j.w + j.L.amax);
    for (int p = 0; p < j.alg.mt; ++p) {
        int64_t ro, rl;
        fmm_part_geom(j.m, j.alg.mt, p, &ro, &rl);
        const int64_t r0 = ro + std::min(a, rl), r1 = ro + std::min(b, rl);
        if (r1 <= r0) continue;
        const int64_t rows_blocks = (r1 - r0 + 255) / 256 * j.alg.kt;
        int cpb = 256;
        while (cpb > 32 && rows_blocks * ((j.d.ke + cpb - 1) / cpb) < 8 * kSms) cpb /= 2;
        dim3 grid((unsigned)((r1 - r0 + 255) / 256), (unsigned)j.alg.kt, (unsigned)((j.d.ke + cpb - 1) / cpb));
        amax_kernel<<<grid, 256, 0, st>>>(j.A, j.lda, j.m, j.k, j.alg.kt, amax, cpb, r0, r1);
        fmm_count_launch(1);
    }
}

/* row exponents and A slices of the products r0 .. r0+np-1 for the S_r rows
 * [a, b) (multiples of 64, or b = m_pad) */
static void job_pack_a_rows(SplitJob& j, int r0, int np, int64_t a, int64_t b, cudaStream_t st)
{
    const Dims& d = j.d;
    if (b <= a) return;
    exps_kernel<<<dim3((unsigned)((b - a + 255) / 256), (unsigned)np), 256, 0, st>>>(
        j.alg.tab, r0, j.m, j.n, j.k, d.m_pad, d.n_pad, (unsigned long long*)(j.w + j.L.amax),
        (unsigned long long*)(j.w + j.L.bmax), (int*)(j.w + j.L.erow), (int*)(j.w + j.L.fcol), a, b);
    PackSel sel;
    sel.b = false;
    sel.ia0 = a;
    sel.ia1 = b;
    launch_packs(j.fmt, j.s, j.alg.tab, r0, np, j.A, j.lda, j.B, j.ldb, j.m, j.n, j.k, d.m_pad, d.n_pad, d.k_pad,
                 (int*)(j.w + j.L.erow), (int*)(j.w + j.L.fcol), j.w + j.L.sa, j.w + j.L.sb, st, st, sel);
    fmm_count_launch(2);
}

static int job_zlevel(const SplitJob& j) { return zlevel_of(j.d, j.s, j.fmt); }
static int job_db(const SplitJob& j) { return j.fmt ? 5 : 8; }
/* exponent of Z's unit relative to 2^(E_i + F_j) */
static int job_ebase(const SplitJob& j) { return 2 - job_db(j) * job_zlevel(j); }

/* the job's Z planes for the C updates */
static ZView job_zview(const SplitJob& j)
{
    ZView v;
    v.base = j.z;
    v.prod = (int64_t)z_bytes(j.d, j.s, j.fmt);
    v.nd = ZPlanes::of(j.s, job_zlevel(j), j.fmt).nd;
    v.group = z_group_bytes(j.d.m_pad, v.nd);
    v.m_pad = (int)j.d.m_pad;
    v.n_pad = (int)j.d.n_pad;
    v.ebase = job_ebase(j);
    return v;
}

/* the job's product group as one problem of a GEMM launch */
/* pair tiles for this job's single-call GEMM launches */
static bool job_pair(const SplitJob& j)
{
    return j.d.me >= g_pair_rows.load(std::memory_order_relaxed) && j.d.m_pad % kPairTileM == 0;
}

/* products [r_first, r_first + np) of the job's group as one problem of a
 * GEMM launch: the tensor maps and Z start at product r_first */
static int job_fill(const SplitJob& j, GemmProblem& gp, int np, int item_begin, bool pair = false, int r_first = 0)
{
    const Dims& d = j.d;
    const size_t esz = j.fmt ? 1 : 2;
    const uint8_t* sa = j.w + j.L.sa + (size_t)r_first * j.s * d.m_pad * d.k_pad * esz;
    const uint8_t* sb = j.w + j.L.sb + (size_t)r_first * j.s * d.n_pad * d.k_pad * esz;
    if (make_slice_map(&gp.tmA, sa, d.k_pad, (int64_t)np * j.s * d.m_pad, kTileM, j.fmt) != FMM_OK)
        return FMM_ERR_CUDA;
    if (make_slice_map(&gp.tmB, sb, d.k_pad, (int64_t)np * j.s * d.n_pad, pair ? kTileN / 2 : kTileN, j.fmt) != FMM_OK)
        return FMM_ERR_CUDA;
    gp.Z = j.z + (size_t)r_first * z_bytes(d, j.s, j.fmt);
    gp.s = j.s;
    gp.zlevel = job_zlevel(j);
    const ZPlanes zp = ZPlanes::of(j.s, gp.zlevel, j.fmt);
    gp.zmin = zp.zmin;
    gp.znd = zp.nd;
    gp.zrow0 = 0;
    gp.nunits = gp.unit_kb = 0;
    gp.kbe = kbe_of(j.fmt);
    gp.nkb = (int)(d.k_pad / gp.kbe);
    gp.db = job_db(j);
    gp.fmt = j.fmt;
    gp.m_pad = (int)d.m_pad;
    gp.n_pad = (int)d.n_pad;
    gp.tiles_m = (int)(d.m_pad / (pair ? kPairTileM : kTileM));
    gp.tiles_n = (int)(d.n_pad / kTileN);
    gp.item_begin = item_begin;
    return FMM_OK;
}

static int64_t job_items(const SplitJob& j, int np, bool pair = false)
{
    return (int64_t)np * (j.d.m_pad / (pair ? kPairTileM : kTileM)) * (j.d.n_pad / kTileN);
}

template <class GL>
static int launch_gemm(GL& gl, int64_t nitems, int nprod_timed, cudaStream_t st, bool pair,
                       bool after_prep = false);

/* The GEMM of the job's current product group, as back-to-back launches of
 * at most K products, K the fewest products that give each launch about 24
 * rounds of work items over the GPU. When the kernels took their items round
 * robin, the persistent CTAs drifted apart over a long launch and shared
 * fewer operand panels in L2, and a new launch started them together again
 * (measured at 16384, two Strassen levels: 92-96 ms of GEMM per step in one
 * launch of 49 products, 86-87 ms in launches of 7). With items drawn
 * dynamically the pair kernel measured the same with 2 or 7 launches per
 * step. */
static int job_gemm(const SplitJob& j, int np, cudaStream_t st)
{
    const bool pair = job_pair(j);
    const int64_t tiles = job_items(j, 1, pair);
    const int64_t units = pair ? kSms / 2 : kSms;
    int K = (int)std::min<int64_t>(np, std::max<int64_t>(1, (24 * units + tiles - 1) / tiles));
    const int nl = (np + K - 1) / K;
    K = (np + nl - 1) / nl;
    GemmLaunch1 gl;
    for (int r = 0; r < np; r += K) {
        const int cnt = std::min(K, np - r);
        memset(&gl, 0, sizeof(gl));
        gl.nprob = 1;
        gl.sched = (unsigned int*)(j.w + j.L.sched);
        if (int rc = job_fill(j, gl.prob[0], cnt, 0, pair, r); rc != FMM_OK) return rc;
        if (int rc = launch_gemm(gl, job_items(j, cnt, pair), cnt, st, pair); rc != FMM_OK) return rc;
    }
    return FMM_OK;
}

/* job_gemm restricted to the tile rows [it0, it1) and tile columns
 * [jt0, jt1) of every product: the A slice map starts it0 tile rows
 * further, the B slice map jt0 * 256 rows further and Z at (it0 tile rows,
 * jt0 * 256 columns), with the same row strides, so each (product, tile)
 * item computes exactly what the full launch computes for it. */
static int job_gemm_block(const SplitJob& j, int np, int64_t it0, int64_t it1, int64_t jt0, int64_t jt1,
                          cudaStream_t st, int slot)
{
    const bool pair = job_pair(j);
    const int64_t tm = it1 - it0, tn = jt1 - jt0;
    if (tm <= 0 || tn <= 0) return FMM_OK;
    const int64_t tiles = tm * tn;
    const int64_t units = pair ? kSms / 2 : kSms;
    int K = (int)std::min<int64_t>(np, std::max<int64_t>(1, (24 * units + tiles - 1) / tiles));
    const int nl = (np + K - 1) / K;
    K = (np + nl - 1) / nl;
    const size_t esz = j.fmt ? 1 : 2;
    const int64_t r0 = it0 * (pair ? kPairTileM : kTileM), c0 = jt0 * kTileN;
    GemmLaunch1 gl;
    for (int r = 0; r < np; r += K) {
        const int cnt = std::min(K, np - r);
        memset(&gl, 0, sizeof(gl));
        gl.nprob = 1;
        gl.sched = (unsigned int*)(j.w + j.L.sched) + slot;
        GemmProblem& gp = gl.prob[0];
        if (int rc = job_fill(j, gp, cnt, 0, pair, r); rc != FMM_OK) return rc;
        const uint8_t* sa = j.w + j.L.sa + ((size_t)r * j.s * j.d.m_pad + (size_t)r0) * j.d.k_pad * esz;
        const uint8_t* sb = j.w + j.L.sb + ((size_t)r * j.s * j.d.n_pad + (size_t)c0) * j.d.k_pad * esz;
        if (make_slice_map(&gp.tmA, sa, j.d.k_pad, (int64_t)cnt * j.s * j.d.m_pad - r0, kTileM, j.fmt) != FMM_OK ||
            make_slice_map(&gp.tmB, sb, j.d.k_pad, (int64_t)cnt * j.s * j.d.n_pad - c0, pair ? kTileN / 2 : kTileN,
                           j.fmt) != FMM_OK)
            return FMM_ERR_CUDA;
        gp.Z += c0 / 4 * z_group_bytes(j.d.m_pad, gp.znd);
        gp.zrow0 = (int)r0;
        gp.tiles_m = (int)tm;
        gp.tiles_n = (int)tn;
        if (int rc = launch_gemm(gl, (int64_t)cnt * tiles, cnt, st, pair); rc != FMM_OK) return rc;
    }
    return FMM_OK;
}

/* rows of a tile of the element-major scatter with T threads; its width is 4 columns */
static int scatter_tile_rows(const SplitJob& j, int T)
{
    return j.classical ? T : T * scatter_cols(j.alg.mt * j.alg.nt) / 4;
}

/* tiles over rows x cols elements of a job (a column range may start inside a group) */
static int64_t scatter_tiles(const SplitJob& j, int64_t rows, int64_t cols, int T)
{
    const int tr = scatter_tile_rows(j, T);
    return (rows + tr - 1) / tr * ((cols + 3) / 4 + 1);
}

/* blocks of one element-major scatter launch: one per tile, at most 16 per SM
 * (each then serves several tiles with one set-up) */
static unsigned scatter_blocks(int64_t tiles) { return (unsigned)std::min<int64_t>(tiles, 16 * kSms); }

/* Whether the element-major C update applies to products [r0, r0 + np): at
 * most 64 sub-blocks whose values (T threads x 2 or 4 columns) and the group's W
 * entries fit its shared memory. T: 32 KB of values, a multiple of 32 up to
 * 256, at least 32; with `small` 16 KB and at most 128, which fits on an SM
 * beside a resident GEMM CTA while P <= 32. */
static bool job_scatter_all(const SplitJob& j, int r0, int np, int* T_out, size_t* smem_out, bool small = false)
{
    const Tab ht = tab_view(j.alg.htab);
    const int P = j.alg.mt * j.alg.nt;
    const int E = ht.w_off[r0 + np] - ht.w_off[r0];
    const int per = 8 * P * scatter_cols(P);   /* bytes of values per thread */
    const int T =
        std::max(32, std::min(small ? 128 : 256, (small ? kScatterAllSmem / 2 : kScatterAllSmem) / per) / 32 * 32);
    const size_t smem = scatter_all_smem(P, T, E, np);
    *T_out = T;
    *smem_out = smem;
    return P <= 64 && smem <= (size_t)kScatterAllMaxSmem;
}

/* Whether the element-major C update is also the faster one. With more than 16
 * sub-blocks its shared memory leaves an SM too few threads (64 sub-blocks:
 * 32-thread blocks, four per SM), and scatter_kernel, which reads Z once per
 * sub-block it feeds but keeps nothing in shared memory, is faster at every
 * grid. From 7 sub-blocks up it is also faster while the element-major form has
 * fewer than two blocks per SM, whose threads take all products one after the
 * other. Calls of k = 48 per sub-block, 6 slices, element-major / per sub-block,
 * us: 9 sub-blocks (333 x1) on a grid of 128 x 256 87 / 77, 500 x 700 165 / 167;
 * 16 (222 x2) 128 x 256 110 / 90, 256 x 512 153 / 173, 1000 x 1000 607 / 790;
 * 16 of 121 products (232 x2) 128 x 256 181 / 121, 500 x 700 544 / 570; 36
 * (322 x2) 256 x 512 424 / 294, 1000 x 1000 2620 / 1732; 64 (222 x3) 1985 / 1188,
 * 13244 / 7758. `tiles`: of the element-major launch that the job would be
 * part of. Calls that need column ranges (host buffers) use it up to 64. */
static bool scatter_all_better(const SplitJob& j, int64_t tiles)
{
    const int P = j.alg.mt * j.alg.nt;
    return P <= 16 && (P <= 6 || tiles >= 2 * kSms);
}

/* beta*C comes with the C updates of the first product group */
static double job_beta(const SplitJob& j, int r0) { return r0 == 0 ? j.beta : 1.0; }

/* the C updates of products [r0, r0 + np) for the product-grid rows
 * [i0, i1) of the columns [j0, j1), element-major form only */
static void job_scatter_block(const SplitJob& j, int r0, int np, int64_t i0, int64_t i1, int64_t j0, int64_t j1,
                              cudaStream_t st, bool small = false)
{
    int T;
    size_t smem;
    job_scatter_all(j, r0, np, &T, &smem, small);
    if (j1 <= j0 || i1 <= i0) return;
    T = (int)std::min<int64_t>(T, round_up((i1 - i0) * T / scatter_tile_rows(j, T), 32));   /* fewer than smem has room for */
    const unsigned nb = scatter_blocks(scatter_tiles(j, i1 - i0, j1 - j0, T));
    const bool row = scatter_cols(j.alg.mt * j.alg.nt) == 4;
    auto* k = j.fmt ? (row ? scatter_all_kernel<1, 4> : scatter_all_kernel<1, 2>)
                    : (row ? scatter_all_kernel<0, 4> : scatter_all_kernel<0, 2>);
    k<<<nb, (unsigned)T, smem, st>>>(j.alg.tab, r0, np, j.m, j.n, j.alpha, job_beta(j, r0), job_zview(j),
                                     (const int*)(j.w + j.L.erow), (const int*)(j.w + j.L.fcol), j.C, j.ldc, (int)j0,
                                     (int)j1, (uint32_t)i0, (uint32_t)(i1 - i0));
    fmm_count_launch(1);
}

/* the C updates of products [r0, r0 + np) for the product-grid columns
 * [j0, j1) (all rows), element-major form only */
static void job_scatter_cols(const SplitJob& j, int r0, int np, int64_t j0, int64_t j1, cudaStream_t st)
{
    job_scatter_block(j, r0, np, 0, j.d.me, j0, j1, st);
}

/* tiles of one sub-block in scatter_kernel, and their rows */
static int64_t scatter_part_tiles(const SplitJob& j, int* tr)
{
    int t = 8;
    while (t < kScatterThreads && t < j.d.me) t *= 2;
    *tr = t;
    const int64_t groups = kScatterThreads / t;
    return (j.d.me + t - 1) / t * (((j.d.ne + 3) / 4 + groups - 1) / groups);
}

/* the C updates of products [r0, r0 + np) by sub-block */
static void job_scatter_parts(const SplitJob& j, int r0, int np, cudaStream_t st)
{
    int tr;
    const int64_t tiles = scatter_part_tiles(j, &tr);
    const bool wide = tr == kScatterThreads;
    auto* k = j.fmt ? (wide ? scatter_kernel<1, true> : scatter_kernel<1, false>)
                    : (wide ? scatter_kernel<0, true> : scatter_kernel<0, false>);
    k<<<dim3((unsigned)tiles, (unsigned)(j.alg.mt * j.alg.nt)), kScatterThreads, 0, st>>>(
        j.alg.tab, r0, np, j.m, j.n, j.alpha, job_beta(j, r0), job_zview(j), (const int*)(j.w + j.L.erow),
        (const int*)(j.w + j.L.fcol), j.C, j.ldc, tr);
    fmm_count_launch(1);
}

/* the C updates of products [r0, r0 + np), in the faster form */
static void job_scatter(const SplitJob& j, int r0, int np, cudaStream_t st, bool small = false)
{
    int T;
    size_t smem;
    if (job_scatter_all(j, r0, np, &T, &smem) && scatter_all_better(j, scatter_tiles(j, j.d.me, j.d.ne, T)))
        job_scatter_block(j, r0, np, 0, j.d.me, 0, j.d.ne, st, small);
    else
        job_scatter_parts(j, r0, np, st);
}

/* dynamic shared memory limits of this file's kernels: per-device attributes, set once per device */
static int kernel_attributes(int dev)
{
    static std::atomic<uint64_t> attr_set{0};
    const uint64_t bit = dev < 64 ? 1ull << dev : 0;
    if (bit != 0 && (attr_set.load(std::memory_order_acquire) & bit)) return FMM_OK;
    auto limit = [](const void* f, size_t bytes) {
        return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess;
    };
    if (!limit((const void*)split_gemm_kernel<GemmLaunch>, kGemmSmem) ||
        !limit((const void*)split_gemm_kernel<GemmLaunch1>, kGemmSmem) ||
        !limit((const void*)split_gemm_pair_kernel<GemmLaunch>, kPairSmem) ||
        !limit((const void*)split_gemm_pair_kernel<GemmLaunch1>, kPairSmem) ||
        !limit((const void*)scatter_all_kernel<0, 2>, kScatterAllMaxSmem) ||
        !limit((const void*)scatter_all_kernel<1, 2>, kScatterAllMaxSmem) ||
        !limit((const void*)scatter_all_kernel<0, 4>, kScatterAllMaxSmem) ||
        !limit((const void*)scatter_all_kernel<1, 4>, kScatterAllMaxSmem) ||
        !limit((const void*)wave_scatter_kernel, kScatterAllMaxSmem))
        return FMM_ERR_CUDA;
    attr_set.fetch_or(bit, std::memory_order_acq_rel);
    return FMM_OK;
}

/* a launch that may start its blocks while the kernel before it on the stream
 * still runs; the kernel waits (sm103::grid_wait) before it reads anything */
template <class K, class... Args>
static int launch_after(K* kernel, dim3 grid, int threads, size_t smem, cudaStream_t st, const Args&... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...) == cudaSuccess ? FMM_OK : FMM_ERR_CUDA;
}

/* after_prep: the kernel before it on the stream is prep_kernel, which zeroes
 * gl.sched and lets this one's blocks start */
template <class GL>
static int launch_gemm(GL& gl, int64_t nitems, int nprod_timed, cudaStream_t st, bool pair, bool after_prep)
{
    int dev = 0, sms = 152;
    if (cudaGetDevice(&dev) != cudaSuccess) return FMM_ERR_CUDA;
    if (int rc = kernel_attributes(dev); rc != FMM_OK) return rc;
    if (nitems > 0x7fffffffLL) return FMM_ERR_UNSUPPORTED;
    if (nitems == 0) return FMM_OK;
    gl.nitems = (int)nitems;
    gl.err = fmm_device_error_word();
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const bool timed = g_timing;
    if (timed) {
        timing_mark(st, true);
        std::lock_guard<std::mutex> lk(g_timing_mu);
        g_timed_products += (uint64_t)nprod_timed;
    }
    /* both kernels draw their work items from gl.sched, zero at launch */
    if (gl.sched == nullptr) return FMM_ERR_CUDA;
    if (!after_prep && cudaMemsetAsync(gl.sched, 0, sizeof(unsigned int), st) != cudaSuccess) return FMM_ERR_CUDA;
    if (pair)   /* clusters of two CTAs, one pair tile each at a time */
        split_gemm_pair_kernel<<<(unsigned)(2 * std::min<int64_t>(nitems, sms / 2)), kGemmThreads, kPairSmem, st>>>(gl);
    else if (after_prep && !timed) {   /* an event between the two kernels ends the overlap */
        if (int rc = launch_after(split_gemm_kernel<GL>, dim3((unsigned)std::min<int64_t>(nitems, sms)), kGemmThreads,
                                  kGemmSmem, st, gl); rc != FMM_OK)
            return rc;
    } else {
        split_gemm_kernel<<<(unsigned)std::min<int64_t>(nitems, sms), kGemmThreads, kGemmSmem, st>>>(gl);
    }
    if (timed) timing_mark(st, false);
    fmm_count_launch(1);
    return FMM_OK;
}

/* Two product groups whose work overlaps: the products split into
 * G1 = ceil(R/2) and R - G1, each group with its own exponents, slices and
 * Z (the second region follows the first; the maxima are shared). Group 1
 * is packed with the whole GPU; group 2's packs (small tiles, pool stream
 * s[3]) then run on the SMs beside group 1's GEMM, and group 1's C updates
 * (small blocks, s[4]) beside group 2's GEMM; group 2's C updates follow on
 * s[4], so every C element still receives the products in increasing order
 * and the result is the single group's bit for bit. The second region's
 * layout: the group part of L1 shifted by its own size. */
struct OverlapPlan {
    WsLayout L1;
    size_t shift = 0;
    bool ok = false;
};

static OverlapPlan overlap_plan(const AlgView& alg, const Dims& d, int64_t m, int64_t n, int s, int fmt,
                                size_t bytes)
{
    OverlapPlan o;
    if (alg.R < 2) return o;
    const int G1 = (alg.R + 1) / 2;
    o.L1 = ws_layout_g(alg, d, m, n, s, G1, fmt);
    o.shift = o.L1.total - o.L1.erow;
    /* each group's GEMM keeps every SM busy for at least 8 rounds of items */
    const int64_t tiles = (d.m_pad / (d.me >= kPairMinRows ? kPairTileM : kTileM)) * (d.n_pad / kTileN);
    o.ok = o.L1.total + o.shift <= bytes && (int64_t)G1 * tiles >= 8 * kSms &&
           (int64_t)G1 * s * std::max(d.m_pad, d.n_pad) <= 0x7fffffffLL;
    return o;
}

static int split_overlap(SplitJob& j, const OverlapPlan& o, void* ws, cudaStream_t st, SidePool* sp)
{
    const int R = j.alg.R, G1 = o.L1.group, G2 = R - G1;
    j.L = o.L1;
    j.w = (uint8_t*)ws;
    j.z = j.w + j.L.z;
    SplitJob j2 = j;
    j2.L.erow += o.shift;
    j2.L.fcol += o.shift;
    j2.L.sa += o.shift;
    j2.L.sb += o.shift;
    j2.L.z += o.shift;
    j2.z += o.shift;
    j2.L.total += o.shift;
    /* the GEMMs on the greatest-priority stream, so the block scheduler
     * places their CTAs first and the side work fills the room they leave */
    cudaStream_t sg = sp->hi, sp2 = sp->s[3], ssc = sp->s[4];
    auto ok = [](cudaError_t e) { return e == cudaSuccess; };
    int rc;
    if ((rc = job_prologue(j, st, sp)) != FMM_OK) return rc;
    if ((rc = job_pack(j, 0, G1, st, sp)) != FMM_OK) return rc;
    if (!ok(cudaEventRecord(sp->chunk[0], st)) || !ok(cudaStreamWaitEvent(sg, sp->chunk[0], 0))) return FMM_ERR_CUDA;
    if ((rc = job_gemm(j, G1, sg)) != FMM_OK) return rc;
    if (!ok(cudaEventRecord(sp->chunk[2], sg))) return FMM_ERR_CUDA;
    /* group 2's packs after the maxima (and group 1's packs), beside GEMM 1 */
    if (!ok(cudaStreamWaitEvent(sp2, sp->chunk[0], 0))) return FMM_ERR_CUDA;
    if ((rc = job_pack(j2, G1, G2, sp2, nullptr, true)) != FMM_OK) return rc;
    if (!ok(cudaEventRecord(sp->chunk[1], sp2))) return FMM_ERR_CUDA;
    /* group 1's C updates beside GEMM 2 */
    if (!ok(cudaStreamWaitEvent(ssc, sp->chunk[2], 0))) return FMM_ERR_CUDA;
    job_scatter(j, 0, G1, ssc, true);
    if (!ok(cudaStreamWaitEvent(sg, sp->chunk[1], 0))) return FMM_ERR_CUDA;
    if ((rc = job_gemm(j2, G2, sg)) != FMM_OK) return rc;
    if (!ok(cudaEventRecord(sp->chunk[3], sg)) || !ok(cudaStreamWaitEvent(ssc, sp->chunk[3], 0))) return FMM_ERR_CUDA;
    job_scatter(j2, G1, G2, ssc);
    if (!ok(cudaEventRecord(sp->chunk[4], ssc)) || !ok(cudaStreamWaitEvent(st, sp->chunk[4], 0))) return FMM_ERR_CUDA;
    return cudaGetLastError() == cudaSuccess ? FMM_OK : FMM_ERR_CUDA;
}

/* CTAs per cluster (k chunks) of prep_kernel for `groups` line groups of depth
 * k_pad: more while the launch has fewer than three CTAs per SM, or a chunk is
 * longer than 1024 k (its 16 lines are read twice, the second time from L2:
 * 128 KB for each of the 608 CTAs in flight), of at least one tile each */
static int prep_ranks(int64_t groups, int64_t k_pad)
{
    int r = 1;
    while (r < 8 && k_pad >= (int64_t)kPrepK * 2 * r && (groups * r < 3 * kSms || k_pad > (int64_t)1024 * r)) r *= 2;
    return r;
}

template <class K, class... Args>
static int launch_clusters(K* kernel, int64_t blocks, int cluster, cudaStream_t st, Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(kPrepThreads);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
    fmm_count_launch(1);
    return e == cudaSuccess ? FMM_OK : FMM_ERR_CUDA;
}

/* exponents and digit slices of both operands of a classical job */
static int job_prep(SplitJob& j, cudaStream_t st)
{
    const Dims& d = j.d;
    const int64_t groups = (d.m_pad + d.n_pad) / kPrepLines;
    const int nrank = prep_ranks(groups, d.k_pad);
    return with_slices(j.fmt, j.s, [&](auto S, auto DB) {
        return launch_clusters(prep_kernel<S(), DB()>, groups * nrank, nrank, st, j.A, j.lda, j.B, j.ldb, j.m, j.n, j.k,
                               d.m_pad, d.n_pad, d.k_pad, (int*)(j.w + j.L.erow), (int*)(j.w + j.L.fcol),
                               j.w + j.L.sa, j.w + j.L.sb, (unsigned int*)(j.w + j.L.sched), nrank);
    });
}

/* whether work enqueued on st is being captured into a graph */
static bool capturing(cudaStream_t st)
{
    cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &c) != cudaSuccess) cudaGetLastError();
    return c != cudaStreamCaptureStatusNone;
}

/* A classical GEMM: one launch for the operands, one for the tiles (or their
 * work units), one for C. With `units`, the units' planes lie behind the job's
 * part of the workspace where the caller's is large enough
 * (fmm_split_full_ws_bytes), else they are a stream-ordered temporary. Without
 * memory, and in a captured call whose workspace has no room, the tiles run
 * whole: a graph with an allocation node could not be cloned or instantiated
 * twice. */
static int split_classical(SplitJob& j, size_t ws_bytes, bool units, cudaStream_t st)
{
    if (int rc = job_prep(j, st); rc != FMM_OK) return rc;
    UnitPlan up;
    if (units) up = unit_plan(j.d, j.s, j.fmt, job_pair(j));
    uint8_t* spare = nullptr;   /* planes in the workspace */
    void* planes = nullptr;     /* planes of their own */
    if (up.nunits != 0) {
        cudaMemPool_t pool = nullptr;
        if (ws_bytes >= j.L.total + up.bytes) {
            spare = j.w + j.L.total;
        } else if (capturing(st) || (pool = fmm_temp_pool()) == nullptr ||
                   cudaMallocFromPoolAsync(&planes, up.bytes, pool, st) != cudaSuccess) {
            cudaGetLastError();
            up = UnitPlan();
        }
    }
    const bool pair = job_pair(j) && up.nunits == 0;
    GemmLaunch1 gl;
    memset(&gl, 0, sizeof(gl));
    gl.nprob = 1;
    gl.sched = (unsigned int*)(j.w + j.L.sched);   /* zeroed by prep_kernel */
    GemmProblem& gp = gl.prob[0];
    if (int rc = job_fill(j, gp, 1, 0, pair); rc != FMM_OK) {
        if (planes) cudaFreeAsync(planes, st);
        return rc;
    }
    if (up.nunits == 0) {
        if (int rc = launch_gemm(gl, job_items(j, 1, pair), 1, st, pair, true); rc != FMM_OK) return rc;
        job_scatter(j, 0, 1, st);
        return cudaGetLastError() == cudaSuccess ? FMM_OK : FMM_ERR_CUDA;
    }
    gp.nunits = up.nunits;
    gp.unit_kb = up.unit_kb;
    gp.Z = spare ? spare : (uint8_t*)planes;
    int rc = launch_gemm(gl, job_items(j, 1) * up.nunits, 1, st, false, true);
    if (rc == FMM_OK) {
        rc = launch_after(scatter_units_kernel, dim3((unsigned)((j.m + 31) / 32), (unsigned)((j.n + 15) / 16)), 128, 0,
                          st, (int)j.m, (int)j.n, j.alpha, j.beta, (const int4*)gp.Z, (int)j.d.m_pad,
                          (int)j.d.n_pad, j.s, gp.nkb, up.unit_kb, up.nunits, job_zlevel(j), job_db(j), job_ebase(j),
                          (const int*)(j.w + j.L.erow), (const int*)(j.w + j.L.fcol), j.C, j.ldc);
        fmm_count_launch(1);
        if (rc == FMM_OK && cudaGetLastError() != cudaSuccess) rc = FMM_ERR_CUDA;
    }
    if (planes != nullptr && cudaFreeAsync(planes, st) != cudaSuccess && rc == FMM_OK) rc = FMM_ERR_CUDA;
    return rc;
}

/* the product groups of a bound job, one after the other */
static int split_groups(SplitJob& j, cudaStream_t st, SidePool* sp)
{
    int rc = job_prologue(j, st, sp);
    if (rc != FMM_OK) return rc;
    const int G = j.L.group;
    for (int r0 = 0; r0 < j.alg.R; r0 += G) {
        const int np = std::min(G, j.alg.R - r0);
        if ((rc = job_pack(j, r0, np, st, sp)) != FMM_OK) return rc;
        if ((rc = job_gemm(j, np, st)) != FMM_OK) return rc;
        job_scatter(j, r0, np, st);
    }
    return cudaGetLastError() == cudaSuccess ? FMM_OK : FMM_ERR_CUDA;
}

static int split_launch_budget(const AlgView& alg, int64_t m, int64_t n, int64_t k, double alpha,
                               const double* A, int64_t lda, const double* B, int64_t ldb, double beta,
                               double* C, int64_t ldc, int s, int fmt, void* ws, size_t ws_bytes, size_t budget,
                               cudaStream_t st, SidePool* sp)
{
    SplitJob j;
    int rc = job_init(j, alg, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, s, fmt);
    if (rc != FMM_OK) return rc;
    if (!j.trivial && sp && ws != nullptr && ((uintptr_t)ws & 255) == 0) {
        const OverlapPlan o = overlap_plan(alg, j.d, m, n, s, fmt, std::min(ws_bytes, budget));
        if (o.ok) return split_overlap(j, o, ws, st, sp);
    }
    if (j.trivial) return job_prologue(j, st);
    if ((rc = job_bind(j, ws, ws_bytes, budget)) != FMM_OK) return rc;
    void* zbuf = nullptr;
    if (j.z == nullptr) {
        const cudaMemPool_t pool = fmm_temp_pool();
        if (pool == nullptr || cudaMallocFromPoolAsync(&zbuf, z_bytes(j.d, s, fmt), pool, st) != cudaSuccess) {
            cudaGetLastError();
            return FMM_ERR_WORKSPACE;
        }
        j.z = (uint8_t*)zbuf;
    }
    rc = j.classical ? split_classical(j, ws_bytes, sp != nullptr, st) : split_groups(j, st, sp);
    if (zbuf != nullptr && cudaFreeAsync(zbuf, st) != cudaSuccess && rc == FMM_OK) rc = FMM_ERR_CUDA;
    return rc;
}

/* ---------------------------------------------------------------------------
 * Host-buffer entry.
 *
 * Operands in host memory: the call owns the device copies and, unless they
 * are small, overlaps the host<->device traffic with the device work. Uploads
 * run on s[1] in the order A, B, C (with the blocked schedule below: A's first
 * row half, B's first column part, A's second half, B's other parts, each
 * block's C before its updates); the A side (row maxima, row exponents, A
 * slices) starts as soon as its rows have arrived, the B side on another stream
 * as soon as its columns have, and C is only needed by the C updates, so its
 * upload runs under the GEMM. The host enqueues in the same order, which keeps
 * the overlap when a copy from pageable memory blocks the host until it is
 * staged. Every host copy touches its host pages first (fmm_touch_host). The
 * operand and workspace buffers are kept per device (grow-only) until
 * fmm_gpu_release_host_buffers.
 * ------------------------------------------------------------------------- */
struct HostBuffers {
    uint8_t* p = nullptr;
    size_t bytes = 0;
};
static std::mutex g_hostbuf_mu;
static HostBuffers g_hostbuf[64];

static uint8_t* host_buffers(size_t bytes)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    HostBuffers& h = g_hostbuf[dev];
    if (h.bytes >= bytes) return h.p;
    if (h.p) cudaFree(h.p);
    h.p = nullptr;
    h.bytes = 0;
    if (cudaMalloc(&h.p, bytes) != cudaSuccess) {
        cudaGetLastError();
        h.p = nullptr;
        return nullptr;
    }
    h.bytes = bytes;
    return h.p;
}

static size_t align256(size_t b) { return (b + 255) / 256 * 256; }

constexpr int kChunks = 8;   /* B uploads and C downloads per host-buffer call */
constexpr size_t kHostSimpleBytes = (size_t)32 << 20;   /* operands up to this size go without the overlapped schedules */

/* A host-buffer call that ends early waits for its streams, so nothing is left
 * in flight on the caller's memory or the kept buffers. */
struct HostCallEnd {
    SidePool* sp;
    bool complete = false;   /* the call waited for its streams itself */
    ~HostCallEnd()
    {
        if (complete) return;
        for (cudaStream_t s : sp->s) cudaStreamSynchronize(s);
        for (cudaStream_t s : sp->top) cudaStreamSynchronize(s);
        cudaStreamSynchronize(sp->hi);
    }
};

int fmm_split_host(const AlgView& alg, int64_t m, int64_t n, int64_t k, double alpha, const double* A,
                   int64_t lda, const double* B, int64_t ldb, double beta, double* C, int64_t ldc, int s, int fmt)
{
    if (m == 0 || n == 0) return FMM_OK;
    std::lock_guard<std::mutex> use(g_side_use);
    std::lock_guard<std::mutex> buf(g_hostbuf_mu);
    SidePool* sp = side_pool();
    if (!sp) return FMM_ERR_CUDA;
    cudaStream_t st = sp->s[2], cs = sp->s[1];
    const int64_t ka = std::max<int64_t>(k, 1);
    const bool trivial = k == 0 || alpha == 0.0;
    if (trivial && beta == 1.0) return FMM_OK;
    /* what the split form refuses is refused before the first copy */
    SplitJob j;
    int rc = job_init(j, alg, m, n, k, alpha, nullptr, m, nullptr, ka, beta, nullptr, m, s, fmt);
    if (rc != FMM_OK) return rc;
    const size_t bA = trivial ? 0 : align256(sizeof(double) * (size_t)(m * ka));
    const size_t bB = trivial ? 0 : align256(sizeof(double) * (size_t)(ka * n));
    const size_t bC = align256(sizeof(double) * (size_t)(m * n));
    const size_t wsb = trivial ? 0 : align256(fmm_split_ws_bytes(alg, m, n, k, s, fmt));
    uint8_t* base = host_buffers(bA + bB + bC + wsb);
    if (!base) return FMM_ERR_ALLOC;
    double* dA = (double*)base;
    double* dB = (double*)(base + bA);
    double* dC = (double*)(base + bA + bB);
    uint8_t* ws = base + bA + bB + bC;
    j.A = dA;
    j.B = dB;
    j.C = dC;
    if ((rc = job_bind(j, ws, wsb, wsb)) != FMM_OK) return rc;
    HostCallEnd end{sp};
    const size_t row = sizeof(double) * (size_t)m;
    auto ok = [](cudaError_t e) { return e == cudaSuccess; };
    const bool tline = g_timeline.load() && !trivial;
    const auto host_t0 = std::chrono::steady_clock::now();
    auto mark = [&](int x, cudaStream_t on) { if (tline) cudaEventRecord(sp->tl[x], on); };
    auto read_timeline = [&]() {
        std::lock_guard<std::mutex> lk(g_timeline_mu);
        for (int x = 1; x <= kTimelinePoints; ++x) {
            float t = 0.f;
            cudaEventElapsedTime(&t, sp->tl[0], sp->tl[x]);
            g_timeline_ms[x - 1] = t;
        }
        g_timeline_ms[kTimelinePoints] =
            std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - host_t0).count();
    };
    if (trivial) {
        /* C := beta*C */
        if (beta != 0.0 && !ok(fmm_copy2d_async(dC, row, C, sizeof(double) * ldc, row, n, cudaMemcpyHostToDevice, st)))
            return FMM_ERR_CUDA;
        if ((rc = fmm_scale_c(m, n, beta, dC, m, st)) != FMM_OK) return rc;
    } else {
        /* Small operands, or many sub-blocks: the device call between plain
         * copies. Overlapping the copies with the work saves at most their
         * time (at about 200 bytes per ns), and the blocked schedule's copies,
         * one per C piece and sub-block, cost about 4 us each: 444 x1 at
         * 1715 x 1867 x 1620, 16 sub-blocks, 1.9 ms blocked. */
        const double piece_ns = 4000.0 * ((double)alg.mt * alg.nt * (double)std::min<int64_t>(16, 1 + (m * n * 8 >> 21)) +
                                          2.0 * alg.mt + 8.0 * alg.nt);
        if (bA + bB + bC <= kHostSimpleBytes || piece_ns > (double)(bA + bB + bC) / 200.0) {
            mark(0, st);
            if (!ok(fmm_copy2d_async(dA, row, A, sizeof(double) * lda, row, k, cudaMemcpyHostToDevice, st)))
                return FMM_ERR_CUDA;
            mark(1, st);
            if (!ok(fmm_copy2d_async(dB, sizeof(double) * k, B, sizeof(double) * ldb, sizeof(double) * k, n,
                                     cudaMemcpyHostToDevice, st)))
                return FMM_ERR_CUDA;
            mark(2, st);
            if (beta != 0.0 &&
                !ok(fmm_copy2d_async(dC, row, C, sizeof(double) * ldc, row, n, cudaMemcpyHostToDevice, st)))
                return FMM_ERR_CUDA;
            mark(3, st);
            if ((rc = split_launch_budget(alg, m, n, k, alpha, dA, m, dB, ka, beta, dC, m, s, fmt, ws, wsb, wsb, st,
                                          sp)) != FMM_OK)
                return rc;
            mark(4, st);
            if (!ok(fmm_copy2d_async(C, sizeof(double) * ldc, dC, row, row, n, cudaMemcpyDeviceToHost, st)))
                return FMM_ERR_CUDA;
            mark(5, st);
            if (!ok(cudaStreamSynchronize(st))) return FMM_ERR_CUDA;
            end.complete = true;
            if (tline) read_timeline();
            return cudaGetLastError() == cudaSuccess ? fmm_device_error_status() : FMM_ERR_CUDA;
        }
        const int G = j.L.group, nt = alg.nt;
        const bool one_group = G >= alg.R;
        cudaStream_t sb = sp->s[0];
        /* Blocked schedule, for one product group with the element-major C
         * update and a product grid of at least two GEMM tiles along a side:
         * the grid splits into up to 2 x 4 blocks of tiles (row halves of A,
         * column parts of B), column by column. A's first row half and B's
         * first column part go up first, so the GEMM of block (0, 0) starts
         * after those; A's second half follows, then B's other parts. A
         * block's C elements are final when its GEMM ends: they are updated
         * and read back while later blocks run, so after the last GEMM only
         * the last block's C is left. Every (product, tile) item and every C
         * element is computed as in the unblocked call: the same bits. */
        {
            const bool pair = job_pair(j);
            const int64_t me = j.d.me, ne = j.d.ne, m_pad = j.d.m_pad, n_pad = j.d.n_pad;
            const int64_t U = pair ? kPairTileM : kTileM;
            const int64_t tiles_m = m_pad / U, tiles_n = n_pad / kTileN;
            const int RH = tiles_m >= 2 ? 2 : 1;
            /* four column parts where a block still has half a round of items
             * (two blocks are in flight at a time) */
            const int CH = tiles_n >= 4 && alg.R * (tiles_m / RH) * (tiles_n / 4) >= (pair ? kSms / 4 : kSms / 2) ? 4
                           : tiles_n >= 2 ? 2 : 1;
            int Tchk;
            size_t smchk;
            if (one_group && RH * CH >= 2 && job_scatter_all(j, 0, alg.R, &Tchk, &smchk)) {
                const int mt = alg.mt;
                const int64_t rcut[3] = {0, RH == 2 ? (tiles_m + 1) / 2 * U : m_pad, m_pad};   /* S_r row halves */
                int64_t ccut[5];                                                               /* T_r column parts */
                for (int x = 0; x <= CH; ++x) ccut[x] = (tiles_n * x + CH - 1) / CH * kTileN;
                /* copies per B part and per block's C: pieces of at least 2 MiB
                 * (a copy and the launches behind it cost about 10 us) */
                auto pieces = [](int64_t elems, int most) {
                    return (int)std::min<int64_t>(most, std::max<int64_t>(1, elems * 8 >> 21));
                };
                const int bchunks = pieces(k * n / CH, 8 / CH), cchunks = pieces(m * n / (RH * CH), 16 / (RH * CH));
                const cudaStream_t ss = sp->top[0], sa = sp->top[1], sb = sp->top[2];
                auto up_a = [&](int h) -> int {
                    /* the A rows ro_p + [rcut[h], rcut[h+1]) of every row part p, then that half's A side */
                    if (RH == 1) {
                        if (!ok(fmm_copy2d_async(dA, row, A, sizeof(double) * lda, row, k, cudaMemcpyHostToDevice, cs)))
                            return FMM_ERR_CUDA;
                    } else {
                        for (int p = 0; p < mt; ++p) {
                            int64_t ro, rl;
                            fmm_part_geom(m, mt, p, &ro, &rl);
                            const int64_t a = ro + std::min(rcut[h], rl), b = ro + std::min(rcut[h + 1], rl);
                            if (b > a && !ok(fmm_copy2d_async(dA + a, row, A + a, sizeof(double) * lda,
                                                               sizeof(double) * (b - a), k, cudaMemcpyHostToDevice, cs)))
                                return FMM_ERR_CUDA;
                        }
                    }
                    if (!ok(cudaEventRecord(sp->blk[h], cs)) || !ok(cudaStreamWaitEvent(sa, sp->blk[h], 0)))
                        return FMM_ERR_CUDA;
                    if (h == 0 && !ok(cudaMemsetAsync(j.w + j.L.amax, 0,
                                                      sizeof(unsigned long long) * (size_t)alg.kt * (size_t)m, sa)))
                        return FMM_ERR_CUDA;
                    job_maxima_a_rows(j, sa, rcut[h], rcut[h + 1]);
                    job_pack_a_rows(j, 0, alg.R, rcut[h], rcut[h + 1], sa);
                    return ok(cudaEventRecord(sp->blk[2 + h], sa)) ? FMM_OK : FMM_ERR_CUDA;
                };
                int xb = 0;
                auto up_b = [&](int h) -> int {
                    /* the T_r columns [ccut[h], ccut[h+1]) in chunks, each chunk's B side behind it */
                    const int64_t w = round_up((ccut[h + 1] - ccut[h] + bchunks - 1) / bchunks, 32);
                    for (int64_t j0 = ccut[h]; j0 < ccut[h + 1]; j0 += w, ++xb) {
                        const int64_t j1 = std::min(j0 + w, ccut[h + 1]);
                        for (int c = 0; c < nt; ++c) {
                            int64_t co, cl;
                            fmm_part_geom(n, nt, c, &co, &cl);
                            const int64_t a = co + std::min(j0, cl), b = co + std::min(j1, cl);
                            if (b > a && !ok(fmm_copy2d_async(dB + a * k, sizeof(double) * k, B + a * ldb,
                                                               sizeof(double) * ldb, sizeof(double) * k, b - a,
                                                               cudaMemcpyHostToDevice, cs)))
                                return FMM_ERR_CUDA;
                        }
                        if (!ok(cudaEventRecord(sp->chunk[xb], cs)) || !ok(cudaStreamWaitEvent(sb, sp->chunk[xb], 0)))
                            return FMM_ERR_CUDA;
                        for (int c = 0; c < nt; ++c) {
                            int64_t co, cl;
                            fmm_part_geom(n, nt, c, &co, &cl);
                            job_maxima_b(j, sb, co + std::min(j0, cl), co + std::min(j1, cl));
                        }
                        job_pack_b_cols(j, 0, alg.R, j0, j1, sb);
                    }
                    return ok(cudaEventRecord(sp->blk[4 + h], sb)) ? FMM_OK : FMM_ERR_CUDA;
                };
                const int nq = RH * CH;   /* block q: rows q % RH, columns q / RH */
                /* GEMM blocks alternate between two streams, each with its
                 * own item counter: a block's CTAs leave as its items run out
                 * and the next block's take their place (a block at 4096 with
                 * one Strassen level is 112 items on 76 CTA pairs). The side
                 * work has priority, or the GEMMs would keep the SMs from the
                 * C updates until the last block. */
                const cudaStream_t gst[2] = {st, sp->s[5]}, ds = sp->s[6];
                auto gemm = [&](int q) -> int {
                    const cudaStream_t on = gst[q & 1];
                    if (!ok(cudaStreamWaitEvent(on, sp->blk[2 + q % RH], 0)) ||
                        !ok(cudaStreamWaitEvent(on, sp->blk[4 + q / RH], 0)))
                        return FMM_ERR_CUDA;
                    if (q == 0) mark(3, on);
                    if (int e = job_gemm_block(j, alg.R, rcut[q % RH] / U, rcut[q % RH + 1] / U,
                                               ccut[q / RH] / kTileN, ccut[q / RH + 1] / kTileN, on, q & 1); e != FMM_OK)
                        return e;
                    if (q + 1 == nq) mark(4, on);
                    return ok(cudaEventRecord(sp->blk[8 + q], on)) ? FMM_OK : FMM_ERR_CUDA;
                };
                /* a block's C updates in column chunks, each with its event */
                struct CChunk {
                    int64_t i0, i1, j0, j1;
                };
                CChunk chunks[16];
                int xc = 0;
                auto update = [&](int q) -> int {
                    if (!ok(cudaStreamWaitEvent(ss, sp->blk[8 + q], 0))) return FMM_ERR_CUDA;
                    const int64_t i0 = rcut[q % RH], i1 = std::min(rcut[q % RH + 1], me);
                    const int64_t a0 = ccut[q / RH], b0 = std::min(ccut[q / RH + 1], ne);
                    if (i1 <= i0 || b0 <= a0) return FMM_OK;
                    const int64_t w = std::max<int64_t>((b0 - a0 + cchunks - 1) / cchunks, 1);
                    for (int64_t j0 = a0; j0 < b0; j0 += w, ++xc) {
                        chunks[xc] = CChunk{i0, i1, j0, std::min(j0 + w, b0)};
                        job_scatter_block(j, 0, alg.R, i0, i1, j0, chunks[xc].j1, ss);
                        if (!ok(cudaEventRecord(sp->chunk[8 + xc], ss))) return FMM_ERR_CUDA;
                    }
                    return FMM_OK;
                };
                /* a block's C elements up, for its updates */
                auto up_c = [&](int q) -> int {
                    if (beta == 0.0) return FMM_OK;
                    for (int p = 0; p < mt; ++p) {
                        int64_t ro, rl;
                        fmm_part_geom(m, mt, p, &ro, &rl);
                        const int64_t ra = ro + std::min(rcut[q % RH], rl), rb = ro + std::min(rcut[q % RH + 1], rl);
                        if (rb <= ra) continue;
                        for (int y = 0; y < nt; ++y) {
                            int64_t co, cl;
                            fmm_part_geom(n, nt, y, &co, &cl);
                            const int64_t ca = co + std::min(ccut[q / RH], cl), cb = co + std::min(ccut[q / RH + 1], cl);
                            if (cb > ca &&
                                !ok(fmm_copy2d_async(dC + ra + ca * m, row, C + ra + ca * ldc, sizeof(double) * ldc,
                                                     sizeof(double) * (rb - ra), cb - ca, cudaMemcpyHostToDevice, cs)))
                                return FMM_ERR_CUDA;
                        }
                    }
                    return ok(cudaEventRecord(sp->chunk[24 + q], cs)) &&
                                   ok(cudaStreamWaitEvent(ss, sp->chunk[24 + q], 0))
                               ? FMM_OK : FMM_ERR_CUDA;
                };
                /* Everything in the order it is needed: what a block's GEMM
                 * waits for, the GEMM, then C for the blocks under way (its
                 * copy and the updates fit under the GEMMs; C last of all
                 * would hold the first update until 3/4 of the call's time).
                 * Streams that share a hardware queue run in enqueue order. */
                mark(0, cs);
                if ((rc = up_a(0)) != FMM_OK) return rc;
                if (RH == 1) mark(1, cs);
                int c_next = 0;   /* the next block whose C goes up */
                for (int x = 0; x < CH; ++x) {
                    if ((rc = up_b(x)) != FMM_OK) return rc;
                    if (x + 1 == CH) mark(2, cs);
                    if ((rc = gemm(x * RH)) != FMM_OK) return rc;
                    if (RH == 2) {
                        if (x == 0) {
                            if ((rc = up_a(1)) != FMM_OK) return rc;
                            mark(1, cs);
                        }
                        if ((rc = gemm(x * RH + 1)) != FMM_OK) return rc;
                    }
                    for (; c_next < (x + 1 == CH ? nq : x * RH + 1); ++c_next)
                        if ((rc = up_c(c_next)) != FMM_OK || (rc = update(c_next)) != FMM_OK) return rc;
                }
                /* each chunk's C elements back on s[6], beside the uploads (enqueued
                 * last: a copy to pageable memory holds the host) */
                for (int x = 0; x < xc; ++x) {
                    const CChunk& c = chunks[x];
                    if (!ok(cudaStreamWaitEvent(ds, sp->chunk[8 + x], 0))) return FMM_ERR_CUDA;
                    for (int p = 0; p < mt; ++p) {
                        int64_t ro, rl;
                        fmm_part_geom(m, mt, p, &ro, &rl);
                        const int64_t ra = ro + std::min(c.i0, rl), rb = ro + std::min(c.i1, rl);
                        if (rb <= ra) continue;
                        for (int y = 0; y < nt; ++y) {
                            int64_t co, cl;
                            fmm_part_geom(n, nt, y, &co, &cl);
                            const int64_t ca = co + std::min(c.j0, cl), cb = co + std::min(c.j1, cl);
                            if (cb > ca &&
                                !ok(fmm_copy2d_async(C + ra + ca * ldc, sizeof(double) * ldc, dC + ra + ca * m, row,
                                                     sizeof(double) * (rb - ra), cb - ca, cudaMemcpyDeviceToHost, ds)))
                                return FMM_ERR_CUDA;
                        }
                    }
                }
                mark(5, ds);
                if (!ok(cudaStreamSynchronize(ds)) || !ok(cudaStreamSynchronize(cs)) || !ok(cudaStreamSynchronize(gst[0])) ||
                    !ok(cudaStreamSynchronize(gst[1])) || !ok(cudaStreamSynchronize(ss)) || !ok(cudaStreamSynchronize(sa)) || !ok(cudaStreamSynchronize(sb)))
                    return FMM_ERR_CUDA;
                end.complete = true;
                if (tline) read_timeline();
                return cudaGetLastError() == cudaSuccess ? fmm_device_error_status() : FMM_ERR_CUDA;
            }
        }
        /* A, then the A side's maxima (and, with one product group, its
         * exponents and slices) */
        mark(0, cs);
        if (!ok(fmm_copy2d_async(dA, row, A, sizeof(double) * lda, row, k, cudaMemcpyHostToDevice, cs)) ||
            !ok(cudaEventRecord(sp->gate[0], cs)) || !ok(cudaStreamWaitEvent(st, sp->gate[0], 0)))
            return FMM_ERR_CUDA;
        mark(1, cs);
        if ((rc = job_maxima_a(j, st)) != FMM_OK) return rc;
        if (one_group) job_pack_a(j, 0, alg.R, st);
        /* B in kChunks chunks of T_r columns [j0, j1): chunk x holds the B
         * columns co_c + [j0, j1) of every column part c, and the B side of
         * those columns (maxima; with one group, exponents and slices) runs
         * on s[0] as soon as the chunk has arrived */
        const int64_t ne = j.d.ne, n_pad = j.d.n_pad;
        const int64_t W = (ne + kChunks * 32 - 1) / (kChunks * 32) * 32;
        int x = 0;
        for (int64_t j0 = 0; j0 < n_pad; j0 += W, ++x) {
            const int64_t j1 = std::min(j0 + W, n_pad);
            for (int c = 0; c < nt; ++c) {
                int64_t co, cl;
                fmm_part_geom(n, nt, c, &co, &cl);
                const int64_t a = co + std::min(j0, cl), b = co + std::min(j1, cl);
                if (b > a && !ok(fmm_copy2d_async(dB + a * k, sizeof(double) * k, B + a * ldb, sizeof(double) * ldb,
                                                   sizeof(double) * k, b - a, cudaMemcpyHostToDevice, cs)))
                    return FMM_ERR_CUDA;
            }
            if (!ok(cudaEventRecord(sp->chunk[x], cs)) || !ok(cudaStreamWaitEvent(sb, sp->chunk[x], 0)))
                return FMM_ERR_CUDA;
            for (int c = 0; c < nt; ++c) {
                int64_t co, cl;
                fmm_part_geom(n, nt, c, &co, &cl);
                job_maxima_b(j, sb, co + std::min(j0, cl), co + std::min(j1, cl));
            }
            if (one_group) job_pack_b_cols(j, 0, alg.R, j0, j1, sb);
        }
        mark(2, cs);
        for (int r0 = 0; r0 < alg.R; r0 += G) {
            const int np = std::min(G, alg.R - r0);
            if (one_group) {
                if ((rc = side_join1(sp, st)) != FMM_OK) return rc;
            } else if ((rc = job_pack(j, r0, np, st, sp)) != FMM_OK) {
                return rc;
            }
            if (r0 == 0) mark(3, st);
            if ((rc = job_gemm(j, np, st)) != FMM_OK) return rc;
            if (r0 + np >= alg.R) mark(4, st);
            if (r0 == 0) {
                /* C under the first GEMM, before the first C updates */
                if (beta != 0.0 &&
                    (!ok(fmm_copy2d_async(dC, row, C, sizeof(double) * ldc, row, n, cudaMemcpyHostToDevice, cs)) ||
                     !ok(cudaEventRecord(sp->gate[2], cs)) || !ok(cudaStreamWaitEvent(st, sp->gate[2], 0))))
                    return FMM_ERR_CUDA;
            }
            int T;
            size_t smem;
            if (r0 + np < alg.R || !job_scatter_all(j, r0, np, &T, &smem)) {
                job_scatter(j, r0, np, st);
                continue;
            }
            /* the last group's C updates in column chunks of the product grid,
             * each chunk's C columns (co_c + [j0, j1) of every column part)
             * read back on s[1] while the next chunk is computed */
            const int64_t W2 = (ne + kChunks - 1) / kChunks;
            x = 0;
            for (int64_t j0 = 0; j0 < ne; j0 += W2, ++x) {
                const int64_t j1 = std::min(j0 + W2, ne);
                job_scatter_cols(j, r0, np, j0, j1, st);
                if (!ok(cudaEventRecord(sp->chunk[kChunks + x], st)) ||
                    !ok(cudaStreamWaitEvent(cs, sp->chunk[kChunks + x], 0)))
                    return FMM_ERR_CUDA;
                for (int c = 0; c < nt; ++c) {
                    int64_t co, cl;
                    fmm_part_geom(n, nt, c, &co, &cl);
                    const int64_t a = co + std::min(j0, cl), b = co + std::min(j1, cl);
                    if (b > a && !ok(fmm_copy2d_async(C + a * ldc, sizeof(double) * ldc, dC + a * m, row, row, b - a,
                                                       cudaMemcpyDeviceToHost, cs)))
                        return FMM_ERR_CUDA;
                }
            }
            mark(5, cs);
            if (!ok(cudaEventRecord(sp->gate[1], cs)) || !ok(cudaStreamSynchronize(cs)) ||
                !ok(cudaStreamSynchronize(st)))
                return FMM_ERR_CUDA;
            end.complete = true;
            if (tline) read_timeline();
            return cudaGetLastError() == cudaSuccess ? fmm_device_error_status() : FMM_ERR_CUDA;
        }
    }
    if (!ok(fmm_copy2d_async(C, sizeof(double) * ldc, dC, row, row, n, cudaMemcpyDeviceToHost, st)) ||
        !ok(cudaStreamSynchronize(st)))
        return FMM_ERR_CUDA;
    end.complete = true;
    /* a kernel whose bounded wait expired left C incomplete: report it */
    return cudaGetLastError() == cudaSuccess ? fmm_device_error_status() : FMM_ERR_CUDA;
}

void fmm_split_host_release()
{
    std::lock_guard<std::mutex> buf(g_hostbuf_mu);
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return;
    if (g_hostbuf[dev].p) cudaFree(g_hostbuf[dev].p);
    g_hostbuf[dev] = HostBuffers();
}

/* Batched split-form GEMMs: problems are taken in order into waves of at
 * most kMaxLaunchProblems whose whole workspaces (all products at once) fit
 * together; per wave every problem is packed, one persistent GEMM launch per
 * tile kind covers all their (problem, product, tile) items, then each
 * problem's C is updated. When the batch needs more than one wave, waves
 * alternate between the two halves of the workspace: a wave's maxima and
 * packs (pack streams s[0..7]) wait only for the C updates of the wave before
 * last, which used the same half, so they run beside the previous wave's GEMM
 * and C updates (scatter streams s[8..15]); the GEMMs run in order on the
 * caller's stream. A problem too large for its share of the workspace runs
 * alone, after everything before it, with the whole workspace and product
 * groups. Every problem's result equals its single-call result. */
/* ------------------------------------------- batched waves: host side ---- */

/* the fields every wave kernel reads, for a bound job (its whole algorithm as one group) */
static WaveProb wave_prob(const SplitJob& j)
{
    WaveProb w;
    memset(&w, 0, sizeof(w));
    w.tab = j.alg.tab;
    w.A = j.A; w.B = j.B; w.C = j.C;
    w.amax = (unsigned long long*)(j.w + j.L.amax);
    w.bmax = (unsigned long long*)(j.w + j.L.bmax);
    w.e_row = (int*)(j.w + j.L.erow);
    w.f_col = (int*)(j.w + j.L.fcol);
    w.sa = j.w + j.L.sa;
    w.sb = j.w + j.L.sb;
    w.Z = job_zview(j);
    w.lda = j.lda; w.ldb = j.ldb; w.ldc = j.ldc;
    w.m = j.m; w.n = j.n; w.k = j.k;
    w.m_pad = j.d.m_pad; w.n_pad = j.d.n_pad; w.k_pad = j.d.k_pad;
    w.alpha = j.alpha; w.beta = j.beta;
    w.R = j.alg.R; w.kt = j.alg.kt; w.fmt = j.fmt;
    return w;
}

/* a table over jobs `qs`, each given gx and its block count by `size`; returns the launch's blocks */
template <class F>
static int64_t wave_table(WaveLaunch& L, const std::vector<SplitJob*>& qs, F size)
{
    L.nprob = 0;
    int64_t acc = 0;
    for (SplitJob* j : qs) {
        WaveProb& w = L.p[L.nprob++];
        w = wave_prob(*j);
        size(*j, w);
        w.b0 = acc;
        acc += w.nb;
    }
    return acc;
}

template <int S, int DB>
static void wave_packs_t(WaveLaunch& L, const std::vector<SplitJob*>& qs, cudaStream_t st)
{
    int64_t nb = wave_table(L, qs, [&](const SplitJob& j, WaveProb& w) {
        w.gx = (int64_t)j.alg.R * (j.d.m_pad / 64);
        w.nb = w.gx * (j.d.k_pad / 64);
    });
    wave_pack_a_kernel<S, DB><<<(unsigned)nb, 256, 0, st>>>(L);
    nb = wave_table(L, qs, [&](const SplitJob& j, WaveProb& w) {
        w.gx = (int64_t)j.alg.R * ((j.d.n_pad + 31) / 32);
        w.nb = w.gx * (j.d.k_pad / 64);
    });
    wave_pack_b_kernel<S, DB><<<(unsigned)nb, 256, 0, st>>>(L);
    fmm_count_launch(2);
}

/* maxima, exponents and digits of classical jobs of one format and slice
 * count: one launch per cluster size among them (chunks of at most 1024 k) */
static int wave_classical(int fmt, int s, WaveLaunch& L, const std::vector<SplitJob*>& qs, cudaStream_t st)
{
    for (int nrank = 1; nrank <= 8; nrank *= 2) {
        std::vector<SplitJob*> sel;
        for (SplitJob* j : qs)
            if (prep_ranks(3 * kSms, j->d.k_pad) == nrank) sel.push_back(j);
        if (sel.empty()) continue;
        const int64_t nb = wave_table(L, sel, [&](const SplitJob& j, WaveProb& w) {
            w.gx = 1;
            w.nb = (j.d.m_pad + j.d.n_pad) / kPrepLines * nrank;
        });
        const int rc = with_slices(fmt, s, [&](auto S, auto DB) {
            return launch_clusters(wave_classical_kernel<S(), DB()>, nb, nrank, st, L, nrank);
        });
        if (rc != FMM_OK) return rc;
    }
    return FMM_OK;
}

/* The side work before a wave's GEMM, one launch per kernel over the bound
 * jobs qs (all products of each as one group). Classical jobs: prep_kernel's
 * work per (slice count, format). Others: maxima zeroing, maxima, exponents,
 * then the packs per (slice count, format). */
static int wave_side_pack(const std::vector<SplitJob*>& all, cudaStream_t st)
{
    WaveLaunch L;
    std::vector<SplitJob*> qs, cl;
    for (SplitJob* j : all) (j->classical ? cl : qs).push_back(j);
    auto each_kind = [](const std::vector<SplitJob*>& js, auto f) -> int {
        std::vector<std::pair<int, int>> kinds;
        for (SplitJob* j : js)
            if (std::find(kinds.begin(), kinds.end(), std::make_pair(j->fmt, j->s)) == kinds.end())
                kinds.emplace_back(j->fmt, j->s);
        for (auto [fmt, sl] : kinds) {
            std::vector<SplitJob*> sel;
            for (SplitJob* j : js)
                if (j->fmt == fmt && j->s == sl) sel.push_back(j);
            if (int rc = f(fmt, sl, sel); rc != FMM_OK) return rc;
        }
        return FMM_OK;
    };
    if (int rc = each_kind(cl, [&](int fmt, int sl, auto& sel) { return wave_classical(fmt, sl, L, sel, st); });
        rc != FMM_OK)
        return rc;
    if (!qs.empty()) {
        int64_t nb = wave_table(L, qs, [](const SplitJob& j, WaveProb& w) {
            const int64_t total = (int64_t)j.alg.kt * (j.m + j.n);
            w.gx = 1;
            w.nb = std::min<int64_t>(std::max<int64_t>((total + 2047) / 2048, 1), 2048);
        });
        wave_prep_kernel<<<(unsigned)nb, 256, 0, st>>>(L);
        nb = wave_table(L, qs, [](const SplitJob& j, WaveProb& w) {
            w.gx = (j.m + 255) / 256 * j.alg.kt * ((j.d.ke + 255) / 256);
            w.nb = w.gx + ((int64_t)j.alg.kt * j.n * 32 + 255) / 256;
        });
        wave_maxima_kernel<<<(unsigned)nb, 256, 0, st>>>(L);
        nb = wave_table(L, qs, [](const SplitJob& j, WaveProb& w) {
            w.gx = (j.d.m_pad + j.d.n_pad + 255) / 256;
            w.nb = w.gx * j.alg.R;
        });
        wave_exps_kernel<<<(unsigned)nb, 256, 0, st>>>(L);
        fmm_count_launch(3);
        each_kind(qs, [&](int fmt, int sl, auto& sel) {
            return with_slices(fmt, sl, [&](auto S, auto DB) {
                wave_packs_t<S(), DB()>(L, sel, st);
                return (int)FMM_OK;
            });
        });
    }
    return cudaGetLastError() == cudaSuccess ? FMM_OK : FMM_ERR_CUDA;
}

/* The C updates after a wave's GEMM, a launch per kind: classical jobs (bound by
 * HBM, no shared memory, full blocks), the other jobs that the element-major
 * form is better for, those of many products among them apart (on st_long), and
 * the rest by sub-block. One element-major launch for all of them would run
 * every job with the fewest threads and the most shared memory any of them
 * needs: 322 x2 at 963 x 267 x 134 with a classical 675 x 2091 x 595, 829 us for
 * the batch against 205. The launches of short blocks run one after the other
 * on one stream: on one each they cost a batch of two kinds 6 us more. */
static int wave_side_scatter(const std::vector<SplitJob*>& qs, cudaStream_t st, cudaStream_t st_long)
{
    /* Classical, element-major (up to kLongProducts products, and more), by sub-block. A job of many products has long
     * blocks; where the launch is about one round of blocks (six per SM), other jobs' blocks in front of them push its
     * last ones into a second round: five problems, 861 of 940 blocks of 232 x2 at 1654 x 1967, 771 us for the batch,
     * 653 with that one in a launch of its own. */
    constexpr int kLongProducts = 64, kBySubBlock = 3;
    std::vector<SplitJob*> kinds[4];
    int T[3] = {256, 256, 256};
    for (SplitJob* j : qs) {
        int Tj;
        size_t sm;
        if (job_scatter_all(*j, 0, j->alg.R, &Tj, &sm) && scatter_all_better(*j, INT64_MAX)) {
            const int x = j->classical ? 0 : j->alg.R <= kLongProducts ? 1 : 2;
            kinds[x].push_back(j);
            T[x] = std::min(T[x], Tj);
        } else {
            kinds[kBySubBlock].push_back(j);
        }
    }
    auto tiles_of = [&](const SplitJob& j, int x) { return scatter_tiles(j, j.d.me, j.d.ne, T[x]); };
    int64_t together = 0;
    for (SplitJob* j : kinds[1]) together += tiles_of(*j, 1);
    for (int x = 1; x < kBySubBlock; ++x) {
        const auto rest = std::stable_partition(kinds[x].begin(), kinds[x].end(), [&](SplitJob* j) {
            return scatter_all_better(*j, x == 1 ? together : tiles_of(*j, x));
        });
        kinds[kBySubBlock].insert(kinds[kBySubBlock].end(), rest, kinds[x].end());
        kinds[x].erase(rest, kinds[x].end());
    }
    /* the only job of a kind: the kernel of single calls, with one form's registers and a hundredth of the parameters */
    for (int x = 0; x <= kBySubBlock; ++x) {
        if (kinds[x].size() != 1) continue;
        const SplitJob& j = *kinds[x][0];
        if (x == kBySubBlock)
            job_scatter_parts(j, 0, j.alg.R, st);
        else
            job_scatter_block(j, 0, j.alg.R, 0, j.d.me, 0, j.d.ne, x == 2 ? st_long : st);
        kinds[x].clear();
    }
    WaveLaunch L;
    for (int x = 0; x < kBySubBlock; ++x) {
        if (kinds[x].empty()) continue;
        /* a job's work: per tile each product's Z, each W entry's update, each sub-block's C in and out */
        std::vector<double> work;
        size_t smem = 0;
        int64_t all_tiles = 0;
        double all_work = 0.0;
        for (SplitJob* j : kinds[x]) {
            const Tab ht = tab_view(j->alg.htab);
            const int P = j->alg.mt * j->alg.nt, E = ht.w_off[j->alg.R] - ht.w_off[0];
            if (x > 0) smem = std::max(smem, scatter_all_smem(P, T[x], E, j->alg.R));
            const int64_t t = tiles_of(*j, x);
            work.push_back((double)t * (double)(j->alg.R + E + 2 * P));
            all_tiles += t;
            all_work += work.back();
        }
        /* a block per tile, or the most blocks of a launch shared out by work, so that a block's set-up serves several
         * tiles in a wave of many problems and no job is left with a few long blocks */
        const double per_work = (double)scatter_blocks(INT64_MAX) / all_work;
        const bool fits = scatter_blocks(all_tiles) == all_tiles;
        size_t q = 0;
        const int64_t nb = wave_table(L, kinds[x], [&](const SplitJob& j, WaveProb& w) {
            const int64_t t = tiles_of(j, x);
            w.gx = 1;
            w.nb = fits ? t : std::min(std::max<int64_t>(1, (int64_t)(per_work * work[q])), t);
            ++q;
        });
        (x == 0 ? wave_scatter_one_kernel : wave_scatter_kernel)<<<(unsigned)nb, (unsigned)T[x], smem,
                                                                     x == 2 ? st_long : st>>>(L);
        fmm_count_launch(1);
    }
    if (!kinds[kBySubBlock].empty()) {
        const int64_t nb = wave_table(L, kinds[kBySubBlock], [&](const SplitJob& j, WaveProb& w) {
            w.gx = scatter_part_tiles(j, &w.tr);
            w.nb = w.gx * j.alg.mt * j.alg.nt;
        });
        wave_scatter_part_kernel<<<(unsigned)nb, kScatterThreads, 0, st>>>(L);
        fmm_count_launch(1);
    }
    return cudaGetLastError() == cudaSuccess ? FMM_OK : FMM_ERR_CUDA;
}

int fmm_split_batch(int count, const SplitJob* jobs_in, void* ws, size_t ws_bytes, cudaStream_t st)
{
    std::lock_guard<std::mutex> use(g_side_use);
    SidePool* sp = side_pool();
    std::vector<SplitJob> jobs(jobs_in, jobs_in + count);
    std::vector<size_t> full(count, 0);
    size_t total = 0;
    int nontrivial = 0;
    for (int i = 0; i < count; ++i)
        if (!jobs[i].trivial) {
            const WsLayout Lf = ws_layout_g(jobs[i].alg, jobs[i].d, jobs[i].m, jobs[i].n, jobs[i].s, jobs[i].alg.R,
                                            jobs[i].fmt);
            full[i] = Lf.total;
            total += (full[i] + 255) / 256 * 256;
            ++nontrivial;
        }
    /* one wave over the whole workspace when everything fits at once;
     * otherwise two halves that waves alternate between */
    const bool halves = sp != nullptr && (total > ws_bytes || nontrivial > kMaxLaunchProblems);
    const size_t share = halves ? ws_bytes / 2 / 256 * 256 : ws_bytes;
    auto pack_st = [&](int x) { return sp ? sp->s[x % kWaveStreams] : st; };
    auto scat_st = [&](int x) { return sp ? sp->s[kWaveStreams + x % kWaveStreams] : st; };
    auto ok = [](cudaError_t e) { return e == cudaSuccess; };
    bool half_used[2] = {false, false};
    struct Wave {
        int i, e, h;
    };
    int wave = 0;

    /* a wave's maxima, exponents and packs on the pack streams, after the C
     * updates of the last wave in its half; the GEMM stream then waits */
    auto pack_wave = [&](const Wave& W) -> int {
        uint8_t* base = (uint8_t*)ws + (size_t)W.h * share;
        if (sp && half_used[W.h])
            for (int x = 0; x < kWaveStreams; ++x)
                for (int y = 0; y < kWaveStreams; ++y)
                    if (!ok(cudaStreamWaitEvent(pack_st(x), sp->wave_sc[W.h][y], 0))) return FMM_ERR_CUDA;
        size_t off = 0;
        std::vector<SplitJob*> qs;
        for (int q = W.i; q < W.e; ++q) {
            SplitJob& j = jobs[q];
            int rc = job_bind_group(j, base + off, full[q], j.alg.R);
            if (rc != FMM_OK) return rc;
            off += (full[q] + 255) / 256 * 256;
            qs.push_back(&j);
        }
        /* the full-size tiles: measured, a wave's side kernels do not overlap the previous wave's GEMM (its
         * CTAs hold the SMs), so the tiles that fit beside a GEMM CTA only make them slower */
        if (int rc = wave_side_pack(qs, pack_st(0)); rc != FMM_OK) return rc;
        if (sp)
            for (int x = 0; x < kWaveStreams; ++x)
                if (!ok(cudaEventRecord(sp->wave_pk[W.h][x], pack_st(x)))) return FMM_ERR_CUDA;
        return FMM_OK;
    };
    /* one persistent GEMM launch per tile kind over the wave's items, the
     * costliest items (slice pairs x k blocks) first so the CTAs' shares end
     * evenly; pair-tile problems and the rest give the same bits per tile */
    auto gemm_wave = [&](const Wave& W) -> int {
        if (sp)
            for (int x = 0; x < kWaveStreams; ++x)
                if (!ok(cudaStreamWaitEvent(st, sp->wave_pk[W.h][x], 0))) return FMM_ERR_CUDA;
        std::vector<int> ord;
        for (int q = W.i; q < W.e; ++q) ord.push_back(q);
        auto item_cost = [&](int q) {
            return (int64_t)jobs[q].s * (jobs[q].s + 1) / 2 * (jobs[q].d.k_pad / kbe_of(jobs[q].fmt)) /
                   (jobs[q].fmt ? 2 : 1);   /* FP8 MMAs run at twice the BF16 rate */
        };
        std::stable_sort(ord.begin(), ord.end(), [&](int a, int b) { return item_cost(a) > item_cost(b); });
        GemmLaunch gl;
        for (int pass = 0; pass < 2; ++pass) {
            const bool pair = pass == 0;
            memset(&gl, 0, sizeof(gl));
            int64_t items = 0;
            int prods = 0;
            for (int q : ord) {
                SplitJob& j = jobs[q];
                if (job_pair(j) != pair) continue;
                if (gl.sched == nullptr) gl.sched = (unsigned int*)(j.w + j.L.sched);
                int rc = job_fill(j, gl.prob[gl.nprob++], j.alg.R, (int)items, pair);
                if (rc != FMM_OK) return rc;
                items += job_items(j, j.alg.R, pair);
                prods += j.alg.R;
            }
            if (gl.nprob == 0) continue;
            if (int rc = launch_gemm(gl, items, prods, st, pair); rc != FMM_OK) return rc;
        }
        if (sp && !ok(cudaEventRecord(sp->wave_gm[W.h], st))) return FMM_ERR_CUDA;
        return FMM_OK;
    };
    /* each problem's C update (disjoint C regions) on the scatter streams */
    auto scatter_wave = [&](const Wave& W) -> int {
        if (sp)
            for (int y = 0; y < kWaveStreams; ++y)
                if (!ok(cudaStreamWaitEvent(scat_st(y), sp->wave_gm[W.h], 0))) return FMM_ERR_CUDA;
        std::vector<SplitJob*> qs;
        for (int q = W.i; q < W.e; ++q) qs.push_back(&jobs[q]);
        if (int rc = wave_side_scatter(qs, scat_st(0), scat_st(1)); rc != FMM_OK) return rc;
        if (sp)
            for (int y = 0; y < kWaveStreams; ++y)
                if (!ok(cudaEventRecord(sp->wave_sc[W.h][y], scat_st(y)))) return FMM_ERR_CUDA;
        half_used[W.h] = true;
        return FMM_OK;
    };

    /* software pipeline, enqueued as GEMM(w), packs(w+1), C updates(w): a pack
     * stream that shares a hardware queue with a scatter stream then never
     * has its work behind the C updates' wait for GEMM(w) */
    bool pending = false;
    Wave P{0, 0, 0};
    auto flush = [&]() -> int {
        if (!pending) return FMM_OK;
        pending = false;
        int rc = gemm_wave(P);
        return rc != FMM_OK ? rc : scatter_wave(P);
    };
    if (int rc = side_fork(sp, st); rc != FMM_OK) return rc;   /* side streams start after the caller's work */
    int i = 0;
    while (i < count) {
        if (jobs[i].trivial) {
            int rc = job_prologue(jobs[i], st);
            if (rc != FMM_OK) return rc;
            ++i;
            continue;
        }
        if (full[i] > share) {
            /* alone, after every wave before it, with the whole workspace */
            SplitJob& j = jobs[i];
            int rc = flush();
            if (rc == FMM_OK) rc = side_join(sp, st);
            if (rc == FMM_OK)
                rc = split_launch_budget(j.alg, j.m, j.n, j.k, j.alpha, j.A, j.lda, j.B, j.ldb, j.beta, j.C, j.ldc,
                                         j.s, j.fmt, ws, ws_bytes, ws_bytes, st, sp);
            if (rc == FMM_OK) rc = side_fork(sp, st);
            if (rc != FMM_OK) return rc;
            half_used[0] = half_used[1] = false;
            ++i;
            continue;
        }
        /* gather a wave */
        int e = i;
        size_t used = 0;
        while (e < count && e - i < kMaxLaunchProblems && !jobs[e].trivial && used + full[e] <= share &&
               (int64_t)jobs[e].alg.R * jobs[e].s * std::max(jobs[e].d.m_pad, jobs[e].d.n_pad) <= 0x7fffffffLL) {
            used += (full[e] + 255) / 256 * 256;
            ++e;
        }
        if (e == i) return FMM_ERR_WORKSPACE;
        const Wave W{i, e, halves ? (wave & 1) : 0};
        ++wave;
        int rc = FMM_OK;
        if (halves) {
            /* W packs into the other half than the pending wave */
            if (pending) rc = gemm_wave(P);
            if (rc == FMM_OK) rc = pack_wave(W);
            if (rc == FMM_OK && pending) rc = scatter_wave(P);
        } else {
            /* one region: the pending wave is done with it first */
            rc = flush();
            if (rc == FMM_OK) rc = pack_wave(W);
        }
        if (rc != FMM_OK) return rc;
        P = W;
        pending = true;
        i = e;
    }
    if (int rc = flush(); rc != FMM_OK) return rc;
    if (int rc = side_join(sp, st); rc != FMM_OK) return rc;   /* the caller's stream waits for everything */
    return cudaGetLastError() == cudaSuccess ? FMM_OK : FMM_ERR_CUDA;
}

/* workspace the batch would use with everything in one wave where possible */
size_t fmm_split_batch_ws(int count, const SplitJob* jobs)
{
    size_t sum = 0, mx = 0;
    for (int i = 0; i < count; ++i) {
        if (jobs[i].trivial) continue;
        const size_t f =
            ws_layout_g(jobs[i].alg, jobs[i].d, jobs[i].m, jobs[i].n, jobs[i].s, jobs[i].alg.R, jobs[i].fmt).total;
        sum += (f + 255) / 256 * 256;
        const size_t one = ws_layout(jobs[i].alg, jobs[i].m, jobs[i].n, jobs[i].k, jobs[i].s, 1, jobs[i].fmt).total;
        mx = std::max(mx, one);
    }
    return std::max(std::min(sum, kGroupBudget), mx);
}

int fmm_split_job_make(SplitJob** out, const AlgView& alg, int64_t m, int64_t n, int64_t k, double alpha,
                       const double* A, int64_t lda, const double* B, int64_t ldb, double beta, double* C,
                       int64_t ldc, int s)
{
    SplitJob* j = new SplitJob;
    int rc = job_init(*j, alg, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, s);
    if (rc != FMM_OK) { delete j; return rc; }
    *out = j;
    return FMM_OK;
}

void fmm_split_job_free(SplitJob* j) { delete j; }

int fmm_split_launch(const AlgView& alg, int64_t m, int64_t n, int64_t k, double alpha,
                     const double* A, int64_t lda, const double* B, int64_t ldb, double beta,
                     double* C, int64_t ldc, int s, int fmt, void* ws, size_t ws_bytes, cudaStream_t st)
{
    /* the group size follows the workspace the caller provides */
    std::lock_guard<std::mutex> use(g_side_use);
    return split_launch_budget(alg, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, s, fmt, ws, ws_bytes,
                               ws_bytes, st, side_pool());
}

/* ---------------------------------------------------------------------------
 * Allocation-free entry point.
 *
 * For callers that must not allocate device memory while they run: stream
 * callbacks and host functions, plug-ins that run on memory handed to them by
 * a host application with its own allocator, or processes whose device memory
 * is already fully reserved. Such callers cannot use fmm_gpu_split_dgemm,
 * whose workspace they would have to obtain, nor the table cache, which
 * allocates on first use of an algorithm. This variant keeps the algorithm
 * table and the whole workspace in one file-scope device array of
 * kNoAllocScratchBytes (64 MiB), which every GPU that loads the library holds
 * until the process exits.
 * ------------------------------------------------------------------------- */
constexpr size_t kNoAllocScratchBytes = (size_t)64 << 20;
static __device__ __align__(256) uint8_t g_noalloc_scratch[kNoAllocScratchBytes];

namespace {
std::mutex g_noalloc_mu;
uint8_t* g_noalloc_ptr[64];

/* One piece of an algorithm table, passed by value: the launch copies the
 * values when it is enqueued, so no host buffer has to outlive the call. */
constexpr int kTabChunkInts = 4000;
struct TabChunk {
    int n;
    int v[kTabChunkInts];
};

__global__ void __launch_bounds__(256) noalloc_table_kernel(int* __restrict__ dst, const __grid_constant__ TabChunk c)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < c.n; i += gridDim.x * blockDim.x) dst[i] = c.v[i];
}
}  // namespace

extern "C" int fmm_gpu_split_dgemm_noalloc(const fmm_t* fmm, int levels, int64_t m, int64_t n, int64_t k,
                                           double alpha, const double* A, int64_t lda, const double* B,
                                           int64_t ldb, double beta, double* C, int64_t ldc, int slices,
                                           void* stream)
{
    if (m < 0 || n < 0 || k < 0 || slices < 2 || slices > 8) return FMM_ERR_ARG;
    if (lda < (m > 1 ? m : 1) || ldb < (k > 1 ? k : 1) || ldc < (m > 1 ? m : 1)) return FMM_ERR_ARG;
    if (m > 0 && n > 0 && C == nullptr) return FMM_ERR_ARG;
    if (m > 0 && n > 0 && k > 0 && (A == nullptr || B == nullptr)) return FMM_ERR_ARG;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return FMM_ERR_CUDA;
    uint8_t* scratch;
    {
        /* once per device, with that device current: the device address of
         * the static array (its host-side name is only a stand-in) */
        std::lock_guard<std::mutex> lk(g_noalloc_mu);
        if (g_noalloc_ptr[dev] == nullptr) {
            void* p = nullptr;
            if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || p == nullptr) return FMM_ERR_CUDA;
            g_noalloc_ptr[dev] = (uint8_t*)p;
        }
        scratch = g_noalloc_ptr[dev];
    }
    fmm_t flat;
    int owned = 0;
    int rc = fmm_flatten(fmm, levels, &flat, &owned);
    if (rc != FMM_OK) return rc;
    std::vector<int> table;
    AlgView alg;
    rc = fmm_alg_describe(&flat, &table, &alg);
    if (owned) free_fmm(flat);
    if (rc != FMM_OK) return rc;
    const size_t tab_bytes = (sizeof(int) * table.size() + 255) / 256 * 256;
    if (tab_bytes >= kNoAllocScratchBytes) return FMM_ERR_SCRATCH;
    const size_t ws_bytes = kNoAllocScratchBytes - tab_bytes;
    if (m > 0 && n > 0 && k > 0 && alpha != 0.0 && ws_layout(alg, m, n, k, slices, ws_bytes).total > ws_bytes)
        return FMM_ERR_SCRATCH;
    if (fmm_device_error_word() == nullptr) return FMM_ERR_CUDA;
    cudaStream_t st = (cudaStream_t)stream;
    /* the table goes to the front of the scratch, written by kernels that
     * carry it as their parameter (never a copy from this call's host vector,
     * which is gone once the call returns) */
    for (size_t off = 0; off < table.size(); off += kTabChunkInts) {
        TabChunk c;
        c.n = (int)std::min<size_t>(kTabChunkInts, table.size() - off);
        std::memcpy(c.v, table.data() + off, sizeof(int) * (size_t)c.n);
        noalloc_table_kernel<<<(c.n + 255) / 256, 256, 0, st>>>((int*)scratch + off, c);
        if (cudaGetLastError() != cudaSuccess) return FMM_ERR_CUDA;
        fmm_count_launch(1);
    }
    alg.tab = (const int*)scratch;
    alg.htab = table.data();
    return split_launch_budget(alg, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, slices, 0, scratch + tab_bytes,
                               ws_bytes, ws_bytes, st, nullptr);
}

/* ---------------------------------------------------------------------------
 * Batched entry point (include/fmm_gb300.h).
 * ------------------------------------------------------------------------- */
namespace {

/* Validates a batch and describes its problems. With `host_tables` (sizing
 * only) the algorithm tables are built on the host and kept in it, so sizing
 * needs no device; otherwise they are the cached device tables. */
int batch_jobs(int count, const fmm_batch_problem* probs, std::vector<SplitJob>& jobs,
               std::vector<int>& f64_idx, std::vector<AlgView>& f64_alg,
               std::deque<std::vector<int>>* host_tables = nullptr)
{
    if (count < 0 || (count > 0 && probs == nullptr)) return FMM_ERR_ARG;
    for (int i = 0; i < count; ++i) {
        const fmm_batch_problem& p = probs[i];
        if (p.m < 0 || p.n < 0 || p.k < 0) return FMM_ERR_ARG;
        if (p.lda < (p.m > 1 ? p.m : 1) || p.ldb < (p.k > 1 ? p.k : 1) || p.ldc < (p.m > 1 ? p.m : 1))
            return FMM_ERR_ARG;
        if (p.m > 0 && p.n > 0 && p.C == nullptr) return FMM_ERR_ARG;
        if (p.m > 0 && p.n > 0 && p.k > 0 && (p.A == nullptr || p.B == nullptr)) return FMM_ERR_ARG;
        if (p.format != 0 && p.format != 1) return FMM_ERR_ARG;
        if (p.slices != 0 && (p.slices < 2 || p.slices > (p.format ? 12 : 8))) return FMM_ERR_ARG;
        fmm_t flat;
        int owned = 0;
        int rc = fmm_flatten(p.fmm, p.fmm ? p.levels : 0, &flat, &owned);
        if (rc != FMM_OK) return rc;
        AlgView alg;
        if (host_tables) {
            host_tables->emplace_back();
            rc = fmm_alg_describe(&flat, &host_tables->back(), &alg);
        } else {
            rc = fmm_alg_get(&flat, &alg);
        }
        if (owned) free_fmm(flat);
        if (rc != FMM_OK) return rc;
        if (p.slices == 0) {
            f64_idx.push_back(i);
            f64_alg.push_back(alg);
            continue;
        }
        SplitJob j;
        rc = job_init(j, alg, p.m, p.n, p.k, p.alpha, p.A, p.lda, p.B, p.ldb, p.beta, p.C, p.ldc, p.slices,
                      p.format);
        if (rc != FMM_OK) return rc;
        jobs.push_back(j);
    }
    return FMM_OK;
}

}  // namespace

/* Batch workspace: the FP64 problems' table, then the split problems' region. */
static size_t batch_f64_bytes(size_t nf64) { return nf64 ? fmm_f64_batch_ws_bytes((int)nf64) : 0; }

extern "C" size_t fmm_gpu_batch_workspace_size(int count, const fmm_batch_problem* probs)
{
    std::vector<SplitJob> jobs;
    std::vector<int> fi;
    std::vector<AlgView> fa;
    std::deque<std::vector<int>> tables;
    if (batch_jobs(count, probs, jobs, fi, fa, &tables) != FMM_OK) return 0;
    const size_t split = jobs.empty() ? 0 : fmm_split_batch_ws((int)jobs.size(), jobs.data());
    return std::max<size_t>(256, batch_f64_bytes(fi.size()) + split);
}

extern "C" int fmm_gpu_batch_dgemm(int count, const fmm_batch_problem* probs, void* workspace,
                                   size_t workspace_bytes, void* stream)
{
    std::vector<SplitJob> jobs;
    std::vector<int> fi;
    std::vector<AlgView> fa;
    int rc = batch_jobs(count, probs, jobs, fi, fa);
    if (rc != FMM_OK) return rc;
    if (fmm_device_error_word() == nullptr) return FMM_ERR_CUDA;
    cudaStream_t st = (cudaStream_t)stream;
    const size_t f64_bytes = batch_f64_bytes(fi.size());
    if (!fi.empty()) {
        /* all FP64 problems in one persistent launch */
        std::vector<F64BatchItem> items(fi.size());
        for (size_t q = 0; q < fi.size(); ++q) {
            const fmm_batch_problem& p = probs[fi[q]];
            items[q] = F64BatchItem{fa[q], p.m, p.n, p.k, p.alpha, p.beta, p.A, p.lda, p.B, p.ldb, p.C, p.ldc};
        }
        rc = fmm_f64_batch_launch((int)items.size(), items.data(), workspace, workspace_bytes, st);
        if (rc != FMM_OK) return rc;
    }
    if (!jobs.empty()) {
        if (workspace_bytes < f64_bytes) return FMM_ERR_WORKSPACE;
        workspace = workspace ? (void*)((uint8_t*)workspace + f64_bytes) : nullptr;
        workspace_bytes -= f64_bytes;
    }
    if (jobs.empty()) return FMM_OK;
    return fmm_split_batch((int)jobs.size(), jobs.data(), workspace, workspace_bytes, st);
}

/* ---------------------------------------------------------------------------
 * Self-test of the failure path every kernel wait relies on: one CTA waits,
 * with the library's bounded mbarrier wait (sm103::mbar_wait, the one the GEMM
 * kernels use), on a barrier that nothing arrives at. After the wait limit it
 * must record `code` in the device error word, raise the CTA's abort flag so
 * the other waiting threads give up too, and return; the kernel then ends
 * normally and the context stays usable.
 * ------------------------------------------------------------------------- */
namespace {
__global__ void __launch_bounds__(64) selftest_wait_kernel(int* err, int code, int* gave_up)
{
    __shared__ uint64_t bar;
    __shared__ volatile int abort_flag;
    if (threadIdx.x == 0) {
        sm103::mbar_init(&bar, 1);     /* one arrival expected; none comes */
        abort_flag = 0;
        sm103::fence_mbar_init();
    }
    __syncthreads();
    const bool ok = sm103::mbar_wait(&bar, 0, &abort_flag, err, code);
    if (!ok) atomicAdd(gave_up, 1);
}
}  // namespace

extern "C" int fmm_gpu_selftest_wait_expiry(int* threads_gave_up)
{
    int* err = fmm_device_error_word();
    if (err == nullptr) return FMM_ERR_CUDA;
    int* d_gave = nullptr;
    if (cudaMalloc(&d_gave, sizeof(int)) != cudaSuccess) return FMM_ERR_ALLOC;
    int rc = FMM_OK;
    if (cudaMemset(d_gave, 0, sizeof(int)) != cudaSuccess) rc = FMM_ERR_CUDA;
    if (rc == FMM_OK) {
        selftest_wait_kernel<<<1, 64>>>(err, 99, d_gave);
        fmm_count_launch(1);
        if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess) rc = FMM_ERR_CUDA;
    }
    int gave = 0;
    if (rc == FMM_OK && cudaMemcpy(&gave, d_gave, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) rc = FMM_ERR_CUDA;
    cudaFree(d_gave);
    if (threads_gave_up) *threads_gave_up = gave;
    if (rc != FMM_OK) return rc;
    return fmm_device_error_status();
}

extern "C" void fmm_gpu_set_host_timeline(int enable) { g_timeline.store(enable != 0); }

extern "C" int fmm_gpu_read_host_timeline(double* ms, int count)
{
    if (ms == nullptr || count < 0) return FMM_ERR_ARG;
    std::lock_guard<std::mutex> lk(g_timeline_mu);
    const int c = std::min(count, kTimelinePoints + 1);
    for (int x = 0; x < c; ++x) ms[x] = g_timeline_ms[x];
    return c;
}
