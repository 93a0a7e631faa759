/*
 * Plain FP64 form of the FMM GEMM (and, with the trivial algorithm, the
 * classical FP64 GEMM it is compared against).
 *
 * On GB300 the FP64 pipe delivers about 2 FMA/clock/SM (1.2 TFLOP/s on the
 * GPU; the FP64 mma.sync path measures slightly slower), so this form is
 * bound by FP64 FMAs and everything else is arranged to cost few of them:
 *
 *  - one CTA owns an output tile position (ti, tj) of the ceil(m/m~) x
 *    ceil(n/n~) product grid and runs every product r over it, so a C
 *    sub-block tile is only ever updated by its owning CTA: no atomics, a
 *    fixed summation order, one launch for the whole algorithm;
 *  - per k step it loads the nnz(U[:,r]) A sub-block tiles and nnz(V[:,r]) B
 *    sub-block tiles straight from the caller's column-major matrices with
 *    coalesced loads, forms the weighted sums in FP64 in registers (the fused
 *    multi-operand pack, plugin/ref_kernels/bli_packm_fmm_ref.c:89-147, with
 *    zero fill past a smaller sub-block as in :133-134) and stores the
 *    combined operand tiles to shared memory;
 *  - a register-blocked DFMA micro-kernel multiplies the tiles (in place of
 *    bli_dgemm_haswell_asm_6x8 called at plugin/ref_kernels/bli_gemm_fmm_ref.c:85-97);
 *  - the k loop stays in registers, and the epilogue adds alpha*W[p,r]*tile
 *    into every C sub-block p with W[p,r] != 0, clipped to its size
 *    (bli_gemm_fmm_ref.c:99-120), with one coalesced read-modify-write per
 *    (product, sub-block) instead of one per KC block.
 */
#include "fmm_internal.h"
#include "sm103_ptx.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

namespace cg = cooperative_groups;

/* k chunks of the small/skinny classical path for an m x n x k FP64
 * problem, 0 when the regular kernel runs it: at most 128 output tiles of
 * 32 x 32, chunks of at least 256 k, at most 8 chunks (a portable cluster)
 * and at most 256 CTAs. A function of the shape only, so single and batched
 * calls take the same path. */
extern "C" int fmm_gpu_f64_sup_splits(int64_t m, int64_t n, int64_t k)
{
    if (m <= 0 || n <= 0 || k <= 0) return 0;
    const int64_t tiles = ((m + 31) / 32) * ((n + 31) / 32);
    if (tiles > 128) return 0;
    const int64_t ks = std::min<int64_t>({8, 256 / tiles, k / 256});
    return ks >= 2 ? (int)ks : 0;
}

/* chunk length: k / ks rounded up to whole 32-k steps; every chunk is
 * non-empty because each holds at least 256 k */
int64_t fmm_f64_sup_chunk(int64_t k, int ks)
{
    return ((k + ks - 1) / ks + 31) / 32 * 32;
}

/* the trivial 1 x 1 x 1 algorithm with all three coefficients +1: the
 * classical GEMM C += alpha * A * B */
bool fmm_plain_classical(const AlgView& alg)
{
    if (alg.R != 1 || alg.mt != 1 || alg.kt != 1 || alg.nt != 1 || alg.htab == nullptr) return false;
    const int* t = alg.htab;
    const int* u_off = t + FMM_ALG_HDR;
    const int* v_off = u_off + 2;
    const int* w_off = v_off + 2;
    const int* u_ent = w_off + 2;
    const int* v_ent = u_ent + 2 * u_off[1];
    const int* w_ent = v_ent + 2 * v_off[1];
    return u_off[1] == 1 && v_off[1] == 1 && w_off[1] == 1 && u_ent[1] == 1 && v_ent[1] == 1 && w_ent[1] == 1;
}

namespace {

constexpr int kMaxEntries = 256;  /* nonzero coefficients per product column */

/* micro-kernel of the plain form (fmm_gpu_set_f64_engine): FMM_F64_DFMA or FMM_F64_MMA */
std::atomic<int> g_f64_engine{FMM_F64_DFMA};

struct Entry {
    const double* base;  /* sub-block origin in the source matrix */
    double coef;         /* small integer coefficient, already a double */
    int rows, cols;      /* sub-block extent */
    int kind;            /* 0: +1, 1: -1, 2: other (no FP64 compare per element) */
    int pad;
};

/* first term of a combination: s[t] = c * v[t], exact like the FP64
 * product; sign flips for c = +-1 keep it off the FP64 pipe that the
 * micro-kernel is bound by. One uniform branch for all of a thread's values. */
template <int N>
__device__ __forceinline__ void scale_first(const Entry& x, double (&s)[N])
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

/* Geometry of the nonzero entries [beg, end) of one product column of U
 * (or V), for a source split rt x ct, into shared memory. */
__device__ void stage_entries(const int* __restrict__ ent, int beg, int end, int ct,
                              int rt, const double* src, int64_t ld, int64_t rows_total,
                              int64_t cols_total, Entry* out)
{
    for (int e = beg + (int)threadIdx.x; e < end; e += blockDim.x) {
        int part = ent[2 * e], coef = ent[2 * e + 1];
        int64_t ro, rl, co, cl;
        fmm_part_geom(rows_total, rt, part / ct, &ro, &rl);
        fmm_part_geom(cols_total, ct, part % ct, &co, &cl);
        Entry x;
        x.base = src + ro + co * ld;
        x.rows = (int)rl;
        x.cols = (int)cl;
        x.coef = (double)coef;
        x.kind = coef == 1 ? 0 : (coef == -1 ? 1 : 2);
        x.pad = 0;
        out[e - beg] = x;
    }
}

/* One output tile position (ti, tj) of the ceil(m/m~) x ceil(n/n~) product
 * grid: every product r of the algorithm over it, with the fused packs, the
 * DFMA micro-kernel and the multi-C epilogue. Shared by the single-problem
 * kernel (one CTA per tile position) and the batched one (a work queue of
 * (problem, tile position) items). */
/* Shared-memory layout of the combined operand tiles. DFMA engine: A as
 * [k][m] and B as [k][n], pitch +1 (the micro-kernel reads a row of each).
 * FP64 MMA engine: A as [k][m] with pitch BM + 8 and B transposed to [n][k]
 * with pitch BK + 4, so both the fused packs' stores (consecutive m, or
 * consecutive k) and the m8n8k4 fragment loads (A[gid][tig], B[tig][gid])
 * hit distinct banks. */
template <int BM, int BN, int BK, bool MMA>
struct F64Smem {
    static constexpr int PA = MMA ? BM + 8 : BM + 1;
    static constexpr int PB = MMA ? BK + 4 : BN + 1;
    static constexpr int A_ELEMS = BK * PA;
    static constexpr int B_ELEMS = MMA ? BN * PB : BK * PB;
    __device__ static __forceinline__ int a(int kk, int mm) { return kk * PA + mm; }
    __device__ static __forceinline__ int b(int kk, int nn) { return MMA ? nn * PB + kk : kk * PB + nn; }
};

/* D += A * B on an 8 x 8 x 4 FP64 tile, one warp (mma.sync.m8n8k4.f64):
 * a = A[gid][tig], b = B[tig][gid], d = D[gid][2 tig .. 2 tig + 1] with
 * gid = lane / 4, tig = lane % 4. */
__device__ __forceinline__ void mma_f64_8x8x4(double (&d)[2], double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

template <int BM, int BN, int BK, int TM, int TN, bool MMA>
__device__ __forceinline__ void f64_tile(const int* __restrict__ tab, int64_t m, int64_t n, int64_t k,
                                         double alpha, const double* __restrict__ A, int64_t lda,
                                         const double* __restrict__ B, int64_t ldb,
                                         double* __restrict__ C, int64_t ldc, int ti, int tj,
                                         double* As, double* Bs,
                                         Entry* ue, Entry* ve, int r_begin, int r_end,
                                         const double* __restrict__ Sp, const double* __restrict__ Tp)
{
    using SM = F64Smem<BM, BN, BK, MMA>;
    constexpr int NT = (BM / TM) * (BN / TN);
    constexpr int RT = BM / TM;  /* thread rows */
    constexpr int CT = BN / TN;  /* thread cols */
    static_assert(NT % BM == 0 && NT % BK == 0, "tile/thread mapping");

    const int mt = tab[0], kt = tab[1], nt = tab[2], R = tab[3];
    const int* u_off = tab + FMM_ALG_HDR;
    const int* v_off = u_off + (R + 1);
    const int* w_off = v_off + (R + 1);
    const int* ents = w_off + (R + 1);          /* (part, coef) pairs */
    const int* u_ent = ents;
    const int* v_ent = ents + 2 * u_off[R];
    const int* w_ent = v_ent + 2 * v_off[R];

    const int64_t me = (m + mt - 1) / mt, ne = (n + nt - 1) / nt, ke = (k + kt - 1) / kt;
    const int64_t i0 = (int64_t)ti * BM, j0 = (int64_t)tj * BN;
    const int tid = threadIdx.x;
    const int tr = tid % RT, tc = tid / RT;
    /* With pre-formed operands (Sp/Tp: S_r, T_r of the products r_begin..,
     * me x ke and ke x ne column-major) every product has one term of
     * coefficient 1, read with those strides; its values are exactly what the
     * fused pack forms. */
    if (Sp) { lda = me; ldb = ke; }
    (void)R;

    for (int r = r_begin; r < r_end; ++r) {
        const int wb = w_off[r], we = w_off[r + 1];
        if (wb == we) continue;
        int ue_n, ve_n;
        __syncthreads();  /* previous product finished with ue/ve */
        if (Sp) {
            ue_n = ve_n = 1;
            if (tid == 0) {
                ue[0] = Entry{Sp + (int64_t)(r - r_begin) * me * ke, 1.0, (int)me, (int)ke, 0, 0};
                ve[0] = Entry{Tp + (int64_t)(r - r_begin) * ke * ne, 1.0, (int)ke, (int)ne, 0, 0};
            }
        } else {
            const int ub = u_off[r], vb = v_off[r];
            ue_n = u_off[r + 1] - ub;
            ve_n = v_off[r + 1] - vb;
            stage_entries(u_ent, ub, ub + ue_n, kt, mt, A, lda, m, k, ue);
            stage_entries(v_ent, vb, vb + ve_n, nt, kt, B, ldb, k, n, ve);
        }
        __syncthreads();

        /* MMA engine: 8 warps in a WGM x (8 / WGM) grid, each an (MB*8) x (NB*8) block of fragments */
        constexpr int WGM = BM >= 64 ? BM / 32 : 4;
        constexpr int WM = BM / WGM, WN = BN / (8 / WGM);
        constexpr int MB = MMA ? WM / 8 : 1, NB = MMA ? WN / 8 : 1;
        static_assert(!MMA || (NT == 256 && WM % 8 == 0 && WN % 8 == 0 && BK % 4 == 0), "MMA warp tiling");
        const int lane = tid % 32, wid = tid / 32, gid = lane / 4, tig = lane % 4;
        const int wm = wid % WGM, wn = wid / WGM;
        double acc[MMA ? 1 : TM][MMA ? 1 : TN];
        double facc[MB][NB][2];
        if (MMA) {
#pragma unroll
            for (int a = 0; a < MB; ++a)
#pragma unroll
                for (int b = 0; b < NB; ++b) facc[a][b][0] = facc[a][b][1] = 0.0;
        } else {
#pragma unroll
            for (int a = 0; a < (MMA ? 1 : TM); ++a)
#pragma unroll
                for (int b = 0; b < (MMA ? 1 : TN); ++b) acc[a][b] = 0.0;
        }

        for (int64_t k0 = 0; k0 < ke; k0 += BK) {
            /* fused pack of the A-side combination: BM x BK. Each term's
             * loads for all of this thread's elements go out together; the
             * first term's coefficient (uniform over the CTA) is applied once
             * after them. */
            {
                constexpr int NA = BM * BK / NT;
                const int li = tid % BM;
                const int64_t gi = i0 + li;
                double s[NA];
#pragma unroll
                for (int t = 0; t < NA; ++t) s[t] = 0.0;
                if (ue_n > 0) {
                    const Entry& x0 = ue[0];
#pragma unroll
                    for (int t = 0; t < NA; ++t) {
                        const int64_t gp = k0 + tid / BM + t * (NT / BM);
                        s[t] = (gi < x0.rows && gp < x0.cols) ? x0.base[gi + gp * lda] : 0.0;
                    }
                    scale_first(x0, s);
                }
                for (int e = 1; e < ue_n; ++e) {
                    const Entry& x = ue[e];
#pragma unroll
                    for (int t = 0; t < NA; ++t) {
                        const int64_t gp = k0 + tid / BM + t * (NT / BM);
                        const double v = (gi < x.rows && gp < x.cols) ? x.base[gi + gp * lda] : 0.0;
                        s[t] = fma(x.coef, v, s[t]);
                    }
                }
#pragma unroll
                for (int t = 0; t < NA; ++t) As[SM::a(tid / BM + t * (NT / BM), li)] = s[t];
            }
            /* fused pack of the B-side combination: BK x BN */
            {
                constexpr int NB = BK * BN / NT;
                const int lp = tid % BK;
                const int64_t gp = k0 + lp;
                double s[NB];
#pragma unroll
                for (int t = 0; t < NB; ++t) s[t] = 0.0;
                if (ve_n > 0) {
                    const Entry& x0 = ve[0];
#pragma unroll
                    for (int t = 0; t < NB; ++t) {
                        const int64_t gj = j0 + tid / BK + t * (NT / BK);
                        s[t] = (gp < x0.rows && gj < x0.cols) ? x0.base[gp + gj * ldb] : 0.0;
                    }
                    scale_first(x0, s);
                }
                for (int e = 1; e < ve_n; ++e) {
                    const Entry& x = ve[e];
#pragma unroll
                    for (int t = 0; t < NB; ++t) {
                        const int64_t gj = j0 + tid / BK + t * (NT / BK);
                        const double v = (gp < x.rows && gj < x.cols) ? x.base[gp + gj * ldb] : 0.0;
                        s[t] = fma(x.coef, v, s[t]);
                    }
                }
#pragma unroll
                for (int t = 0; t < NB; ++t) Bs[SM::b(lp, tid / BK + t * (NT / BK))] = s[t];
            }
            __syncthreads();
            if (MMA) {
#pragma unroll 2
                for (int kk = 0; kk < BK; kk += 4) {
                    double a[MB], b[NB];
#pragma unroll
                    for (int x = 0; x < MB; ++x) a[x] = As[SM::a(kk + tig, wm * WM + x * 8 + gid)];
#pragma unroll
                    for (int y = 0; y < NB; ++y) b[y] = Bs[SM::b(kk + tig, wn * WN + y * 8 + gid)];
#pragma unroll
                    for (int x = 0; x < MB; ++x)
#pragma unroll
                        for (int y = 0; y < NB; ++y) mma_f64_8x8x4(facc[x][y], a[x], b[y]);
                }
            } else {
#pragma unroll 4
                for (int kk = 0; kk < BK; ++kk) {
                    double a[MMA ? 1 : TM], b[MMA ? 1 : TN];
#pragma unroll
                    for (int x = 0; x < (MMA ? 1 : TM); ++x) a[x] = As[SM::a(kk, tr + x * RT)];
#pragma unroll
                    for (int y = 0; y < (MMA ? 1 : TN); ++y) b[y] = Bs[SM::b(kk, tc + y * CT)];
#pragma unroll
                    for (int x = 0; x < (MMA ? 1 : TM); ++x)
#pragma unroll
                        for (int y = 0; y < (MMA ? 1 : TN); ++y) acc[x][y] = fma(a[x], b[y], acc[x][y]);
                }
            }
            __syncthreads();
        }

        /* multi-C epilogue */
        for (int e = wb; e < we; ++e) {
            const int part = w_ent[2 * e];
            const double lam = alpha * (double)w_ent[2 * e + 1];
            int64_t ro, rl, co, cl;
            fmm_part_geom(m, mt, part / nt, &ro, &rl);
            fmm_part_geom(n, nt, part % nt, &co, &cl);
            double* cb = C + ro + co * ldc;
            if (MMA) {
#pragma unroll
                for (int y = 0; y < NB; ++y)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int64_t gj = j0 + wn * WN + y * 8 + 2 * tig + h;
                        if (gj >= cl) continue;
#pragma unroll
                        for (int x = 0; x < MB; ++x) {
                            const int64_t gi = i0 + wm * WM + x * 8 + gid;
                            if (gi < rl) {
                                double* p = cb + gi + gj * ldc;
                                *p = fma(lam, facc[x][y][h], *p);
                            }
                        }
                    }
            } else {
#pragma unroll
                for (int y = 0; y < (MMA ? 1 : TN); ++y) {
                    const int64_t gj = j0 + tc + y * CT;
                    if (gj >= cl) continue;
#pragma unroll
                    for (int x = 0; x < (MMA ? 1 : TM); ++x) {
                        const int64_t gi = i0 + tr + x * RT;
                        if (gi < rl) {
                            double* p = cb + gi + gj * ldc;
                            *p = fma(lam, acc[x][y], *p);
                        }
                    }
                }
            }
        }
    }
    (void)me; (void)ne;
}

template <int BM, int BN, int BK, int TM, int TN, bool MMA>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
fmm_f64_kernel(const int* __restrict__ tab, int64_t m, int64_t n, int64_t k,
               double alpha, const double* __restrict__ A, int64_t lda,
               const double* __restrict__ B, int64_t ldb,
               double* __restrict__ C, int64_t ldc, int tiles_m, int r_begin, int r_end,
               const double* __restrict__ Sp, const double* __restrict__ Tp)
{
    using SM = F64Smem<BM, BN, BK, MMA>;
    __shared__ double As[SM::A_ELEMS];
    __shared__ double Bs[SM::B_ELEMS];
    __shared__ Entry ue[kMaxEntries];
    __shared__ Entry ve[kMaxEntries];
    f64_tile<BM, BN, BK, TM, TN, MMA>(tab, m, n, k, alpha, A, lda, B, ldb, C, ldc, (int)(blockIdx.x % tiles_m),
                                      (int)(blockIdx.x / tiles_m), As, Bs, ue, ve, r_begin, r_end, Sp, Tp);
}

/* ------------------------------------- pipelined single-term tiles ---- */

using sm103::cp_async8;
using sm103::cp_async_commit;
using sm103::cp_async_wait;

/* Tile geometry of the pipelined kernels: BM x BN outputs per CTA, TM x TN per
 * thread, k steps of kPipeBk in a ring of kPipeStages shared-memory stages
 * (A as [k][m]; B as [k][n] with an odd pitch, as its copies run along k). */
constexpr int kPipeBk = 16, kPipeStages = 4;
template <int BM, int BN, int TM, int TN>
struct PipeTile {
    static constexpr int RT = BM / TM, CT = BN / TN, NT = RT * CT;
    static constexpr int PB = BN + 1;
    static constexpr int STAGE = kPipeBk * (BM + PB);            /* doubles */
    static constexpr size_t SMEM = sizeof(double) * STAGE * kPipeStages;
    static_assert(NT % BM == 0 && NT % kPipeBk == 0, "tile/thread mapping");

    /* the stage's copies: rows [i0, i0 + BM) x k [k0, k0 + kPipeBk) of A and
     * the same k x columns [j0, j0 + BN) of B, zero outside rows/cols/kend */
    __device__ static __forceinline__ void issue(double* st, const double* __restrict__ A, int64_t lda, int64_t rows,
                                                 const double* __restrict__ B, int64_t ldb, int64_t cols, int64_t i0,
                                                 int64_t j0, int64_t k0, int64_t kend)
    {
        const int tid = threadIdx.x;
        {
            const int li = tid % BM, lk = tid / BM;
            const int64_t gi = i0 + li;
            const bool ok = gi < rows;
            const double* p = A + (ok ? gi : 0) + k0 * lda;
            double* d = st + li;
#pragma unroll
            for (int t = 0; t < kPipeBk * BM / NT; ++t) {
                const int kk = lk + t * (NT / BM);
                const bool in = ok && k0 + kk < kend;
                cp_async8(d + kk * BM, in ? p + kk * lda : A, in);
            }
        }
        {
            const int kk = tid % kPipeBk, lj = tid / kPipeBk;
            const bool ok = k0 + kk < kend;
            const double* p = B + (ok ? k0 + kk : 0);
            double* d = st + kPipeBk * BM + kk * PB;
#pragma unroll
            for (int t = 0; t < kPipeBk * BN / NT; ++t) {
                const int jj = lj + t * (NT / kPipeBk);
                const bool in = ok && j0 + jj < cols;
                cp_async8(d + jj, in ? p + (j0 + jj) * ldb : B, in);
            }
        }
    }

    /* acc += the stage's kn rows, k in increasing order */
    __device__ static __forceinline__ void multiply(const double* st, int kn, double (&acc)[TM][TN])
    {
        const int tr = threadIdx.x % RT, tc = threadIdx.x / RT;
        const double* as = st + tr;
        const double* bs = st + kPipeBk * BM + tc;
#pragma unroll 4
        for (int kk = 0; kk < kn; ++kk) {
            double a[TM], b[TN];
#pragma unroll
            for (int x = 0; x < TM; ++x) a[x] = as[kk * BM + x * RT];
#pragma unroll
            for (int y = 0; y < TN; ++y) b[y] = bs[kk * PB + y * CT];
#pragma unroll
            for (int x = 0; x < TM; ++x)
#pragma unroll
                for (int y = 0; y < TN; ++y) acc[x][y] = fma(a[x], b[y], acc[x][y]);
        }
    }
};

/* The FP64 FMM GEMM over single-term operands (the classical GEMM, or the
 * pre-formed S_r, T_r of the products r_begin..): one CTA per output tile
 * position runs every product over it, as fmm_f64_kernel does and in the same
 * order (the same bits), with the operand copies of the next steps, across
 * products too, in flight under the DFMAs. Bound by the FP64 pipe, 2 FMA per
 * clock and SM, which eight warps keep busy; the CTAs are small so that the
 * SMs' shares of the tiles differ little. */
template <int BM, int BN, int TM, int TN, int MINB>
__global__ void __launch_bounds__(PipeTile<BM, BN, TM, TN>::NT, MINB)
fmm_f64_pipe_kernel(const int* __restrict__ tab, int64_t m, int64_t n, int64_t k, double alpha,
                    const double* __restrict__ A, int64_t lda, const double* __restrict__ B, int64_t ldb,
                    double* __restrict__ C, int64_t ldc, int tiles_m, int r_begin, int r_end,
                    const double* __restrict__ Sp, const double* __restrict__ Tp)
{
    using PT = PipeTile<BM, BN, TM, TN>;
    extern __shared__ double f64_stages[];
    const int mt = tab[0], kt = tab[1], nt = tab[2], R = tab[3];
    const int* u_off = tab + FMM_ALG_HDR;
    const int* v_off = u_off + (R + 1);
    const int* w_off = v_off + (R + 1);
    const int* w_ent = w_off + (R + 1) + 2 * u_off[R] + 2 * v_off[R];
    const int64_t me = (m + mt - 1) / mt, ne = (n + nt - 1) / nt, ke = (k + kt - 1) / kt;
    const int64_t i0 = (int64_t)(blockIdx.x % (unsigned)tiles_m) * BM, j0 = (int64_t)(blockIdx.x / (unsigned)tiles_m) * BN;
    const int tr = threadIdx.x % PT::RT, tc = threadIdx.x / PT::RT;
    if (Sp) {
        A = Sp;
        lda = me;
        B = Tp;
        ldb = ke;
    }
    const int64_t sa = Sp ? me * ke : 0, sb = Sp ? ke * ne : 0;   /* operands of the next product */
    const int64_t nk = (ke + kPipeBk - 1) / kPipeBk;
    int lr = r_begin;      /* the next step to copy: product lr, k from lk */
    int64_t lk = 0;
    const double *la = A, *lb = B;
    int ls = 0;            /* its stage */
    auto copy_next = [&]() {
        if (lr < r_end) {
            PT::issue(f64_stages + ls * PT::STAGE, la, lda, me, lb, ldb, ne, i0, j0, lk, ke);
            lk += kPipeBk;
            if (lk >= ke) {
                lk = 0;
                ++lr;
                la += sa;
                lb += sb;
            }
            ls = ls + 1 == kPipeStages ? 0 : ls + 1;
        }
        cp_async_commit();
    };
#pragma unroll
    for (int x = 0; x < kPipeStages - 1; ++x) copy_next();
    int cs = 0;            /* the stage to multiply */
    for (int r = r_begin; r < r_end; ++r) {
        double acc[TM][TN];
#pragma unroll
        for (int x = 0; x < TM; ++x)
#pragma unroll
            for (int y = 0; y < TN; ++y) acc[x][y] = 0.0;
        for (int64_t q = 0; q < nk; ++q) {
            cp_async_wait<kPipeStages - 2>();
            __syncthreads();   /* the step's copies are in, and the stage copied to next is read out */
            copy_next();
            const int64_t left = ke - q * kPipeBk;
            if (left >= kPipeBk)
                PT::multiply(f64_stages + cs * PT::STAGE, kPipeBk, acc);
            else
                PT::multiply(f64_stages + cs * PT::STAGE, (int)left, acc);
            cs = cs + 1 == kPipeStages ? 0 : cs + 1;
        }
        /* multi-C epilogue */
        for (int e = w_off[r]; e < w_off[r + 1]; ++e) {
            const int part = w_ent[2 * e];
            const double lam = alpha * (double)w_ent[2 * e + 1];
            int64_t ro, rl, co, cl;
            fmm_part_geom(m, mt, part / nt, &ro, &rl);
            fmm_part_geom(n, nt, part % nt, &co, &cl);
            double* cb = C + (ro + i0 + tr) + (co + j0 + tc) * ldc;
            const int64_t il = rl - i0 - tr, jl = cl - j0 - tc;   /* rows and columns left from this thread's first */
            double c[TM][TN];
#pragma unroll
            for (int y = 0; y < TN; ++y)
#pragma unroll
                for (int x = 0; x < TM; ++x)
                    if (x * PT::RT < il && y * PT::CT < jl) c[x][y] = cb[x * PT::RT + y * PT::CT * ldc];
#pragma unroll
            for (int y = 0; y < TN; ++y)
#pragma unroll
                for (int x = 0; x < TM; ++x)
                    if (x * PT::RT < il && y * PT::CT < jl)
                        cb[x * PT::RT + y * PT::CT * ldc] = fma(lam, acc[x][y], c[x][y]);
        }
    }
}

/* --------------------------------------------- small FMM problems ---- */

/* A whole small FMM GEMM in one launch: a CTA owns an 8 x 8 tile position, its
 * groups of 64 threads (one element each) take the products in turn, packs
 * fused in with the terms' loads one k step ahead, and leave each M_r in shared
 * memory; then every C sub-block's element gets beta*C and the products in
 * increasing order. The values and orders are the general path's (the same
 * bits). Bound by latency: a product's k sum is one chain of dependent DFMAs
 * per element (about 120 clocks each), so the products run side by side, and
 * the general path's two packing launches, its C scaling and its temporary
 * cost more than the whole problem. 222 x1 at 97 x 61 x 45: 28.7 us general. */
constexpr int kSmallTile = 8, kSmallBk = 16, kSmallGroup = kSmallTile * kSmallTile, kSmallGroups = 8;
constexpr int kSmallMaxR = 64;
constexpr int kSmallA = kSmallBk * kSmallTile, kSmallB = kSmallBk * (kSmallTile + 1);   /* one operand tile, doubles */
constexpr int kSmallTerms = 4;   /* terms in flight together */

/* shared memory: operand tiles (two per group), M_r, entries */
size_t small_smem(int R, int nu, int nv)
{
    const int G = std::min(R, kSmallGroups);
    return sizeof(double) * ((size_t)2 * G * (kSmallA + kSmallB) + (size_t)R * kSmallGroup) +
           sizeof(Entry) * (size_t)(nu + nv);
}

/* this thread's two elements of the terms [x0, x0 + kSmallTerms) of a
 * combination at (i, j) and (i + di, j + dj) of its sub-blocks */
struct SmallTerms {
    double v[kSmallTerms][2];

    __device__ __forceinline__ void load(const Entry* e, int n, int64_t i, int64_t j, int64_t di, int64_t dj, int64_t ld)
    {
#pragma unroll
        for (int x = 0; x < kSmallTerms; ++x)
            if (x < n) {
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    const int64_t a = i + t * di, b = j + t * dj;
                    v[x][t] = a < e[x].rows && b < e[x].cols ? e[x].base[a + b * ld] : 0.0;
                }
            }
    }
    /* s (+)= the terms, in order; the first one by its kind */
    __device__ __forceinline__ void sum(const Entry* e, int n, bool first, double (&s)[2]) const
    {
#pragma unroll
        for (int x = 0; x < kSmallTerms; ++x)
            if (x < n) {
                if (x == 0 && first) {
                    s[0] = v[0][0];
                    s[1] = v[0][1];
                    scale_first(e[0], s);
                } else {
                    s[0] = fma(e[x].coef, v[x][0], s[0]);
                    s[1] = fma(e[x].coef, v[x][1], s[1]);
                }
            }
    }
    /* the whole combination, its first terms already loaded */
    __device__ __forceinline__ void combine(const Entry* e, int n, int64_t i, int64_t j, int64_t di, int64_t dj,
                                            int64_t ld, double (&s)[2])
    {
        s[0] = s[1] = 0.0;
        sum(e, n, true, s);
        for (int x = kSmallTerms; x < n; x += kSmallTerms) {
            load(e + x, n - x, i, j, di, dj, ld);
            sum(e + x, n - x, false, s);
        }
    }
};

__global__ void __launch_bounds__(kSmallGroup * kSmallGroups)
fmm_f64_small_kernel(const int* __restrict__ tab, int64_t m, int64_t n, int64_t k, double alpha,
                     const double* __restrict__ A, int64_t lda, const double* __restrict__ B, int64_t ldb, double beta,
                     double* __restrict__ C, int64_t ldc, int tiles_m)
{
    extern __shared__ double f64_stages[];
    const int mt = tab[0], kt = tab[1], nt = tab[2], R = tab[3];
    const int* u_off = tab + FMM_ALG_HDR;
    const int* v_off = u_off + (R + 1);
    const int* w_off = v_off + (R + 1);
    const int* u_ent = w_off + (R + 1);
    const int nu = u_off[R], nv = v_off[R], nw = w_off[R];
    const int* v_ent = u_ent + 2 * nu;
    const int* wp_off = v_ent + 2 * nv + 2 * nw;
    const int* wp_ent = wp_off + (mt * nt + 1);
    const int G = (int)blockDim.x / kSmallGroup, g = (int)threadIdx.x / kSmallGroup, tid = (int)threadIdx.x % kSmallGroup;
    double* tiles = f64_stages + (size_t)g * 2 * (kSmallA + kSmallB);                  /* [2][A, B] */
    double* M = f64_stages + (size_t)G * 2 * (kSmallA + kSmallB);                      /* [R][64] */
    Entry* ue = (Entry*)(M + (size_t)R * kSmallGroup);
    Entry* ve = ue + nu;
    stage_entries(u_ent, 0, nu, kt, mt, A, lda, m, k, ue);
    stage_entries(v_ent, 0, nv, nt, kt, B, ldb, k, n, ve);
    __syncthreads();
    const int64_t ke = (k + kt - 1) / kt;
    const int64_t i0 = (int64_t)(blockIdx.x % (unsigned)tiles_m) * kSmallTile;
    const int64_t j0 = (int64_t)(blockIdx.x / (unsigned)tiles_m) * kSmallTile;
    const int tr = tid % kSmallTile, tc = tid / kSmallTile;   /* the thread's element, and its A copies (row, k) */
    const int bk = tid % kSmallBk, bj = tid / kSmallBk;       /* its B copies: k, columns bj and bj + 4 */
    SmallTerms ta, tb;
    auto fetch = [&](int r, int64_t k0) {
        ta.load(ue + u_off[r], u_off[r + 1] - u_off[r], i0 + tr, k0 + tc, 0, 8, lda);
        tb.load(ve + v_off[r], v_off[r + 1] - v_off[r], k0 + bk, j0 + bj, 0, 4, ldb);
    };
    auto put = [&](int r, int64_t k0, double* t) {
        double s[2];
        ta.combine(ue + u_off[r], u_off[r + 1] - u_off[r], i0 + tr, k0 + tc, 0, 8, lda, s);
        t[tc * kSmallTile + tr] = s[0];
        t[(tc + 8) * kSmallTile + tr] = s[1];
        tb.combine(ve + v_off[r], v_off[r + 1] - v_off[r], k0 + bk, j0 + bj, 0, 4, ldb, s);
        t[kSmallA + bk * (kSmallTile + 1) + bj] = s[0];
        t[kSmallA + bk * (kSmallTile + 1) + bj + 4] = s[1];
    };
    auto group_sync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(g + 1) : "memory"); };
    int buf = 0;
    if (g < R) {
        fetch(g, 0);
        put(g, 0, tiles);
    }
    for (int r = g; r < R; r += G) {
        double acc = 0.0;
        for (int64_t k0 = 0; k0 < ke; k0 += kSmallBk) {
            group_sync();   /* the step's tile is in, the other one read out */
            const bool last = k0 + kSmallBk >= ke;
            const int rn = last ? r + G : r;
            const int64_t kn = last ? 0 : k0 + kSmallBk;
            if (rn < R) fetch(rn, kn);
            const double* t = tiles + buf * (kSmallA + kSmallB);
            const int kc = (int)(ke - k0 < kSmallBk ? ke - k0 : kSmallBk);
#pragma unroll 4
            for (int kk = 0; kk < kc; ++kk)
                acc = fma(t[kk * kSmallTile + tr], t[kSmallA + kk * (kSmallTile + 1) + tc], acc);
            buf ^= 1;
            if (rn < R) put(rn, kn, tiles + buf * (kSmallA + kSmallB));
        }
        M[r * kSmallGroup + tid] = acc;
    }
    __syncthreads();
    /* the C sub-blocks, shared out over the groups */
    for (int p = g; p < mt * nt; p += G) {
        int64_t ro, rl, co, cl;
        fmm_part_geom(m, mt, p / nt, &ro, &rl);
        fmm_part_geom(n, nt, p % nt, &co, &cl);
        if (i0 + tr >= rl || j0 + tc >= cl) continue;
        double* cp = C + ro + i0 + tr + (co + j0 + tc) * ldc;
        double c = beta == 1.0 ? *cp : (beta == 0.0 ? 0.0 : beta * *cp);
        for (int e = wp_off[p]; e < wp_off[p + 1]; ++e)
            c = fma(alpha * (double)wp_ent[2 * e + 1], M[wp_ent[2 * e] * kSmallGroup + tid], c);
        *cp = c;
    }
}

/* ------------------------------------------------------------ batched -- */

/* One problem of a batched FP64 launch; problems are laid out in the order
 * their work items are handed out (item_begin increasing). */
struct F64Prob {
    const int* tab;
    int64_t m, n, k;
    double alpha, beta;
    const double* A;
    int64_t lda;
    const double* B;
    int64_t ldb;
    double* C;
    int64_t ldc;
    int64_t item_begin;   /* first (tile position) item of this problem */
    int tiles_m, tile;    /* tile: items are tile x tile positions (64, 32 or 16) */
};

constexpr int kF64BatchThreads = 256;
constexpr int kF64TableChunk = 256;   /* problems per table-writer launch (parameter space) */

struct F64TableChunk {
    F64Prob* dst;
    int count;
    F64Prob p[kF64TableChunk];
};

/* copies a chunk of the problem table (passed by value, so a captured graph
 * holds it) into device memory */
__global__ void f64_table_write(const __grid_constant__ F64TableChunk c)
{
    for (int i = threadIdx.x; i < c.count; i += blockDim.x) c.dst[i] = c.p[i];
}

/* One item: beta applied to the C elements its threads own in every
 * sub-block of the tile position, then the tile as the single-problem kernels
 * run it (every tile shape accumulates in the same order: the same bits). */
template <int B, int T, bool MMA>
__device__ __forceinline__ void f64_batch_item(const F64Prob& P, int ti, int tj, double* As, double* Bs, Entry* ue,
                                               Entry* ve)
{
    constexpr int RT = B / T;
    const int tr = threadIdx.x % RT, tc = threadIdx.x / RT;
    const int mt = P.tab[0], nt = P.tab[2];
    if (P.beta != 1.0) {
        for (int part = 0; part < mt * nt; ++part) {
            int64_t ro, rl, co, cl;
            fmm_part_geom(P.m, mt, part / nt, &ro, &rl);
            fmm_part_geom(P.n, nt, part % nt, &co, &cl);
            for (int y = 0; y < T; ++y) {
                const int64_t gj = (int64_t)tj * B + tc + y * RT;
                if (gj >= cl) continue;
                for (int x = 0; x < T; ++x) {
                    const int64_t gi = (int64_t)ti * B + tr + x * RT;
                    if (gi < rl) {
                        double* q = P.C + ro + gi + (co + gj) * P.ldc;
                        *q = P.beta == 0.0 ? 0.0 : P.beta * *q;
                    }
                }
            }
        }
    }
    if (P.k == 0 || P.alpha == 0.0) return;
    f64_tile<B, B, 32, T, T, MMA>(P.tab, P.m, P.n, P.k, P.alpha, P.A, P.lda, P.B, P.ldb, P.C, P.ldc, ti, tj, As, Bs, ue,
                                  ve, 0, P.tab[3], nullptr, nullptr);
}

/* Batched FP64 FMM GEMM: one persistent launch over all (problem, tile
 * position) items of a batch. A CTA takes the next item from an atomic
 * counter (problems sorted by per-item work, largest first, so the long
 * items go out first). The FP64 MMA engine has no 16 x 16 tile (its eight
 * warps need 8 x 8 fragments). */
template <bool MMA>
__global__ void __launch_bounds__(kF64BatchThreads)
fmm_f64_batch_kernel(const F64Prob* __restrict__ probs, int nprob, int64_t nitems,
                     unsigned long long* __restrict__ counter)
{
    using SM = F64Smem<64, 64, 32, MMA>;
    __shared__ double As[SM::A_ELEMS];
    __shared__ double Bs[SM::B_ELEMS];
    __shared__ Entry ue[kMaxEntries];
    __shared__ Entry ve[kMaxEntries];
    __shared__ long long next;
    for (;;) {
        __syncthreads();   /* the previous item is done with next, ue and ve */
        if (threadIdx.x == 0) next = (long long)atomicAdd(counter, 1ull);
        __syncthreads();
        const int64_t b = next;
        if (b >= nitems) break;
        int lo = 0, hi = nprob - 1;        /* last problem with item_begin <= b */
        while (lo < hi) {
            const int mid = (lo + hi + 1) / 2;
            if (probs[mid].item_begin <= b) lo = mid; else hi = mid - 1;
        }
        const F64Prob P = probs[lo];
        const int64_t local = b - P.item_begin;
        const int ti = (int)(local % P.tiles_m), tj = (int)(local / P.tiles_m);
        if (P.tile == 64)
            f64_batch_item<64, 4, MMA>(P, ti, tj, As, Bs, ue, ve);
        else if (MMA || P.tile == 32)
            f64_batch_item<32, 2, MMA>(P, ti, tj, As, Bs, ue, ve);
        else
            f64_batch_item<16, 1, false>(P, ti, tj, As, Bs, ue, ve);
    }
}

/* Pre-formed operand combinations for the products r0 .. r0+np-1:
 * S[q][i + p*me] = sum_e U[e,r] A_e[i,p] (A side) or T[q][p + j*ke] =
 * sum_e V[e,r] B_e[p,j] (B side), zero past a smaller sub-block, summed
 * exactly as the fused pack does (the first term's coefficient, then FMAs in
 * entry order), so the GEMM over them gives the fused kernel's bits. One
 * thread per element down a column (coalesced loads and stores); the product
 * index runs fastest in the block order so the products at one position read
 * their shared sub-blocks through L2 once. */
template <bool A_SIDE>
__global__ void __launch_bounds__(256)
f64_combine_kernel(const int* __restrict__ tab, int r0, int np, const double* __restrict__ X, int64_t ldx,
                   int64_t m, int64_t n, int64_t k, double* __restrict__ out)
{
    __shared__ Entry ent[kMaxEntries];
    const int mt = tab[0], kt = tab[1], nt = tab[2], R = tab[3];
    const int* u_off = tab + FMM_ALG_HDR;
    const int* v_off = u_off + (R + 1);
    const int* w_off = v_off + (R + 1);
    const int* u_ent = w_off + (R + 1);
    const int* v_ent = u_ent + 2 * u_off[R];
    const int64_t me = (m + mt - 1) / mt, ne = (n + nt - 1) / nt, ke = (k + kt - 1) / kt;
    const int64_t rows = A_SIDE ? me : ke, cols = A_SIDE ? ke : ne;
    const int q = (int)(blockIdx.x % (unsigned)np), r = r0 + q;
    const int64_t i = (int64_t)(blockIdx.x / (unsigned)np) * blockDim.x + threadIdx.x;
    int ne_;
    if (A_SIDE) {
        ne_ = u_off[r + 1] - u_off[r];
        stage_entries(u_ent, u_off[r], u_off[r + 1], kt, mt, X, ldx, m, k, ent);
    } else {
        ne_ = v_off[r + 1] - v_off[r];
        stage_entries(v_ent, v_off[r], v_off[r + 1], nt, kt, X, ldx, k, n, ent);
    }
    __syncthreads();
    if (i >= rows) return;
    double* o = out + (int64_t)q * rows * cols;
    for (int64_t c = blockIdx.y; c < cols; c += gridDim.y) {
        double sv[1] = {0.0};
        if (ne_ > 0) {
            const Entry& x0 = ent[0];
            sv[0] = (i < x0.rows && c < x0.cols) ? x0.base[i + c * ldx] : 0.0;
            scale_first(x0, sv);
        }
        for (int e = 1; e < ne_; ++e) {
            const Entry& x = ent[e];
            const double v = (i < x.rows && c < x.cols) ? x.base[i + c * ldx] : 0.0;
            sv[0] = fma(x.coef, v, sv[0]);
        }
        o[i + c * rows] = sv[0];
    }
}

__global__ void scale_c_kernel(int64_t m, int64_t n, double beta, double* C, int64_t ldc)
{
    const int64_t total = m * n;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = idx % m, j = idx / m;
        double* p = C + i + j * ldc;
        *p = beta == 0.0 ? 0.0 : beta * *p;
    }
}

/* ------------------------------------------- small/skinny classical ---- */

/* The classical FP64 GEMM of a small output (at most 128 tiles of 32 x 32)
 * with a long k (the BLIS "sup" shapes, blis/kernels/haswell/3/sup): the
 * regular kernel would run one CTA per tile down the whole of k on a few
 * SMs. Here a cluster of ks CTAs (one per k chunk of kc elements) computes
 * each tile: every CTA accumulates its chunk in k order (the pipelined tile),
 * leaves its partial tile in shared memory, and after a cluster
 * barrier the first CTA, one element per thread, sums the ks partials
 * through distributed shared memory, always in chunk order
 * (((p_0 + p_1) + p_2) + ...), and applies C := fma(alpha, sum, C). The
 * result depends only on (m, n, k): the batched call runs these problems
 * through the same kernel. */
template <int BM, int BN, int TM, int TN, int MINB>
__global__ void __launch_bounds__(PipeTile<BM, BN, TM, TN>::NT, MINB)
fmm_f64_sup_kernel(int64_t m, int64_t n, int64_t k, double alpha, const double* __restrict__ A, int64_t lda,
                   const double* __restrict__ B, int64_t ldb, double* __restrict__ C, int64_t ldc, int tiles_m,
                   int ks, int64_t kc)
{
    using PT = PipeTile<BM, BN, TM, TN>;
    extern __shared__ double f64_stages[];
    __shared__ double Ps[BM * BN];                /* this CTA's partial tile, element i + BM j */
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();        /* the k chunk */
    const int tile = (int)(blockIdx.x / (unsigned)ks);
    const int64_t i0 = (int64_t)(tile % tiles_m) * BM, j0 = (int64_t)(tile / tiles_m) * BN;
    const int64_t kb = (int64_t)rank * kc, kend = kb + kc < k ? kb + kc : k;
    const int tid = threadIdx.x, tr = tid % PT::RT, tc = tid / PT::RT;
    double acc[TM][TN];
#pragma unroll
    for (int x = 0; x < TM; ++x)
#pragma unroll
        for (int y = 0; y < TN; ++y) acc[x][y] = 0.0;
    int64_t lk = kb;
    int ls = 0, cs = 0;
    auto copy_next = [&]() {
        if (lk < kend) {
            PT::issue(f64_stages + ls * PT::STAGE, A, lda, m, B, ldb, n, i0, j0, lk, kend);
            lk += kPipeBk;
            ls = ls + 1 == kPipeStages ? 0 : ls + 1;
        }
        cp_async_commit();
    };
#pragma unroll
    for (int x = 0; x < kPipeStages - 1; ++x) copy_next();
    for (int64_t k0 = kb; k0 < kend; k0 += kPipeBk) {
        cp_async_wait<kPipeStages - 2>();
        __syncthreads();   /* the step's copies are in, and the stage copied to next is read out */
        copy_next();
        PT::multiply(f64_stages + cs * PT::STAGE, (int)(kend - k0 < kPipeBk ? kend - k0 : kPipeBk), acc);
        cs = cs + 1 == kPipeStages ? 0 : cs + 1;
    }
#pragma unroll
    for (int x = 0; x < TM; ++x)
#pragma unroll
        for (int y = 0; y < TN; ++y) Ps[(tr + x * PT::RT) + BM * (tc + y * PT::CT)] = acc[x][y];
    cl.sync();   /* every partial tile of the cluster is in place */
    static_assert(BM * BN == PT::NT, "one element per thread");
    if (rank == 0) {
        double s = Ps[tid];
        for (int q = 1; q < ks; ++q) s = s + *cl.map_shared_rank(Ps + tid, q);
        const int64_t gi = i0 + tid % BM, gj = j0 + tid / BM;
        if (gi < m && gj < n) {
            double* p = C + gi + gj * ldc;
            *p = fma(alpha, s, *p);
        }
    }
    cl.sync();   /* no CTA leaves while another still reads its partial */
}

template <int BM, int BN, int TM, int TN, int MINB>
int sup_launch_t(int64_t m, int64_t n, int64_t k, double alpha, const double* A, int64_t lda, const double* B,
                 int64_t ldb, double* C, int64_t ldc, int ks, cudaStream_t st)
{
    using PT = PipeTile<BM, BN, TM, TN>;
    const int64_t tm = (m + BM - 1) / BM, tn = (n + BN - 1) / BN;
    const int64_t kc = fmm_f64_sup_chunk(k, ks);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tm * tn * ks));
    cfg.blockDim = dim3(PT::NT);
    cfg.dynamicSmemBytes = PT::SMEM;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)ks;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, fmm_f64_sup_kernel<BM, BN, TM, TN, MINB>, m, n, k, alpha, A, lda, B,
                                             ldb, C, ldc, (int)tm, ks, kc);
    fmm_count_launch(1);
    return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? FMM_OK : FMM_ERR_CUDA;
}

/* Tile of the cluster path: 16 x 8 or 8 x 8, whichever loads the busiest SM
 * less (ks CTAs per tile), the smaller one at the lower measured efficiency.
 * The bits do not depend on it. Measured (us, 16 x 8 / 8 x 8; 32 x 32 before):
 * 128 x 128 x 16384 536 / 522 (1047), 250 x 120 x 12000 676 / 753,
 * 257 x 129 x 2048 146 / 166 (218), 33 x 700 x 3000 197 / 162 (316),
 * 8 x 320 x 16384 201 / 131. */
int sup_launch(int64_t m, int64_t n, int64_t k, double alpha, const double* A, int64_t lda, const double* B,
               int64_t ldb, double* C, int64_t ldc, int ks, cudaStream_t st)
{
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    auto load = [&](int bm, int bn, double eff) {
        const int64_t ctas = ((m + bm - 1) / bm) * ((n + bn - 1) / bn) * ks;
        return (double)((ctas + sms - 1) / sms) * (bm * bn) / eff;
    };
    if (load(8, 8, 0.85) < load(16, 8, 0.95))
        return sup_launch_t<8, 8, 1, 1, 8>(m, n, k, alpha, A, lda, B, ldb, C, ldc, ks, st);
    return sup_launch_t<16, 8, 1, 1, 6>(m, n, k, alpha, A, lda, B, ldb, C, ldc, ks, st);
}

template <int BM, int BN, int BK, int TM, int TN, bool MMA>
int launch_cfg(const AlgView& alg, int64_t m, int64_t n, int64_t k, double alpha,
               const double* A, int64_t lda, const double* B, int64_t ldb, double* C,
               int64_t ldc, int r_begin, int r_end, const double* Sp, const double* Tp, cudaStream_t st)
{
    const int64_t me = (m + alg.mt - 1) / alg.mt, ne = (n + alg.nt - 1) / alg.nt;
    const int64_t tm = (me + BM - 1) / BM, tn = (ne + BN - 1) / BN;
    if (tm * tn > 0x7fffffffLL) return FMM_ERR_UNSUPPORTED;
    fmm_f64_kernel<BM, BN, BK, TM, TN, MMA><<<(unsigned)(tm * tn), (BM / TM) * (BN / TN), 0, st>>>(
        alg.tab, m, n, k, alpha, A, lda, B, ldb, C, ldc, (int)tm, r_begin, r_end, Sp, Tp);
    fmm_count_launch(1);
    return cudaGetLastError() == cudaSuccess ? FMM_OK : FMM_ERR_CUDA;
}

template <int BM, int BN, int TM, int TN, int MINB>
int launch_pipe(const AlgView& alg, int64_t m, int64_t n, int64_t k, double alpha, const double* A, int64_t lda,
                const double* B, int64_t ldb, double* C, int64_t ldc, int r_begin, int r_end, const double* Sp,
                const double* Tp, cudaStream_t st)
{
    using PT = PipeTile<BM, BN, TM, TN>;
    const int64_t me = (m + alg.mt - 1) / alg.mt, ne = (n + alg.nt - 1) / alg.nt;
    const int64_t tm = (me + BM - 1) / BM, tn = (ne + BN - 1) / BN;
    if (tm * tn > 0x7fffffffLL) return FMM_ERR_UNSUPPORTED;
    if (PT::SMEM > 48 * 1024) {
        static std::atomic<uint64_t> attr_set{0};   /* a per-device attribute of the kernel: set once per device */
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess) return FMM_ERR_CUDA;
        const uint64_t bit = dev < 64 ? 1ull << dev : 0;
        if (bit == 0 || !(attr_set.load(std::memory_order_acquire) & bit)) {
            if (cudaFuncSetAttribute(fmm_f64_pipe_kernel<BM, BN, TM, TN, MINB>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PT::SMEM) != cudaSuccess)
                return FMM_ERR_CUDA;
            attr_set.fetch_or(bit, std::memory_order_acq_rel);
        }
    }
    fmm_f64_pipe_kernel<BM, BN, TM, TN, MINB><<<(unsigned)(tm * tn), PT::NT, PT::SMEM, st>>>(
        alg.tab, m, n, k, alpha, A, lda, B, ldb, C, ldc, (int)tm, r_begin, r_end, Sp, Tp);
    fmm_count_launch(1);
    return cudaGetLastError() == cudaSuccess ? FMM_OK : FMM_ERR_CUDA;
}

/* the kernels a call runs its tiles on */
enum F64Pick {
    kPipe64, kPipe16x8, kPipe8,                       /* pipelined DFMA tiles, single-term operands */
    kFused64, kFused32,                               /* DFMA with the packs fused in */
    kMma64, kMma128x64, kMma64x128, kMma32            /* FP64 MMA engine */
};

int launch_pick(F64Pick pick, const AlgView& alg, int64_t m, int64_t n, int64_t k, double alpha, const double* A,
                int64_t lda, const double* B, int64_t ldb, double* C, int64_t ldc, int r_begin, int r_end,
                const double* Sp, const double* Tp, cudaStream_t st)
{
    auto go = [&](auto f) { return f(alg, m, n, k, alpha, A, lda, B, ldb, C, ldc, r_begin, r_end, Sp, Tp, st); };
    switch (pick) {
    case kPipe64: return go(launch_pipe<64, 64, 4, 4, 2>);
    case kPipe16x8: return go(launch_pipe<16, 8, 1, 1, 6>);
    case kPipe8: return go(launch_pipe<8, 8, 1, 1, 8>);
    case kFused64: return go(launch_cfg<64, 64, 32, 4, 4, false>);
    case kFused32: return go(launch_cfg<32, 32, 32, 2, 2, false>);
    case kMma64: return go(launch_cfg<64, 64, 32, 4, 4, true>);
    case kMma128x64: return go(launch_cfg<128, 64, 16, 8, 4, true>);
    case kMma64x128: return go(launch_cfg<64, 128, 16, 4, 8, true>);
    default: return go(launch_cfg<32, 32, 32, 2, 2, true>);
    }
}

/* the cheapest of a list of tiles, by the most loaded SM's FP64 work */
struct F64Cand {
    F64Pick pick;
    int bm, bn;
    double eff;   /* measured share of the FP64 pipe's rate when the SMs' shares are equal */
};

/* Pipelined tiles: an SM's CTAs share its FP64 pipe and a finished CTA's place
 * is taken at once, so the SM with the most tiles sets the time. Measured
 * (us, tiles 64 x 64 / 16 x 8 / 8 x 8; the kernel before: 64 or 32 wide):
 * classical 4096^3 110038 / 110443 / 109979, classical 1000 x 1200 x 900
 * 1811 / 1787 / 1779 (1876), 222 x1 2048^3 14502 / 12360 / 12578 (12895),
 * 333 x1 4097 x 3001 x 3500 81199 / 61521 / 61097 (69717), classical 512^3
 * 525 / 234 / 247 (265), 222 x1 400^3 - / 159 / 137 (463). */
constexpr F64Cand kPipeCands[] = {{kPipe64, 64, 64, 0.985}, {kPipe16x8, 16, 8, 0.97}, {kPipe8, 8, 8, 0.85}};

F64Pick pick_pipe(int64_t me, int64_t ne, int sms)
{
    F64Pick best = kPipe64;
    double least = 0.0;
    for (const F64Cand& c : kPipeCands) {
        const int64_t tiles = ((me + c.bm - 1) / c.bm) * ((ne + c.bn - 1) / c.bn);
        const double est = (double)((tiles + sms - 1) / sms) * (c.bm * c.bn) / c.eff;
        if (least == 0.0 || est < least) { least = est; best = c.pick; }
    }
    return best;
}

/* Tiles with the packs fused in (and the MMA engine's): waves of two CTAs per
 * SM, times the FMAs per tile including the pack additions (nu, nv terms per
 * operand), over the tile's efficiency. */
F64Pick pick_fused(bool mma, int64_t me, int64_t ne, double nu, double nv, int sms)
{
    static constexpr F64Cand dfma[] = {{kFused64, 64, 64, 1.0}, {kFused32, 32, 32, 0.8}};
    static constexpr F64Cand mmac[] = {{kMma64, 64, 64, 1.0}, {kMma128x64, 128, 64, 0.99}, {kMma64x128, 64, 128, 0.99},
                                       {kMma32, 32, 32, 0.8}};
    F64Pick best = kFused64;
    double least = 0.0;
    for (int x = 0; x < (mma ? 4 : 2); ++x) {
        const F64Cand& c = mma ? mmac[x] : dfma[x];
        const int64_t tiles = ((me + c.bm - 1) / c.bm) * ((ne + c.bn - 1) / c.bn);
        const double waves = (double)((tiles + 2 * (int64_t)sms - 1) / (2 * (int64_t)sms));
        const double work = (double)(c.bm * c.bn) *
                            (1.0 + (nu - 1.0) / c.bn + (nv - 1.0) / c.bm + 4.0 / c.bm);
        if (least == 0.0 || waves * work / c.eff < least) { least = waves * work / c.eff; best = c.pick; }
    }
    return best;
}

/* Stream-ordered temporaries (pre-formed operands, work units' planes) from the library's own
 * memory pool of the device, which keeps up to 256 MiB between calls: the
 * device's default pool gives everything back at each synchronization, and
 * getting it again cost a synchronous caller about 200 us per call. Given back
 * by fmm_gpu_release_host_buffers. */
constexpr uint64_t kTempPoolKeep = (uint64_t)256 << 20;
std::mutex g_pool_mu;
cudaMemPool_t g_pools[64];

}  // namespace

namespace {
/* puts the thread's stream capture mode back */
struct CaptureModeBack {
    cudaStreamCaptureMode mode;
    ~CaptureModeBack()
    {
        cudaStreamCaptureMode m = mode;
        cudaThreadExchangeStreamCaptureMode(&m);
    }
};
}  // namespace

cudaMemPool_t fmm_temp_pool()
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    std::lock_guard<std::mutex> lk(g_pool_mu);
    if (g_pools[dev] == nullptr) {
        /* a pool may be made while the calling thread captures a stream: no stream's work is part of it */
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) return nullptr;
        const CaptureModeBack back{mode};
        cudaMemPoolProps props;
        memset(&props, 0, sizeof(props));
        props.allocType = cudaMemAllocationTypePinned;
        props.handleTypes = cudaMemHandleTypeNone;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t p = nullptr;
        uint64_t keep = kTempPoolKeep;
        if (cudaMemPoolCreate(&p, &props) != cudaSuccess) return nullptr;
        if (cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
            cudaMemPoolDestroy(p);
            return nullptr;
        }
        g_pools[dev] = p;
    }
    return g_pools[dev];
}

namespace {

/* bytes of pre-formed operands a product group may hold at once */
constexpr size_t kPrepackBudget = (size_t)4 << 30;

}  // namespace

int fmm_scale_c(int64_t m, int64_t n, double beta, double* C, int64_t ldc, cudaStream_t st)
{
    if (beta == 1.0 || m == 0 || n == 0) return FMM_OK;
    int64_t total = m * n;
    int blocks = (int)std::min<int64_t>((total + 255) / 256, 152 * 16);
    scale_c_kernel<<<blocks, 256, 0, st>>>(m, n, beta, C, ldc);
    fmm_count_launch(1);
    return cudaGetLastError() == cudaSuccess ? FMM_OK : FMM_ERR_CUDA;
}

namespace {

/* Whether a problem runs as fmm_f64_small_kernel: its busiest SM's FP64 work
 * (8 x 8 tiles, the packs adding about a quarter) within 50000 clocks, about
 * where the general path's fewer DFMAs make up for its launches (256^3 222 x1
 * is just past it), and the shared memory it needs. */
bool small_fmm(const AlgView& alg, int64_t me, int64_t ne, int64_t ke, int sms, size_t* smem)
{
    if (alg.R < 2 || alg.R > kSmallMaxR || alg.htab == nullptr) return false;
    const int* u_off = alg.htab + FMM_ALG_HDR;
    const int nu = u_off[alg.R], nv = u_off[alg.R + 1 + alg.R];
    if (nu > kMaxEntries || nv > kMaxEntries) return false;
    const int64_t tiles = ((me + kSmallTile - 1) / kSmallTile) * ((ne + kSmallTile - 1) / kSmallTile);
    if (tiles > (int64_t)64 * sms) return false;
    const double clocks = (double)((tiles + sms - 1) / sms) * kSmallGroup * alg.R * (double)ke * 1.25 / 2.0;
    *smem = small_smem(alg.R, nu, nv);
    return clocks <= 50000.0 && *smem <= (size_t)100 * 1024;
}

int launch_small(const AlgView& alg, int64_t m, int64_t n, int64_t k, double alpha, const double* A, int64_t lda,
                 const double* B, int64_t ldb, double beta, double* C, int64_t ldc, size_t smem, cudaStream_t st)
{
    static std::atomic<uint64_t> attr_set{0};   /* a per-device attribute of the kernel: set once per device */
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return FMM_ERR_CUDA;
    const uint64_t bit = dev < 64 ? 1ull << dev : 0;
    if (bit == 0 || !(attr_set.load(std::memory_order_acquire) & bit)) {
        if (cudaFuncSetAttribute(fmm_f64_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024) !=
            cudaSuccess)
            return FMM_ERR_CUDA;
        attr_set.fetch_or(bit, std::memory_order_acq_rel);
    }
    const int64_t me = (m + alg.mt - 1) / alg.mt, ne = (n + alg.nt - 1) / alg.nt;
    const int64_t tm = (me + kSmallTile - 1) / kSmallTile, tn = (ne + kSmallTile - 1) / kSmallTile;
    fmm_f64_small_kernel<<<(unsigned)(tm * tn), kSmallGroup * std::min(alg.R, kSmallGroups), smem, st>>>(
        alg.tab, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, (int)tm);
    fmm_count_launch(1);
    return cudaGetLastError() == cudaSuccess ? FMM_OK : FMM_ERR_CUDA;
}

}  // namespace

void fmm_f64_release_temp()
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return;
    std::lock_guard<std::mutex> lk(g_pool_mu);
    if (g_pools[dev]) cudaMemPoolTrimTo(g_pools[dev], 0);
}

int fmm_f64_launch(const AlgView& alg, int64_t m, int64_t n, int64_t k, double alpha,
                   const double* A, int64_t lda, const double* B, int64_t ldb,
                   double beta, double* C, int64_t ldc, cudaStream_t st)
{
    if (m == 0 || n == 0 || k == 0 || alpha == 0.0) return fmm_scale_c(m, n, beta, C, ldc, st);
    if (alg.max_nnz_u > kMaxEntries || alg.max_nnz_v > kMaxEntries) return FMM_ERR_UNSUPPORTED;

    const bool mma = g_f64_engine.load(std::memory_order_relaxed) == FMM_F64_MMA;
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int64_t me = (m + alg.mt - 1) / alg.mt, ne = (n + alg.nt - 1) / alg.nt, ke = (k + alg.kt - 1) / alg.kt;
    size_t smem = 0;
    if (!mma && small_fmm(alg, me, ne, ke, sms, &smem))
        return launch_small(alg, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, smem, st);
    int rc = fmm_scale_c(m, n, beta, C, ldc, st);
    if (rc != FMM_OK) return rc;
    const bool classical = fmm_plain_classical(alg);
    if (classical) {
        const int ks = fmm_gpu_f64_sup_splits(m, n, k);
        if (ks >= 2) return sup_launch(m, n, k, alpha, A, lda, B, ldb, C, ldc, ks, st);
    }
    /* FMM algorithms form each product's operand combinations once, ahead of
     * the tiles (a stream-ordered temporary of at most kPrepackBudget per
     * product group), instead of once per tile position inside the kernel;
     * the values, and so the results, are the same either way. */
    if (alg.R > 1) {
        const F64Pick pick = mma ? pick_fused(true, me, ne, 1.0, 1.0, sms) : pick_pipe(me, ne, sms);
        const size_t per = (size_t)(me * ke + ke * ne) * sizeof(double);
        const int G = (int)std::max<size_t>(1, std::min<size_t>((size_t)alg.R, kPrepackBudget / std::max<size_t>(per, 1)));
        void* buf = nullptr;
        const cudaMemPool_t pool = fmm_temp_pool();
        if (pool != nullptr && cudaMallocFromPoolAsync(&buf, (size_t)G * per, pool, st) == cudaSuccess) {
            double* Sbuf = (double*)buf;
            double* Tbuf = Sbuf + (size_t)G * me * ke;
            for (int r0 = 0; r0 < alg.R && rc == FMM_OK; r0 += G) {
                const int np = std::min(G, alg.R - r0);
                f64_combine_kernel<true><<<dim3((unsigned)(np * ((me + 255) / 256)), (unsigned)std::min<int64_t>(ke, 65535)),
                                           256, 0, st>>>(alg.tab, r0, np, A, lda, m, n, k, Sbuf);
                f64_combine_kernel<false><<<dim3((unsigned)(np * ((ke + 255) / 256)), (unsigned)std::min<int64_t>(ne, 65535)),
                                            256, 0, st>>>(alg.tab, r0, np, B, ldb, m, n, k, Tbuf);
                fmm_count_launch(2);
                rc = launch_pick(pick, alg, m, n, k, alpha, A, lda, B, ldb, C, ldc, r0, r0 + np, Sbuf, Tbuf, st);
            }
            if (cudaFreeAsync(buf, st) != cudaSuccess && rc == FMM_OK) rc = FMM_ERR_CUDA;
            return rc;
        }
        cudaGetLastError();   /* no temporary: the combinations stay fused into the kernel */
    }
    const F64Pick pick = classical && !mma ? pick_pipe(me, ne, sms)
                                           : pick_fused(mma, me, ne, alg.avg_nnz_u, alg.avg_nnz_v, sms);
    return launch_pick(pick, alg, m, n, k, alpha, A, lda, B, ldb, C, ldc, 0, alg.R, nullptr, nullptr, st);
}

/* Workspace of a batched FP64 launch: the work counter and the problem table. */
size_t fmm_f64_batch_ws_bytes(int count)
{
    return 256 + ((size_t)std::max(count, 0) * sizeof(F64Prob) + 255) / 256 * 256;
}

/* All problems of a batch in one persistent launch (plus the table-writer
 * launches and a counter reset). Problems are ordered by the FP64 work of one
 * of their items, largest first. Each result is identical to the problem
 * issued alone through fmm_f64_launch: every tile shape accumulates the
 * packed sums, the k loop and the products in the same order. */
namespace {
std::atomic<int> g_f64_batch_ctas{0};   /* 0: two CTAs per SM */
}  // namespace

extern "C" int fmm_gpu_set_f64_batch_ctas(int max_ctas)
{
    return g_f64_batch_ctas.exchange(max_ctas > 0 ? max_ctas : 0);
}

namespace {

/* Item tiles of a batch. One 64 x 64 item of a deep problem can last as long as
 * the whole batch (1024^3 222 x1: 14.7 M FMAs, 7 ms on half an SM), so a
 * problem's tile shrinks to 32, then 16, while its items hold more than an
 * eighth of a CTA's share of the batch: 24 problems of 256 to 1024 7.25 ms, 7.8
 * with 64 x 64 alone. That is within 3% of the best limit for 258 drawn
 * batches but for those whose items are nearly all alike, where smaller tiles
 * only cost more and whole rounds of items decide: for these the tile with the
 * least batch_rounds times batch_item_cost is taken if it saves 3%. Tiles of 64
 * / 32 / 16 / the rule, us: 2048^3 222 x1 15204 / 13633 / 16552 / 13640; 1912 x
 * 2475 x 97 232 x1 1522 / 1580 / 2015 / 1522; 1024^3 222 x1 3992 / 1966 / 2388
 * / 1966; 512^3 222 x1 2019 / 586 / 319 / 319; classical 1216 x 1024 x 500 1048
 * / 1052 / 1212 / 1048. */

/* FP64 pipe time of an item (a tile of all products) in FMAs at a 64 x 64
 * tile's rate. Smaller tiles pay for the pack additions of more tiles per
 * operand element (nn terms per product on both sides), 16 x 16 also for fewer
 * FMAs per shared-memory load and for the C updates of a short k. */
double batch_item_cost(const F64BatchItem& it, int tile, bool mma)
{
    const double ke = (double)((it.k + it.alg.kt - 1) / it.alg.kt), nn = it.alg.avg_nnz_u + it.alg.avg_nnz_v;
    double rel = 1.0;
    if (tile == 32)
        rel = mma ? 1.01 + 0.11 * (nn - 2.0) : 1.01 + 0.016 * (nn - 2.0) + 3.0 / ke;
    else if (tile == 16)
        rel = 1.14 + 0.085 * (nn - 2.0) + 11.0 / ke;
    return rel * tile * tile * it.alg.R * (ke + 1.0);
}

/* Time of n like items on `sms` SMs, in times of one item with an SM's FP64
 * pipe to itself: two CTAs of an SM share the pipe, the items of a last part
 * round are alone on their SM or nearly, and a CTA alone does not fill the
 * pipe, the less the smaller its tile and the more terms its packs have. */
double batch_rounds(double n, int sms, int tile, double nn)
{
    const double alone = tile == 64 ? std::max(1.05, 1.0 + 0.1 * (nn - 2.0))
                                    : tile == 32 ? 1.15 + 0.16 * (nn - 2.0) : 1.5 + 0.35 * (nn - 2.0);
    if (n <= sms) return alone;
    const double full = std::floor(n / (2.0 * sms)), left = n - full * 2.0 * sms;
    return 2.0 * full + (left <= 0.0 ? 0.0 : left <= sms ? std::min(2.0, 1.08 * alone) : 2.0);
}

/* each problem's tile, by the rule above, for `ctas` CTAs on `sms` SMs; items(i, tile): a problem's items */
template <class Items>
void batch_tiles(const F64BatchItem* p, const std::vector<int>& order, bool mma, int64_t ctas, int sms, Items items,
                 std::vector<int>& tile)
{
    const int least = mma ? 32 : 16;
    auto idle = [&](int i) { return p[i].k == 0 || p[i].alpha == 0.0; };   /* C := beta*C only */
    auto fmas = [&](int i, int t) {
        return idle(i) ? 1.0 : (double)t * t * p[i].alg.R * (double)((p[i].k + p[i].alg.kt - 1) / p[i].alg.kt + 1);
    };
    double total = 0.0, work = 0.0, most = 0.0;
    int heavy = -1;   /* the problem with the most work */
    for (int i : order) {
        total += fmas(i, 32) * (double)items(i, 32);
        const double w = fmas(i, 64) * (double)items(i, 64);
        work += w;
        if (!idle(i) && w > most) {
            most = w;
            heavy = i;
        }
    }
    for (int i : order) {
        tile[i] = 64;
        while (tile[i] > least && fmas(i, tile[i]) > total / (double)ctas / 8) tile[i] /= 2;
    }
    if (heavy < 0) return;
    /* the problems whose items are within a tenth of the heavy one's */
    const double len = fmas(heavy, 64);
    auto alike = [&](int i) { return !idle(i) && fmas(i, 64) <= len * 1.1 && fmas(i, 64) >= len / 1.1; };
    double part = 0.0;
    for (int i : order)
        if (alike(i)) part += fmas(i, 64) * (double)items(i, 64);
    if (part < 0.95 * work) return;
    const int slots = (int)std::min<int64_t>(ctas, sms);
    auto estimate = [&](int t) {
        double n = 0.0, longest = 0.0;
        for (int i : order)
            if (alike(i)) {
                n += (double)items(i, t);
                longest = std::max(longest, batch_item_cost(p[i], t, mma));
            }
        return longest * batch_rounds(n, slots, t, p[heavy].alg.avg_nnz_u + p[heavy].alg.avg_nnz_v);
    };
    double best = 0.97 * estimate(tile[heavy]);
    int to = tile[heavy];
    for (int t = 64; t >= least; t /= 2) {
        const double e = t == tile[heavy] ? best : estimate(t);
        if (e < best) {
            best = e;
            to = t;
        }
    }
    if (to != tile[heavy])
        for (int i : order)
            if (alike(i)) tile[i] = to;
}

}  // namespace

int fmm_f64_batch_launch(int count, const F64BatchItem* items, void* ws, size_t ws_bytes, cudaStream_t st)
{
    if (count <= 0) return FMM_OK;
    if (ws == nullptr || ws_bytes < fmm_f64_batch_ws_bytes(count)) return FMM_ERR_WORKSPACE;
    if (((uintptr_t)ws & 255) != 0) return FMM_ERR_ARG;
    std::vector<int> order;
    std::vector<double> cost(count, 0.0);
    for (int i = 0; i < count; ++i) {
        const F64BatchItem& it = items[i];
        if (it.alg.max_nnz_u > kMaxEntries || it.alg.max_nnz_v > kMaxEntries) return FMM_ERR_UNSUPPORTED;
        if (it.m == 0 || it.n == 0) continue;   /* nothing to do at all */
        if (it.k > 0 && it.alpha != 0.0 && fmm_plain_classical(it.alg)) {
            /* small/skinny classical problems take the same kernel as their
             * single calls (C := beta*C first, as there) */
            const int ks = fmm_gpu_f64_sup_splits(it.m, it.n, it.k);
            if (ks >= 2) {
                int rc = fmm_scale_c(it.m, it.n, it.beta, it.C, it.ldc, st);
                if (rc == FMM_OK) rc = sup_launch(it.m, it.n, it.k, it.alpha, it.A, it.lda, it.B, it.ldb, it.C,
                                                  it.ldc, ks, st);
                if (rc != FMM_OK) return rc;
                continue;
            }
        }
        order.push_back(i);
    }
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const bool mma = g_f64_engine.load(std::memory_order_relaxed) == FMM_F64_MMA;
    int64_t ctas = 2 * (int64_t)sms;
    const int cap = g_f64_batch_ctas.load();
    if (cap > 0) ctas = std::min<int64_t>(ctas, cap);
    auto tiles_of = [&](int i, int tile, int64_t* tm) {
        const F64BatchItem& it = items[i];
        const int64_t me = (it.m + it.alg.mt - 1) / it.alg.mt, ne = (it.n + it.alg.nt - 1) / it.alg.nt;
        *tm = (me + tile - 1) / tile;
        return *tm * ((ne + tile - 1) / tile);
    };
    std::vector<int> tile(count, 64);
    int64_t tm = 0;
    batch_tiles(items, order, mma, ctas, sms, [&](int i, int t) { return tiles_of(i, t, &tm); }, tile);
    for (int i : order) {
        const F64BatchItem& it = items[i];
        cost[i] = it.k == 0 || it.alpha == 0.0
                      ? 1.0 : (double)tile[i] * tile[i] * it.alg.R * (double)((it.k + it.alg.kt - 1) / it.alg.kt + 1);
    }
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return cost[a] > cost[b]; });
    std::vector<F64Prob> tab(order.size());
    int64_t items_total = 0;
    for (size_t q = 0; q < order.size(); ++q) {
        const F64BatchItem& it = items[order[q]];
        F64Prob& P = tab[q];
        P.tab = it.alg.tab;
        P.m = it.m; P.n = it.n; P.k = it.k;
        P.alpha = it.alpha; P.beta = it.beta;
        P.A = it.A; P.lda = it.lda; P.B = it.B; P.ldb = it.ldb; P.C = it.C; P.ldc = it.ldc;
        P.tile = tile[order[q]];
        const int64_t tiles = tiles_of(order[q], P.tile, &tm);
        if (tm > 0x7fffffffLL || tiles / tm > 0x7fffffffLL) return FMM_ERR_UNSUPPORTED;
        P.tiles_m = (int)tm;
        P.item_begin = items_total;
        items_total += tiles;
    }
    if (tab.empty()) return FMM_OK;
    unsigned long long* counter = (unsigned long long*)ws;
    F64Prob* dtab = (F64Prob*)((uint8_t*)ws + 256);
    if (cudaMemsetAsync(counter, 0, sizeof(unsigned long long), st) != cudaSuccess) return FMM_ERR_CUDA;
    for (size_t c0 = 0; c0 < tab.size(); c0 += kF64TableChunk) {
        F64TableChunk ch;
        ch.dst = dtab + c0;
        ch.count = (int)std::min<size_t>(kF64TableChunk, tab.size() - c0);
        memcpy(ch.p, tab.data() + c0, sizeof(F64Prob) * (size_t)ch.count);
        f64_table_write<<<1, 128, 0, st>>>(ch);
        fmm_count_launch(1);
    }
    const int64_t grid = std::min<int64_t>(items_total, ctas);   /* items are drawn from a counter: any grid finishes them */
    if (mma)
        fmm_f64_batch_kernel<true><<<(unsigned)grid, kF64BatchThreads, 0, st>>>(dtab, (int)tab.size(), items_total, counter);
    else
        fmm_f64_batch_kernel<false><<<(unsigned)grid, kF64BatchThreads, 0, st>>>(dtab, (int)tab.size(), items_total, counter);
    fmm_count_launch(1);
    return cudaGetLastError() == cudaSuccess ? FMM_OK : FMM_ERR_CUDA;
}

/* ---------------------------------------------------------------------------
 * Peak rates of the two FP64 paths of the SM, measured by compute-only
 * kernels (no memory traffic inside the loop): DFMA (fma.rn.f64, the plain
 * form's micro-kernel) and the FP64 tensor-core MMA (mma.sync m8n8k4 f64).
 * Each thread (DFMA) or warp (MMA) runs independent accumulation chains, so
 * the issue rate, not a dependency, bounds the loop.
 * ------------------------------------------------------------------------- */
namespace {

constexpr int kRateChains = 8;

/* NF DFMA chains per thread and NM FP64 MMA chains per warp, interleaved,
 * every chain with its own operand registers. On GB300 this compute-only loop
 * measures below what the DFMA GEMM kernel itself reaches (1.06 against
 * 1.25 TFLOP/s for the classical FP64 GEMM at 16384^3), so its figures are a
 * relative comparison of the two paths, not the pipe's peak. */
template <int NF, int NM>
__global__ void __launch_bounds__(256) fp64_rate_kernel(double* __restrict__ out, int iters)
{
    const int lane = threadIdx.x % 32;
    double a[kRateChains], bb[kRateChains], cc[kRateChains], d[kRateChains][2], x[kRateChains], y[kRateChains];
#pragma unroll
    for (int u = 0; u < kRateChains; ++u) {
        a[u] = 1e-3 * (threadIdx.x + u);
        bb[u] = 0.999999 - 1e-8 * u;
        cc[u] = 1e-9 * (u + 1);
        d[u][0] = 0.0;
        d[u][1] = 0.0;
        x[u] = 1e-3 * (lane + 1 + u);
        y[u] = 0.5 - 1e-3 * u;
    }
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int u = 0; u < kRateChains; ++u) {
            if (u < NF) a[u] = fma(a[u], bb[u], cc[u]);
            if (u < NM)
                asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                             : "+d"(d[u][0]), "+d"(d[u][1])
                             : "d"(x[u]), "d"(y[u]));
        }
    }
    double sum = 0.0;
#pragma unroll
    for (int u = 0; u < kRateChains; ++u) sum += a[u] + d[u][0] + d[u][1];
    out[blockIdx.x * (int64_t)blockDim.x + threadIdx.x] = sum;
}

}  // namespace

extern "C" int fmm_gpu_fp64_pipe_rates(double* dfma_tflops, double* dmma_tflops, double* mixed_tflops)
{
    if (dfma_tflops == nullptr || dmma_tflops == nullptr || mixed_tflops == nullptr) return FMM_ERR_ARG;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
        return FMM_ERR_CUDA;
    const int blocks = 8 * sms, threads = 256, iters = 16384;
    double* out = nullptr;
    if (cudaMalloc(&out, sizeof(double) * (size_t)blocks * threads) != cudaSuccess) return FMM_ERR_ALLOC;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    int rc = FMM_OK;
    float ms[3] = {0.f, 0.f, 0.f};
    for (int which = 0; which < 3 && rc == FMM_OK; ++which) {
        for (int rep = 0; rep < 3; ++rep) {   /* the first launch warms up */
            cudaEventRecord(e0);
            if (which == 0) fp64_rate_kernel<kRateChains, 0><<<blocks, threads>>>(out, iters);
            else if (which == 1) fp64_rate_kernel<0, kRateChains><<<blocks, threads>>>(out, iters);
            else fp64_rate_kernel<kRateChains / 2, kRateChains / 2><<<blocks, threads>>>(out, iters);
            cudaEventRecord(e1);
            fmm_count_launch(1);
            if (cudaEventSynchronize(e1) != cudaSuccess || cudaGetLastError() != cudaSuccess) { rc = FMM_ERR_CUDA; break; }
            float t = 0.f;
            cudaEventElapsedTime(&t, e0, e1);
            if (rep > 0 && (ms[which] == 0.f || t < ms[which])) ms[which] = t;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(out);
    if (rc != FMM_OK) return rc;
    const double threads_total = (double)blocks * threads;
    const double fma_flops = threads_total * iters * 2.0, mma_flops = threads_total / 32.0 * iters * (2.0 * 8 * 8 * 4);
    *dfma_tflops = fma_flops * kRateChains / (ms[0] * 1e-3) / 1e12;
    *dmma_tflops = mma_flops * kRateChains / (ms[1] * 1e-3) / 1e12;
    *mixed_tflops = (fma_flops + mma_flops) * (kRateChains / 2) / (ms[2] * 1e-3) / 1e12;
    return FMM_OK;
}

extern "C" int fmm_gpu_set_f64_engine(int engine)
{
    if (engine != FMM_F64_DFMA && engine != FMM_F64_MMA) return -1;
    return g_f64_engine.exchange(engine);
}
