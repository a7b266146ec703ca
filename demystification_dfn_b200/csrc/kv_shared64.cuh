// kv_shared64.cuh — FP64 K.V of a batch whose networks share one kernel
// matrix (DFN_STORE_FP64_SHARED). The R slip-rate vectors of a stage meet the
// same K, so K.V is a GEMM, C[k][m] = sum_l K[k][l] V_m[l] (rows k with their
// shear and normal entries, members m), in FP64 with K streamed from HBM once
// per member tile. It is the FP64 counterpart of the tensor-core batch
// (tc_gemm.cuh): same K sharing, FP64 products and sums, so that the two
// isolate what the BF16 hi+lo arithmetic itself gains. (The reference has one
// network per process and no batch.)
//
// The products run on the FP64 matrix instructions (mma.sync m16n8k4.f64:
// IEEE FP64 products and sums): the contraction is bound by the FP64 unit for
// R >= 16 (16 flop per byte of K at R = 64), and against scalar FMAs one
// instruction replaces 16 per lane and a fragment load serves 16 rows x 8
// members.
//
// K is stored row-major, N rows of Np columns (Np = N padded to S64_COLS with
// zero columns), {K_T, K_N} per column in mode II; the V of all members is
// packed per stage into vt[m][l] (members padded to 8, columns to Np, zeros).
// A CTA of four warps takes S64_ROWS rows (16 per warp) x 8 NT members (a
// member tile; NT the smallest that covers R in as few tiles as fill the GPU,
// so that padding costs at most 7 members per tile) and streams the columns in
// chunks of S64_COLS through a ring of shared-memory stages (cp.async, 16
// bytes per copy). A chunk is four instructions per group of eight members and
// component: in the j-th, lane (g, t) of a warp holds rows g, g + 8 of column
// t + 4 j. The stage rows are padded so that a quarter-warp's 16-byte reads of
// K and a half-warp's 8-byte reads of V cover all banks once.
//
// Split of the work: the (row tile, member tile, column chunk) steps form one
// sequence that the CTAs of a single wave share evenly (CTA b takes steps
// b*I/G .. (b+1)*I/G), so no last wave is partly empty and a row tile is cut
// into few pieces. The piece of CTA b of a tile that starts in CTA b0 goes to
// part[poff_m + (b - b0)*N + k]; the tile's last CTA zeroes the unused slots.
// The stage kernel adds the slots in fixed order: deterministic.
//
// Measured at N = 8 272, R = 50, mode II: 0.879 -> 0.479 ms per K.V (scalar
// FMAs on 32 x 64 tiles with 12 splits before; 32 TFLOP/s on the 56 padded
// members, the instruction alone reaches 37). What mattered besides the
// instruction: the loader's addresses advance by additions (recomputing them
// with divisions per chunk left the matrix unit idle a third of the time,
// 0.635 ms); more warps per scheduler (8 warps of half the members, or one
// component each) gave nothing (0.630-0.666 ms).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

constexpr int S64_ROWS = 64;
constexpr int S64_COLS = 16;
constexpr int S64_THREADS = 128;
constexpr int S64_NT = 8;                        // at most 8 tiles of 8 members per CTA
// Chunks a CTA gets at least. A chunk takes about 0.8 us, so small matrices
// are spread thin: N = 305, R = 43 takes 31 / 16.5 / 14.5 / 14.4 us with 8 / 4
// / 2 / 1 (one only adds partial sums); from N = 2000 on no difference.
constexpr int S64_MIN_STEPS = 2;
// Steps per SM below which the member tiles are narrowed, and the groups of
// eight members up to which one tile takes them all: a small matrix with wide
// tiles is a few CTAs of long, unevenly shared steps. K.V in us, scalar FMAs
// before / the fewest tiles / this rule, mode II: N = 100, R = 64 12.5 / 18.6 /
// 6.6; 200, 128 13.3 / 21.2 / 8.4; 450, 192 24.7 / 27.0 / 18.8; 1150, 64 34.9 /
// 40.7 / 22; 1386, 64 43.2 / 45.8 / 30.9. No size from 39 to 4000 with 2 to 256
// members is slower than with the scalar FMAs; with 8 steps 1150, 64 is, with
// 12 1386, 64, and with 16 or 24, or fewer groups narrowed too, others lose
// what these gain (1500, 17 15.5 -> 16.7; 850, 130 29.6 -> 33.5).
constexpr int S64_FILL = 14;
constexpr int S64_WHOLE = 4;
constexpr int S64_VROW = S64_COLS + 4;           // doubles of a staged V row (160 bytes)

// doubles of a staged K row: 320 bytes (mode II) or 160
__host__ __device__ constexpr int s64_krow(int mode) { return mode == 2 ? 2 * S64_COLS + 8 : S64_COLS + 4; }
__host__ __device__ constexpr int s64_stage_doubles(int mode, int nt)
{
    return S64_ROWS * s64_krow(mode) + 8 * nt * S64_VROW;
}
// stages that fit two CTAs per SM, at most 6
__host__ __device__ constexpr int s64_stages(int mode, int nt)
{
    return 108 * 1024 / (8 * s64_stage_doubles(mode, nt)) < 6 ? 108 * 1024 / (8 * s64_stage_doubles(mode, nt)) : 6;
}
__host__ __device__ constexpr size_t s64_smem_bytes(int mode, int nt)
{
    return sizeof(double) * (size_t)s64_stages(mode, nt) * s64_stage_doubles(mode, nt);
}

// The work of one launch: steps per row tile, steps in all, CTAs, tiles.
struct S64Plan {
    int nt = 1;            // tiles of 8 members per CTA
    int mtiles = 1;        // member tiles
    int nkc = 0;           // column chunks
    int rtiles = 0;        // row tiles
    int64_t steps = 0;     // rtiles * mtiles * nkc
    int64_t ctas = 0;
    int slots = 1;         // partial sums per element
};
// first step of CTA b, and the CTA that holds a step
__host__ __device__ inline int64_t s64_first(int64_t b, int64_t steps, int64_t ctas) { return b * steps / ctas; }
__host__ __device__ inline int64_t s64_cta_of(int64_t step, int64_t steps, int64_t ctas)
{
    int64_t b = step * ctas / steps;
    while (b + 1 < ctas && s64_first(b + 1, steps, ctas) <= step) b++;
    while (s64_first(b, steps, ctas) > step) b--;
    return b;
}

inline S64Plan s64_plan(int64_t N, int R, int sms)
{
    S64Plan p;
    const int n8 = (R + 7) / 8;
    p.nkc = (int)((N + S64_COLS - 1) / S64_COLS);
    p.rtiles = (int)((N + S64_ROWS - 1) / S64_ROWS);
    for (int tiles = (n8 + S64_NT - 1) / S64_NT;; tiles++) {
        p.nt = (n8 + tiles - 1) / tiles;
        p.mtiles = (n8 + p.nt - 1) / p.nt;
        p.steps = (int64_t)p.rtiles * p.mtiles * p.nkc;
        if (p.nt == 1 || n8 <= S64_WHOLE || p.steps >= (int64_t)S64_FILL * sms) break;
    }
    p.ctas = p.steps / S64_MIN_STEPS < 1 ? 1 : p.steps / S64_MIN_STEPS;
    if (p.ctas > 2 * (int64_t)sms) p.ctas = 2 * (int64_t)sms;
    for (int64_t t = 0; t < (int64_t)p.rtiles * p.mtiles; t++) {
        const int64_t n = s64_cta_of((t + 1) * p.nkc - 1, p.steps, p.ctas) - s64_cta_of(t * p.nkc, p.steps, p.ctas) + 1;
        if (n > p.slots) p.slots = (int)n;
    }
    return p;
}

// 16-byte copy; bytes = 0 writes zeros (src is not read then)
__device__ __forceinline__ void s64_cp16(void *smem_dst, const void *gmem_src, uint32_t bytes)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(static_cast<uint32_t>(
                     __cvta_generic_to_shared(smem_dst))),
                 "l"(gmem_src), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void s64_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void s64_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// C (16 x 8) += A (16 x 4) B (4 x 8): a[0], a[1] rows g, g + 8 of column t,
// b row t of column g, c rows g, g, g + 8, g + 8 of columns 2t, 2t + 1
__device__ __forceinline__ void s64_mma(double c[4], const double a[2], double b)
{
    asm volatile("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                 : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
                 : "d"(a[0]), "d"(a[1]), "d"(b));
}
// Whether any of the R networks takes part in a launch (CTA-uniform; a
// barrier): a shared K.V serves all of them or none.
__device__ __forceinline__ bool any_takes_part(const StepCtl *ctl, int R, int mask)
{
    int on = 0;
    for (int r = threadIdx.x; r < R; r += blockDim.x) on |= takes_part(ctl, r, mask);
    return __syncthreads_or(on) != 0;
}

// vt[m * Np + l] = V of member m at column l (zero beyond N and R); V of
// member m is Vbase[vmul * eoff_m + l]. grid (ceil(Np / 256), RP)
__global__ void s64_pack_v_kernel(const double *Vbase, int vmul, const Inst *__restrict__ inst,
                                  int64_t N, int R, int64_t Np, double *__restrict__ vt)
{
    const int64_t l = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int m = blockIdx.y;
    pdl_wait();
    pdl_trigger();
    if (l >= Np) return;
    vt[(int64_t)m * Np + l] = (l < N && m < R) ? Vbase[(int64_t)vmul * inst[m].eoff + l] : 0.0;
}

template <int MODE, int NT>
__global__ void __launch_bounds__(S64_THREADS, 2)
    s64_gemm_kernel(const double *__restrict__ K, const double *vt, const Inst *__restrict__ inst,
                    const StepCtl *ctl, int mask, int64_t N, int64_t Np, int R, S64Plan pl,
                    double *__restrict__ partT, double *__restrict__ partN)
{
    constexpr int CPE = (MODE == 2) ? 2 : 1;             // doubles per stored entry
    constexpr int KLD = s64_krow(MODE);
    constexpr int KSZ = S64_ROWS * KLD;
    constexpr int STAGE = s64_stage_doubles(MODE, NT);
    constexpr int ST = s64_stages(MODE, NT);
    extern __shared__ __align__(16) double s64_smem[];

    pdl_wait();
    pdl_trigger();
    if (!any_takes_part(ctl, R, mask)) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t4 = lane & 3;
    const int64_t s0 = s64_first(blockIdx.x, pl.steps, pl.ctas), s1 = s64_first(blockIdx.x + 1, pl.steps, pl.ctas);

    // Loader: the chunks of this CTA in order, each thread the same 16-byte
    // copies of every chunk (K rows krow + i * KRS, V members mrow + i * MRS),
    // from pointers that advance by one chunk and are set anew at a tile.
    constexpr int KV = S64_COLS * CPE / 2, KRS = S64_THREADS / KV, KN = S64_ROWS / KRS;
    constexpr int VV = S64_COLS / 2, MRS = S64_THREADS / VV, VN = (8 * NT + MRS - 1) / MRS;
    const int krow = tid / KV, kq = tid % KV, mrow = tid / VV, mq = tid % VV;
    const int64_t kstep = (int64_t)KRS * Np * CPE, vstep = (int64_t)MRS * Np;
    const double *kp = nullptr, *vp = nullptr;
    int lc = 0, ltile = 0, rows_left = 0;
    auto set_tile = [&](int tile, int c) {
        const int64_t r0 = (int64_t)(tile / pl.mtiles) * S64_ROWS, m0 = (int64_t)(tile % pl.mtiles) * (8 * NT);
        ltile = tile;
        lc = c;
        rows_left = (int)(N - r0 < S64_ROWS ? N - r0 : S64_ROWS);
        kp = K + ((r0 + krow) * Np + (int64_t)c * S64_COLS) * CPE + 2 * kq;
        vp = vt + (m0 + mrow) * Np + (int64_t)c * S64_COLS + 2 * mq;
    };
    auto load = [&](int st) {
        double *kd = s64_smem + st * STAGE + krow * KLD + 2 * kq;
        double *vd = s64_smem + st * STAGE + KSZ + mrow * S64_VROW + 2 * mq;
#pragma unroll
        for (int i = 0; i < KN; i++) {
            const bool on = krow + i * KRS < rows_left;   // rows beyond N: zeros
            s64_cp16(kd + i * KRS * KLD, on ? kp + i * kstep : K, on ? 16u : 0u);
        }
#pragma unroll
        for (int i = 0; i < VN; i++)
            if (VN * MRS == 8 * NT || mrow + i * MRS < 8 * NT) s64_cp16(vd + i * MRS * S64_VROW, vp + i * vstep, 16u);
        if (++lc == pl.nkc) {
            set_tile(ltile + 1, 0);
        } else {
            kp += S64_COLS * CPE;
            vp += S64_COLS;
        }
    };
    set_tile((int)(s0 / pl.nkc), (int)(s0 % pl.nkc));

    double cT[NT][4], cN[NT][4];
    auto zero = [&]() {
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
            for (int j = 0; j < 4; j++) { cT[n][j] = 0.0; cN[n][j] = 0.0; }
    };
    zero();
    const int nsteps = (int)(s1 - s0);
#pragma unroll
    for (int q = 0; q < ST - 1; q++) {
        if (q < nsteps) load(q);
        s64_commit();
    }
    int st = 0, tile = (int)(s0 / pl.nkc), c = (int)(s0 % pl.nkc);
    for (int step = 0; step < nsteps; step++) {
        s64_wait<ST - 2>();
        __syncthreads();   // stage st is complete; the stage before it has been read by all
        if (step + ST - 1 < nsteps) load(st == 0 ? ST - 1 : st - 1);
        s64_commit();
        const double *kb = s64_smem + st * STAGE + (16 * warp + g) * KLD;
        const double *vb = s64_smem + st * STAGE + KSZ + g * S64_VROW + t4;
        // one k step of 4 columns at a time over all members and components:
        // consecutive instructions are independent (a k chain within one
        // accumulator would wait for the unit's latency)
#pragma unroll
        for (int j = 0; j < 4; j++) {
            double aT[2], aN[2];
#pragma unroll
            for (int i = 0; i < 2; i++) {
                if (MODE == 2) {
                    const double2 kk = *reinterpret_cast<const double2 *>(kb + i * 8 * KLD + 2 * (t4 + 4 * j));
                    aT[i] = kk.x;
                    aN[i] = kk.y;
                } else {
                    aT[i] = kb[i * 8 * KLD + t4 + 4 * j];
                }
            }
#pragma unroll
            for (int n = 0; n < NT; n++) {
                const double b = vb[n * 8 * S64_VROW + 4 * j];
                s64_mma(cT[n], aT, b);
                if (MODE == 2) s64_mma(cN[n], aN, b);
            }
        }
        st = st == ST - 1 ? 0 : st + 1;
        const bool last = ++c == pl.nkc;
        if (last || step + 1 == nsteps) {
            // end of this CTA's piece of the tile
            const int64_t b0 = s64_cta_of((int64_t)tile * pl.nkc, pl.steps, pl.ctas);
            const int slot = (int)(blockIdx.x - b0);
            const int64_t r0 = (int64_t)(tile / pl.mtiles) * S64_ROWS + 16 * warp + g;
            const int m0 = tile % pl.mtiles * (8 * NT) + 2 * t4;
#pragma unroll
            for (int n = 0; n < NT; n++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int64_t row = r0 + 8 * (j >> 1);
                    const int m = m0 + 8 * n + (j & 1);
                    if (row < N && m < R) {
                        const int64_t o = inst[m].poff + row;
                        partT[o + (int64_t)slot * N] = cT[n][j];
                        if (MODE == 2) partN[o + (int64_t)slot * N] = cN[n][j];
                        if (last)
                            for (int q = slot + 1; q < pl.slots; q++) {
                                partT[o + (int64_t)q * N] = 0.0;
                                if (MODE == 2) partN[o + (int64_t)q * N] = 0.0;
                            }
                    }
                }
            zero();
            tile++;
            c = 0;
        }
    }
}
