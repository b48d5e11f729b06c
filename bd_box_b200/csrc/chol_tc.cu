// Mixed-precision blocked Cholesky for sm_100a: FP64 panels, FP16-split
// trailing updates on the 5th-generation tensor cores (tcgen05), and the
// plain FP64 path's updates on the FP64 tensor instruction (DMMA).
//
// M is FP32 (lower triangle: the factor, upper: D, never written here) or
// FP64 on the FP64 path. Super-panel P covers columns p0 = 128P .. p0+127:
//   k_potrf128  one CTA factors the 128x128 diagonal block in FP64 by 8
//               columns (each 8x8 pivot block factored and inverted by the
//               pivot warp while the other warps form and solve their
//               tiles), and hands L_PP and the inverses W_kk of its 8x8 diagonal tiles on
//               to the panel solve;
//   k_trsm128   the rows below, X L_PP^T = A, by blocked forward substitution
//               in FP64 (one warp per 8 rows, DMMA); each row goes to M and,
//               on the mixed path, as an FP16 hi/lo pair of the row scaled
//               by a power of two (k_panel_scale) to two panel buffers;
//   k_syrk_tc   C -= L_i L_j^T for single 128x128 tiles and block columns
//               (the next three block columns), and
//   k_syrk_tc2  for 256x256 blocks on CTA pairs (the columns beyond), two
//               panels per pass over C, with
//               L_i L_j^T ~= (Lhi_i Lhi_j^T + Lhi_i Llo_j^T + Llo_i Lhi_j^T)
//                            / scale^2
//               (the dropped lo*lo term is ~2^-22 relative: FP32 accuracy);
//   k_syrk64    the FP64 path's updates on mma.sync.m8n8k4.f64;
//   k_syrk_diag the next diagonal tile's update, on both paths.
//
// The update kernels are persistent and warp-specialised:
//   warp 0    TMA producer: per K chunk of 64 columns, four 128x64 FP16
//             boxes (A_hi, A_lo, B_hi, B_lo, 128-byte swizzle) into a
//             3-stage ring;
//   warp 1    MMA issuer: tcgen05.mma.kind::f16 (K=16), three per K step,
//             into one of two TMEM accumulators; tcgen05.commit frees a ring
//             stage / publishes an accumulator;
//   warps 2-5 epilogue: tcgen05.ld of the accumulator (warp w reads TMEM
//             lanes 32(w%4)..), hand the accumulator back, then
//             -acc / scale^2 per 128x32 box into a 2-box shared-memory ring
//             and a TMA reduce-add into C (lower triangle only on diagonal
//             tiles); C is never loaded.
// The epilogue of tile t overlaps the MMAs of tile t+1 and the loads of the
// tiles after it. Every mbarrier wait is bounded; a time-out sets
// ST_TIMEOUT and a shared abort flag that stops all roles, and the CTA frees
// its tensor memory before returning.
//
// Kernels are chained as programmatic dependents (griddepcontrol): each
// reads its inputs only after griddepcontrol.wait. Where the dependent is a
// small kernel of the panel chain, it is released early so that its launch
// overlaps; where it is a full grid (the next bulk update, the side
// stream's column update), only near the end, since its CTAs would hold the
// free SMs in their wait for as long as the releasing kernel runs.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <cuda_fp16.h>

#include <algorithm>

#include "bdb_common.cuh"
#include "sm100.cuh"

namespace bdb {

static constexpr int PW = 128;                    // super-panel width = tile size
static constexpr int KC = 32;                     // FP32 columns of a box of the C update (128 B)
static constexpr int KCP = 64;                    // panel K columns per TMA box (128 B of FP16)
static constexpr int NCHUNK = PW / KCP;           // 2 boxes per panel
static constexpr int KSTEPS = KCP / 16;           // MMA k-steps per box (K = 16 for kind::f16)
static constexpr int STAGES = 3;
static constexpr int BOX_BYTES = PW * KC * 4;     // 16 KB: a C box, and a panel box (PW x KCP x 2 B)
static_assert(PW * KCP * 2 == BOX_BYTES, "panel and C boxes have the same size");
static constexpr int STAGE_BYTES = 4 * BOX_BYTES; // A_hi, A_lo, B_hi, B_lo
static constexpr int C_BOXES = 2;                 // staging ring of 128x32 boxes for the C update
static constexpr int SYRK_SMEM = STAGES * STAGE_BYTES + C_BOXES * BOX_BYTES + 1024;

// C[tile] += smem tile (FP32 add in L2, no load of C by the SM)
__device__ __forceinline__ void tma_reduce_add_2d(const CUtensorMap* map, uint32_t src, int x, int y)
{
    asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
                 "r"(x), "r"(y), "r"(src)
                 : "memory");
}

__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }

// wait until at most C_BOXES-1 of this thread's bulk groups still read
// shared memory
__device__ __forceinline__ void bulk_wait_read_ring()
{
    static_assert(C_BOXES == 2, "wait_group count below");
    asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
}

__device__ __forceinline__ void bulk_wait0() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// barrier 1 among the 128 epilogue threads only
__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// barrier 1 with an OR over the 128 epilogue threads: all of them see the
// same answer, so they leave their loop together
__device__ __forceinline__ bool epi_any(bool x)
{
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 q, %1, 0;\n\t"
        "bar.red.or.pred p, 1, 128, q;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)x)
        : "memory");
    return r != 0;
}

// UMMA shared-memory descriptor: K-major, 128-byte swizzle, 8-row groups
// 1024 bytes apart (SBO = 64 x 16 B), LBO = 1 (unused for swizzled K-major),
// version 1 (sm_100), layout type 2 (SWIZZLE_128B).
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr)
{
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)1u << 16;
    d |= (uint64_t)64u << 32;
    d |= (uint64_t)1u << 46;
    d |= (uint64_t)2u << 61;
    return d;
}

// instruction descriptor: D=F32, A=B=F16, both K-major, N=128, M=128
__host__ __device__ constexpr uint32_t idesc_f16_128x128()
{
    return (1u << 4) | (0u << 7) | (0u << 10) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
}

__device__ __forceinline__ void umma_f16(uint32_t tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void umma_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}

__device__ __forceinline__ void tri_index(int idx, int& ti, int& tj)
{
    int i = (int)((sqrtf(8.0f * (float)idx + 1.0f) - 1.0f) * 0.5f);
    while ((i + 1) * (i + 2) / 2 <= idx) ++i;
    while (i * (i + 1) / 2 > idx) --i;
    ti = i;
    tj = idx - i * (i + 1) / 2;
}

// tile t of a launch -> (ti, tj) relative to the first trailing block:
// mode 2 only block column 1, 3 block columns 2 and beyond, 4 block column 0
// below its diagonal tile (which is k_syrk_diag's), 5 only block column 2
__device__ __forceinline__ void tile_of_mode(int t, int mode, int& ti, int& tj)
{
    if (mode == 5) {
        ti = t + 2;
        tj = 2;
    } else if (mode == 4) {
        ti = t + 1;
        tj = 0;
    } else if (mode == 2) {
        ti = t + 1;
        tj = 1;
    } else {
        tri_index(t, ti, tj);
        ti += 2;
        tj += 2;
    }
}

// the mixed path's panel operands: x = (hi + lo) / scale with hi and lo in
// FP16 (11 significant bits each, 22 together: the accuracy class of a
// TF32 hi/lo split, at twice the tensor rate and half the bytes). scale is
// a power of two chosen per factorisation from D's largest diagonal entry
// (|L_ij| <= sqrt(D_ii)), so that every entry stays in FP16's normal range
// where it matters; the products are unscaled exactly in the epilogue.
__device__ __forceinline__ void f16_split(float x, float scale, __half& hi, __half& lo)
{
    const float xs = x * scale;
    hi = __float2half_rn(xs);
    lo = __float2half_rn(xs - __half2float(hi));
}

// ------------------------------------------------------------ FP64 panel

// FP64 tensor-core MMA (the only FP64 tensor instruction on sm_100a; the
// tcgen05 kinds have no FP64): D = A B + C for an 8x8 tile, k = 4. Lane l
// holds A[l/4][l%4], B[l%4][l/4] and C/D[l/4][2(l%4) + {0,1}].
__device__ __forceinline__ void dmma884(double& d0, double& d1, double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// Every product here is X Y^T of 8x8 tiles, summed over their columns, so the
// columns may be taken in any order that both operands share: k-step h of a
// DMMA takes columns 2 q + h (q = lane mod 4). A lane's A fragments of X and B
// fragments of Y^T are then the pair [l/4][2 (l%4) + {0, 1}], the lane's own
// elements of a C fragment: tiles are kept by rows, one 16-byte load gives
// both k-steps, and an accumulator is the next product's operand as it is.
// tile (g, n), n <= g, of the lower triangle of 16 x 16 tiles
__device__ __forceinline__ int tix(int g, int n) { return g * (g + 1) / 2 + n; }

// 1/x for x > 0 in FP64: the hardware's FP64 reciprocal estimate (no
// conversions on the pivot chain) refined by one Newton-Raphson step
// q <- q + q (1 - x q), which squares its relative error.
__device__ __forceinline__ double rcp_nr(double x)
{
    double q;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(q) : "d"(x));
    return fma(q, fma(-x, q, 1.0), q);
}

// 1/sqrt(x) for the pivots: the hardware's FP64 estimate (~20 bits) and, with
// e = 1 - x y^2, one step of third order y <- y + y e (1/2 + 3/8 e) (its error
// is 5/16 e^3, below FP64 rounding of the FP32 factor that leaves; one dependent
// operation more than a Newton-Raphson step, which leaves 2^-40), or two
// Newton-Raphson steps with kFull (FP64 rounding)
template <bool kFull>
__device__ __forceinline__ double pivot_rsqrt(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-(x * y), y, 1.0);
    if (!kFull) return fma(y * e, fma(0.375, e, 0.5), y);
    y = fma(0.5 * y, e, y);
    return fma(0.5 * y, fma(-(x * y), y, 1.0), y);
}

// The 8x8 pivot block and every row that meets it. Dg ([8][DLD], lower
// triangle) is factored in registers, every lane of the pivot warp the whole
// of it (nothing passes between lanes): elimination on the unscaled Schur
// complements with q_j = 1/a_jj, the next pivot a_{j+1,j+1} -= a_{j+1,j}^2 q_j
// first (the square is formed while q_j is computed, so one reciprocal and
// one FMA separate two pivots), then the other entries as a_ic -= a_ij t_c, t_c
// = a_cj q_j. The t_c replace column j; a_jj becomes 1/sqrt(a_jj) = 1/L_jj.
// Columns [J0, J1).
static constexpr int DLD = 10;   // row stride of 8x8 blocks kept by rows (16-byte rows, distinct banks)

template <bool kFull, int J0, int J1>
__device__ __forceinline__ bool pivot8(double (&a)[8][8])
{
    bool ok = true;
#pragma unroll
    for (int j = J0; j < J1; ++j) {
        if (!(a[j][j] > 0.0)) ok = false;
        double q = rcp_nr(a[j][j]);
        if (kFull) q = fma(q, fma(-a[j][j], q, 1.0), q);
        if (j + 1 < 8) a[j + 1][j + 1] = fma(-(a[j + 1][j] * a[j + 1][j]), q, a[j + 1][j + 1]);
        double t[8];
#pragma unroll
        for (int k = j + 1; k < 8; ++k) t[k] = a[k][j] * q;
#pragma unroll
        for (int r = j + 1; r < 8; ++r)
#pragma unroll
            for (int k = j + 1; k <= r; ++k)
                if (r != j + 1) a[r][k] = fma(-a[r][j], t[k], a[r][k]);
#pragma unroll
        for (int k = j + 1; k < 8; ++k) a[k][j] = t[k];
        a[j][j] = pivot_rsqrt<kFull>(a[j][j]);
    }
    return ok;
}

// x L^T = c for one row c per lane, columns [J0, J1), from pivot8's t and
// 1/L_jj: the rows of L[k+1][k] from those of C[k+1][k], the columns of W_kk =
// L_kk^-1 from unit rows, the rows of L_kk from those of the block itself. (The
// scaling by 1/L_jj is left to the end: c_j enters the later columns unscaled.)
template <int J0, int J1>
__device__ __forceinline__ void pivot8_row(const double (&t)[8][8], double (&c)[8])
{
#pragma unroll
    for (int j = J0; j < J1; ++j)
#pragma unroll
        for (int k = j + 1; k < 8; ++k) c[k] = fma(-c[j], t[k][j], c[k]);
}

// two consecutive elements of an FP32 or FP64 matrix as doubles, and back
__device__ __forceinline__ double2 ld_pair(const float* p)
{
    const float2 v = *reinterpret_cast<const float2*>(p);
    return make_double2(v.x, v.y);
}
__device__ __forceinline__ double2 ld_pair(const double* p) { return *reinterpret_cast<const double2*>(p); }
__device__ __forceinline__ void st_pair(float* p, double a, double b)
{
    *reinterpret_cast<float2*>(p) = make_float2((float)a, (float)b);
}
__device__ __forceinline__ void st_pair(double* p, double a, double b)
{
    *reinterpret_cast<double2*>(p) = make_double2(a, b);
}

static constexpr int POTRF_THREADS = 512;
static constexpr int NT = PW / 8;                  // 16 row groups of 8 rows
static constexpr int NTILE = NT * (NT + 1) / 2;    // 136 tiles in the lower triangle
// Lt tiles, W_kk, the 8x8 block being factored, and per step a hand-over slot
// of two tiles
static constexpr int HAND = 8 * DLD + 64;
static constexpr int POTRF_SMEM = (NTILE * 64 + NT * 64 + 8 * DLD + NT * HAND) * 8;
// factor hand-off to the panel solve: L_PP tiles then the W_kk, by rows
static constexpr int PANEL_FAC = (NTILE + NT) * 64;

// row group owned by a warp: warp 0 runs the pivots; warps 4, 8, 12 share
// its scheduler (warp w issues on sub-partition w mod 4) and own the row
// groups with the least work (1, 2, 3); the other 12 warps own 4..15
__device__ __forceinline__ int row_group_of(int warp)
{
    return (warp & 3) ? 4 + warp - 1 - (warp >> 2) : warp >> 2;
}

// progress counters of k_potrf128: each is raised by one warp at a time, after
// what it announces
struct PotrfFlags {
    int piv;        // L_kk, W_kk and L[k+1][k] published for k < piv
    int hand;       // hand-over slots 1 .. hand written
    int row[NT];    // tiles (g, m), m < row[g], published by row group g's owner
};

__device__ __forceinline__ void flag_set(int* f, int v)
{
    asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(smem_u32(f)), "r"(v) : "memory");
}

// all 32 lanes poll until *f >= v, at most `limit` times; false on a time-out
// or an abort. (An mbarrier's try_wait suspends the warp: it woke 230 cycles
// after the arrival, a poll sees a flag within about 40; a relaxed wait polls
// less often and leaves the issue slots to others.)
__device__ __forceinline__ bool flag_wait(const int* f, int v, volatile int* abort_flag, uint32_t limit,
                                          bool relaxed = false)
{
    bool ok = false;
    for (uint32_t it = 0; it < limit; ++it) {
        int x;
        asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(x) : "r"(smem_u32(f)) : "memory");
        if (x >= v) {
            ok = true;
            break;
        }
        if ((it & 1023) == 1023 && *abort_flag) break;
        if (relaxed) __nanosleep(64);
    }
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) *abort_flag = 1;
    return ok;
}

// A solved off-diagonal tile X (C fragments x0, x1 of lane (fr, fq)) of
// L_PP, tile index t = tix(g, n): to the FP64 hand-off for the panel solve and,
// in M's precision, to M
template <typename T>
__device__ __forceinline__ void put_tile(double* Wt, T* M, size_t row0, size_t col0, int npad, int t,
                                         int lane, double x0, double x1)
{
    *reinterpret_cast<double2*>(Wt + t * 64 + 2 * lane) = make_double2(x0, x1);
    st_pair(M + (row0 + (lane >> 2)) * npad + col0 + 2 * (lane & 3), x0, x1);
}

// FP64 factorisation L_PP of the 128x128 diagonal block (P, P) and the
// inverses W_kk of its 8x8 diagonal tiles, over 16 blocks of 8 columns. One
// warp runs the pivots, the warp owning row group g forms its tiles (g, n) left
// to right, each when its column's turn comes, from tiles in shared memory; no
// CTA-wide barrier orders the steps, progress counters carry exactly what each
// warp needs:
//   pivot warp, step k: factor tile (k, k) (pivot8, every lane the whole
//     factorisation) with one more row per lane carried along (pivot8_row),
//     which gives in lanes 0-7 the rows of L[k+1][k], in lanes 8-15 W_kk, in
//     lanes 16-23 L_kk -> publish all three; update tile (k+1, k+1) with
//     L[k+1][k] and go on to pivot k+1;
//   owner g, step k <= g-2: C[g][k] -= sum over m < k of L[g][m] L[k][m]^T (row
//     group k is complete once pivot k-1 is published), then L[g][k] = C[g][k]
//     W_kk^T -> publish. Its last two tiles (g, g-1) and (g, g) take every
//     column as it comes; at k = g-2 they are complete up to it and are handed
//     to the pivot warp.
// So the pivot chain holds, per 8 columns, one pivot block (8 reciprocals) and
// one rank-8 update; the hand-over of row group k+1 (one solve and one update
// behind pivot k-1) is made while the first half of pivot block k is
// eliminated. The owners' sums of a step are at most 56 tile products over
// three schedulers (right-looking updates, 100 in the first steps, stood in
// front of the hand-over on the FP64 tensor pipes: 3,700 cycles a step there,
// against 2,000 of the chain itself).
// Each solved tile goes to M and to the FP64 hand-off Wt for the panel solve
// (by rows: the 136 L_PP tiles, then the 16 W_kk; PANEL_FAC doubles) as soon as
// it is final, so nothing is left to store at the end. Every wait is bounded:
// a time-out sets ST_TIMEOUT and every warp runs out to the final barrier.
// Bound by the pivot chain's latency: a block by itself took 21.9 us with
// right-looking updates and mbarriers (FP64 path 23.6);
// now 16.3 and 17.3.
template <typename T>
__global__ void __launch_bounds__(POTRF_THREADS, 1) k_potrf128(T* __restrict__ M, int npad, int P,
                                                            double* __restrict__ Wt, unsigned* __restrict__ status,
                                                            uint32_t wlim)
{
    extern __shared__ double sh[];
    double* Lt = sh;                       // [NTILE][64] tiles by rows: M's, then L's
    double* Wa = Lt + NTILE * 64;          // [NT][64] W_kk by rows
    double* Dg = Wa + NT * 64;             // [8][DLD] diagonal block being factored
    double* Hd = Dg + 8 * DLD;             // [NT][HAND] hand-over slots: (g, g-1) as [8][DLD], (g, g) by rows
    __shared__ PotrfFlags fl;
    __shared__ int bad;
    __shared__ volatile int abort_flag;
    {
        // the warp roles assume this exact launch shape
        uint32_t dyn;
        asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
        if (blockDim.x != POTRF_THREADS || dyn < (uint32_t)POTRF_SMEM) {
            if (threadIdx.x == 0) atomicOr(status, ST_LAUNCH);
            return;
        }
    }
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int fr = lane >> 2, fq = lane & 3;
    const size_t base = (size_t)P * PW;
    const int g = row_group_of(warp);
    if (tid < NT) fl.row[tid] = 0;
    if (tid == 0) {
        fl.piv = fl.hand = 0;
        bad = 0;
        abort_flag = 0;
    }
    __syncthreads();
    // launched as a programmatic dependent of the update of this block
    // column: the set-up above overlaps its tail, M is read only after it
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (warp == 0) {
        // ---------------------------------------------------- pivot warp
        // tile (0, 0) to Dg, tiles (1, 0) and (1, 1) to the first hand-over
        // slot (nothing updates them before step 0)
        {
            const double2 d = ld_pair(M + (base + fr) * npad + base + 2 * fq);
            const double2 a = ld_pair(M + (base + 8 + fr) * npad + base + 2 * fq);
            const double2 b = ld_pair(M + (base + 8 + fr) * npad + base + 8 + 2 * fq);
            *reinterpret_cast<double2*>(Dg + fr * DLD + 2 * fq) = d;
            *reinterpret_cast<double2*>(Hd + fr * DLD + 2 * fq) = a;
            *reinterpret_cast<double2*>(Hd + 8 * DLD + 2 * lane) = b;
        }
        __syncwarp();
        const int role = lane >> 3, row = lane & 7;   // 0: L[k+1][k], 1: W_kk, 2: L_kk, 3: none
        for (int k = 0; k < NT; ++k) {
            // the dependent (block row P+1's solve, 4 CTAs) launches for the
            // last steps only: launched at the start, its CTAs held 4 SMs in
            // their wait for the whole factorisation
            if (k == NT - 6) asm volatile("griddepcontrol.launch_dependents;");
            double a[8][8], c[8];
#pragma unroll
            for (int r = 0; r < 8; ++r)
#pragma unroll
                for (int j = 0; j <= r; j += 2) {
                    const double2 v = *reinterpret_cast<const double2*>(Dg + r * DLD + j);
                    a[r][j] = v.x;
                    if (j + 1 <= r) a[r][j + 1] = v.y;
                }
            bool ok = pivot8<sizeof(T) == 8, 0, 4>(a);
            // tiles (k+1, k) and (k+1, k+1) through column k-1
            const double* h0 = Hd + (size_t)k * HAND;
            if (k + 1 < NT && !flag_wait(&fl.hand, k, &abort_flag, wlim)) break;
            const double* src = role == 0 ? h0 + row * DLD : Dg + row * DLD;
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
                const double2 v = *reinterpret_cast<const double2*>(src + j);
                c[j] = role == 1 ? (row == j ? 1.0 : 0.0) : v.x;
                c[j + 1] = role == 1 ? (row == j + 1 ? 1.0 : 0.0) : v.y;
            }
            const double2 t2 = *reinterpret_cast<const double2*>(h0 + 8 * DLD + 2 * lane);
            pivot8_row<0, 4>(a, c);
            ok &= pivot8<sizeof(T) == 8, 4, 8>(a);
            pivot8_row<4, 8>(a, c);
            if (!ok && lane == 0) bad = 1;
#pragma unroll
            for (int j = 0; j < 8; ++j) c[j] *= a[j][j];
            // rows of L and columns of W_kk (zero before its diagonal: so are
            // c's entries there), one store for all three roles: branches by
            // role took 170 cycles more. L_kk's upper half is never read.
            double* dst = role == 0 ? Lt + tix(k + 1, k) * 64 + row * 8
                          : role == 1 ? Wa + k * 64 + row
                                      : Lt + tix(k, k) * 64 + row * 8;
            const int step = role == 1 ? 8 : 1;
            if (role < 3 && (role > 0 || k + 1 < NT)) {
#pragma unroll
                for (int j = 0; j < 8; ++j) dst[j * step] = c[j];
            }
            __syncwarp();
            if (lane == 0) flag_set(&fl.piv, k + 1);
            if (k + 1 == NT) break;
            // tile (k+1, k+1) -= L[k+1][k] L[k+1][k]^T: the next pivot block
            const double2 av = *reinterpret_cast<const double2*>(Lt + tix(k + 1, k) * 64 + 2 * lane);
            double e0 = t2.x, e1 = t2.y, f0 = 0.0, f1 = 0.0;
            dmma884(e0, e1, -av.x, av.x);
            dmma884(f0, f1, -av.y, av.y);
            *reinterpret_cast<double2*>(Dg + fr * DLD + 2 * fq) = make_double2(e0 + f0, e1 + f1);
            __syncwarp();
        }
    } else if (g == 1) {
        // ------------------------------------------------------ store warp
        // (row group 1 needs no owner: the pivot warp takes its tiles). It
        // copies the pivot warp's results to global memory off the pivot
        // chain, once published: L_kk, W_kk and L[k+1][k]; FP64 to Wt, L in M's
        // precision to M
        for (int k = 0; k < NT; ++k) {
            if (!flag_wait(&fl.piv, k + 1, &abort_flag, wlim, true)) break;
            const double2 l = *reinterpret_cast<const double2*>(Lt + tix(k, k) * 64 + 2 * lane);
            *reinterpret_cast<double2*>(Wt + tix(k, k) * 64 + 2 * lane) = l;
            *reinterpret_cast<double2*>(Wt + (NTILE + k) * 64 + 2 * lane) =
                *reinterpret_cast<const double2*>(Wa + k * 64 + 2 * lane);
            T* m = M + (base + 8 * k + fr) * npad + base + 8 * k + 2 * fq;
            if (2 * fq <= fr) m[0] = (T)l.x;
            if (2 * fq + 1 <= fr) m[1] = (T)l.y;
            if (k + 1 == NT) break;
            const double2 x = *reinterpret_cast<const double2*>(Lt + tix(k + 1, k) * 64 + 2 * lane);
            put_tile(Wt, M, base + 8 * (k + 1), base + 8 * k, npad, tix(k + 1, k), lane, x.x, x.y);
        }
    } else {
        // -------------------------------------------------- tile owners
        double s0, s1, d0, d1;   // tiles (g, g-1) and (g, g)
        {
            double2 v[NT];
#pragma unroll
            for (int n = 0; n < NT; ++n)
                if (n <= g) v[n] = ld_pair(M + (base + 8 * g + fr) * npad + base + 8 * n + 2 * fq);
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                if (n + 2 <= g) *reinterpret_cast<double2*>(Lt + tix(g, n) * 64 + 2 * lane) = v[n];
                if (n + 1 == g) s0 = v[n].x, s1 = v[n].y;
                if (n == g) d0 = v[n].x, d1 = v[n].y;
            }
        }
        double* Lg = Lt + tix(g, 0) * 64 + 2 * lane;
        double x0 = 0.0, x1 = 0.0;   // L[g][k-1]
        for (int k = 0; k + 1 < g; ++k) {
            // C[g][k], four running sums
            double2 c = *reinterpret_cast<const double2*>(Lg + k * 64);
            {
                const double* Lk = Lt + tix(k, 0) * 64 + 2 * lane;
                double p0 = 0.0, p1 = 0.0, q0 = 0.0, q1 = 0.0, r0 = 0.0, r1 = 0.0;
                int m = 0;
                for (; m + 2 <= k; m += 2) {
                    const double2 a0 = *reinterpret_cast<const double2*>(Lg + m * 64);
                    const double2 b0 = *reinterpret_cast<const double2*>(Lk + m * 64);
                    const double2 a1 = *reinterpret_cast<const double2*>(Lg + m * 64 + 64);
                    const double2 b1 = *reinterpret_cast<const double2*>(Lk + m * 64 + 64);
                    dmma884(c.x, c.y, -a0.x, b0.x);
                    dmma884(p0, p1, -a0.y, b0.y);
                    dmma884(q0, q1, -a1.x, b1.x);
                    dmma884(r0, r1, -a1.y, b1.y);
                }
                if (m < k) {
                    const double2 b0 = *reinterpret_cast<const double2*>(Lk + m * 64);
                    dmma884(c.x, c.y, -x0, b0.x);
                    dmma884(p0, p1, -x1, b0.y);
                }
                c.x += p0 + (q0 + r0);
                c.y += p1 + (q1 + r1);
            }
            if (k > 0) {
                // column k-1 of tile (g, g-1)
                if (!flag_wait(&fl.row[g - 1], k, &abort_flag, wlim)) break;
                const double2 b = *reinterpret_cast<const double2*>(Lt + tix(g - 1, k - 1) * 64 + 2 * lane);
                dmma884(s0, s1, -x0, b.x);
                dmma884(s0, s1, -x1, b.y);
            }
            if (!flag_wait(&fl.piv, k + 1, &abort_flag, wlim, k + 4 < g)) break;
            // L[g][k] = C[g][k] W_kk^T
            const double2 wb = *reinterpret_cast<const double2*>(Wa + k * 64 + 2 * lane);
            double y0 = 0.0, y1 = 0.0;
            x0 = x1 = 0.0;
            dmma884(x0, x1, c.x, wb.x);
            dmma884(y0, y1, c.y, wb.y);
            x0 += y0;
            x1 += y1;
            *reinterpret_cast<double2*>(Lg + k * 64) = make_double2(x0, x1);
            if (k + 2 == g) {
                // the last two tiles through column k, for the pivot warp
                // (whose row g-1 of column k came with W_kk)
                const double2 b = *reinterpret_cast<const double2*>(Lt + tix(g - 1, k) * 64 + 2 * lane);
                double t0 = 0.0, t1 = 0.0, u0 = 0.0, u1 = 0.0;
                dmma884(s0, s1, -x0, b.x);
                dmma884(t0, t1, -x1, b.y);
                dmma884(d0, d1, -x0, x0);
                dmma884(u0, u1, -x1, x1);
                double* h = Hd + (size_t)(k + 1) * HAND;
                *reinterpret_cast<double2*>(h + fr * DLD + 2 * fq) = make_double2(s0 + t0, s1 + t1);
                *reinterpret_cast<double2*>(h + 8 * DLD + 2 * lane) = make_double2(d0 + u0, d1 + u1);
            }
            __syncwarp();
            if (lane == 0) {
                if (k + 2 == g) flag_set(&fl.hand, k + 1);
                flag_set(&fl.row[g], k + 1);
            }
            put_tile(Wt, M, base + 8 * g, base + 8 * k, npad, tix(g, k), lane, x0, x1);
            if (k + 2 < g) {
                dmma884(d0, d1, -x0, x0);
                dmma884(d0, d1, -x1, x1);
            }
        }
    }
    __syncthreads();
    if (tid == 0) {
        if (bad) atomicOr(status, ST_NOT_SPD);
        if (abort_flag) atomicOr(status, ST_TIMEOUT);
    }
}

// Rows below block P: X L_PP^T = A by blocked forward substitution in FP64
// on the DMMA path, from the tiles of L_PP and the inverses W_kk of its
// diagonal tiles (k_potrf128). Work unit = one row group of 8 rows, owned by
// one warp, which keeps the unit's 16 tiles C_n (8x8, 32 doubles per lane)
// as DMMA accumulators loaded straight from M. For n = 0..15:
//   X_n = C_n W_nn^T                       (two DMMAs),
//   C_n' -= X_n L_n'n^T for n' > n         (two DMMAs each),
// 272 DMMAs per unit; a C fragment is the next A fragment (k_potrf128's column order). The CTA copies the
// factor (76 KB) into shared memory once. The grid is persistent: unit u goes
// to warp slot u mod (8 grid), slots ordered so that the first 4 grid slots
// put one warp on every SM sub-partition, the next 4 grid a second one.
// Writes the rows to M and, for the mixed path (T = float), their FP16
// split L s = hi + lo (f16_split, s = pscale[0]) to the panel buffers; for
// the FP64 path (T = double) the rows in FP64 to one panel buffer (Lhi, as
// doubles; Llo unused).
static constexpr int TRSM_THREADS = 256;
static constexpr int TRSM_SMEM = PANEL_FAC * 8;

template <typename T>
__global__ void __launch_bounds__(TRSM_THREADS, 1) k_trsm128(T* __restrict__ M, int npad, int P, int unit0, int units,
                                                          const double* __restrict__ Lf, float* __restrict__ Lhi,
                                                          float* __restrict__ Llo, unsigned* __restrict__ status,
                                                          const float* __restrict__ pscale)
{
    {
        uint32_t dyn;
        asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
        if (blockDim.x != TRSM_THREADS || dyn < (uint32_t)TRSM_SMEM) {
            if (threadIdx.x == 0) atomicOr(status, ST_LAUNCH);
            return;
        }
    }
    // block row P+1 (unit0 = 0) releases its dependent, the chain's update of
    // the next diagonal tile (k_syrk_diag, 10 CTAs), at once; the rows below only as their warps finish, because
    // theirs is the side stream's column update, a grid that would
    // otherwise wait on the free SMs the chain needs while this runs
    if (unit0 == 0) asm volatile("griddepcontrol.launch_dependents;");
    extern __shared__ double sh[];
    const double2* Ls = reinterpret_cast<const double2*>(sh);               // [NTILE][32] pairs
    const double2* Ws = reinterpret_cast<const double2*>(sh + NTILE * 64);  // [NT][32] pairs
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int fr = lane >> 2, fq = lane & 3;
    const size_t base = (size_t)P * PW;
    // units unit0 .. unit0 + units - 1 of 8 rows below the block
    const size_t row0 = base + PW + (size_t)8 * unit0;
    // block row P+1 is launched as a programmatic dependent of the diagonal
    // block's factorisation (a no-op wait for the rows below, a plain
    // launch): nothing is read before this
    asm volatile("griddepcontrol.wait;" ::: "memory");
    {
        // the factor, by asynchronous 16-byte copies (no register staging)
        const char* src = reinterpret_cast<const char*>(Lf);
        const uint32_t dst = smem_u32(sh);
        for (int f = tid; f < PANEL_FAC / 2; f += TRSM_THREADS)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * f), "l"(src + 16 * (size_t)f)
                         : "memory");
        asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const int slot = (warp >> 2) * 4 * gridDim.x + blockIdx.x * 4 + (warp & 3);
    for (int u = slot; u < units; u += TRSM_THREADS / 32 * gridDim.x) {
        const size_t row = row0 + (size_t)8 * u + fr;
        double c[16][2];
#pragma unroll
        for (int n = 0; n < 16; ++n) {
            const double2 v = ld_pair(M + row * npad + base + 8 * n + 2 * fq);
            c[n][0] = v.x;
            c[n][1] = v.y;
        }
#pragma unroll
        for (int n = 0; n < 16; ++n) {
            double x0 = 0.0, x1 = 0.0;
            const double2 w = Ws[n * 32 + lane];
            dmma884(x0, x1, c[n][0], w.x);
            dmma884(x0, x1, c[n][1], w.y);
            const int col = 8 * n + 2 * fq;
            if constexpr (sizeof(T) == 4) {
                const float o0 = (float)x0, o1 = (float)x1;
                *reinterpret_cast<float2*>(M + row * npad + base + col) = make_float2(o0, o1);
                __half2 h, l;
                f16_split(o0, pscale[0], h.x, l.x);
                f16_split(o1, pscale[0], h.y, l.y);
                *reinterpret_cast<__half2*>(reinterpret_cast<__half*>(Lhi) + row * PW + col) = h;
                *reinterpret_cast<__half2*>(reinterpret_cast<__half*>(Llo) + row * PW + col) = l;
            } else {
                st_pair(M + row * npad + base + col, x0, x1);
                st_pair(reinterpret_cast<double*>(Lhi) + row * PW + col, x0, x1);
            }
            if (n < 15) {
#pragma unroll
                for (int n2 = n + 1; n2 < 16; ++n2) {
                    const double2 b = Ls[tix(n2, n) * 32 + lane];
                    dmma884(c[n2][0], c[n2][1], -x0, b.x);
                    dmma884(c[n2][0], c[n2][1], -x1, b.y);
                }
            }
        }
    }
    asm volatile("griddepcontrol.launch_dependents;");
}

// ------------------------------------------------------- tensor-core update

struct SyrkBars {
    uint64_t full[STAGES], empty[STAGES], accfull[2], accempty[2], drain;
};

// Staging slot cc of the C update in shared memory: one 128x32 box, 128
// rows of 128 bytes with the 128-byte swizzle (16-byte chunk j of row r at
// position j ^ (r mod 8)), the layout the TMA reduce reads.
__device__ __forceinline__ float4* c_chunk(unsigned char* cbuf, int cc, int r, int j)
{
    return reinterpret_cast<float4*>(cbuf + cc * BOX_BYTES + r * 128 + ((j ^ (r & 7)) << 4));
}

__global__ void __launch_bounds__(192, 1)
k_syrk_tc(const __grid_constant__ CUtensorMap map_hi, const __grid_constant__ CUtensorMap map_lo,
          const __grid_constant__ CUtensorMap map_c, int t0, int ntiles, int mode, unsigned* __restrict__ status,
          uint32_t wlim, const float* __restrict__ pscale)
{
    {
        uint32_t dyn;
        asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
        if (blockDim.x != 192 || dyn < (uint32_t)SYRK_SMEM) {
            if (threadIdx.x == 0) atomicOr(status, ST_LAUNCH);
            return;
        }
    }
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ SyrkBars bars;
    __shared__ uint32_t tmem_base_sh;
    __shared__ volatile int abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t sbase = smem_u32(sm);
    unsigned char* cbuf = sm + STAGES * STAGE_BYTES;
    const uint32_t cbase = sbase + STAGES * STAGE_BYTES;
    if (tid == 0) {
        abort_flag = 0;
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_u32(&bars.full[s]), 1);
            mbar_init(smem_u32(&bars.empty[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&bars.accfull[b]), 1);
            mbar_init(smem_u32(&bars.accempty[b]), 4);
        }
        mbar_init(smem_u32(&bars.drain), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_sh)),
                     "r"(256));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base_sh;
    // launched as a programmatic dependent of the previous kernel on the
    // stream: the set-up above overlaps its tail; nothing below may read or
    // write what it produces before this wait (a no-op for a plain launch)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    // The side stream's update (mode 4) lets its dependent launch at once.
    // A bulk update's dependent is the next bulk update, a full grid of CTAs
    // that, launched early, would sit on every free SM in its
    // griddepcontrol.wait for as long as this launch runs, SMs the chain
    // needs meanwhile: bulk updates release it only once their last loads
    // are issued (below).
    if (mode == 4) asm volatile("griddepcontrol.launch_dependents;");

    if (warp == 0) {
        if (lane == 0) {
            // TMA producer of the four K chunks of A/B (hi and lo) per tile
            uint32_t g = 0;
            for (int t = blockIdx.x; t < ntiles && !abort_flag; t += gridDim.x) {
                int ti, tj;
                tile_of_mode(t, mode, ti, tj);
                const int ra = (t0 + ti) * PW, rb = (t0 + tj) * PW;
                for (int kc = 0; kc < NCHUNK; ++kc, ++g) {
                    const int s = g % STAGES;
                    if (!mbar_wait(smem_u32(&bars.empty[s]), ((g / STAGES) & 1) ^ 1, &abort_flag, wlim)) break;
                    const uint32_t st = sbase + s * STAGE_BYTES;
                    const uint32_t fb = smem_u32(&bars.full[s]);
                    mbar_expect_tx(fb, STAGE_BYTES);
                    tma_load_2d(st, &map_hi, kc * KCP, ra, fb);
                    tma_load_2d(st + BOX_BYTES, &map_lo, kc * KCP, ra, fb);
                    tma_load_2d(st + 2 * BOX_BYTES, &map_hi, kc * KCP, rb, fb);
                    tma_load_2d(st + 3 * BOX_BYTES, &map_lo, kc * KCP, rb, fb);
                }
            }
            if (mode != 1 && mode != 4) asm volatile("griddepcontrol.launch_dependents;");
            if (abort_flag) {
                // the loads still in flight (the last fill of each stage)
                // must land before the CTA exits
                volatile int never = 0;
                for (uint32_t j = g > (uint32_t)STAGES ? g - STAGES : 0; j < g; ++j)
                    mbar_wait(smem_u32(&bars.full[j % STAGES]), (j / STAGES) & 1, &never);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // MMA issuer
            const uint32_t idesc = idesc_f16_128x128();
            uint32_t g = 0, tl = 0;
            for (int t = blockIdx.x; t < ntiles && !abort_flag; t += gridDim.x, ++tl) {
                const uint32_t b = tl & 1;
                if (!mbar_wait(smem_u32(&bars.accempty[b]), ((tl >> 1) & 1) ^ 1, &abort_flag, wlim)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc = tmem + b * 128;
                bool ok = true;
                for (int kc = 0; kc < NCHUNK; ++kc, ++g) {
                    const int s = g % STAGES;
                    if (!mbar_wait(smem_u32(&bars.full[s]), (g / STAGES) & 1, &abort_flag, wlim)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t ah = sbase + s * STAGE_BYTES, al = ah + BOX_BYTES;
                    const uint32_t bh = ah + 2 * BOX_BYTES, bl = ah + 3 * BOX_BYTES;
#pragma unroll
                    for (int ks = 0; ks < KSTEPS; ++ks) {
                        const uint32_t off = ks * 32;   // 16 FP16 of K
                        umma_f16(acc, umma_desc_sw128(ah + off), umma_desc_sw128(bh + off), idesc,
                                 (kc | ks) ? 1u : 0u);
                        umma_f16(acc, umma_desc_sw128(ah + off), umma_desc_sw128(bl + off), idesc, 1u);
                        umma_f16(acc, umma_desc_sw128(al + off), umma_desc_sw128(bh + off), idesc, 1u);
                    }
                    umma_commit(smem_u32(&bars.empty[s]));
                }
                if (!ok) break;
                umma_commit(smem_u32(&bars.accfull[b]));
            }
            if (abort_flag) {
                // every MMA issued so far completes before the tensor
                // memory is freed: commit once more and wait for it
                volatile int never = 0;
                umma_commit(smem_u32(&bars.drain));
                mbar_wait(smem_u32(&bars.drain), 0, &never);
            }
        }
    } else {
        // epilogue warps 2..5: TMEM lane quarter = warp % 4. C is never
        // loaded: each 128x32 box of -acc goes to shared memory and a TMA
        // reduce-add applies it in L2 (C - acc and C + (-acc) are the same
        // IEEE sum). On diagonal tiles the upper triangle (D, kept intact)
        // receives -0.0, which leaves every value as it is.
        const int quarter = warp & 3;
        const int rl = 32 * quarter + lane;   // row inside the tile
        const float is2 = pscale[1];         // 1 / scale^2: the panels' FP16 scaling undone, exactly
        uint32_t tl = 0;
        for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++tl) {
            int ti, tj;
            tile_of_mode(t, mode, ti, tj);
            const bool diag = ti == tj;
            const int ra = (t0 + ti) * PW, rb = (t0 + tj) * PW;
            const uint32_t b = tl & 1;
            // a time-out or abort seen by any epilogue thread stops all of
            // them before the next barrier
            if (epi_any(!mbar_wait(smem_u32(&bars.accfull[b]), (tl >> 1) & 1, &abort_flag, wlim))) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
            for (int cc = 0; cc < PW / 32; ++cc) {
                uint32_t v[32];
                const uint32_t taddr = tmem + b * 128 + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(32 * cc);
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
                    "%13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, "
                    "%31}, [%32];"
                    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                      "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                      "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]),
                      "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]),
                      "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                    : "r"(taddr));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (cc == PW / 32 - 1) {
                    // the accumulator is free once all its columns are read
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&bars.accempty[b]));
                }
                // the reduce that last used this ring slot must have read it
                if (tid == 64) bulk_wait_read_ring();
                epi_sync();
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int c = 32 * cc + 4 * j;   // column inside the tile
                    float4 d;
                    d.x = (!diag || c <= rl) ? -is2 * __uint_as_float(v[4 * j]) : -0.0f;
                    d.y = (!diag || c + 1 <= rl) ? -is2 * __uint_as_float(v[4 * j + 1]) : -0.0f;
                    d.z = (!diag || c + 2 <= rl) ? -is2 * __uint_as_float(v[4 * j + 2]) : -0.0f;
                    d.w = (!diag || c + 3 <= rl) ? -is2 * __uint_as_float(v[4 * j + 3]) : -0.0f;
                    *c_chunk(cbuf, cc % C_BOXES, rl, j) = d;
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                epi_sync();
                if (tid == 64) {
                    tma_reduce_add_2d(&map_c, cbase + (cc % C_BOXES) * BOX_BYTES, rb + cc * KC, ra);
                    bulk_commit();
                }
            }
        }
        if (tid == 64) bulk_wait0();
    }
    if (abort_flag && tid == 0) atomicOr(status, ST_TIMEOUT);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256));
    }
}

// ------------------------------------------- 2-SM tensor-core bulk update
//
// Block columns 2 and beyond of the trailing update (mode 3, most of the
// factorisation's work) on CTA pairs: a cluster of two CTAs computes a
// 256x256 block (2x2 tiles) of -L_i L_j^T with tcgen05.mma.cta_group::2,
// M = N = 256. CTA r of the pair stages the 128 rows of tile row 2I+r (its
// half of A) and of tile column 2J+r (its half of B) in the same ring as the
// 1-SM kernel, so each SM pulls the same 64 KB per K chunk from L2 for twice
// the MMA work: the operand feed that bounds the 1-SM kernel is halved.
// CTA r's tensor memory holds its 128 rows x 256 columns of the block, two
// buffers (all 512 columns). Protocol: the leader (rank 0) owns the full
// barriers (it expects both CTAs' bytes; each CTA's loads complete on the
// leader's barrier) and the accumulator-empty barriers (both CTAs' epilogue
// warps arrive there); its single MMA thread commits stage release and
// accumulator-full to both CTAs at once. Every wait is bounded; a time-out in
// either CTA stops both. With npan = 2 the block takes the updates of two
// panels at once (K = 256: the second panel's maps continue the K loop), so
// C is read and written once for both.
__host__ __device__ constexpr uint32_t idesc_f16_256x256()
{
    return (1u << 4) | (0u << 7) | (0u << 10) | ((256u >> 3) << 17) | ((256u >> 4) << 24);
}

__device__ __forceinline__ void umma_f16_pair(uint32_t tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                              uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// arrive once on the barrier at offset `bar` of both CTAs of the pair when
// this thread's MMAs so far have completed
__device__ __forceinline__ void umma_commit_pair(uint32_t bar)
{
    asm volatile(
        "{\n\t.reg .b16 m;\n\tmov.b16 m, 3;\n\t"
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], m;\n\t}" ::"r"(
            bar)
        : "memory");
}

// shared::cluster address of `addr` (a shared::cta address of this CTA) in
// CTA `rank` of the cluster
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

__device__ __forceinline__ void cluster_sync_all()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// 2-D load into this CTA's shared memory whose completion is counted on the
// pair leader's barrier (cluster address `bar`); the data lands in this
// CTA's shared memory only
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
        "[%4];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

struct PairBars {
    uint64_t full[STAGES], empty[STAGES], accfull[2], accempty[2], drain;
};

// block t of the lower triangle of 256-wide blocks over the trailing tile
// columns c0 .. cols-1 -> tile row and column of its top-left tile
__device__ __forceinline__ void pair_block(int t, int c0, int& ti, int& tj)
{
    int bi, bj;
    tri_index(t, bi, bj);
    ti = c0 + 2 * bi;
    tj = c0 + 2 * bj;
}

__global__ void __launch_bounds__(192, 1)
k_syrk_tc2(const __grid_constant__ CUtensorMap map_hi, const __grid_constant__ CUtensorMap map_lo,
           const __grid_constant__ CUtensorMap map_hi2, const __grid_constant__ CUtensorMap map_lo2,
           const __grid_constant__ CUtensorMap map_c, int t0, int c0, int cols, int npan, unsigned* __restrict__ status,
           uint32_t wlim, const float* __restrict__ pscale)
{
    {
        uint32_t dyn, ncta;
        asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
        asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(ncta));
        if (blockDim.x != 192 || dyn < (uint32_t)SYRK_SMEM || ncta != 2 || npan < 1 || npan > 2) {
            if (threadIdx.x == 0) atomicOr(status, ST_LAUNCH);
            return;
        }
    }
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ PairBars bars;
    __shared__ uint32_t tmem_base_sh;
    __shared__ volatile int abort_flag;
    uint32_t rank, cid, ncl;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm("mov.u32 %0, %%clusterid.x;" : "=r"(cid));
    asm("mov.u32 %0, %%nclusterid.x;" : "=r"(ncl));
    const bool leader = rank == 0;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t sbase = smem_u32(sm);
    unsigned char* cbuf = sm + STAGES * STAGE_BYTES;
    const uint32_t cbase = sbase + STAGES * STAGE_BYTES;
    // the other CTA's abort flag: a time-out here stops the pair
    const uint32_t peer_abort = cluster_addr(smem_u32((const void*)&abort_flag), rank ^ 1u);
    auto stop_pair = [&]() {
        abort_flag = 1;
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(peer_abort), "r"(1) : "memory");
    };
    if (tid == 0) {
        abort_flag = 0;
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_u32(&bars.full[s]), 1);
            mbar_init(smem_u32(&bars.empty[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&bars.accfull[b]), 1);
            mbar_init(smem_u32(&bars.accempty[b]), 8);   // 4 epilogue warps x 2 CTAs
        }
        mbar_init(smem_u32(&bars.drain), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_sh)),
                     "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    // both CTAs' barriers are initialised (and their flags cleared) before
    // either signals the other's
    cluster_sync_all();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base_sh;
    // a bulk update: its dependent (the next bulk update) is released only
    // once this CTA's last loads are issued, so that its CTAs do not wait on
    // SMs the chain needs for as long as this launch runs
    asm volatile("griddepcontrol.wait;" ::: "memory");

    const int nb = (cols - c0 + 1) / 2;   // 256-wide block columns
    const int nblocks = nb * (nb + 1) / 2;
    const int nchunk = NCHUNK * npan;     // K chunks of a block
    if (warp == 0) {
        if (lane == 0) {
            // TMA producer: this CTA's half of A (tile row ti + rank) and of B
            // (tile column tj + rank); rows past the matrix read as zeros
            uint32_t g = 0;
            const uint32_t full0 = cluster_addr(smem_u32(&bars.full[0]), 0);
            for (int t = cid; t < nblocks && !abort_flag; t += ncl) {
                int ti, tj;
                pair_block(t, c0, ti, tj);
                const int ra = (t0 + ti + (int)rank) * PW, rb = (t0 + tj + (int)rank) * PW;
                bool ok = true;
                for (int kc = 0; kc < nchunk; ++kc, ++g) {
                    const int s = g % STAGES;
                    if (!mbar_wait(smem_u32(&bars.empty[s]), ((g / STAGES) & 1) ^ 1, &abort_flag, wlim)) {
                        ok = false;
                        break;
                    }
                    const uint32_t st = sbase + s * STAGE_BYTES;
                    const uint32_t fb = full0 + s * sizeof(uint64_t);
                    const CUtensorMap* mh = kc < NCHUNK ? &map_hi : &map_hi2;
                    const CUtensorMap* ml = kc < NCHUNK ? &map_lo : &map_lo2;
                    const int x = (kc % NCHUNK) * KCP;
                    if (leader) mbar_expect_tx(smem_u32(&bars.full[s]), 2 * STAGE_BYTES);
                    tma_load_2d_pair(st, mh, x, ra, fb);
                    tma_load_2d_pair(st + BOX_BYTES, ml, x, ra, fb);
                    tma_load_2d_pair(st + 2 * BOX_BYTES, mh, x, rb, fb);
                    tma_load_2d_pair(st + 3 * BOX_BYTES, ml, x, rb, fb);
                }
                if (!ok) {
                    stop_pair();
                    break;
                }
            }
            asm volatile("griddepcontrol.launch_dependents;");
            if (abort_flag && leader) {
                // the loads still in flight (the last fill of each stage, both
                // CTAs' bytes) land before the pair exits
                volatile int never = 0;
                for (uint32_t j = g > (uint32_t)STAGES ? g - STAGES : 0; j < g; ++j)
                    mbar_wait(smem_u32(&bars.full[j % STAGES]), (j / STAGES) & 1, &never);
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && leader) {
            // the pair's MMA issuer
            const uint32_t idesc = idesc_f16_256x256();
            uint32_t g = 0, tl = 0;
            for (int t = cid; t < nblocks && !abort_flag; t += ncl, ++tl) {
                const uint32_t b = tl & 1;
                if (!mbar_wait(smem_u32(&bars.accempty[b]), ((tl >> 1) & 1) ^ 1, &abort_flag, wlim)) {
                    stop_pair();
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc = tmem + b * 256;
                bool ok = true;
                for (int kc = 0; kc < nchunk; ++kc, ++g) {
                    const int s = g % STAGES;
                    if (!mbar_wait(smem_u32(&bars.full[s]), (g / STAGES) & 1, &abort_flag, wlim)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t ah = sbase + s * STAGE_BYTES, al = ah + BOX_BYTES;
                    const uint32_t bh = ah + 2 * BOX_BYTES, bl = ah + 3 * BOX_BYTES;
#pragma unroll
                    for (int ks = 0; ks < KSTEPS; ++ks) {
                        const uint32_t off = ks * 32;   // 16 FP16 of K
                        umma_f16_pair(acc, umma_desc_sw128(ah + off), umma_desc_sw128(bh + off), idesc,
                                      (kc | ks) ? 1u : 0u);
                        umma_f16_pair(acc, umma_desc_sw128(ah + off), umma_desc_sw128(bl + off), idesc, 1u);
                        umma_f16_pair(acc, umma_desc_sw128(al + off), umma_desc_sw128(bh + off), idesc, 1u);
                    }
                    umma_commit_pair(smem_u32(&bars.empty[s]));
                }
                if (!ok) {
                    stop_pair();
                    break;
                }
                umma_commit_pair(smem_u32(&bars.accfull[b]));
            }
            if (abort_flag) {
                volatile int never = 0;
                asm volatile(
                    "{\n\t.reg .b16 m;\n\tmov.b16 m, 1;\n\t"
                    "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], "
                    "m;\n\t}" ::"r"(smem_u32(&bars.drain))
                    : "memory");
                mbar_wait(smem_u32(&bars.drain), 0, &never);
            }
        }
    } else {
        // epilogue warps 2..5: this CTA's 128 rows (tile row ti + rank) of
        // the block, its two 128-column tiles in turn; tiles above the
        // diagonal or past the matrix are read from tensor memory (so that
        // the buffer's release is counted alike) but not written
        const int quarter = warp & 3;
        const int rl = 32 * quarter + lane;
        const float is2 = pscale[1];   // 1 / scale^2: the panels' FP16 scaling undone, exactly
        const uint32_t accempty0 = cluster_addr(smem_u32(&bars.accempty[0]), 0);
        uint32_t tl = 0;
        for (int t = cid; t < nblocks; t += ncl, ++tl) {
            int ti, tj;
            pair_block(t, c0, ti, tj);
            ti += (int)rank;
            const uint32_t b = tl & 1;
            if (epi_any(!mbar_wait(smem_u32(&bars.accfull[b]), (tl >> 1) & 1, &abort_flag, wlim))) {
                if (tid == 64) stop_pair();
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
                const int tjh = tj + h;
                const bool live = ti < cols && tjh <= ti;
                const bool diag = ti == tjh;
                const int ra = (t0 + ti) * PW, rb = (t0 + tjh) * PW;
#pragma unroll 1
                for (int cc = 0; cc < PW / 32; ++cc) {
                    uint32_t v[32];
                    const uint32_t taddr =
                        tmem + b * 256 + h * 128 + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(32 * cc);
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
                        "%12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, "
                        "%30, %31}, [%32];"
                        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
                          "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
                          "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]),
                          "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]),
                          "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                        : "r"(taddr));
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (h == 1 && cc == PW / 32 - 1) {
                        // the buffer is free once both CTAs have read it all
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        __syncwarp();
                        if (lane == 0)
                            asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(
                                             accempty0 + b * (uint32_t)sizeof(uint64_t))
                                         : "memory");
                    }
                    if (!live) continue;
                    if (tid == 64) bulk_wait_read_ring();
                    epi_sync();
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int c = 32 * cc + 4 * j;
                        float4 d;
                        d.x = (!diag || c <= rl) ? -is2 * __uint_as_float(v[4 * j]) : -0.0f;
                        d.y = (!diag || c + 1 <= rl) ? -is2 * __uint_as_float(v[4 * j + 1]) : -0.0f;
                        d.z = (!diag || c + 2 <= rl) ? -is2 * __uint_as_float(v[4 * j + 2]) : -0.0f;
                        d.w = (!diag || c + 3 <= rl) ? -is2 * __uint_as_float(v[4 * j + 3]) : -0.0f;
                        *c_chunk(cbuf, cc % C_BOXES, rl, j) = d;
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    epi_sync();
                    if (tid == 64) {
                        tma_reduce_add_2d(&map_c, cbase + (cc % C_BOXES) * BOX_BYTES, rb + cc * KC, ra);
                        bulk_commit();
                    }
                }
            }
        }
        if (tid == 64) bulk_wait0();
    }
    if (abort_flag && tid == 0) atomicOr(status, ST_TIMEOUT);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    // neither CTA frees its tensor memory or exits while the other may still
    // signal its barriers or (the leader's MMAs) write its tensor memory
    cluster_sync_all();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
    }
}

// ------------------------------------------------- FP64 trailing update
//
// The plain FP64 path's C -= L_i L_j^T on the FP64 tensor instruction
// (mma.sync m8n8k4 f64; tcgen05 has no FP64): a persistent CTA of 4 warps per
// 64x128 half tile, warp w owning rows 32 (w mod 2).. and columns 64 (w / 2)..
// as 32 accumulator tiles in registers, initialised from C and stored back
// (lower triangle only on diagonal tiles, whose upper triangle holds D; the
// warp that lies above the diagonal does nothing). Two CTAs fit an SM, so that
// one multiplies while the other loads or stores its C; a whole tile on 8
// warps (one CTA, 242 registers a thread) left the FP64 pipe idle meanwhile,
// and a panel of few tiles left half the SMs without one. (mean launch
// of a factorisation, n = 1536: 29.5 us before, 18.3 now; n = 6003: 51, 44.) The panel rows
// stream through shared memory in chunks of 16 columns (cp.async, two
// stages). k-step h of 8 columns takes columns 2 q + h (q = lane mod 4), so one
// 16-byte shared load feeds two k-steps. Rows padded to 24 doubles (a quarter-warp's 16-byte loads then
// hit distinct banks). Every accumulator takes its k-steps in order.
static constexpr int S64_THREADS = 128;
static constexpr int S64_ROWS = 64;                      // rows of a half tile
static constexpr int S64_KC = 16;                        // panel columns per staged chunk
static constexpr int S64_LD = 24;                        // padded row stride of a staged chunk (doubles)
static constexpr int S64_STAGE = (S64_ROWS + PW) * S64_LD;   // doubles of one stage (A and B chunks)
static constexpr int S64_SMEM = 2 * S64_STAGE * 8;       // two stages: 72 KB

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// columns [k0, k0 + 16) of panel rows ra.. (64, A) and rb.. (128, B), as stored:
// 8 16-byte pieces a row, 12 a thread
__device__ __forceinline__ void s64_stage(double* st, const double* __restrict__ Lp, int ra, int rb, int k0, int tid)
{
    constexpr int PIECES = S64_KC / 2;
#pragma unroll
    for (int q = tid; q < (S64_ROWS + PW) * PIECES; q += S64_THREADS) {
        const int r = q / PIECES, c = (q % PIECES) * 2;
        const int row = r < S64_ROWS ? ra + r : rb + r - S64_ROWS;
        cp_async16(smem_u32(st + r * S64_LD + c), Lp + (size_t)row * PW + k0 + c);
    }
}

__global__ void __launch_bounds__(S64_THREADS, 2) k_syrk64(double* __restrict__ M, int npad,
                                                         const double* __restrict__ Lp, int t0, int ntiles, int mode,
                                                         unsigned* __restrict__ status)
{
    extern __shared__ __align__(16) double sm64[];
    {
        uint32_t dyn;
        asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
        if (blockDim.x != S64_THREADS || dyn < (uint32_t)S64_SMEM) {
            if (threadIdx.x == 0) atomicOr(status, ST_LAUNCH);
            return;
        }
    }
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int fr = lane >> 2, fq = lane & 3;
    const int wr = warp & 1, wc = warp >> 1;
    // a programmatic dependent of the previous kernel on the stream: nothing
    // it produces is read before this. Dependents launch at once after the
    // side stream's update (mode 4), after a bulk
    // update only when each CTA starts its last tile (a bulk dependent
    // launched early would hold free SMs in its wait)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (mode == 4) asm volatile("griddepcontrol.launch_dependents;");
    constexpr int NCH = PW / S64_KC;
    for (int t = blockIdx.x; t < 2 * ntiles; t += gridDim.x) {
        if (t + (int)gridDim.x >= 2 * ntiles) asm volatile("griddepcontrol.launch_dependents;");
        int ti, tj;
        tile_of_mode(t >> 1, mode, ti, tj);
        const int half = t & 1;
        const int ra = (t0 + ti) * PW + S64_ROWS * half, rb = (t0 + tj) * PW;
        const bool diag = ti == tj;
        const bool work = !(diag && half == 0 && wc == 1);   // else above the diagonal
        s64_stage(sm64, Lp, ra, rb, 0, tid);
        cp_async_commit();
        double acc[4][8][2];
#pragma unroll
        for (int rt = 0; rt < 4; ++rt)
#pragma unroll
            for (int ct = 0; ct < 8; ++ct) {
                const size_t row = (size_t)ra + 32 * wr + 8 * rt + fr;
                const double2 v = work ? *reinterpret_cast<const double2*>(M + row * npad + rb + 64 * wc + 8 * ct + 2 * fq)
                                       : make_double2(0.0, 0.0);
                acc[rt][ct][0] = v.x;
                acc[rt][ct][1] = v.y;
            }
#pragma unroll 1
        for (int kc = 0; kc < NCH; ++kc) {
            const double* As = sm64 + (kc & 1) * S64_STAGE;
            const double* Bs = As + S64_ROWS * S64_LD;
            if (kc + 1 < NCH) {
                s64_stage(sm64 + ((kc + 1) & 1) * S64_STAGE, Lp, ra, rb, (kc + 1) * S64_KC, tid);
                cp_async_commit();
                cp_async_wait<1>();
            } else {
                cp_async_wait<0>();
            }
            __syncthreads();
            if (work) {
#pragma unroll
                for (int kk = 0; kk < S64_KC; kk += 8) {
                    // this lane's fragments of two k-steps
                    double2 a[4], b[8];
#pragma unroll
                    for (int rt = 0; rt < 4; ++rt) {
                        const double2 v =
                            *reinterpret_cast<const double2*>(As + (32 * wr + 8 * rt + fr) * S64_LD + kk + 2 * fq);
                        a[rt] = make_double2(-v.x, -v.y);
                    }
#pragma unroll
                    for (int ct = 0; ct < 8; ++ct)
                        b[ct] = *reinterpret_cast<const double2*>(Bs + (64 * wc + 8 * ct + fr) * S64_LD + kk + 2 * fq);
#pragma unroll
                    for (int rt = 0; rt < 4; ++rt)
#pragma unroll
                        for (int ct = 0; ct < 8; ++ct) dmma884(acc[rt][ct][0], acc[rt][ct][1], a[rt].x, b[ct].x);
#pragma unroll
                    for (int rt = 0; rt < 4; ++rt)
#pragma unroll
                        for (int ct = 0; ct < 8; ++ct) dmma884(acc[rt][ct][0], acc[rt][ct][1], a[rt].y, b[ct].y);
                }
            }
            __syncthreads();   // this stage is read; it may be staged again
        }
        if (!work) continue;
#pragma unroll
        for (int rt = 0; rt < 4; ++rt)
#pragma unroll
            for (int ct = 0; ct < 8; ++ct) {
                const int r = S64_ROWS * half + 32 * wr + 8 * rt + fr, c = 64 * wc + 8 * ct + 2 * fq;
                double* dst = M + ((size_t)ra + 32 * wr + 8 * rt + fr) * npad + rb + c;
                if (!diag) {
                    *reinterpret_cast<double2*>(dst) = make_double2(acc[rt][ct][0], acc[rt][ct][1]);
                } else {
                    if (c <= r) dst[0] = acc[rt][ct][0];
                    if (c + 1 <= r) dst[1] = acc[rt][ct][1];
                }
            }
    }
}

// The chain's update of one diagonal tile (block b, the next to be factored)
// with panel b-1, C -= L_b L_b^T, in FP64 from M's own rows (in L2: the panel
// solve has just written them), on both precisions' paths. The chain waits for
// it, so it is spread over 10 CTAs of 32x32 outputs (lower triangle), a warp
// 16x16, and its 2 x 32 panel rows are staged at once (one load latency). Bound
// by launch and that latency. FP64: on one or two SMs the FP64 pipe alone takes
// 10 us; the same bits as k_syrk64. Mixed: one tensor-core CTA set up its tensor
// memory, loaded split panels and went through all stages for one tile (a
// predictor-corrector step at 3N = 3003 took 1653 us with it, 1603 with this;
// rounded once a panel as there, its products exact).
static constexpr int SYRKD_GRID = 10, SYRKD_LD = PW + 8;   // (rows in distinct banks)
template <typename T>
static constexpr int SYRKD_SMEM = 64 * SYRKD_LD * (int)sizeof(T);
template <typename T>
__global__ void __launch_bounds__(128) k_syrk_diag(T* __restrict__ M, int npad, int b)
{
    extern __shared__ __align__(16) unsigned char syrkd_smem[];
    T* Ls = reinterpret_cast<T*>(syrkd_smem);   // [32 rows of block row bi, 32 of bj][LD]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int fr = lane >> 2, fq = lane & 3;
    int bi, bj;
    tri_index(blockIdx.x, bi, bj);
    const int rw = 16 * (warp & 1), cw = 16 * (warp >> 1);
    const int r0 = 32 * bi + rw, c0 = 32 * bj + cw;   // within the tile
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
    const size_t base = (size_t)b * PW;
    constexpr int VE = 16 / (int)sizeof(T), PIECES = PW / VE;
    for (int e = tid; e < 64 * PIECES; e += 128) {
        const int r = e / PIECES, c = VE * (e % PIECES);
        const size_t row = base + (r < 32 ? 32 * bi + r : 32 * bj + r - 32);
        cp_async16(smem_u32(Ls + r * SYRKD_LD + c), M + row * npad + base - PW + c);
    }
    cp_async_commit();
    double acc[2][2][2];
#pragma unroll
    for (int rt = 0; rt < 2; ++rt)
#pragma unroll
        for (int ct = 0; ct < 2; ++ct) {
            const double2 v = ld_pair(M + (base + r0 + 8 * rt + fr) * npad + base + c0 + 8 * ct + 2 * fq);
            acc[rt][ct][0] = v.x;
            acc[rt][ct][1] = v.y;
        }
    cp_async_wait<0>();
    __syncthreads();
    if (c0 > r0 + 15) return;   // above the diagonal
    const T* pa = Ls + (rw + fr) * SYRKD_LD + 2 * fq;
    const T* pb = Ls + (32 + cw + fr) * SYRKD_LD + 2 * fq;
#pragma unroll 4
    for (int k = 0; k < PW; k += 8) {
        double2 x[2], y[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            x[h] = ld_pair(pa + 8 * h * SYRKD_LD + k);
            y[h] = ld_pair(pb + 8 * h * SYRKD_LD + k);
        }
#pragma unroll
        for (int rt = 0; rt < 2; ++rt)
#pragma unroll
            for (int ct = 0; ct < 2; ++ct) dmma884(acc[rt][ct][0], acc[rt][ct][1], -x[rt].x, y[ct].x);
#pragma unroll
        for (int rt = 0; rt < 2; ++rt)
#pragma unroll
            for (int ct = 0; ct < 2; ++ct) dmma884(acc[rt][ct][0], acc[rt][ct][1], -x[rt].y, y[ct].y);
    }
#pragma unroll
    for (int rt = 0; rt < 2; ++rt)
#pragma unroll
        for (int ct = 0; ct < 2; ++ct) {
            const int r = r0 + 8 * rt + fr, c = c0 + 8 * ct + 2 * fq;
            T* dst = M + (base + r) * npad + base + c;
            if (c <= r) dst[0] = (T)acc[rt][ct][0];
            if (c + 1 <= r) dst[1] = (T)acc[rt][ct][1];
        }
}

// ---------------------------------------------------------------- host side

// row-major FP32 [rows][cols] buffer, boxes of 128 rows x 32 columns
// (f16: an FP16 panel buffer [rows][128], boxes of 128 rows x 64 columns;
// otherwise FP32, boxes of 128 rows x 32 columns; 128 bytes a box row)
static int make_panel_map(void* buf, int rows, CUtensorMap* map, int cols = PW, bool f16 = false)
{
    auto enc = get_encode();
    if (!enc) return fail(BDB_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
    if (reinterpret_cast<uintptr_t>(buf) % 16) return fail(BDB_ERR_ARG, "panel buffer not 16-byte aligned");
    const size_t es = f16 ? 2 : 4;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)cols * es};
    cuuint32_t box[2] = {(cuuint32_t)(f16 ? KCP : KC), PW};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(map, f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, buf, dims,
                     strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(BDB_ERR_CUDA, "cuTensorMapEncodeTiled failed");
    return BDB_OK;
}

// scratch layout in panel64: four panel buffer sets (hi, lo: FP32
// [npad][128] each; on the FP64 path one FP64 [npad][128] panel in their
// room), then four FP64 128x128 hand-offs of L_PP / W_kk; panel P uses set
// P mod 4, so a panel's updates may still read its set (and the previous
// panel's) while the next two panels are solved
static constexpr int PANEL_SETS = 4;

static void panel_ptrs(bdb_system* s, int set, float** hi, float** lo, double** lkk)
{
    const size_t pan = (size_t)s->npad * PW;
    float* base = reinterpret_cast<float*>(s->panel64.p);
    *hi = base + (size_t)set * 2 * pan;
    *lo = *hi + pan;
    *lkk = reinterpret_cast<double*>(base + (size_t)PANEL_SETS * 2 * pan) + (size_t)set * PANEL_FAC;
}

static int tc_setup(bdb_system* s)
{
    if (s->tc_map_ok) return BDB_OK;
    const size_t pan = (size_t)s->npad * PW;
    // floats of the panel sets are counted as half a double each
    if (s->panel64.alloc((size_t)PANEL_SETS * pan + (size_t)PANEL_SETS * PANEL_FAC + 64)) return BDB_ERR_NOMEM;
    BDB_CUDA(dzero(s, s->panel64.p, s->panel64.n * sizeof(double)));
    static_assert(sizeof(CUtensorMap) * (2 * PANEL_SETS + 1) <= sizeof(bdb_system::tc_map), "tensor-map storage");
    CUtensorMap* maps = reinterpret_cast<CUtensorMap*>(s->tc_map);   // hi0, lo0, ..., hi3, lo3, M
    for (int set = 0; set < PANEL_SETS; ++set) {
        float *hi, *lo;
        double* lkk;
        panel_ptrs(s, set, &hi, &lo, &lkk);
        int rc = make_panel_map(hi, s->npad, &maps[2 * set], PW, true);
        if (rc) return rc;
        rc = make_panel_map(lo, s->npad, &maps[2 * set + 1], PW, true);
        if (rc) return rc;
    }
    int rc = make_panel_map(s->M32.p, s->npad, &maps[2 * PANEL_SETS], s->npad);
    if (rc) return rc;
    BDB_CUDA(cudaFuncSetAttribute(k_syrk_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, SYRK_SMEM));
    BDB_CUDA(cudaFuncSetAttribute(k_syrk_tc2, cudaFuncAttributeMaxDynamicSharedMemorySize, SYRK_SMEM));
    if (s->pscale.alloc(2)) return BDB_ERR_NOMEM;
    BDB_CUDA(cudaFuncSetAttribute(k_potrf128<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, POTRF_SMEM));
    BDB_CUDA(cudaFuncSetAttribute(k_syrk_diag<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, SYRKD_SMEM<float>));
    BDB_CUDA(cudaFuncSetAttribute(k_trsm128<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, TRSM_SMEM));
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    s->sm_count = sms;
    s->tc_map_ok = true;
    return BDB_OK;
}

// k_syrk_tc as a programmatic dependent launch: its CTAs may start while the
// previous kernel on the stream drains and wait in griddepcontrol.wait.
static cudaError_t launch_syrk(bdb_system* s, int grid, cudaStream_t st, const CUtensorMap& hi, const CUtensorMap& lo,
                               const CUtensorMap& c, int t0, int ntiles, int mode)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(192);
    cfg.dynamicSmemBytes = SYRK_SMEM;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_syrk_tc, hi, lo, c, t0, ntiles, mode, s->status.p, (uint32_t)s->wait_limit,
                              (const float*)s->pscale.p);
}

// k_syrk_tc2 on `clusters` CTA pairs over block columns c0 .. cols-1 of
// the trailing matrix at block t0 with the updates of npan panels (the
// first in hi / lo, the second in hi2 / lo2), behind the previous kernel on
// the stream like launch_syrk
static cudaError_t launch_syrk_pair(bdb_system* s, int clusters, cudaStream_t st, const CUtensorMap& hi,
                                    const CUtensorMap& lo, const CUtensorMap& hi2, const CUtensorMap& lo2,
                                    const CUtensorMap& c, int t0, int c0, int cols, int npan)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * clusters);
    cfg.blockDim = dim3(192);
    cfg.dynamicSmemBytes = SYRK_SMEM;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = 2;
    at[1].val.clusterDim.y = 1;
    at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, k_syrk_tc2, hi, lo, hi2, lo2, c, t0, c0, cols, npan, s->status.p,
                              (uint32_t)s->wait_limit, (const float*)s->pscale.p);
}

// the chain's kernels the same way: the next diagonal tile's update, and its
// factorisation behind it
template <typename T>
static cudaError_t launch_syrk_diag(bdb_system* s, cudaStream_t st, T* M, int b)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(SYRKD_GRID);
    cfg.blockDim = dim3(128);
    cfg.dynamicSmemBytes = SYRKD_SMEM<T>;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_syrk_diag<T>, M, s->npad, b);
}

template <typename T>
static cudaError_t launch_potrf(bdb_system* s, cudaStream_t st, T* M, int P, double* lkk)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1);
    cfg.blockDim = dim3(POTRF_THREADS);
    cfg.dynamicSmemBytes = POTRF_SMEM;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_potrf128<T>, M, s->npad, P, lkk, s->status.p, (uint32_t)s->wait_limit);
}

// block row P+1 of panel P's solve (k_trsm128, units 0..15 on 4 CTAs) as a
// programmatic dependent of the diagonal block's factorisation, so that its
// launch overlaps that kernel's tail
template <typename T>
static cudaError_t launch_trsm_top(bdb_system* s, cudaStream_t st, T* M, int P, int units, const double* lkk,
                                   float* hi, float* lo, const float* pscale)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(units / 4);
    cfg.blockDim = dim3(TRSM_THREADS);
    cfg.dynamicSmemBytes = TRSM_SMEM;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_trsm128<T>, M, s->npad, P, 0, units, lkk, hi, lo, s->status.p, pscale);
}

// The factorisation schedule, on three streams. Panel P's trailing update
// is split four ways: the diagonal tile of block column P+1 (A0), the rest
// of that column (A1), block column P+2 (B) and block columns P+3 on (C);
// its panel solve two ways: block row P+1 (top) and the rows below (rest).
//   chain stream: top(P) -> A0(P) -> diagonal block P+1 -> top(P+1) -> ...
//   side stream:  rest(P) -> A1(P) -> rest(P+1) -> ...
//   bulk stream:  B(P) -> C(P) -> B(P+1) -> C(P+1) -> ...
// So the diagonal block P+1 waits only for one panel-solve block row and
// one tile update, while the rest of panel P's solve and of its column
// update run beside it; the bulk updates of panel P run beside the next two
// steps of the chain. Hand-offs:
//   rest(P) after the diagonal block P; top(P) after A1(P-1) and B(P-1)
//   (both update block column P or P+1 before panel P's updates do);
//   A1(P) after top(P) (its B operand rows) and B(P-1); B(P) once the whole
//   panel is solved.
// The mixed path (T = float) pairs the panels for C: an even panel P
// updates block column P+3 alone, and the odd panel P+1 applies both
// panels' updates to block columns P+4 on in one K = 256 pass on CTA pairs,
// which halves the reads and writes of C, the bulk's largest cost. Every tile
// receives the same updates in the same order whatever the GPU split (the
// same bits for every chain_sms). Four panel-buffer sets let C(P) read
// panels P-1 and P while panels P+1 and P+2 are solved. The persistent bulk
// updates leave s->chain_sms SMs to the chain and side kernels (tuned).
template <typename T, typename Update>
static int factor_schedule(bdb_system* s, T* M, Update update)
{
    const int nt = s->npad / PW;
    cudaStream_t st = s->stream, st2 = s->stream2, st3 = s->stream3;
    cudaEvent_t ev_potrf = s->la_ev[0], ev_top = s->la_ev[1], ev_rest = s->la_ev[2], ev_side = s->la_ev[3],
                ev_b = s->la_ev[4], ev_end = s->la_ev[5];
    const int chain = std::min(std::max(s->chain_sms, 1), s->sm_count - 1);
    const int bulk_sms = std::max(1, s->sm_count - chain);
    const int per_cta = TRSM_THREADS / 32, units_top = PW / 8;
    // the side kernels take the chain's SMs but five: the diagonal block and
    // the four CTAs of the top panel solve. k_syrk_diag runs between those two,
    // when their five SMs are free, and its small CTAs (128 threads, 35 KB; 70
    // in FP64) also fit beside the side kernels'. The panel solve two CTAs per SM
    // (its registers and shared memory allow it), for more warps on the FP64
    // pipes
    const int side = std::max(1, chain - 5);
    constexpr bool kPairs = sizeof(T) == 4;   // two panels per pass over C (mixed path)
    const float* pscale = sizeof(T) == 4 ? s->pscale.p : nullptr;   // FP16 panel scale (mixed path)
    float *hi, *lo;
    double* lkk;
    panel_ptrs(s, 0, &hi, &lo, &lkk);
    phase_mark_on(s, P_POTRF, st);
    BDB_CUDA(launch_potrf(s, st, M, 0, lkk));
    phase_mark_on(s, P_POTRF, st);
    s->launches += 1;
    if (nt > 1) {
        BDB_CUDA(cudaEventRecord(ev_potrf, st));
        BDB_CUDA(cudaStreamWaitEvent(st2, ev_potrf, 0));   // the bulk stream starts after what came before
    }
    for (int P = 0; P + 1 < nt; ++P) {
        const int set = P % PANEL_SETS;
        panel_ptrs(s, set, &hi, &lo, &lkk);
        const int rem = nt - P - 1;   // trailing block columns
        const int units_rest = (rem - 1) * PW / 8;
        // side: the panel solve below block row P+1
        BDB_CUDA(cudaStreamWaitEvent(st3, ev_potrf, 0));
        if (units_rest > 0) {
            k_trsm128<T><<<std::min(2 * side, (units_rest + per_cta - 1) / per_cta), TRSM_THREADS, TRSM_SMEM, st3>>>(
                M, s->npad, P, units_top, units_rest, lkk, hi, lo, s->status.p, pscale);
            BDB_CUDA(cudaGetLastError());
            s->launches += 1;
        }
        BDB_CUDA(cudaEventRecord(ev_rest, st3));
        // chain: block row P+1 of the panel solve
        if (P > 0) {
            BDB_CUDA(cudaStreamWaitEvent(st, ev_side, 0));   // A1(P-1)
            BDB_CUDA(cudaStreamWaitEvent(st, ev_b, 0));      // B(P-1)
        }
        phase_mark_on(s, P_TRSM, st);
        // block row P+1: its 16 units on 4 CTAs, so that each unit's warp
        // has an SM sub-partition (and its FP64 pipe) to itself
        BDB_CUDA(launch_trsm_top(s, st, M, P, units_top, lkk, hi, lo, pscale));
        phase_mark_on(s, P_TRSM, st);
        BDB_CUDA(cudaEventRecord(ev_top, st));
        // side: block column P+1 below its diagonal tile
        BDB_CUDA(cudaStreamWaitEvent(st3, ev_top, 0));
        if (P > 0) BDB_CUDA(cudaStreamWaitEvent(st3, ev_b, 0));   // B(P-1)
        if (rem > 1) {
            BDB_CUDA(update(st3, kPairs ? std::min(rem - 1, side) : side, set, -1, P + 1, rem - 1, 4));
            s->launches += 1;
        }
        BDB_CUDA(cudaEventRecord(ev_side, st3));
        // bulk: block column P+2, then the rest
        BDB_CUDA(cudaStreamWaitEvent(st2, ev_top, 0));
        BDB_CUDA(cudaStreamWaitEvent(st2, ev_rest, 0));
        phase_mark_on(s, P_SYRK_REST, st2);
        if (rem >= 2) {
            BDB_CUDA(update(st2, kPairs ? std::min(bulk_sms, rem - 1) : bulk_sms, set, -1, P + 1, rem - 1, 2));
            s->launches += 1;
        }
        BDB_CUDA(cudaEventRecord(ev_b, st2));
        if (rem >= 3) {
            if (kPairs && P % 2 == 0) {
                // block column P+3 alone; the columns beyond take this
                // panel's update together with panel P+1's
                BDB_CUDA(update(st2, std::min(bulk_sms, rem - 2), set, -1, P + 1, rem - 2, 5));
            } else {
                // block columns P+3 on: panel P, and on the mixed path panel
                // P-1 (deferred there) in the same pass
                const int ntc = (rem - 2) * (rem - 1) / 2;
                const int set_prev = kPairs ? (P - 1) % PANEL_SETS : -1;
                BDB_CUDA(update(st2, kPairs ? std::min(bulk_sms, ntc) : bulk_sms, set, set_prev, P + 1, ntc, 3));
            }
            s->launches += 1;
        }
        phase_mark_on(s, P_SYRK_REST, st2);
        // chain: the diagonal tile of block column P+1, then its factorisation
        phase_mark_on(s, P_SYRK_COL, st);
        BDB_CUDA(launch_syrk_diag(s, st, M, P + 1));
        phase_mark_on(s, P_SYRK_COL, st);
        double* lkk1;
        float *hi1, *lo1;
        panel_ptrs(s, (P + 1) % PANEL_SETS, &hi1, &lo1, &lkk1);
        phase_mark_on(s, P_POTRF, st);
        BDB_CUDA(launch_potrf(s, st, M, P + 1, lkk1));
        phase_mark_on(s, P_POTRF, st);
        BDB_CUDA(cudaEventRecord(ev_potrf, st));
        s->launches += 3;
    }
    // join the side and bulk streams (a single panel has not used them: in a
    // capture the side stream would not belong to it)
    if (nt == 1) return BDB_OK;
    BDB_CUDA(cudaEventRecord(ev_side, st3));
    BDB_CUDA(cudaStreamWaitEvent(st, ev_side, 0));
    BDB_CUDA(cudaEventRecord(ev_end, st2));
    BDB_CUDA(cudaStreamWaitEvent(st, ev_end, 0));
    BDB_CUDA(cudaGetLastError());
    return BDB_OK;
}

// The FP16 panel scale of a factorisation, from D's diagonal (dD): 2^e with
// the largest sqrt(D_ii) -- a bound of every |L_ij| -- just below 2^14;
// pscale[0] = 2^e, pscale[1] = 2^-2e. One CTA.
__global__ void k_panel_scale(const double* __restrict__ dD, int n3, float* __restrict__ pscale)
{
    __shared__ double red[32];
    double m = 0.0;
    for (int i = threadIdx.x; i < n3; i += blockDim.x) m = fmax(m, dD[i]);
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = fmax(m, red[w]);
        int e = 0, sh = 0;
        if (m > 0.0 && isfinite(m)) {
            frexp(sqrt(m), &e);   // sqrt(m) < 2^e
            sh = 14 - e;
        }
        sh = max(-60, min(60, sh));
        pscale[0] = ldexpf(1.0f, sh);
        pscale[1] = ldexpf(1.0f, -2 * sh);
    }
}

int factor_mixed_tc(bdb_system* s)
{
    int rc = tc_setup(s);
    if (rc) return rc;
    k_panel_scale<<<1, 1024, 0, s->stream>>>(s->dD.p, s->n3, s->pscale.p);
    BDB_CUDA(cudaGetLastError());
    s->launches += 1;
    const CUtensorMap* maps = reinterpret_cast<const CUtensorMap*>(s->tc_map);
    const int nt = s->npad / PW;
    return factor_schedule(s, s->M32.p, [&](cudaStream_t stream, int grid, int set, int set_prev, int t0, int ntiles,
                                            int mode) {
        if (mode == 3) {
            // block columns 2.. of the trailing matrix: 256-wide blocks on
            // CTA pairs, with the previous panel's update too if it is given
            const int cols = nt - t0, nb = (cols - 1) / 2;
            const int clusters = std::max(1, std::min(grid / 2, nb * (nb + 1) / 2));
            const int first = set_prev >= 0 ? set_prev : set;
            return launch_syrk_pair(s, clusters, stream, maps[2 * first], maps[2 * first + 1], maps[2 * set],
                                    maps[2 * set + 1], maps[2 * PANEL_SETS], t0, 2, cols, set_prev >= 0 ? 2 : 1);
        }
        return launch_syrk(s, grid, stream, maps[2 * set], maps[2 * set + 1], maps[2 * PANEL_SETS], t0, ntiles, mode);
    });
}

// ------------------------------------------------------ FP64 factorisation

static int tc64_setup(bdb_system* s)
{
    if (s->tc64_ok) return BDB_OK;
    const size_t pan = (size_t)s->npad * PW;
    // one FP64 panel buffer per set (the room of a mixed-path hi/lo pair)
    if (s->panel64.alloc((size_t)PANEL_SETS * pan + (size_t)PANEL_SETS * PANEL_FAC + 64)) return BDB_ERR_NOMEM;
    BDB_CUDA(dzero(s, s->panel64.p, s->panel64.n * sizeof(double)));
    BDB_CUDA(cudaFuncSetAttribute(k_potrf128<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, POTRF_SMEM));
    BDB_CUDA(cudaFuncSetAttribute(k_syrk_diag<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, SYRKD_SMEM<double>));
    BDB_CUDA(cudaFuncSetAttribute(k_trsm128<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, TRSM_SMEM));
    BDB_CUDA(cudaFuncSetAttribute(k_syrk64, cudaFuncAttributeMaxDynamicSharedMemorySize, S64_SMEM));
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    s->sm_count = sms;
    s->tc64_ok = true;
    return BDB_OK;
}

// grid: SMs the update may take
static cudaError_t launch_syrk64(bdb_system* s, int grid, cudaStream_t st, const double* Lp, int t0, int ntiles,
                                 int mode)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(std::min(2 * grid, 2 * ntiles));
    cfg.blockDim = dim3(S64_THREADS);
    cfg.dynamicSmemBytes = S64_SMEM;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_syrk64, s->M64.p, s->npad, Lp, t0, ntiles, mode, s->status.p);
}

// The plain FP64 path: the same schedule with FP64 panels and FP64 DMMA
// trailing updates
int factor_fp64_tc(bdb_system* s)
{
    int rc = tc64_setup(s);
    if (rc) return rc;
    return factor_schedule(s, s->M64.p, [&](cudaStream_t stream, int grid, int set, int, int t0, int ntiles,
                                            int mode) {
        float *hi, *lo;
        double* lkk;
        panel_ptrs(s, set, &hi, &lo, &lkk);
        return launch_syrk64(s, grid, stream, reinterpret_cast<const double*>(hi), t0, ntiles, mode);
    });
}

}  // namespace bdb
