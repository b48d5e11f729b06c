// Matrix-free D.F (compute_Rf_geyer_in_fly, diff_equation.c:55-117) and the
// Geyer-Winter noise of the same tensor (compute_r DIFF_GEYER,
// diff_rand.c:86-230).
//
// 1. k_tea_pairs: every bead pair once. Beads are cut into tiles of 32; a job
//    is a warp's share of the pairs of a row tile I with a run of column
//    tiles J <= I. Lane l keeps row bead l (position, F, X and its sums) in
//    registers and walks the 32 columns rotated by its lane: at step s it
//    meets column (l + s) mod 32, whose sums travel with it -- after every
//    step each lane hands its column sums to the lane that meets that column
//    next. So both sides of a pair are summed in registers, at 9 shuffles per
//    step, with no reduction across lanes and no barrier.
// 2. k_tea_finish: one CTA per bead tile adds the tile's records in a fixed
//    order, forms eps and beta of its segment (diff_rand.c:197-217) from the
//    jobs' partials, and writes Rf and Rs.
// Bound by instruction issue: per pair the tile (~30), two sets of products
// (~60) and a ninth of the hand-over each, ~150 in all in FP32; in FP64 by the
// FP64 pipe. One row sum per lane over 5 exchanges of 9 values per pair, as a
// warp holding rows of a tile needs, took more than the tile itself: N = 3000
// in FP64 124 -> 50 us, the 256-replica batch 748 -> 342 us per step (319 with
// FP32 sums over whole tiles, single FP32 records and eps in FP32, which lost
// precision against that form).
// Which warp runs a job does not change a bit: each job writes records of its
// own, and they are added in the order of the job list.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "bdb_common.cuh"
#include "ewald_fast.cuh"
#include "tensor_args.cuh"

namespace bdb {

static constexpr int TT = 32;            // beads per tile
static constexpr int TEA_WARPS = 4;      // independent warps (jobs) per CTA
static constexpr int REC = 9 * TT;       // values of one record: [9][32]
static constexpr int CHUNK = 8;          // steps of an FP32 partial sum
// the sums of a bead: D F (3), then C (3) and D X (3)
enum { JOB_ROWS1 = 0, JOB_DIAG = 1, JOB_ROWS2 = 2 };
// tiles: free space; the reference's lattice sums; their converged split
enum { TILE_FREE = 0, TILE_EWALD = 1, TILE_FAST = 2 };
template <int KIND>
using FastArg = typename std::conditional<KIND == TILE_FAST, EwaldFast, NoFast>::type;

struct TeaSeg {
    int begin, count, tile0, ntile, job0, job1;
};

// records of a bead tile: row records first, then column records
struct TeaTile {
    int rec0, nslot, seg, pad;
};

// T-typed bead data of the column tile, one 16-byte vector load per group
template <typename T>
struct ColData;
template <>
struct ColData<float> {
    float4 hi_w[TT], lo_inv[TT], f_x0[TT];   // position (hi), radius; position (lo), 1/D_jj; F, X_0
    float2 x12[TT];                          // X_1, X_2
};
template <>
struct ColData<double> {
    double2 xy[TT], zw[TT], f01[TT], f2_inv[TT], x01[TT];
    double x2[TT];
};

template <typename T>
struct Bead {
    T x[3], lo[3], w, inv, f[3], g[3];   // position (FP32: relative to the job's origin, hi + lo), radius, 1/D, F, X
};

// Positions in FP32 pairs: the length unit and the step of hi's grid (a power
// of two)
struct PairUnits {
    double unit, step, inv_step;
};

// A bead's position relative to the job's origin as the FP32 pair hi + lo, so
// that the difference of two beads needs no FP64 subtractions and conversions
// per pair. hi is a multiple of `step` below 2^23 steps: the difference of two
// is then exact, and with lo's (below a step, rounded 2^-24 of that) the
// separation is the FP64 difference rounded to FP32 once. Farther out hi is
// the FP32 value, and the difference rounds twice.
template <typename T, bool RS>
__device__ __forceinline__ void load_bead(Bead<T>& b, const TensorArgs& A, const double4* __restrict__ pos,
                                          const double* __restrict__ F, const double* __restrict__ X, int i, bool ok,
                                          const double4& org, const PairUnits& u)
{
    const double4 p = pos[i];
    if constexpr (sizeof(T) == 4) {
        const double d[3] = {(p.x - org.x) * u.unit, (p.y - org.y) * u.unit, (p.z - org.z) * u.unit};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const double q = rint(d[k] * u.inv_step);
            b.x[k] = fabs(q) < 8388608.0 ? (float)(q * u.step) : (float)d[k];
            b.lo[k] = (float)(d[k] - (double)b.x[k]);
        }
    } else {
        b.x[0] = p.x;
        b.x[1] = p.y;
        b.x[2] = p.z;
    }
    b.w = (T)p.w;
    b.inv = ok ? (T)(p.w / A.preDii) : (T)0;   // 1/diag_D (diff_decl.c:94-99)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        b.f[k] = ok ? (T)F[3 * i + k] : (T)0;
        b.g[k] = RS && ok ? (T)X[3 * i + k] : (T)0;
    }
}

template <bool RS>
__device__ __forceinline__ void put_col(ColData<float>& s, int l, const Bead<float>& b)
{
    s.hi_w[l] = make_float4(b.x[0], b.x[1], b.x[2], b.w);
    s.lo_inv[l] = make_float4(b.lo[0], b.lo[1], b.lo[2], b.inv);
    s.f_x0[l] = make_float4(b.f[0], b.f[1], b.f[2], b.g[0]);
    if (RS) s.x12[l] = make_float2(b.g[1], b.g[2]);
}
template <bool RS>
__device__ __forceinline__ void get_col(const ColData<float>& s, int l, Bead<float>& b)
{
    const float4 a = s.hi_w[l], c = s.lo_inv[l], d = s.f_x0[l];
    b.x[0] = a.x;
    b.x[1] = a.y;
    b.x[2] = a.z;
    b.w = a.w;
    b.lo[0] = c.x;
    b.lo[1] = c.y;
    b.lo[2] = c.z;
    b.inv = c.w;
    b.f[0] = d.x;
    b.f[1] = d.y;
    b.f[2] = d.z;
    b.g[0] = d.w;
    if (RS) {
        const float2 e = s.x12[l];
        b.g[1] = e.x;
        b.g[2] = e.y;
    }
}
template <bool RS>
__device__ __forceinline__ void put_col(ColData<double>& s, int l, const Bead<double>& b)
{
    s.xy[l] = make_double2(b.x[0], b.x[1]);
    s.zw[l] = make_double2(b.x[2], b.w);
    s.f01[l] = make_double2(b.f[0], b.f[1]);
    s.f2_inv[l] = make_double2(b.f[2], b.inv);
    if (RS) {
        s.x01[l] = make_double2(b.g[0], b.g[1]);
        s.x2[l] = b.g[2];
    }
}
template <bool RS>
__device__ __forceinline__ void get_col(const ColData<double>& s, int l, Bead<double>& b)
{
    const double2 a = s.xy[l], c = s.zw[l], d = s.f01[l], e = s.f2_inv[l];
    b.x[0] = a.x;
    b.x[1] = a.y;
    b.x[2] = c.x;
    b.w = c.y;
    b.f[0] = d.x;
    b.f[1] = d.y;
    b.f[2] = e.x;
    b.inv = e.y;
    if (RS) {
        const double2 h = s.x01[l];
        b.g[0] = h.x;
        b.g[1] = h.y;
        b.g[2] = s.x2[l];
    }
}

// products of a tile with its bead b: D F, and with RS the squared rows of D
// over D_bb (q) and D X; on top of v (first: of nothing)
template <typename T, bool RS>
__device__ __forceinline__ void products(const T* t, const T* q, const Bead<T>& b, T* v, bool first)
{
    const T m[3][3] = {{t[0], t[3], t[4]}, {t[3], t[1], t[5]}, {t[4], t[5], t[2]}};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        v[k] = (first ? m[k][0] * b.f[0] : v[k] + m[k][0] * b.f[0]) + m[k][1] * b.f[1] + m[k][2] * b.f[2];
        if (RS) {
            v[3 + k] = first ? q[k] * b.inv : v[3 + k] + q[k] * b.inv;
            v[6 + k] = (first ? m[k][0] * b.g[0] : v[6 + k] + m[k][0] * b.g[0]) + m[k][1] * b.g[1] + m[k][2] * b.g[2];
        }
    }
}

// pairs the converged split does not cover
__device__ __noinline__ void ewald_pair(const TensorArgs& A, const double4* __restrict__ pos, int i, int j, float* t)
{
    tile_of_k<float, true>(A, pos, i, j, t);
}

// The tile of row bead a (index i) with column bead b (j). Free space: from
// the separation in T. Lattice sums: from the positions. Converged split: from
// the separation in L; pairs of other radii, overlapping ones, those so far
// apart in the box that the reference's sphere truncates (7.5e-5 of them at
// R = 4) and those outside the box (positions set by a caller) take the
// lattice sums.
template <typename T, int KIND>
__device__ __forceinline__ void pair_tile(const TensorArgs& A, const FastArg<KIND>& E, const double4* __restrict__ pos,
                                          const Bead<T>& a, const Bead<T>& b, int i, int j, T* t)
{
    if constexpr (KIND == TILE_EWALD) {
        tile_of_k<T, true>(A, pos, i, j, t);
        return;
    } else {
        T d[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            d[k] = a.x[k] - b.x[k];
            if constexpr (sizeof(T) == 4) d[k] += a.lo[k] - b.lo[k];
        }
        if constexpr (KIND == TILE_FAST) {
            const float far = fmaxf(fabsf(d[0]), fmaxf(fabsf(d[1]), fabsf(d[2])));
            const float dd = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
            if (a.w == E.radius && b.w == E.radius && far < 1.0001f && dd >= E.near_sq && dd <= E.far_sq)
                ewald_fast_tile(E, d, t);
            else
                ewald_pair(A, pos, i, j, t);
        } else {
            rpy_free_sep<T>(d, a.w, b.w, (T)A.preDii, (T)A.preDij, t);
        }
    }
}

// Steps s0 .. s1-1 of NR row tiles (bead i0 + 32 r per lane) against the
// column tile at bead j0; column sums are left with the lane that would meet
// the column at step s1. diag: the tile with itself, steps 1 .. 16 (at step
// 16 only half of the lanes, so that every pair is met once).
template <typename T, int KIND, bool RS, int NR>
__device__ __forceinline__ void tea_steps(const TensorArgs& A, const FastArg<KIND>& E,
                                          const double4* __restrict__ pos, const ColData<T>& cols,
                                          const Bead<T> (&row)[NR], int i0, int ni, int j0, int nj, int s0, int s1,
                                          bool diag, T (&racc)[NR][RS ? 9 : 3], T (&cacc)[RS ? 9 : 3], T& eps)
{
    constexpr int NV = RS ? 9 : 3;
    const int lane = threadIdx.x & 31;
    const bool edge = ni < TT * NR || nj < TT;
#pragma unroll 1
    for (int s = s0; s < s1; ++s) {
        const int c = (lane + s) & 31;
        Bead<T> b;
        get_col<RS>(cols, c, b);
        T cv[NV];   // the rows' products with this column, joined before they meet its larger sum
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const bool off = (edge && (c >= nj || lane + TT * r >= ni)) || (diag && s == TT / 2 && lane >= TT / 2);
            T t[6] = {0, 0, 0, 0, 0, 0};
            if (KIND == TILE_FREE || !off) pair_tile<T, KIND>(A, E, pos, row[r], b, i0 + TT * r + lane, j0 + c, t);
            if (off)
#pragma unroll
                for (int k = 0; k < 6; ++k) t[k] = 0;
            T q[3];
            if (RS) {
                q[0] = t[0] * t[0] + t[3] * t[3] + t[4] * t[4];
                q[1] = t[3] * t[3] + t[1] * t[1] + t[5] * t[5];
                q[2] = t[4] * t[4] + t[5] * t[5] + t[2] * t[2];
                eps += (t[0] + t[1] + t[2]) + 2 * (t[3] + t[4] + t[5]);
            }
            T v[NV];
            products<T, RS>(t, q, b, v, true);
#pragma unroll
            for (int k = 0; k < NV; ++k) racc[r][k] += v[k];
            products<T, RS>(t, q, row[r], cv, r == 0);
        }
#pragma unroll
        for (int k = 0; k < NV; ++k) cacc[k] += cv[k];
#pragma unroll
        for (int k = 0; k < NV; ++k) cacc[k] = __shfl_sync(0xffffffffu, cacc[k], (lane + 1) & 31);
    }
}

// One warp per job. Records are written in T: in FP32 a record holds one tile's
// sums; the row sums of a job with several column tiles take two.
template <typename T, int KIND, bool RS>
__global__ void __launch_bounds__(32 * TEA_WARPS, sizeof(T) == 4 && KIND == TILE_FREE ? 4 : 3)
k_tea_pairs(const __grid_constant__ TensorArgs A, const __grid_constant__ FastArg<KIND> E,
            const TileJob* __restrict__ jobs, int n_jobs, const int* __restrict__ col_rec,
            const TeaSeg* __restrict__ segs, const double4* __restrict__ pos, const double* __restrict__ F,
            const double* __restrict__ X, T* __restrict__ part, double* __restrict__ eps_part, const PairUnits units)
{
    constexpr int NV = RS ? 9 : 3;
    constexpr int MAXR = sizeof(T) == 4 && KIND == TILE_FREE ? 2 : 1;   // row tiles a job may hold
    __shared__ ColData<T> s_col[TEA_WARPS];
    __shared__ double s_sum[TEA_WARPS][sizeof(T) == 4 ? NV : 1][TT];
    __shared__ double s_row[TEA_WARPS][sizeof(T) == 4 ? MAXR * NV : 1][TT];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int job = blockIdx.x * TEA_WARPS + warp;
    if (job >= n_jobs) return;
    const TileJob jb = jobs[job];
    const TeaSeg sg = segs[jb.seg];
    ColData<T>& cols = s_col[warp];
    const int end = sg.begin + sg.count;
    const int i0 = sg.begin + TT * jb.I, ni = end - i0;
    const double4 org = pos[i0];
    const bool one = jb.nJ == 1 && jb.s1 - jb.s0 <= CHUNK;   // FP32: a single chunk
    double eps = 0;   // FP32: a chunk's sum at a time (at most 16 pairs a lane)
    Bead<T> b;

    auto columns = [&](int J) {
        const int j0 = sg.begin + TT * J, j = j0 + lane;
        load_bead<T, RS>(b, A, pos, F, X, min(j, end - 1), j < end, org, units);
        __syncwarp();
        put_col<RS>(cols, lane, b);
        __syncwarp();
    };
    auto put_record = [&](int rec, int l, const T* v) {
        T* o = part + (size_t)rec * REC + l;
#pragma unroll
        for (int k = 0; k < NV; ++k) o[TT * k] = v[k];
    };
    auto rows = [&](auto nr_c) {
        constexpr int NR = decltype(nr_c)::value;
        Bead<T> row[NR];
        T racc[NR][NV];
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const int i = i0 + TT * r + lane;
            load_bead<T, RS>(row[r], A, pos, F, X, min(i, end - 1), i < end, org, units);
#pragma unroll
            for (int k = 0; k < NV; ++k) racc[r][k] = 0;
        }
        for (int q = 0; q < jb.nJ; ++q) {
            const int J = jb.J0 + q, j0 = sg.begin + TT * J;
            T cacc[NV];
#pragma unroll
            for (int k = 0; k < NV; ++k) cacc[k] = 0;
            columns(J);
            if constexpr (sizeof(T) == 8) {
                tea_steps<T, KIND, RS, NR>(A, E, pos, cols, row, i0, ni, j0, end - j0, jb.s0, jb.s1,
                                           jb.type == JOB_DIAG, racc, cacc, eps);
            } else {
                // FP32 sums of 8 steps at a time, the chunks' sums in FP64, in
                // shared memory at the bead's own slot (the column's at its
                // number): rows over the whole job, columns over the tile. A
                // job of one chunk keeps its sums in registers (N = 1000:
                // 43.0 -> 41.1 us a step).
                for (int s = jb.s0; s < jb.s1; s += CHUNK) {
                    const int e = min(s + CHUNK, jb.s1), l = (lane + e) & 31;
                    T eps_c = 0;
#pragma unroll
                    for (int k = 0; k < NV; ++k) {
                        cacc[k] = 0;
#pragma unroll
                        for (int r = 0; r < NR; ++r) racc[r][k] = 0;
                    }
                    tea_steps<T, KIND, RS, NR>(A, E, pos, cols, row, i0, ni, j0, end - j0, s, e, jb.type == JOB_DIAG,
                                               racc, cacc, eps_c);
                    eps += (double)eps_c;
                    if (one) break;
                    __syncwarp();   // lanes take turns at a column's slot
#pragma unroll
                    for (int k = 0; k < NV; ++k) {
                        double* o = &s_sum[warp][k][l];
                        *o = s == jb.s0 ? (double)cacc[k] : *o + (double)cacc[k];
#pragma unroll
                        for (int r = 0; r < NR; ++r) {
                            double* p = &s_row[warp][NV * r + k][lane];
                            *p = q == 0 && s == jb.s0 ? (double)racc[r][k] : *p + (double)racc[r][k];
                        }
                    }
                }
                if (!one) {
                    __syncwarp();
#pragma unroll
                    for (int k = 0; k < NV; ++k) cacc[k] = (T)s_sum[warp][k][(lane + jb.s1) & 31];
                    __syncwarp();
                }
            }
            if (jb.type == JOB_DIAG) {
                // row and column sums of the same beads: one record in FP64,
                // one each in FP32, where joining them would round again
                if constexpr (sizeof(T) == 8) {
#pragma unroll
                    for (int k = 0; k < NV; ++k) racc[0][k] += __shfl_sync(0xffffffffu, cacc[k], (lane - jb.s1) & 31);
                } else {
                    put_record(jb.rec0 + 1, (lane + jb.s1) & 31, cacc);
                }
            } else {
                put_record(col_rec[jb.col0 + q], (lane + jb.s1) & 31, cacc);
            }
        }
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const int rec = r ? jb.rec1 : jb.rec0;
            if (sizeof(T) == 4 && !one) {
                // the FP64 sum over several tiles goes out as two FP32
                // records, its FP32 value and what that leaves
                T lo[NV];
#pragma unroll
                for (int k = 0; k < NV; ++k) {
                    const double v = s_row[warp][sizeof(T) == 4 ? NV * r + k : 0][lane];
                    racc[r][k] = (T)v;
                    lo[k] = (T)(v - (double)racc[r][k]);
                }
                if (jb.nJ > 1) put_record(rec + 1, lane, lo);
            }
            put_record(rec, lane, racc[r]);
        }
    };
    if constexpr (MAXR == 2) {
        if (jb.type == JOB_ROWS2) rows(std::integral_constant<int, 2>{});
        else rows(std::integral_constant<int, 1>{});
    } else {
        rows(std::integral_constant<int, 1>{});
    }
    if (RS) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) eps += __shfl_xor_sync(0xffffffffu, eps, o);
        if (lane == 0) eps_part[job] = eps;
    }
}

// One CTA per bead tile and NK coordinates (all three, or one each where
// few tiles would leave SMs idle): warp w adds records w, w + 8, ... of the
// tile (lane = bead, coalesced), the warps' sums are added in order.
static constexpr int FIN_WARPS = 8;

template <typename T, bool RS, int NK>
__global__ void __launch_bounds__(32 * FIN_WARPS)
k_tea_finish(TensorArgs A, const TeaSeg* __restrict__ segs, const TeaTile* __restrict__ tiles,
             const T* __restrict__ part, const double* __restrict__ eps_part, const double4* __restrict__ pos,
             const double* __restrict__ F, const double* __restrict__ X, double pre_f, double* __restrict__ Rf,
             double* __restrict__ Rs)
{
    constexpr int NG = RS ? 3 : 1;   // sums of a coordinate: D F, C, D X
    __shared__ double sh[FIN_WARPS][NG * NK][TT];
    __shared__ double se[FIN_WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, k0 = blockIdx.y;
    const TeaTile tl = tiles[blockIdx.x];
    const TeaSeg sg = segs[tl.seg];
    double acc[NG][NK];
#pragma unroll
    for (int g = 0; g < NG; ++g)
#pragma unroll
        for (int c = 0; c < NK; ++c) acc[g][c] = 0;
    const T* src = part + (size_t)tl.rec0 * REC + TT * k0 + lane;
#pragma unroll(NK == 1 ? 4 : 2)
    for (int u = warp; u < tl.nslot; u += FIN_WARPS)
#pragma unroll
        for (int g = 0; g < NG; ++g)
#pragma unroll
            for (int c = 0; c < NK; ++c) acc[g][c] += (double)src[(size_t)u * REC + TT * (3 * g + c)];
#pragma unroll
    for (int g = 0; g < NG; ++g)
#pragma unroll
        for (int c = 0; c < NK; ++c) sh[warp][g * NK + c][lane] = acc[g][c];
    if (RS) {
        // eps of the segment: the same sum in every CTA of it
        double e = 0;
        for (int q = sg.job0 + threadIdx.x; q < sg.job1; q += 32 * FIN_WARPS) e += eps_part[q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
        if (lane == 0) se[warp] = e;
    }
    __syncthreads();
    const int k = k0 + warp, i = sg.begin + TT * (blockIdx.x - sg.tile0) + lane, q = 3 * i + k;
    if (warp >= NK || i >= sg.begin + sg.count) return;
    double v[NG];
#pragma unroll
    for (int g = 0; g < NG; ++g) {
        v[g] = 0;
        for (int w = 0; w < FIN_WARPS; ++w) v[g] += sh[w][g * NK + warp][lane];
    }
    // self tile: D.F uses only its diagonal (diff_equation.c:96-102)
    double self[6];
    tile_of<double>(A, pos, i, i, self);
    const double d = A.preDii / pos[i].w;   // diag_D (diff_decl.c:94-99)
    Rf[q] = (v[0] + F[q] * self[k]) * pre_f;
    if constexpr (RS) {
        double eps = 0;
        for (int w = 0; w < FIN_WARPS; ++w) eps += se[w];
        const int n3 = 3 * sg.count;
        eps /= n3;
        eps /= (n3 - 1);
        eps *= 2;
        if (eps > 1.0) eps = 1.0;
        const double aa = (n3 - 1) * eps * eps - (n3 - 2) * eps;
        double beta;
        if (fabs(aa) < (double)0.0000001f) beta = 0.5;
        else beta = (1 - sqrt(1 - aa)) / aa;
        double c = v[1] * (beta * beta * (1 / d));
        c = 1 / (1 + c);
        c = sqrt(c);
        Rs[q] = c * (beta * v[2] + d * X[q]);
    }
}

// hydro none (diff_rand.c:55-63): X already carries sqrt(2 dt D_ii)
__global__ void k_diag_drift(int n, double preDii, const double4* __restrict__ pos, const double* __restrict__ F,
                             const double* __restrict__ X, double pre_f, int want_rs, double* __restrict__ Rf,
                             double* __restrict__ Rs)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= 3 * n) return;
    const double d = preDii / pos[q / 3].w;
    Rf[q] = pre_f * d * F[q];
    if (want_rs) Rs[q] = X[q];
}

template <typename T, int KIND, bool RS>
static void tea_pairs(bdb_system* s, const TensorArgs& A, const FastArg<KIND>& E, const TeaSeg* segs)
{
    // steps of a 256th of the least radius reach 2^15 of them; in L (the converged split)
    // steps of 2^-22 reach two boxes
    PairUnits u;
    u.unit = KIND == TILE_FAST ? A.ec.inv_L : 1.0;
    u.step = KIND == TILE_FAST ? std::ldexp(1.0, -22) : std::ldexp(1.0, std::ilogb(s->radius_min) - 8);
    u.inv_step = 1 / u.step;
    k_tea_pairs<T, KIND, RS><<<(s->n_jobs + TEA_WARPS - 1) / TEA_WARPS, 32 * TEA_WARPS, 0, s->stream>>>(
        A, E, s->jobs.p, s->n_jobs, s->tea_cols.p, segs, s->pos.p, s->F.p, s->X.p, reinterpret_cast<T*>(s->part.p),
        s->eps_part.p, u);
}

template <bool RS>
static void tea_dispatch_rs(bdb_system* s, const TensorArgs& A, const TeaSeg* segs)
{
    if (s->p.precision == BDB_PREC_FP64) {
        if (A.ewald) tea_pairs<double, TILE_EWALD, RS>(s, A, NoFast(), segs);
        else tea_pairs<double, TILE_FREE, RS>(s, A, NoFast(), segs);
    } else {
        if (s->ewald_fast) tea_pairs<float, TILE_FAST, RS>(s, A, *s->ewald_fast, segs);
        else if (A.ewald) tea_pairs<float, TILE_EWALD, RS>(s, A, NoFast(), segs);
        else tea_pairs<float, TILE_FREE, RS>(s, A, NoFast(), segs);
    }
}

static void tea_dispatch(bdb_system* s, const TensorArgs& A, const TeaSeg* segs, bool want_rs)
{
    if (want_rs) tea_dispatch_rs<true>(s, A, segs);
    else tea_dispatch_rs<false>(s, A, segs);
}

template <typename T, bool RS, int NK>
static void tea_finish_nk(bdb_system* s, const TensorArgs& A, const TeaSeg* segs, const TeaTile* tiles)
{
    k_tea_finish<T, RS, NK><<<dim3(s->tea_tiles, 3 / NK), 32 * FIN_WARPS, 0, s->stream>>>(
        A, segs, tiles, reinterpret_cast<const T*>(s->part.p), s->eps_part.p, s->pos.p, s->F.p, s->X.p,
        s->p.dt / (BDB_KB * s->p.T), s->Rf.p, s->Rs.p);
}

// three CTAs a tile up to 2 tiles per SM (N = 3000 in FP64: 10.7 -> 6.5 us
// with 94 tiles; the 256-replica batch's 4,400 tiles: 24 us, 48 with three)
template <typename T>
static void tea_finish(bdb_system* s, const TensorArgs& A, const TeaSeg* segs, const TeaTile* tiles, bool want_rs)
{
    const bool wide = s->tea_tiles <= 2 * s->sm_count;
    if (want_rs) wide ? tea_finish_nk<T, true, 1>(s, A, segs, tiles) : tea_finish_nk<T, true, 3>(s, A, segs, tiles);
    else wide ? tea_finish_nk<T, false, 1>(s, A, segs, tiles) : tea_finish_nk<T, false, 3>(s, A, segs, tiles);
}

// Work list of k_tea_pairs and the record layout, for the segments of the
// system. The size of a job follows from the number of tile pairs against
// the warps the GPU holds: with few pairs a tile pair's 32 steps are cut into
// up to 8 jobs, with many a job takes several column tiles (fewer row
// records) and, in FP32 and free space, two row tiles (each column load and
// hand-over serves two pairs). tea_tile 16 (tunable) makes jobs half as long.
static int tea_setup(bdb_system* s)
{
    long long pairs = 0;
    for (const Segment& sg : s->segs) {
        const long long nt = (sg.count + TT - 1) / TT;
        pairs += nt * (nt + 1) / 2;
    }
    // jobs that fill the GPU a few times over; lattice sums, thousands of
    // operations a pair, are cut finer
    const long long fill = 16ll * s->sm_count * (s->tea_tile == 16 ? 2 : 1);
    const int max_split = s->p.ewald ? 16 : 8;
    int split = 1, run = 1;
    while (split < max_split && pairs * split < (s->p.ewald ? 2 * fill : fill / 2)) split *= 2;
    const bool fp64 = s->p.precision == BDB_PREC_FP64;
    const bool two = !s->p.ewald && !fp64 && pairs >= 4 * fill;
    while (run < 8 && pairs / (2 * run * (two ? 2 : 1)) >= 4 * fill) run *= 2;
    std::vector<TileJob> jobs;
    std::vector<int> cols;           // column record of (job, column tile): slot, turned into an index below
    std::vector<int> col_tile;
    std::vector<TeaSeg> ts;
    std::vector<TeaTile> tiles;
    std::vector<int> nrow, ncol;
    for (size_t g = 0; g < s->segs.size(); ++g) {
        const Segment& sg = s->segs[g];
        TeaSeg t;
        t.begin = sg.begin;
        t.count = sg.count;
        t.tile0 = (int)tiles.size();
        t.ntile = (sg.count + TT - 1) / TT;
        t.job0 = (int)jobs.size();
        tiles.resize(tiles.size() + t.ntile, TeaTile{0, 0, (int)g, 0});
        nrow.resize(tiles.size(), 0);
        ncol.resize(tiles.size(), 0);
        auto add = [&](int type, int I, int J0, int nJ, int s0, int s1) {
            TileJob j;
            j.seg = (int)g;
            j.I = I;
            j.J0 = J0;
            j.nJ = nJ;
            j.s0 = s0;
            j.s1 = s1;
            j.type = type;
            j.col0 = (int)cols.size();
            const int nrec = !fp64 && (type == JOB_DIAG || nJ > 1) ? 2 : 1;   // row records of the job
            j.rec0 = nrow[t.tile0 + I];
            nrow[t.tile0 + I] += nrec;
            j.rec1 = 0;
            if (type == JOB_ROWS2) {
                j.rec1 = nrow[t.tile0 + I + 1];
                nrow[t.tile0 + I + 1] += nrec;
            }
            if (type != JOB_DIAG)
                for (int q = 0; q < nJ; ++q) {
                    cols.push_back(ncol[t.tile0 + J0 + q]++);
                    col_tile.push_back(t.tile0 + J0 + q);
                }
            jobs.push_back(j);
        };
        auto strip = [&](int type, int I, int J_end) {
            for (int J = 0; J < J_end; J += run)
                for (int u = 0; u < split; ++u)
                    add(type, I, J, std::min(run, J_end - J), TT * u / split, TT * (u + 1) / split);
        };
        for (int I = t.ntile - 1; I >= 0; --I) {
            // long strips first
            if (two && I % 2 == 1) {
                strip(JOB_ROWS2, I - 1, I - 1);
                add(JOB_ROWS1, I, I - 1, 1, 0, TT);
            } else if (!two || I == t.ntile - 1) {
                strip(JOB_ROWS1, I, I);
            }
        }
        for (int I = 0; I < t.ntile; ++I)
            for (int u = 0; u < split; ++u)
                add(JOB_DIAG, I, I, 1, 1 + TT / 2 * u / split, 1 + TT / 2 * (u + 1) / split);
        t.job1 = (int)jobs.size();
        ts.push_back(t);
    }
    size_t rec = 0;
    for (size_t b = 0; b < tiles.size(); ++b) {
        tiles[b].rec0 = (int)rec;
        tiles[b].nslot = nrow[b] + ncol[b];
        rec += tiles[b].nslot;
    }
    for (size_t q = 0; q < cols.size(); ++q) cols[q] += tiles[col_tile[q]].rec0 + nrow[col_tile[q]];
    for (TileJob& j : jobs) {
        const int t0 = ts[j.seg].tile0;
        j.rec0 += tiles[t0 + j.I].rec0;
        if (j.type == JOB_ROWS2) j.rec1 += tiles[t0 + j.I + 1].rec0;
    }
    if (rec > (size_t)1 << 30) return fail(BDB_ERR_NOMEM, "too many bead tiles for the pair sums");
    s->n_jobs = (int)jobs.size();
    s->tea_tiles = (int)tiles.size();
    const size_t el = fp64 ? sizeof(double) : sizeof(float);
    if (s->jobs.alloc(jobs.size()) || s->tea_cols.alloc(std::max<size_t>(1, cols.size())) ||
        s->eps_part.alloc(jobs.size()) || s->part.alloc((rec * REC * el + sizeof(double) - 1) / sizeof(double)) ||
        s->tea_meta.alloc(sizeof(TeaTile) * tiles.size() + sizeof(TeaSeg) * ts.size()))
        return BDB_ERR_NOMEM;
    BDB_CUDA(h2d(s, s->jobs.p, jobs.data(), sizeof(TileJob) * jobs.size()));
    BDB_CUDA(h2d(s, s->tea_cols.p, cols.data(), sizeof(int) * cols.size()));
    BDB_CUDA(h2d(s, s->tea_meta.p, tiles.data(), sizeof(TeaTile) * tiles.size()));
    BDB_CUDA(h2d(s, s->tea_meta.p + sizeof(TeaTile) * tiles.size(), ts.data(), sizeof(TeaSeg) * ts.size()));
    return BDB_OK;
}

static const TeaTile* tea_tile_table(const bdb_system* s) { return reinterpret_cast<const TeaTile*>(s->tea_meta.p); }
static const TeaSeg* tea_seg_table(const bdb_system* s)
{
    return reinterpret_cast<const TeaSeg*>(s->tea_meta.p + sizeof(TeaTile) * s->tea_tiles);
}

// Autotuning of the job length (tea_tile 16 or 32): each candidate's work
// list is built and its pair kernel timed twice on the system's stream; the
// faster one is kept. Runs at the first TEA call of a system with
// autotuning on (which comes before any graph capture).
static int tea_tune(bdb_system* s, bool want_rs)
{
    const int cands[2] = {16, 32};
    float best_ms = 1e30f;
    int best = s->tea_tile;
    cudaEvent_t e0, e1;
    BDB_CUDA(cudaEventCreate(&e0));
    BDB_CUDA(cudaEventCreate(&e1));
    for (int c : cands) {
        s->tea_tile = c;
        int rc = tea_setup(s);
        if (rc) return rc;
        if (int rc_e = ewald_tables(s)) return rc_e;
        const TensorArgs A = targs(s);
        tea_dispatch(s, A, tea_seg_table(s), want_rs);   // warm-up
        BDB_CUDA(cudaEventRecord(e0, s->stream));
        tea_dispatch(s, A, tea_seg_table(s), want_rs);
        tea_dispatch(s, A, tea_seg_table(s), want_rs);
        BDB_CUDA(cudaEventRecord(e1, s->stream));
        BDB_CUDA(cudaEventSynchronize(e1));
        float ms = 0;
        BDB_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        s->launches += 3;
        if (ms < best_ms) {
            best_ms = ms;
            best = c;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    s->tea_tile = best;
    s->tea_tuned = true;
    return tea_setup(s);
}

int tea_run(bdb_system* s, bool want_rs)
{
    if (!s->p.hydro) {
        const double pre_f = s->p.dt / (BDB_KB * s->p.T);
        k_diag_drift<<<(s->n3 + 127) / 128, 128, 0, s->stream>>>(s->n, s->preDii, s->pos.p, s->F.p, s->X.p, pre_f,
                                                                 want_rs, s->Rf.p, s->Rs.p);
        BDB_CUDA(cudaGetLastError());
        s->launches += 1;
        return BDB_OK;
    }
    if (s->autotune && !s->tea_tuned) {
        int rc = tea_tune(s, want_rs);
        if (rc) return rc;
    } else if (!s->tea_meta.p) {
        int rc = tea_setup(s);
        if (rc) return rc;
    }
    if (int rc_e = ewald_tables(s)) return rc_e;
    const TensorArgs A = targs(s);
    tea_dispatch(s, A, tea_seg_table(s), want_rs);
    BDB_CUDA(cudaGetLastError());
    if (s->p.precision == BDB_PREC_FP64) tea_finish<double>(s, A, tea_seg_table(s), tea_tile_table(s), want_rs);
    else tea_finish<float>(s, A, tea_seg_table(s), tea_tile_table(s), want_rs);
    BDB_CUDA(cudaGetLastError());
    s->launches += 2;
    return BDB_OK;
}

}  // namespace bdb
