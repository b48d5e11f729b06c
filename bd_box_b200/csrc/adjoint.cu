// Hand-written adjoint of the Ermak-McCammon step with Cholesky noise.
//
// One step (diff_equation.c:216-286 with compute_r's Cholesky branch,
// diff_rand.c:64-85) maps x to
//     x' = x + c D(x) F(x; theta) + B(x) X,   c = dt/(kB T), B = chol(D),
// with X = sqrt(2 dt) xi the step's fixed noise. Given lambda' = dL/dx', the
// adjoint step returns
//     lambda = lambda' + c [ (dD/dx : F)^T lambda' + (dF/dx)^T (D lambda') ]
//                     + (d(B X)/dx)^T lambda'
//     theta_bar += c (D lambda')^T dF/dtheta.
// * D is a sum of pair tiles T(x_i - x_j) (free-space RPY with the overlap
//   form; the diagonal tiles do not depend on x), so every x-derivative of a
//   contraction <G, D> is a pair sum of grad_r <G_ij, T(r)> (k_tile_grad).
// * The forces are conservative, dF/dx is symmetric, and its product with
//   u = D lambda' is a pair sum over bonds, LJ and Debye-Hueckel pairs with
//   the forward pass's cutoffs and bonded scaling (k_force_jvp), which also
//   accumulates u^T dF/dtheta for the four force-field scale factors.
// * The Cholesky factor's derivative dB = B Phi(B^-1 dD B^-T), Phi = lower
//   triangle with half the diagonal, gives
//     lambda'^T dB X = <Dbar, dD>,  Dbar = B^-T Phi(v X^T) B^-1,  v = B^T lambda',
//   formed from the inverse of B by products of full tiles (adjoint_linalg).
// The forward pass is recomputed from checkpoints every `checkpoint` steps. A
// segment's steps leave what their reverse needs -- positions and, where the
// device has room for them, forces, D and B -- so that each step is factored
// once more, not twice; the last segment's are kept by the forward pass itself.
// Without that room forces, D and B are computed again from the positions.
// Precision follows the system's: FP64 throughout for an FP64 system; for a
// mixed-precision system (FP32 tensor, FP16-split Cholesky) the forward steps
// are the mixed path's, and the backward's O(n^3) part -- the inverse and the
// products with Phi(v X^T) B^-1 -- runs in FP32 on its FP32 factor, while the
// O(N^2) tile gradients and force products keep FP64 arithmetic and FP64 sums.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "bdb_common.cuh"

namespace bdb {

// ---------------------------------------------------------------- tiles

// T(r) = A(r) I + Bc(r) e e^T (rpy_free); the gradient of <G, T(r)> with
// respect to r = x_i - x_j needs A', Bc and Bc'. si is bead j's radius, sj
// bead i's.
__device__ __forceinline__ void tile_grad(const double* r, double si, double sj, double preDii, double preDij,
                                          const double* G, double* g)
{
    const double r_sq = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
    const double rn = sqrt(r_sq);
    const double e[3] = {r[0] / rn, r[1] / rn, r[2] / rn};
    double Bc, dA, dB;
    if (rn < si + sj) {
        const double sigma = (si + sj) / 2;
        const double pre = preDii / sigma;
        Bc = pre * 3 * rn / (32 * sigma);
        dA = -9 * pre / (32 * sigma);
        dB = 3 * pre / (32 * sigma);
    } else {
        const double S = si * si + sj * sj;
        Bc = preDij / rn - preDij * S / (rn * r_sq);
        dA = -preDij / r_sq - preDij * S / (r_sq * r_sq);
        dB = -preDij / r_sq + 3 * preDij * S / (r_sq * r_sq);
    }
    const double tr = G[0] + G[4] + G[8];
    double Ge[3], GTe[3];
    for (int a = 0; a < 3; ++a) {
        Ge[a] = G[3 * a] * e[0] + G[3 * a + 1] * e[1] + G[3 * a + 2] * e[2];
        GTe[a] = G[a] * e[0] + G[3 + a] * e[1] + G[6 + a] * e[2];
    }
    const double eGe = e[0] * Ge[0] + e[1] * Ge[1] + e[2] * Ge[2];
    for (int a = 0; a < 3; ++a)
        g[a] = (dA * tr + dB * eGe) * e[a] + Bc / rn * (Ge[a] + GTe[a] - 2 * eGe * e[a]);
}

// grad_i += sum_{j != i} grad_r <G_ij, T(x_i - x_j)> with
//   G_ij = c (lam_i F_j^T + lam_j F_i^T) + S_ij,
// S the (symmetric) noise weight matrix Z + Z^T (3x3 tile ij, row-major, ld),
// or none. One warp per bead, lanes over j, fixed-order reduction.
template <typename T>
__global__ void k_tile_grad(int n, const double4* __restrict__ pos, double preDii, double preDij, double c,
                            const double* __restrict__ lam, const double* __restrict__ F,
                            const T* __restrict__ S, int ld, double* __restrict__ grad)
{
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i >= n) return;
    const double4 pi = pos[i];
    double li[3], fi[3];
    for (int a = 0; a < 3; ++a) {
        li[a] = lam[3 * i + a];
        fi[a] = F[3 * i + a];
    }
    double acc[3] = {0, 0, 0};
    for (int j = lane; j < n; j += 32) {
        if (j == i) continue;
        const double4 pj = pos[j];
        const double r[3] = {pi.x - pj.x, pi.y - pj.y, pi.z - pj.z};
        double G[9];
        for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b)
                G[3 * a + b] = c * (li[a] * F[3 * j + b] + lam[3 * j + a] * fi[b]) +
                               (S ? (double)S[(size_t)(3 * i + a) * ld + 3 * j + b] : 0.0);
        double g[3];
        tile_grad(r, pj.w, pi.w, preDii, preDij, G, g);
        acc[0] += g[0];
        acc[1] += g[1];
        acc[2] += g[2];
    }
    for (int o = 16; o > 0; o >>= 1)
        for (int a = 0; a < 3; ++a) acc[a] += __shfl_xor_sync(0xffffffffu, acc[a], o);
    if (lane == 0)
        for (int a = 0; a < 3; ++a) grad[3 * i + a] += acc[a];
}

// ---------------------------------------------------------------- forces

struct AdjForce {
    int elec;
    double epsilon_c, kappa_c, gamma_c, cutoff_c;
    double alpha_lj, cutoff_lj, lj6;
    double bond_lj_scale, bond_c_scale;
    int conn_live;
};

__device__ __forceinline__ bool adj_conn(const int* conn_ptr, const int* conn_list, int i, int j)
{
    for (int k = conn_ptr[i]; k < conn_ptr[i + 1]; ++k)
        if (conn_list[k] == j) return true;
    return false;
}

// the pair force on bead i is Fm(r) d / r with d = x_i - x_j; add the
// directional derivative along du = u_i - u_j and the parameter terms
__device__ __forceinline__ void pair_jvp(double Fm, double dFm, const double* d, double rn, const double* du,
                                         double* jvp)
{
    const double phi = Fm / rn;
    const double k2 = (dFm * rn - Fm) / (rn * rn * rn);
    const double dd = d[0] * du[0] + d[1] * du[1] + d[2] * du[2];
    for (int a = 0; a < 3; ++a) jvp[a] += phi * du[a] + k2 * dd * d[a];
}

// grad_i += c (dF/dx u)_i and ppart[4 i + k] += c u_i . dF_i/ds_k for the
// scale factors s = (LJ epsilon, LJ sigma, bond H, Debye length), following
// force_single (calc_func.c:370-409), LJ_force (LJ.c:37-64), electro_force
// (electro.c:36-56) and bond_calc (bond.c:43-85). One warp per bead: lanes
// over all other beads (the forward pass's cutoffs and 1-2 scaling decide
// which pairs act), then the bead's bonds.
__global__ void k_force_jvp(int n, AdjForce fp, const double4* __restrict__ pos, const double* __restrict__ Q,
                            const double2* __restrict__ LJ, const int* __restrict__ conn_ptr,
                            const int* __restrict__ conn_list, const int* __restrict__ bptr,
                            const int* __restrict__ blist, const int* __restrict__ bond_pairs,
                            const double* __restrict__ bond_parms, const double* __restrict__ u, double c,
                            double* __restrict__ grad, double* __restrict__ ppart)
{
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i >= n) return;
    const double4 pi = pos[i];
    const double ui[3] = {u[3 * i], u[3 * i + 1], u[3 * i + 2]};
    double jvp[3] = {0, 0, 0}, pp[4] = {0, 0, 0, 0};
    for (int j = lane; j < n; j += 32) {
        if (j == i) continue;
        const int a = min(i, j), b = max(i, j);
        const double4 pj = pos[j];
        const double d[3] = {pi.x - pj.x, pi.y - pj.y, pi.z - pj.z};
        const double r_sq = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
        const double rn = sqrt(r_sq);
        const double2 la = LJ[a], lb = LJ[b];
        const double sig = la.x + lb.x;
        const double lj_lim = fp.cutoff_lj > 0.0 ? fp.cutoff_lj : (double)1.122462f * sig;
        const bool elec_in = fp.elec && rn <= fp.cutoff_c;
        const bool lj_in = fp.alpha_lj != 0.0 && rn <= lj_lim;
        if (!elec_in && !lj_in) continue;
        const bool conn = fp.conn_live && adj_conn(conn_ptr, conn_list, a, b);
        double Fm = 0, dFm = 0;
        const double du[3] = {ui[0] - u[3 * j], ui[1] - u[3 * j + 1], ui[2] - u[3 * j + 2]};
        const double ud = (ui[0] * d[0] + ui[1] * d[1] + ui[2] * d[2]) / rn;
        if (elec_in && (!conn || fp.bond_c_scale != 0.0)) {
            const double scale = conn ? fp.bond_c_scale : 1.0;
            const double gq = scale * fp.gamma_c / fp.epsilon_c * Q[a] * Q[b];
            const double kap = fp.kappa_c;
            const double ex = exp(-kap * rn);
            Fm += gq * (1 + kap * rn) * ex / r_sq;
            dFm += gq * ex * (-kap * kap / rn - 2 * (1 + kap * rn) / (r_sq * rn));
            pp[3] += ud * gq * kap * kap * ex;   // kappa -> kappa / s
        }
        if (lj_in && (!conn || fp.bond_lj_scale != 0.0)) {
            const double scale = conn ? fp.bond_lj_scale : 1.0;
            const double K = scale * fp.alpha_lj * sqrt(la.y * lb.y) * 6;
            double s6 = sig / rn;
            s6 *= s6;
            s6 *= s6 * s6;
            const double F = K * s6 * (2 * s6 - fp.lj6) / rn;
            Fm += F;
            dFm += K * s6 * (6 * fp.lj6 - 24 * s6) / r_sq - F / rn;
            pp[0] += ud * F;
            pp[1] += ud * K * s6 * (24 * s6 - 6 * fp.lj6) / rn;
        }
        pair_jvp(Fm, dFm, d, rn, du, jvp);
    }
    for (int k = bptr[i] + lane; k < bptr[i + 1]; k += 32) {
        const int t = blist[k];
        const int j = bond_pairs[2 * t] == i ? bond_pairs[2 * t + 1] : bond_pairs[2 * t];
        const double r0 = bond_parms[3 * t], rmax = bond_parms[3 * t + 1], H = bond_parms[3 * t + 2];
        const double4 pj = pos[j];
        const double d[3] = {pi.x - pj.x, pi.y - pj.y, pi.z - pj.z};
        const double r_sq = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
        const double rn = sqrt(r_sq);
        const double q = 1 - r_sq / (rmax * rmax);
        const double Ff = H * (r0 - rn) / q;
        const double dFf = (-H * q + H * (r0 - rn) * 2 * rn / (rmax * rmax)) / (q * q);
        const double du[3] = {ui[0] - u[3 * j], ui[1] - u[3 * j + 1], ui[2] - u[3 * j + 2]};
        pair_jvp(Ff, dFf, d, rn, du, jvp);
        pp[2] += (ui[0] * d[0] + ui[1] * d[1] + ui[2] * d[2]) / rn * Ff;
    }
    for (int o = 16; o > 0; o >>= 1) {
        for (int a = 0; a < 3; ++a) jvp[a] += __shfl_xor_sync(0xffffffffu, jvp[a], o);
        for (int k = 0; k < 4; ++k) pp[k] += __shfl_xor_sync(0xffffffffu, pp[k], o);
    }
    if (lane == 0) {
        for (int a = 0; a < 3; ++a) grad[3 * i + a] += c * jvp[a];
        for (int k = 0; k < 4; ++k) ppart[4 * i + k] += c * pp[k];
    }
}

// ---------------------------------------------------------------- dense

// One pass over the stored matrix M (strict upper: D, lower with diagonal:
// B = chol(D)) for u = D lam (with dD the diagonal) and v = B^T lam. A CTA
// covers 64 columns x 256 rows; thread (row group g, column q) walks 64 rows.
// Partial sums: colp[rb][q] = (lower, upper) column sums of row block rb,
// rowp[cb][p] = upper row sums of column block cb; k_mv2_finish adds them
// in a fixed order.
static constexpr int MV2_COLS = 64, MV2_ROWS = 256;

template <typename TM>
__global__ void __launch_bounds__(256) k_mv2(const TM* __restrict__ M, int n, int ld,
                                             const double* __restrict__ lam, double* __restrict__ colp,
                                             double* __restrict__ rowp)
{
    __shared__ double cl[4][MV2_COLS], cu[4][MV2_COLS];
    __shared__ double rs[MV2_ROWS][MV2_COLS / 16 + 1];
    const int q = threadIdx.x & 63, g = threadIdx.x >> 6;
    const int cb = blockIdx.x, rb = blockIdx.y;
    const int col = cb * MV2_COLS + q;
    double sl = 0, su = 0;
    for (int k = 0; k < 64; ++k) {
        const int row = rb * MV2_ROWS + g * 64 + k;
        double rsum = 0;
        if (row < n && col < n) {
            const double m = (double)M[(size_t)row * ld + col];
            const double lr = lam[row];
            if (col <= row) {
                sl += m * lr;
            } else {
                su += m * lr;
                rsum = m * lam[col];
            }
        }
        // row sum of the upper part over this CTA's 64 columns: 16 lanes per
        // partial, then 4 partials in a fixed order
        for (int o = 8; o > 0; o >>= 1) rsum += __shfl_xor_sync(0xffffffffu, rsum, o, 16);
        if ((q & 15) == 0) rs[g * 64 + k][q >> 4] = rsum;
    }
    cl[g][q] = sl;
    cu[g][q] = su;
    __syncthreads();
    if (g == 0 && col < n) {
        colp[((size_t)rb * n + col) * 2] = cl[0][q] + cl[1][q] + cl[2][q] + cl[3][q];
        colp[((size_t)rb * n + col) * 2 + 1] = cu[0][q] + cu[1][q] + cu[2][q] + cu[3][q];
    }
    for (int r = threadIdx.x; r < MV2_ROWS; r += blockDim.x) {
        const int row = rb * MV2_ROWS + r;
        if (row < n) rowp[(size_t)cb * n + row] = rs[r][0] + rs[r][1] + rs[r][2] + rs[r][3];
    }
}

__global__ void k_mv2_finish(int n, int nrb, int ncb, const double* __restrict__ colp,
                             const double* __restrict__ rowp, const double* __restrict__ dD,
                             const double* __restrict__ lam, double* __restrict__ u, double* __restrict__ v)
{
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= n) return;
    double sl = 0, su = 0, sr = 0;
    for (int rb = 0; rb < nrb; ++rb) {
        sl += colp[((size_t)rb * n + a) * 2];
        su += colp[((size_t)rb * n + a) * 2 + 1];
    }
    for (int cb = 0; cb < ncb; ++cb) sr += rowp[(size_t)cb * n + a];
    u[a] = dD[a] * lam[a] + su + sr;
    v[a] = sl;
}

// The Cholesky factor's adjoint as products of full matrices. With A = B^-1
// (lower triangular) Dbar = A^T Phi(v X^T) A, and Phi(v X^T) A needs no
// product: row a of it is v_a times the running sum over c < a of X_c A_c (half
// of c = a), O(n^2). So with G = Phi A
//     S = Z + Z^T = A^T G + G^T A,  S_ij = sum over k >= max(i, j),
// n^3/3 multiply-adds for one half of it and n^3/6 for the inverse, all in
// 128 x 128 tiles, in about 18 launches; two blocked triangular solves with n
// right-hand sides take n^3 in 190 launches of narrow updates (n = 3072, FP32:
// 4.2 ms a step before, 1.34 now).

// Room: A and G are lower triangular and share one buffer, n rows of n + 128:
// row block C (128 rows) of G lies in row block nb - 1 - C, right of A's last
// block there. W, the partial sums of G and then S share another (n x n): each
// is read for the last time before the next is written. So two matrices beside
// the system's own, as the two right-hand sides of the solves took.
template <typename T>
struct PlainRows {
    const T* p;
    size_t ld;
    __device__ const T* at(int r) const { return p + (size_t)r * ld; }
};
template <typename T>
struct GRows {
    T* p;
    size_t ld;
    int nb;
    __device__ T* at(int r) const
    {
        const int C = r >> 7;
        return p + (size_t)(128 * (nb - 1 - C) + (r & 127)) * ld + 128 * (nb - C);
    }
};

// inverses of the 64x64 diagonal blocks of the lower-triangular B (ld) into A
// (lda, zero above the diagonal), column c by forward substitution: four
// lanes share a column's dot products (one lane each: 83 us at n = 3072),
// accumulated in FP64 over the column's entries as stored (T)
template <typename TM, typename T>
__global__ void __launch_bounds__(256) k_trinv64(const TM* __restrict__ B, int ld, T* __restrict__ A, size_t lda)
{
    extern __shared__ __align__(16) unsigned char trinv_smem[];
    T(*Bs)[65] = reinterpret_cast<T(*)[65]>(trinv_smem);
    T(*W)[65] = reinterpret_cast<T(*)[65]>(trinv_smem + sizeof(T) * 64 * 65);
    __shared__ double dinv[64];
    const int tid = threadIdx.x, c = tid >> 2, q = tid & 3;
    const size_t o = (size_t)blockIdx.x * 64;
    for (int e = tid; e < 64 * 64; e += 256) {
        const int r = e >> 6, k = e & 63;
        Bs[r][k] = k <= r ? (T)B[(o + r) * ld + o + k] : (T)0;
        if (k > r) W[r][k] = (T)0;
    }
    if (tid < 64) dinv[tid] = 1.0 / (double)B[(o + tid) * ld + o + tid];
    __syncthreads();
    for (int i = 8 * (tid >> 5); i < 64; ++i) {   // rows above the warp's columns are zero
        double a = 0.0;
        for (int m = c + q; m < i; m += 4) a += (double)Bs[i][m] * (double)W[m][c];
        a += __shfl_xor_sync(0xffffffffu, a, 1);
        a += __shfl_xor_sync(0xffffffffu, a, 2);
        if (q == 0 && i >= c) W[i][c] = (T)(((i == c ? 1.0 : 0.0) - a) * dinv[i]);
        __syncwarp();
    }
    __syncthreads();
    for (int e = tid; e < 64 * 64; e += 256) A[(o + (e >> 6)) * lda + o + (e & 63)] = W[e >> 6][e & 63];
}

// ---- tile products: TILE x TILE (128 or 64) on TILE^2 / 64 threads with 8 x 8
// outputs each (rows and columns 4 t and TILE/2 + 4 t of the tile), K in steps
// of 16 through two shared-memory stages; the next step's operands are loaded
// into registers while the present one is multiplied. FP32 or FP64
// multiply-adds as the matrices are stored; bound by those.
static constexpr int GT = 128, GK = 16;
constexpr int gemm_threads(int tile) { return tile * tile / 64; }

// In FP32 a thread's sums over 64 k are added to their running sums in shared
// memory (a 64th of the multiply-adds), so that a sum of thousands rounds like
// one of a hundred.
static constexpr int GFLUSH = 64;

template <typename T, int TILE>
struct GemmSmem {
    T a[2][GK][TILE + 4], b[2][GK][TILE + 4];
    T sum[sizeof(T) == 4 ? 64 : 1][sizeof(T) == 4 ? gemm_threads(TILE) : 1];
};

// 8 consecutive elements (16-byte aligned)
__device__ __forceinline__ void load8(const float* p, float* v)
{
    const float4 x = *reinterpret_cast<const float4*>(p), y = *reinterpret_cast<const float4*>(p + 4);
    v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w, v[4] = y.x, v[5] = y.y, v[6] = y.z, v[7] = y.w;
}
__device__ __forceinline__ void load8(const double* p, double* v)
{
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
        const double2 x = *reinterpret_cast<const double2*>(p + k);
        v[k] = x.x, v[k + 1] = x.y;
    }
}

// acc += op(A) B over k0 <= k < k1 (multiples of 16). op(A)(m, k) is row m of
// A at k or, with TA, row k of A at ma + m; B(k, c) is row k of B at nb + c. Rows
// m >= ml and columns c >= nl (multiples of 8) are zero.
template <typename T, bool TA, int TILE, class RA, class RB>
__device__ __forceinline__ void gemm_tile(GemmSmem<T, TILE>& sm, const RA A, int ma, const RB B, int nb, int k0, int k1,
                                          int ml, int nl, T (&acc)[8][8])
{
    constexpr int NT = gemm_threads(TILE), NP = 2 * TILE / NT;   // pieces of 8 per thread and operand
    constexpr int HX = TILE / 8;                                 // threads along a tile's side
    const int tid = threadIdx.x, tx = tid % HX, ty = tid / HX;
    T ra[NP][8], rb[NP][8];
    // 16 rows from a multiple of 16: in one row block of 128
    const T* a0 = TA ? A.at(k0) + ma : nullptr;
    const T* b0 = B.at(k0) + nb;
    auto load = [&](int k) {
        if (k > k0) {
            const bool next = (k & 127) == 0;
            if (TA) a0 = next ? A.at(k) + ma : a0 + 16 * A.ld;
            b0 = next ? B.at(k) + nb : b0 + 16 * B.ld;
        }
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            const int e = tid + NT * p, kr = e / HX, c8 = 8 * (e % HX);   // a row of TILE in pieces of 8
            const int mr = e >> 1, k8 = 8 * (e & 1);                      // 16 k of one row
#pragma unroll
            for (int u = 0; u < 8; ++u) ra[p][u] = rb[p][u] = (T)0;
            if (TA) {
                if (c8 < ml) load8(a0 + (size_t)kr * A.ld + c8, ra[p]);
            } else {
                if (mr < ml) load8(A.at(mr) + k + k8, ra[p]);
            }
            if (c8 < nl) load8(b0 + (size_t)kr * B.ld + c8, rb[p]);
        }
    };
    auto store = [&](int st) {
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            const int e = tid + NT * p, kr = e / HX, c8 = 8 * (e % HX), mr = e >> 1, k8 = 8 * (e & 1);
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (TA) sm.a[st][kr][c8 + u] = ra[p][u];
                else sm.a[st][k8 + u][mr] = ra[p][u];
                sm.b[st][kr][c8 + u] = rb[p][u];
            }
        }
    };
    if (k0 >= k1) return;
    load(k0);
    __syncthreads();   // an earlier product's stages are read
    int since = 0;
    store(0);
    __syncthreads();
    int st = 0;
    for (int k = k0; k < k1; k += GK, st ^= 1) {
        const bool more = k + GK < k1;
        if (more) load(k + GK);
#pragma unroll
        for (int kk = 0; kk < GK; ++kk) {
            T a[8], b[8];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                a[u] = sm.a[st][kk][4 * ty + u];
                a[4 + u] = sm.a[st][kk][TILE / 2 + 4 * ty + u];
                b[u] = sm.b[st][kk][4 * tx + u];
                b[4 + u] = sm.b[st][kk][TILE / 2 + 4 * tx + u];
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] += a[i] * b[j];
        }
        if (more) store(st ^ 1);
        if (sizeof(T) == 4 && ((since += GK) == GFLUSH)) {
            since = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    sm.sum[8 * i + j][tid] += acc[i][j];
                    acc[i][j] = (T)0;
                }
        }
        __syncthreads();
    }
}

// a thread's sums before and after its products
template <typename T, int TILE>
__device__ __forceinline__ void gemm_begin(GemmSmem<T, TILE>& sm, T (&acc)[8][8])
{
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            acc[i][j] = (T)0;
            if (sizeof(T) == 4) sm.sum[8 * i + j][threadIdx.x] = (T)0;
        }
}
template <typename T, int TILE>
__device__ __forceinline__ void gemm_end(const GemmSmem<T, TILE>& sm, T (&acc)[8][8])
{
    if (sizeof(T) == 4)
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[i][j] += sm.sum[8 * i + j][threadIdx.x];
}

// row or column u of a thread's 8
template <int TILE>
__device__ __forceinline__ int gemm_at(int t, int u)
{
    return (u < 4 ? 0 : TILE / 2 - 4) + 4 * t + u;
}

// One level of the inverse: blocks of s rows are inverted; pair z joins block
// 2 z (rows c0) and 2 z + 1 (rows r0, cut at n): A21 = -A22 (B21 A11). STAGE 0:
// W21 = B21 A11, STAGE 1: A21 = -A22 W21 (W: n x n scratch). 64 x 64 tiles: the
// levels have few outputs and long sums (n = 3072: 128 tiles of 128 with k up
// to 2048 at the last one, 0.92 ms in all levels; 0.69 with 64).
template <typename T, int STAGE>
__global__ void __launch_bounds__(gemm_threads(64), sizeof(T) == 4 ? 6 : 4)
k_tri_level(int n, int s, const T* __restrict__ B, int ldb, T* __restrict__ A, size_t lda, T* __restrict__ W)
{
    extern __shared__ __align__(16) unsigned char gemm_smem[];
    constexpr int TL = 64;
    GemmSmem<T, TL>& sm = *reinterpret_cast<GemmSmem<T, TL>*>(gemm_smem);
    const int c0 = 2 * blockIdx.z * s, r0 = c0 + s;
    const int m0 = blockIdx.y * TL, n0 = blockIdx.x * TL;
    const int ml = min(s, n - r0) - m0, nl = s - n0;   // rows and columns left
    if (ml <= 0 || nl <= 0) return;
    T acc[8][8];
    gemm_begin(sm, acc);
    if (STAGE == 0)   // A11 is zero above its diagonal: k >= n0
        gemm_tile<T, false, TL>(sm, PlainRows<T>{B + (size_t)(r0 + m0) * ldb + c0, (size_t)ldb}, 0,
                                PlainRows<T>{A + (size_t)c0 * lda + c0, lda}, n0, n0, s, ml, nl, acc);
    else              // A22 likewise: k < m0 + 64
        gemm_tile<T, false, TL>(sm, PlainRows<T>{A + (size_t)(r0 + m0) * lda + r0, lda}, 0,
                                PlainRows<T>{W + (size_t)r0 * n + c0, (size_t)n}, n0, 0,
                                min(m0 + TL, min(s, n - r0)), ml, nl, acc);
    gemm_end(sm, acc);
    const size_t ldo = STAGE == 0 ? (size_t)n : lda;
    T* O = (STAGE == 0 ? W : A) + (size_t)(r0 + m0) * ldo + c0 + n0;
    const int tx = threadIdx.x % (TL / 8), ty = threadIdx.x / (TL / 8);
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int r = gemm_at<TL>(ty, i), c = gemm_at<TL>(tx, j);
            if (r < ml && c < nl) O[(size_t)r * ldo + c] = STAGE == 0 ? acc[i][j] : -acc[i][j];
        }
}

// G = Phi(v X^T) A in two passes over blocks of 64 rows: the blocks' sums of
// X_c A_c, then each block's running sum from those before it (FP64)
template <typename T>
__global__ void k_phi_sums(int n, const double* __restrict__ X, const T* __restrict__ A, size_t lda,
                           double* __restrict__ sums)
{
    const int b = blockIdx.x * blockDim.x + threadIdx.x, r0 = 64 * blockIdx.y;
    if (b >= n) return;
    double a = 0;
    if (b < r0 + 64)
        for (int c = r0; c < r0 + 64; ++c) a += X[c] * (double)A[(size_t)c * lda + b];
    sums[(size_t)blockIdx.y * n + b] = a;
}
template <typename T>
__global__ void k_phi_rows(int n, const double* __restrict__ v, const double* __restrict__ X, const T* A, size_t lda,
                           const double* __restrict__ sums, const GRows<T> G)
{
    const int b = blockIdx.x * blockDim.x + threadIdx.x, r0 = 64 * blockIdx.y;
    if (b >= (r0 / 128 + 1) * 128) return;   // G's row block ends at its diagonal block
    double run = 0;
    for (int q = b / 64; q < (int)blockIdx.y; ++q) run += sums[(size_t)q * n + b];
    T* g = G.at(r0) + b;
    for (int c = r0; c < r0 + 64; ++c) {
        const double t = b <= c ? X[c] * (double)A[(size_t)c * lda + b] : 0.0;
        g[(size_t)(c - r0) * lda] = (T)(v[c] * (run + 0.5 * t));
        run += t;
    }
}

// S pieces: tile (i, j), i >= j, of 128 x 128 over 128 i + sk q <= k <
// 128 i + sk (q + 1): A^T G + G^T A. The sum over k is longest where tiles are
// fewest (k >= 128 i), so it is cut into at most 8 pieces (adj_piece): 1,000
// pieces of 384 at n = 3072 for 296 CTA slots. k_adj_join adds a tile's pieces
// in order and writes the tile and its mirror image. Rows of tiles are taken
// in rounds of at most ADJ_ROUND pieces (one row where that has more): seven
// waves of CTAs, all of n = 3072 in one, and 128 KB (FP64) a piece of room.
static constexpr int ADJ_ROUND = 2048;
__host__ __device__ inline int adj_piece(int nb) { return GT * (nb > 24 ? (nb + 7) / 8 : 3); }
__host__ __device__ inline int adj_pieces_of(int nb, int i)
{
    const int sk = adj_piece(nb);
    return (GT * (nb - i) + sk - 1) / sk;
}
__host__ __device__ inline int adj_pieces_before(int nb, int i)
{
    int p = 0;
    for (int q = 0; q < i; ++q) p += (q + 1) * adj_pieces_of(nb, q);
    return p;
}

// end of the round that starts with row i0
static int adj_round_end(int nb, int i0)
{
    int i1 = i0, p = 0;
    do p += (i1 + 1) * adj_pieces_of(nb, i1);
    while (++i1 < nb && p + (i1 + 1) * adj_pieces_of(nb, i1) <= ADJ_ROUND);
    return i1;
}
// pieces of the largest round
static int adj_round_pieces(int nb)
{
    int most = 0;
    for (int i0 = 0, i1; i0 < nb; i0 = i1) {
        i1 = adj_round_end(nb, i0);
        most = std::max(most, adj_pieces_before(nb, i1) - adj_pieces_before(nb, i0));
    }
    return most;
}

// the pieces from number p0 on
template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 2 : 1)
k_adj_pieces(int n, int p0, const PlainRows<T> A, const GRows<T> G, T* __restrict__ part)
{
    extern __shared__ __align__(16) unsigned char gemm_smem[];
    GemmSmem<T, GT>& sm = *reinterpret_cast<GemmSmem<T, GT>*>(gemm_smem);
    const int nb = n / GT;
    int i = 0, p = p0 + blockIdx.x;
    while (p >= (i + 1) * adj_pieces_of(nb, i)) p -= (i + 1) * adj_pieces_of(nb, i++);
    const int np = adj_pieces_of(nb, i), j = p / np, q = p % np;
    const int sk = adj_piece(nb), k0 = GT * i + sk * q, k1 = min(n, k0 + sk);
    T acc[8][8];
    gemm_begin(sm, acc);
    gemm_tile<T, true, GT>(sm, A, GT * i, G, GT * j, k0, k1, GT, GT, acc);
    gemm_tile<T, true, GT>(sm, G, GT * i, A, GT * j, k0, k1, GT, GT, acc);
    gemm_end(sm, acc);
    T* O = part + (size_t)blockIdx.x * GT * GT;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int c = 0; c < 8; ++c) O[gemm_at<GT>(ty, r) * GT + gemm_at<GT>(tx, c)] = acc[r][c];
}

// 32 x 32 of tile (i, j) per CTA (blockIdx.z = 0..15), rows i0 .. of tiles
template <typename T>
__global__ void __launch_bounds__(256) k_adj_join(int n, int i0, int p0, const T* __restrict__ part, T* __restrict__ S)
{
    const int i = i0 + blockIdx.y, j = blockIdx.x;
    if (j > i) return;
    __shared__ T t[32][33];
    const int nb = n / GT, np = adj_pieces_of(nb, i);
    const T* src = part + (size_t)(adj_pieces_before(nb, i) - p0 + j * np) * GT * GT;
    const int r0 = 32 * (blockIdx.z >> 2), c0 = 32 * (blockIdx.z & 3);
    const int x = threadIdx.x & 31;
    for (int y = threadIdx.x >> 5; y < 32; y += 8) {
        T a = (T)0;
        for (int q = 0; q < np; ++q) a += src[(size_t)q * GT * GT + (r0 + y) * GT + c0 + x];
        t[y][x] = a;
        S[(size_t)(GT * i + r0 + y) * n + GT * j + c0 + x] = a;
    }
    if (i == j) return;
    __syncthreads();
    for (int y = threadIdx.x >> 5; y < 32; y += 8) S[(size_t)(GT * j + c0 + y) * n + GT * i + r0 + x] = t[x][y];
}

// ---------------------------------------------------------------- driver

template <typename T>
struct Scratch {
    T* p = nullptr;
    ~Scratch()
    {
        if (p) cudaFree(p);
    }
    int alloc(size_t n)
    {
        return cudaMalloc(reinterpret_cast<void**>(&p), sizeof(T) * std::max<size_t>(n, 1)) == cudaSuccess ? 0 : 1;
    }
};

// n elements at a 256-byte offset of a shared allocation
template <typename T>
struct Part {
    T* p = nullptr;
    size_t at = 0;
    void place(size_t& bytes, size_t n)
    {
        at = bytes;
        bytes += (sizeof(T) * n + 255) / 256 * 256;
    }
    void set(unsigned char* base) { p = reinterpret_cast<T*>(base + at); }
};

// Work buffers of adjoint_linalg, T elements: the inverse (zero above the
// diagonal) with G, S (also W, and the sums of G, [np / 64][np] in FP64) and
// the pieces of S
template <typename T>
struct AdjLinalg {
    T *A = nullptr, *S = nullptr, *part = nullptr;
};
static size_t adj_dense(int np)   // elements of the three
{
    return (size_t)np * (np + GT) + (size_t)np * np + (size_t)adj_round_pieces(np / GT) * GT * GT;
}

// u = D lam and v = B^T lam from the stored matrix M (D upper, B lower), then
// S = Z + Z^T with Z^T = Dbar = B^-T Phi(v X^T) B^-1
template <typename T>
static int adjoint_linalg(bdb_system* s, const T* M, int np, int n3, int nrb, int ncb, const double* lam,
                          double* colp, double* rowp, double* u, double* v, const double* Xp, const AdjLinalg<T>& w)
{
    cudaStream_t st = s->stream;
    const int smem = (int)sizeof(GemmSmem<T, GT>), lev_smem = (int)sizeof(GemmSmem<T, 64>);
    const int tri_smem = 2 * 64 * 65 * (int)sizeof(T);
    BDB_CUDA(cudaFuncSetAttribute(k_trinv64<T, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, tri_smem));
    BDB_CUDA(cudaFuncSetAttribute(k_tri_level<T, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, lev_smem));
    BDB_CUDA(cudaFuncSetAttribute(k_tri_level<T, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, lev_smem));
    BDB_CUDA(cudaFuncSetAttribute(k_adj_pieces<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    k_mv2<T><<<dim3(ncb, nrb), 256, 0, st>>>(M, n3, np, lam, colp, rowp);
    k_mv2_finish<<<(n3 + 255) / 256, 256, 0, st>>>(n3, nrb, ncb, colp, rowp, s->dD.p, lam, u, v);
    const size_t lda = (size_t)np + GT;
    double* sums = reinterpret_cast<double*>(w.S);
    k_trinv64<T, T><<<np / 64, 256, tri_smem, st>>>(M, np, w.A, lda);
    s->launches += 5;
    for (int h = 64; h < np; h *= 2) {
        const dim3 grid(h / 64, std::min(h, np - h) / 64, (np + h - 1) / (2 * h));
        k_tri_level<T, 0><<<grid, gemm_threads(64), lev_smem, st>>>(np, h, M, np, w.A, lda, w.S);
        k_tri_level<T, 1><<<grid, gemm_threads(64), lev_smem, st>>>(np, h, M, np, w.A, lda, w.S);
        s->launches += 2;
    }
    const dim3 cols((np + 127) / 128, np / 64);
    const int nb = np / GT;
    const GRows<T> G{w.A, lda, nb};
    k_phi_sums<T><<<cols, 128, 0, st>>>(np, Xp, w.A, lda, sums);
    k_phi_rows<T><<<cols, 128, 0, st>>>(np, v, Xp, w.A, lda, sums, G);
    for (int i0 = 0, i1; i0 < nb; i0 = i1) {
        i1 = adj_round_end(nb, i0);
        const int p0 = adj_pieces_before(nb, i0), p1 = adj_pieces_before(nb, i1);
        k_adj_pieces<T><<<p1 - p0, 256, smem, st>>>(np, p0, PlainRows<T>{w.A, lda}, G, w.part);
        k_adj_join<T><<<dim3(i1, i1 - i0, 16), 256, 0, st>>>(np, i0, p0, w.part, w.S);
        s->launches += 2;
    }
    BDB_CUDA(cudaGetLastError());
    return BDB_OK;
}

static int set_counter(bdb_system* s, unsigned long long v)
{
    const unsigned long long c[2] = {v, 0ull};
    BDB_CUDA(cudaMemcpyAsync(s->ctr.p, c, sizeof(c), cudaMemcpyHostToDevice, s->stream));
    return BDB_OK;
}

static int set_positions(bdb_system* s, const double4* src)
{
    BDB_CUDA(cudaMemcpyAsync(s->pos.p, src, sizeof(double4) * s->n, cudaMemcpyDeviceToDevice, s->stream));
    BDB_CUDA(cudaMemsetAsync(s->cells_built.p, 0, sizeof(int) * s->segs.size(), s->stream));
    s->have_forces = false;
    s->factor_valid = false;
    return BDB_OK;
}

}  // namespace bdb

using namespace bdb;

extern "C" int bdb_adjoint(bdb_system* s, int K, int checkpoint, int npairs, const int* pairs,
                           const double* targets, double* loss, double* grad_coord, double* grad_params)
{
    if (!s || K < 1 || checkpoint < 1 || npairs < 1 || !pairs || !targets || !loss || !grad_coord || !grad_params)
        return fail(BDB_ERR_ARG, "bad arguments");
    if (s->p.hydro != BDB_HYDRO_CHOLESKY || s->p.refresh != 1 || s->p.noise != BDB_NOISE_PHILOX || s->p.bc != 0 ||
        s->segs.size() != 1)
        return fail(BDB_ERR_UNSUPPORTED,
                    "the adjoint needs one free-space system, hydro cholesky, refresh 1 and device noise");
    const bool mixed = s->p.precision == BDB_PREC_MIXED;
    if (s->p.e_ext && s->p.e_type != 0)
        return fail(BDB_ERR_UNSUPPORTED, "the adjoint takes a constant (DC) external field only");
    if (s->n_angle || s->n_angle_cos || s->n_dihe || s->n_dihe_angle)
        return fail(BDB_ERR_UNSUPPORTED, "the adjoint covers bonds, LJ and Debye-Hueckel terms only");
    for (int p = 0; p < 2 * npairs; ++p)
        if (pairs[p] < 0 || pairs[p] >= s->n) return fail(BDB_ERR_ARG, "loss pair references a missing bead");
    const int n = s->n, n3 = s->n3, np = s->npad;
    const double c = s->p.dt / (BDB_KB * s->p.T);
    cudaStream_t st = s->stream;
    int rc;
    if ((rc = ensure_matrix(s))) return rc;
    // bead -> bond list (host CSR, fixed order)
    std::vector<int> bp_h(2 * std::max(1, s->n_bond)), bptr(n + 1, 0), blist;
    if (s->n_bond)
        BDB_CUDA(d2h(s, bp_h.data(), s->bond_pairs.p, sizeof(int) * 2 * s->n_bond));
    for (int t = 0; t < s->n_bond; ++t) {
        bptr[bp_h[2 * t] + 1]++;
        bptr[bp_h[2 * t + 1] + 1]++;
    }
    for (int i = 0; i < n; ++i) bptr[i + 1] += bptr[i];
    blist.resize(std::max(1, bptr[n]));
    {
        std::vector<int> fill(bptr.begin(), bptr.end() - 1);
        for (int t = 0; t < s->n_bond; ++t) {
            blist[fill[bp_h[2 * t]]++] = t;
            blist[fill[bp_h[2 * t + 1]]++] = t;
        }
    }
    const int nck = (K + checkpoint - 1) / checkpoint, seg_len = std::min(K, checkpoint);
    const int nrb = (n3 + MV2_ROWS - 1) / MV2_ROWS, ncb = (n3 + MV2_COLS - 1) / MV2_COLS;
    const size_t nn = (size_t)np * np, el = mixed ? sizeof(float) : sizeof(double);
    // one allocation for the matrices, vectors and lists, one for what is
    // kept. A call's time spreads with the driver's share of it: 40 calls at
    // n = 3072 in each of three processes had a median of 27.8 ms, means of 28,
    // 29 and 47 and slowest calls of 55, 57 and 718 ms; an allocation or free of
    // such a size by itself takes 0.4 to 0.8 ms, at times 100
    Part<double> lam, lam2, u, v, Xp, colp, rowp, ppart;
    Part<double4> ckpt, seg, xK;
    Part<int> d_bptr, d_blist;
    Scratch<unsigned char> vecs, kept;
    size_t bytes = 0;
    Part<unsigned char> dense;
    dense.place(bytes, adj_dense(np) * el), lam.place(bytes, np), lam2.place(bytes, np), u.place(bytes, np);
    v.place(bytes, np), Xp.place(bytes, np), colp.place(bytes, (size_t)nrb * n3 * 2);
    rowp.place(bytes, (size_t)ncb * n3), ppart.place(bytes, 4 * (size_t)n), ckpt.place(bytes, (size_t)nck * n);
    seg.place(bytes, (size_t)seg_len * n), xK.place(bytes, n);
    d_bptr.place(bytes, n + 1), d_blist.place(bytes, blist.size());
    if (vecs.alloc(bytes)) return fail(BDB_ERR_NOMEM, "adjoint scratch allocation failed");
    dense.set(vecs.p);
    for (Part<double>* q : {&lam, &lam2, &u, &v, &Xp, &colp, &rowp, &ppart}) q->set(vecs.p);
    for (Part<double4>* q : {&ckpt, &seg, &xK}) q->set(vecs.p);
    for (Part<int>* q : {&d_bptr, &d_blist}) q->set(vecs.p);
    // a segment's matrices and forces, where they fit in the bytes that the
    // caller allows (bdb_set_adjoint_keep), by default half of what is free
    bool keep = false;
    const size_t fbytes = (sizeof(double) * (size_t)seg_len * n3 + 255) / 256 * 256;
    const size_t kbytes = fbytes + (size_t)seg_len * nn * el;
    {
        size_t room = 0, total_b = 0;
        if (s->adjoint_keep >= 0) room = (size_t)s->adjoint_keep;
        else if (cudaMemGetInfo(&room, &total_b) == cudaSuccess) room /= 2;
        else room = 0;
        if (kbytes <= room) keep = !kept.alloc(kbytes);
        if (!keep) cudaGetLastError();   // too little room is no error: the steps are computed again
    }
    double* Fseg = reinterpret_cast<double*>(kept.p);
    unsigned char* Mseg = kept.p + fbytes;
    BDB_CUDA(h2d(s, d_bptr.p, bptr.data(), sizeof(int) * (n + 1)));
    BDB_CUDA(h2d(s, d_blist.p, blist.data(), sizeof(int) * blist.size()));
    BDB_CUDA(cudaMemsetAsync(dense.p, 0, (nn + (size_t)np * GT) * el, st));   // the inverse: zero above its diagonal
    BDB_CUDA(cudaMemsetAsync(ppart.p, 0, sizeof(double) * 4 * n, st));
    BDB_CUDA(cudaMemsetAsync(u.p, 0, sizeof(double) * np, st));
    BDB_CUDA(cudaMemsetAsync(v.p, 0, sizeof(double) * np, st));
    BDB_CUDA(cudaMemsetAsync(Xp.p, 0, sizeof(double) * np, st));
    BDB_CUDA(cudaMemsetAsync(lam.p, 0, sizeof(double) * np, st));
    BDB_CUDA(cudaMemsetAsync(lam2.p, 0, sizeof(double) * np, st));
    unsigned long long base = 0;
    BDB_CUDA(cudaMemcpyAsync(&base, s->ctr.p, sizeof(base), cudaMemcpyDeviceToHost, st));
    BDB_CUDA(cudaStreamSynchronize(st));
    BDB_CUDA(cudaMemsetAsync(s->status.p, 0, sizeof(unsigned), st));

    // one forward step from the current positions; slot >= 0: what its
    // reverse needs goes to that slot of the segment
    auto forward = [&](int slot) -> int {
        int r = 0;
        if (slot >= 0) {
            BDB_CUDA(cudaMemcpyAsync(seg.p + (size_t)slot * n, s->pos.p, sizeof(double4) * n, cudaMemcpyDeviceToDevice,
                                     st));
            if (keep) {
                if (!s->have_forces && (r = forces_run(s, false, false))) return r;
                BDB_CUDA(cudaMemcpyAsync(Fseg + (size_t)slot * n3, s->F.p, sizeof(double) * n3,
                                         cudaMemcpyDeviceToDevice, st));
            }
        }
        if ((r = engine_step(s))) return r;
        if (slot >= 0 && keep)   // refresh 1: the matrix still holds this step's D and B
            BDB_CUDA(cudaMemcpyAsync(Mseg + (size_t)slot * nn * el,
                                     mixed ? (const void*)s->M32.p : (const void*)s->M64.p, nn * el,
                                     cudaMemcpyDeviceToDevice, st));
        return BDB_OK;
    };
    // forward, keeping the positions at every checkpoint
    for (int k = 0; k < K; ++k) {
        if (k % checkpoint == 0)
            BDB_CUDA(cudaMemcpyAsync(ckpt.p + (size_t)(k / checkpoint) * n, s->pos.p, sizeof(double4) * n,
                                     cudaMemcpyDeviceToDevice, st));
        const int last0 = (nck - 1) * checkpoint;
        if ((rc = forward(k >= last0 ? k - last0 : -1))) return rc;
    }
    BDB_CUDA(cudaMemcpyAsync(xK.p, s->pos.p, sizeof(double4) * n, cudaMemcpyDeviceToDevice, st));

    // loss = mean over pairs of (|x_b - x_a| - target)^2 and its gradient
    std::vector<double4> xh(n);
    BDB_CUDA(cudaMemcpyAsync(xh.data(), s->pos.p, sizeof(double4) * n, cudaMemcpyDeviceToHost, st));
    BDB_CUDA(cudaStreamSynchronize(st));
    std::vector<double> lh(np, 0.0);
    double L = 0;
    for (int p = 0; p < npairs; ++p) {
        const int a = pairs[2 * p], b = pairs[2 * p + 1];
        const double d[3] = {xh[b].x - xh[a].x, xh[b].y - xh[a].y, xh[b].z - xh[a].z};
        const double r = std::sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
        const double dev = r - targets[p];
        L += dev * dev / npairs;
        for (int k = 0; k < 3; ++k) {
            const double g = 2 * dev / npairs * d[k] / r;
            lh[3 * b + k] += g;
            lh[3 * a + k] -= g;
        }
    }
    BDB_CUDA(cudaMemcpyAsync(lam.p, lh.data(), sizeof(double) * n3, cudaMemcpyHostToDevice, st));
    std::vector<double> gp(4, 0.0);
    AdjForce fp;
    fp.elec = s->p.elec;
    fp.epsilon_c = s->p.epsilon_c;
    fp.kappa_c = s->p.kappa_c;
    fp.gamma_c = s->p.gamma_c;
    fp.cutoff_c = s->p.cutoff_c;
    fp.alpha_lj = s->p.alpha_lj;
    fp.cutoff_lj = s->p.cutoff_lj;
    fp.lj6 = s->p.lj_6_term;
    fp.bond_lj_scale = s->p.bond_lj_scale;
    fp.bond_c_scale = s->p.bond_c_scale;
    fp.conn_live = s->conn_live;
    std::vector<double> pph(4 * (size_t)n);
    const int warps_blocks = (n * 32 + 255) / 256;

    // backward, one checkpoint segment at a time (recomputed forward, but for
    // the last)
    for (int sg = nck - 1; sg >= 0; --sg) {
        const int k0 = sg * checkpoint, k1 = std::min(K, k0 + checkpoint);
        if (sg < nck - 1) {
            if ((rc = set_positions(s, ckpt.p + (size_t)sg * n)) || (rc = set_counter(s, base + k0))) return rc;
            for (int k = k0; k < k1; ++k)
                if ((rc = forward(k - k0))) return rc;
        }
        for (int k = k1 - 1; k >= k0; --k) {
            // the forward quantities of step k: F(x_k), D(x_k), B(x_k), X_k
            const int slot = k - k0;
            const double4* x = seg.p + (size_t)slot * n;
            const double* Fk = keep ? Fseg + (size_t)slot * n3 : s->F.p;
            if (!keep && ((rc = set_positions(s, x)) || (rc = forces_run(s, false, false)) || (rc = tensor_build(s)) ||
                          (rc = factor_run(s))))
                return rc;
            if ((rc = set_counter(s, base + k)) || (rc = noise_fill(s, nullptr))) return rc;
            BDB_CUDA(cudaMemcpyAsync(Xp.p, s->X.p, sizeof(double) * n3, cudaMemcpyDeviceToDevice, st));
            // u = D lam, v = B^T lam; S = Z + Z^T with Z^T = Dbar = B^-T Phi(v X^T) B^-1;
            // lam_k = lam + c (dD/dx : F)^T lam + (d(BX)/dx)^T lam + c (dF/dx) u
            auto reverse = [&](auto type, const auto* M) -> int {
                using T = decltype(type);
                AdjLinalg<T> w;
                w.A = reinterpret_cast<T*>(dense.p);
                w.S = w.A + nn + (size_t)np * GT;
                w.part = w.S + nn;
                const T* Mk = keep ? reinterpret_cast<const T*>(Mseg) + (size_t)slot * nn : M;
                const int r = adjoint_linalg<T>(s, Mk, np, n3, nrb, ncb, lam.p, colp.p, rowp.p, u.p, v.p, Xp.p, w);
                if (r) return r;
                BDB_CUDA(cudaMemcpyAsync(lam2.p, lam.p, sizeof(double) * n3, cudaMemcpyDeviceToDevice, st));
                k_tile_grad<T><<<warps_blocks, 256, 0, st>>>(n, x, s->preDii, s->preDij, c, lam.p, Fk, w.S, np, lam2.p);
                return BDB_OK;
            };
            rc = mixed ? reverse(0.0f, (const float*)s->M32.p) : reverse(0.0, (const double*)s->M64.p);
            if (rc) return rc;
            k_force_jvp<<<warps_blocks, 256, 0, st>>>(n, fp, x, s->Q.p, s->LJ.p, s->conn_ptr.p,
                                                     s->conn_list.p, d_bptr.p, d_blist.p, s->bond_pairs.p,
                                                     s->bond_parms.p, u.p, c, lam2.p, ppart.p);
            BDB_CUDA(cudaGetLastError());
            s->launches += 3;
            std::swap(lam.p, lam2.p);
        }
    }
    BDB_CUDA(cudaMemcpyAsync(pph.data(), ppart.p, sizeof(double) * 4 * n, cudaMemcpyDeviceToHost, st));
    BDB_CUDA(cudaStreamSynchronize(st));
    for (int i = 0; i < n; ++i)
        for (int q = 0; q < 4; ++q) gp[q] += pph[4 * (size_t)i + q];
    BDB_CUDA(cudaMemcpyAsync(grad_coord, lam.p, sizeof(double) * n3, cudaMemcpyDeviceToHost, st));
    if ((rc = set_positions(s, xK.p)) || (rc = set_counter(s, base + K))) return rc;
    unsigned stw = 0;
    BDB_CUDA(cudaMemcpyAsync(&stw, s->status.p, sizeof(unsigned), cudaMemcpyDeviceToHost, st));
    BDB_CUDA(cudaStreamSynchronize(st));
    if (stw & ST_NOT_SPD) return fail(BDB_ERR_NOT_SPD, "Cholesky decomposition error: non-positive pivot");
    if (stw & ST_BOND) return fail(BDB_ERR_BOND, "Overstretched bond (bond.c:73-78)");
    for (int q = 0; q < 4; ++q) grad_params[q] = gp[q];
    *loss = L;
    return BDB_OK;
}

extern "C" int bdb_set_adjoint_keep(bdb_system* s, long long bytes)
{
    if (!s) return fail(BDB_ERR_ARG, "null system");
    s->adjoint_keep = bytes < 0 ? -1 : bytes;
    return BDB_OK;
}
