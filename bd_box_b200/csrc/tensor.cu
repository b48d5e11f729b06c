// Diffusion tensor on the device.
//
// k_build: the stored 3N x 3N tensor of compute_D (diff_tensor.c:472-544)
//    for the Cholesky path. One CTA per 32x32-bead tile (I >= J) evaluates
//    the 1024 RPY tiles into shared memory and writes the 96x96 block twice
//    with coalesced rows: as rows of block (I, J) below the diagonal and,
//    transposed through shared memory, as rows of block (J, I) above it.
//    The factorisation later overwrites the lower triangle with L; the upper
//    triangle keeps D (the reference keeps Ds and S separately,
//    diff_rand.c:76-82). The diagonal of D goes to dD.
// The matrix-free pair sums (D.F, TEA noise) are in tea.cu.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "bdb_common.cuh"
#include "ewald_fast.cuh"
#include "tensor_args.cuh"

namespace bdb {

static constexpr int TB = 32;   // beads per tile

// Constants of a system's Ewald sums (no device data).
static EwaldConst system_ewald(const bdb_system* s)
{
    EwaldConst e;
    if (!s->p.ewald) return e;
    e.smith = s->p.ewald_method == BDB_EWALD_SMITH;
    e.R = s->p.ewald_real;
    e.L = s->p.box[0];
    e.inv_L = s->inv_L[0];
    e.alpha = e.smith && s->p.ewald_alpha > 0 ? s->p.ewald_alpha : BDB_SQRTPI;
    e.a2 = e.alpha * e.alpha;
    e.isp = e.smith ? BDB_M1_SQRTPI : 1 / BDB_SQRTPI;
    // of the images' polynomials (diff_tensor.c:336-356): a multiple of
    // alpha^n / sqrt(pi) each
    const long double a = e.alpha, a2 = a * a;
    const long double p1 = e.smith ? a * (long double)BDB_M1_SQRTPI : a / (long double)BDB_SQRTPI;
    const long double p3 = p1 * a2, p5 = p3 * a2, p7 = p5 * a2;
    e.e2 = (double)(2 * p1);
    e.as = (double)p1;
    e.c0[0] = (double)(-4.5L * p1);
    e.c0[1] = (double)(14 * p3);
    e.c1[0] = (double)(3 * p3);
    e.c1[1] = (double)(-20 * p5);
    e.c2 = (double)(4 * p7);
    e.d0[0] = (double)(1.5L * p1);
    e.d0[1] = (double)(-2 * p3);
    e.d1[0] = (double)(-3 * p3);
    e.d1[1] = (double)(16 * p5);
    volatile float pif = BDB_M_PIF;
    volatile float two = 2 * pif;
    e.two_pif = two;
    e.kappa = std::exp(-2 * e.a2);
    for (int q = 0; q <= e.R * e.R; ++q) e.extent[q] = (signed char)std::sqrt((double)(e.R * e.R - q));
    // images beyond 2.5 L (Beenakker), 4.45/alpha (Smith): erfc ~ 3e-10
    const double rc = e.smith ? 4.45 / e.alpha : 2.5;
    e.rcut_sq = (float)(rc * rc);
    return e;
}

// the reciprocal weights I and e e^T of a vector of |k|^2 = k_sq: {I, ee} and
// the same of the terms in s2. The k-only factors are the reference's
// (diff_tensor.c:360-395, :206-239), with its float constants; Beenakker's
// k^2/alpha^2 is formed there as (2 pi_f k)^2 over alpha^2 = pi/L^2, which
// leaves weights of exp(-pi L^2 k^2): zero for boxes above ~15.
static void recip_weights(const EwaldConst& ec, double k_sq, double* w)
{
    volatile float pif = BDB_M_PIF;
    if (ec.smith) {
        volatile float npif2 = -pif * pif;
        volatile float four_pif = 4 * pif;
        const double m = (double)npif2 / ec.a2 * k_sq;
        const double ex = std::exp(m);
        const double A = 2 * ex / ((double)pif * k_sq);
        w[0] = 0.75 * A;
        w[1] = 0.75 * A * (-1 + m);
        w[2] = 0;
        w[3] = 0.5 * (double)four_pif * ex;
    } else {
        volatile float four = 4 * pif;
        volatile float four2 = four * pif;
        volatile float six = 6 * pif;
        const double k2 = k_sq * (double)four2;
        const double alpha = ec.alpha * ec.inv_L, ia2 = 1.0f / (alpha * alpha);
        double P = 1 + (ia2 * k2 / 4) * (1 + ia2 * k2 / 2);
        P *= (double)six * std::exp(-ia2 * k2 / 4) / k2;
        w[0] = P * ec.inv_L * ec.inv_L;
        w[1] = -w[0];
        w[2] = -k2 / 3 * P;
        w[3] = -w[2];
    }
}

// Real-space scalars of an image (RealSpace::image) on the host, the parts
// without and with s2: A0, B0, A1, B1
static void real_scalars(const EwaldConst& ec, double r2, double* q)
{
    const double a = ec.alpha, a3 = a * ec.a2, a5 = a3 * ec.a2, a7 = a5 * ec.a2;
    const double r = std::sqrt(r2), i = 1 / r, i2 = 1 / r2;
    const double ex = std::exp(-ec.a2 * r2), er = std::erfc(a * r) * i;
    if (ec.smith) {
        const double E = 2 * a * ec.isp * ex, sq = i2 * (er + E);
        q[0] = 0.75 * er;
        q[1] = 0.75 * (er + E) * i2;
        q[2] = 0.5 * sq;
        q[3] = 0.5 * (-3 * sq - 2 * ec.a2 * E) * i2;
    } else {
        const double g = ec.isp * ex;
        q[0] = (-4.5 * a + 3 * a3 * r2) * g + 0.75 * er;
        q[1] = ((1.5 * a - 3 * a3 * r2) * g + 0.75 * er) * i2;
        q[2] = (a * i2 + 14 * a3 - 20 * a5 * r2 + 4 * a7 * r2 * r2) * g + 0.5 * er * i2;
        q[3] = ((-3 * a * i2 - 2 * a3 + 16 * a5 * r2 - 4 * a7 * r2 * r2) * g - 1.5 * er * i2) * i2;
    }
}

// S(v) of the reference on the host, v in L (raw), s2 = sigma^2/L^2: the
// sphere of images and the reciprocal sum
static void reference_sum(const EwaldConst& ec, const double* v, double s2, double* S)
{
    const int R = ec.R;
    for (int k = 0; k < 6; ++k) S[k] = 0;
    for (int h = -R; h <= R; ++h)
        for (int f = -R; f <= R; ++f)
            for (int g = -R; g <= R; ++g) {
                const int m2 = h * h + f * f + g * g;
                if (m2 > R * R) continue;
                const double x[3] = {v[0] + h, v[1] + f, v[2] + g};
                double q[4], A = 0, B = 0;
                real_scalars(ec, x[0] * x[0] + x[1] * x[1] + x[2] * x[2], q);
                A = q[0] + s2 * q[2];
                B = q[1] + s2 * q[3];
                S[0] += A + B * x[0] * x[0];
                S[1] += A + B * x[1] * x[1];
                S[2] += A + B * x[2] * x[2];
                S[3] += B * x[0] * x[1];
                S[4] += B * x[0] * x[2];
                S[5] += B * x[1] * x[2];
                if (m2 == 0) continue;
                recip_weights(ec, m2, q);
                const double cs = std::cos(ec.two_pif * (v[0] * h + v[1] * f + v[2] * g));
                const double ci = (q[0] + s2 * q[2]) * cs, ce = (q[1] + s2 * q[3]) * cs / m2;
                S[0] += ci + ce * h * h;
                S[1] += ci + ce * f * f;
                S[2] += ci + ce * g * g;
                S[3] += ce * h * f;
                S[4] += ce * h * g;
                S[5] += ce * f * g;
            }
}

// Fourier weights {I, ee} at |k|^2 = k_sq of the converged split (see
// ewald_fast.cuh), on top of the near part
static void fast_weights(const EwaldConst& ec, double k_sq, double s2, double* w)
{
    const double b = EF_SPLIT * BDB_SQRTPI, y = BDB_PI_D * BDB_PI_D * k_sq / (b * b), ex = std::exp(-y);
    w[0] = 1.5 * ex / (BDB_PI_D * k_sq);
    w[1] = -w[0] * (1 + y) + 2 * BDB_PI_D * s2 * ex;
    if (ec.smith) return;
    // Beenakker's screening of the same tensor at alpha = sqrt(pi)/L, whose
    // real-space sum the reference takes, and the reference's reciprocal sum
    const double k2 = 4 * BDB_PI_D * BDB_PI_D * k_sq, x = k2 / (4 * ec.a2);
    const double P = (1 + x + 2 * x * x) * 6 * BDB_PI_D * std::exp(-x) / k2 * (1 - s2 * k2 / 3);
    w[0] -= P;
    w[1] += P;
    if (k_sq <= ec.R * ec.R) {
        double q[4];
        recip_weights(ec, k_sq, q);
        w[0] += q[0] + s2 * q[2];
        w[1] += q[1] + s2 * q[3];
    }
}

// The converged split for a mixed system, or nothing (false) where the
// reference's truncated sums differ from it. The sphere of images truncates
// first for separations far apart in the box, so the two are compared there:
// at |v| = 1.5 and within (they must agree to 2e-7 in preDii/L, where the tile
// is ~1 and its FP32 rounding in the reference's split ~7e-7), then in the
// box's corners, without which the split covers |v| <= 1.5 only. At the
// default alpha, Beenakker: 2.4e-8 at R = 4 within 1.5 (1e-5 in the
// corners), 2.5e-4 at R = 3.
static bool ewald_fast_setup(const bdb_system* s, EwaldFast* E)
{
    const EwaldConst ec = system_ewald(s);
    const double a = s->radius0, s2 = a * a * ec.inv_L * ec.inv_L, b = EF_SPLIT * BDB_SQRTPI;
    if (!(s2 < 0.25)) return false;
    static const double pt[10][3] = {{0.31, 0.17, 0.23},   {0.49, 0.48, 0.47},    {0.97, 0.03, 0.99}, {0.07, 0.04, 0.09},
                                     {0.97, 0.81, -0.81},  {-0.99, -0.99, 0.53},  {0.866, 0.866, 0.866},
                                     {0.96, -0.97, 0.98},  {-0.995, -0.99, 0.999}, {0.99, 0.98, -0.7}};
    static const int corner0 = 7;   // the last three lie beyond 1.5
    double dev[10][6], C = 0;
    std::vector<double> w;
    for (int h = 0; h <= EF_K; ++h)
        for (int f = 0; f <= EF_K; ++f)
            for (int g = 0; g <= EF_K; ++g) {
                const int m2 = h * h + f * f + g * g;
                if (m2 > EF_K2) continue;
                double q[6] = {0, 0, 0, 0, 0, 0}, c[2];
                if (m2) {
                    const double mult = (h ? 2.0 : 1.0) * (f ? 2.0 : 1.0) * (g ? 2.0 : 1.0);
                    fast_weights(ec, m2, s2, c);
                    q[0] = mult * (c[0] + c[1] * h * h / m2);
                    q[1] = mult * (c[0] + c[1] * f * f / m2);
                    q[2] = mult * (c[0] + c[1] * g * g / m2);
                    q[3] = -mult * c[1] * h * f / m2;
                    q[4] = -mult * c[1] * h * g / m2;
                    q[5] = -mult * c[1] * f * g / m2;
                }
                w.insert(w.end(), q, q + 6);
            }
    EwaldConst near;   // Smith's real-space functions at the split's screening
    near.smith = 1;
    near.alpha = b;
    near.a2 = b * b;
    near.isp = 1 / BDB_SQRTPI;
    for (int p = 0; p < 10; ++p) {
        double S[6], o[6] = {0, 0, 0, 0, 0, 0}, u[3], sg[3];
        reference_sum(ec, pt[p], s2, S);
        for (int k = 0; k < 3; ++k) {
            u[k] = pt[p][k] - std::rint(pt[p][k]);
            sg[k] = u[k] < 0 ? -1 : 1;
            u[k] = std::fabs(u[k]);
        }
        for (int m = 0; m < 8; ++m) {
            const double x[3] = {u[0] - (m & 1), u[1] - ((m >> 1) & 1), u[2] - (m >> 2)};
            double q[4];
            real_scalars(near, x[0] * x[0] + x[1] * x[1] + x[2] * x[2], q);
            const double A = q[0] + s2 * q[2], B = q[1] + s2 * q[3];
            for (int k = 0; k < 3; ++k) o[k] += A + B * x[k] * x[k];
            o[3] += B * x[0] * x[1];
            o[4] += B * x[0] * x[2];
            o[5] += B * x[1] * x[2];
        }
        size_t n = 0;
        const double tp = 2 * BDB_PI_D;
        for (int h = 0; h <= EF_K; ++h)
            for (int f = 0; f <= EF_K; ++f)
                for (int g = 0; g <= EF_K; ++g) {
                    if (h * h + f * f + g * g > EF_K2) continue;
                    const double cx = std::cos(tp * h * u[0]), sx = std::sin(tp * h * u[0]), cy = std::cos(tp * f * u[1]),
                                 sy = std::sin(tp * f * u[1]), cz = std::cos(tp * g * u[2]), sz = std::sin(tp * g * u[2]);
                    const double* q = &w[n];
                    for (int k = 0; k < 3; ++k) o[k] += q[k] * cx * cy * cz;
                    o[3] += q[3] * sx * sy * cz;
                    o[4] += q[4] * sx * cy * sz;
                    o[5] += q[5] * cx * sy * sz;
                    n += 6;
                }
        o[3] *= sg[0] * sg[1];
        o[4] *= sg[0] * sg[2];
        o[5] *= sg[1] * sg[2];
        for (int k = 0; k < 6; ++k) dev[p][k] = S[k] - o[k];
        for (int k = 0; k < 3 && p < corner0; ++k) C += dev[p][k] / (3 * corner0);
    }
    bool corners = true;
    for (int p = 0; p < 10; ++p)
        for (int k = 0; k < 6; ++k)
            if (!(std::fabs(dev[p][k] - (k < 3 ? C : 0.0)) < 2e-7)) {
                if (p < corner0) return false;
                corners = false;
            }
    for (size_t q = 0; q < w.size(); ++q) E->w[q / 6][q % 6] = (float)w[q];
    E->beta = (float)b;
    E->b2 = (float)(b * b);
    E->e2 = (float)(2 * b / BDB_SQRTPI);
    E->hs = (float)(0.5 * s2);
    E->diag = (float)C;
    E->radius = (float)a;
    const Gauss32 gauss(b * b);
    E->g_hi = gauss.hi;
    E->g_lo = gauss.lo;
    E->near_sq = (float)(4 * s2);
    E->far_sq = corners ? 3.01f : 2.25f;
    E->pre = (float)(s->preDii * ec.inv_L);
    return true;
}

// The reciprocal weight table and a bead's sum over its own images, once per
// system (see EwaldConst)
int ewald_tables(bdb_system* s)
{
    if (!s->p.ewald || s->ewald_tab.p) return BDB_OK;
    const EwaldConst ec = system_ewald(s);
    const int R = ec.R;
    std::vector<double> rk;
    double self0 = 0, self1 = 0;
    bool any = false;
    for (int h = 0; h <= R; ++h)
        for (int f = 0; f <= ec.extent[h * h]; ++f)
            for (int g = 0; g <= ec.extent[h * h + f * f]; ++g) {
                double w[12] = {0};
                const double k_sq = (double)(h * h + f * f + g * g);
                if (k_sq > 0) {
                    const double mult = (h ? 2.0 : 1.0) * (f ? 2.0 : 1.0) * (g ? 2.0 : 1.0);
                    const double ik = 1 / std::sqrt(k_sq), e[3] = {h * ik, f * ik, g * ik};
                    double c[4];
                    recip_weights(ec, k_sq, c);
                    for (int q = 0; q < 2; ++q) {
                        for (int k = 0; k < 3; ++k) w[6 * q + k] = mult * (c[2 * q] + c[2 * q + 1] * e[k] * e[k]);
                        // cos of a sum with both signs of two axes: -sin sin
                        w[6 * q + 3] = -mult * c[2 * q + 1] * e[0] * e[1];
                        w[6 * q + 4] = -mult * c[2 * q + 1] * e[0] * e[2];
                        w[6 * q + 5] = -mult * c[2 * q + 1] * e[1] * e[2];
                    }
                    self0 += w[0];
                    self1 += w[6];
                    // the sphere's images of a bead itself: mean of the three axes
                    double q[4];
                    real_scalars(ec, k_sq, q);
                    self0 += mult * (q[0] + q[1] * h * h);
                    self1 += mult * (q[2] + q[3] * h * h);
                }
                for (double x : w) any = any || x != 0.0;
                rk.insert(rk.end(), w, w + 12);
            }
    if (s->ewald_tab.alloc(rk.size())) return BDB_ERR_NOMEM;
    BDB_CUDA(h2d(s, s->ewald_tab.p, rk.data(), sizeof(double) * rk.size()));
    s->ewald_self[0] = self0;
    s->ewald_self[1] = self1;
    s->ewald_recip = any;
    if (s->p.precision != BDB_PREC_FP64) {
        s->ewald_fast = std::make_shared<EwaldFast>();
        if (!ewald_fast_setup(s, s->ewald_fast.get())) s->ewald_fast.reset();
    }
    return BDB_OK;
}

TensorArgs targs(const bdb_system* s)
{
    TensorArgs a;
    a.n = s->n;
    a.npad = s->npad;
    a.preDii = s->preDii;
    a.preDij = s->preDij;
    a.ewald = s->p.ewald;
    a.ec = system_ewald(s);
    a.ec.rk = s->ewald_tab.p;
    a.ec.recip = s->ewald_recip;
    a.ec.self0 = s->ewald_self[0];
    a.ec.self1 = s->ewald_self[1];
    return a;
}

// One CTA per pair of 32-bead blocks (I >= J): the 96x96 tile of D in
// shared memory, then stored straight and (off the diagonal) transposed,
// both triangles, one warp per matrix row so that every store of a warp is
// one contiguous run of the row. The free-space variant (kEwald false)
// carries none of the Ewald code, so it keeps few registers and several
// CTAs per SM.
template <typename T, bool kEwald>
__global__ void __launch_bounds__(256) k_build(TensorArgs A, const double4* __restrict__ pos, T* __restrict__ M,
                                               double* __restrict__ dD)
{
    extern __shared__ __align__(16) unsigned char build_smem[];
    T(*tile)[3 * TB + 1] = reinterpret_cast<T(*)[3 * TB + 1]>(build_smem);
    const int I = blockIdx.y, J = blockIdx.x;
    if (J > I) return;
    const int tid = threadIdx.x;
    const int n3 = 3 * A.n;
    for (int p = tid; p < TB * TB; p += blockDim.x) {
        const int li = p / TB, lj = p % TB;
        const int i = I * TB + li, j = J * TB + lj;
        T t[6] = {0, 0, 0, 0, 0, 0};
        if (i < A.n && j < A.n) tile_of_k<T, kEwald>(A, pos, i, j, t);
        const int r = 3 * li, c = 3 * lj;
        tile[r][c] = t[0];
        tile[r + 1][c + 1] = t[1];
        tile[r + 2][c + 2] = t[2];
        tile[r][c + 1] = tile[r + 1][c] = t[3];
        tile[r][c + 2] = tile[r + 2][c] = t[4];
        tile[r + 1][c + 2] = tile[r + 2][c + 1] = t[5];
    }
    __syncthreads();
    const int r0 = 3 * TB * I, c0 = 3 * TB * J;
    const int warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
    const int rows = min(3 * TB, n3 - r0), cols = min(3 * TB, n3 - c0);
    for (int r = warp; r < rows; r += nw) {
        T* dst = M + (size_t)(r0 + r) * A.npad + c0;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int c = lane + 32 * k;
            if (c < cols) dst[c] = tile[r][c];
        }
    }
    if (I != J) {
        for (int c = warp; c < cols; c += nw) {
            T* dst = M + (size_t)(c0 + c) * A.npad + r0;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int r = lane + 32 * k;
                if (r < rows) dst[r] = tile[r][c];
            }
        }
    } else {
        for (int r = tid; r < 3 * TB; r += blockDim.x)
            if (r0 + r < n3) dD[r0 + r] = (double)tile[r][r];
    }
}

template <typename T>
static size_t build_smem_bytes()
{
    return sizeof(T) * 3 * TB * (3 * TB + 1);
}


static int tensor_attrs();

int tensor_build(bdb_system* s)
{
    int rc = tensor_attrs();
    if (rc) return rc;
    if (int rc_e = ewald_tables(s)) return rc_e;
    const TensorArgs A = targs(s);
    const int nt = (s->n + TB - 1) / TB;
    dim3 grid(nt, nt);
    if (s->p.precision == BDB_PREC_FP64) {
        if (A.ewald)
            k_build<double, true><<<grid, 256, build_smem_bytes<double>(), s->stream>>>(A, s->pos.p, s->M64.p, s->dD.p);
        else
            k_build<double, false><<<grid, 256, build_smem_bytes<double>(), s->stream>>>(A, s->pos.p, s->M64.p,
                                                                                        s->dD.p);
    } else {
        if (A.ewald)
            k_build<float, true><<<grid, 256, build_smem_bytes<float>(), s->stream>>>(A, s->pos.p, s->M32.p, s->dD.p);
        else
            k_build<float, false><<<grid, 256, build_smem_bytes<float>(), s->stream>>>(A, s->pos.p, s->M32.p, s->dD.p);
    }
    s->launches += 1;
    BDB_CUDA(cudaGetLastError());
    return BDB_OK;
}

__global__ void k_one_tile(TensorArgs A, const double4* pos, int i, int j, double* out)
{
    double t[6];
    tile_of<double>(A, pos, i, j, t);
    out[0] = t[0];
    out[4] = t[1];
    out[8] = t[2];
    out[1] = out[3] = t[3];
    out[2] = out[6] = t[4];
    out[5] = out[7] = t[5];
}

int tensor_tile_host(bdb_system* s, int i, int j, double* tD)
{
    if (int rc_e = ewald_tables(s)) return rc_e;
    const TensorArgs A = targs(s);
    double* d = s->work.p;
    k_one_tile<<<1, 1, 0, s->stream>>>(A, s->pos.p, i, j, d);
    BDB_CUDA(cudaGetLastError());
    BDB_CUDA(cudaMemcpyAsync(tD, d, 9 * sizeof(double), cudaMemcpyDeviceToHost, s->stream));
    BDB_CUDA(cudaStreamSynchronize(s->stream));
    return BDB_OK;
}

static int tensor_attrs()
{
    static bool done = false;
    if (done) return BDB_OK;
    BDB_CUDA(cudaFuncSetAttribute(k_build<double, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)build_smem_bytes<double>()));
    BDB_CUDA(cudaFuncSetAttribute(k_build<double, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)build_smem_bytes<double>()));
    BDB_CUDA(cudaFuncSetAttribute(k_build<float, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)build_smem_bytes<float>()));
    BDB_CUDA(cudaFuncSetAttribute(k_build<float, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)build_smem_bytes<float>()));
    done = true;
    return BDB_OK;
}

}  // namespace bdb
