// RPY diffusion-tensor tiles, shared by the stored-D build and the
// matrix-free D.F / TEA kernels.
//
// A tile is the symmetric 3x3 block D_ij, kept as 6 values
// {xx, yy, zz, xy, xz, yz}.
//  * rpy_free: diff_tensor_calc_pos (diff_alg/diff_tensor.c:45-92), the
//    free-space Rotne-Prager-Yamakawa tensor with the overlap form for
//    r < a_i + a_j.
//  * rpy_ewald: the lattice sums of diff_tensor_calc_ewald_beenakker
//    (diff_tensor.c:265-401) and diff_tensor_calc_ewald_smith (:102-243) with
//    their self terms (:404-422, :245-263): real-space images r + L m and
//    reciprocal vectors over the same sphere |m|^2 <= R^2, overlap correction
//    on the raw (not minimum-image) separation. Beenakker's alpha is
//    sqrt(pi)/L (init_tensor, :546-559), Smith's ewald_alpha/L. Constants that
//    the reference forms from the float literal M_PIF are formed the same way
//    on the host.
//
// The sums are evaluated in units of L: v = r/L, s2 = sigma^2/L^2 and the
// dimensionless alpha; the tile is preDii/L times the sum.
#pragma once

#include <type_traits>

#include "bdb_common.cuh"

namespace bdb {

// 1/sqrt(pi) as the reference's double build spells it (data.h:228)
#define BDB_M1_SQRTPI 0.5641895835

static constexpr int EWALD_MAX_R = 5;

struct EwaldConst {
    int smith = 0, R = 0;
    double L = 0, inv_L = 0;
    double alpha = 0, a2 = 0;       // alpha L and its square
    double isp = 0;                 // 1/sqrt(pi), spelled as each method spells it
    // RealSpace's constants, [0] + [1] sigma^2/L^2, each rounded once from
    // extended precision: their rounding is the same in every image of every
    // pair, and with it the tensor's mean
    double e2 = 0, as = 0, c0[2] = {0, 0}, c1[2] = {0, 0}, c2 = 0, d0[2] = {0, 0}, d1[2] = {0, 0};
    double two_pif = 0;             // 2*M_PIF evaluated in float
    double kappa = 0;               // exp(-2 a2): second ratio of the Gaussian along an axis
    // isqrt(R^2 - q), the extent of a row of the sphere, for q = 0 .. R^2
    signed char extent[EWALD_MAX_R * EWALD_MAX_R + 1] = {};
    // reciprocal weights (device memory), see ewald_tables: for h, f, g >= 0
    // in the sphere, 12 values: the coefficients of xx, yy, zz (with
    // cos cos cos), xy (sin sin cos), xz (sin cos sin), yz (cos sin sin), then
    // the same of the terms in s2. recip is 0 when every weight is zero.
    const double* rk = nullptr;
    int recip = 0;
    // the lattice sum of a bead with its own images: self0 + self1 s2
    double self0 = 0, self1 = 0;
    float rcut_sq = 0;              // mixed precision: images beyond this are dropped (erfc ~ 3e-10)
};

// 1/sqrt(x) for normal x: the hardware's estimate and Newton-Raphson steps in
// residual form, y <- y + y/2 (1 - x y^2). FP64: the estimate has ~20 bits, two
// steps leave its rounding (1 ulp). FP32: one step, 0.8 ulp against 2 of the
// estimate; inv_sqrt_half, for the free-space tile, which takes its cube, puts
// the rounding of x y back as well: 0.5 ulp.
__device__ __forceinline__ double inv_sqrt(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    y = fma(0.5 * y, fma(-(x * y), y, 1.0), y);
    return fma(0.5 * y, fma(-(x * y), y, 1.0), y);
}
__device__ __forceinline__ float inv_sqrt(float x)
{
    const float y = rsqrtf(x);
    return fmaf(0.5f * y, fmaf(-(x * y), y, 1.0f), y);
}
__device__ __forceinline__ double inv_sqrt_half(double x) { return inv_sqrt(x); }
__device__ __forceinline__ float inv_sqrt_half(float x)
{
    const float y = rsqrtf(x), p = x * y;
    return fmaf(0.5f * y, fmaf(-fmaf(x, y, -p), y, fmaf(-p, y, 1.0f)), y);
}

// A squared separation that has overflowed (beads 1.8e19 apart in FP32, 1.3e154
// in FP64) as the largest finite number, or the residual above is inf * 0: the
// tile is then as good as zero, not NaN. One integer (FP64) or minimum
// operation a pair; a NaN stays one through the separation itself.
__device__ __forceinline__ float below_inf(float x) { return fminf(x, 3.402823466e38f); }
__device__ __forceinline__ double below_inf(double x)
{
    return __hiloint2double(min(__double2hiint(x), 0x7fefffff), __double2loint(x));
}

// diff_tensor_calc_pos(i, j) from the separation d = r_i - r_j and the two
// radii (which enter symmetrically): A I + B d d^T, with one reciprocal
// square root instead of a square root and four divisions.
template <typename T>
__device__ __forceinline__ void rpy_free_sep(const T* d, T si, T sj, T preDii, T preDij, T* t)
{
    const T r_sq = below_inf(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
    const T inv = inv_sqrt_half(r_sq);
    const T inv_sq = inv * inv, r = r_sq * inv;
    T A, B;
    if (r < si + sj) {
        const T sigma = (si + sj) / 2;
        const T pre = preDii / sigma;
        const T q = r / (32 * sigma);
        A = (1 - 9 * q) * pre;
        B = 3 * q * pre * inv_sq;
    } else {
        const T pre = preDij * inv;
        const T sigm_r = (si * si + sj * sj) * inv_sq;
        A = (1 + sigm_r * ((T)1 / 3)) * pre;
        B = (1 - sigm_r) * pre * inv_sq;
    }
    const T bx = B * d[0], by = B * d[1], bz = B * d[2];
    t[0] = A + bx * d[0];
    t[1] = A + by * d[1];
    t[2] = A + bz * d[2];
    t[3] = bx * d[1];
    t[4] = bx * d[2];
    t[5] = by * d[2];
}

template <typename T>
__device__ __forceinline__ void rpy_free(const double4& pi, const double4& pj, T preDii, T preDij, T* t)
{
    const T d[3] = {(T)(pi.x - pj.x), (T)(pi.y - pj.y), (T)(pi.z - pj.z)};
    rpy_free_sep<T>(d, (T)pi.w, (T)pj.w, preDii, preDij, t);
}

// ---- the scaled complementary error function, erfcx(x) = exp(x^2) erfc(x),
// for x >= 0: (1 + 2x) erfcx(x) as a polynomial in t = (x - K)/(x + K), the
// transformation of Shepherd and Laframboise (Math. Comp. 36, 249 (1981)).
// The coefficients are Chebyshev interpolants at K = 3.5 (FP64, 1.2e-16 on
// x >= 0) and K = 2.5 (FP32, 1.2e-7 on 0 <= x <= 9), computed in 50 digits.
// One reciprocal serves both quotients: d = 1/((x + K)(1 + 2x)).
// constant memory: a constant operand of the multiply-add, where a 64-bit
// immediate would take two more instructions
static __constant__ double kErfcx64[24] = {
    1.2423492448711544, -0.1400091801376197, -0.010555596332221669, 0.09751909515328706,
    -0.11508959816003075, 0.08798315382403678, -0.04882332583088402, 0.019099330953271165,
    -0.004215019879774186, -0.0003022679534333239, 0.0005643842668705102, -0.00012151212091980101,
    -4.2781739959539994e-05, 2.4260300984917994e-05, 2.3273309537791425e-06, -3.814012584490695e-06,
    -4.309237398316666e-08, 6.014823849950426e-07, -8.611571571113718e-09, -9.64004253144383e-08,
    6.651894382376532e-10, 1.3624442778701048e-08, 6.040390099342991e-11, -1.1656687889203665e-09};
__device__ __forceinline__ double erfcx_pos(double x)
{
    const double p = x + 3.5, q = fma(2.0, x, 1.0), pq = p * q;
    double d;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(d) : "d"(pq));
    d = fma(d, fma(-pq, d, 1.0), d);
    d = fma(d, fma(-pq, d, 1.0), d);
    const double t = (x - 3.5) * (q * d);
    // even and odd powers side by side: two chains of 11 instead of one of 23
    const double u = t * t;
    double e = kErfcx64[22], o = kErfcx64[23];
#pragma unroll
    for (int k = 20; k >= 0; k -= 2) {
        e = fma(e, u, kErfcx64[k]);
        o = fma(o, u, kErfcx64[k + 1]);
    }
    const double r = fma(o, t, e);
    return r * (p * d);
}
__device__ __forceinline__ float erfcx_pos(float x)
{
    const float p = x + 2.5f, q = fmaf(2.0f, x, 1.0f);
    float d;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(d) : "f"(p * q));
    const float t = (x - 2.5f) * (q * d);
    float r = 0.0004457839258919816f;
    r = fmaf(r, t, 0.00030503612796383756f);
    r = fmaf(r, t, -0.004302876907248387f);
    r = fmaf(r, t, 0.0010337509324308317f);
    r = fmaf(r, t, 0.03274950128568062f);
    r = fmaf(r, t, -0.1029877887892802f);
    r = fmaf(r, t, 0.15763045854613184f);
    r = fmaf(r, t, -0.09902309465772124f);
    r = fmaf(r, t, -0.12235677564486401f);
    r = fmaf(r, t, 1.2648381682779481f);
    return r * (p * d);
}

// exp(-a2 r2) in FP32 for a2 = -(hi + lo) ln 2: the exponent's rounding error
// is put back, so that the hardware's exp2 (2 ulp) is what is left of it --
// __expf loses |a2 r2| half-ulps, 1e-6 at the cutoff
struct Gauss32 {
    float hi, lo;
    __host__ __device__ explicit Gauss32(double a2)
    {
        const double c = -a2 * 1.4426950408889634074;   // log2(e)
        hi = (float)c;
        lo = (float)(c - (double)hi);
    }
    __device__ __forceinline__ float operator()(float r2) const
    {
        const float t = hi * r2, d = fmaf(lo, r2, fmaf(hi, r2, -t));
        float e;
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(t));
        return fmaf(e, d * 0.693147181f, e);
    }
};

// Real-space scalars of one image at squared distance r2 (in L^2), its term
// being A I + B x x^T; ex = exp(-a2 r2). Beenakker's polynomials in r2 have
// constants of alpha and s2, times 1/sqrt(pi). In FP32 every constant's own
// rounding would bias all images of all pairs alike (and with them eps, the
// tensor's mean), so it is carried along as a second FP32 number.
template <typename T>
struct Const2 {
    T hi, lo;
    __device__ Const2() {}
    __device__ explicit Const2(double c) : hi((T)c), lo((T)(c - (double)(T)c)) {}
};

template <typename T>
struct RealSpace {
    Const2<T> alpha, e2, as, c0, c1, c2, d0, d1;   // e2: 2 alpha / sqrt(pi); the others times 1/sqrt(pi)
    T s2, hs, a2;                                  // hs: s2/2
    bool smith;
    static constexpr bool kLo = sizeof(T) == 4;
    __device__ RealSpace(const EwaldConst& ec, double s2d)
    {
        alpha = Const2<T>(ec.alpha);
        e2 = Const2<T>(ec.e2);
        as = Const2<T>(ec.as * s2d);
        c0 = Const2<T>(fma(ec.c0[1], s2d, ec.c0[0]));
        c1 = Const2<T>(fma(ec.c1[1], s2d, ec.c1[0]));
        c2 = Const2<T>(ec.c2 * s2d);
        d0 = Const2<T>(fma(ec.d0[1], s2d, ec.d0[0]));
        d1 = Const2<T>(fma(ec.d1[1], s2d, ec.d1[0]));
        a2 = (T)ec.a2;
        s2 = (T)s2d;
        hs = (T)(0.5 * s2d);
        smith = ec.smith;
    }
    __device__ __forceinline__ void image(T r2, T ex, T& A, T& B) const
    {
        const T i = inv_sqrt(r2), i2 = i * i, r = r2 * i;
        T x = alpha.hi * r;
        if (kLo) x += alpha.lo * r;
        const T er = ex * erfcx_pos(x) * i;      // erfc(alpha r)/r
        if (smith) {
            T E = e2.hi * ex;
            if (kLo) E += e2.lo * ex;
            const T sq = i2 * (er + E);
            A = (T)0.75 * er + hs * sq;
            B = ((T)0.75 * (er + E) - hs * (3 * sq + 2 * a2 * E)) * i2;
        } else {
            const T q = s2 * i2, t = as.hi * i2, r4 = c2.hi * r2;
            T p = t + c0.hi + (c1.hi + r4) * r2, u = d0.hi - 3 * t + (d1.hi - r4) * r2;
            if (kLo) {
                p += c0.lo + c1.lo * r2;
                u += d0.lo + d1.lo * r2;
            }
            A = p * ex + er * ((T)0.75 + (T)0.5 * q);
            B = (u * ex + er * ((T)0.75 - (T)1.5 * q)) * i2;
        }
    }
};

__device__ __forceinline__ void add_image(double* o, double A, double B, double x, double y, double z)
{
    const double bx = B * x, by = B * y;
    o[0] += A + bx * x;
    o[1] += A + by * y;
    o[2] += A + B * z * z;
    o[3] += bx * y;
    o[4] += bx * z;
    o[5] += by * z;
}
__device__ __forceinline__ void add_image(float* o, float A, float B, float x, float y, float z)
{
    const float bx = B * x, by = B * y, bz = B * z;
    o[0] += A + bx * x;
    o[1] += A + by * y;
    o[2] += A + bz * z;
    o[3] += bx * y;
    o[4] += bx * z;
    o[5] += by * z;
}

// every image of the FP64 sum with an exponential of its own (see lattice_sum)
static __device__ __noinline__ void images_one_by_one(const EwaldConst& ec, const double* v, double s2, double* o)
{
    const RealSpace<double> rs(ec, s2);
    for (int h = -ec.R; h <= ec.R; ++h)
        for (int f = -ec.extent[h * h]; f <= ec.extent[h * h]; ++f) {
            const int ng = ec.extent[h * h + f * f];
            for (int g = -ng; g <= ng; ++g) {
                const double x = v[0] + h, y = v[1] + f, z = v[2] + g, r2 = x * x + y * y + z * z;
                if (r2 == 0.0) continue;
                double A, B;
                rs.image(r2, exp(-ec.a2 * r2), A, B);
                add_image(o, A, B, x, y, z);
            }
        }
}

// The lattice sum S(v) over the reference's sphere of images and reciprocal
// vectors, v = (r_i - r_j)/L as it is (no minimum image). Bound by FP64
// multiply-adds and their latency (about 90 a image; N = 777, R = 3, Smith:
// 941 -> 347 us per pass over all pairs, against exp, erfc, two square roots or
// divisions per image and a cosine per reciprocal vector).
//
// FP64: every image of the sphere. An image costs one Gaussian, one erfcx and
// the rational terms; the Gaussian along a row of images (g = 0, +-1, ...)
// follows from its neighbour's by two multiplications (exp(-a2 (z+1)^2) =
// exp(-a2 z^2) rho, rho' = rho kappa), started at g = 0 where it is largest.
// With MIXED the images are summed in FP32 and those beyond rcut are dropped.
// Reciprocal space, FP64 in both: the vectors (+-h, +-f, +-g) share their
// weight up to signs, so their cosines collapse to products of the axes'
// cosines and sines: 12 weights and 4 products per class of up to 8 vectors,
// and no cosine beyond one per axis.
template <bool MIXED>
__device__ __forceinline__ void lattice_sum(const EwaldConst& ec, const double* v, double s2, double* S)
{
    const int R = ec.R;
    using T = typename std::conditional<MIXED, float, double>::type;
    T o[6] = {0, 0, 0, 0, 0, 0};
    const RealSpace<T> rs(ec, s2);
    if constexpr (MIXED) {
        const Gauss32 gauss(ec.a2);
        for (int h = -R; h <= R; ++h) {
            const float x = (float)v[0] + h;
            const int nf = ec.extent[h * h];
            for (int f = -nf; f <= nf; ++f) {
                const float y = (float)v[1] + f, xy = x * x + y * y;
                if (xy > ec.rcut_sq) continue;
                const int ng = ec.extent[h * h + f * f];
                for (int g = -ng; g <= ng; ++g) {
                    const float z = (float)v[2] + g, r2 = xy + z * z;
                    if (r2 == 0.f || r2 > ec.rcut_sq) continue;
                    float A, B;
                    rs.image(r2, gauss(r2), A, B);
                    add_image(o, A, B, x, y, z);
                }
            }
        }
    } else {
        // The recurrence holds while up0 and down0 stay finite and the Gaussian
        // at g = 0 does not underflow: positions in the box have |v_k| <= 1
        // (m = 1). Beyond (strong screening; positions that a caller has set
        // many boxes away, 0 * inf from |z0| ~ 113 at alpha = sqrt(pi)) every
        // image takes its own exponential. a2 (1 + 2 |z0|) <= a2 (R + 1 + m)^2.
        const double m = R + 1 + fmax(1.0, fmax(fabs(v[0]), fmax(fabs(v[1]), fabs(v[2]))));
        const double z0 = v[2];
        const double up0 = exp(-ec.a2 * (1 + 2 * z0)), down0 = exp(-ec.a2 * (1 - 2 * z0));
        const bool run = ec.a2 * m * m < 600.0;
        if (!run) {
            const double w[3] = {v[0], v[1], v[2]};
            double e[6] = {0, 0, 0, 0, 0, 0};
            images_one_by_one(ec, w, s2, e);
#pragma unroll
            for (int k = 0; k < 6; ++k) o[k] = e[k];
        }
        for (int h = run ? -R : R + 1; h <= R; ++h) {
            const double x = v[0] + h;
            const int nf = ec.extent[h * h];
            for (int f = -nf; f <= nf; ++f) {
                const double y = v[1] + f, xy = x * x + y * y;
                const int ng = ec.extent[h * h + f * f];
                const double mid = exp(-ec.a2 * (xy + z0 * z0));
                for (int dir = 0; dir < 2; ++dir) {
                    // g = 0, 1, .. ng, then g = -1, .. -ng
                    double ex = dir ? mid * down0 : mid;
                    double rho = dir ? down0 * ec.kappa : up0;
                    const double step = dir ? -1.0 : 1.0;
                    double z = dir ? z0 - 1.0 : z0;
                    for (int g = dir; g <= ng; ++g) {
                        const double r2 = xy + z * z;
                        if (r2 != 0.0) {
                            double A, B;
                            rs.image(r2, ex, A, B);
                            add_image(o, A, B, x, y, z);
                        }
                        z += step;
                        ex *= rho;
                        rho *= ec.kappa;
                    }
                }
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) S[k] = o[k];
    if (!ec.recip) return;
    double cx1, sx1, cy1, sy1, cz1, sz1;
    sincos(ec.two_pif * v[0], &sx1, &cx1);
    sincos(ec.two_pif * v[1], &sy1, &cy1);
    sincos(ec.two_pif * v[2], &sz1, &cz1);
    const double* w = ec.rk;
    double cx = 1, sx = 0;
    for (int h = 0; h <= R; ++h) {
        double cy = 1, sy = 0;
        const int nf = ec.extent[h * h];
        for (int f = 0; f <= nf; ++f) {
            double q[6] = {0, 0, 0, 0, 0, 0};
            double cz = 1, sz = 0;
            const int ng = ec.extent[h * h + f * f];
            for (int g = 0; g <= ng; ++g, w += 12) {
#pragma unroll
                for (int k = 0; k < 6; ++k) q[k] += (w[k] + s2 * w[6 + k]) * (k < 4 ? cz : sz);
                const double c = cz * cz1 - sz * sz1;
                sz = sz * cz1 + cz * sz1;
                cz = c;
            }
            const double cc = cx * cy;
            S[0] += cc * q[0];
            S[1] += cc * q[1];
            S[2] += cc * q[2];
            S[3] += sx * sy * q[3];
            S[4] += sx * cy * q[4];
            S[5] += cx * sy * q[5];
            const double c = cy * cy1 - sy * sy1;
            sy = sy * cy1 + cy * sy1;
            cy = c;
        }
        const double c = cx * cx1 - sx * sx1;
        sx = sx * cx1 + cx * sx1;
        cx = c;
    }
}

// The self tile of a bead of radius a (diagonal, isotropic): its own term,
// the method's self correction and its images.
__device__ __forceinline__ double ewald_self(const EwaldConst& ec, double a, double preDii)
{
    const double il = ec.inv_L, a3 = ec.alpha * ec.a2, q = a * il;
    double sc;
    if (ec.smith) {
        sc = ec.alpha * a * il;
        sc = sc * sc * sc * BDB_M1_SQRTPI / 3;
        sc = -(0.75 * il * 1.5 * ec.alpha * a * BDB_M1_SQRTPI * il + 0.5 * a * a * il * il * il * sc);
    } else {
        sc = (-6 * ec.alpha + 40 * a3 * q * q / 3) / BDB_SQRTPI * il;
    }
    return preDii / a + sc * preDii + preDii * (il * (ec.self0 + ec.self1 * q * q));
}

// diff_tensor_calc_ewald_* (i, j), and _diag for i == j
template <bool MIXED>
__device__ __forceinline__ void rpy_ewald(const double4& pi, const double4& pj, bool self, double preDii,
                                          double preDij, const EwaldConst& ec, double* t)
{
    if (self) {
        t[0] = t[1] = t[2] = ewald_self(ec, pi.w, preDii);
        t[3] = t[4] = t[5] = 0;
        return;
    }
    const double r0 = pi.x - pj.x, r1 = pi.y - pj.y, r2 = pi.z - pj.z;
    const double sum = pi.w + pj.w, ss = pi.w * pi.w + pj.w * pj.w;
    for (int k = 0; k < 6; ++k) t[k] = 0;
    const double rr = r0 * r0 + r1 * r1 + r2 * r2;
    if (rr < sum * sum) {
        // the overlap form in place of the far field
        const double r = sqrt(rr), inv = 1 / r, sigma = sum / 2;
        const double pre = preDii / sigma, q = r / (32 * sigma), pre2 = preDij * inv, sr = ss / rr;
        const double A = pre * (1 - 9 * q) - pre2 * (1 + sr / 3), B = pre * 3 * q - pre2 * (1 - sr);
        const double e[3] = {r0 * inv, r1 * inv, r2 * inv};
        t[0] = A + B * e[0] * e[0];
        t[1] = A + B * e[1] * e[1];
        t[2] = A + B * e[2] * e[2];
        t[3] = B * e[0] * e[1];
        t[4] = B * e[0] * e[2];
        t[5] = B * e[1] * e[2];
    }
    const double v[3] = {r0 * ec.inv_L, r1 * ec.inv_L, r2 * ec.inv_L};
    double S[6];
    lattice_sum<MIXED>(ec, v, 0.5 * ss * ec.inv_L * ec.inv_L, S);
    const double pre = preDii * ec.inv_L;
    for (int k = 0; k < 6; ++k) t[k] += pre * S[k];
}

}  // namespace bdb
