// The converged Ewald sums of the mixed path with another split.
//
// At R >= 4 (default alpha) the reference's sphere of images is the periodic
// sum to ~1e-9, and that sum can be split at any screening. The reference's
// alpha = sqrt(pi)/L leaves ~65 images within 2.5 L per pair. Here the
// screening is 2.5 times stronger, so that only the 8 images around the pair's
// cell matter (the next lie beyond erfc ~ 3e-10), and the rest is a Fourier
// sum over |k|^2 <= 36 whose vectors collapse into 163 classes of signs: six
// multiply-adds each on 21 cosines and sines built from one sincos per axis.
// About 2,700 instructions per pair (74% of the issue slots), against ~65
// images of ~60 and 128 cosines in the reference's split, with lanes idle at
// its cutoff: N = 4096, R = 4 (Beenakker): pair kernel 8.13 -> 0.77 ms.
// The near part is the RPY tensor screened as in Smith's sums (Hasimoto's
// functions: the least Fourier tail); the Fourier weights are its complement
// for the periodic RPY tensor (Smith) or, for Beenakker's sums, the
// difference of the two screenings of the same tensor plus the reference's own
// reciprocal weights. A constant on the diagonal, from the k = 0 terms, is
// fixed by the reference's sum at given points, which also decide whether
// the two agree (ewald_fast_setup).
// Weights and sums are FP32, the Fourier sum's too, where the reference's split
// on this path adds its reciprocal vectors in FP64 (lattice_sum). The error is
// smaller all the same, since that split sums ~65 images in FP32: D F and TEA
// noise against FP64 at N = 4096, R = 4: Beenakker 4.6e-7 and 1.0e-7 relative
// (8.6e-7 and 9.4e-7 by the reference's split), Smith 7.1e-7 and 5.5e-8 (8.2e-7 and
// 6.8e-8); N = 600, R = 4 and 5, three seeds, lower in each.
#pragma once

#include "rpy_tile.cuh"

namespace bdb {

static constexpr int EF_K = 6;                   // |k| <= 6
static constexpr int EF_K2 = EF_K * EF_K;
static constexpr double EF_SPLIT = 2.5;          // screening in units of sqrt(pi)/L

constexpr int ef_classes()
{
    int n = 0;
    for (int h = 0; h <= EF_K; ++h)
        for (int f = 0; f <= EF_K; ++f)
            for (int g = 0; g <= EF_K; ++g) n += h * h + f * f + g * g <= EF_K2;
    return n;
}

// kernel parameter (constant bank): weights in the order the loops below
// visit (h, f, g), {xx, yy, zz, xy, xz, yz}
struct EwaldFast {
    float w[ef_classes()][6];
    float beta, b2, e2;       // screening, its square, 2 beta/sqrt(pi)
    float g_hi, g_lo;         // Gauss32 of the square
    float hs;                 // s2/2
    float diag;               // constant of the diagonal
    float radius;             // the radius the weights hold for
    float near_sq, far_sq;    // squared separations covered: (2 radius / L)^2 (overlap below) to far_sq
    float pre;                // preDii / L
};
struct NoFast {};

// Tile of the raw separation v (in L) of two beads of radius E.radius that do
// not overlap, |v_k| <= 1, |v|^2 <= E.far_sq
__device__ __forceinline__ void ewald_fast_tile(const EwaldFast& E, const float* v, float* t)
{
    float sg[3], x[3][2], xx[3][2], c[3][EF_K + 1], s[3][EF_K + 1];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        // nearest image, folded into the positive octant: the tile is even,
        // and a reflection changes the sign of its off-diagonal entries
        const float u = v[d] - rintf(v[d]), a = fabsf(u);
        sg[d] = copysignf(1.0f, u);
        x[d][0] = a;
        x[d][1] = a - 1.0f;
        xx[d][0] = x[d][0] * x[d][0];
        xx[d][1] = x[d][1] * x[d][1];
        c[d][0] = 1.0f;
        s[d][0] = 0.0f;
        sincospif(2.0f * a, &s[d][1], &c[d][1]);
#pragma unroll
        for (int k = 2; k <= EF_K; ++k) {
            c[d][k] = c[d][k - 1] * c[d][1] - s[d][k - 1] * s[d][1];
            s[d][k] = s[d][k - 1] * c[d][1] + c[d][k - 1] * s[d][1];
        }
    }
    Gauss32 gauss(0.0);
    gauss.hi = E.g_hi;
    gauss.lo = E.g_lo;
    float o[6] = {E.diag, E.diag, E.diag, 0, 0, 0};
    int n = 0;
#pragma unroll
    for (int h = 0; h <= EF_K; ++h)
#pragma unroll
        for (int f = 0; f <= EF_K; ++f) {
            if (h * h + f * f > EF_K2) continue;
            float q[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
            for (int g = 0; g <= EF_K; ++g) {
                if (h * h + f * f + g * g > EF_K2) continue;
                if (h + f + g > 0) {
#pragma unroll
                    for (int k = 0; k < 3; ++k) q[k] = g ? fmaf(E.w[n][k], c[2][g], q[k]) : E.w[n][k];
                    if (h && f) q[3] = g ? fmaf(E.w[n][3], c[2][g], q[3]) : E.w[n][3];
                    if (h && g) q[4] = fmaf(E.w[n][4], s[2][g], q[4]);
                    if (f && g) q[5] = fmaf(E.w[n][5], s[2][g], q[5]);
                }
                ++n;
            }
            const float cc = c[0][h] * c[1][f];
#pragma unroll
            for (int k = 0; k < 3; ++k) o[k] = fmaf(cc, q[k], o[k]);
            if (h && f) o[3] = fmaf(s[0][h] * s[1][f], q[3], o[3]);
            if (h) o[4] = fmaf(s[0][h] * c[1][f], q[4], o[4]);
            if (f) o[5] = fmaf(c[0][h] * s[1][f], q[5], o[5]);
        }
    // the 8 images around the cell
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        const int i0 = m & 1, i1 = (m >> 1) & 1, i2_ = m >> 2;
        const float r2 = xx[0][i0] + (xx[1][i1] + xx[2][i2_]);
        const float i = inv_sqrt(r2), i2 = i * i, r = r2 * i;
        const float ex = gauss(r2);
        const float er = ex * erfcx_pos(E.beta * r) * i, e = E.e2 * ex;
        const float sq = i2 * (er + e);
        const float A = fmaf(0.75f, er, E.hs * sq);
        const float B = (0.75f * (er + e) - E.hs * (3.0f * sq + 2.0f * E.b2 * e)) * i2;
        add_image(o, A, B, x[0][i0], x[1][i1], x[2][i2_]);
    }
    t[0] = E.pre * o[0];
    t[1] = E.pre * o[1];
    t[2] = E.pre * o[2];
    t[3] = E.pre * (sg[0] * sg[1]) * o[3];
    t[4] = E.pre * (sg[0] * sg[2]) * o[4];
    t[5] = E.pre * (sg[1] * sg[2]) * o[5];
}

}  // namespace bdb
