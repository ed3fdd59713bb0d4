// nufft_taps.cuh -- the tap run of one point on an antenna's oversampled grid, shared by the
// interpolation-form kernels.
#pragma once
#include "bp_kernels.cuh"
#include "es_taps.cuh"

namespace mmn {

// First grid cell of N * (u mod 1), u = d slope/c, and the fractional offset less 1/2: both by
// the 1.5*2^52 rounding constant (no conversion instructions), clamped so that a NaN or a
// fraction that rounds up to 1 still reads inside the row.  T: the offset's type.
template <class T>
__device__ __forceinline__ void nufft_cell(double d, double uq, int n, int &cell, T &offset) {
    const double kRound = 6755399441055744.0;  // 1.5 * 2^52
    const double u = d * uq;
    double uf = u - ((u + kRound) - kRound);  // [-1/2, 1/2]
    uf = uf < 0.0 ? uf + 1.0 : uf;            // [0, 1]
    const double x = uf * (double)n;
    const double xt = x + kRound;
    int ix = __double2loint(xt);
    double fr = x - (xt - kRound);             // [-1/2, 1/2]
    ix = fr < 0.0 ? ix - 1 : ix;
    fr = fr < 0.0 ? fr + 1.0 : fr;
    const bool lo = !(ix >= 0), hi = ix >= n;
    cell = lo ? 0 : (hi ? n - 1 : ix);
    offset = lo ? (T)-0.5 : (hi ? (T)0.5 : (T)(fr - 0.5));
}

// First grid cell and the 8 tap weights: the weights from es_taps.cuh, P_i(t) and P_i(-t) from
// one even and one odd part.
// offset: if not null, receives the fractional offset less 1/2.
__device__ __forceinline__ void nufft_taps(double d, double uq, int n, int &cell,
                                           float (&w)[kNuW], float *offset = nullptr) {
    float t;
    nufft_cell(d, uq, n, cell, t);
    const float t2 = t * t;
    if (offset) *offset = t;
#pragma unroll
    for (int i = 0; i < kNuW / 2; ++i) {
        float e = kEsEven[i][kEsEvenTerms - 1];
#pragma unroll
        for (int q = kEsEvenTerms - 2; q >= 0; --q) e = fmaf(e, t2, kEsEven[i][q]);
        float od = kEsOdd[i][kEsOddTerms - 1];
#pragma unroll
        for (int q = kEsOddTerms - 2; q >= 0; --q) od = fmaf(od, t2, kEsOdd[i][q]);
        w[i] = fmaf(t, od, e);
        w[kNuW - 1 - i] = fmaf(-t, od, e);
    }
}

// The same weights in FP64.
__device__ __forceinline__ void nufft_taps64(double d, double uq, int n, int &cell,
                                             double (&w)[kNuW]) {
    double t;
    nufft_cell(d, uq, n, cell, t);
    const double t2 = t * t;
#pragma unroll
    for (int i = 0; i < kNuW / 2; ++i) {
        double e = kEsEven64[i][kEsEvenTerms - 1];
#pragma unroll
        for (int q = kEsEvenTerms - 2; q >= 0; --q) e = fma(e, t2, kEsEven64[i][q]);
        double od = kEsOdd64[i][kEsOddTerms - 1];
#pragma unroll
        for (int q = kEsOddTerms - 2; q >= 0; --q) od = fma(od, t2, kEsOdd64[i][q]);
        w[i] = fma(t, od, e);
        w[kNuW - 1 - i] = fma(-t, od, e);
    }
}

// Per (voxel, antenna) geometry of the interpolation form.
//   d      round-trip range in FP64.  Each leg's square root starts from an FP32 rsqrt of the
//          FP32 difference vector and takes one FP64 Newton step (relative error ~1e-13, far
//          below what the phase needs), which avoids the IEEE FP64 square root's slow path.
//   e3     -(unit(v - tx) + unit(v - rx)) in FP32 (the derivative of d with respect to an
//          antenna offset; a direction needs no more).
//   ix, w  the tap run (nufft_taps).
struct NuPair {
    double d;
    float e3[3];
    int ix;
    float w[kNuW];
};

__device__ __forceinline__ void nufft_pair(double vxd, double vyd, double vzd, float vx, float vy,
                                           float vz, const AntRec &ar, const float (&txf)[3],
                                           const float (&rxf)[3], bool mono, double ti, double uq,
                                           int n, NuPair &o) {
    const float ax = vx - txf[0], ay = vy - txf[1], az = vz - txf[2];
    const float rf = rsqrtf(fmaf(ax, ax, fmaf(ay, ay, az * az)));
    const double dx = vxd - ar.tx[0], dy = vyd - ar.tx[1], dz = vzd - ar.tx[2];
    const double D = fma(dx, dx, fma(dy, dy, dz * dz));
    const double r = (double)rf;
    double f = D * r;
    f = fma(fma(-f, f, D), 0.5 * r, f);
    double b = f;
    float bx = ax, by = ay, bz = az, rb = rf;
    if (!mono) {
        bx = vx - rxf[0];
        by = vy - rxf[1];
        bz = vz - rxf[2];
        rb = rsqrtf(fmaf(bx, bx, fmaf(by, by, bz * bz)));
        const double ex = vxd - ar.rx[0], ey = vyd - ar.rx[1], ez = vzd - ar.rx[2];
        const double B = fma(ex, ex, fma(ey, ey, ez * ez));
        const double rr = (double)rb;
        b = B * rr;
        b = fma(fma(-b, b, B), 0.5 * rr, b);
    }
    o.d = f + b + ti;
    o.e3[0] = -fmaf(ax, rf, bx * rb);
    o.e3[1] = -fmaf(ay, rf, by * rb);
    o.e3[2] = -fmaf(az, rf, bz * rb);
    nufft_taps(o.d, uq, n, o.ix, o.w);
}

// Centre and half width of an antenna's round-trip range over a box of voxels (without the
// TI offset), from the legs' separate extremes in FP32, widened by their rounding.  A NaN or
// infinite antenna or box gives a half width that is not finite.
__device__ __forceinline__ void range_bounds(const float (&lo)[3], const float (&hi)[3],
                                             const float (&t)[3], const float (&r)[3],
                                             float &centre, float &half, float &dmax) {
    float near2[2] = {0.f, 0.f}, far2[2] = {0.f, 0.f}, mag = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
#pragma unroll
        for (int l = 0; l < 2; ++l) {
            const float p = l ? r[k] : t[k];
            const float a = lo[k] - p, b = p - hi[k];
            const float n = fmaxf(fmaxf(a, b), 0.f), f = fmaxf(fabsf(a), fabsf(b));
            near2[l] = fmaf(n, n, near2[l]);
            far2[l] = fmaf(f, f, far2[l]);
            mag += fabsf(p);
        }
    }
    dmax = sqrtf(far2[0]) + sqrtf(far2[1]);
    const float dmin = sqrtf(near2[0]) + sqrtf(near2[1]);
    centre = 0.5f * (dmin + dmax);
    half = 0.5f * (dmax - dmin) + 1e-6f * (mag + dmax) + 1e-9f;
}

}  // namespace mmn
