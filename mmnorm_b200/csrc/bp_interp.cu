// bp_interp.cu -- interpolated-mode backprojection and normal vote (the reference's
// shipped default, src/utils/params.json:4 "use_interpolated_processing": true).
//
// Per (voxel, virtual antenna) the reference takes ONE sample -- the range-FFT bin
// floor(d/fft_spacing/2) -- and ONE phasor exp(-j*2*pi*d/lambda) evaluated in FP64
// (imaging_gpu.cu:90-105; surface_normal_est.cu:99-124).  The exact form gives that
// arithmetic's bits (FP32 distance, the FP32 roundings of the FP64 cos and sin, FP32
// accumulation in antenna order), so its outputs reproduce the reference's kernels; what
// changes is the structure around it: the antenna geometry streams through shared memory in
// chunks, each thread's two voxels ride in the halves of packed FP32 instructions, the
// measurement gather is a single 8-byte load of the complex bin, the phasor comes from a short
// FP64 evaluation that proves its own FP32 rounding (phasor2_exact), and the image pass can
// fuse the vote vector W = sum_i c_i (tx_i + o_i/2 - v).
#include <atomic>

#include "bp_kernels.cuh"

namespace mmn {

// Form of the fast passes: 0 packed voxel pairs (default), 1 scalar.
std::atomic<int> g_interp_fast_form{0};

namespace {
constexpr int kInterpThreads = 256;
// antennas per loop pass (exact: 1 measured 13.80 ms, 2 13.54; fast: 1 7.06, 2 6.91, 4 6.78)
constexpr int kExactUnroll = 2, kFastUnroll = 4;
constexpr int kInterpChunk = 256;  // antennas staged per shared-memory chunk
}  // namespace

// ---------------------------------------------------------------------------------
// Fast form.  The path length and the range bin are the reference's (same FP32
// operations, so the same bin is gathered); only the phasor exp(-j 2 pi path/lambda) is
// formed differently: instead of an FP64 cos and sin of the ~1e3-radian phase, the turn
// count path/lambda is formed as a double-float product (1/lambda = hi + lo, both FP32;
// the rounding error of path*hi recovered exactly by an FMA), its integer part removed
// exactly, and the hardware sine/cosine (__sincosf, absolute error about 2^-21.4 on
// [-pi, pi]) evaluated on the wrapped angle.  Phase error ~2e-7 turns + 4e-7 absolute in
// each phasor component: about 5e-7 relative per term against the reference's phasor.
// ---------------------------------------------------------------------------------
namespace {
constexpr int kFastT = 2;                  // voxels per thread
constexpr float kRoundMagic = 12582912.f;  // 1.5 * 2^23: (x + M) - M rounds |x| < 2^22

// Range antenna record of the fast kernels: TX, RX offset and the vote anchor TX + o/2
// (formed in FP32 as surface_normal_est.cu:128-130 does).
struct __align__(16) FastAnt {
    float4 t, o, u;
};

__device__ __forceinline__ void stage_fast_chunk(const InterpParams &p, int a0, int n,
                                                 FastAnt *sh) {
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        const int i = a0 + j;
        const int rx = i % p.num_rx;
        const float tx = p.ant[3 * i + 0], ty = p.ant[3 * i + 1], tz = p.ant[3 * i + 2];
        const float ox = p.rxo[3 * rx + 0], oy = p.rxo[3 * rx + 1], oz = p.rxo[3 * rx + 2];
        FastAnt a;
        a.t = make_float4(tx, ty, tz, 0.f);
        a.o = make_float4(ox, oy, oz, 0.f);
        a.u = make_float4(tx + ox / 2, ty + oy / 2, tz + oz / 2, 0.f);
        sh[j] = a;
    }
}

// floor(RN(path / fsp) / 2), the reference's range bin (imaging_gpu.cu:100), for
// 0 <= path <= fsp * nbins.  h = path * (1/(2 fsp)) is within 2e-7 h of the rounded
// quotient's half, so floor(h) is that bin unless h lies within 1.2e-6 h of an integer;
// then the reference's own division decides.  The floor comes from the rounding constant
// (no conversion instruction): bits(h + M) - bits(M) = rint(h) for 0 <= h < 2^22.
__device__ __forceinline__ int fast_bin(float path, float fsp, float half_inv) {
    const float h = path * half_inv;
    const float hm = h + kRoundMagic;
    const float r = hm - kRoundMagic;
    const bool above = r > h;
    const float fr = h - (above ? r - 1.f : r);
    const float tol = fmaxf(h, 1.f) * 1.2e-6f;
    if (fr < tol || fr > 1.f - tol) return (int)floorf(path / fsp / 2);
    return __float_as_int(hm) - __float_as_int(kRoundMagic) - (above ? 1 : 0);
}

// (cos, sin) of -2 pi path / lambda with 1/lambda = hi + lo.
__device__ __forceinline__ void fast_phasor(float path, float hi, float lo, float &c,
                                            float &s) {
    const float q = path * hi;
    const float e = fmaf(path, hi, -q);        // exact: path*hi = q + e
    const float n = (q + kRoundMagic) - kRoundMagic;
    const float f = (q - n) + fmaf(path, lo, e);  // path/lambda - n; |f| <= 0.5 + ulp(q)
    __sincosf(-6.28318530717958647692f * f, &s, &c);
}

template <bool MONO>
__device__ __forceinline__ float2 fast_contrib(const InterpParams &p, size_t row, float vx,
                                               float vy, float vz, const FastAnt &a,
                                               float range_max) {
    const float dx = vx - a.t.x;
    const float dy = vy - a.t.y;
    const float dz = vz - a.t.z;
    const float leg_out = sqrtf(dx * dx +
                                dy * dy +
                                dz * dz);
    float path;
    if (MONO) {
        path = leg_out + leg_out;  // the return leg with a zero offset is the same value
    } else {
        const float leg_back = sqrtf((dx - a.o.x) * (dx - a.o.x) +
                                     (dy - a.o.y) * (dy - a.o.y) +
                                     (dz - a.o.z) * (dz - a.o.z));
        path = leg_out + leg_back;
    }
    if (p.is_ti != 0) {
        path += 0.15;
    }
    const bool valid = !(path < 0 || path > range_max);
    const int bin = valid ? fast_bin(path, p.fft_spacing, p.half_inv_fsp) : 0;
    float m_re, m_im;
    if (p.meas) {
        const float2 m = __ldg(p.meas + row + bin);
        m_re = m.x;
        m_im = m.y;
    } else {
        m_re = __ldg(p.meas_r + row + bin);
        m_im = __ldg(p.meas_i + row + bin);
    }
    float c, s;
    fast_phasor(path, p.inv_lambda_hi, p.inv_lambda_lo, c, s);
    const float re = fmaf(m_re, c, -m_im * s);
    const float im = fmaf(m_re, s, m_im * c);
    return valid ? make_float2(re, im) : make_float2(0.f, 0.f);
}

// Does any staged antenna of this chunk have a non-zero RX offset?  (Uniform per CTA.)
__device__ __forceinline__ bool chunk_has_offsets(const FastAnt *sh, int n) {
    bool any = false;
    for (int j = threadIdx.x; j < n; j += blockDim.x)
        any |= (sh[j].o.x != 0.f) | (sh[j].o.y != 0.f) | (sh[j].o.z != 0.f);
    return __syncthreads_or(any) != 0;
}

template <bool MONO, bool VOTE>
__device__ __forceinline__ void fast_image_chunk(const InterpParams &p, const FastAnt *sh,
                                                 int a0, int n, float range_max,
                                                 const float (&vx)[kFastT],
                                                 const float (&vy)[kFastT],
                                                 const float (&vz)[kFastT],
                                                 float (&acc)[kFastT][8]) {
#pragma unroll 2
    for (int j = 0; j < n; ++j) {
        const FastAnt a = sh[j];
        const size_t row = (size_t)(a0 + j) * (size_t)p.nbins;
#pragma unroll
        for (int k = 0; k < kFastT; ++k) {
            const float2 c = fast_contrib<MONO>(p, row, vx[k], vy[k], vz[k], a, range_max);
            acc[k][0] += c.x;
            acc[k][1] += c.y;
            if (VOTE) {
                const float ex = a.u.x - vx[k], ey = a.u.y - vy[k], ez = a.u.z - vz[k];
                acc[k][2] = fmaf(c.x, ex, acc[k][2]);
                acc[k][3] = fmaf(c.y, ex, acc[k][3]);
                acc[k][4] = fmaf(c.x, ey, acc[k][4]);
                acc[k][5] = fmaf(c.y, ey, acc[k][5]);
                acc[k][6] = fmaf(c.x, ez, acc[k][6]);
                acc[k][7] = fmaf(c.y, ez, acc[k][7]);
            }
        }
    }
}
}  // namespace

// Image pass in fast form, kFastT voxels per thread (strided by the block size so loads
// and stores coalesce), optionally fusing the vote vector.
__global__ void __launch_bounds__(kInterpThreads) interp_image_fast_kernel(const InterpParams p) {
    __shared__ FastAnt sh[kInterpChunk];
    const int64_t nyz = (int64_t)p.ny * p.nz;
    const float range_max = p.fft_spacing * p.nbins;
    int64_t vox[kFastT];
    bool active[kFastT];
    float vx[kFastT], vy[kFastT], vz[kFastT];
    float acc[kFastT][8];
#pragma unroll
    for (int k = 0; k < kFastT; ++k) {
        const int64_t rel = ((int64_t)blockIdx.x * kFastT + k) * blockDim.x + threadIdx.x;
        active[k] = rel < p.count && rel + p.start < p.nvox;
        const int64_t v = active[k] ? rel + p.start : 0;
        vox[k] = v;
        const int x = (int)(v / nyz);
        const int y = (int)((v - (int64_t)x * nyz) / p.nz);
        const int z = (int)(v - (int64_t)x * nyz - (int64_t)y * p.nz);
        vx[k] = p.x_locs[x];
        vy[k] = p.y_locs[y];
        vz[k] = p.z_locs[z];
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[k][q] = 0.f;
    }
    for (int a0 = 0; a0 < p.num_ant; a0 += kInterpChunk) {
        const int n = min(kInterpChunk, p.num_ant - a0);
        __syncthreads();
        stage_fast_chunk(p, a0, n, sh);
        __syncthreads();
        const bool offsets = chunk_has_offsets(sh, n);
        if (p.vote) {
            if (offsets) fast_image_chunk<false, true>(p, sh, a0, n, range_max, vx, vy, vz, acc);
            else fast_image_chunk<true, true>(p, sh, a0, n, range_max, vx, vy, vz, acc);
        } else {
            if (offsets) fast_image_chunk<false, false>(p, sh, a0, n, range_max, vx, vy, vz, acc);
            else fast_image_chunk<true, false>(p, sh, a0, n, range_max, vx, vy, vz, acc);
        }
    }
#pragma unroll
    for (int k = 0; k < kFastT; ++k) {
        if (!active[k]) continue;
        const int64_t v = vox[k];
        if (p.out_r) {
            p.out_r[v] = acc[k][0];
            p.out_i[v] = acc[k][1];
        }
        if (p.image) p.image[v] = make_float2(acc[k][0], acc[k][1]);
        if (p.vote) {
            p.vote[v] = make_float2(acc[k][2], acc[k][3]);
            p.vote[p.nvox + v] = make_float2(acc[k][4], acc[k][5]);
            p.vote[2 * p.nvox + v] = make_float2(acc[k][6], acc[k][7]);
        }
    }
}

// Normal pass in fast form over a valid-voxel list (one voxel per thread).
__global__ void __launch_bounds__(kInterpThreads) interp_normals_fast_kernel(const InterpParams p) {
    __shared__ FastAnt sh[kInterpChunk];
    const int64_t rel = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t ind64 = rel + p.start;
    const bool active = rel < p.count && ind64 < p.num_valid && ind64 >= 0;
    const int ind = active ? (int)ind64 : 0;
    int x = 0, y = 0, z = 0;
    if (active) {
        x = p.vidx_x[ind];
        y = p.vidx_y[ind];
        z = p.vidx_z[ind];
    }
    const float vx = p.x_locs[x], vy = p.y_locs[y], vz = p.z_locs[z];
    const int64_t v = ((int64_t)x * p.ny + y) * p.nz + z;
    const float i_re = active ? p.img_r[v] : 1.f;
    const float i_im = active ? p.img_i[v] : 0.f;
    const float inv_mag = 1.f / sqrtf(i_re * i_re + i_im * i_im);
    const float range_max = p.fft_spacing * p.nbins;
    float acc_x = 0.f, acc_y = 0.f, acc_z = 0.f;
    for (int a0 = 0; a0 < p.num_ant; a0 += kInterpChunk) {
        const int n = min(kInterpChunk, p.num_ant - a0);
        __syncthreads();
        stage_fast_chunk(p, a0, n, sh);
        __syncthreads();
        const bool offsets = chunk_has_offsets(sh, n);
        if (!active) continue;
#pragma unroll 2
        for (int j = 0; j < n; ++j) {
            const FastAnt a = sh[j];
            const size_t row = (size_t)(a0 + j) * (size_t)p.nbins;
            const float2 c = offsets ? fast_contrib<false>(p, row, vx, vy, vz, a, range_max)
                                     : fast_contrib<true>(p, row, vx, vy, vz, a, range_max);
            const float wgt = fmaf(c.x, i_re, c.y * i_im) * inv_mag;
            acc_x = fmaf(a.u.x - vx, wgt, acc_x);
            acc_y = fmaf(a.u.y - vy, wgt, acc_y);
            acc_z = fmaf(a.u.z - vz, wgt, acc_z);
        }
    }
    if (!active) return;
    p.n_x[ind] = acc_x;
    p.n_y[ind] = acc_y;
    p.n_z[ind] = acc_z;
}

// ---------------------------------------------------------------------------------
// Packed kernels (both forms): each thread's two voxels ride in the two halves of Blackwell's packed
// FP32 instructions (FADD2 / FMUL2 / FFMA2; each half rounds exactly like the scalar
// instruction), so the per-pair arithmetic -- differences, squared range, range bin,
// turn count, complex product, vote -- issues once per voxel pair.  The square roots, the
// sine/cosine and the gathers stay per voxel.  The squared range must reproduce the
// reference's FP32 value bit for bit (its path length selects the bin and sets the phase
// to ~1e-4 rad per ulp): nvcc contracts the reference's dx*dx + dy*dy + dz*dz into
// fma(dz, dz, fma(dx, dx, dy*dy)), which sumsq2 repeats.  (Measured: that order gives the
// bit-exact kernel's bins and phases, 7.5e-7 from it at the 128^3 / 16384-antenna
// workload; the order fma(dz, dz, fma(dy, dy, dx*dx)) is 2.5e-4 away.)
// ---------------------------------------------------------------------------------
namespace {
// Staged antenna of the packed form: values pre-negated and duplicated in both halves, so
// one 16-byte shared load feeds a packed instruction directly.
struct __align__(16) PackAnt {
    float2 ntx, nty, ntz, pad0;  // -TX
    float2 nox, noy, noz, pad1;  // -RX offset
    float2 ux, uy, uz, pad2;     // TX + o/2 (vote anchor)
};

__device__ __forceinline__ float2 dup(float a) { return make_float2(a, a); }

__device__ __forceinline__ void stage_pack_chunk(const InterpParams &p, int a0, int n,
                                                 PackAnt *sh) {
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        const int i = a0 + j;
        const int rx = i % p.num_rx;
        const float tx = p.ant[3 * i + 0], ty = p.ant[3 * i + 1], tz = p.ant[3 * i + 2];
        const float ox = p.rxo[3 * rx + 0], oy = p.rxo[3 * rx + 1], oz = p.rxo[3 * rx + 2];
        PackAnt a;
        a.ntx = dup(-tx);
        a.nty = dup(-ty);
        a.ntz = dup(-tz);
        a.nox = dup(-ox);
        a.noy = dup(-oy);
        a.noz = dup(-oz);
        a.ux = dup(tx + ox / 2);
        a.uy = dup(ty + oy / 2);
        a.uz = dup(tz + oz / 2);
        a.pad0 = a.pad1 = a.pad2 = dup(0.f);
        sh[j] = a;
    }
}

__device__ __forceinline__ bool pack_chunk_has_offsets(const PackAnt *sh, int n) {
    bool any = false;
    for (int j = threadIdx.x; j < n; j += blockDim.x)
        any |= (sh[j].nox.x != 0.f) | (sh[j].noy.x != 0.f) | (sh[j].noz.x != 0.f);
    return __syncthreads_or(any) != 0;
}

// Correctly rounded square roots of two values: s = x y from the hardware reciprocal square root
// y, then Heron's step s + (x - s^2) y / 2 with the residual exact in one FMA (Markstein, IBM J.
// Res. Dev. 34, 1990).  That rounds like sqrtf for every mantissa and exponent parity (checked
// exhaustively over [1, 4), 2^24 inputs); outside [2^-100, 2^100], and for NaN, sqrtf itself.
__device__ __forceinline__ float2 sqrt2(float2 x) {
    float2 y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y.x) : "f"(x.x));
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y.y) : "f"(x.y));
    const float2 s = __fmul2_rn(x, y);
    const float2 h = __fmul2_rn(y, dup(0.5f));
    const float2 e = __ffma2_rn(make_float2(-s.x, -s.y), s, x);
    float2 r = __ffma2_rn(e, h, s);
    if (!(fminf(x.x, x.y) >= 7.888609052210118e-31f && fmaxf(x.x, x.y) <= 1.2676506002282294e30f) ||
        !(x.x == x.x && x.y == x.y))
        r = make_float2(sqrtf(x.x), sqrtf(x.y));
    return r;
}

__device__ __forceinline__ float2 sumsq2(float2 dx, float2 dy, float2 dz) {
    return __ffma2_rn(dz, dz, __ffma2_rn(dx, dx, __fmul2_rn(dy, dy)));
}

// The two voxels' FP32 path lengths, as imaging_gpu.cu:70-89 forms them.
template <bool MONO>
__device__ __forceinline__ float2 path2(float2 vx, float2 vy, float2 vz, const PackAnt &a,
                                        bool ti) {
    const float2 dx = __fadd2_rn(vx, a.ntx);
    const float2 dy = __fadd2_rn(vy, a.nty);
    const float2 dz = __fadd2_rn(vz, a.ntz);
    const float2 s = sumsq2(dx, dy, dz);
    const float2 leg = sqrt2(s);
    float2 path;
    if (MONO) {
        path = __fadd2_rn(leg, leg);
    } else {
        const float2 bx = __fadd2_rn(dx, a.nox);
        const float2 by = __fadd2_rn(dy, a.noy);
        const float2 bz = __fadd2_rn(dz, a.noz);
        const float2 sb = sumsq2(bx, by, bz);
        path = __fadd2_rn(leg, sqrt2(sb));
    }
    if (ti) {  // float += double, as the reference adds its 0.15 m
        path.x += 0.15;
        path.y += 0.15;
    }
    return path;
}

// The reference's range bin floor(RN(path / fsp) / 2) (imaging_gpu.cu:100) of two paths, plus
// kBinBias and clamped to bin nbins - 1 (an in-range path's bin is at most nbins / 2; anything
// else, a NaN's too, must only stay inside the row).  h = path * (1/(2 fsp)) is within 2e-7 h of
// the rounded quotient's half, so floor(h) -- one addition rounded down -- is that bin unless h
// lies within 1.2e-6 (h + 1) of an integer; then, and for a NaN (a path's, or half_inv's, which
// sends every path here), the reference's own division decides.
constexpr uint32_t kBinBias = 0x4B000000u;  // bits of 2^23
__device__ __forceinline__ uint2 bin2(float2 path, float fsp, float half_inv, uint32_t nbins) {
    const float2 h = __fmul2_rn(path, dup(half_inv));
    const float2 hm = make_float2(__fadd_rd(h.x, 8388608.f), __fadd_rd(h.y, 8388608.f));
    const float2 fr = __fadd2_rn(h, __fadd2_rn(dup(8388608.f), make_float2(-hm.x, -hm.y)));
    const float2 mid = __fadd2_rn(fr, dup(-0.5f));
    const float2 lim = __ffma2_rn(h, dup(-1.2e-6f), dup(0.5f - 1.2e-6f));
    uint2 b = make_uint2(__float_as_uint(hm.x), __float_as_uint(hm.y));
    if (!(fabsf(mid.x) < lim.x)) b.x = (uint32_t)(int)floorf(path.x / fsp / 2) + kBinBias;
    if (!(fabsf(mid.y) < lim.y)) b.y = (uint32_t)(int)floorf(path.y / fsp / 2) + kBinBias;
    b.x = min(b.x, nbins - 1u + kBinBias);
    b.y = min(b.y, nbins - 1u + kBinBias);
    return b;
}

// fast_phasor for two paths: returns (cos, sin) of -2 pi path / lambda per half.
__device__ __forceinline__ void phasor2(float2 path, float hi, float lo, float2 &c,
                                        float2 &s) {
    const float2 qn = __fmul2_rn(path, dup(-hi));               // -q
    const float2 e = __ffma2_rn(path, dup(hi), qn);             // path*hi - q, exact
    const float2 nn = __fadd2_rn(__fadd2_rn(qn, dup(kRoundMagic)), dup(-kRoundMagic));  // -n
    const float2 g = __ffma2_rn(nn, dup(-1.f), qn);             // -(q - n), exact
    const float2 w = __ffma2_rn(path, dup(lo), e);              // path*lo + e
    const float2 f = __ffma2_rn(g, dup(-1.f), w);               // (q - n) + w
    const float2 ang = __fmul2_rn(f, dup(-6.28318530717958647692f));
    __sincosf(ang.x, &s.x, &c.x);
    __sincosf(ang.y, &s.y, &c.y);
}

// The reference's own phasor (FP64 phase, cos, sin, rounded to FP32): the fallback of
// phasor2_exact.
__device__ __noinline__ float2 phasor_library(float path, float wavelength) {
    float ph_re = cos(-2 * kPi * path / wavelength);
    float ph_im = sin(-2 * kPi * path / wavelength);
    return make_float2(ph_re, ph_im);
}

// FP64 (cos, sin) of -2 pi path / lambda as bounds: the turns path * (-1/lambda), reduced to
// half a turn in one FMA, then polynomials in r^2 (fitted at Chebyshev nodes on |r| <= 1/4: sine
// 7.8e-14, cosine 1.9e-15).  The reference's rounded phase and this one differ by less than
// 3.8e-16 relative (two roundings and the rounded pi there, the rounded 1/lambda here), i.e. by
// less than 2.4e-15 path / lambda radians; with 1.5e-13 for the fits, the evaluation and the
// library functions' ulps,
//     delta = 2.5e-15 path / lambda + 1.5e-13
// bounds the distance of both components.  lo and hi are the FP32 roundings of the bounds'
// ends: where they agree, every value between them, the reference's among them, rounds to that.
__device__ __forceinline__ bool phasor_exact(float path, double ninv, float &c, float &s) {
    const double kM = 3377699720527872.0;  // 1.5 * 2^51: the sum rounds to half turns
    const double P = (double)path;
    const double t = fma(P, ninv, kM);
    const uint32_t flip = (uint32_t)__double2loint(t) << 31;  // odd half turns negate both
    const double r = fma(P, ninv, kM - t);
    const double y = r * r;
    double p = fma(3.6658551595639612, y, -15.081483206893);
    p = fma(p, y, 42.058134871372054);
    p = fma(p, y, -76.70584754377326);
    p = fma(p, y, 81.60524914901583);
    p = fma(p, y, -41.341702239903675);
    p = fma(p, y, 6.28318530717927);
    const double sn = p * r;
    double g = fma(-1.6452233497893094, y, 7.896555735851554);
    g = fma(g, y, -26.42588874334368);
    g = fma(g, y, 60.24463060817376);
    g = fma(g, y, -85.45681703563287);
    g = fma(g, y, 64.93939402133272);
    g = fma(g, y, -19.739208802174744);
    g = fma(g, y, 0.9999999999999981);
    const double delta = fma(P, -2.5e-15 * ninv, 1.5e-13);
    const float c_lo = (float)(g - delta), c_hi = (float)(g + delta);
    const float s_lo = (float)(sn - delta), s_hi = (float)(sn + delta);
    c = __uint_as_float(__float_as_uint(c_lo) ^ flip);
    s = __uint_as_float(__float_as_uint(s_lo) ^ flip);
    return c_lo == c_hi && s_lo == s_hi;
}

// The reference's FP32 phasors of two paths, bit for bit: about one evaluation in 4000 cannot
// decide its rounding and takes the library functions.  Bound: instruction issue (142 a pair,
// active 79 % of cycles), then the conversions and root seeds (XU 41 %).  90 x 100 x 70 voxels x 4096 antennas, four
// receivers, TI offset: 20.3 ms with the two library calls per pair, 13.5 ms.
__device__ __forceinline__ void phasor2_exact(float2 path, float wavelength, double ninv,
                                              float2 &c, float2 &s) {
    if (!phasor_exact(path.x, ninv, c.x, s.x)) {
        const float2 a = phasor_library(path.x, wavelength);
        c.x = a.x;
        s.x = a.y;
    }
    if (!phasor_exact(path.y, ninv, c.y, s.y)) {
        const float2 a = phasor_library(path.y, wavelength);
        c.y = a.x;
        s.y = a.y;
    }
}

// c_i of two voxels of the given paths against one antenna, as imaging_gpu.cu:90-105; v0, v1: the
// path lies in the measured range (the reference skips the others).
template <bool SOA, bool EXACT>
__device__ __forceinline__ void pack_terms(const InterpParams &p, ptrdiff_t row, float range_max,
                                           float2 path, float2 &re, float2 &im, bool &v0,
                                           bool &v1) {
    v0 = !(path.x > range_max);  // a path is never negative
    v1 = !(path.y > range_max);
    const uint2 b = bin2(path, p.fft_spacing, p.half_inv_fsp, (uint32_t)p.nbins);
    float2 mre, mim;
    if (SOA) {
        const float *mr = p.meas_r + row - kBinBias, *mi = p.meas_i + row - kBinBias;
        mre = make_float2(__ldg(mr + b.x), __ldg(mr + b.y));
        mim = make_float2(__ldg(mi + b.x), __ldg(mi + b.y));
    } else {
        const float2 *m = p.meas + row - kBinBias;
        const float2 m0 = __ldg(m + b.x), m1 = __ldg(m + b.y);
        mre = make_float2(m0.x, m1.x);
        mim = make_float2(m0.y, m1.y);
    }
    float2 c, s;
    if (EXACT) phasor2_exact(path, p.wavelength, p.neg_inv_lambda, c, s);
    else phasor2(path, p.inv_lambda_hi, p.inv_lambda_lo, c, s);
    // the reference kernel's products as they are contracted: fma(m_re, c, -(m_im s)) and
    // fma(m_im, c, m_re s)
    re = __ffma2_rn(mre, c, __fmul2_rn(mim, make_float2(-s.x, -s.y)));
    im = __ffma2_rn(mim, c, __fmul2_rn(mre, s));
}

template <bool MONO, bool VOTE, bool SOA, bool EXACT>
__device__ __forceinline__ void pack_image_chunk(const InterpParams &p, const PackAnt *sh,
                                                 int a0, int n, float range_max, bool ti,
                                                 float2 vx, float2 vy, float2 vz, float2 nvx,
                                                 float2 nvy, float2 nvz, float2 (&acc)[8]) {
    constexpr int kUnroll = EXACT ? kExactUnroll : kFastUnroll;
#pragma unroll kUnroll
    for (int j = 0; j < n; ++j) {
        const PackAnt &a = sh[j];
        const ptrdiff_t row = (ptrdiff_t)(a0 + j) * p.nbins;
        float2 re, im;
        bool v0, v1;
        pack_terms<SOA, EXACT>(p, row, range_max, path2<MONO>(vx, vy, vz, a, ti), re, im, v0, v1);
        float2 ex = __fadd2_rn(a.ux, nvx);
        float2 ey = __fadd2_rn(a.uy, nvy);
        float2 ez = __fadd2_rn(a.uz, nvz);
        if (!(v0 && v1)) {  // a skipped pair adds nothing, whatever its vector is
            re = make_float2(v0 ? re.x : 0.f, v1 ? re.y : 0.f);
            im = make_float2(v0 ? im.x : 0.f, v1 ? im.y : 0.f);
            ex = make_float2(v0 ? ex.x : 0.f, v1 ? ex.y : 0.f);
            ey = make_float2(v0 ? ey.x : 0.f, v1 ? ey.y : 0.f);
            ez = make_float2(v0 ? ez.x : 0.f, v1 ? ez.y : 0.f);
        }
        acc[0] = __fadd2_rn(acc[0], re);
        acc[1] = __fadd2_rn(acc[1], im);
        if (VOTE) {
            acc[2] = __ffma2_rn(re, ex, acc[2]);
            acc[3] = __ffma2_rn(im, ex, acc[3]);
            acc[4] = __ffma2_rn(re, ey, acc[4]);
            acc[5] = __ffma2_rn(im, ey, acc[5]);
            acc[6] = __ffma2_rn(re, ez, acc[6]);
            acc[7] = __ffma2_rn(im, ez, acc[7]);
        }
    }
}

template <bool VOTE, bool SOA, bool EXACT>
__device__ __forceinline__ void pack_image_dispatch(const InterpParams &p, const PackAnt *sh,
                                                    int a0, int n, float range_max, bool ti,
                                                    bool offsets, float2 vx, float2 vy,
                                                    float2 vz, float2 nvx, float2 nvy,
                                                    float2 nvz, float2 (&acc)[8]) {
    if (offsets)
        pack_image_chunk<false, VOTE, SOA, EXACT>(p, sh, a0, n, range_max, ti, vx, vy, vz, nvx,
                                                  nvy, nvz, acc);
    else
        pack_image_chunk<true, VOTE, SOA, EXACT>(p, sh, a0, n, range_max, ti, vx, vy, vz, nvx,
                                                 nvy, nvz, acc);
}
}  // namespace

// Image pass: voxels rel and rel + blockDim of each 2*blockDim tile (coalesced stores),
// optionally fusing the vote vector.
template <bool EXACT>
__global__ void __launch_bounds__(kInterpThreads) interp_image_pack_kernel(const InterpParams p) {
    __shared__ PackAnt sh[kInterpChunk];
    const int64_t nyz = (int64_t)p.ny * p.nz;
    const float range_max = p.fft_spacing * p.nbins;
    const bool ti = p.is_ti != 0;
    int64_t vox[2];
    bool active[2];
    float px[2], py[2], pz[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int64_t rel = ((int64_t)blockIdx.x * 2 + k) * blockDim.x + threadIdx.x;
        active[k] = rel < p.count && rel + p.start < p.nvox;
        const int64_t v = active[k] ? rel + p.start : 0;
        vox[k] = v;
        const int x = (int)(v / nyz);
        const int y = (int)((v - (int64_t)x * nyz) / p.nz);
        const int z = (int)(v - (int64_t)x * nyz - (int64_t)y * p.nz);
        px[k] = p.x_locs[x];
        py[k] = p.y_locs[y];
        pz[k] = p.z_locs[z];
    }
    const float2 vx = make_float2(px[0], px[1]), vy = make_float2(py[0], py[1]),
                 vz = make_float2(pz[0], pz[1]);
    const float2 nvx = make_float2(-px[0], -px[1]), nvy = make_float2(-py[0], -py[1]),
                 nvz = make_float2(-pz[0], -pz[1]);
    float2 acc[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) acc[q] = dup(0.f);
    const bool soa = p.meas == nullptr;
    for (int a0 = 0; a0 < p.num_ant; a0 += kInterpChunk) {
        const int n = min(kInterpChunk, p.num_ant - a0);
        __syncthreads();
        stage_pack_chunk(p, a0, n, sh);
        __syncthreads();
        const bool offsets = pack_chunk_has_offsets(sh, n);
        if (p.vote) {
            if (soa) pack_image_dispatch<true, true, EXACT>(p, sh, a0, n, range_max, ti, offsets,
                                                            vx, vy, vz, nvx, nvy, nvz, acc);
            else pack_image_dispatch<true, false, EXACT>(p, sh, a0, n, range_max, ti, offsets,
                                                         vx, vy, vz, nvx, nvy, nvz, acc);
        } else {
            if (soa) pack_image_dispatch<false, true, EXACT>(p, sh, a0, n, range_max, ti,
                                                             offsets, vx, vy, vz, nvx, nvy, nvz,
                                                             acc);
            else pack_image_dispatch<false, false, EXACT>(p, sh, a0, n, range_max, ti, offsets,
                                                          vx, vy, vz, nvx, nvy, nvz, acc);
        }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        if (!active[k]) continue;
        const int64_t v = vox[k];
        const float re = k ? acc[0].y : acc[0].x, im = k ? acc[1].y : acc[1].x;
        if (p.out_r) {
            p.out_r[v] = re;
            p.out_i[v] = im;
        }
        if (p.image) p.image[v] = make_float2(re, im);
        if (p.vote) {
            p.vote[v] = make_float2(k ? acc[2].y : acc[2].x, k ? acc[3].y : acc[3].x);
            p.vote[p.nvox + v] = make_float2(k ? acc[4].y : acc[4].x, k ? acc[5].y : acc[5].x);
            p.vote[2 * p.nvox + v] = make_float2(k ? acc[6].y : acc[6].x,
                                                 k ? acc[7].y : acc[7].x);
        }
    }
}

// Image pass with each thread's two voxels in one grid column (z 2 r, 2 r + 1): the reference's
// squared legs are contracted fma(dz, dz, fma(dx, dx, dy dy)), so the lateral part -- and the
// vote's lateral vector -- is formed once for both.  The same bits as the flat kernel above.  CTAs
// of 128 threads, 7 (exact) or 9 (fast) to an SM.  90 x 100 x 70 voxels x 4096 antennas, four
// receivers, TI offset: exact 13.4 ms flat, 12.8; 80 x 96 x 64 x 4000, fast form: 6.2 ms flat,
// 5.8.  Four voxels a thread share more but leave 16 warps on an SM with gathers to wait for:
// 15.6 and 7.7 ms.
namespace {
constexpr int kRun = 2, kRunThreads = 128;

template <bool MONO, bool VOTE, bool SOA, bool EXACT>
__device__ __forceinline__ void run_image_chunk(const InterpParams &p, const PackAnt *sh, int a0,
                                                int n, float range_max, bool ti, float vx,
                                                float vy, const float2 (&vz)[kRun / 2],
                                                float2 (&acc)[kRun / 2][8]) {
    constexpr int kUnroll = EXACT ? 1 : 2;
#pragma unroll kUnroll
    for (int j = 0; j < n; ++j) {
        const PackAnt &a = sh[j];
        const ptrdiff_t row = (ptrdiff_t)(a0 + j) * p.nbins;
        const float dx = vx + a.ntx.x, dy = vy + a.nty.x;
        const float2 sxy = dup(__fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
        float2 txy = sxy;
        if (!MONO) {
            const float bx = dx + a.nox.x, by = dy + a.noy.x;
            txy = dup(__fmaf_rn(bx, bx, __fmul_rn(by, by)));
        }
        const float2 ex0 = dup(a.ux.x - vx), ey0 = dup(a.uy.x - vy);
#pragma unroll
        for (int q = 0; q < kRun / 2; ++q) {
            const float2 dz = __fadd2_rn(vz[q], a.ntz);
            const float2 leg = sqrt2(__ffma2_rn(dz, dz, sxy));
            float2 path;
            if (MONO) {
                path = __fadd2_rn(leg, leg);
            } else {
                const float2 bz = __fadd2_rn(dz, a.noz);
                path = __fadd2_rn(leg, sqrt2(__ffma2_rn(bz, bz, txy)));
            }
            if (ti) {  // float += double, as the reference adds its 0.15 m
                path.x += 0.15;
                path.y += 0.15;
            }
            float2 re, im;
            bool v0, v1;
            pack_terms<SOA, EXACT>(p, row, range_max, path, re, im, v0, v1);
            float2 ex = ex0, ey = ey0;
            float2 ez = __fadd2_rn(a.uz, make_float2(-vz[q].x, -vz[q].y));
            if (!(v0 && v1)) {  // a skipped pair adds nothing, whatever its vector is
                re = make_float2(v0 ? re.x : 0.f, v1 ? re.y : 0.f);
                im = make_float2(v0 ? im.x : 0.f, v1 ? im.y : 0.f);
                ex = make_float2(v0 ? ex.x : 0.f, v1 ? ex.y : 0.f);
                ey = make_float2(v0 ? ey.x : 0.f, v1 ? ey.y : 0.f);
                ez = make_float2(v0 ? ez.x : 0.f, v1 ? ez.y : 0.f);
            }
            acc[q][0] = __fadd2_rn(acc[q][0], re);
            acc[q][1] = __fadd2_rn(acc[q][1], im);
            if (VOTE) {
                acc[q][2] = __ffma2_rn(re, ex, acc[q][2]);
                acc[q][3] = __ffma2_rn(im, ex, acc[q][3]);
                acc[q][4] = __ffma2_rn(re, ey, acc[q][4]);
                acc[q][5] = __ffma2_rn(im, ey, acc[q][5]);
                acc[q][6] = __ffma2_rn(re, ez, acc[q][6]);
                acc[q][7] = __ffma2_rn(im, ez, acc[q][7]);
            }
        }
    }
}

template <bool VOTE, bool SOA, bool EXACT>
__device__ __forceinline__ void run_image_dispatch(const InterpParams &p, const PackAnt *sh,
                                                   int a0, int n, float range_max, bool ti,
                                                   bool offsets, float vx, float vy,
                                                   const float2 (&vz)[kRun / 2],
                                                   float2 (&acc)[kRun / 2][8]) {
    if (offsets) run_image_chunk<false, VOTE, SOA, EXACT>(p, sh, a0, n, range_max, ti, vx, vy, vz, acc);
    else run_image_chunk<true, VOTE, SOA, EXACT>(p, sh, a0, n, range_max, ti, vx, vy, vz, acc);
}
}  // namespace

// first, runs: the first grid column of the launch and its runs per column.
template <bool EXACT>
__global__ void __launch_bounds__(kRunThreads, EXACT ? 7 : 9)
    interp_image_run_kernel(const InterpParams p, int64_t first, int runs) {
    __shared__ PackAnt sh[kInterpChunk];
    const float range_max = p.fft_spacing * p.nbins;
    const bool ti = p.is_ti != 0;
    const int64_t slot = (int64_t)blockIdx.x * kRunThreads + threadIdx.x;
    const int64_t col = first + slot / runs;
    const int z0 = (int)(slot % runs) * kRun;
    const int64_t v0 = col * p.nz + z0;  // flat index of the run's first voxel
    const int64_t columns = (int64_t)p.nx * p.ny;
    const int64_t c = col < columns ? col : columns - 1;
    const float vx = p.x_locs[c / p.ny], vy = p.y_locs[c % p.ny];
    float pz[kRun];
#pragma unroll
    for (int k = 0; k < kRun; ++k) pz[k] = p.z_locs[min(z0 + k, p.nz - 1)];
    float2 vz[kRun / 2];
#pragma unroll
    for (int q = 0; q < kRun / 2; ++q) vz[q] = make_float2(pz[2 * q], pz[2 * q + 1]);
    float2 acc[kRun / 2][8];
#pragma unroll
    for (int q = 0; q < kRun / 2; ++q)
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[q][k] = dup(0.f);
    const bool soa = p.meas == nullptr;
    for (int a0 = 0; a0 < p.num_ant; a0 += kInterpChunk) {
        const int n = min(kInterpChunk, p.num_ant - a0);
        __syncthreads();
        stage_pack_chunk(p, a0, n, sh);
        __syncthreads();
        const bool offsets = pack_chunk_has_offsets(sh, n);
        if (p.vote) {
            if (soa) run_image_dispatch<true, true, EXACT>(p, sh, a0, n, range_max, ti, offsets, vx, vy, vz, acc);
            else run_image_dispatch<true, false, EXACT>(p, sh, a0, n, range_max, ti, offsets, vx, vy, vz, acc);
        } else {
            if (soa) run_image_dispatch<false, true, EXACT>(p, sh, a0, n, range_max, ti, offsets, vx, vy, vz, acc);
            else run_image_dispatch<false, false, EXACT>(p, sh, a0, n, range_max, ti, offsets, vx, vy, vz, acc);
        }
    }
#pragma unroll
    for (int k = 0; k < kRun; ++k) {
        const int64_t v = v0 + k;
        if (col >= columns || z0 + k >= p.nz || v < p.start || v >= p.start + p.count) continue;
        const int q = k / 2;
        const bool hi = k & 1;
        const float re = hi ? acc[q][0].y : acc[q][0].x, im = hi ? acc[q][1].y : acc[q][1].x;
        if (p.out_r) {
            p.out_r[v] = re;
            p.out_i[v] = im;
        }
        if (p.image) p.image[v] = make_float2(re, im);
        if (p.vote) {
            p.vote[v] = make_float2(hi ? acc[q][2].y : acc[q][2].x, hi ? acc[q][3].y : acc[q][3].x);
            p.vote[p.nvox + v] =
                make_float2(hi ? acc[q][4].y : acc[q][4].x, hi ? acc[q][5].y : acc[q][5].x);
            p.vote[2 * p.nvox + v] =
                make_float2(hi ? acc[q][6].y : acc[q][6].x, hi ? acc[q][7].y : acc[q][7].x);
        }
    }
}

namespace {
// mag: |I| of the two voxels (exact form, the reference's quotient) or 1/|I| (fast form).
template <bool MONO, bool SOA, bool EXACT>
__device__ __forceinline__ void pack_normals_chunk(const InterpParams &p, const PackAnt *sh,
                                                   int a0, int n, float range_max, bool ti,
                                                   float2 vx, float2 vy, float2 vz, float2 nvx,
                                                   float2 nvy, float2 nvz, float2 ire,
                                                   float2 iim, float2 mag, float2 (&acc)[3]) {
    constexpr int kUnroll = EXACT ? kExactUnroll : kFastUnroll;
#pragma unroll kUnroll
    for (int j = 0; j < n; ++j) {
        const PackAnt &a = sh[j];
        const ptrdiff_t row = (ptrdiff_t)(a0 + j) * p.nbins;
        float2 re, im;
        bool v0, v1;
        pack_terms<SOA, EXACT>(p, row, range_max, path2<MONO>(vx, vy, vz, a, ti), re, im, v0, v1);
        // weight Re(c conj(I)) / |I| (surface_normal_est.cu:138-139)
        float2 w = __ffma2_rn(re, ire, __fmul2_rn(im, iim));
        if (EXACT) w = make_float2(w.x / mag.x, w.y / mag.y);
        else w = __fmul2_rn(w, mag);
        float2 ex = __fadd2_rn(a.ux, nvx);
        float2 ey = __fadd2_rn(a.uy, nvy);
        float2 ez = __fadd2_rn(a.uz, nvz);
        if (!(v0 && v1)) {  // a skipped pair adds nothing, whatever its vector is
            w = make_float2(v0 ? w.x : 0.f, v1 ? w.y : 0.f);
            ex = make_float2(v0 ? ex.x : 0.f, v1 ? ex.y : 0.f);
            ey = make_float2(v0 ? ey.x : 0.f, v1 ? ey.y : 0.f);
            ez = make_float2(v0 ? ez.x : 0.f, v1 ? ez.y : 0.f);
        }
        acc[0] = __ffma2_rn(ex, w, acc[0]);
        acc[1] = __ffma2_rn(ey, w, acc[1]);
        acc[2] = __ffma2_rn(ez, w, acc[2]);
    }
}
}  // namespace

// Normal pass (cuda_sn_est, surface_normal_est.cu:63-149) over a valid-voxel list: entries ind
// and ind + blockDim of each 2*blockDim tile per thread.
template <bool EXACT>
__global__ void __launch_bounds__(kInterpThreads) interp_normals_pack_kernel(const InterpParams p) {
    __shared__ PackAnt sh[kInterpChunk];
    const float range_max = p.fft_spacing * p.nbins;
    const bool ti = p.is_ti != 0;
    int ind[2];
    bool active[2];
    float px[2], py[2], pz[2], pr[2], pi[2], pm[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int64_t rel = ((int64_t)blockIdx.x * 2 + k) * blockDim.x + threadIdx.x;
        const int64_t i64 = rel + p.start;
        active[k] = rel < p.count && i64 < p.num_valid && i64 >= 0;
        ind[k] = active[k] ? (int)i64 : 0;
        int x = 0, y = 0, z = 0;
        if (active[k]) {
            x = p.vidx_x[ind[k]];
            y = p.vidx_y[ind[k]];
            z = p.vidx_z[ind[k]];
        }
        px[k] = p.x_locs[x];
        py[k] = p.y_locs[y];
        pz[k] = p.z_locs[z];
        const int64_t v = ((int64_t)x * p.ny + y) * p.nz + z;
        pr[k] = active[k] ? p.img_r[v] : 1.f;
        pi[k] = active[k] ? p.img_i[v] : 0.f;
        pm[k] = sqrtf(fmaf(pr[k], pr[k], pi[k] * pi[k]));
        if (!EXACT) pm[k] = 1.f / pm[k];
    }
    const float2 vx = make_float2(px[0], px[1]), vy = make_float2(py[0], py[1]),
                 vz = make_float2(pz[0], pz[1]);
    const float2 nvx = make_float2(-px[0], -px[1]), nvy = make_float2(-py[0], -py[1]),
                 nvz = make_float2(-pz[0], -pz[1]);
    const float2 ire = make_float2(pr[0], pr[1]), iim = make_float2(pi[0], pi[1]),
                 mag = make_float2(pm[0], pm[1]);
    float2 acc[3] = {dup(0.f), dup(0.f), dup(0.f)};
    const bool soa = p.meas == nullptr;
    for (int a0 = 0; a0 < p.num_ant; a0 += kInterpChunk) {
        const int n = min(kInterpChunk, p.num_ant - a0);
        __syncthreads();
        stage_pack_chunk(p, a0, n, sh);
        __syncthreads();
        const bool offsets = pack_chunk_has_offsets(sh, n);
        if (!active[0] && !active[1]) continue;
        if (offsets) {
            if (soa) pack_normals_chunk<false, true, EXACT>(p, sh, a0, n, range_max, ti, vx, vy, vz,
                                                     nvx, nvy, nvz, ire, iim, mag, acc);
            else pack_normals_chunk<false, false, EXACT>(p, sh, a0, n, range_max, ti, vx, vy, vz, nvx,
                                                  nvy, nvz, ire, iim, mag, acc);
        } else {
            if (soa) pack_normals_chunk<true, true, EXACT>(p, sh, a0, n, range_max, ti, vx, vy, vz,
                                                    nvx, nvy, nvz, ire, iim, mag, acc);
            else pack_normals_chunk<true, false, EXACT>(p, sh, a0, n, range_max, ti, vx, vy, vz, nvx,
                                                 nvy, nvz, ire, iim, mag, acc);
        }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        if (!active[k]) continue;
        p.n_x[ind[k]] = k ? acc[0].y : acc[0].x;
        p.n_y[ind[k]] = k ? acc[1].y : acc[1].x;
        p.n_z[ind[k]] = k ? acc[2].y : acc[2].x;
    }
}

namespace {
unsigned pack_blocks(int64_t count) {
    const int64_t per = (int64_t)kInterpThreads * 2;
    return (unsigned)((count + per - 1) / per);
}
}  // namespace

// The run kernel where it wastes little: whole columns of the grid are covered, so the slots past
// a column's end (nz odd) and the parts of the first and last column outside
// [start, start + count) are idle.
static bool image_runs(const InterpParams &p, int64_t *first, int *runs, unsigned *blocks) {
    *first = p.start / p.nz;
    *runs = (p.nz + kRun - 1) / kRun;
    const int64_t columns = (p.start + p.count - 1) / p.nz - *first + 1;
    const int64_t slots = columns * *runs;
    *blocks = (unsigned)((slots + kRunThreads - 1) / kRunThreads);
    return slots * kRun <= p.count + p.count / 8;
}

cudaError_t launch_interp_image(const InterpParams &p, cudaStream_t stream) {
    if (p.count <= 0) return cudaSuccess;
    int64_t first;
    int runs;
    unsigned blocks;
    if (image_runs(p, &first, &runs, &blocks))
        interp_image_run_kernel<true><<<blocks, kRunThreads, 0, stream>>>(p, first, runs);
    else
        interp_image_pack_kernel<true><<<pack_blocks(p.count), kInterpThreads, 0, stream>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_interp_normals(const InterpParams &p, cudaStream_t stream) {
    if (p.count <= 0) return cudaSuccess;
    interp_normals_pack_kernel<true><<<pack_blocks(p.count), kInterpThreads, 0, stream>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_interp_image_fast(const InterpParams &p, cudaStream_t stream) {
    if (p.count <= 0) return cudaSuccess;
    const unsigned blocks = pack_blocks(p.count);  // kFastT == 2
    int64_t first;
    int runs;
    unsigned run_blocks;
    if (g_interp_fast_form.load() == 1)
        interp_image_fast_kernel<<<blocks, kInterpThreads, 0, stream>>>(p);
    else if (image_runs(p, &first, &runs, &run_blocks))
        interp_image_run_kernel<false><<<run_blocks, kRunThreads, 0, stream>>>(p, first, runs);
    else
        interp_image_pack_kernel<false><<<blocks, kInterpThreads, 0, stream>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_interp_normals_fast(const InterpParams &p, cudaStream_t stream) {
    if (p.count <= 0) return cudaSuccess;
    if (g_interp_fast_form.load() == 1) {
        const int64_t blocks = (p.count + kInterpThreads - 1) / kInterpThreads;
        interp_normals_fast_kernel<<<(unsigned)blocks, kInterpThreads, 0, stream>>>(p);
    } else {
        interp_normals_pack_kernel<false>
            <<<pack_blocks(p.count), kInterpThreads, 0, stream>>>(p);
    }
    return cudaGetLastError();
}

}  // namespace mmn

namespace mmn {
namespace {

__device__ __forceinline__ bool same_float(float a, float b) {
    return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b);
}

// Whether the exact form's short evaluations give the library functions' bits, for the floats with
// bit patterns first .. first + count - 1: counts[0] square roots that differ (either half of
// sqrt2), counts[1] phasors of a path that differ, counts[2] phasors that took the library.
__global__ void exact_probe_kernel(uint32_t first, uint64_t count, float wavelength, double ninv,
                                   unsigned long long *counts) {
    unsigned long long bad_root = 0, bad_phasor = 0, library = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const float x = __uint_as_float(first + (uint32_t)i);
        const float2 r = sqrt2(make_float2(x, 2.f)), s = sqrt2(make_float2(2.f, x));
        const float root = sqrtf(x);
        if (!same_float(r.x, root) || !same_float(s.y, root)) ++bad_root;
        if (wavelength > 0.f) {
            float c, sn;
            if (!phasor_exact(x, ninv, c, sn)) {
                ++library;
            } else {
                const float2 l = phasor_library(x, wavelength);
                if (!same_float(c, l.x) || !same_float(sn, l.y)) ++bad_phasor;
            }
        }
    }
    atomicAdd(counts, bad_root);
    atomicAdd(counts + 1, bad_phasor);
    atomicAdd(counts + 2, library);
}

}  // namespace
}  // namespace mmn

extern "C" int mmn_interp_exact_probe(uint32_t first, uint64_t count, float wavelength,
                                      uint64_t *counts, cudaStream_t stream) {
    if (count < 1 || count > 0x100000000ull) return MMN_ERR_INVALID_ARGUMENT;
    if (!counts) return MMN_ERR_NULL_POINTER;
    if (cudaMemsetAsync(counts, 0, 3 * sizeof(uint64_t), stream) != cudaSuccess)
        return MMN_ERR_CUDA;
    mmn::exact_probe_kernel<<<148 * 8, 256, 0, stream>>>(
        first, count, wavelength, -1.0 / (double)wavelength,
        reinterpret_cast<unsigned long long *>(counts));
    return cudaGetLastError() == cudaSuccess ? MMN_OK : MMN_ERR_CUDA;
}
