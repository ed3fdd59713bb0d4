// bp_local.cu -- the interpolation form by tile-local polynomials: the forward kernel of mode
// "nufft" (mmn_backproject_nufft) and the default kernels of both gradients.
//
// One antenna's sample sum is e^{-2pi i d t0c} M(u), u = d slope/c, with M band-limited
// (bp_nufft.cu).  Over a compact box of voxels u covers a short interval only, on which M is a
// polynomial of low degree to FP32 accuracy.  So a CTA takes a box of up to 512 voxels (8 x 8 x
// 8 on a large grid) and, for 32 antennas at a time,
//   1. bounds each antenna's range over the box: centre d_c, half width D (FP32, widened);
//   2. evaluates M at NN Chebyshev nodes of [d_c - D, d_c + D] by the 8-tap gather from the
//      antenna's grid row (global memory: the few cells a box needs stay in L1/L2);
//   3. turns the node values into polynomial coefficients in shared memory;
//   4. runs its voxels through FP64 range, FP64-wrapped anchor, one Horner evaluation and the
//      image + vote sums.
// Per (voxel, antenna) that leaves NN packed FMAs on coefficients that all voxels of the thread
// share, where a tap run per pair costs 44 FMAs of weights, 8 shared loads and the FP64 cell
// index.  A thread owns 4 voxels in a row along one axis, whose lateral distance is one.
//
// NN follows from theta = pi F |slope| / c * D, the largest phase excursion of M over the half
// width (local_nodes).  Up to NN = 12 the polynomial is evaluated in monomials by Horner (theta
// <= 2.6, so the coefficients' sum, and with it the FP32 rounding, stays within a few units).  An
// antenna whose theta is larger (from a 7 to 11 mm voxel pitch on at 4 GHz of bandwidth), or not a
// number, takes a tap run per pair (local_chunk).
//
// Bound: no single unit.  64^3 x 4096 x 128: 58 instructions a pair, issue 61 % active, FMA lanes
// 50 % (a packed instruction holds them two cycles), FP64 23 %, conversions 29 %, with the four
// warps a scheduler that 128 registers leave waiting out fixed latencies.  Measured on 96^3 voxels
// x 4096 antennas x 200 samples: 23.5 ms for the whole forward with a tap run per pair, 9.0 ms with
// this kernel; error against 64 bits 1.1e-6 before, 2.3e-7 now (sums over 32 antennas at a time).  96 or 80
// registers (5 or 6 CTAs per SM) measured the same or 2 % slower than 128.  The hardware sine
// and cosine in place of cis_half_pair: 8.1 ms, but 2.2e-7 of error on short sums, more than
// the tap form's.
#include <algorithm>
#include <cmath>
#include <cstddef>

#include "bp_stage.cuh"
#include "nufft_taps.cuh"

namespace mmn {

namespace {

constexpr int kLocThreads = 128;
constexpr int kLocRun = 4;      // voxels of a thread, consecutive in z
constexpr int kLocAnts = 32;    // antennas per chunk
constexpr int kLocNodes = 24;   // most nodes (measurement pass)
constexpr int kLocHorner = 12;  // most nodes evaluated, in monomials (forward, position pass)
constexpr int kLocWide = 99;

// Monomial coefficients of the Chebyshev polynomials T_0 .. T_11.
__constant__ float kChebMono[kLocHorner][kLocHorner] = {
    {1, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0},
    {0, 1, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0},
    {-1, 0, 2, 0, 0, 0, 0, 0, 0, 0, 0, 0},
    {0, -3, 0, 4, 0, 0, 0, 0, 0, 0, 0, 0},
    {1, 0, -8, 0, 8, 0, 0, 0, 0, 0, 0, 0},
    {0, 5, 0, -20, 0, 16, 0, 0, 0, 0, 0, 0},
    {-1, 0, 18, 0, -48, 0, 32, 0, 0, 0, 0, 0},
    {0, -7, 0, 56, 0, -112, 0, 64, 0, 0, 0, 0},
    {1, 0, -32, 0, 160, 0, -256, 0, 128, 0, 0, 0},
    {0, 9, 0, -120, 0, 432, 0, -576, 0, 256, 0, 0},
    {-1, 0, 50, 0, -400, 0, 1120, 0, -1280, 0, 512, 0},
    {0, -11, 0, 220, 0, -1232, 0, 2816, 0, -2816, 0, 1024},
};

// Nodes for a phase excursion theta: 2 (theta/2)^NN / NN! < 1.2e-7 at the band's edge, which
// is about 3e-8 rms over its samples (the error of sample j' goes with |2 j'/F|^NN);
// kLocWide: too wide for any.
__device__ __forceinline__ int local_nodes(float theta) {
    if (theta <= 0.94f) return 8;
    if (theta <= 1.72f) return 10;
    if (theta <= 2.64f) return 12;
    if (theta <= 4.8f) return 16;
    if (theta <= 9.8f) return 24;
    return kLocWide;  // NaN lands here too
}

// One antenna of a chunk, as the voxel loop reads it.
struct __align__(16) LocRec {
    double tx[3], rx[3];
    double inv, off;  // x = d * inv + off on [-1, 1]
    float txf[3], rxf[3], u[3];
    int nn;           // nodes; 0: a tap run per voxel; -1: that, and anchors from FP64 phases
};
static_assert(sizeof(LocRec) % 16 == 0, "LocRec rows are read in 16-byte words");

// Minima and maxima over the warp.
__device__ __forceinline__ void warp_bounds(float (&lo)[3], float (&hi)[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
            hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
        }
}

// Voxel box of a tile, by all threads of the CTA: per-axis minimum and maximum of the
// coordinates it covers (any order of the coordinate arrays).
__device__ __forceinline__ void tile_box(const float *locs, int first, int count, int total,
                                         float &lo, float &hi) {
    const int lane = threadIdx.x & 31;
    float a = __int_as_float(0x7f800000), b = -a;
    for (int i = lane; i < count && first + i < total; i += 32) {
        const float v = __ldg(locs + first + i);
        a = fminf(a, v);
        b = fmaxf(b, v);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a = fminf(a, __shfl_xor_sync(0xffffffffu, a, o));
        b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, o));
    }
    lo = a;
    hi = b;
}

// ... of a tile on every axis, in the boxes' axis order.
__device__ __forceinline__ void tile_bounds(const LocalParams &q, int tile, float (&lo)[3],
                                            float (&hi)[3]) {
    const LocalTiles &t = q.t;
    const int tz = tile % t.tiles_z, txy = tile / t.tiles_z;
    tile_box(q.locs[0], txy / t.tiles_y * t.bx, t.bx, t.dim[0], lo[0], hi[0]);
    tile_box(q.locs[1], txy % t.tiles_y * t.by, t.by, t.dim[1], lo[1], hi[1]);
    tile_box(q.locs[2], tz * t.runs * kLocRun, t.runs * kLocRun, t.dim[2], lo[2], hi[2]);
}

// A thread's place in its tile and its voxels' coordinates (clamped into the grid, so that
// an idle slot repeats a voxel of the box).
struct LocSlot {
    float vx, vy, vz[kLocRun];  // along the boxes' axes
    int64_t v;                  // flat index of the run's first voxel
    int count;                  // voxels of the run inside the grid; 0: an idle slot
};
// COMPACT: 32 consecutive slots are 8 x 4 columns of one layer of runs (measurement pass), not rows
// of columns of all runs.
template <bool COMPACT>
__device__ __forceinline__ LocSlot local_slot(const LocalParams &q, int tile, int slot) {
    const LocalTiles &t = q.t;
    const int tz = tile % t.tiles_z, txy = tile / t.tiles_z;
    const int ty = txy % t.tiles_y, tx = txy / t.tiles_y;
    const int used = t.bx * t.by * t.runs;
    const int s = min(slot, used - 1);
    int run = s % t.runs, c = s / t.runs, cx = c / t.by, cy = c - cx * t.by;
    if (COMPACT) {
        const int columns = t.bx * t.by, band = min(8, t.by) * t.bx;
        run = s / columns;
        c = s - run * columns;
        const int b = c / band, width = min(8, t.by - 8 * b);  // band of up to 8 columns in y
        c -= b * band;
        cx = c / width;
        cy = 8 * b + c - cx * width;
    }
    const int ix = tx * t.bx + cx, iy = ty * t.by + cy;
    const int iz = (tz * t.runs + run) * kLocRun;
    LocSlot o;
    o.vx = __ldg(q.locs[0] + min(ix, t.dim[0] - 1));
    o.vy = __ldg(q.locs[1] + min(iy, t.dim[1] - 1));
#pragma unroll
    for (int k = 0; k < kLocRun; ++k) o.vz[k] = __ldg(q.locs[2] + min(iz + k, t.dim[2] - 1));
    o.v = ix * t.stride[0] + iy * t.stride[1] + iz * t.stride[2];
    o.count = slot < used && ix < t.dim[0] && iy < t.dim[1]
                  ? max(0, min(kLocRun, t.dim[2] - iz)) : 0;
    return o;
}
// Table cos(pi m / (2 NN)), m < 4 NN, and the nodes cos(pi (i + 1/2) / NN).
__device__ __forceinline__ void cheb_tables(int nn, double *table, double *node) {
    for (int m = threadIdx.x; m < 4 * nn; m += blockDim.x) {
        const double c = cospi((double)m / (2 * nn));
        table[m] = c;
        if ((m & 1) && m < 2 * nn) node[m >> 1] = c;
    }
}

// h_k = sum_q cf[q] x_k^q for the thread's voxels.
template <int NN>
__device__ __forceinline__ void eval_mono(const float2 *cf, const float (&x)[kLocRun],
                                          float2 (&h)[kLocRun]) {
    const float4 *c4 = reinterpret_cast<const float4 *>(cf);
    const float4 top = c4[NN / 2 - 1];
#pragma unroll
    for (int k = 0; k < kLocRun; ++k)
        h[k] = __ffma2_rn(make_float2(top.z, top.w), make_float2(x[k], x[k]),
                          make_float2(top.x, top.y));
#pragma unroll
    for (int q = NN / 2 - 2; q >= 0; --q) {
        const float4 c = c4[q];
#pragma unroll
        for (int k = 0; k < kLocRun; ++k) {
            const float2 xx = make_float2(x[k], x[k]);
            h[k] = __ffma2_rn(h[k], xx, make_float2(c.z, c.w));
            h[k] = __ffma2_rn(h[k], xx, make_float2(c.x, c.y));
        }
    }
}

// h_k and its derivative g_k in x.
template <int NN>
__device__ __forceinline__ void eval_mono_d(const float2 *cf, const float (&x)[kLocRun],
                                            float2 (&h)[kLocRun], float2 (&g)[kLocRun]) {
    const float4 *c4 = reinterpret_cast<const float4 *>(cf);
    const float4 top = c4[NN / 2 - 1];
#pragma unroll
    for (int k = 0; k < kLocRun; ++k) {
        g[k] = make_float2(top.z, top.w);
        h[k] = __ffma2_rn(g[k], make_float2(x[k], x[k]), make_float2(top.x, top.y));
    }
#pragma unroll
    for (int q = NN / 2 - 2; q >= 0; --q) {
        const float4 c = c4[q];
#pragma unroll
        for (int k = 0; k < kLocRun; ++k) {
            const float2 xx = make_float2(x[k], x[k]);
            g[k] = __ffma2_rn(g[k], xx, h[k]);
            h[k] = __ffma2_rn(h[k], xx, make_float2(c.z, c.w));
            g[k] = __ffma2_rn(g[k], xx, h[k]);
            h[k] = __ffma2_rn(h[k], xx, make_float2(c.x, c.y));
        }
    }
}

// M at one node by a tap run from the antenna's row in global memory, in FP64.
__device__ __forceinline__ double2 tap_run64(const float2 *row, double d, double uq, int n) {
    int ix;
    double w[kNuW];
    nufft_taps64(d, uq, n, ix, w);
    double2 h = make_double2(0.0, 0.0);
#pragma unroll
    for (int i = 0; i < kNuW; ++i) {
        const float2 g = __ldg(row + ix + i);
        h.x = fma(w[i], (double)g.x, h.x);
        h.y = fma(w[i], (double)g.y, h.y);
    }
    return h;
}

// M at one range by a tap run.
__device__ __forceinline__ float2 tap_run(const float2 *row, double d, double uq, int n) {
    int ix;
    float w[kNuW];
    nufft_taps(d, uq, n, ix, w);
    float2 h = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < kNuW; ++i)
        h = __ffma2_rn(make_float2(w[i], w[i]), __ldg(row + ix + i), h);
    return h;
}

// The anchors e^{-2 pi i d t0c} of two ranges: wrapped turns in 2^-32 steps, or, for ranges beyond
// what those hold (local_chunk), FP64 phases.  (cos, cos, sin, sin)
__device__ __noinline__ float4 cis_wide_pair(double d0, double d1, double k0c) {
    const float2 a = cis_fp64_phase(-d0 * k0c), b = cis_fp64_phase(-d1 * k0c);
    return make_float4(a.x, b.x, a.y, b.y);
}
__device__ __forceinline__ void anchor_pair(const LocalParams &q, double d0, double d1, bool wide,
                                            float2 &c, float2 &s) {
    const double kM = 6755399441055744.0;  // 1.5 * 2^52
    if (!wide) {
        cis_half_pair(__double2loint(fma(d0, q.t0c_fixed, kM)),
                      __double2loint(fma(d1, q.t0c_fixed, kM)), c, s);
    } else {
        const float4 w = cis_wide_pair(d0, d1, q.k0c);
        c = make_float2(w.x, w.y);
        s = make_float2(w.z, w.w);
    }
}

// 1/sqrt of a sum of squares, subnormals flushed: one MUFU.
__device__ __forceinline__ float rsqrt_seed(float s) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(fmaxf(s, 1e-30f)));
    return r;
}

// Round-trip ranges of the thread's run in FP64.  Each leg is f = D r with r an FP32
// reciprocal-square-root seed of the FP32 difference vector, plus one Newton correction
// (D - f^2) r / 2 (relative error ~1e-13).
// rf, rb: the FP32 reciprocal legs.
template <bool MONO>
__device__ __forceinline__ void run_ranges(const LocRec &a, float vx, float vy,
                                           const float (&vz)[kLocRun], double ti,
                                           double (&d)[kLocRun], float (&rf)[kLocRun],
                                           float (&rb)[kLocRun]) {
    const float ax = vx - a.txf[0], ay = vy - a.txf[1];
    const float sxy = fmaf(ax, ax, ay * ay);
    const double dx = (double)vx - a.tx[0], dy = (double)vy - a.tx[1];
    const double Dxy = fma(dx, dx, dy * dy);
    const float bx = vx - a.rxf[0], by = vy - a.rxf[1];
    const float txy = fmaf(bx, bx, by * by);
    const double ex = (double)vx - a.rx[0], ey = (double)vy - a.rx[1];
    const double Exy = fma(ex, ex, ey * ey);
#pragma unroll
    for (int k = 0; k < kLocRun; ++k) {
        const float az = vz[k] - a.txf[2];
        rf[k] = rsqrt_seed(fmaf(az, az, sxy));
        const double r = (double)rf[k];
        const double dz = (double)vz[k] - a.tx[2];
        const double D = fma(dz, dz, Dxy);
        const double f = D * r, e = fma(-f, f, D);
        if (MONO) {
            d[k] = fma(e, r, fma(2.0, f, ti));  // twice the leg
        } else {
            const float bz = vz[k] - a.rxf[2];
            rb[k] = rsqrt_seed(fmaf(bz, bz, txy));
            const double s = (double)rb[k];
            const double ez = (double)vz[k] - a.rx[2];
            const double E = fma(ez, ez, Exy);
            const double g = E * s, h = fma(-g, g, E);
            d[k] = fma(0.5, fma(h, s, e * r), f + (g + ti));
        }
    }
}

// Shared memory of one CTA.
struct __align__(16) LocShared {
    LocRec rec[kLocAnts];
    double2 node_val[kLocAnts][kLocHorner];
    float2 coef[kLocAnts][kLocHorner];  // monomials
    double centre[kLocAnts], half[kLocAnts];
    double node[kLocHorner];
    double table[4 * kLocHorner];
    double basis[kLocHorner * kLocHorner];  // monomials from node values
    int nn, taps;
};
static_assert(offsetof(LocShared, node_val) % 16 == 0 && offsetof(LocShared, coef) % 16 == 0 &&
                  sizeof(float2) * kLocHorner % 16 == 0,
              "node values and monomials are read in 16-byte words");

// An antenna's positions in the boxes' axis order; t, o: TX and RX in FP32.
__device__ __forceinline__ void load_antenna(const AntRec *ar, const LocalTiles &lt, LocRec &r,
                                             float (&t)[3], float (&o)[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int x = lt.axis[k];
        r.tx[k] = ar->tx[x];
        r.rx[k] = ar->rx[x];
        r.u[k] = ar->virt[x];
        r.txf[k] = t[k] = (float)r.tx[k];
        r.rxf[k] = o[k] = (float)r.rx[k];
    }
}

// Steps 1 to 3 for antennas a0 .. a0 + na - 1.  Returns the node count of those whose boxes take
// kLocHorner nodes at most (0: none); taps: whether any takes tap runs instead.  Called by all
// threads; barriers inside.
// 16 and 24 nodes by Clenshaw's recurrence measured slower than a tap run per pair (64^3 voxels at
// a 14 mm pitch x 1024 antennas x 128 samples at 4 GHz: forward 2.47 ms and position pass 5.1;
// tap runs 1.54 and 2.38).
// Node values and coefficients are formed in FP64: their rounding is shared by all voxels of a
// box, and in FP32 it put the sums of 256 antennas 2.06e-7 from 64 bits (position gradient
// 2.27e-7), where tap runs per pair were 1.75e-7 (2.05e-7) and this is 1.78e-7 (1.98e-7).  The
// products with one basis matrix in place of two transforms pay for it: 96^3 x 4096 x 200 went
// from 9.17 to 9.02 ms.
__device__ __forceinline__ int local_chunk(const LocalParams &q, LocShared &sh, int a0, int na,
                                           const float (&lo)[3], const float (&hi)[3],
                                           int &table_nn, bool &taps) {
    const FwdParams &p = q.f;
    __syncthreads();  // the previous chunk's readers are done
    if (threadIdx.x == 0) sh.nn = sh.taps = 0;
    __syncthreads();
    if (threadIdx.x < na) {
        LocRec &r = sh.rec[threadIdx.x];
        float t[3], o[3];
        load_antenna(p.ant + a0 + threadIdx.x, q.t, r, t, o);
        float c, half, dmax;
        range_bounds(lo, hi, t, o, c, half, dmax);
        half = fmaxf(half, q.half_min);
        const double centre = (double)c + p.ti;
        sh.centre[threadIdx.x] = centre;
        sh.half[threadIdx.x] = (double)half;
        // the anchor's turn count must fit the fixed-point reduction (|turns| < 2^18)
        const bool fits = ((double)dmax + p.ti) * fabs(q.t0c) < 262144.0;
        const int nodes = local_nodes(q.theta_per_m * half);
        r.nn = !fits ? -1 : (nodes > kLocHorner ? 0 : nodes);
        const double inv = r.nn > 0 ? 1.0 / (double)half : 0.0;
        r.inv = inv;
        r.off = r.nn > 0 ? -centre * inv : 0.0;
        if (r.nn > 0) atomicMax(&sh.nn, r.nn);
        else sh.taps = 1;
    }
    __syncthreads();
    const int nn = sh.nn;
    taps = sh.taps != 0;
    if (nn == 0) return 0;
    if (nn != table_nn) {
        cheb_tables(nn, sh.table, sh.node);
        table_nn = nn;
        __syncthreads();
        // monomial c of the interpolant: sum_j basis[c][j] M_j
        for (int i = threadIdx.x; i < nn * nn; i += kLocThreads) {
            const int c = i / nn, j = i - c * nn;
            double s = 0.0;
            for (int m = c; m < nn; m += 2)
                s = fma((double)kChebMono[m][c] * (m == 0 ? 1.0 : 2.0),
                        sh.table[m * (2 * j + 1) % (4 * nn)], s);
            sh.basis[i] = s / nn;
        }
        __syncthreads();
    }
    for (int i = threadIdx.x; i < na * nn; i += kLocThreads) {
        const int la = i / nn, j = i - la * nn;
        // (an antenna with tap runs: the zero polynomial, so that the loop over the monomials
        // needs no test)
        sh.node_val[la][j] = make_double2(0.0, 0.0);
        if (sh.rec[la].nn <= 0) continue;
        const double d = fma(sh.node[j], sh.half[la], sh.centre[la]);
        sh.node_val[la][j] = tap_run64(q.rows + (size_t)(a0 + la) * q.row, d, q.uq, q.n);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < na * nn; i += kLocThreads) {
        const int la = i / nn, c = i - la * nn;
        const double *b = sh.basis + c * nn;
        double2 s = make_double2(0.0, 0.0);
        for (int j = 0; j < nn; ++j) {
            const double2 v = sh.node_val[la][j];
            s.x = fma(b[j], v.x, s.x);
            s.y = fma(b[j], v.y, s.y);
        }
        sh.coef[la][c] = make_float2((float)s.x, (float)s.y);
    }
    __syncthreads();
    return nn;
}

// Step 4 for one chunk.  NN: 8, 10 or 12, the monomials (zero for the antennas with tap runs); 0:
// those antennas.
template <bool MONO, int NN>
__device__ __forceinline__ void local_forward(const LocalParams &q, const LocShared &sh, int a0,
                                              int na, float vx, float vy,
                                              const float (&vz)[kLocRun],
                                              float2 (&acc)[kLocRun][4]) {
    for (int la = 0; la < na; ++la) {
        const LocRec &a = sh.rec[la];
        if (NN == 0 && a.nn > 0) continue;
        double d[kLocRun];
        float rf[kLocRun], rb[kLocRun];
        run_ranges<MONO>(a, vx, vy, vz, q.f.ti, d, rf, rb);
        float2 h[kLocRun];
        if (NN > 0) {
            float x[kLocRun];
#pragma unroll
            for (int k = 0; k < kLocRun; ++k) x[k] = (float)fma(d[k], a.inv, a.off);
            eval_mono<(NN > 0 ? NN : 8)>(sh.coef[la], x, h);
        } else {
            const float2 *row = q.rows + (size_t)(a0 + la) * q.row;
#pragma unroll
            for (int k = 0; k < kLocRun; ++k) h[k] = tap_run(row, d[k], q.uq, q.n);
        }
#pragma unroll
        for (int k = 0; k < kLocRun; k += 2) {
            float2 c, s;
            anchor_pair(q, d[k], d[k + 1], NN == 0 && a.nn < 0, c, s);
            h[k] = make_float2(fmaf(c.x, h[k].x, -s.x * h[k].y), fmaf(c.x, h[k].y, s.x * h[k].x));
            h[k + 1] = make_float2(fmaf(c.y, h[k + 1].x, -s.y * h[k + 1].y),
                                   fmaf(c.y, h[k + 1].y, s.y * h[k + 1].x));
        }
        // the vote about the run's first voxel: the others' share is (z_0 - z_k) I at the end
        const float ux = a.u[0] - vx, uy = a.u[1] - vy, uz = a.u[2] - vz[0];
#pragma unroll
        for (int k = 0; k < kLocRun; ++k) {
            acc[k][0] = __fadd2_rn(acc[k][0], h[k]);
            acc[k][1] = __ffma2_rn(h[k], make_float2(ux, ux), acc[k][1]);
            acc[k][2] = __ffma2_rn(h[k], make_float2(uy, uy), acc[k][2]);
            acc[k][3] = __ffma2_rn(h[k], make_float2(uz, uz), acc[k][3]);
        }
    }
}

template <bool MONO>
__device__ __forceinline__ void local_forward_nn(const LocalParams &q, const LocShared &sh, int a0,
                                                 int na, int nn, float vx, float vy,
                                                 const float (&vz)[kLocRun],
                                                 float2 (&acc)[kLocRun][4]) {
    if (nn == 8) local_forward<MONO, 8>(q, sh, a0, na, vx, vy, vz, acc);
    else if (nn == 10) local_forward<MONO, 10>(q, sh, a0, na, vx, vy, vz, acc);
    else if (nn == 12) local_forward<MONO, 12>(q, sh, a0, na, vx, vy, vz, acc);
    else local_forward<MONO, 0>(q, sh, a0, na, vx, vy, vz, acc);
}

}  // namespace

// grid = tiles x antenna splits.
__global__ void __launch_bounds__(kLocThreads, 4) bp_fwd_local_kernel(const LocalParams q) {
    __shared__ LocShared sh;
    // sums over the chunks done: a chunk's 32 antennas are summed in registers and added here,
    // which keeps the FP32 rounding of the long antenna sum down
    __shared__ float2 total[kLocRun][4][kLocThreads];
    const FwdParams &p = q.f;
    const int tile = blockIdx.x % p.num_tiles, split = blockIdx.x / p.num_tiles;
    const int a_begin = split * p.ant_per_split;
    const int a_end = min(p.num_ant, a_begin + p.ant_per_split);
    float lo[3], hi[3];
    tile_bounds(q, tile, lo, hi);
    const LocSlot s = local_slot<false>(q, tile, threadIdx.x);
    float2 acc[kLocRun][4];
#pragma unroll
    for (int k = 0; k < kLocRun; ++k)
#pragma unroll
        for (int c = 0; c < 4; ++c) total[k][c][threadIdx.x] = make_float2(0.f, 0.f);
    const bool mono = *p.mono_flag != 0;
    int table_nn = 0;
    for (int a0 = a_begin; a0 < a_end; a0 += kLocAnts) {
        const int na = min(kLocAnts, a_end - a0);
        bool taps;
        const int nn = local_chunk(q, sh, a0, na, lo, hi, table_nn, taps);
        // the antennas with monomials, then those with tap runs
        for (int pass = nn > 0 ? nn : 0;;) {
#pragma unroll
            for (int k = 0; k < kLocRun; ++k)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[k][c] = make_float2(0.f, 0.f);
            if (mono) local_forward_nn<true>(q, sh, a0, na, pass, s.vx, s.vy, s.vz, acc);
            else local_forward_nn<false>(q, sh, a0, na, pass, s.vx, s.vy, s.vz, acc);
#pragma unroll
            for (int k = 0; k < kLocRun; ++k)
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    total[k][c][threadIdx.x] = __fadd2_rn(total[k][c][threadIdx.x], acc[k][c]);
            if (pass == 0 || !taps) break;
            pass = 0;
        }
    }
    const LocSlot e = local_slot<false>(q, tile, threadIdx.x);  // (again: nothing of it stays in the loop)
    // W's components back in the grid's axis order
    int from[3];
#pragma unroll
    for (int o = 0; o < 3; ++o) from[o] = q.t.axis[0] == o ? 1 : (q.t.axis[1] == o ? 2 : 3);
#pragma unroll
    for (int k = 0; k < kLocRun; ++k) {
        if (k >= e.count) continue;
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[k][c] = total[k][c][threadIdx.x];
        const float dz = e.vz[0] - e.vz[k];
        acc[k][3] = __ffma2_rn(acc[k][0], make_float2(dz, dz), acc[k][3]);
        float a[8] = {acc[k][0].x, acc[k][0].y};
#pragma unroll
        for (int o = 0; o < 3; ++o) {
            const float2 w = from[o] == 1 ? acc[k][1] : (from[o] == 2 ? acc[k][2] : acc[k][3]);
            a[2 + 2 * o] = w.x;
            a[3 + 2 * o] = w.y;
        }
        store_voxel(p, split, e.v + k * q.t.stride[2], a);
    }
}

// ---------------------------------------------------------------- position pass
// dL/ddelta_a = sum_v Im(conj(G) c') (-(e_tx + e_rx)) + Re(conj(gW) c) (bp_backward.cu) with c'
// = sum_j kappa_j m_j p_j = i dc/dd: the derivative of the same polynomial, so the pass needs
// no second grid (M' enters scaled by bandwidth / carrier, a few per cent of c').  The four
// voxels of a thread share their lateral legs; a warp's three sums per antenna go through one
// transposed reduction (6 shuffles) and the CTA's to the per-tile partials.
namespace {

// M and dM/dd of a pair by a tap run (wide boxes).
__device__ __forceinline__ float4 tap_run_d(const float2 *row, double d, double uq, int n) {
    int ix;
    float w[kNuW], t;
    nufft_taps(d, uq, n, ix, w, &t);
    const float t2 = t * t;
    float2 h = make_float2(0.f, 0.f), g = h;
#pragma unroll
    for (int i = 0; i < kNuW; ++i) {
        // P_i'(t) = sum 2q e_q t^(2q-1) + (2q+1) o_q t^(2q); mirror taps: -P_i'(-t)
        const int m = i < kNuW / 2 ? i : kNuW - 1 - i;
        float e = (2.f * (kEsEvenTerms - 1)) * kEsEven[m][kEsEvenTerms - 1];
#pragma unroll
        for (int q = kEsEvenTerms - 2; q >= 1; --q) e = fmaf(e, t2, 2.f * q * kEsEven[m][q]);
        float o = (2.f * kEsOddTerms - 1.f) * kEsOdd[m][kEsOddTerms - 1];
#pragma unroll
        for (int q = kEsOddTerms - 2; q >= 0; --q) o = fmaf(o, t2, (2.f * q + 1.f) * kEsOdd[m][q]);
        const float wd = i < kNuW / 2 ? fmaf(t, e, o) : fmaf(t, e, -o);
        const float2 c = __ldg(row + ix + i);
        h = __ffma2_rn(make_float2(w[i], w[i]), c, h);
        g = __ffma2_rn(make_float2(wd, wd), c, g);
    }
    const float s = (float)(uq * n);
    return make_float4(h.x, h.y, g.x * s, g.y * s);
}

// Sums of v0, v1, v2 over the warp: in lanes 0-7, 8-15 and 16-23.
__device__ __forceinline__ float warp_sum3(float v0, float v1, float v2) {
    const int lane = threadIdx.x & 31;
    const bool hi = lane & 16, mid = lane & 8;
    float a = (hi ? v2 : v0) + __shfl_xor_sync(0xffffffffu, hi ? v0 : v2, 16);
    float b = v1 + __shfl_xor_sync(0xffffffffu, v1, 16);
    a = (mid ? b : a) + __shfl_xor_sync(0xffffffffu, mid ? a : b, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    return a;
}

// NN: 8, 10 or 12, the monomials (zero for the antennas with tap runs); 0: those antennas, after
// the others.
template <bool VOTE, bool MONO, int NN>
__device__ __forceinline__ void local_position(const LocalParams &q, const LocShared &sh, int a0,
                                               int na, float vx, float vy,
                                               const float (&vz)[kLocRun],
                                               const float2 (&gi)[kLocRun],
                                               const float2 (&gw)[kLocRun][3], float *wsum) {
    const int lane = threadIdx.x & 31;
    const float k0c = (float)q.k0c;
    for (int la = 0; la < na; ++la) {
        const LocRec &a = sh.rec[la];
        if (NN == 0 && a.nn > 0) continue;
        double d[kLocRun];
        float rf[kLocRun], rb[kLocRun];
        run_ranges<MONO>(a, vx, vy, vz, q.f.ti, d, rf, rb);
        float2 h[kLocRun], g[kLocRun];  // M, dM/dd
        if (NN > 0) {
            float x[kLocRun];
#pragma unroll
            for (int k = 0; k < kLocRun; ++k) x[k] = (float)fma(d[k], a.inv, a.off);
            eval_mono_d<(NN > 0 ? NN : 8)>(sh.coef[la], x, h, g);
            const float inv = (float)a.inv;
#pragma unroll
            for (int k = 0; k < kLocRun; ++k) g[k] = __fmul2_rn(g[k], make_float2(inv, inv));
        } else {
            const float2 *row = q.rows + (size_t)(a0 + la) * q.row;
#pragma unroll
            for (int k = 0; k < kLocRun; ++k) {
                const float4 t = tap_run_d(row, d[k], q.uq, q.n);
                h[k] = make_float2(t.x, t.y);
                g[k] = make_float2(t.z, t.w);
            }
        }
        const float ax = vx - a.txf[0], ay = vy - a.txf[1];
        const float bx = vx - a.rxf[0], by = vy - a.rxf[1];
        const float ux = a.u[0] - vx, uy = a.u[1] - vy;
        float sf = 0.f, sb = 0.f, g0 = 0.f, g1 = 0.f, g2 = 0.f;
#pragma unroll
        for (int k = 0; k < kLocRun; k += 2) {
            float2 ac, as;
            anchor_pair(q, d[k], d[k + 1], NN == 0 && a.nn < 0, ac, as);
#pragma unroll
            for (int l = 0; l < 2; ++l) {
                const int j = k + l;
                const float c = l ? ac.y : ac.x, s = l ? as.y : as.x;
                // c' = anchor (k0c M + i M')
                const float tr = fmaf(k0c, h[j].x, -g[j].y), ti = fmaf(k0c, h[j].y, g[j].x);
                float Gr = gi[j].x, Gi = gi[j].y;
                if (VOTE) {
                    const float uz = a.u[2] - vz[j];
                    Gr = fmaf(gw[j][0].x, ux, fmaf(gw[j][1].x, uy, fmaf(gw[j][2].x, uz, Gr)));
                    Gi = fmaf(gw[j][0].y, ux, fmaf(gw[j][1].y, uy, fmaf(gw[j][2].y, uz, Gi)));
                }
                // Im(conj(G) anchor T) = Im(B T), B = conj(G) anchor
                const float Br = fmaf(Gr, c, Gi * s), Bi = fmaf(Gr, s, -Gi * c);
                const float s1 = fmaf(Br, ti, Bi * tr);
                const float tf = s1 * rf[j];
                sf += tf;
                g2 = fmaf(-tf, vz[j] - a.txf[2], g2);
                const float tb = MONO ? tf : s1 * rb[j];
                if (!MONO) sb += tb;
                if (!MONO) g2 = fmaf(-tb, vz[j] - a.rxf[2], g2);
                if (VOTE) {
                    const float cr = fmaf(c, h[j].x, -s * h[j].y), ci = fmaf(c, h[j].y, s * h[j].x);
                    g0 = fmaf(gw[j][0].x, cr, fmaf(gw[j][0].y, ci, g0));
                    g1 = fmaf(gw[j][1].x, cr, fmaf(gw[j][1].y, ci, g1));
                    if (MONO)  // g2 is doubled below
                        g2 = fmaf(0.5f * gw[j][2].x, cr, fmaf(0.5f * gw[j][2].y, ci, g2));
                    else
                        g2 = fmaf(gw[j][2].x, cr, fmaf(gw[j][2].y, ci, g2));
                }
            }
        }
        if (MONO) {
            g0 = fmaf(-2.f * ax, sf, g0);
            g1 = fmaf(-2.f * ay, sf, g1);
            g2 += g2;
        } else {
            g0 = fmaf(-ax, sf, fmaf(-bx, sb, g0));
            g1 = fmaf(-ay, sf, fmaf(-by, sb, g1));
        }
        const float s = warp_sum3(g0, g1, g2);
        if ((lane & 7) == 0 && lane < 24) wsum[la * 3 + (lane >> 3)] = s;
    }
}

template <bool VOTE, bool MONO>
__device__ __forceinline__ void local_position_nn(const LocalParams &q, const LocShared &sh,
                                                  int a0, int na, int nn, bool taps, float vx,
                                                  float vy,
                                                  const float (&vz)[kLocRun],
                                                  const float2 (&gi)[kLocRun],
                                                  const float2 (&gw)[kLocRun][3], float *wsum) {
    if (nn == 8) local_position<VOTE, MONO, 8>(q, sh, a0, na, vx, vy, vz, gi, gw, wsum);
    else if (nn == 10) local_position<VOTE, MONO, 10>(q, sh, a0, na, vx, vy, vz, gi, gw, wsum);
    else if (nn == 12) local_position<VOTE, MONO, 12>(q, sh, a0, na, vx, vy, vz, gi, gw, wsum);
    if (taps) local_position<VOTE, MONO, 0>(q, sh, a0, na, vx, vy, vz, gi, gw, wsum);
}

}  // namespace

// grid = tiles x antenna splits.  VOTE: the loss has a vote term.
template <bool VOTE>
__global__ void __launch_bounds__(kLocThreads, 4) bp_bwd_pos_local_kernel(const LocalParams q) {
    __shared__ LocShared sh;
    __shared__ float wsum[kLocThreads / 32][kLocAnts * 3];
    const FwdParams &p = q.f;
    const int tile = blockIdx.x % p.num_tiles, split = blockIdx.x / p.num_tiles;
    const int a_begin = split * p.ant_per_split;
    const int a_end = min(p.num_ant, a_begin + p.ant_per_split);
    float lo[3], hi[3];
    tile_bounds(q, tile, lo, hi);
    const LocSlot s = local_slot<false>(q, tile, threadIdx.x);
    float2 gi[kLocRun], gw[kLocRun][3];
#pragma unroll
    for (int k = 0; k < kLocRun; ++k) {
        const bool ok = k < s.count;
        const int64_t v = ok ? s.v + k * q.t.stride[2] : 0;
        gi[k] = ok && q.grad_image ? q.grad_image[v] : make_float2(0.f, 0.f);
#pragma unroll
        for (int c = 0; c < 3; ++c)
            gw[k][c] = VOTE && ok ? q.grad_vote[q.t.axis[c] * p.nvox + v] : make_float2(0.f, 0.f);
    }
    const bool mono = *p.mono_flag != 0;
    float *mine = wsum[threadIdx.x >> 5];
    int table_nn = 0;
    for (int a0 = a_begin; a0 < a_end; a0 += kLocAnts) {
        const int na = min(kLocAnts, a_end - a0);
        bool taps;
        const int nn = local_chunk(q, sh, a0, na, lo, hi, table_nn, taps);
        if (mono)
            local_position_nn<VOTE, true>(q, sh, a0, na, nn, taps, s.vx, s.vy, s.vz, gi, gw, mine);
        else
            local_position_nn<VOTE, false>(q, sh, a0, na, nn, taps, s.vx, s.vy, s.vz, gi, gw, mine);
        __syncthreads();
        for (int i = threadIdx.x; i < na * 3; i += kLocThreads) {
            float t = 0.f;
#pragma unroll
            for (int w = 0; w < kLocThreads / 32; ++w) t += wsum[w][i];
            const int la = i / 3, c = i - 3 * la;
            q.pos_partial[((size_t)tile * p.num_ant + a0 + la) * 3 + q.t.axis[c]] = t;
        }
    }
}

const void *bwd_pos_local_kernel_ptr(bool vote, int *threads) {
    *threads = kLocThreads;
    return vote ? reinterpret_cast<const void *>(&bp_bwd_pos_local_kernel<true>)
                : reinterpret_cast<const void *>(&bp_bwd_pos_local_kernel<false>);
}

// ------------------------------------------------------------- measurement pass
// dL/dm[a, J0+j'] = sum_v h_v e^{2 pi i j' u_v}, h_v = G_a(v) conj(anchor): the transpose of the
// forward's evaluation.  Per (box, antenna) the voxels' h are reduced to NN Chebyshev moments
// sum_v h_v T_q(x_v) in registers (two packed instructions each); the transposed interpolation
// turns the moments into NN node values, and only those are spread onto the antenna's grid row
// (8 cells each).  A warp owns one antenna and its row and walks a range of boxes, 32 voxel
// runs at a time; everything is summed in a fixed order.  Boxes too wide for the nodes go in parts,
// and parts of 128 voxels that still are spread every voxel.
//
// A box costs some 700 instructions besides its voxels' 90 each (bounds, the warp sums, the
// spread), so boxes are larger than the forward's where enough of them remain to fill the GPU:
// 2048, else 1024, else 512 voxels.  64^3 voxels x 4096 antennas x 128 samples (this pass):
// 16.3 ms with a spread per voxel, 6.2 / 5.1 / 4.5 ms with boxes of 512 / 1024 / 2048.  Bound as
// the forward: 94 instructions a pair, issue 62 % active, FMA lanes 49 %, conversions 29 %.
namespace {

constexpr int kLocMeasWarps = 4;

// Voxel records in box order: per box q.slots x (x, y, -, -), (z_0 .. z_3), then per run
// position k (gI) or (gI, gW_x), (gW_y, gW_z); and the boxes' bounds.
struct LocVox {
    float4 *xy, *z, *box;  // [tiles][slots], [tiles][slots], [tiles][2]
    float4 *g;             // vote: [tiles][4][2][slots] float4; image only: [tiles][4][slots] float2
};
__device__ __forceinline__ LocVox loc_vox(const LocalParams &q) {
    LocVox r;
    const size_t n = (size_t)q.f.num_tiles * q.slots;
    r.box = q.vox;
    r.xy = r.box + 2 * (size_t)q.f.num_tiles;
    r.z = r.xy + n;
    r.g = r.z + n;
    return r;
}

__global__ void __launch_bounds__(512) local_vox_kernel(const LocalParams q) {
    const FwdParams &p = q.f;
    const int tile = blockIdx.x, slot = threadIdx.x;
    const LocVox r = loc_vox(q);
    float lo[3], hi[3];
    tile_bounds(q, tile, lo, hi);
    if (slot == 0) {
        r.box[2 * tile] = make_float4(lo[0], lo[1], lo[2], 0.f);
        r.box[2 * tile + 1] = make_float4(hi[0], hi[1], hi[2], 0.f);
    }
    const LocSlot s = local_slot<true>(q, tile, slot);
    const size_t at = (size_t)tile * q.slots + slot;
    r.xy[at] = make_float4(s.vx, s.vy, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < kLocRun; ++k) {
        const bool ok = k < s.count;
        const int64_t v = ok ? s.v + k * q.t.stride[2] : 0;
        const float2 zero = make_float2(0.f, 0.f);
        const float2 gi = ok && q.grad_image ? q.grad_image[v] : zero;
        const size_t gk = (size_t)tile * kLocRun + k;
        if (q.grad_vote) {
            const float2 a = ok ? q.grad_vote[q.t.axis[0] * p.nvox + v] : zero,
                         b = ok ? q.grad_vote[q.t.axis[1] * p.nvox + v] : zero,
                         c = ok ? q.grad_vote[q.t.axis[2] * p.nvox + v] : zero;
            r.g[(2 * gk) * q.slots + slot] = make_float4(gi.x, gi.y, a.x, a.y);
            r.g[(2 * gk + 1) * q.slots + slot] = make_float4(b.x, b.y, c.x, c.y);
        } else {
            reinterpret_cast<float2 *>(r.g)[gk * q.slots + slot] = gi;
        }
    }
    r.z[at] = make_float4(s.vz[0], s.vz[1], s.vz[2], s.vz[3]);
}

// Tables of every node count, back to back: cos(pi m / (2 NN)), m < 4 NN, and the nodes.
constexpr int kNodeTotal = 8 + 10 + 12 + 16 + 24;
__device__ __forceinline__ int node_offset(int nn) {  // sum of the smaller counts
    return nn == 8 ? 0 : nn == 10 ? 8 : nn == 12 ? 18 : nn == 16 ? 30 : 46;
}

constexpr int kNuWin = 16;  // cells of a window (spread_voxels)

// Per-warp scratch of the spread.
struct __align__(16) LocSpread {
    union {
        float2 w[32][kNuW];       // node values: tap weights by lane
        float2 win[kNuWin][32];   // voxels: a window's cells by lane
    };
    int ix[32];
    float box[6];             // bounds of a part of a box
    double centre, half;      // its range interval, and slots a part, kept out of registers
    int part;
    alignas(16) double mom[2 * kLocNodes];  // (re, im) pairs
};
static_assert(offsetof(LocSpread, mom) % 16 == 0 && sizeof(LocSpread) % 16 == 0,
              "moments are read in 16-byte words");

// Adds a node value per active lane times its tap weights at range d to the warp's grid row, in
// lane order per cell.  The weights are formed in FP64 (their rounding would be all of the box's
// voxels').
__device__ __noinline__ void spread_row(LocSpread &sp, float2 *row, int mrow, double d,
                                        float2 value, bool active, double uq, int n) {
    const int lane = threadIdx.x & 31;
    int ix;
    float w[kNuW];
    {
        double w64[kNuW];
        nufft_taps64(d, uq, n, ix, w64);
#pragma unroll
        for (int i = 0; i < kNuW; ++i) w[i] = (float)w64[i];
    }
#pragma unroll
    for (int i = 0; i < kNuW; ++i) sp.w[lane][i] = make_float2(value.x * w[i], value.y * w[i]);
    sp.ix[lane] = ix;
    __syncwarp();
    unsigned pending = __ballot_sync(0xffffffffu, active);
    while (pending) {
        const bool mine_p = (pending >> lane) & 1u;
        const int base = __reduce_min_sync(0xffffffffu, mine_p ? ix : 0x7fffffff);
        const unsigned mine = __ballot_sync(0xffffffffu, mine_p && ix - base <= 32 - kNuW);
        float2 s = make_float2(0.f, 0.f);
        for (unsigned m = mine; m; m &= m - 1) {
            const int i = __ffs(m) - 1;
            const unsigned o = (unsigned)(base + lane - sp.ix[i]);
            if (o < (unsigned)kNuW) s = __fadd2_rn(s, sp.w[i][o]);
        }
        if (base + lane < mrow) row[base + lane] = __fadd2_rn(row[base + lane], s);
        pending &= ~mine;
        // the next window, 25 cells on or less where the row wraps, reads cells that other lanes
        // wrote here (the ballot orders no memory); it also frees the scratch for the next call
        __syncwarp();
    }
}

// The same for a voxel per lane: windows of 16 cells from the least cell left, each lane's products
// with its weights (FP32) put into its column of the window, 32 components summed over the lanes by
// a transposing reduction.  (Column entry s of lane l holds component s ^ l, cell by cell: every
// access of a half-warp falls in 16 different banks.)  A fifth of spread_row's instructions where
// all 32 lanes have values.
__device__ __noinline__ void spread_voxels(LocSpread &sp, float2 *row, double d, float2 value,
                                           double uq, int n) {
    const int lane = threadIdx.x & 31;
    int ix;
    float w[kNuW];
    nufft_taps(d, uq, n, ix, w);
    const bool odd = lane & 1;  // odd lanes keep (im, re)
    const float h0 = odd ? value.y : value.x, h1 = odd ? value.x : value.y;
    float *rowf = reinterpret_cast<float *>(row);
    unsigned pending = 0xffffffffu;
    while (pending) {
        const bool left = (pending >> lane) & 1u;
        const int base = __reduce_min_sync(0xffffffffu, left ? ix : 0x7fffffff);
        const int off = ix - base;
        const bool mine = left && off <= kNuWin - kNuW;
        if (mine) {
#pragma unroll
            for (int i = 0; i < kNuW; ++i)
                sp.win[off + i][lane] = make_float2(h0 * w[i], h1 * w[i]);
        }
        float v[32];
#pragma unroll
        for (int s = 0; s < kNuWin; ++s) {
            const int cell = s ^ (lane >> 1), i = cell - off;
            float2 t = make_float2(0.f, 0.f);
            if (mine && i >= 0 && i < kNuW) t = sp.win[cell][lane];
            v[2 * s] = t.x;
            v[2 * s + 1] = t.y;
        }
#pragma unroll
        for (int h = 16; h >= 1; h >>= 1) {
#pragma unroll
            for (int i = 0; i < h; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i + h], h);
        }
        rowf[2 * (base + (lane >> 1)) + (lane & 1)] += v[0];
        pending &= ~__ballot_sync(0xffffffffu, mine);
        __syncwarp();  // the next window reads cells that other lanes wrote here
    }
}

// Transposed warp sum of N (a power of two) values: out[i] = sum over lanes of v[i].  FP64 past
// the first level, which halves their number.
template <int N>
__device__ __forceinline__ void warp_sums(const float *v, double *out) {
    const int lane = threadIdx.x & 31;
    constexpr int H = N / 2;
    double w[H];
    int at = 0;  // index of w[0] in the original order
    {
        const bool up = lane & 16;
#pragma unroll
        for (int i = 0; i < H; ++i) {
            const float send = up ? v[i] : v[i + H], keep = up ? v[i + H] : v[i];
            w[i] = (double)keep + (double)__shfl_xor_sync(0xffffffffu, send, 16);
        }
        at += up ? H : 0;
    }
    int bit = 8;
#pragma unroll
    for (int h = H / 2; h >= 1; h >>= 1, bit >>= 1) {
        const bool up = lane & bit;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const double send = up ? w[i] : w[i + h], keep = up ? w[i + h] : w[i];
            w[i] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
        }
        at += up ? h : 0;
    }
#pragma unroll
    for (; bit >= 1; bit >>= 1) w[0] += __shfl_xor_sync(0xffffffffu, w[0], bit);
    out[at] = w[0];  // the lanes of a group write the same value
}

// Bounds of `count` slots (a multiple of 32) of the records xys, zs into box, by the warp.
__device__ __noinline__ void slot_bounds(const float4 *xys, const float4 *zs, int count,
                                         float *box) {
    const float inf = __int_as_float(0x7f800000);
    float lo[3] = {inf, inf, inf}, hi[3] = {-inf, -inf, -inf};
    for (int i = threadIdx.x & 31; i < count; i += 32) {
        const float4 xy = __ldg(xys + i), z = __ldg(zs + i);
        lo[0] = fminf(lo[0], xy.x);
        hi[0] = fmaxf(hi[0], xy.x);
        lo[1] = fminf(lo[1], xy.y);
        hi[1] = fmaxf(hi[1], xy.y);
        lo[2] = fminf(lo[2], fminf(fminf(z.x, z.y), fminf(z.z, z.w)));
        hi[2] = fmaxf(hi[2], fmaxf(fmaxf(z.x, z.y), fmaxf(z.z, z.w)));
    }
    warp_bounds(lo, hi);
    __syncwarp();
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            box[k] = lo[k];
            box[3 + k] = hi[k];
        }
    __syncwarp();
}

// A part of a box against the warp's antenna: the moments into sp.mom (NN > 0), or every voxel's
// spread (NN = 0).
template <bool VOTE, bool MONO, int NN>
__device__ __forceinline__ void box_moments(const LocalParams &q, const LocVox &vx, int tile,
                                            int s0, int s1, const LocRec &a, LocSpread &sp,
                                            float2 *row, int mrow) {
    const double kM = 6755399441055744.0;  // 1.5 * 2^52
    const int lane = threadIdx.x & 31;
    constexpr int NV = NN > 0 ? NN : 1;
    // Voxels of a run taken together: their terms are added up before they join a moment, which
    // halves the additions to it (all four measured 2 % slower in registers spilled).  With that,
    // the warp sums and node values in FP64 and FP64 weights of the nodes, the gradient is 1.62e-7
    // from 64 bits, where a term at a time and FP32 throughout were 1.92e-7 and a spread per voxel
    // 1.59e-7.
    constexpr int L = 2;
    float2 mom[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) mom[i] = make_float2(0.f, 0.f);
    // The coordinates lead the FP64 chain and come from L2: a run ahead (64^3 voxels x 4096 antennas x
    // 128 samples, forward and backward: 12.56 -> 12.36 ms).
    const float4 *pxy = vx.xy + (size_t)tile * q.slots, *pz = vx.z + (size_t)tile * q.slots;
    float4 nxy = __ldg(pxy + s0 + lane), nz = __ldg(pz + s0 + lane);
#pragma unroll 1
    for (int slot = s0 + lane; slot < s1; slot += 32) {
        const float4 xy = nxy, z4 = nz;
        if (slot + 32 < s1) {
            nxy = __ldg(pxy + slot + 32);
            nz = __ldg(pz + slot + 32);
        }
        const float vz[kLocRun] = {z4.x, z4.y, z4.z, z4.w};
        double d[kLocRun];
        float rf[kLocRun], rb[kLocRun];
        run_ranges<MONO>(a, xy.x, xy.y, vz, q.f.ti, d, rf, rb);
        const float ux = a.u[0] - xy.x, uy = a.u[1] - xy.y;
#pragma unroll
        for (int k = 0; k < kLocRun; k += L) {
            float2 t0[L], t1[L];
            float x[L];
#pragma unroll
            for (int l = 0; l < L; ++l) {
                const int j = k + l;
                const size_t gk = (size_t)tile * kLocRun + j;
                float Gr, Gi;
                if (VOTE) {
                    const float4 g0 = __ldg(vx.g + (2 * gk) * q.slots + slot);
                    const float4 g1 = __ldg(vx.g + (2 * gk + 1) * q.slots + slot);
                    const float uz = a.u[2] - vz[j];
                    Gr = fmaf(g1.z, uz, fmaf(g1.x, uy, fmaf(g0.z, ux, g0.x)));
                    Gi = fmaf(g1.w, uz, fmaf(g1.y, uy, fmaf(g0.w, ux, g0.y)));
                } else {
                    const float2 g = __ldg(reinterpret_cast<const float2 *>(vx.g) +
                                           gk * q.slots + slot);
                    Gr = g.x;
                    Gi = g.y;
                }
                t0[l] = make_float2(Gr, Gi);
            }
            if (NN > 0) {
                float2 ac, as;
                cis_half_pair(__double2loint(fma(d[k], q.t0c_fixed, kM)),
                              __double2loint(fma(d[k + 1], q.t0c_fixed, kM)), ac, as);
                const float2 g = t0[0], h = t0[1];
                t0[0] = make_float2(fmaf(g.x, ac.x, g.y * as.x), fmaf(g.y, ac.x, -g.x * as.x));
                t0[1] = make_float2(fmaf(h.x, ac.y, h.y * as.y), fmaf(h.y, ac.y, -h.x * as.y));
#pragma unroll
                for (int l = 0; l < L; ++l) {
                    x[l] = (float)fma(d[k + l], a.inv, a.off);
                    t1[l] = __fmul2_rn(make_float2(x[l], x[l]), t0[l]);
                    x[l] += x[l];
                }
                mom[0] = __fadd2_rn(mom[0], __fadd2_rn(t0[0], t0[1]));
                mom[1 % NV] = __fadd2_rn(mom[1 % NV], __fadd2_rn(t1[0], t1[1]));
#pragma unroll
                for (int i = 2; i < NN; ++i) {
#pragma unroll
                    for (int l = 0; l < L; ++l) {
                        const float2 t2 = __ffma2_rn(make_float2(x[l], x[l]), t1[l],
                                                     make_float2(-t0[l].x, -t0[l].y));
                        t0[l] = t1[l];
                        t1[l] = t2;
                    }
                    mom[i % NV] = __fadd2_rn(mom[i % NV], __fadd2_rn(t1[0], t1[1]));
                }
            } else {
#pragma unroll
                for (int l = 0; l < L; ++l) {
                    const float2 an = cis_fp64_phase(-d[k + l] * q.k0c);
                    spread_voxels(sp, row, d[k + l],
                                  make_float2(fmaf(t0[l].x, an.x, t0[l].y * an.y),
                                              fmaf(t0[l].y, an.x, -t0[l].x * an.y)),
                                  q.uq, q.n);
                }
            }
        }
    }
    if (NN > 0) {
        float *v = reinterpret_cast<float *>(mom);
        if (NN == 8) warp_sums<16>(v, sp.mom);
        if (NN == 10) {
            warp_sums<16>(v, sp.mom);
            warp_sums<4>(v + 16, sp.mom + 16);
        }
        if (NN == 12) {
            warp_sums<16>(v, sp.mom);
            warp_sums<8>(v + 16, sp.mom + 16);
        }
        if (NN == 16) warp_sums<32>(v, sp.mom);
        if (NN == 24) {
            warp_sums<32>(v, sp.mom);
            warp_sums<16>(v + 32, sp.mom + 32);
        }
        __syncwarp();
    }
}

template <bool VOTE, bool MONO>
__device__ __forceinline__ void box_moments_nn(const LocalParams &q, const LocVox &vx, int tile,
                                               int s0, int s1, const LocRec &a, LocSpread &sp, float2 *row,
                                               int mrow) {
    switch (a.nn) {
        case 8: box_moments<VOTE, MONO, 8>(q, vx, tile, s0, s1, a, sp, row, mrow); break;
        case 10: box_moments<VOTE, MONO, 10>(q, vx, tile, s0, s1, a, sp, row, mrow); break;
        case 12: box_moments<VOTE, MONO, 12>(q, vx, tile, s0, s1, a, sp, row, mrow); break;
        case 16: box_moments<VOTE, MONO, 16>(q, vx, tile, s0, s1, a, sp, row, mrow); break;
        case 24: box_moments<VOTE, MONO, 24>(q, vx, tile, s0, s1, a, sp, row, mrow); break;
        default: box_moments<VOTE, MONO, 0>(q, vx, tile, s0, s1, a, sp, row, mrow);
    }
}

}  // namespace

// blockIdx.x = antenna group (one antenna per warp) + groups * box range.
template <bool VOTE>
__global__ void __launch_bounds__(kLocMeasWarps * 32, 4)
    bp_bwd_meas_local_kernel(const LocalParams q, float2 *part, int mrow, int tiles_per_range) {
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ LocRec s_rec[kLocMeasWarps];
    __shared__ LocSpread s_spread[kLocMeasWarps];
    __shared__ double s_node[kNodeTotal];
    __shared__ double s_table[4 * kNodeTotal];
    const FwdParams &p = q.f;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int groups = (p.num_ant + kLocMeasWarps - 1) / kLocMeasWarps;
    const int a = blockIdx.x % groups * kLocMeasWarps + warp, range = blockIdx.x / groups;
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        const int nn = c < 3 ? 8 + 2 * c : 8 * (c - 1);
        cheb_tables(nn, s_table + 4 * node_offset(nn), s_node + node_offset(nn));
    }
    __syncthreads();
    if (a >= p.num_ant) return;  // warps are independent from here on
    float2 *row = reinterpret_cast<float2 *>(dyn) + (size_t)warp * mrow;
    for (int c = lane; c < mrow; c += 32) row[c] = make_float2(0.f, 0.f);
    LocRec &rec = s_rec[warp];
    LocSpread &sp = s_spread[warp];
    float t[3], r[3];
    {
        LocRec mine;
        load_antenna(p.ant + a, q.t, mine, t, r);
        if (lane == 0) rec = mine;
    }
    const bool mono = *p.mono_flag != 0;
    const LocVox vx = loc_vox(q);
    const int t0 = range * tiles_per_range, t1 = min(p.num_tiles, t0 + tiles_per_range);
    // a box too wide for kLocNodes goes in parts, down to 32 slots
    int tile = t0, s0 = 0;
    if (lane == 0) sp.part = q.slots;
    __syncwarp();
    while (tile < t1) {
        int s1 = min(s0 + sp.part, q.slots);
        float4 l4, h4;
        if (s1 - s0 == q.slots) {
            l4 = __ldg(vx.box + 2 * tile);
            h4 = __ldg(vx.box + 2 * tile + 1);
        } else {
            const size_t at = (size_t)tile * q.slots + s0;
            slot_bounds(vx.xy + at, vx.z + at, s1 - s0, sp.box);
            l4 = make_float4(sp.box[0], sp.box[1], sp.box[2], 0.f);
            h4 = make_float4(sp.box[3], sp.box[4], sp.box[5], 0.f);
        }
        const float lo[3] = {l4.x, l4.y, l4.z}, hi[3] = {h4.x, h4.y, h4.z};
        float c, half, dmax;
        range_bounds(lo, hi, t, r, c, half, dmax);
        half = fmaxf(half, q.half_min);
        const double centre = (double)c + p.ti;
        const bool fits = ((double)dmax + p.ti) * fabs(q.t0c) < 262144.0;
        const int nodes = local_nodes(q.theta_per_m * half);
        if (fits && nodes == kLocWide && s1 - s0 > 32) {
            __syncwarp();
            if (lane == 0) sp.part = ((s1 - s0) / 2 + 31) / 32 * 32;
            __syncwarp();
            continue;
        }
        const int nn = fits && nodes != kLocWide ? nodes : 0;
        if (nn == 0) s1 = q.slots;  // the rest of the box by voxels too
        __syncwarp();
        if (lane == 0) {
            const double inv = 1.0 / (double)half;
            rec.inv = inv;
            rec.off = -centre * inv;
            rec.nn = nn;
            sp.centre = centre;
            sp.half = (double)half;
        }
        __syncwarp();
        if (mono) box_moments_nn<VOTE, true>(q, vx, tile, s0, s1, rec, sp, row, mrow);
        else box_moments_nn<VOTE, false>(q, vx, tile, s0, s1, rec, sp, row, mrow);
        if (nn > 0) {
            // node values: sum_q (2 - [q = 0]) / NN cos(pi q (2 i + 1) / (2 NN)) moment_q
            const int no = node_offset(nn), i = min(lane, nn - 1);
            const double *table = s_table + 4 * no;
            const double2 *mom = reinterpret_cast<const double2 *>(sp.mom);
            double2 s = make_double2(0.5 * mom[0].x, 0.5 * mom[0].y);
            int m = 2 * i + 1;
            for (int k = 1; k < nn; ++k) {
                const double w = table[m];
                s.x = fma(w, mom[k].x, s.x);
                s.y = fma(w, mom[k].y, s.y);
                m += 2 * i + 1;
                if (m >= 4 * nn) m -= 4 * nn;
            }
            const double sc = 2.0 / nn;
            spread_row(sp, row, mrow, fma(s_node[no + i], sp.half, sp.centre),
                       make_float2((float)(s.x * sc), (float)(s.y * sc)), lane < nn, q.uq, q.n);
        }
        s0 = s1 < q.slots ? s1 : 0;
        if (s0 == 0) {
            ++tile;
            __syncwarp();
            if (lane == 0) sp.part = min(2 * sp.part, q.slots);
            __syncwarp();
        }
    }
    __syncwarp();
    float2 *dst = part + ((size_t)range * p.num_ant + a) * mrow;
    for (int c = lane; c < mrow; c += 32) dst[c] = row[c];
}

size_t local_meas_vox_bytes(int64_t tiles, int slots) {
    return (size_t)tiles * (2 + (size_t)slots * (2 + 2 * kLocRun)) * sizeof(float4);
}

size_t local_meas_smem(int mrow) { return (size_t)kLocMeasWarps * mrow * sizeof(float2); }

int local_meas_warps() { return kLocMeasWarps; }

const void *local_meas_kernel_ptr(bool vote) {
    return vote ? reinterpret_cast<const void *>(&bp_bwd_meas_local_kernel<true>)
                : reinterpret_cast<const void *>(&bp_bwd_meas_local_kernel<false>);
}

cudaError_t launch_local_meas(const LocalParams &q, float2 *part, int mrow, int ranges,
                              int tiles_per_range, cudaStream_t stream) {
    local_vox_kernel<<<q.f.num_tiles, q.slots, 0, stream>>>(q);
    const void *fn = local_meas_kernel_ptr(q.grad_vote != nullptr);
    const size_t smem = local_meas_smem(mrow);
    if (smem > 24 * 1024)
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const int groups = (q.f.num_ant + kLocMeasWarps - 1) / kLocMeasWarps;
    void *args[] = {const_cast<LocalParams *>(&q), &part, &mrow, &tiles_per_range};
    return cudaLaunchKernel(fn, dim3((unsigned)((int64_t)groups * ranges)),
                            dim3(kLocMeasWarps * 32), args, smem, stream);
}

// Box shape for one order of the axes (the grid's extents along them, the runs' last): columns
// bx x by and runs, at most `most` runs in all and at most `side` columns or voxels a side, chosen
// for few boxes (idle slots of a ragged grid cost as much as used ones) with a charge for elongated
// ones, whose wider range interval needs more nodes.  8 x 8 x 8 on a large grid.  Returns the cost.
static double plan_order(const int (&dim)[3], int most, int side, LocalTiles *t) {
    double best = 1e300;
    const int zr = (dim[2] + kLocRun - 1) / kLocRun;
    const double cube = std::sqrt(3.0) * std::cbrt((double)most * kLocRun);
    for (int r = 1; r <= std::min({zr, most, std::max(side / 2, 1)}); ++r)
        for (int y = 1; y <= std::min(dim[1], side) && r * y <= most; ++y) {
            const int x = std::min({dim[0], most / (r * y), side});
            const double tiles = (double)((dim[0] + x - 1) / x) * ((dim[1] + y - 1) / y) *
                                 ((zr + r - 1) / r);
            const double diag2 = (double)x * x + (double)y * y +
                                 (double)(kLocRun * r) * (kLocRun * r);
            const double cost = tiles * (1.0 + 0.01 * std::max(0.0, std::sqrt(diag2) - cube));
            if (cost < best) {
                best = cost;
                t->bx = x;
                t->by = y;
                t->runs = r;
            }
        }
    return best;
}

// The runs lie along z unless that leaves over a quarter of the slots idle (a grid thin in z: a
// plane used one voxel of a run's four, 1.9 ms for 300 x 300 x 1 voxels x 2048 antennas x 128
// samples; along y 0.6) and another axis does at least a tenth better.  Lines and bars also get
// longer boxes than the 32 a side that wider grids do (8192 voxels in a row x 4096 antennas: 1.6 ms
// with 16 of 128 threads at work, 0.17 so).
void plan_local_tiles(int nx, int ny, int nz, int most, LocalTiles *t) {
    static const int order[3][3] = {{0, 1, 2}, {0, 2, 1}, {1, 2, 0}};
    const int n[3] = {nx, ny, nz};
    const int64_t stride[3] = {(int64_t)ny * nz, nz, 1};
    const auto share = [&](double cost) {  // of the slots in use, if boxes are not elongated
        return (double)nx * ny * nz / (cost * most * kLocRun);
    };
    double best = 1e300;
    for (int side : {32, 2 * most}) {
        for (const auto &o : order) {
            LocalTiles c;
            const int dim[3] = {n[o[0]], n[o[1]], n[o[2]]};
            const double cost = plan_order(dim, most, side, &c);
            if (cost >= 0.9 * best) continue;
            best = cost;
            *t = c;
            for (int k = 0; k < 3; ++k) {
                t->axis[k] = o[k];
                t->dim[k] = dim[k];
                t->stride[k] = stride[o[k]];
            }
            if (share(best) > 0.75) break;
        }
        if (share(best) > 0.5) break;
    }
    t->tiles_y = (t->dim[1] + t->by - 1) / t->by;
    t->tiles_z = (t->dim[2] + kLocRun * t->runs - 1) / (kLocRun * t->runs);
    t->tiles = (int64_t)((t->dim[0] + t->bx - 1) / t->bx) * t->tiles_y * t->tiles_z;
}

const void *fwd_local_kernel_ptr(int *threads) {
    *threads = kLocThreads;
    return reinterpret_cast<const void *>(&bp_fwd_local_kernel);
}

int local_chunk_antennas() { return kLocAnts; }

}  // namespace mmn
