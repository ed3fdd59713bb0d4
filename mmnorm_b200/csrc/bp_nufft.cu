// bp_nufft.cu -- the adjoint's two passes in interpolation form.
//
// Position pass.  The position gradient needs, per (voxel v, antenna a), the two sums
//   c_a(v)  = sum_j m[a,j] p_aj(v),   c'_a(v) = sum_j kappa_j m[a,j] p_aj(v),
//   p_aj = exp(-i d kappa_j),  kappa_j = 2pi(1/lambda + j slope/c).
// Both are one antenna's discrete-time Fourier sum evaluated at the point
// u = d slope / c (turns per sample):  c = e^{-2pi i d (1/lambda + J0 slope/c)} M(u) with
// M(u) = sum_j' m[J0+j'] e^{-2pi i j' u},  j' = j - J0 centred on J0 = F/2.  M is
// evaluated as a type-2 non-uniform FFT: on a grid of N = 2F cells,
//   M(u) ~= sum_k phi(N u - k) G_k,   G_k = sum_j' (m / phihat(j'/N)) e^{-2pi i j' k / N},
// with phi the exponential-of-semicircle kernel exp(beta (sqrt(1 - (2z/W)^2) - 1)),
// W = 8 cells, beta = 2.3 W, and phihat its Fourier transform.  Per (voxel, antenna) that
// is eight taps -- weights from degree-8 polynomials in the fractional cell offset
// (es_taps.cuh; mirror taps share one even and one odd part), one 16-byte shared load of
// (G'.re, G.re, G'.im, G.im) and two FFMA2 each -- in place of two F-step Horner chains.
// Accuracy ~1e-7 relative (the FP32 Horner chains' level).
//
// Measurement pass.  dL/dm[a, J0+j'] = sum_v G_a(v) conj(p) = sum_v h_v e^{2pi i j' u_v} with
// h_v = G_a(v) conj(anchor): the transposed (type-1) transform.  Each voxel spreads
// h_v phi(N u_v - k) onto the same 8 cells it would read, the cells are summed over all
// voxels into the antenna's grid S_k, and dL/dm[a, J0+j'] = sum_k S_k e^{2pi i j' k/N} /
// phihat(j'/N) per antenna.  The spread onto S_k is bp_local.cu's (moments per voxel box, node
// values spread without atomics); this file holds the transform out of S_k.
//
// Kernels: nufft_tables_kernel (1/phihat by midpoint quadrature in FP64, twiddles, the voxel
// box), nufft_grid_window_kernel (the forward's per-antenna grids, only the cells that the
// voxel box can reach; bp_local.cu reads them), nufft_grid_kernel (per-antenna grids by a
// direct FP64 transform: F x (N + W - 1) per antenna), bp_bwd_pos_nufft_kernel (the forward's tiling and
// double-buffered antenna staging, rows of N + W - 1 cells so no tap wraps; per-antenna
// sums over a CTA's voxels go to the same per-tile partials as the Horner form),
// nufft_meas_out_kernel (measurement pass).
#include <algorithm>

#include "bp_stage.cuh"
#include "nufft_taps.cuh"

namespace mmn {

namespace {

constexpr double kNuBeta = 2.30 * kNuW;
constexpr int kNuQuad = 256;  // midpoint nodes on [0, W/2]: 1/phihat to ~1e-11

__device__ __forceinline__ double es_kernel(double z) {
    const double t = 2.0 * z / kNuW;
    const double q = 1.0 - t * t;
    return q > 0.0 ? exp(kNuBeta * (sqrt(q) - 1.0)) : 0.0;
}

}  // namespace

// Per-axis bounds of the voxel coordinates, by one block: box = (min x, y, z, max x, y, z).
__device__ void coordinate_box(const float *xs, int nx, const float *ys, int ny, const float *zs,
                               int nz, float *box) {
    __shared__ float s_lo[3][32], s_hi[3][32];
    const float *arr[3] = {xs, ys, zs};
    const int cnt[3] = {nx, ny, nz};
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float lo = __int_as_float(0x7f800000), hi = -lo;
        for (int i = threadIdx.x; i < cnt[k]; i += blockDim.x) {
            const float v = arr[k][i];
            lo = fminf(lo, v);
            hi = fmaxf(hi, v);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        if (lane == 0) {
            s_lo[k][warp] = lo;
            s_hi[k][warp] = hi;
        }
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        const int k = threadIdx.x;
        float lo = s_lo[k][0], hi = s_hi[k][0];
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) {
            lo = fminf(lo, s_lo[k][w]);
            hi = fmaxf(hi, s_hi[k][w]);
        }
        box[k] = lo;
        box[3 + k] = hi;
    }
}

// sc[j] = 1 / phihat((j - J0) / N) for j < F (one warp per j), tw[k] = e^{-2pi i k/N}; the
// last block writes the voxel box.
__global__ void nufft_tables_kernel(int F, int N, int J0, double *__restrict__ sc,
                                    double2 *__restrict__ tw, const float *xs, int nx,
                                    const float *ys, int ny, const float *zs, int nz,
                                    float *__restrict__ box) {
    if (blockIdx.x == gridDim.x - 1) {
        coordinate_box(xs, nx, ys, ny, zs, nz, box);
        return;
    }
    const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t gw = gid >> 5;
    const int lane = threadIdx.x & 31;
    if (gw < F) {
        const double xi = (double)(gw - J0) / N;
        const double h = 0.5 * kNuW / kNuQuad;
        double s = 0.0;
        for (int q = lane; q < kNuQuad; q += 32) {
            const double z = (q + 0.5) * h;
            s += es_kernel(z) * cospi(2.0 * xi * z);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) sc[gw] = 1.0 / (2.0 * h * s);
    }
    if (gid < N) {
        double sn, cs;
        sincospi(2.0 * (double)gid / N, &sn, &cs);
        tw[gid] = make_double2(cs, -sn);
    }
}

// The cells an antenna's tap runs can touch while its range stays inside the voxel box:
// first cell (any integer, to be taken mod N) and count; all N when the window is not shorter
// or not a number.
__device__ __forceinline__ void cell_window(const float *box, const AntRec &ar, double ti,
                                            double uq, int N, int &first, int &count) {
    const float lo[3] = {box[0], box[1], box[2]}, hi[3] = {box[3], box[4], box[5]};
    const float t[3] = {(float)ar.tx[0], (float)ar.tx[1], (float)ar.tx[2]};
    const float r[3] = {(float)ar.rx[0], (float)ar.rx[1], (float)ar.rx[2]};
    float c, half, dmax;
    range_bounds(lo, hi, t, r, c, half, dmax);
    // (the local kernels may widen a box by a third of a cell: one cell of slack either side)
    const double a = ((double)c - half + ti) * uq * N, b = ((double)c + half + ti) * uq * N;
    const double k0 = floor(fmin(a, b)) - kNuW / 2, k1 = floor(fmax(a, b)) + kNuW / 2 + 1;
    first = 0;
    count = N;
    if (k1 - k0 + 1.0 < (double)N && fabs(k0) < 1e9) {
        first = (int)k0;
        count = (int)(k1 - k0) + 1;
    }
}

// Forward rows: rows[a][jj] = (G_k.re, G_k.im) for cell k = (jj - (W/2 - 1)) mod N, jj < row.
// One block per antenna, one lane per cell, a quarter of the samples per warp (their sums added in
// order), over the cells of the antenna's window only: a 0.19 m grid at 4 GHz touches about 30 of
// the 400 cells of 200 samples (592 us for all cells of 4096 antennas).  Cells outside the window
// are left unwritten and are never read.  blockIdx.y: every gridDim.y-th 32 cells of a window.
// Both splits are for few antennas, whose windows a warp or two took long over: 4 antennas x 1000
// samples over a 10 m scene, the whole image 0.88 ms with a warp an antenna, 0.15 with a warp per
// 32 cells, 0.076 so.
constexpr int kGridWarps = 4;
__global__ void __launch_bounds__(kGridWarps * 32)
    nufft_grid_window_kernel(const float2 *__restrict__ meas, int F, int N, int J0, int row,
                             const double *__restrict__ sc, const double2 *__restrict__ tw,
                             const AntRec *__restrict__ ant, const float *__restrict__ box,
                             double ti, double uq, float2 *__restrict__ rows) {
    __shared__ double2 part[kGridWarps][32];
    const int a = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int first, count;
    cell_window(box, ant[a], ti, uq, N, first, count);
    const float2 *m = meas + (size_t)a * F;
    float2 *out = rows + (size_t)a * row;
    const int j0 = (int)((int64_t)F * warp / kGridWarps);
    const int j1 = (int)((int64_t)F * (warp + 1) / kGridWarps);
    for (int c0 = blockIdx.y * 32; c0 < count; c0 += 32 * gridDim.y) {
        const int k = (int)((((int64_t)first + min(c0 + lane, count - 1)) % N + N) % N);
        int idx = (int)((((int64_t)(j0 - J0) * k) % N + N) % N);  // (j - J0) k mod N at j = j0
        double gr = 0.0, gi = 0.0;
#pragma unroll 4
        for (int j = j0; j < j1; ++j) {
            const float2 mv = __ldg(m + j);
            const double s = __ldg(sc + j);
            const double2 t = __ldg(tw + idx);
            const double ar = s * (double)mv.x, ai = s * (double)mv.y;
            gr += fma(ar, t.x, -ai * t.y);
            gi += fma(ar, t.y, ai * t.x);
            idx += k;
            if (idx >= N) idx -= N;
        }
        part[warp][lane] = make_double2(gr, gi);
        __syncthreads();
        if (warp == 0 && c0 + lane < count) {
#pragma unroll
            for (int w = 1; w < kGridWarps; ++w) {
                gr += part[w][lane].x;
                gi += part[w][lane].y;
            }
            for (int jj = (k + kNuW / 2 - 1) % N; jj < row; jj += N)
                out[jj] = make_float2((float)gr, (float)gi);
        }
        __syncthreads();
    }
}

// rows[a][jj] = (G'_k.re, G_k.re, G'_k.im, G_k.im) for cell k = (jj - (W/2 - 1)) mod N,
// jj < N + W - 1: a tap run starting at any cell reads W consecutive entries.
__global__ void nufft_grid_kernel(const float2 *__restrict__ meas, int F, int N, int J0, int row,
                                  double k0, double kd, const double *__restrict__ sc,
                                  const double2 *__restrict__ tw, float4 *__restrict__ rows,
                                  int blocks_per_row) {
    const int a = blockIdx.x / blocks_per_row;
    const int jj = (blockIdx.x - a * blocks_per_row) * blockDim.x + threadIdx.x;
    if (jj >= row) return;
    const int k = ((jj - (kNuW / 2 - 1)) % N + N) % N;
    int idx = (int)((((int64_t)(-J0) * k) % N + N) % N);  // (j - J0) k mod N at j = 0
    const float2 *m = meas + (size_t)a * F;
    double gr = 0.0, gi = 0.0, hr = 0.0, hi = 0.0;
    for (int j = 0; j < F; ++j) {
        const float2 mv = __ldg(m + j);
        const double s = __ldg(sc + j);
        const double2 t = __ldg(tw + idx);
        const double ar = s * (double)mv.x, ai = s * (double)mv.y;
        const double pr = fma(ar, t.x, -ai * t.y), pi = fma(ar, t.y, ai * t.x);
        gr += pr;
        gi += pi;
        const double kap = fma((double)j, kd, k0);
        hr = fma(kap, pr, hr);
        hi = fma(kap, pi, hi);
        idx += k;
        if (idx >= N) idx -= N;
    }
    rows[(size_t)a * row + jj] = make_float4((float)hr, (float)gr, (float)hi, (float)gi);
}

// Position pass, interpolation form.  VOTE: the loss has a vote term (grad_vote set).
template <int T, int NT, bool VOTE>
__global__ void __launch_bounds__(NT) bp_bwd_pos_nufft_kernel(const BwdParams bp) {
    const FwdParams &p = bp.f;
    extern __shared__ __align__(128) unsigned char smem[];
    Stage st;
    st.bars = reinterpret_cast<uint64_t *>(smem);
    st.base = smem + 128;
    st.nas = p.ant_per_stage;
    st.esz = 16;
    st.fp = p.fp;  // grid row length N + W - 1
    st.stage_bytes = (size_t)st.nas * sizeof(AntRec) + (size_t)st.nas * st.fp * st.esz;
    float *wsum = reinterpret_cast<float *>(st.base + 2 * st.stage_bytes);  // [NT/32][nas][3]
    constexpr int NW = NT / 32;
    const int row_len = p.fp;
    const int n = bp.nu_n;
    const double uq = bp.nu_u, k0c = bp.nu_k0c;
    const int tile = blockIdx.x % p.num_tiles;
    const int split = blockIdx.x / p.num_tiles;
    const int a_begin = split * p.ant_per_split;
    const int a_end = min(p.num_ant, a_begin + p.ant_per_split);
    const int n_chunks = a_end > a_begin ? (a_end - a_begin + st.nas - 1) / st.nas : 0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        mbar_init(&st.bars[0], 1);
        mbar_init(&st.bars[1], 1);
        fence_mbar_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (n_chunks > 0) st.issue(p, 0, a_begin, a_end);
        if (n_chunks > 1) st.issue(p, 1, a_begin, a_end);
    }

    const int64_t rbase = (int64_t)tile * (NT * T) + threadIdx.x;
    float vx[T], vy[T], vz[T];
    double vxd[T], vyd[T], vzd[T];
    float2 gi[T], gw[T][3];
#pragma unroll
    for (int k = 0; k < T; ++k) {
        const int64_t rel = rbase + (int64_t)k * NT;
        decode_voxel(p, rel, vx[k], vy[k], vz[k]);
        vxd[k] = vx[k];
        vyd[k] = vy[k];
        vzd[k] = vz[k];
        const bool ok = rel < p.vox_count;
        const int64_t v = p.vox_start + (ok ? rel : 0);
        gi[k] = (ok && bp.grad_image) ? bp.grad_image[v] : make_float2(0.f, 0.f);
#pragma unroll
        for (int q = 0; q < 3; ++q)
            gw[k][q] = (VOTE && ok) ? bp.grad_vote[q * p.nvox + v] : make_float2(0.f, 0.f);
    }
    const bool mono = *p.mono_flag != 0;

    int c_failed = -1;  // chunk whose wait gave up; the drain runs after the loop
    for (int c = 0; c < n_chunks; ++c) {
        const int s = c & 1;
        bool ok = mbar_wait_bounded(&st.bars[s], (uint32_t)((c >> 1) & 1), p.status);
        if (!__syncthreads_and(ok)) {
            c_failed = c;
            break;
        }
        const AntRec *ants = st.ants(s);
        const float4 *mstage = reinterpret_cast<const float4 *>(st.meas(s));
        const int a0 = a_begin + c * st.nas;
        const int na = min(st.nas, a_end - a0);

        for (int a = 0; a < na; ++a) {
            const AntRec &ar = ants[a];
            const float4 *row = mstage + (size_t)a * row_len;
            // FP32 antenna positions for the gradient directions (a direction needs no more)
            const float txf[3] = {(float)ar.tx[0], (float)ar.tx[1], (float)ar.tx[2]};
            const float rxf[3] = {(float)ar.rx[0], (float)ar.rx[1], (float)ar.rx[2]};
            float g3[3] = {0.f, 0.f, 0.f};
#pragma unroll
            for (int k = 0; k < T; ++k) {
                NuPair g;
                nufft_pair(vxd[k], vyd[k], vzd[k], vx[k], vy[k], vz[k], ar, txf, rxf, mono, p.ti,
                           uq, n, g);
                const double d = g.d;
                const float *e3 = g.e3;
                float2 acc_r = make_float2(0.f, 0.f), acc_i = make_float2(0.f, 0.f);
#pragma unroll
                for (int i = 0; i < kNuW; ++i) {
                    const float4 e = row[g.ix + i];
                    acc_r = __ffma2_rn(make_float2(g.w[i], g.w[i]), make_float2(e.x, e.y), acc_r);
                    acc_i = __ffma2_rn(make_float2(g.w[i], g.w[i]), make_float2(e.z, e.w), acc_i);
                }
                // rotate by the anchor e^{-2pi i d (1/lambda + J0 slope/c)}: .x c', .y c
                const float2 an = cis_fp64_phase(-d * k0c);
                const float2 anr = make_float2(an.x, an.x), ani = make_float2(an.y, an.y);
                const float2 cr = __ffma2_rn(anr, acc_r, __fmul2_rn(make_float2(-an.y, -an.y), acc_i));
                const float2 ci = __ffma2_rn(anr, acc_i, __fmul2_rn(ani, acc_r));

                float Gr = gi[k].x, Gi = gi[k].y;
                if (VOTE) {
                    const float uu[3] = {ar.virt[0] - vx[k], ar.virt[1] - vy[k],
                                         ar.virt[2] - vz[k]};
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        Gr = fmaf(gw[k][q].x, uu[q], Gr);
                        Gi = fmaf(gw[k][q].y, uu[q], Gi);
                    }
                }
                const float s1 = Gr * ci.x - Gi * cr.x;  // Im(conj(G) c')
#pragma unroll
                for (int q = 0; q < 3; ++q)
                    g3[q] += VOTE ? fmaf(s1, e3[q], gw[k][q].x * cr.y + gw[k][q].y * ci.y)
                                  : s1 * e3[q];
            }
#pragma unroll
            for (int q = 0; q < 3; ++q) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) g3[q] += __shfl_xor_sync(0xffffffffu, g3[q], o);
            }
            if (lane == 0) {
                wsum[(warp * st.nas + a) * 3 + 0] = g3[0];
                wsum[(warp * st.nas + a) * 3 + 1] = g3[1];
                wsum[(warp * st.nas + a) * 3 + 2] = g3[2];
            }
        }
        __syncthreads();
        for (int idx = threadIdx.x; idx < na * 3; idx += NT) {
            float sum = 0.f;
#pragma unroll
            for (int w = 0; w < NW; ++w) sum += wsum[w * st.nas * 3 + idx];
            bp.pos_partial[((size_t)tile * p.num_ant + a0) * 3 + idx] = sum;
        }
        __syncthreads();
        if (threadIdx.x == 0 && c + 2 < n_chunks) st.issue(p, c + 2, a_begin, a_end);
    }
    if (c_failed >= 0) {
        st.drain_after_timeout((uint32_t)c_failed, c_failed + 1 < n_chunks, p.status);
        return;
    }
}

// Launch shapes (voxels per thread, threads per CTA, cap on one shared-memory stage).
struct NuVariant {
    int t, nt, stage_cap;
    const void *fn_vote, *fn_img;
    const char *name;
};

#define MMN_NU_VARIANT(T, NT, CAP)                                                         \
    {T, NT, CAP, reinterpret_cast<const void *>(&bp_bwd_pos_nufft_kernel<T, NT, true>),     \
     reinterpret_cast<const void *>(&bp_bwd_pos_nufft_kernel<T, NT, false>),               \
     "interp_t" #T "_n" #NT "_s" #CAP}

// Variant 0, the default, is the tile-local form (bp_local.cu; its pointers are filled in by
// bwd_pos_nufft_kernel_ptr).  The others are launch shapes of this file's tap-run kernel: at
// 64^3 voxels, 4096 antennas, 128 samples (position pass alone; with vote term / image loss
// only) 9.08/8.22, 12.1/11.8, 10.6/9.82 and 8.97/8.21 ms in this order (4.55/3.73 the default).  The
// last was variant 0 before the local form; it keeps its name, at the end.
const NuVariant kNuVariants[] = {
    {4, 128, 0, nullptr, nullptr, "interp_local_t4_n128"},
    MMN_NU_VARIANT(2, 256, 24),
    MMN_NU_VARIANT(1, 256, 48),
    MMN_NU_VARIANT(1, 128, 16),
    MMN_NU_VARIANT(2, 128, 24),
};
#undef MMN_NU_VARIANT

// ------------------------------------------------------------- measurement pass

// Per antenna (one block): S_k = sum over box ranges and over the row cells that wrap onto
// cell k, then dL/dm[a, j] = sc[j] sum_k S_k e^{2pi i (j - J0) k / N} in FP64 over the cells
// that are not zero (a box of voxels reaches a few tens of the N cells), in ascending order.
__global__ void nufft_meas_out_kernel(const NuMeasParams q) {
    extern __shared__ __align__(16) unsigned char smem_out[];
    double2 *S = reinterpret_cast<double2 *>(smem_out);
    int *cell = reinterpret_cast<int *>(S + q.n);
    __shared__ int s_count;
    const int a = blockIdx.x;
    const int n = q.n;
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        double sr = 0.0, si = 0.0;
        for (int r = 0; r < q.ranges; ++r) {
            const float2 *row = q.part + ((size_t)r * q.num_ant + a) * q.mrow;
            for (int jj = (k + kNuW / 2 - 1) % n; jj < q.mrow; jj += n) {
                sr += row[jj].x;
                si += row[jj].y;
            }
        }
        S[k] = make_double2(sr, si);
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        int count = 0;
        for (int k0 = 0; k0 < n; k0 += 32) {
            const int k = k0 + threadIdx.x;
            const bool some = k < n && !(S[k].x == 0.0 && S[k].y == 0.0);
            const unsigned b = __ballot_sync(0xffffffffu, some);
            if (some) cell[count + __popc(b & ((1u << threadIdx.x) - 1u))] = k;
            count += __popc(b);
        }
        if (threadIdx.x == 0) s_count = count;
    }
    __syncthreads();
    const int count = s_count;
    for (int j = threadIdx.x; j < q.F; j += blockDim.x) {
        const int step = ((j - q.J0) % n + n) % n;
        double er = 0.0, ei = 0.0;
        int idx = 0, at = 0;  // idx = step * at mod N
        for (int c = 0; c < count; ++c) {
            const int k = cell[c];
            idx = k == at + 1 ? idx + step : (int)((int64_t)step * k % n);
            if (idx >= n) idx -= n;
            at = k;
            const double2 t = q.tw[idx];  // e^{-2pi i idx/N}; the transform needs its conjugate
            const double2 sk = S[k];
            er = fma(sk.x, t.x, fma(sk.y, t.y, er));
            ei = fma(sk.y, t.x, fma(-sk.x, t.y, ei));
        }
        const double sc = q.sc[j];
        q.grad_meas[(size_t)a * q.F + j] = make_float2((float)(er * sc), (float)(ei * sc));
    }
}

cudaError_t launch_nufft_meas_out(const NuMeasParams &q, cudaStream_t stream) {
    const size_t osmem = (size_t)q.n * (sizeof(double2) + sizeof(int));
    if (osmem > 47 * 1024)
        cudaFuncSetAttribute(reinterpret_cast<const void *>(&nufft_meas_out_kernel),
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)osmem);
    nufft_meas_out_kernel<<<q.num_ant, 256, osmem, stream>>>(q);
    return cudaGetLastError();
}

int bwd_pos_nufft_num_variants() { return (int)(sizeof(kNuVariants) / sizeof(kNuVariants[0])); }

const char *bwd_pos_nufft_variant_name(int variant) {
    return variant >= 0 && variant < bwd_pos_nufft_num_variants() ? kNuVariants[variant].name
                                                                   : nullptr;
}

const void *bwd_pos_nufft_kernel_ptr(int variant, bool vote, int *threads, int *voxels_per_thread,
                                     int *stage_cap_bytes) {
    if (variant < 0 || variant >= bwd_pos_nufft_num_variants()) variant = 0;
    const NuVariant &v = kNuVariants[variant];
    *threads = v.nt;
    *voxels_per_thread = v.t;
    *stage_cap_bytes = v.stage_cap * 1024;
    if (!v.fn_vote) return bwd_pos_local_kernel_ptr(vote, threads);
    return vote ? v.fn_vote : v.fn_img;
}

cudaError_t launch_nufft_tables(const FwdParams &p, int F, int N, int J0, double *sc, double2 *tw,
                                float *box, cudaStream_t stream) {
    const int nt = 256;
    const int64_t tthreads = std::max<int64_t>((int64_t)F * 32, N);
    nufft_tables_kernel<<<(unsigned)((tthreads + nt - 1) / nt) + 1, nt, 0, stream>>>(
        F, N, J0, sc, tw, p.x_locs, p.nx, p.y_locs, p.ny, p.z_locs, p.nz, box);
    return cudaGetLastError();
}

cudaError_t launch_nufft_grid(const float *meas, int A, int F, int N, int J0, double k0,
                              double kd, const double *sc, const double2 *tw, float4 *rows,
                              cudaStream_t stream) {
    const int nt = 256;
    const int row = nufft_row(N);
    const int bpr = (row + nt - 1) / nt;
    nufft_grid_kernel<<<(unsigned)((int64_t)A * bpr), nt, 0, stream>>>(
        reinterpret_cast<const float2 *>(meas), F, N, J0, row, k0, kd, sc, tw, rows, bpr);
    return cudaGetLastError();
}

cudaError_t launch_nufft_grid_window(const float *meas, int A, int F, int N, int J0, int row,
                                     const double *sc, const double2 *tw, const AntRec *ant,
                                     const float *box, double ti, double uq, float2 *rows,
                                     cudaStream_t stream) {
    const int parts = std::max(1, std::min((N + 31) / 32, 148 * 8 / A));
    nufft_grid_window_kernel<<<dim3(A, parts), kGridWarps * 32, 0, stream>>>(
        reinterpret_cast<const float2 *>(meas), F, N, J0, row, sc, tw, ant, box, ti, uq, rows);
    return cudaGetLastError();
}

}  // namespace mmn
