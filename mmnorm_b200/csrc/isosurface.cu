// isosurface.cu -- mmWave channels simulated from an isosurface of the RSDF: ray marching
// fused with the channel synthesis.
//
// Reference: _simulate_channels (src/data_processing/isosurface_optimization.py:116-208)
// and the ray-marching extension it calls (src/data_processing/cuda/ray_tracing_kernel.cu:
// GenerateRay :60-120, ValueAt :200-290, Intersect :292-400).  For one antenna and one
// isosurface offset tau per RSDF component, width x height rays leave the antenna over the
// field of view; each marches the grid (rsdf - tau) with steps equal to the trilinear SDF
// value (MIN_STEP where a corner is undefined) until the value drops below one voxel; the
// hit is refined by one more step of the trilinear value at the hit voxel
// (_compute_intersection_pos :66-92), and every hit adds exp(j 2 pi d / lambda_k), d the
// round trip (+0.15 m for the TI radar), to the antenna's channel at every wavelength.
//
// Ray generation and marching repeat the reference kernel's FP32 arithmetic expression for
// expression (including its float-valued flat index), so the hits and rough positions are
// the reference's; the refinement repeats the torch expressions with one rounding per
// operation, as torch evaluates them; the distance is FP64 (the reference subtracts the
// FP32 hit from the FP64 antenna position).  The synthesis evaluates
// exp(j 2 pi d f_k / c) from an exact fixed-point phase per (hit, wavelength) and the
// hardware sincos on the wrapped angle (f_k uniform, f_k = c / lambda_k).
//
// Work item = (offset set t, antenna a); grid = (ray blocks, items).  A block takes every
// blocks-per-item-th tile of 256 rays, gathers the rays that can reach the box into batches,
// marches them through every component, collects the hits in ray order and adds them to its
// partial channel [K]; a second kernel adds the blocks' partials in a fixed order (FP64) --
// deterministic run to run.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "mmn_internal.cuh"

namespace mmn {
namespace {

constexpr float kPiF = 3.14159265358979323846f;
constexpr float kUndef = -50.f;
constexpr float kMinStep = 0.005;   // a double literal narrowed to float, as the reference
constexpr int kMaxSteps = 1000;
constexpr int kIsoThreads = 256;

struct IsoParams {
    const float *grids;        // [C][NX][NY][NZ] RSDF, kUndef where undefined
    const float *taus;         // [T][C] offsets (already clipped to their bounds)
    const double *rx_locs;     // [A][3] antenna positions (FP64, for the distance)
    const float *rx_dirs;      // [A][3]
    int num_comp, num_ant, num_items;
    int width, height;
    float width_fov, height_fov;
    float bb_min_x, bb_min_y, bb_min_z, bb_max_x, bb_max_y, bb_max_z;
    int res_x, res_y, res_z;
    float voxel_size_ref;      // the voxel size the refinement step uses (voxel_size)
    float lower_x, lower_y, lower_z;  // bounding_box_lower (FP32)
    double range_offset;       // 0.15 for the TI radar, else 0
    double f0_over_c, df_over_c;  // f_k / c = f0_over_c + k * df_over_c (1/m)
    int num_wl;
    float2 *partial;           // [items][blocks][K]
    int32_t *block_hits;       // [items][blocks]
    int blocks_per_item;
    int32_t *status;
    float *plane;              // [width + height] view-plane coordinates of columns and rows
    float *basis;              // [A][12] RayBasis of each antenna
    int32_t *defined;          // [6] largest index + 1 and N - smallest index per axis of the
                               // voxels that may be defined; null: not formed
};

__device__ __forceinline__ float deg_to_rad(const float &deg) { return (deg * (kPiF / 180.f)); }

__device__ __forceinline__ float vlen(const float x, const float y, const float z) {
    return sqrtf(powf(x, 2) + powf(y, 2) + powf(z, 2));
}

// the antenna's view frame (w along the antenna direction, u = up x w, v = w x u) and the
// field of view in radians: the same for every ray of an antenna, formed once per block
struct RayBasis {
    float w_x, w_y, w_z, u_x, u_y, u_z, v_x, v_y, v_z, horiz_fov, vert_fov;
};

__device__ RayBasis ray_basis(const IsoParams &p, float rdx, float rdy, float rdz) {
    RayBasis b;
    const float up_x = 1, up_y = 0, up_z = 0;
    b.vert_fov = deg_to_rad(p.height_fov);
    b.horiz_fov = deg_to_rad(p.width_fov);
    b.w_x = (rdx) / vlen(rdx, rdy, rdz);
    b.w_y = (rdy) / vlen(rdx, rdy, rdz);
    b.w_z = (rdz) / vlen(rdx, rdy, rdz);
    const float cuw_x = up_y * b.w_z - up_z * b.w_y;
    const float cuw_y = up_z * b.w_x - up_x * b.w_z;
    const float cuw_z = up_x * b.w_y - up_y * b.w_x;
    b.u_x = (cuw_x) / vlen(cuw_x, cuw_y, cuw_z);
    b.u_y = (cuw_y) / vlen(cuw_x, cuw_y, cuw_z);
    b.u_z = (cuw_z) / vlen(cuw_x, cuw_y, cuw_z);
    b.v_x = b.w_y * b.u_z - b.w_z * b.u_y;
    b.v_y = b.w_z * b.u_x - b.w_x * b.u_z;
    b.v_z = b.w_x * b.u_y - b.w_y * b.u_x;
    return b;
}

// view-plane coordinate of column (or row) i of n: the angle is formed in double (a float plus
// 0.5) and narrowed, as the reference does
__device__ float view_plane(float fov, int i, int n) {
    const float angle = -fov + (fov*2) * (__int2float_rd(i) + 0.5)/ __int2float_rd(n);
    return tan(angle);
}

// ray direction through a point of the view plane
__device__ void ray_direction(const RayBasis &b, float view_plane_x, float view_plane_y,
                              float &dx, float &dy, float &dz) {
    const float s_x = view_plane_x * b.u_x + view_plane_y * b.v_x - b.w_x;
    const float s_y = view_plane_x * b.u_y + view_plane_y * b.v_y - b.w_y;
    const float s_z = view_plane_x * b.u_z + view_plane_y * b.v_z - b.w_z;
    const float len = vlen(s_x, s_y, s_z);
    dx = s_x / len;
    dy = s_y / len;
    dz = s_z / len;
}

__device__ __forceinline__ bool inside_box(const IsoParams &p, float x, float y, float z) {
    return (x >= p.bb_min_x) && (x <= p.bb_max_x) && (y >= p.bb_min_y) && (y <= p.bb_max_y) &&
           (z >= p.bb_min_z) && (z <= p.bb_max_z);
}

// distance along the ray to the bounding box from outside (-1: none)
__device__ float box_distance(const IsoParams &p, float px, float py, float pz, float dx, float dy,
                              float dz) {
    float dist = -1.f;
    dx = dx / vlen(dx, dy, dz);
    dy = dy / vlen(dx, dy, dz);
    dz = dz / vlen(dx, dy, dz);
    const float vs[3] = {px, py, pz};
    const float ds[3] = {dx, dy, dz};
    const float lo[3] = {p.bb_min_x, p.bb_min_y, p.bb_min_z};
    const float hi[3] = {p.bb_max_x, p.bb_max_y, p.bb_max_z};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float v = vs[k], d = ds[k];
        if (dist == -1) {
            if ((v < lo[k]) && (d > 0)) { dist = (lo[k] - v) / d; }
            if ((v > hi[k]) && (d < 0)) { dist = (hi[k] - v) / d; }
        } else {
            if ((v < lo[k]) && (d > 0)) { dist = fmaxf(dist, (lo[k] - v) / d); }
            if ((v > hi[k]) && (d < 0)) { dist = fmaxf(dist, (hi[k] - v) / d); }
        }
    }
    return dist;
}

// the reference's flat index: integer parts recombined in FP32 (exact below 2^24 voxels)
__device__ __forceinline__ int flat_index(float const x, float const y, float const z, int const rx,
                                          int const ry, int const rz) {
    (void)rx;
    return __int2float_rd(z) + __int2float_rd(y) * rz + __int2float_rd(x) * rz * ry;
}

__device__ __forceinline__ float grid_at(const float *g, float tau, int idx, int n, bool &ok) {
    if (idx < 0 || idx >= n) {
        ok = false;
        return 0.f;
    }
    return __fsub_rn(g[idx], tau);
}

// Constants of the march, the same at every step.
struct MarchGrid {
    float voxel_size, inv;             // and its reciprocal
    float edge_x, edge_y, edge_z;      // (max - min) / voxel_size
    bool exact;                        // flat indices are exact in FP32
};
__device__ __forceinline__ MarchGrid march_grid(const IsoParams &p) {
    MarchGrid m;
    m.voxel_size = (p.bb_max_y - p.bb_min_y) / (p.res_y - 1);
    m.inv = 1.f / m.voxel_size;
    m.edge_x = (p.bb_max_x - p.bb_min_x) / m.voxel_size;
    m.edge_y = (p.bb_max_y - p.bb_min_y) / m.voxel_size;
    m.edge_z = (p.bb_max_z - p.bb_min_z) / m.voxel_size;
    m.exact = ((int64_t)p.res_x + 2) * (p.res_y + 2) * (p.res_z + 2) < (1 << 24);
    return m;
}

// floorf(a / voxel_size) for a >= 0: a * inv is within 3e-7 of the rounded quotient, relative, so
// its floor -- one addition rounded down -- is the quotient's unless it lies within 1.2e-6 (h + 1)
// of an integer (or the quotient is beyond 2^22, or NaN); then the division decides.
__device__ __forceinline__ float floor_cell(float a, const MarchGrid &m) {
    const float h = a * m.inv;
    const float r = __fadd_rd(h, 8388608.f) - 8388608.f;
    if (fabsf((h - r) - 0.5f) < fmaf(h, -1.2e-6f, 0.5f - 1.2e-6f) && h < 4194304.f) return r;
    return floorf(a / m.voxel_size);
}

// signed distance at a point (the reference's ValueAt); ok=false if an index left the grid
__device__ __forceinline__ float value_at(const IsoParams &p, const MarchGrid &mg, const float *g,
                                          float tau, float px, float py, float pz, float dx,
                                          float dy, float dz, bool first_time, bool &ok) {
    if (!inside_box(p, px, py, pz)) {
        if (first_time)
            return box_distance(p, px, py, pz, dx, dy, dz) + 0.00001f;
        return -1;
    }
    const int n = p.res_x * p.res_y * p.res_z;
    const float voxel_size = mg.voxel_size;
    float mx = floor_cell(px - p.bb_min_x, mg);
    float my = floor_cell(py - p.bb_min_y, mg);
    float mz = floor_cell(pz - p.bb_min_z, mg);
    if (mx == mg.edge_x) mx = mg.edge_x - 1;
    if (my == mg.edge_y) my = mg.edge_y - 1;
    if (mz == mg.edge_z) mz = mg.edge_z - 1;
    const int rx = p.res_x, ry = p.res_y, rz = p.res_z;
    float g000, g010, g001, g011, g100, g110, g101, g111;
    if (mg.exact) {
        // every index the reference forms in FP32 is exact: one base and integer strides
        const int base = ((int)mx * ry + (int)my) * rz + (int)mz;
        const int sx = ry * rz;
        if (base < 0 || base + sx + rz + 1 >= n) {
            ok = false;
            return 0.f;
        }
        const float *q = g + base;
        g000 = __ldg(q);
        g001 = __ldg(q + 1);
        g010 = __ldg(q + rz);
        g011 = __ldg(q + rz + 1);
        g100 = __ldg(q + sx);
        g101 = __ldg(q + sx + 1);
        g110 = __ldg(q + sx + rz);
        g111 = __ldg(q + sx + rz + 1);
        // the subtraction of tau keeps the order, so the least corner decides for all (a NaN
        // corner compares false in the reference too, and fminf passes it over)
        const float least = fminf(fminf(fminf(g000, g001), fminf(g010, g011)),
                                  fminf(fminf(g100, g101), fminf(g110, g111)));
        if (__fsub_rn(least, tau) < kUndef + 10) return kMinStep;
        g000 = __fsub_rn(g000, tau);
        g001 = __fsub_rn(g001, tau);
        g010 = __fsub_rn(g010, tau);
        g011 = __fsub_rn(g011, tau);
        g100 = __fsub_rn(g100, tau);
        g101 = __fsub_rn(g101, tau);
        g110 = __fsub_rn(g110, tau);
        g111 = __fsub_rn(g111, tau);
    } else {
        g000 = grid_at(g, tau, flat_index(mx, my, mz, rx, ry, rz), n, ok);
        g010 = grid_at(g, tau, flat_index(mx, my + 1, mz, rx, ry, rz), n, ok);
        g001 = grid_at(g, tau, flat_index(mx, my, mz + 1, rx, ry, rz), n, ok);
        g011 = grid_at(g, tau, flat_index(mx, my + 1, mz + 1, rx, ry, rz), n, ok);
        g100 = grid_at(g, tau, flat_index(mx + 1, my, mz, rx, ry, rz), n, ok);
        g110 = grid_at(g, tau, flat_index(mx + 1, my + 1, mz, rx, ry, rz), n, ok);
        g101 = grid_at(g, tau, flat_index(mx + 1, my, mz + 1, rx, ry, rz), n, ok);
        g111 = grid_at(g, tau, flat_index(mx + 1, my + 1, mz + 1, rx, ry, rz), n, ok);
        if (g000 < kUndef + 10 || g010 < kUndef + 10 || g001 < kUndef + 10 || g011 < kUndef + 10 ||
            g100 < kUndef + 10 || g110 < kUndef + 10 || g101 < kUndef + 10 || g111 < kUndef + 10)
            return kMinStep;
    }
    const float tx = (px - (p.bb_min_x + mx * voxel_size)) / voxel_size;
    const float ex_y0z0 = (1.f - tx) * g000 + tx * g100;
    const float ex_y1z0 = (1.f - tx) * g010 + tx * g110;
    const float ex_y0z1 = (1.f - tx) * g001 + tx * g101;
    const float ex_y1z1 = (1.f - tx) * g011 + tx * g111;
    const float ty = (py - (p.bb_min_y + my * voxel_size)) / voxel_size;
    const float fz0 = (1.f - ty) * ex_y0z0 + ty * ex_y1z0;
    const float fz1 = (1.f - ty) * ex_y0z1 + ty * ex_y1z1;
    const float tz = (pz - (p.bb_min_z + mz * voxel_size)) / voxel_size;
    return (1.f - tz) * fz0 + tz * fz1;
}

// marches one ray; on a hit returns true with the rough point and its voxel index
__device__ bool march(const IsoParams &p, const float *g, float tau, float ox, float oy, float oz,
                      float dx, float dy, float dz, float &hx, float &hy, float &hz, float &vx,
                      float &vy, float &vz) {
    const MarchGrid mg = march_grid(p);
    const float voxel_size = mg.voxel_size;
    bool first_time = true;
    float depth = 0;
    for (int steps = 0; steps < kMaxSteps; steps++) {
        const float rx = ox + depth * dx;
        const float ry = oy + depth * dy;
        const float rz = oz + depth * dz;
        bool ok = true;
        const float distance = value_at(p, mg, g, tau, rx, ry, rz, dx, dy, dz, first_time, ok);
        if (!ok) return false;
        first_time = false;
        if (distance == -1) return false;
        if (distance < voxel_size && distance) {
            vx = floorf((rx - p.bb_min_x) / voxel_size);
            vy = floorf((ry - p.bb_min_y) / voxel_size);
            vz = floorf((rz - p.bb_min_z) / voxel_size);
            if (vx == p.res_x - 1) vx = vx - 1;
            if (vy == p.res_y - 1) vy = vy - 1;
            if (vz == p.res_z - 1) vz = vz - 1;
            hx = rx;
            hy = ry;
            hz = rz;
            return true;
        }
        depth += distance;
    }
    return false;
}

// _compute_intersection_pos for one hit, one rounding per torch operation; ok=false when the
// hit's voxel is not inside the grid (the reference would index outside its tensor)
__device__ bool refine(const IsoParams &p, const float *g, float tau, float hx, float hy, float hz,
                       float vx, float vy, float vz, float dx, float dy, float dz, float &ix,
                       float &iy, float &iz) {
    const int x = (int)(vx == -1.f ? 0.f : vx), y = (int)(vy == -1.f ? 0.f : vy),
              z = (int)(vz == -1.f ? 0.f : vz);
    if (x < 0 || y < 0 || z < 0 || x + 1 >= p.res_x || y + 1 >= p.res_y || z + 1 >= p.res_z)
        return false;
    auto at = [&](int a, int b, int c) {
        return __fsub_rn(g[((int64_t)a * p.res_y + b) * p.res_z + c], tau);
    };
    const float vs = p.voxel_size_ref;
    const float mnx = __fadd_rn(p.lower_x, __fmul_rn(vx, vs));
    const float mny = __fadd_rn(p.lower_y, __fmul_rn(vy, vs));
    const float mnz = __fadd_rn(p.lower_z, __fmul_rn(vz, vs));
    auto lerp = [](float t, float a, float b) {
        return __fadd_rn(__fmul_rn(__fsub_rn(1.f, t), a), __fmul_rn(t, b));
    };
    const float tx = __fdiv_rn(__fsub_rn(hx, mnx), vs);
    const float ex_y0z0 = lerp(tx, at(x, y, z), at(x + 1, y, z));
    const float ex_y1z0 = lerp(tx, at(x, y + 1, z), at(x + 1, y + 1, z));
    const float ex_y0z1 = lerp(tx, at(x, y, z + 1), at(x + 1, y, z + 1));
    const float ex_y1z1 = lerp(tx, at(x, y + 1, z + 1), at(x + 1, y + 1, z + 1));
    const float ty = __fdiv_rn(__fsub_rn(hy, mny), vs);
    const float fz0 = lerp(ty, ex_y0z0, ex_y1z0);
    const float fz1 = lerp(ty, ex_y0z1, ex_y1z1);
    const float tz = __fdiv_rn(__fsub_rn(hz, mnz), vs);
    const float sdf = lerp(tz, fz0, fz1);
    ix = __fadd_rn(hx, __fmul_rn(dx, sdf));
    iy = __fadd_rn(hy, __fmul_rn(dy, sdf));
    iz = __fadd_rn(hz, __fmul_rn(dz, sdf));
    return true;
}

// Bounds of the voxels that may be defined, over every component: anything above kUndef + 5 (and
// NaN).  Only a cell whose corners are all defined can be hit, so rays need not march where none
// is; a block takes whole rows along z.
constexpr float kMaybe = kUndef + 5.f;
__global__ void __launch_bounds__(256) iso_defined_kernel(const IsoParams p) {
    const int64_t rows = (int64_t)p.num_comp * p.res_x * p.res_y;
    const int lane = threadIdx.x & 31;
    int hi[3] = {0, 0, 0}, lo[3] = {0, 0, 0};
    for (int64_t r = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); r < rows;
         r += (int64_t)gridDim.x * 8) {
        const float *g = p.grids + r * p.res_z;
        int first = p.res_z, last = -1;
        for (int z = lane; z < p.res_z; z += 32)
            if (!(__ldg(g + z) <= kMaybe)) {
                first = min(first, z);
                last = z;
            }
        if (last >= 0) {
            const int y = (int)(r % p.res_y), x = (int)(r / p.res_y % p.res_x);
            hi[0] = max(hi[0], x + 1);
            hi[1] = max(hi[1], y + 1);
            hi[2] = max(hi[2], last + 1);
            lo[0] = max(lo[0], p.res_x - x);
            lo[1] = max(lo[1], p.res_y - y);
            lo[2] = max(lo[2], p.res_z - first);
        }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        hi[k] = __reduce_max_sync(0xffffffffu, hi[k]);
        lo[k] = __reduce_max_sync(0xffffffffu, lo[k]);
        if (lane == 0 && hi[k] > 0) {
            atomicMax(p.defined + k, hi[k]);
            atomicMax(p.defined + 3 + k, lo[k]);
        }
    }
}

// Whether the line through the eye and a point of the view plane misses the box grown
// by `margin`.  A ray can only hit where its first step from the eye -- to the box's entry, or,
// for a ray that no face of the box receives, the step of -1 + 1e-5 that the reference's sentinel
// turns into -- lands inside the box, and both points lie on that line.  The slab test's FP32
// rounding (about 1e-6 of the distance) is far inside the margin; NaN rejects nothing.  (A first
// step shorter than a voxel, the sentinel's among them, is a hit at the eye itself: it counts only
// if the eye's cell is in the grid, so an eye within two voxels of the box, or of the grid's cells
// where these reach past it, keeps every ray.)
__device__ __forceinline__ bool line_misses(const float (&lo)[3], const float (&hi)[3],
                                            const RayBasis &b, float margin, float ex, float ey,
                                            float ez, float vx, float vy) {
    const float s[3] = {vx * b.u_x + vy * b.v_x - b.w_x, vx * b.u_y + vy * b.v_y - b.w_y,
                        vx * b.u_z + vy * b.v_z - b.w_z};
    const float o[3] = {ex, ey, ez};
    float t0 = -__int_as_float(0x7f800000), t1 = -t0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float inv = __fdividef(1.f, copysignf(fmaxf(fabsf(s[k]), 1e-12f), s[k]));
        const float a = (lo[k] - margin - o[k]) * inv, c = (hi[k] + margin - o[k]) * inv;
        t0 = fmaxf(t0, fminf(a, c));
        t1 = fminf(t1, fmaxf(a, c));
    }
    return t0 > t1;
}

// The tables that every block of an antenna shares: view-plane coordinates and view frames (the
// frame alone is 27 powf calls, which each thread of each block formed for itself before).
__global__ void iso_prep_kernel(const IsoParams p) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < p.width) {
        p.plane[i] = view_plane(deg_to_rad(p.width_fov), i, p.width);
    } else if (i < p.width + p.height) {
        p.plane[i] = view_plane(deg_to_rad(p.height_fov), i - p.width, p.height);
    } else if (i - p.width - p.height < p.num_ant) {
        const int a = i - p.width - p.height;
        const RayBasis b = ray_basis(p, p.rx_dirs[3 * a], p.rx_dirs[3 * a + 1], p.rx_dirs[3 * a + 2]);
        float *o = p.basis + 12 * a;
        o[0] = b.w_x;
        o[1] = b.w_y;
        o[2] = b.w_z;
        o[3] = b.u_x;
        o[4] = b.u_y;
        o[5] = b.u_z;
        o[6] = b.v_x;
        o[7] = b.v_y;
        o[8] = b.v_z;
    }
}

// Rays whose line misses the box (99 % of them at +-80 degrees over a 0.2 m object at 0.45 m) are
// dropped before the exact direction and march, whose 12 powf calls, divisions and two steps they
// spent on finding that out; the rest are gathered into batches of 256, so that the warps that
// march are full.  30 items of 1024 x 1024 rays: 1520 us, 860 without the misses, 716 with the
// batches, 490 with integer cell indices and one comparison for a cell's eight corners, 440 with
// 5 CTAs on an SM, 237 with the defined voxels' box in place of the grid's.
__global__ void __launch_bounds__(kIsoThreads, 5) iso_channel_kernel(const IsoParams p) {
    __shared__ unsigned long long s_ph0[kIsoThreads], s_stp[kIsoThreads];
    __shared__ int s_warp[kIsoThreads / 32 + 1];
    __shared__ int s_ray[2 * kIsoThreads];  // a batch and what one more tile can add
    const int item = blockIdx.y;
    const int t = item / p.num_ant, a = item % p.num_ant;
    const int npix = p.width * p.height;
    const int ntiles = (npix + kIsoThreads - 1) / kIsoThreads;
    const float eye_x = (float)p.rx_locs[3 * a], eye_y = (float)p.rx_locs[3 * a + 1],
                eye_z = (float)p.rx_locs[3 * a + 2];
    RayBasis basis;
    {
        const float *o = p.basis + 12 * a;
        basis.w_x = o[0];
        basis.w_y = o[1];
        basis.w_z = o[2];
        basis.u_x = o[3];
        basis.u_y = o[4];
        basis.u_z = o[5];
        basis.v_x = o[6];
        basis.v_y = o[7];
        basis.v_z = o[8];
    }
    // 1e-4 of the farthest box point's distance, and more than the first step's 1e-5
    const float margin =
        2e-5f + 1e-4f * (fmaxf(fabsf(p.bb_min_x - eye_x), fabsf(p.bb_max_x - eye_x)) +
                         fmaxf(fabsf(p.bb_min_y - eye_y), fabsf(p.bb_max_y - eye_y)) +
                         fmaxf(fabsf(p.bb_min_z - eye_z), fabsf(p.bb_max_z - eye_z)));
    const float vs = (p.bb_max_y - p.bb_min_y) / (p.res_y - 1);
    const float skin = 2.f * fmaxf(p.voxel_size_ref, vs);
    // a cell is vs wide on every axis, whatever the box's own spacing there
    const bool beside =
        !(eye_x < p.bb_min_x - skin || eye_x > fmaxf(p.bb_max_x, p.bb_min_x + p.res_x * vs) + skin ||
          eye_y < p.bb_min_y - skin || eye_y > fmaxf(p.bb_max_y, p.bb_min_y + p.res_y * vs) + skin ||
          eye_z < p.bb_min_z - skin || eye_z > fmaxf(p.bb_max_z, p.bb_min_z + p.res_z * vs) + skin);
    // the box that rays have to reach: the whole grid's, or, where it is known and every undefined
    // cell is one to the march too (its step longer than a voxel, tau within the bounds' slack),
    // the defined voxels'.  Past its last layer of voxels a box has cells whose corners are the
    // next row's voxels: no narrowing then (a hundredth of a cell is rounding: added below).
    float box_lo[3] = {p.bb_min_x, p.bb_min_y, p.bb_min_z};
    float box_hi[3] = {p.bb_max_x, p.bb_max_y, p.bb_max_z};
    {
        bool narrow = p.defined != nullptr && vs <= kMinStep &&
                      p.bb_max_x - p.bb_min_x <= (p.res_x - 0.99f) * vs &&
                      p.bb_max_z - p.bb_min_z <= (p.res_z - 0.99f) * vs;
        for (int c = 0; c < p.num_comp; ++c)
            narrow = narrow && p.taus[(int64_t)t * p.num_comp + c] > -4.9f;
        if (narrow) {
            const int res[3] = {p.res_x, p.res_y, p.res_z};
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const float low = box_lo[k];
                box_lo[k] = low + (res[k] - p.defined[3 + k]) * vs;
                box_hi[k] = low + (p.defined[k] - 0.99f) * vs;
            }
        }
    }
    const int64_t ncell = (int64_t)p.res_x * p.res_y * p.res_z;
    const int64_t bslot = (int64_t)item * p.blocks_per_item + blockIdx.x;
    float2 *dst = p.partial + bslot * p.num_wl;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int total = 0;  // block-uniform: hits added to dst so far
    int count = 0;  // block-uniform: rays waiting in s_ray
    int tile = blockIdx.x;
    for (;;) {
        // this block's tiles of 256 rays, in order, until a full batch of rays can reach the box
        while (count < kIsoThreads && tile < ntiles) {
            const int pixel = tile * kIsoThreads + threadIdx.x;
            const int py = min(pixel, npix - 1) / p.width;
            const float plane_x = __ldg(p.plane + (min(pixel, npix - 1) - py * p.width));
            const float plane_y = __ldg(p.plane + p.width + py);
            const bool reach = pixel < npix &&
                               (beside || !line_misses(box_lo, box_hi, basis, margin, eye_x, eye_y,
                                                       eye_z, plane_x, plane_y));
            tile += p.blocks_per_item;
            if (!__syncthreads_or(reach)) continue;
            const unsigned ball = __ballot_sync(0xffffffffu, reach);
            if (lane == 0) s_warp[warp] = __popc(ball);
            __syncthreads();
            int at = count + __popc(ball & ((1u << lane) - 1u)), sum = 0;
#pragma unroll
            for (int w = 0; w < kIsoThreads / 32; ++w) {
                const int cnt = s_warp[w];
                at += w < warp ? cnt : 0;
                sum += cnt;
            }
            if (reach) s_ray[at] = pixel;
            count += sum;
            __syncthreads();  // the counts are rewritten by the next tile
        }
        if (count == 0) break;
        const bool mine = threadIdx.x < count;
        float dx = 0.f, dy = 0.f, dz = 0.f;
        if (mine) {
            const int pixel = s_ray[threadIdx.x], py = pixel / p.width;
            ray_direction(basis, __ldg(p.plane + (pixel - py * p.width)),
                          __ldg(p.plane + p.width + py), dx, dy, dz);
        }
        // the rest of the list moves to its front (barriers of the loop below order the writes)
        const int left = max(count - kIsoThreads, 0);
        const int later = threadIdx.x < left ? s_ray[kIsoThreads + threadIdx.x] : 0;
        __syncthreads();
        if (threadIdx.x < left) s_ray[threadIdx.x] = later;
        count = left;
        // every component's isosurface in turn (the reference sums the components' channels)
        for (int c = 0; c < p.num_comp; ++c) {
            const float *g = p.grids + (int64_t)c * ncell;
            const float tau = p.taus[(int64_t)t * p.num_comp + c];
            bool hit = false;
            double d = 0.0;
            if (mine) {
                float hx, hy, hz, vx, vy, vz, ix, iy, iz;
                if (march(p, g, tau, eye_x, eye_y, eye_z, dx, dy, dz, hx, hy, hz, vx, vy, vz) &&
                    refine(p, g, tau, hx, hy, hz, vx, vy, vz, dx, dy, dz, ix, iy, iz)) {
                    const double ex = p.rx_locs[3 * a] - (double)ix;
                    const double ey = p.rx_locs[3 * a + 1] - (double)iy;
                    const double ez = p.rx_locs[3 * a + 2] - (double)iz;
                    d = sqrt(ex * ex + ey * ey + ez * ez) * 2.0 + p.range_offset;
                    hit = true;
                }
            }
            // the hits of this batch and component, compacted in ray order
            const unsigned ball = __ballot_sync(0xffffffffu, hit);
            if (lane == 0) s_warp[warp] = __popc(ball);
            __syncthreads();
            if (threadIdx.x == 0) {
                int run = 0;
                for (int w = 0; w < kIsoThreads / 32; ++w) {
                    const int cnt = s_warp[w];
                    s_warp[w] = run;
                    run += cnt;
                }
                s_warp[kIsoThreads / 32] = run;
            }
            __syncthreads();
            if (hit) {
                const int slot = s_warp[warp] + __popc(ball & ((1u << lane) - 1u));
                s_ph0[slot] = turns_to_fixed(d * p.f0_over_c);
                s_stp[slot] = turns_to_fixed(d * p.df_over_c);
            }
            __syncthreads();
            const int nh = s_warp[kIsoThreads / 32];
            if (nh > 0) {
                for (int k = threadIdx.x; k < p.num_wl; k += kIsoThreads) {
                    float sr = 0.f, si = 0.f;
                    for (int h = 0; h < nh; ++h) {
                        float cs, sn;
                        fixed_cis(s_ph0[h] + (unsigned long long)k * s_stp[h], cs, sn);
                        sr += cs;
                        si += sn;
                    }
                    if (total > 0) {
                        const float2 o = dst[k];
                        sr += o.x;
                        si += o.y;
                    }
                    dst[k] = make_float2(sr, si);
                }
            }
            total += nh;
            __syncthreads();  // the shared hit lists are refilled by the next pass
        }
    }
    if (threadIdx.x == 0) p.block_hits[bslot] = total;
}

// channel[item][k] = sum over the item's blocks of their partials in FP64: 32 wavelengths per
// block, kIsoReduceWarps warps taking every kIsoReduceWarps-th ray block that hit anything, their
// sums added in warp order (one thread per wavelength walked the 1184 ray blocks alone: 95 us for
// 30 items of 512 wavelengths).
constexpr int kIsoReduceWarps = 16;
__global__ void __launch_bounds__(kIsoReduceWarps * 32)
    iso_reduce_kernel(const IsoParams p, float2 *__restrict__ channel) {
    __shared__ double2 part[kIsoReduceWarps][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int item = blockIdx.y, k = blockIdx.x * 32 + lane;
    double sr = 0.0, si = 0.0;
    if (k < p.num_wl) {
#pragma unroll 4
        for (int b = warp; b < p.blocks_per_item; b += kIsoReduceWarps) {
            const int64_t bslot = (int64_t)item * p.blocks_per_item + b;
            if (p.block_hits[bslot] == 0) continue;
            const float2 v = p.partial[bslot * p.num_wl + k];
            sr += v.x;
            si += v.y;
        }
    }
    part[warp][lane] = make_double2(sr, si);
    __syncthreads();
    if (warp != 0 || k >= p.num_wl) return;
    for (int w = 1; w < kIsoReduceWarps; ++w) {
        sr += part[w][lane].x;
        si += part[w][lane].y;
    }
    channel[(int64_t)item * p.num_wl + k] = make_float2((float)sr, (float)si);
}

// rough hits of one antenna's rays (for tests against the reference extension): per pixel
// the rough point (-1 if none), the voxel index (-1 if none) and the ray direction
__global__ void iso_march_debug_kernel(const IsoParams p, int comp, float tau, int ant,
                                       float *rough, float *voxel, float *dir) {
    const int pixel = blockIdx.x * blockDim.x + threadIdx.x;
    if (pixel >= p.width * p.height) return;
    float dx, dy, dz;
    const RayBasis basis =
        ray_basis(p, p.rx_dirs[3 * ant], p.rx_dirs[3 * ant + 1], p.rx_dirs[3 * ant + 2]);
    ray_direction(basis, view_plane(basis.horiz_fov, pixel % p.width, p.width),
                  view_plane(basis.vert_fov, pixel / p.width, p.height), dx, dy, dz);
    const int64_t ncell = (int64_t)p.res_x * p.res_y * p.res_z;
    float hx = -1, hy = -1, hz = -1, vx = -1, vy = -1, vz = -1;
    if (!march(p, p.grids + comp * ncell, tau, (float)p.rx_locs[3 * ant],
               (float)p.rx_locs[3 * ant + 1], (float)p.rx_locs[3 * ant + 2], dx, dy, dz, hx, hy,
               hz, vx, vy, vz)) {
        hx = hy = hz = vx = vy = vz = -1;
    }
    rough[3 * pixel] = hx;
    rough[3 * pixel + 1] = hy;
    rough[3 * pixel + 2] = hz;
    voxel[3 * pixel] = vx;
    voxel[3 * pixel + 1] = vy;
    voxel[3 * pixel + 2] = vz;
    dir[3 * pixel] = dx;
    dir[3 * pixel + 1] = dy;
    dir[3 * pixel + 2] = dz;
}

}  // namespace
}  // namespace mmn

// ----------------------------------------------------------------------------- C ABI
// (the ABI types come in through mmn_internal.cuh)

namespace {
constexpr size_t kIsoStatus = 256;
inline size_t iso_up(size_t x) { return (x + 255) & ~(size_t)255; }

int iso_check(const mmn_iso_scene *s) {
    if (!s) return MMN_ERR_NULL_POINTER;
    if (!s->grids) return MMN_ERR_NULL_POINTER;
    if (s->num_comp < 1 || s->res_x < 2 || s->res_y < 2 || s->res_z < 2 || s->width < 1 ||
        s->height < 1 || s->num_wl < 1)
        return MMN_ERR_INVALID_ARGUMENT;
    if ((int64_t)s->res_x * s->res_y * s->res_z >= ((int64_t)1 << 31)) return MMN_ERR_TOO_LARGE;
    if ((int64_t)s->width * s->height >= ((int64_t)1 << 31)) return MMN_ERR_TOO_LARGE;
    return MMN_OK;
}

// Ray-tile blocks per work item: some 12 per SM over all items, at most 8 per SM for one (each
// loops over its share of the tiles), and an odd number, so that the stride from tile to tile
// does not keep a block in one column of the view (4 tiles to a row of 1024 rays: half the blocks
// never saw the object).
int64_t iso_blocks(const mmn_iso_scene *s, int64_t items) {
    const int64_t npix = (int64_t)s->width * s->height;
    const int64_t tiles = (npix + mmn::kIsoThreads - 1) / mmn::kIsoThreads;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int64_t want = std::max<int64_t>(16, (int64_t)sms * 12 / std::max<int64_t>(items, 1));
    return std::min<int64_t>(tiles, std::min<int64_t>(want, (int64_t)sms * 8) | 1);
}

// Partial slots (items x blocks) that a workspace for `items` holds: enough for any smaller count
// too, whose blocks per item are more.
int64_t iso_slots(const mmn_iso_scene *s, int64_t items) {
    int64_t slots = items * iso_blocks(s, items);
    for (int64_t i = 1; i <= items && i <= 512; ++i) {
        const int64_t b = iso_blocks(s, i);
        slots = std::max(slots, i * b);
        if (b <= 17) break;  // the least: constant from here on
    }
    return slots;
}

mmn::IsoParams iso_params(const mmn_iso_scene *s) {
    mmn::IsoParams p;
    std::memset(&p, 0, sizeof(p));
    p.grids = s->grids;
    p.num_comp = s->num_comp;
    p.width = s->width;
    p.height = s->height;
    p.width_fov = s->width_fov;
    p.height_fov = s->height_fov;
    p.bb_min_x = s->bbox[0];
    p.bb_min_y = s->bbox[1];
    p.bb_min_z = s->bbox[2];
    p.bb_max_x = s->bbox[3];
    p.bb_max_y = s->bbox[4];
    p.bb_max_z = s->bbox[5];
    p.res_x = s->res_x;
    p.res_y = s->res_y;
    p.res_z = s->res_z;
    p.voxel_size_ref = s->voxel_size;
    p.lower_x = s->lower[0];
    p.lower_y = s->lower[1];
    p.lower_z = s->lower[2];
    p.range_offset = s->range_offset;
    p.f0_over_c = s->f0_over_c;
    p.df_over_c = s->df_over_c;
    p.num_wl = s->num_wl;
    return p;
}
}  // namespace

extern "C" size_t mmn_iso_channels_workspace_bytes(const mmn_iso_scene *s, int32_t num_sets,
                                                   int32_t num_antennas) {
    if (iso_check(s) != MMN_OK || num_sets < 1 || num_antennas < 1) return 0;
    const int64_t items = (int64_t)num_sets * num_antennas;
    const int64_t slots = iso_slots(s, items);
    return kIsoStatus + iso_up((size_t)slots * sizeof(int32_t)) +
           iso_up((size_t)slots * s->num_wl * sizeof(float2)) +
           iso_up(((size_t)s->width + s->height + 12 * (size_t)num_antennas) * sizeof(float));
}

extern "C" int mmn_iso_channels(const mmn_iso_scene *s, const float *taus, int32_t num_sets,
                                const double *rx_locs, const float *rx_dirs,
                                int32_t num_antennas, float *channels, void *workspace,
                                size_t workspace_bytes, cudaStream_t stream) {
    int rc = iso_check(s);
    if (rc != MMN_OK) return rc;
    if (!taus || !rx_locs || !rx_dirs || !channels) return MMN_ERR_NULL_POINTER;
    if (num_sets < 1 || num_antennas < 1) return MMN_ERR_INVALID_ARGUMENT;
    const int64_t items = (int64_t)num_sets * num_antennas;
    if (items > 65535) return MMN_ERR_TOO_LARGE;  // grid.y
    const size_t need = mmn_iso_channels_workspace_bytes(s, num_sets, num_antennas);
    if (!workspace || workspace_bytes < need || (reinterpret_cast<uintptr_t>(workspace) & 255))
        return MMN_ERR_WORKSPACE;
    const int blocks = (int)iso_blocks(s, items);
    unsigned char *w = static_cast<unsigned char *>(workspace);
    mmn::IsoParams p = iso_params(s);
    p.taus = taus;
    p.rx_locs = rx_locs;
    p.rx_dirs = rx_dirs;
    p.num_ant = num_antennas;
    p.num_items = (int)items;
    p.blocks_per_item = blocks;
    p.status = reinterpret_cast<int32_t *>(w);
    p.block_hits = reinterpret_cast<int32_t *>(w + kIsoStatus);
    p.partial = reinterpret_cast<float2 *>(w + kIsoStatus +
                                           iso_up((size_t)items * blocks * sizeof(int32_t)));
    p.plane = reinterpret_cast<float *>(w + kIsoStatus +
                                        iso_up((size_t)items * blocks * sizeof(int32_t)) +
                                        iso_up((size_t)items * blocks * s->num_wl *
                                               sizeof(float2)));
    p.basis = p.plane + s->width + s->height;
    if (cudaMemsetAsync(w, 0, kIsoStatus, stream) != cudaSuccess) return MMN_ERR_CUDA;
    // the scan for defined voxels reads the grids once: worth it beside as many rays as voxels
    const int64_t voxels = (int64_t)s->num_comp * s->res_x * s->res_y * s->res_z;
    // (only where FP32 flat indices are exact: a rounded one reads another voxel)
    const bool exact = ((int64_t)s->res_x + 2) * (s->res_y + 2) * (s->res_z + 2) < (1 << 24);
    if (exact && items * s->width * s->height >= voxels) {
        p.defined = reinterpret_cast<int32_t *>(w + 64);
        mmn::iso_defined_kernel<<<148 * 8, 256, 0, stream>>>(p);
    }
    const int64_t prep = (int64_t)s->width + s->height + num_antennas;
    mmn::iso_prep_kernel<<<(unsigned)((prep + 127) / 128), 128, 0, stream>>>(p);
    mmn::iso_channel_kernel<<<dim3(blocks, (unsigned)items), mmn::kIsoThreads, 0, stream>>>(p);
    mmn::iso_reduce_kernel<<<dim3((unsigned)((s->num_wl + 31) / 32), (unsigned)items),
                             mmn::kIsoReduceWarps * 32, 0, stream>>>(
        p, reinterpret_cast<float2 *>(channels));
    return cudaGetLastError() == cudaSuccess ? MMN_OK : MMN_ERR_CUDA;
}

extern "C" int mmn_iso_march(const mmn_iso_scene *s, int32_t comp, float tau,
                             const double *rx_loc, const float *rx_dir, float *rough,
                             float *voxel, float *direction, cudaStream_t stream) {
    int rc = iso_check(s);
    if (rc != MMN_OK) return rc;
    if (!rx_loc || !rx_dir || !rough || !voxel || !direction) return MMN_ERR_NULL_POINTER;
    if (comp < 0 || comp >= s->num_comp) return MMN_ERR_INVALID_ARGUMENT;
    mmn::IsoParams p = iso_params(s);
    p.rx_locs = rx_loc;
    p.rx_dirs = rx_dir;
    p.num_ant = 1;
    const int64_t npix = (int64_t)s->width * s->height;
    mmn::iso_march_debug_kernel<<<(unsigned)((npix + 255) / 256), 256, 0, stream>>>(
        p, comp, tau, 0, rough, voxel, direction);
    return cudaGetLastError() == cudaSuccess ? MMN_OK : MMN_ERR_CUDA;
}
