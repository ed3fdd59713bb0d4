// rsdf.cu -- connected components of the normal mask and the relative signed distance
// field (RSDF) integrated from the normals by breadth-first search, on the GPU.
//
// Reference: src/data_processing/sdf.py:94-120 (_find_connected_components, which calls
// cc3d.connected_components(mask, connectivity=6)) and sdf.py:122-224
// (_construct_rsdf_components): for each valid component a FIFO breadth-first search
// from a seed voxel visits the 6-neighbours in the order (-x, +y, +x, -y, +z, -z) and sets
//     rsdf[adj] = rsdf[cell] + dot(step * dx, normal[adj])            (sdf.py:222)
// when it enqueues adj.  The value a voxel receives depends on which cell enqueued it,
// i.e. on the queue order, so the search here is level-synchronous but keeps that order
// exactly:
//   * the frontier of level k is stored in queue order;
//   * every (frontier position i, direction d) that reaches an unvisited voxel of the
//     component bids key 6*i + d for it (atomicMin): the smallest key is the cell
//     that dequeues first, which is the cell that enqueues the voxel sequentially;
//   * the winning bids, read in key order (an exclusive scan over the 6*|frontier| slots),
//     are the next level's queue order -- the order in which the sequential search appends
//     them.
// The increment is computed as numpy's dot of two 3-vectors: a running FP64 sum of the
// three products, without contraction, so the values are the reference's bit for bit.
//
// Components: lock-free union-find over the +x/+y/+z neighbours, always linking the larger
// root under the smaller, so every component ends with the smallest flat index in it as its
// root, whatever the order of the unions.  Every retry loop is bounded; a bound that runs
// out records MMN_ERR_TIMEOUT in the status word.
#include <cmath>
#include <cstring>

#include "mmn_internal.cuh"

namespace mmn {
namespace {

// parent[x] <= x always (atomicMin only lowers it), so paths strictly decrease and every
// loop below ends by construction; the bounds only guard against a broken invariant
constexpr int kUfMaxSteps = 1 << 26;   // steps of one find
constexpr int kUfMaxRetries = 1 << 16; // link attempts of one union

// parent entries change under other threads' atomicMin: read them through volatile so every
// step loads the current value
__device__ __forceinline__ int32_t uf_find(const int32_t *parent, int32_t a, int32_t *status) {
    const volatile int32_t *vp = parent;
    for (int s = 0; s < kUfMaxSteps; ++s) {
        const int32_t p = vp[a];
        if (p == a) return a;
        a = p;
    }
    set_status(status, MMN_ERR_TIMEOUT);
    return a;
}

__device__ void uf_union(int32_t *parent, int32_t a, int32_t b, int32_t *status) {
    for (int s = 0; s < kUfMaxRetries; ++s) {
        a = uf_find(parent, a, status);
        b = uf_find(parent, b, status);
        if (a == b) return;
        if (a < b) {
            const int32_t old = atomicMin(&parent[b], a);
            if (old == b) return;
            b = old;
        } else {
            const int32_t old = atomicMin(&parent[a], b);
            if (old == a) return;
            a = old;
        }
    }
    set_status(status, MMN_ERR_TIMEOUT);
}

// parent = the first voxel of the run along z as far back as this warp's 32 voxels reach (a run
// that enters the warp links to the voxel before it), so the z direction needs no unions; -1
// outside the mask.
__global__ void cc_init_kernel(const uint8_t *__restrict__ mask, int64_t n, int nz,
                               int32_t *__restrict__ parent, int32_t *__restrict__ count) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const bool in = v < n && mask[v];
    const int iz = v < n ? (int)((uint32_t)v % (uint32_t)nz) : 0;
    // lanes that continue the run of the lane before them
    const unsigned m = __ballot_sync(0xffffffffu, in);
    const unsigned cont = __ballot_sync(
        0xffffffffu, in && iz > 0 && (lane > 0 ? (m >> (lane - 1)) & 1u : mask[v - 1] != 0));
    if (v >= n) return;
    count[v] = 0;
    if (!in) {
        parent[v] = -1;
        return;
    }
    // the nearest lane at or below this one that does not continue a run
    const unsigned stops = ~cont & (lane == 31 ? 0xffffffffu : (1u << (lane + 1)) - 1u);
    const int first = stops ? 31 - __clz(stops) : -1;
    parent[v] = (int32_t)(v - lane + first);  // first = -1: the voxel before the warp's
}

// Unions with the +x and +y neighbours, only where two runs begin to touch: if the voxels before
// both along z are in the mask too, those two are already being joined.
__global__ void cc_union_kernel(const uint8_t *__restrict__ mask, int nx, int ny, int nz,
                                int32_t *parent, int32_t *status) {
    const uint32_t n = (uint32_t)nx * ny * nz;
    const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n || !mask[v]) return;
    const uint32_t nyz = (uint32_t)ny * nz;
    const int ix = (int)(v / nyz);
    const int iz = (int)(v % (uint32_t)nz), iy = (int)(v / (uint32_t)nz % (uint32_t)ny);
    const bool before = iz > 0 && mask[v - 1];
    if (ix + 1 < nx && mask[v + nyz] && !(before && mask[v + nyz - 1]))
        uf_union(parent, (int32_t)v, (int32_t)(v + nyz), status);
    if (iy + 1 < ny && mask[v + nz] && !(before && mask[v + nz - 1]))
        uf_union(parent, (int32_t)v, (int32_t)(v + nz), status);
}

// Roots, and the components' sizes (one atomic per warp and root: a component's voxels all add to
// one word).
__global__ void cc_flatten_kernel(int64_t n, int32_t *parent, int32_t *__restrict__ count,
                                  int32_t *status) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = v < n && parent[v] >= 0;
    const unsigned active = __ballot_sync(0xffffffffu, in);
    if (!in) return;
    const int32_t r = uf_find(parent, (int32_t)v, status);
    parent[v] = r;
    const unsigned same = __match_any_sync(active, r);
    if ((int)(threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&count[r], __popc(same));
}

// ------------------------------------------------------------------ breadth-first search
struct BfsArgs {
    int nx, ny, nz;
    const double *normals;   // [V, 3]
    uint32_t *state;         // [V] all-ones: open; 0: closed (visited, NaN or another component);
                             // during a level an open voxel holds its smallest bid (key + 1)
    double *rsdf;            // [V]
    double dx;
};

// One word per voxel says whether it can still be reached: a bid is one atomicMin whatever it
// meets (0 stays the least), and a voxel is won by the key it then holds.
__global__ void bfs_state_kernel(const double *__restrict__ normals,
                                 const int32_t *__restrict__ root, int32_t comp_root, int64_t n,
                                 uint32_t *__restrict__ state) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    state[v] = root[v] == comp_root && !isnan(normals[3 * v]) ? 0xffffffffu : 0u;
}

struct Cell {
    int ix, iy, iz;
};
__device__ __forceinline__ Cell cell_of(const BfsArgs &a, int32_t v) {
    const uint32_t t = (uint32_t)v / (uint32_t)a.nz;
    Cell c;
    c.iz = (int)((uint32_t)v - t * (uint32_t)a.nz);
    c.ix = (int)(t / (uint32_t)a.ny);
    c.iy = (int)(t - (uint32_t)c.ix * (uint32_t)a.ny);
    return c;
}

// neighbour in direction d: (-x, +y, +x, -y, +z, -z), sdf.py's dX/dY/dZ order
__device__ __forceinline__ bool neighbour(const BfsArgs &a, int32_t v, const Cell &c, int d,
                                          int32_t &out) {
    switch (d) {
        case 0: out = v - a.ny * a.nz; return c.ix > 0;
        case 1: out = v + a.nz; return c.iy + 1 < a.ny;
        case 2: out = v + a.ny * a.nz; return c.ix + 1 < a.nx;
        case 3: out = v - a.nz; return c.iy > 0;
        case 4: out = v + 1; return c.iz + 1 < a.nz;
        default: out = v - 1; return c.iz > 0;
    }
}

// value of voxel n reached in direction d from a cell of value `from`: step * dx as numpy forms
// it, then dot(): 0 + s0*n0 + s1*n1 + s2*n2 in FP64, in order
__device__ __forceinline__ double step_value(const BfsArgs &a, int32_t n, int d, double from) {
    const double sx = d == 0 ? -1.0 : (d == 2 ? 1.0 : 0.0);
    const double sy = d == 1 ? 1.0 : (d == 3 ? -1.0 : 0.0);
    const double sz = d == 4 ? 1.0 : (d == 5 ? -1.0 : 0.0);
    const double *nv = a.normals + 3 * (int64_t)n;
    double acc = 0.0;
    acc = __dadd_rn(acc, __dmul_rn(__dmul_rn(sx, a.dx), __ldg(nv)));
    acc = __dadd_rn(acc, __dmul_rn(__dmul_rn(sy, a.dx), __ldg(nv + 1)));
    acc = __dadd_rn(acc, __dmul_rn(__dmul_rn(sz, a.dx), __ldg(nv + 2)));
    return __dadd_rn(from, acc);
}

__global__ void bfs_bid_kernel(const BfsArgs a, const int32_t *__restrict__ frontier, int64_t nf) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nf * 6) return;
    const int32_t v = frontier[k / 6];
    int32_t n;
    if (neighbour(a, v, cell_of(a, v), (int)(k % 6), n)) atomicMin(&a.state[n], (uint32_t)k + 1u);
}

__global__ void bfs_flag_kernel(const BfsArgs a, const int32_t *__restrict__ frontier, int64_t nf,
                                int32_t *__restrict__ flag) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nf * 6) return;
    const int32_t v = frontier[k / 6];
    int32_t n;
    flag[k] = neighbour(a, v, cell_of(a, v), (int)(k % 6), n) && a.state[n] == (uint32_t)k + 1u;
}

// after the exclusive scan pos[k] is the winner's place in the next frontier
__global__ void bfs_emit_kernel(const BfsArgs a, const int32_t *__restrict__ frontier, int64_t nf,
                                const int32_t *__restrict__ pos, int32_t *__restrict__ next) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nf * 6) return;
    const int32_t v = frontier[k / 6];
    const int d = (int)(k % 6);
    int32_t n;
    if (!neighbour(a, v, cell_of(a, v), d, n) || a.state[n] != (uint32_t)k + 1u) return;
    a.rsdf[n] = step_value(a, n, d, a.rsdf[v]);
    next[pos[k]] = n;
}

__global__ void bfs_mark_kernel(const int32_t *__restrict__ next, int64_t n, uint32_t *state) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) state[next[k]] = 0;
}

__global__ void bfs_seed_kernel(int32_t seed, int32_t *frontier, uint32_t *state, double *rsdf) {
    frontier[0] = seed;
    state[seed] = 0;
    rsdf[seed] = 0.0;
}

// Small frontiers: one CTA runs whole levels -- the same bids, winners, queue positions
// and rsdf values as the per-level kernels above, with __syncthreads between the phases
// instead of kernel boundaries and a host read-back -- until the frontier empties or grows
// past kSmallFrontier entries (then the per-level kernels take over from the frontier it
// leaves in global memory).  The frontier stays in shared memory; a thread owns consecutive
// entries, all six directions of one at a time, so that a level's latency is one round of
// reductions, one of loads and one of normals.  What bounds it then is one SM's scattered traffic
// (a 32-byte sector a bid), so a bit per open voxel is kept in shared memory too, where it fits
// (MASK), and only open neighbours cost a bid and a load.  100 x 96 x 72 cap: 2.85 ms when each
// slot walked frontier, visited, normal, root and bid in turn; 1.21 ms; 0.89 ms with the bits (86 levels).
// A block-wide exclusive scan of the threads' winner counts gives the queue order.  The
// loop ends: every level marks at least one new voxel of a finite component.
constexpr int kSmallThreads = 1024;
constexpr int kSmallFrontier = 4096;
constexpr int kSmallPer = kSmallFrontier / kSmallThreads;  // entries per thread, at most
constexpr size_t kSmallBytes = 2 * kSmallFrontier * sizeof(int32_t);
constexpr size_t kSmallMost = 224 * 1024;  // shared memory of one CTA, less the static part

struct SmallState {
    int64_t nf;       // frontier size on exit (0: the search is complete)
    int64_t visited;  // voxels marked by this launch
    int32_t parity;   // 1: the exit frontier is in the second buffer
    int32_t pad;
};

template <bool MASK>
__global__ void __launch_bounds__(kSmallThreads) bfs_small_kernel(const BfsArgs a, int32_t *fa,
                                                                  int32_t *fb, int64_t nf0,
                                                                  SmallState *state) {
    extern __shared__ __align__(16) unsigned char dyn[];
    int32_t *cell = reinterpret_cast<int32_t *>(dyn);                      // [2][kSmallFrontier]
    uint32_t *open = reinterpret_cast<uint32_t *>(cell + 2 * kSmallFrontier);  // MASK: [V / 32]
    __shared__ int32_t warp_tot[kSmallThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int nf = (int)nf0, cur = 0;
    int64_t marked = 0;
    for (int i = tid; i < nf; i += kSmallThreads) cell[i] = fa[i];
    if (MASK) {
        const int nvox = a.nx * a.ny * a.nz;
        for (int v0 = 0; v0 < nvox; v0 += kSmallThreads) {
            const int v = v0 + tid;
            const unsigned b = __ballot_sync(0xffffffffu, v < nvox && __ldcg(&a.state[v]) != 0u);
            if (lane == 0 && v < nvox) open[v >> 5] = b;
        }
    }
    __syncthreads();
    bool spilled = false;  // the next frontier went to global memory
    while (nf > 0 && !spilled) {
        const int32_t *cc = cell + cur * kSmallFrontier;
        int32_t *nc = cell + (cur ^ 1) * kSmallFrontier;
        const int per = (nf + kSmallThreads - 1) / kSmallThreads;
        const int i0 = tid * per, i1 = min(i0 + per, nf);
        // bids
        uint32_t bid = 0;
        for (int i = i0; i < i1; ++i) {
            const int32_t v = cc[i];
            const Cell c = cell_of(a, v);
#pragma unroll
            for (int d = 0; d < 6; ++d) {
                int32_t n;
                if (neighbour(a, v, c, d, n) && (!MASK || open[n >> 5] >> (n & 31) & 1u)) {
                    atomicMin(&a.state[n], (uint32_t)(6 * i + d) + 1u);
                    bid |= 1u << (6 * (i - i0) + d);
                }
            }
        }
        __syncthreads();
        // winners of this thread's slots; the bids came from atomics at L2: read them past L1
        uint32_t won = 0;
        for (int i = i0; i < i1; ++i) {
            const uint32_t mine = bid >> (6 * (i - i0)) & 63u;
            if (!mine) continue;
            const int32_t v = cc[i];
            const Cell c = cell_of(a, v);
            uint32_t got[6];
#pragma unroll
            for (int d = 0; d < 6; ++d) {
                int32_t n;
                neighbour(a, v, c, d, n);
                got[d] = mine >> d & 1u ? __ldcg(&a.state[n]) : 0u;
            }
#pragma unroll
            for (int d = 0; d < 6; ++d)
                if (got[d] == (uint32_t)(6 * i + d) + 1u) won |= 1u << (6 * (i - i0) + d);
        }
        // exclusive scan of the counts over the block, in thread (= slot) order
        const int32_t cnt = __popc(won);
        int32_t incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) warp_tot[warp] = incl;
        __syncthreads();
        int32_t w = warp_tot[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        const int32_t total = __shfl_sync(0xffffffffu, w, 31);
        const int32_t before = __shfl_sync(0xffffffffu, w, warp > 0 ? warp - 1 : 0);
        int32_t pos = incl - cnt + (warp > 0 ? before : 0);
        spilled = total > kSmallFrontier;
        // emit in queue order
        for (int i = i0; i < i1; ++i) {
            const uint32_t mine = won >> (6 * (i - i0)) & 63u;
            if (!mine) continue;
            const int32_t v = cc[i];
            const Cell c = cell_of(a, v);
            const double from = a.rsdf[v];
#pragma unroll
            for (int d = 0; d < 6; ++d) {
                if (!(mine >> d & 1u)) continue;
                int32_t n;
                neighbour(a, v, c, d, n);
                const double x = step_value(a, n, d, from);
                a.rsdf[n] = x;
                a.state[n] = 0;
                if (MASK) atomicAnd(&open[n >> 5], ~(1u << (n & 31)));
                (spilled ? fb : nc)[pos++] = n;
            }
        }
        __syncthreads();
        marked += total;
        nf = total;
        cur ^= 1;
    }
    if (tid == 0) {
        state->nf = nf;
        state->visited = marked;
        state->parity = spilled ? 1 : 0;
    }
}
static_assert(6 * kSmallPer <= 32, "a thread's winners are bits of one word");

// ---------------------------------------------------------------- exclusive int32 scan
constexpr int kScanThreads = 256;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;  // 1024 values per block

__global__ void scan_block_kernel(int32_t *data, int64_t n, int32_t *block_sums) {
    __shared__ int32_t warp_sums[kScanThreads / 32];
    const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
    int32_t v[kScanItems];
    int32_t run = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        v[i] = base + i < n ? data[base + i] : 0;
        const int32_t t = v[i];
        v[i] = run;  // exclusive within the thread
        run += t;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t incl = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        int32_t w = lane < kScanThreads / 32 ? warp_sums[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < kScanThreads / 32) warp_sums[lane] = w;  // inclusive over warps
    }
    __syncthreads();
    const int32_t offset = (incl - run) + (warp > 0 ? warp_sums[warp - 1] : 0);
#pragma unroll
    for (int i = 0; i < kScanItems; ++i)
        if (base + i < n) data[base + i] = v[i] + offset;
    if (threadIdx.x == kScanThreads - 1) block_sums[blockIdx.x] = offset + run;
}

__global__ void scan_add_kernel(int32_t *data, int64_t n, const int32_t *block_offsets) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) data[k] += block_offsets[k / kScanTile];
}

size_t scan_temp_elems(int64_t n) {
    size_t total = 0;
    while (n > 1) {
        n = (n + kScanTile - 1) / kScanTile;
        total += (size_t)n + 1;
    }
    return total + 2;
}

// exclusive scan of data[0..n) in place; data[n] (one past the end) receives the total
cudaError_t scan_exclusive(int32_t *data, int64_t n, int32_t *temp, cudaStream_t stream) {
    const int64_t blocks = (n + kScanTile - 1) / kScanTile;
    int32_t *sums = temp;
    scan_block_kernel<<<(unsigned)blocks, kScanThreads, 0, stream>>>(data, n, sums);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (blocks > 1) {
        // scan the block totals (recursively), then add each block's offset
        e = scan_exclusive(sums, blocks, temp + blocks + 1, stream);
        if (e != cudaSuccess) return e;
        scan_add_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(data, n, sums);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        return cudaMemcpyAsync(data + n, sums + blocks, sizeof(int32_t),
                               cudaMemcpyDeviceToDevice, stream);
    }
    return cudaMemcpyAsync(data + n, sums, sizeof(int32_t), cudaMemcpyDeviceToDevice, stream);
}

inline unsigned grid_for(int64_t n, int nt) { return (unsigned)((n + nt - 1) / nt); }

}  // namespace
}  // namespace mmn

using namespace mmn;

namespace {
constexpr size_t kStatus = 256;
inline size_t up256(size_t x) { return (x + 255) & ~(size_t)255; }

bool bad_dims(int32_t nx, int32_t ny, int32_t nz) {
    if (nx < 1 || ny < 1 || nz < 1) return true;
    const int64_t v = (int64_t)nx * ny * nz;
    return v > (int64_t)INT32_MAX / 6;  // flat indices and 6 bids per voxel fit in int32
}
}  // namespace

extern "C" size_t mmn_components_workspace_bytes(int64_t num_voxels) {
    (void)num_voxels;
    return kStatus;
}

extern "C" int mmn_components(int32_t nx, int32_t ny, int32_t nz, const uint8_t *mask,
                              int32_t *root, int32_t *count, void *workspace,
                              size_t workspace_bytes, cudaStream_t stream) {
    if (bad_dims(nx, ny, nz)) return MMN_ERR_INVALID_ARGUMENT;
    if (!mask || !root || !count) return MMN_ERR_NULL_POINTER;
    if (!workspace || workspace_bytes < kStatus ||
        (reinterpret_cast<uintptr_t>(workspace) & 255))
        return MMN_ERR_WORKSPACE;
    const int64_t n = (int64_t)nx * ny * nz;
    int32_t *status = static_cast<int32_t *>(workspace);
    if (cudaMemsetAsync(status, 0, kStatus, stream) != cudaSuccess) return MMN_ERR_CUDA;
    cc_init_kernel<<<grid_for(n, 256), 256, 0, stream>>>(mask, n, nz, root, count);
    cc_union_kernel<<<grid_for(n, 256), 256, 0, stream>>>(mask, nx, ny, nz, root, status);
    cc_flatten_kernel<<<grid_for(n, 256), 256, 0, stream>>>(n, root, count, status);
    return cudaGetLastError() == cudaSuccess ? MMN_OK : MMN_ERR_CUDA;
}

// Start voxel of a component's search (sdf.py:187-193), on the host: the voxel nearest the mean of
// its voxels' coordinates, the first among ties, in numpy's order of operations -- the mean's sums
// row by row, each distance sqrt((x x + y y) + z z) -- so the choice is numpy's.  flat: the
// component's flat indices, ascending; x, y, z: the axes.  numpy's own calls build the coordinate
// rows and seven temporaries: 4.5 ms for 97,000 voxels, here under 1.
extern "C" int mmn_rsdf_seed(const int64_t *flat, int64_t count, int32_t ny, int32_t nz,
                             const double *x, const double *y, const double *z, int64_t *seed) {
    if (count < 1 || ny < 1 || nz < 1) return MMN_ERR_INVALID_ARGUMENT;
    if (!flat || !x || !y || !z || !seed) return MMN_ERR_NULL_POINTER;
    // walks the ascending list row by row: f(index, x, y, z) for every voxel
    auto each = [&](auto &&f) {
        int64_t row = -1, first = 0, past = 0;
        double xv = 0.0, yv = 0.0;
        for (int64_t i = 0; i < count; ++i) {
            const int64_t v = flat[i];
            if (v < first || v >= past) {
                row = v / nz;
                first = row * nz;
                past = first + nz;
                xv = x[row / ny];
                yv = y[row % ny];
            }
            f(i, xv, yv, z[v - first]);
        }
    };
    double sx = 0.0, sy = 0.0, sz = 0.0;
    each([&](int64_t, double a, double b, double c) {
        sx += a;
        sy += b;
        sz += c;
    });
    const double mx = sx / (double)count, my = sy / (double)count, mz = sz / (double)count;
    double best = 0.0;
    int64_t at = -1;
    bool nan = false;
    each([&](int64_t i, double a, double b, double c) {
        const double ex = a - mx, ey = b - my, ez = c - mz;
        const double xx = ex * ex, yy = ey * ey, zz = ez * ez;
        const double s = xx + yy;
        const double d = std::sqrt(s + zz);
        // argmin: the first least, or the first NaN
        if (at < 0 || (!nan && (d < best || d != d))) {
            best = d;
            at = i;
            nan = d != d;
        }
    });
    *seed = flat[at];
    return MMN_OK;
}

extern "C" size_t mmn_rsdf_workspace_bytes(int32_t nx, int32_t ny, int32_t nz) {
    if (bad_dims(nx, ny, nz)) return 0;
    const int64_t n = (int64_t)nx * ny * nz;
    return kStatus + up256((size_t)n * 4) + 2 * up256((size_t)n * 4) +
           up256(((size_t)6 * n + 1) * 4) + up256(scan_temp_elems(6 * n) * 4) + 256;
}

extern "C" int mmn_rsdf_component(int32_t nx, int32_t ny, int32_t nz, const double *normals,
                                  const int32_t *root, int32_t comp_root, int32_t seed,
                                  double dx, double *rsdf, int64_t *visited_count,
                                  void *workspace, size_t workspace_bytes,
                                  cudaStream_t stream) {
    if (bad_dims(nx, ny, nz)) return MMN_ERR_INVALID_ARGUMENT;
    if (!normals || !root || !rsdf) return MMN_ERR_NULL_POINTER;
    const int64_t n = (int64_t)nx * ny * nz;
    if (seed < 0 || seed >= n || comp_root < 0 || comp_root >= n || !(dx > 0.0))
        return MMN_ERR_INVALID_ARGUMENT;
    const size_t need = mmn_rsdf_workspace_bytes(nx, ny, nz);
    if (!workspace || workspace_bytes < need || (reinterpret_cast<uintptr_t>(workspace) & 255))
        return MMN_ERR_WORKSPACE;
    unsigned char *w = static_cast<unsigned char *>(workspace);
    size_t off = kStatus;
    uint32_t *state = reinterpret_cast<uint32_t *>(w + off);
    off += up256((size_t)n * 4);
    int32_t *fa = reinterpret_cast<int32_t *>(w + off);
    off += up256((size_t)n * 4);
    int32_t *fb = reinterpret_cast<int32_t *>(w + off);
    off += up256((size_t)n * 4);
    int32_t *flag = reinterpret_cast<int32_t *>(w + off);
    off += up256(((size_t)6 * n + 1) * 4);
    int32_t *temp = reinterpret_cast<int32_t *>(w + off);

    if (cudaMemsetAsync(w, 0, kStatus, stream) != cudaSuccess) return MMN_ERR_CUDA;
    BfsArgs a;
    a.nx = nx;
    a.ny = ny;
    a.nz = nz;
    a.normals = normals;
    a.state = state;
    a.rsdf = rsdf;
    a.dx = dx;
    bfs_state_kernel<<<grid_for(n, 256), 256, 0, stream>>>(normals, root, comp_root, n, state);
    bfs_seed_kernel<<<1, 1, 0, stream>>>(seed, fa, state, rsdf);
    const size_t with_bits = kSmallBytes + ((size_t)n + 31) / 32 * 4;
    const bool bits = with_bits <= kSmallMost;
    const size_t small_bytes = bits ? with_bits : kSmallBytes;
    const void *small_fn = bits ? reinterpret_cast<const void *>(&bfs_small_kernel<true>)
                                : reinterpret_cast<const void *>(&bfs_small_kernel<false>);
    if (cudaFuncSetAttribute(small_fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)small_bytes) != cudaSuccess)
        return MMN_ERR_CUDA;
    int64_t nf = 1, total = 1;
    // the single-CTA search's exit state, in the workspace header after the status word
    SmallState *small = reinterpret_cast<SmallState *>(w + 64);
    // every level (and every single-CTA launch) adds at least one voxel, so n rounds bound
    // the search
    for (int64_t level = 0; nf > 0 && level <= n; ++level) {
        if (nf <= kSmallFrontier) {
            void *args[] = {&a, &fa, &fb, &nf, &small};
            if (cudaLaunchKernel(small_fn, dim3(1), dim3(kSmallThreads), args, small_bytes,
                                 stream) != cudaSuccess)
                return MMN_ERR_CUDA;
            SmallState hs;
            if (cudaGetLastError() != cudaSuccess ||
                cudaMemcpyAsync(&hs, small, sizeof(hs), cudaMemcpyDeviceToHost, stream) !=
                    cudaSuccess ||
                cudaStreamSynchronize(stream) != cudaSuccess)
                return MMN_ERR_CUDA;
            total += hs.visited;
            nf = hs.nf;
            if (hs.parity) {
                int32_t *t = fa;
                fa = fb;
                fb = t;
            }
            continue;
        }
        const int64_t slots = nf * 6;
        bfs_bid_kernel<<<grid_for(slots, 256), 256, 0, stream>>>(a, fa, nf);
        bfs_flag_kernel<<<grid_for(slots, 256), 256, 0, stream>>>(a, fa, nf, flag);
        if (scan_exclusive(flag, slots, temp, stream) != cudaSuccess) return MMN_ERR_CUDA;
        bfs_emit_kernel<<<grid_for(slots, 256), 256, 0, stream>>>(a, fa, nf, flag, fb);
        int32_t next_n = 0;
        if (cudaMemcpyAsync(&next_n, flag + slots, sizeof(int32_t), cudaMemcpyDeviceToHost,
                            stream) != cudaSuccess ||
            cudaStreamSynchronize(stream) != cudaSuccess)
            return MMN_ERR_CUDA;
        if (next_n > 0)
            bfs_mark_kernel<<<grid_for(next_n, 256), 256, 0, stream>>>(fb, next_n, state);
        if (cudaGetLastError() != cudaSuccess) return MMN_ERR_CUDA;
        nf = next_n;
        total += next_n;
        int32_t *t = fa;
        fa = fb;
        fb = t;
    }
    if (visited_count) *visited_count = total;
    int32_t st = 0;
    if (cudaMemcpyAsync(&st, w, sizeof(int32_t), cudaMemcpyDeviceToHost, stream) != cudaSuccess ||
        cudaStreamSynchronize(stream) != cudaSuccess)
        return MMN_ERR_CUDA;
    return st ? st : MMN_OK;
}
