"""The measurement gradient's spreads onto an antenna's grid row (spread_row for node values,
spread_voxels, bp_local.cu), run on the host by 32 threads: every access to the warp's shared memory is recorded with the number of
warp barriers its lane has passed, and two lanes that touch one cell between the same two barriers,
one of them writing, are a race (ballots and reductions order no memory).  The row's sums are
checked too, against numpy's (FP32 sums of at most 32 terms: 1e-5 relative)."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SOURCE = os.path.join(HERE, "..", "mmnorm_b200", "csrc", "bp_local.cu")

HARNESS = r"""
#include <barrier>
#include <cstdint>
#include <map>
#include <mutex>
#include <set>
#include <thread>
#include <vector>
constexpr int kNuW = 8;
static std::barrier<> g_bar(32);
static std::mutex g_lock;
static const char *g_lo, *g_hi;   // shared memory: row and scratch
static int g_races;
struct Dim { int x; };
static thread_local Dim threadIdx;
static thread_local int t_epoch;
struct Use { int epoch = -1; std::set<int> readers, writers; };
static std::map<const void *, Use> g_use;
static void touch(const void *p, bool write) {
    if ((const char *)p < g_lo || (const char *)p >= g_hi) return;
    std::lock_guard<std::mutex> l(g_lock);
    Use &u = g_use[p];
    if (u.epoch != t_epoch) { u.epoch = t_epoch; u.readers.clear(); u.writers.clear(); }
    const int me = threadIdx.x;
    for (int w : u.writers) g_races += w != me;
    if (write) for (int r : u.readers) g_races += r != me;
    (write ? u.writers : u.readers).insert(me);
}
struct float2 {
    float x, y;
    float2() {}
    float2(float a, float b) : x(a), y(b) {}
    float2(const float2 &o) { touch(&o, false); x = o.x; y = o.y; }
    float2 &operator=(const float2 &o) { touch(&o, false); touch(this, true); x = o.x; y = o.y; return *this; }
};
struct Cell {
    int v;
    operator int() const { touch(this, false); return v; }
    Cell &operator=(int a) { touch(this, true); v = a; return *this; }
};
struct Comp {   // a float of the row
    float v;
    Comp &operator+=(float a) { touch(this, false); touch(this, true); v += a; return *this; }
};
constexpr int kNuWin = 16;
struct LocSpread { float2 w[32][kNuW]; float2 win[kNuWin][32]; Cell ix[32]; };
static float2 make_float2(float a, float b) { return float2(a, b); }
static float2 __fadd2_rn(float2 a, float2 b) { return float2(a.x + b.x, a.y + b.y); }
static int __ffs(unsigned m) { return __builtin_ffs(m); }
static void __syncwarp() { g_bar.arrive_and_wait(); ++t_epoch; g_bar.arrive_and_wait(); }
static int g_vals[32];
static unsigned __ballot_sync(unsigned, bool b) {
    g_vals[threadIdx.x] = b; g_bar.arrive_and_wait();
    unsigned m = 0; for (int i = 0; i < 32; ++i) m |= (unsigned)g_vals[i] << i;
    g_bar.arrive_and_wait(); return m;
}
static int __reduce_min_sync(unsigned, int v) {
    g_vals[threadIdx.x] = v; g_bar.arrive_and_wait();
    int m = g_vals[0]; for (int i = 1; i < 32; ++i) m = g_vals[i] < m ? g_vals[i] : m;
    g_bar.arrive_and_wait(); return m;
}
static float g_fvals[32];
static float __shfl_xor_sync(unsigned, float v, int m) {
    g_fvals[threadIdx.x] = v; g_bar.arrive_and_wait();
    const float r = g_fvals[threadIdx.x ^ m];
    g_bar.arrive_and_wait(); return r;
}
static const int *g_cell;
static void nufft_taps(double, double, int, int &cell, float (&w)[kNuW]) {
    cell = g_cell[threadIdx.x];
    for (int i = 0; i < kNuW; ++i) w[i] = 1.f + i;
}
static void nufft_taps64(double, double, int, int &cell, double (&w)[kNuW]) {
    cell = g_cell[threadIdx.x];
    for (int i = 0; i < kNuW; ++i) w[i] = 1.0 + i;
}
#define __device__
#define __noinline__
#define __forceinline__
@FUNCTION@
struct Shared { LocSpread sp; float2 row[4096]; };
extern "C" int spread(const int *cells, const int *active, int calls, int mrow, float *out, int voxels) {
    static Shared sh;
    g_lo = (const char *)&sh; g_hi = (const char *)(&sh + 1);
    g_races = 0; g_use.clear();
    for (int i = 0; i < mrow; ++i) sh.row[i].x = sh.row[i].y = 0.f;
    for (int c = 0; c < calls; ++c) {
        g_cell = cells + 32 * c;
        std::vector<std::thread> t;
        for (int l = 0; l < 32; ++l)
            t.emplace_back([&, l, c] {
                threadIdx.x = l; t_epoch = 1000 * c;
                const float2 v = make_float2(1.f + l, -2.f * l);
                const bool on = active[32 * c + l] != 0;
                if (voxels) spread_voxels(sh.sp, sh.row, 0.0, v, 0.0, 0);
                else spread_row(sh.sp, sh.row, mrow, 0.0, v, on, 0.0, 0);
            });
        for (auto &x : t) x.join();
    }
    for (int i = 0; i < mrow; ++i) { out[2 * i] = sh.row[i].x; out[2 * i + 1] = sh.row[i].y; }
    return g_races;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    with open(SOURCE) as f:
        text = f.read()
    body = ""
    for name in ("spread_row", "spread_voxels"):
        m = re.search(r"__device__ [^\n]*void %s\(.*?\n}\n" % name, text, re.S)
        assert m, name + " not found"
        body += m.group(0)
    body = body.replace("float *rowf = reinterpret_cast<float *>", "Comp *rowf = reinterpret_cast<Comp *>")
    d = tmp_path_factory.mktemp("spread")
    src, out = str(d / "spread.cpp"), str(d / "spread.so")
    with open(src, "w") as f:
        f.write(HARNESS.replace("@FUNCTION@", body))
    subprocess.run(["g++", "-std=c++20", "-O1", "-shared", "-fPIC", "-pthread", "-w", "-o", out,
                    src], check=True)
    return ctypes.CDLL(out)


@pytest.mark.parametrize("voxels", [False, True])
@pytest.mark.parametrize("n,lo,hi,active", [
    (256, 40, 60, 32),     # one window
    (256, 40, 60, 8),      # node values of a box: a lane each
    (256, 10, 240, 32),    # a wide box
    (256, 100, 127, 24),   # a second window that starts where the first ends
    (48, 30, 70, 32),      # a short grid, cells that wrap past its end
    (32, 0, 32, 32),
])
def test_no_lane_reads_what_another_wrote(lib, n, lo, hi, active, voxels):
    rng = np.random.default_rng(n + hi)
    active = 32 if voxels else active
    calls, mrow = 3, n + 16
    cells = np.sort(rng.integers(lo, hi, (calls, 32)) % n, axis=1).astype(np.int32)
    rng.shuffle(cells, axis=1)
    act = np.zeros((calls, 32), np.int32)
    act[:, :active] = 1
    out = np.zeros((mrow, 2), np.float32)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    races = lib.spread(p(cells), p(act), calls, mrow, p(out), int(voxels))
    ref = np.zeros((mrow, 2))
    for c in range(calls):
        for lane in range(active):
            for i in range(8):
                ref[cells[c, lane] + i] += (1 + i) * np.array([1.0 + lane, -2.0 * lane])
    np.testing.assert_allclose(out, ref, rtol=1e-5, atol=1e-5 * np.abs(ref).max())
    assert races == 0
