"""The channel kernel's ray culling and batching against a march of every ray (mmn_iso_march,
which drops none): views of one pixel, partial ray tiles, rows that are a power of two, more
reachable rays in one tile than a batch holds, the eye inside the box, the box behind the eye
(the reference's -1 sentinel steps backwards), two components, several offset sets.

Channels of the marched hits are formed in numpy (the refinement in FP32 as the kernel states it,
the phasors in FP64).  Tolerance 5e-6 relative: phase steps of 2^-32 turns, the hardware sine's
4e-7 and FP32 sums of at most a few thousand unit phasors."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

C = 2.99792458e8
f32 = np.float32


def _refined(grid, tau, rough, voxel, dirs, vs, lower):
    """Hit points float32 [n, 3] of the rough hits, one rounding per operation."""
    # a hit counts if its cell is in the grid (-1 counts as 0); no hit: rough and voxel all -1
    cell = np.where(voxel == -1, 0, voxel)
    hit = np.all((cell >= 0) & (cell + 1 < grid.shape), axis=1) & \
        ~np.all((voxel == -1) & (rough == -1), axis=1)
    v, h, d = voxel[hit], rough[hit], dirs[hit]
    i = cell[hit].astype(int)
    at = lambda a, b, c: (grid[i[:, 0] + a, i[:, 1] + b, i[:, 2] + c] - f32(tau)).astype(f32)
    lerp = lambda t, a, b: ((f32(1) - t) * a + t * b).astype(f32)
    t = [((h[:, k] - (f32(lower[k]) + v[:, k] * f32(vs)).astype(f32)) / f32(vs)).astype(f32)
         for k in range(3)]
    e = {(b, c): lerp(t[0], at(0, b, c), at(1, b, c)) for b in (0, 1) for c in (0, 1)}
    z = [lerp(t[1], e[0, c], e[1, c]) for c in (0, 1)]
    sdf = lerp(t[2], z[0], z[1])
    return (h + (d * sdf[:, None]).astype(f32)).astype(f32)


@pytest.mark.parametrize("w,h,fov,centre_z,eye_z,comps,sets", [
    (1, 1, 0.5, 0.3, 0.0, 1, 1),
    (37, 23, 20.0, 0.3, 0.0, 1, 2),
    (256, 40, 12.0, 0.25, 0.0, 2, 1),
    (300, 70, 4.0, 0.3, 0.0, 1, 3),     # every ray reaches the box
    (64, 64, 80.0, 0.02, 0.02, 1, 1),   # the eye inside the box
    (90, 50, 40.0, -1.0, 0.0, 1, 1),    # a metre behind the eye
    (64, 30, 80.0, 0.0194, 0.0, 1, 1),  # the eye 0.4 of a voxel outside the box
])
def test_channels_of_every_ray(cuda_dev, w, h, fov, centre_z, eye_z, comps, sets):
    import torch
    from mmnorm_b200 import _lib, isosurface
    from mmnorm_b200.ops import _stream, _vp
    rng = np.random.default_rng(w + h)
    vs, n = 0.001, (41, 43, 39)
    lo = np.array([-0.02, -0.021, centre_z - 0.019])
    ax = [lo[k] + vs * np.arange(n[k]) for k in range(3)]
    X, Y, Z = np.meshgrid(*ax, indexing="ij")
    r = np.sqrt(X ** 2 + (Y - 0.001) ** 2 + (Z - centre_z) ** 2) - 0.013
    shell = np.abs(r) < 0.005
    parts = [np.where(shell, r, -50.0)] if comps == 1 else \
        [np.where(shell & (X < 0), r, -50.0), np.where(shell & (X >= 0), r, -50.0)]
    sdf = np.stack(parts, -1).astype(f32)
    bbox = [a[0] for a in ax] + [a[-1] for a in ax]
    K = 33
    wl = C / (77.5e9 + np.arange(K) * 3e9 / K)
    scene = isosurface.make_scene(sdf, bbox, vs, wl, w, h, fov, fov, True)
    A = 3
    loc = np.concatenate([rng.uniform(-0.004, 0.004, (A, 2)), np.full((A, 1), eye_z)], 1)
    dirs = np.tile(np.array([[0.02, -0.01, -1.0]], f32), (A, 1))
    taus = rng.uniform(-0.002, 0.002, (sets, comps)).astype(f32)
    ch = isosurface.simulate_channels_batch(scene, torch.as_tensor(taus), loc, dirs).cpu().numpy()
    lib = _lib.load()
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=cuda_dev)
    hits = 0
    for s in range(sets):
        for a in range(A):
            ref = np.zeros(K, np.complex128)
            for c in range(comps):
                rough, voxel, ray = (torch.empty((w * h, 3), dtype=torch.float32, device=cuda_dev)
                                     for _ in range(3))
                one, rd = t(loc[a]), t(dirs[a])
                _lib.check(lib.mmn_iso_march(ctypes.byref(scene.scene), c, float(taus[s, c]),
                                             _vp(one), _vp(rd), _vp(rough), _vp(voxel), _vp(ray),
                                             _stream(cuda_dev)), "mmn_iso_march")
                pts = _refined(sdf[..., c], taus[s, c], *(v.cpu().numpy() for v in
                                                          (rough, voxel, ray)), vs, lo)
                d = 2 * np.linalg.norm(loc[a] - pts.astype(np.float64), axis=1) + 0.15
                hits += len(d)
                ref += np.exp(2j * np.pi * d[:, None] / wl[None]).sum(0)
            assert np.linalg.norm(ch[s, a] - ref) <= 5e-6 * max(np.linalg.norm(ref), 1.0)
    assert hits > 0 or centre_z < 0
