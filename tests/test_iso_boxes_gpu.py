"""The channel kernel's two shortcuts -- rays kept only if they can reach the defined voxels' box,
cells read by integer strides -- where their conditions change: most cases have at least as many
rays as voxels, so the box is formed wherever it may be.  Two components; the eye inside the box, beside
it, and past it where the grid's cells reach further than the box (voxels flatter in z than in y);
a box that ends between two cells (reads wrap into the next row there); the box behind the eye; a
shell in a corner; a field that is defined nowhere, or everywhere; an offset that defines voxels
below the bounds' slack; voxels above the undefined cells' 5 mm step; a grid whose flat indices
are not exact in FP32.  Against a march of every ray (mmn_iso_march), as in test_iso_batches_gpu,
with its tolerance."""
import ctypes

import numpy as np
import pytest

from test_iso_batches_gpu import C, _refined, f32

pytestmark = pytest.mark.gpu


def _check(dev, sdf, bbox, vs, loc, dirs, taus, w, h, fov):
    """Compares the channels; the number of hits."""
    import torch
    from mmnorm_b200 import _lib, isosurface
    from mmnorm_b200.ops import _stream, _vp
    K = 33
    wl = C / (77.5e9 + np.arange(K) * 3e9 / K)
    scene = isosurface.make_scene(sdf, bbox, vs, wl, w, h, fov, fov, True)
    ch = isosurface.simulate_channels_batch(scene, torch.as_tensor(taus), loc, dirs).cpu().numpy()
    lib = _lib.load()
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)
    hits = 0
    for s in range(len(taus)):
        for a in range(len(loc)):
            ref = np.zeros(K, np.complex128)
            for c in range(sdf.shape[-1]):
                rough, voxel, ray = (torch.empty((w * h, 3), dtype=torch.float32, device=dev)
                                     for _ in range(3))
                one, rd = t(loc[a]), t(dirs[a])
                _lib.check(lib.mmn_iso_march(ctypes.byref(scene.scene), c, float(taus[s, c]),
                                             _vp(one), _vp(rd), _vp(rough), _vp(voxel), _vp(ray),
                                             _stream(dev)), "mmn_iso_march")
                pts = _refined(sdf[..., c], taus[s, c], *(v.cpu().numpy() for v in
                                                          (rough, voxel, ray)), vs, bbox[:3])
                d = 2 * np.linalg.norm(loc[a] - pts.astype(np.float64), axis=1) + 0.15
                hits += len(d)
                ref += np.exp(2j * np.pi * d[:, None] / wl[None]).sum(0)
            assert np.linalg.norm(ch[s, a] - ref) <= 5e-6 * max(np.linalg.norm(ref), 1.0)
    return hits


@pytest.mark.parametrize("name,grid,vs,eye_z,fov,some", [
    ("two", (21, 23, 19), 0.001, 0.0, 6.0, True),
    ("inside", (21, 23, 19), 0.001, 0.3, 80.0, True),
    ("beside", (21, 23, 19), 0.001, 0.2906, 80.0, True),
    ("behind", (21, 23, 19), 0.001, 0.6, 40.0, False),
    ("corner", (31, 29, 27), 0.001, 0.0, 7.0, True),
    ("nowhere", (21, 23, 19), 0.001, 0.0, 6.0, False),
    ("low", (21, 23, 19), 0.001, 0.0, 6.0, True),
    ("coarse", (21, 23, 19), 0.006, 0.0, 40.0, True),
    ("flat", (21, 23, 39), 0.001, 0.314, 80.0, True),
    ("wrap", (21, 23, 19), 0.001, 0.3095, 3.0, True),
    ("large", (258, 256, 255), 0.001, 0.0, 30.0, True),
])
def test_channels_of_every_ray(cuda_dev, name, grid, vs, eye_z, fov, some):
    rng = np.random.default_rng(len(name) + grid[2])
    n, w, h = grid, 96, 64
    lo = np.array([-0.5 * (n[0] - 1), -0.5 * (n[1] - 1), -0.5 * (n[2] - 1)]) * vs
    lo[2] += 0.3
    ax = [lo[k] + vs * np.arange(n[k]) for k in range(3)]
    bbox = [a[0] for a in ax] + [a[-1] for a in ax]
    X, Y, Z = np.meshgrid(*ax, indexing="ij", sparse=True)
    c = (0.0, 0.0, 0.3) if name != "corner" else (0.009, -0.008, 0.307)
    radius = min(0.3 * vs * min(n), 0.02)
    r = np.sqrt((X - c[0]) ** 2 + (Y - c[1]) ** 2 + (Z - c[2]) ** 2) - radius
    sdf = np.where(np.abs(r) < 3 * vs, r, -50.0)[..., None]
    comps, taus = 1, rng.uniform(-0.3, 0.3, (2, 1)).astype(f32) * f32(vs)
    loc = np.array([[0.001, -0.002, eye_z], [-0.003, 0.001, eye_z], [0.0, 0.004, eye_z]])
    dirs = np.tile(np.array([[0.02, -0.01, -1.0]], f32), (3, 1))
    if name == "two":
        comps = 2
        sdf = np.concatenate([np.where(X < 0, sdf[..., 0], -50.0)[..., None],
                              np.where(X < 0, -50.0, sdf[..., 0])[..., None]], -1)
        taus = rng.uniform(-3e-4, 3e-4, (2, 2)).astype(f32)
    elif name == "nowhere":
        sdf[:] = -50.0
    elif name == "low":
        sdf[:, :, :4] = -46.0       # undefined, but not once an offset of -6.5 is taken off
        taus = np.array([[-6.5], [0.0]], f32)
    elif name == "flat":            # the box holds the lower half of the cells' extent
        bbox[5] = bbox[2] + 0.5 * (bbox[5] - bbox[2])
        taus = taus[:1]             # fewer rays than voxels: the grid's box; it lies behind the eye
        sdf[:] = 0.0004
    elif name == "wrap":            # the box ends 0.9 of a voxel above the last layer
        bbox[5] += 0.0009
        sdf = sdf * 0 + f32(0.0004)
        loc = np.array([[-0.1, 0.001, eye_z], [-0.2, -0.002, eye_z], [-0.15, 0.0, eye_z]])
        dirs = np.tile(np.array([[-1.0, 0.0, 0.0005]], f32), (3, 1))
    if name not in ("flat", "large"):
        assert 2 * 3 * w * h >= comps * np.prod(n)
    hits = _check(cuda_dev, np.ascontiguousarray(sdf.astype(f32)), bbox, vs, loc, dirs, taus, w, h,
                  fov)
    assert (hits > 0) == some
