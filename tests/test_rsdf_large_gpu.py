"""The relative signed distance search past its single-CTA kernel's limits: a frontier that
outgrows its 4096 entries and shrinks again (spill, per-level kernels, return), and grids whose
open bits do not fit shared memory (over about 1.57 M voxels), alone and with such a frontier.
Bit for bit against the sequential search.  Components with runs along z over several warps."""
import numpy as np
import pytest

from test_rsdf_gpu import _field

pytestmark = pytest.mark.gpu


def _shell_sizes(normals, seed):
    """Sizes of the search's levels on the voxels with a normal, from voxel ``seed``."""
    free = ~np.isnan(normals[..., 0])
    level = np.zeros(free.shape, bool)
    level[seed] = True
    sizes = []
    while level.any():
        sizes.append(int(level.sum()))
        free &= ~level
        grow = np.zeros_like(level)
        for ax in range(3):
            a, b = [slice(None)] * 3, [slice(None)] * 3
            a[ax], b[ax] = slice(1, None), slice(None, -1)
            grow[tuple(a)] |= level[tuple(b)]
            grow[tuple(b)] |= level[tuple(a)]
        level = grow & free
    return sizes


@pytest.mark.parametrize("grid,part,large", [
    ((64, 64, 64), (64, 64, 64), True),      # open bits in shared memory, frontier over 4096
    ((96, 128, 130), (40, 30, 3), False),    # no open bits: 1.6 M voxels, a small component
    ((70, 66, 350), (64, 63, 65), True),     # neither
])
def test_search_against_the_sequential_one(cuda_dev, grid, part, large):
    from oracle import rsdf_oracle as RO
    from mmnorm_b200 import rsdf
    rng = np.random.default_rng(sum(grid))
    n = np.full(grid + (3,), np.nan)
    at = [(g - p) // 2 for g, p in zip(grid, part)]
    where = tuple(slice(a, a + p) for a, p in zip(at, part))
    n[where] = rng.standard_normal(part + (3,))
    n[where] /= np.linalg.norm(n[where], axis=-1, keepdims=True)
    dx = 0.004
    ax = [np.arange(g) * dx - 0.1 for g in grid]
    out, labeled, valid, _ = rsdf.compute_rsdf(n, *ax)
    assert len(valid) == 1
    ref = RO.rsdf(n[where], RO.coords(*(a[s] for a, s in zip(ax, where))), labeled[where], valid,
                  ax[0])
    np.testing.assert_array_equal(out[where], ref)
    assert np.isnan(out).sum() == out.size - ref.size
    start = tuple(int(v[0]) for v in np.nonzero(ref == 0))
    assert (max(_shell_sizes(n[where], start)) > 4096) == large


@pytest.mark.parametrize("shape,seed", [((3, 4, 200), 11), ((2, 40, 65), 12), ((40, 3, 31), 13)])
def test_components_with_long_runs(cuda_dev, shape, seed):
    import torch
    from scipy import ndimage
    from mmnorm_b200 import rsdf
    _, mask = _field(shape, seed, level=-0.8)
    root = rsdf.component_roots(torch.as_tensor(mask, device=cuda_dev))[0].cpu().numpy()
    lab, n = ndimage.label(mask, structure=ndimage.generate_binary_structure(3, 1))
    flat = np.arange(mask.size).reshape(shape)
    assert np.all((root >= 0) == mask)
    for k in range(1, n + 1):
        assert np.all(root[lab == k] == flat[lab == k].min())
