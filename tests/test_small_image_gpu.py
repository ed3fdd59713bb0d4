"""Small problems: the one-launch normals of a small image (both sides of its size limit, an
image of one voxel, zeros and NaN) give the bits of the two-pass kernels; a problem with too
few voxel tiles to fill the GPU (short antenna stages, up to 64 splits, the grouped split
reduction) matches the FP64 oracle at the mixed form's tolerance and repeats bit for bit."""
import numpy as np
import pytest

from mmnorm_b200 import scenes
from test_forward_gpu import TOL_MIXED, run_ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 4096, 32767, 32768, 32769])
@pytest.mark.parametrize("special", [False, True])
def test_small_normals_bits(cuda_dev, n, special):
    import torch
    from mmnorm_b200 import ops
    g = torch.Generator(device=cuda_dev).manual_seed(n)
    image = torch.randn(n, dtype=torch.complex64, device=cuda_dev, generator=g)
    vote = torch.randn((3, n), dtype=torch.complex64, device=cuda_dev, generator=g)
    if special:
        image[:: max(1, n // 3)] = 0
        image[n // 2] = complex("nan")
    a = ops.surface_normals(image, vote, 0.3, want_raw=True)
    b = ops.surface_normals_from_max(image, vote, ops.image_max_abs(image), 0.3, want_raw=True)
    assert a[1].dtype == torch.bool and torch.equal(a[1], b[1])
    for x, y in ((a[0], b[0]), (a[2], b[2])):
        assert torch.equal(x.view(torch.int32), y.view(torch.int32))


@pytest.mark.parametrize("n_vox,n_ap", [(1, 3), (4, 9), (9, 33), (16, 17)])
def test_few_tiles_many_splits(cuda_dev, oracle, n_vox, n_ap):
    sc = scenes.sphere_scene(seed=n_ap, n_ap=n_ap, nf=64, n_vox=n_vox, n_pts=12)
    I, W = run_ops(cuda_dev, sc, "mixed")
    I2, W2 = run_ops(cuda_dev, sc, "mixed")
    assert np.array_equal(I, I2) and np.array_equal(W, W2)
    Io, Wo = oracle.full(sc.voxel_centres(), sc.antenna_locs, np.zeros((1, 3)), sc.meas,
                         sc.wavelength, sc.slope)
    assert oracle.rel_l2(I, Io) < TOL_MIXED and oracle.rel_l2(W, Wo) < TOL_MIXED
