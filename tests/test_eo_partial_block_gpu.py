"""The default mixed variant's last partial block (even / odd second-order chains at the
block's own length): every remainder class -- one sample, odd counts (the sample above is a
padded zero), rows shorter than a block, a remainder of 32 in unpadded rows -- and the warps
that fall back to first-order sums because cos 2 phi is too near 1 (short ranges).

Tolerance 3e-6 relative L2 against the FP64 oracle: the form's documented 3.4e-6 is at 256
samples on a defocused scene; these sums are of at most 130 samples and few antennas (FP32
chains of 32 steps, anchors of 4e-7)."""
import numpy as np
import pytest

from mmnorm_b200 import scenes
from test_forward_gpu import run_ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nf", [1, 2, 3, 31, 32, 33, 63, 65, 77, 96, 127, 130])
@pytest.mark.parametrize("near", [False, True])
def test_partial_blocks(cuda_dev, oracle, nf, near):
    sc = scenes.sphere_scene(seed=nf, n_ap=5, nf=64, n_vox=7, n_pts=9)
    rng = np.random.default_rng(nf)
    meas = (rng.standard_normal((25, nf)) + 1j * rng.standard_normal((25, nf))).astype(np.complex64)
    if near:   # 2 phi below the form's limit for every pair
        sc.z_locs = (sc.z_locs - sc.z_locs.min() + 0.02).astype(np.float32)
    I, W = run_ops(cuda_dev, sc, "mixed", meas=meas)
    Io, Wo = oracle.full(sc.voxel_centres(), sc.antenna_locs, np.zeros((1, 3)), meas,
                         sc.wavelength, sc.slope)
    assert oracle.rel_l2(I, Io) < 3e-6 and oracle.rel_l2(W, Wo) < 3e-6
