"""The tile-local kernels are no further from 64 bits than the tap runs per (voxel, antenna) that
they replaced: root mean squares of the relative L2 errors over eight scenes (sums over 256
antennas; 8, 10, 12 and 16 nodes) against the FP64 oracle.  The bounds are the replaced kernels'
own errors on these scenes, and 3 % for the spread of such a mean."""
import numpy as np
import pytest

from test_local_polynomials_gpu import _scene
from test_forward_gpu import _t

pytestmark = pytest.mark.gpu

# image, vote, measurement gradient, position gradient of the replaced kernels
REPLACED = (1.752e-7, 1.758e-7, 1.594e-7, 2.047e-7)


def errors(dev, oracle):
    from mmnorm_b200 import ops
    out = []
    rxo = np.zeros((1, 3), np.float32)
    for seed, (spacing, nf) in enumerate([(0.001, 64), (0.002, 77), (0.003, 100), (0.004, 128),
                                          (0.005, 60), (0.006, 90), (0.008, 110), (0.011, 70)]):
        sc = _scene((20, 21, 23), 256, nf, spacing, 500 + seed)
        rng = np.random.default_rng(seed)
        V = sc.num_voxels
        c = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
        gI, gW = c(V), c(3, V)
        args = [_t(a, dev) for a in (sc.x_locs, sc.y_locs, sc.z_locs, sc.antenna_locs, rxo,
                                     sc.meas)] + [sc.wavelength, sc.slope]
        I, W = ops.backproject(*args, mode="nufft")
        gm, gp = ops.backproject_backward(*args, _t(gI, dev), _t(gW, dev))
        geo = (sc.voxel_centres(), sc.antenna_locs, rxo, sc.meas, sc.wavelength, sc.slope)
        Io, Wo = oracle.full(*geo)
        gm_o, gp_o = oracle.full_backward(*geo, gI.astype(np.complex128),
                                          gW.T.astype(np.complex128))
        n = lambda a, dt=np.complex128: a.cpu().numpy().astype(dt)
        out.append([oracle.rel_l2(n(I).ravel(), Io), oracle.rel_l2(n(W).reshape(3, -1).T, Wo),
                    oracle.rel_l2(n(gm), gm_o), oracle.rel_l2(n(gp, np.float64), gp_o)])
    return np.sqrt(np.mean(np.square(out), axis=0))


def test_no_further_from_64_bits_than_tap_runs(cuda_dev, oracle):
    err = errors(cuda_dev, oracle)
    assert np.all(err <= 1.03 * np.array(REPLACED)), err
