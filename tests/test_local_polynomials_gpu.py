"""The tile-local polynomial kernels of the interpolation form at the sizes where they can go
wrong: tile remainders on every axis, antenna-chunk remainders (chunks of 32), each node count
(set by the voxel pitch) and the tap-run path of a box too wide for any of them, unordered
coordinate arrays, several receivers.

Tolerance 2e-6 relative L2 against the FP64 oracle: anchor polynomials 1.7e-7 at most, node
interpolation 1.2e-7 at the band's edge, FP32 Horner with coefficient sums up to e^2.6 = 13
(8e-7 at worst), the tap fit and the FP32 sums of a few 1e-8.  The position gradient adds FP32
directions and a sum of terms of either sign over the voxels: 1e-5."""
import numpy as np
import pytest

from mmnorm_b200 import scenes
from test_forward_gpu import _t, run_ops

pytestmark = pytest.mark.gpu

TOL = 2e-6


def _scene(shape, ants, nf, spacing, seed):
    rng = np.random.default_rng(seed)
    sc = scenes.sphere_scene(seed=seed, n_ap=2, nf=nf, n_vox=4, n_pts=4)
    axes = [(c + spacing * (np.arange(n) - (n - 1) / 2.0)).astype(np.float32)
            for n, c in zip(shape, (0.01, -0.02, 0.6))]
    sc.x_locs, sc.y_locs, sc.z_locs = axes
    sc.antenna_locs = (0.15 * rng.uniform(-1, 1, (ants, 3)) * [1, 1, 0.1]).astype(np.float32)
    sc.meas = (rng.standard_normal((ants, nf)) +
               1j * rng.standard_normal((ants, nf))).astype(np.complex64)
    return sc


SHAPES = pytest.mark.parametrize("shape,ants,spacing", [
    ((1, 1, 1), 1, 0.003),
    ((9, 8, 7), 31, 0.0005),    # 8 nodes
    ((5, 17, 9), 33, 0.004),
    ((8, 8, 16), 64, 0.0045),   # 10 nodes
    ((7, 3, 33), 65, 0.006),    # 12 nodes
    ((10, 9, 10), 40, 0.012),   # 16 nodes
    ((9, 9, 9), 37, 0.022),     # 24 nodes
    ((8, 9, 8), 33, 0.05),      # tap runs
])


@SHAPES
@pytest.mark.parametrize("rx", [1, 3])
def test_forward_edges(cuda_dev, oracle, shape, ants, spacing, rx):
    sc = _scene(shape, ants, 50, spacing, 100 + ants)
    rxo = np.array([[0, 0, 0], [0.004, -0.01, 0], [0.02, 0.003, 0.001]], np.float32)[-rx:]
    I, W = run_ops(cuda_dev, sc, "nufft", rxo=rxo, ti=rx == 3)
    Io, Wo = oracle.full(sc.voxel_centres(), sc.antenna_locs, rxo, sc.meas, sc.wavelength,
                         sc.slope, is_ti=rx == 3)
    assert oracle.rel_l2(I, Io) < TOL and oracle.rel_l2(W, Wo) < TOL


@SHAPES
@pytest.mark.parametrize("rx,vote", [(1, True), (1, False), (3, True), (3, False)])
def test_gradient_edges(cuda_dev, oracle, shape, ants, spacing, rx, vote):
    from mmnorm_b200 import ops
    sc = _scene(shape, ants, 50, spacing, 200 + ants)
    rng = np.random.default_rng(ants)
    rxo = np.array([[0, 0, 0], [0.004, -0.01, 0], [0.02, 0.003, 0.001]], np.float32)[-rx:]
    V = sc.num_voxels
    gI = (rng.standard_normal(V) + 1j * rng.standard_normal(V)).astype(np.complex64)
    gW = (rng.standard_normal((3, V)) + 1j * rng.standard_normal((3, V))).astype(np.complex64)
    gW = gW if vote else np.zeros_like(gW)
    args = [_t(a, cuda_dev) for a in (sc.x_locs, sc.y_locs, sc.z_locs, sc.antenna_locs, rxo,
                                      sc.meas)]
    gm, gp = ops.backproject_backward(*args, sc.wavelength, sc.slope, _t(gI, cuda_dev),
                                      _t(gW, cuda_dev) if vote else None, is_ti_radar=rx == 3)
    gm_o, gp_o = oracle.full_backward(sc.voxel_centres(), sc.antenna_locs, rxo, sc.meas,
                                   sc.wavelength, sc.slope, gI.astype(np.complex128),
                                   gW.T.astype(np.complex128), is_ti=rx == 3)
    assert oracle.rel_l2(gp.cpu().numpy().astype(np.float64), gp_o) < 1e-5
    assert oracle.rel_l2(gm.cpu().numpy().astype(np.complex128), gm_o) < TOL


def test_forward_unordered_axes(cuda_dev, oracle):
    sc = _scene((11, 10, 13), 40, 33, 0.003, 7)
    rng = np.random.default_rng(8)
    sc.x_locs, sc.y_locs, sc.z_locs = (np.ascontiguousarray(rng.permutation(a))
                                       for a in (sc.x_locs, sc.y_locs[::-1], sc.z_locs))
    I, W = run_ops(cuda_dev, sc, "nufft")
    Io, Wo = oracle.full(sc.voxel_centres(), sc.antenna_locs, np.zeros((1, 3)), sc.meas,
                         sc.wavelength, sc.slope)
    assert oracle.rel_l2(I, Io) < TOL and oracle.rel_l2(W, Wo) < TOL
