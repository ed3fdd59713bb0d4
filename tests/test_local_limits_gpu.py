"""The tile-local kernels of the interpolation form at the limits of their approximations, against
the FP64 oracle: short antenna grids (32 to 64 cells) on which a box's cells wrap past the row's
end, with boxes narrow enough for the nodes and too wide for them.

Tolerance 2e-6 relative L2, as for these kernels at ordinary sizes (test_local_polynomials_gpu)."""
import numpy as np
import pytest

from test_local_polynomials_gpu import TOL, _scene
from test_forward_gpu import _t, run_ops

pytestmark = pytest.mark.gpu


def _gradients(dev, oracle, sc, rxo, ti, seed):
    """(measurement, position) gradients twice, and the oracle's."""
    from mmnorm_b200 import ops
    rng = np.random.default_rng(seed)
    V = sc.num_voxels
    gI = (rng.standard_normal(V) + 1j * rng.standard_normal(V)).astype(np.complex64)
    gW = (rng.standard_normal((3, V)) + 1j * rng.standard_normal((3, V))).astype(np.complex64)
    args = [_t(a, dev) for a in (sc.x_locs, sc.y_locs, sc.z_locs, sc.antenna_locs, rxo, sc.meas)]
    runs = [[g.cpu().numpy() for g in ops.backproject_backward(
        *args, sc.wavelength, sc.slope, _t(gI, dev), _t(gW, dev), is_ti_radar=ti)]
        for _ in range(2)]
    ref = oracle.full_backward(sc.voxel_centres(), sc.antenna_locs, rxo, sc.meas, sc.wavelength,
                               sc.slope, gI.astype(np.complex128), gW.T.astype(np.complex128),
                               is_ti=ti)
    return runs, ref


@pytest.mark.parametrize("nf", [16, 21, 32])
@pytest.mark.parametrize("shape,spacing", [((9, 8, 7), 0.004), ((10, 9, 10), 0.012),
                                           ((8, 9, 8), 0.05), ((3, 2, 13), 0.11)])
def test_short_grids_that_wrap(cuda_dev, oracle, nf, shape, spacing):
    sc = _scene(shape, 37, nf, spacing, 300 + nf)
    # the grid's period of c / slope ends inside the scene (round-trip ranges near 1.2 m)
    sc.f_hi = sc.f_lo + (nf - 1) * 2.99792458e8 / 1.2
    runs, (gm_o, _) = _gradients(cuda_dev, oracle, sc, np.zeros((1, 3), np.float32), False, nf)
    assert np.array_equal(runs[0][0], runs[1][0])
    assert oracle.rel_l2(runs[0][0].astype(np.complex128), gm_o) < TOL


@pytest.mark.parametrize("wavelength", [2.1e-6, 0.9e-6])
@pytest.mark.parametrize("rx", [1, 3])
def test_anchors_beyond_the_fixed_point_range(cuda_dev, oracle, wavelength, rx):
    """Ranges of 5.7e5 and 1.3e6 wavelengths, past the 2^18 turns that the 2^-32-turn anchors
    hold.  The ranges' FP64 Newton step (1.5e-13 relative) is up to 1.3e-6 rad of anchor phase
    here: 3e-6 for the sums and, with the 1e-5 of the position gradient's FP32 directions, 1.2e-5
    for that."""
    sc = _scene((6, 7, 9), 35, 40, 0.004, 400)
    sc.f_lo, sc.f_hi = 2.99792458e8 / wavelength, 2.99792458e8 / wavelength + 4e9
    rxo = np.array([[0, 0, 0], [0.004, -0.01, 0], [0.02, 0.003, 0.001]], np.float32)[-rx:]
    I, W = run_ops(cuda_dev, sc, "nufft", rxo=rxo, ti=rx == 3)
    Io, Wo = oracle.full(sc.voxel_centres(), sc.antenna_locs, rxo, sc.meas, sc.wavelength,
                         sc.slope, is_ti=rx == 3)
    assert oracle.rel_l2(I, Io) < 3e-6 and oracle.rel_l2(W, Wo) < 3e-6
    runs, (gm_o, gp_o) = _gradients(cuda_dev, oracle, sc, rxo, rx == 3, rx)
    assert oracle.rel_l2(runs[0][0].astype(np.complex128), gm_o) < 3e-6
    assert oracle.rel_l2(runs[0][1].astype(np.float64), gp_o) < 1.2e-5


@pytest.mark.parametrize("ants,nf,spacing", [(1, 40, 0.3), (3, 300, 0.25), (4, 17, 0.3),
                                             (5, 300, 0.004), (9, 700, 0.4)])
def test_few_antennas_with_wide_windows(cuda_dev, oracle, ants, nf, spacing):
    """Grid windows of up to all 2 F cells, spread over several warps an antenna.  Ranges of some
    metres: FP32 anchors and tap offsets as at ordinary sizes (2e-6)."""
    sc = _scene((6, 5, 9), ants, nf, spacing, 600 + nf)
    I, W = run_ops(cuda_dev, sc, "nufft")
    Io, Wo = oracle.full(sc.voxel_centres(), sc.antenna_locs, np.zeros((1, 3)), sc.meas,
                         sc.wavelength, sc.slope)
    assert oracle.rel_l2(I, Io) < TOL and oracle.rel_l2(W, Wo) < TOL
    runs, (_, gp_o) = _gradients(cuda_dev, oracle, sc, np.zeros((1, 3), np.float32), False, nf)
    assert oracle.rel_l2(runs[0][1].astype(np.float64), gp_o) < 1e-5


@pytest.mark.parametrize("spacing,nf", [(0.004, 50), (0.008, 64), (0.016, 33)])
@pytest.mark.parametrize("rx", [1, 3])
def test_chunks_of_narrow_and_wide_boxes(cuda_dev, oracle, spacing, nf, rx):
    """Columns of voxels seen by antennas from the side, whose range over a box varies little, and
    from below, where it takes tap runs: both in the same chunks of 32."""
    sc = _scene((3, 4, 70), 75, nf, spacing, 800 + nf)
    sc.antenna_locs[::2] += np.array([0.9, 0.2, 0.6], np.float32)
    rxo = np.array([[0, 0, 0], [0.004, -0.01, 0], [0.02, 0.003, 0.001]], np.float32)[-rx:]
    I, W = run_ops(cuda_dev, sc, "nufft", rxo=rxo)
    Io, Wo = oracle.full(sc.voxel_centres(), sc.antenna_locs, rxo, sc.meas, sc.wavelength,
                         sc.slope)
    assert oracle.rel_l2(I, Io) < TOL and oracle.rel_l2(W, Wo) < TOL
    runs, (gm_o, gp_o) = _gradients(cuda_dev, oracle, sc, rxo, False, rx)
    assert oracle.rel_l2(runs[0][0].astype(np.complex128), gm_o) < TOL
    assert oracle.rel_l2(runs[0][1].astype(np.float64), gp_o) < 1e-5


@pytest.mark.parametrize("spacing", [0.006, 0.011, 0.016, 0.021, 0.035])
def test_measurement_boxes_in_parts(cuda_dev, oracle, spacing):
    """Boxes of 2048 voxels that are narrow enough, too wide as a whole, in halves, and down to
    128 voxels, whose parts then go by moments or voxel by voxel."""
    sc = _scene((48, 50, 54), 75, 16, spacing, 900)
    sc.f_hi = sc.f_lo + 4e9
    runs, (gm_o, _) = _gradients(cuda_dev, oracle, sc, np.zeros((1, 3), np.float32), False, 1)
    assert np.array_equal(runs[0][0], runs[1][0])
    assert oracle.rel_l2(runs[0][0].astype(np.complex128), gm_o) < TOL
