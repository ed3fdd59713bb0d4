"""The tile-local kernels where their voxel runs lie along x or y: planes, slabs, lines and bars
with the short axes at either end, box remainders along the runs, several receivers.  Tolerances of
the same kernels at ordinary shapes (test_local_polynomials_gpu)."""
import numpy as np
import pytest

from test_local_limits_gpu import _gradients
from test_local_polynomials_gpu import TOL, _scene
from test_forward_gpu import run_ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,spacing", [
    ((41, 37, 1), 0.002), ((43, 1, 39), 0.002), ((1, 47, 35), 0.002),
    ((35, 31, 2), 0.003), ((30, 37, 3), 0.003), ((2, 29, 41), 0.003),
    ((701, 1, 1), 0.0003), ((1, 701, 1), 0.0003), ((1, 1, 701), 0.0003),
    ((333, 3, 2), 0.0005), ((2, 401, 3), 0.0005), ((150, 1, 1), 0.01),
    ((33, 1, 1), 0.002), ((1, 30, 1), 0.002), ((5, 5, 1), 0.002),
])
@pytest.mark.parametrize("rx", [1, 3])
def test_runs_along_other_axes(cuda_dev, oracle, shape, spacing, rx):
    sc = _scene(shape, 35, 50, spacing, 700 + sum(shape))
    rxo = np.array([[0, 0, 0], [0.004, -0.01, 0], [0.02, 0.003, 0.001]], np.float32)[-rx:]
    I, W = run_ops(cuda_dev, sc, "nufft", rxo=rxo, ti=rx == 3)
    Io, Wo = oracle.full(sc.voxel_centres(), sc.antenna_locs, rxo, sc.meas, sc.wavelength,
                         sc.slope, is_ti=rx == 3)
    assert oracle.rel_l2(I, Io) < TOL and oracle.rel_l2(W, Wo) < TOL
    runs, (gm_o, gp_o) = _gradients(cuda_dev, oracle, sc, rxo, rx == 3, rx)
    assert oracle.rel_l2(runs[0][0].astype(np.complex128), gm_o) < TOL
    assert oracle.rel_l2(runs[0][1].astype(np.float64), gp_o) < 1e-5
