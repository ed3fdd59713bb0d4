"""The default mixed variant's block phases: exact modular steps of 64 samples whatever the phase
step per sample, up to 2^19 turns of it (here 1e4 and 1e5: a block's 64 steps pass 2^19 turns),
over rows of two and three blocks, partial ones among them, and rows of over 1024 samples; single
and batched.

Tolerance 2e-5 relative L2 against the FP64 oracle, as for the mixed form at ordinary slopes; the
range's FP64 Newton step (1.5e-13 relative) adds up to 6e-6 rad at 6.5e6 turns."""
import numpy as np
import pytest

from test_forward_gpu import TOL_MIXED, _t, run_ops, small_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nf,turns", [(65, 1e4), (130, 1e4), (100, 3e4), (65, 1e5), (1100, 0.4)])
@pytest.mark.parametrize("batched", [False, True])
def test_wide_steps(cuda_dev, oracle, nf, turns, batched):
    from mmnorm_b200 import ops
    sc = small_scene(seed=9, n_ap=6, nf=nf, n_vox=6)
    mid = np.array([a.mean() for a in (sc.x_locs, sc.y_locs, sc.z_locs)])
    d = 2 * np.linalg.norm(mid - sc.antenna_locs.mean(0))
    sc.f_hi = sc.f_lo + (nf - 1) * turns * 2.99792458e8 / d
    Io, Wo = oracle.full(sc.voxel_centres(), sc.antenna_locs, np.zeros((1, 3)), sc.meas,
                         sc.wavelength, sc.slope)
    if batched:
        t = lambda a: _t(a, cuda_dev)
        plan = ops.BatchPlan([dict(
            x_locs=t(sc.x_locs), y_locs=t(sc.y_locs), z_locs=t(sc.z_locs),
            antenna_locs=t(sc.antenna_locs), rx_offsets=t(np.zeros((1, 3), np.float32)),
            meas=t(sc.meas), wavelength=sc.wavelength, slope=sc.slope)])
        plan.run()
        I, W = (v.cpu().numpy() for v in plan.results()[0])
        I, W = I.ravel(), W.reshape(3, -1).T
    else:
        I, W = run_ops(cuda_dev, sc)
    assert oracle.rel_l2(I, Io) < TOL_MIXED and oracle.rel_l2(W, Wo) < TOL_MIXED
