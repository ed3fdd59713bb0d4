"""Voxel boxes of thin grids: the backward's workspace, most of it per box and slot, does not depend
on which axis of a plane, a slab or a line is the short one (boxes that always ran along z took up to
four times the slots of a plane in z, and 32 times those of a line).  CPU only: no call launches."""
import ctypes
import itertools

import pytest


def _bytes(shape, antennas=64, samples=40):
    from mmnorm_b200 import _lib
    p = _lib.MmnProblem()
    p.num_x, p.num_y, p.num_z = shape
    p.num_antennas, p.num_rx, p.num_samples = antennas, 1, samples
    p.wavelength, p.slope, p.fft_spacing = 0.004, 1e8, 0.01
    for name in ("x_locs", "y_locs", "z_locs", "antenna_locs", "rx_offsets", "meas"):
        setattr(p, name, 4096)   # looked at, never read: no launch
    return _lib.load().mmn_backward_workspace_bytes(ctypes.byref(p))


@pytest.mark.parametrize("shape", [(1, 300, 280), (2, 250, 200), (3, 200, 190), (1, 1, 20000),
                                   (2, 3, 9000)])
def test_short_axis_anywhere(shape):
    sizes = [_bytes(s) for s in set(itertools.permutations(shape))]
    assert min(sizes) > 0
    assert max(sizes) < 1.34 * min(sizes), sizes   # up to a quarter of the slots may be idle


@pytest.mark.parametrize("shape", [(1, 1, 20000), (20000, 1, 1), (300, 280, 1), (1, 1, 7),
                                   (64, 64, 64)])
def test_slots_are_used(shape):
    """Against the bytes of the records alone: 160 a run of four voxels, most slots in use."""
    n = shape[0] * shape[1] * shape[2]
    base = _bytes((1, 1, 1))
    assert _bytes(shape) - base < 2.2 * (n * (160 / 4 + 48)) + 4e6
