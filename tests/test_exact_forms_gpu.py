"""The exact interpolated form's square root and phasor against sqrtf and the FP64 cos and sin they
stand for, input by input: every float as a squared leg (all mantissas and exponents, zero,
subnormals, infinities, NaN, negative ones, both ends of the range that the short form takes), and
every float of three stretches as a path.  Equality of bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _counts(dev, first, count, wavelength):
    import torch
    from mmnorm_b200 import _lib
    from mmnorm_b200.ops import _stream, _vp
    out = torch.zeros(3, dtype=torch.int64, device=dev)
    _lib.check(_lib.load().mmn_interp_exact_probe(first, count, wavelength, _vp(out),
                                                  _stream(dev)), "mmn_interp_exact_probe")
    return out.tolist()


def _bits(x):
    return int(np.float32(x).view(np.uint32))


def test_square_root_of_every_float(cuda_dev):
    assert _counts(cuda_dev, 0, 1 << 32, 0.0)[0] == 0


@pytest.mark.parametrize("lo,hi,wavelength", [
    (2.0 ** -12, 0.25, 2.99792458e8 / 77e9), (0.25, 8.0, 2.99792458e8 / 77e9),
    (8.0, 600.0, 2.99792458e8 / 81e9), (0.25, 4.0, 2.99792458e8 / 60e9), (1.0, 64.0, 0.0125)])
def test_phasor_of_every_path(cuda_dev, lo, hi, wavelength):
    n = _bits(hi) - _bits(lo)
    _, bad, library = _counts(cuda_dev, _bits(lo), n, float(np.float32(wavelength)))
    assert bad == 0
    # undecided when a rounding boundary lies in the bounds' width: 2 delta / ulp of the smaller
    # component, delta = 2.5e-15 turns + 1.5e-13 (a few in 10^4 at ordinary paths)
    turns = hi / wavelength
    assert library < n * (1e-3 + 40 * 2.5e-15 * turns * 2 ** 24)
