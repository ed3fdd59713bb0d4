"""Interpolated mode, exact form: the kernels' bits against a numpy restatement of the
reference's arithmetic (FP32 legs, path and range bin, FP64 phase, cos and sin rounded to FP32,
FP32 sums in antenna order, each product and sum contracted as the reference kernel's), at the
sizes where the packed kernels can go wrong: odd voxel counts (two voxels a thread), one
antenna, antenna chunks of 256 with a remainder, paths beyond the measured range, paths on a
bin's edge, several receivers, the TI offset.  Equality of bits: no tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

f32, ld = np.float32, np.longdouble


def _fma(a, b, c):
    return (a.astype(ld) * ld(1) * b + c).astype(f32)


def _terms(vox, tx, off, meas, fsp, lam, ti):
    """(re, im, valid) float32 of one antenna for every voxel."""
    d = [(vox[:, k] - tx[k]).astype(f32) for k in range(3)]
    b = [(d[k] - off[k]).astype(f32) for k in range(3)]
    leg = [np.sqrt(_fma(e[2], e[2], _fma(e[0], e[0], (e[1] * e[1]).astype(f32)))) for e in (d, b)]
    path = (leg[0] + leg[1]).astype(f32)
    if ti:
        path = (path.astype(np.float64) + 0.15).astype(f32)
    valid = ~(path > f32(fsp) * f32(len(meas)))
    q = (path / f32(fsp)).astype(f32) / f32(2)
    m = meas[np.where(valid, np.floor(q), 0).astype(np.int64)]
    t = (-2 * np.pi * path.astype(np.float64)) / np.float64(f32(lam))
    c, s = np.cos(t.astype(ld)).astype(f32), np.sin(t.astype(ld)).astype(f32)
    re = _fma(m.real, c, -(m.imag * s).astype(f32))
    im = _fma(m.imag, c, (m.real * s).astype(f32))
    return re, im, valid


def _restated(x, y, z, ant, rxo, meas, fsp, lam, ti, image=None):
    vox = np.stack(np.meshgrid(x, y, z, indexing="ij"), -1).reshape(-1, 3).astype(f32)
    acc = np.zeros((8, len(vox)), f32)
    nrm = np.zeros((3, len(vox)), f32)
    if image is not None:
        ir, ii = image.real.ravel(), image.imag.ravel()
        mag = np.sqrt(_fma(ir, ir, (ii * ii).astype(f32)))
    for i, tx in enumerate(ant):
        off = rxo[i % len(rxo)]
        re, im, ok = _terms(vox, tx, off, meas[i], fsp, lam, ti)
        add = lambda a, v: np.where(ok, v, a)
        acc[0], acc[1] = add(acc[0], acc[0] + re), add(acc[1], acc[1] + im)
        if image is not None:
            w = (_fma(re, ir, (im * ii).astype(f32)) / mag).astype(f32)
        for k in range(3):
            e = (f32(tx[k] + off[k] / f32(2)) - vox[:, k]).astype(f32)
            acc[2 + 2 * k] = add(acc[2 + 2 * k], _fma(re, e, acc[2 + 2 * k]))
            acc[3 + 2 * k] = add(acc[3 + 2 * k], _fma(im, e, acc[3 + 2 * k]))
            if image is not None:
                nrm[k] = add(nrm[k], _fma(e, w, nrm[k]))
    return acc, nrm


@pytest.mark.parametrize("shape,ants,rx,ti,bins,far", [
    ((1, 1, 1), 1, 1, False, 64, False),
    ((7, 5, 3), 1, 3, True, 512, False),
    ((9, 8, 15), 13, 1, False, 4096, False),
    ((8, 8, 8), 257, 4, True, 256, False),
    ((5, 16, 13), 300, 1, True, 1024, True),
    ((16, 11, 3), 24, 4, False, 2048, True),
    ((3, 5, 9), 20, 4, True, 512, False),    # columns of an odd length in pairs along z
    ((4, 1, 64), 70, 1, True, 512, True),
])
def test_bits(cuda_dev, shape, ants, rx, ti, bins, far):
    import torch
    from mmnorm_b200 import ops, py_sn_est_gpu
    rng = np.random.default_rng(ants + bins)
    x, y, z = (f32(c) + f32(0.004) * np.arange(n, dtype=f32)
               for n, c in zip(shape, (-0.02, 0.01, 0.4)))
    tx = (0.1 * rng.uniform(-1, 1, (-(-ants // rx), 3)) * [1, 1, 0.2]).astype(f32)
    ant = np.repeat(tx, rx, axis=0)[:ants]
    rxo = np.zeros((1, 3), f32) if rx == 1 else rng.uniform(-0.01, 0.01, (rx, 3)).astype(f32)
    meas = (rng.standard_normal((ants, bins)) +
            1j * rng.standard_normal((ants, bins))).astype(np.complex64)
    lam, slope = 2.99792458e8 / 77e9, 4e9 / 99
    # `far`: the measured range ends inside the grid, at a path that is a whole bin
    fsp = float(f32((0.9 + 0.15 * ti) / bins if far else 3.0 / bins))
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=cuda_dev)
    image, vote = ops.backproject(t(x), t(y), t(z), t(ant), t(rxo), t(meas), lam, slope,
                                  mode="interp", fft_spacing=fsp, is_ti_radar=ti)
    got = np.concatenate([np.stack([v.real.ravel(), v.imag.ravel()]) for v in
                          [image.cpu().numpy()] + list(vote.cpu().numpy())])
    ref, _ = _restated(x, y, z, ant, rxo, meas, fsp, lam, ti)
    assert np.array_equal(got, ref)
    # the normal pass, over every voxel with |I| > 0 of the image just made
    if ants % rx:
        return
    img = image.cpu().numpy()
    data = meas.reshape(ants // rx, rx, bins).transpose(0, 2, 1)
    bandwidth, samples = 4e9, 100
    fsp_n = float(f32(3e8 / (2 * bandwidth) * samples / bins))
    raw = py_sn_est_gpu.sn_est_cuda(img, x, y, z, tx, data, rxo, slope, lam, bandwidth, samples,
                                    use_4_rx=True, is_ti_radar=ti, initial_filter_percent=0.0)
    _, nrm = _restated(x, y, z, ant, rxo, meas, fsp_n, lam, ti, image=img)
    ok = np.abs(img).ravel() > 0
    assert np.array_equal(raw.reshape(-1, 3)[ok].astype(f32), nrm.T[ok])
