"""The work a user of this package has it do, as a list of timed cases.

Each case is a dict of plain values.  ``listed()`` holds the fixed ones, ``draw(rng)`` makes
one more from the same ranges, ``prepare`` builds what a program holds before the call (on
the GPU, or on the host where the path takes host arrays), ``run`` makes one pass through
the public entry points, ``work`` states what the path cannot do without and ``exact`` the
result in 64 bits.  Scenes are point scatterers on a sphere or cylinder shell seen by a
planar 77-81 GHz aperture, with noise, as in the package's own scene generators.
"""
import math

import numpy as np
import torch

C = 2.99792458e8
F_LO, F_HI = 77e9, 81e9
PI2 = 2.0 * math.pi


def listed():
    return [
        # the smallest useful call: one object in a coarse box, image and masked normals;
        # launches and host work decide
        dict(name="image_tiny", kind="image", mode="mixed", nx=16, ny=16, nz=16, ant=256, rx=1,
             freqs=64, ti=False, pos=False, normals=True),
        # the small planar workload of the benchmark: 48^3 voxels, 32 x 32 antennas, 64 samples
        dict(name="image_48", kind="image", mode="mixed", nx=48, ny=48, nz=48, ant=1024, rx=1,
             freqs=64, ti=False, pos=False, normals=True),
        # a TI radar with four receivers and a trajectory correction: ragged grid, odd antenna
        # and sample counts
        dict(name="image_ragged_4rx", kind="image", mode="mixed", nx=75, ny=61, nz=53, ant=1236,
             rx=4, freqs=100, ti=True, pos=True, normals=False),
        # the large grid of the benchmark with a quarter of its aperture: the arithmetic decides
        dict(name="image_128", kind="image", mode="mixed", nx=128, ny=128, nz=128, ant=4096,
             rx=1, freqs=256, ti=False, pos=False, normals=False),
        # the same sums from per-antenna oversampled spectra
        dict(name="nufft_96", kind="image", mode="nufft", nx=96, ny=96, nz=96, ant=4096, rx=1,
             freqs=200, ti=False, pos=False, normals=False),
        # the interpolated mode (the reference's shipped default): range bins of a 4096-point
        # FFT, four receivers
        dict(name="interp_exact_4rx", kind="interp", nx=90, ny=100, nz=70, ant=4096, rx=4,
             freqs=256, bins=4096, ti=True),
        # a whole imaging + normals call from raw samples: range FFT, image, normals, in the
        # interpolated mode's fast form
        dict(name="stage1_fast", kind="stage1", nx=80, ny=96, nz=64, ant=1000, rx=4, freqs=256,
             ti=True),
        # one calibration step: image and vote forward, gradients to measurements and antenna
        # positions (the benchmark's adjoint workload)
        dict(name="train_64", kind="train", nx=64, ny=64, nz=64, ant=4096, freqs=128),
        # an image-only loss on a ragged grid: both gradients, no vote term
        dict(name="adjoint_image_odd", kind="adjoint", nx=41, ny=53, nz=37, ant=1111, freqs=77),
        # many objects of uneven sizes in one plan, re-run for each new capture
        dict(name="batch_uneven", kind="batch", grids="32,48,64,32,96,48,33,40",
             ants="32,64,32,64,32,48,32,33", freqs="64,200,256,77,128,100,90,250"),
        # the relative signed distance field of a masked normal field (host arrays in and out)
        dict(name="rsdf_cap", kind="rsdf", nx=100, ny=96, nz=72, spacing=0.0015),
        # channels simulated from an isosurface: the inner step of the offset search
        dict(name="iso_channels", kind="iso", nx=200, ny=220, nz=120, rays=1024, ant=10, sets=3,
             wavelengths=512),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["image", "image", "image", "nufft", "interp", "interp", "stage1", "train",
                       "adjoint", "batch", "rsdf", "iso"])
    g = lambda lo, hi: dict(nx=_log(rng, lo, hi), ny=_log(rng, lo, hi), nz=_log(rng, lo, hi))
    if kind in ("image", "nufft"):
        rx = rng.choice([1, 1, 4])
        c = dict(kind="image", mode="mixed" if kind == "image" else "nufft", **g(14, 128),
                 ant=rx * _log(rng, 200 // rx, 4096 // rx), rx=rx, freqs=_log(rng, 60, 256),
                 ti=rx == 4, pos=rng.random() < 0.3, normals=rng.random() < 0.5)
        return c
    if kind == "interp":
        rx = rng.choice([1, 4, 4])
        return dict(kind="interp", **g(16, 100), ant=rx * _log(rng, 200 // rx, 4096 // rx),
                    rx=rx, freqs=rng.choice([100, 128, 256]), bins=rng.choice([512, 2048, 4096]),
                    ti=rx == 4)
    if kind == "stage1":
        return dict(kind="stage1", **g(20, 100), ant=_log(rng, 60, 1000),
                    rx=rng.choice([1, 4]), freqs=rng.choice([100, 128, 256]),
                    ti=rng.random() < 0.5)
    if kind == "train":
        return dict(kind="train", **g(16, 64), ant=_log(rng, 256, 4096),
                    freqs=_log(rng, 60, 200))
    if kind == "adjoint":
        return dict(kind="adjoint", **g(16, 64), ant=_log(rng, 256, 4096),
                    freqs=_log(rng, 60, 200))
    if kind == "batch":
        n = rng.randint(3, 8)
        j = lambda lo, hi: ",".join(str(_log(rng, lo, hi)) for _ in range(n))
        return dict(kind="batch", grids=j(24, 72), ants=j(20, 64), freqs=j(60, 256))
    if kind == "rsdf":
        return dict(kind="rsdf", nx=rng.randint(50, 100), ny=rng.randint(50, 96),
                    nz=rng.randint(40, 72), spacing=0.0015)
    return dict(kind="iso", nx=rng.randint(100, 200), ny=rng.randint(100, 220),
                nz=rng.randint(80, 120), rays=rng.choice([256, 500, 1024]),
                ant=rng.randint(2, 10), sets=rng.randint(1, 3),
                wavelengths=rng.choice([64, 200, 512]))


# ------------------------------------------------------------------------------- inputs

def _f32(v):
    return float(np.float32(v))


def _axes(shape, spacing, centre, dev):
    out = []
    for n, c in zip(shape, centre):
        k = (torch.arange(n, dtype=torch.float64, device=dev) - (n - 1) / 2.0) * spacing + c
        out.append(k.to(torch.float32))
    return out


def _aperture(n, pitch, dev):
    """n positions of a raster about as wide as high in the plane z = 0."""
    w = max(1, int(round(math.sqrt(n))))
    i = torch.arange(n, device=dev)
    x, y = (i % w).double(), torch.div(i, w, rounding_mode="floor").double()
    p = torch.stack([(x - x.mean()) * pitch, (y - y.mean()) * pitch, torch.zeros_like(x)], dim=1)
    return p.to(torch.float32)


def _rx_offsets(rx, dev):
    o = torch.zeros((rx, 3), dtype=torch.float32, device=dev)
    o[:, 0] = 0.0019 * torch.arange(rx, device=dev) + (0.005 if rx > 1 else 0.0)
    return o


def _scatterers(gen, extent, centre, dev, n=160):
    v = torch.randn((n, 3), generator=gen, dtype=torch.float64, device=dev)
    v /= v.norm(dim=1, keepdim=True)
    rho = 0.3 + 0.7 * torch.rand(n, generator=gen, dtype=torch.float64, device=dev)
    return v * (0.33 * extent) + torch.tensor(centre, dtype=torch.float64, device=dev), rho


def _samples(gen, tx, rx_pos, pts, rho, freqs, ti):
    """Echoes complex64 [A, F] of the scatterers, with noise 20 dB below them."""
    dev = tx.device
    f = F_LO + torch.arange(freqs, dtype=torch.float64, device=dev) * (F_HI - F_LO) / (freqs - 1)
    out = torch.empty((tx.shape[0], freqs), dtype=torch.complex128, device=dev)
    step = max(1, (1 << 24) // (freqs * pts.shape[0]))
    for a in range(0, tx.shape[0], step):
        r1, r2 = torch.cdist(tx[a:a + step], pts), torch.cdist(rx_pos[a:a + step], pts)
        ph = (r1 + r2 + ti)[:, :, None] * (PI2 / C * f)
        out[a:a + step] = torch.einsum("ap,apf->af", (rho / (r1 * r2)).to(torch.complex128),
                                       torch.polar(torch.ones_like(ph), ph))
    s = math.sqrt(float((out.abs() ** 2).mean()) / 200.0)
    noise = torch.randn((tx.shape[0], freqs, 2), generator=gen, dtype=torch.float64, device=dev)
    return (out + s * torch.view_as_complex(noise)).to(torch.complex64)


def _scene(shape, ant, rx, freqs, ti, seed, spacing=None):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(1000003 * seed + 17)
    jit = (torch.rand(3, generator=gen, dtype=torch.float64, device=dev) - 0.5).cpu().numpy()
    centre = (0.01 * jit[0], 0.01 * jit[1], 0.42 + 0.04 * jit[2])
    spacing = spacing or 0.19 / max(shape)
    x, y, z = _axes(shape, spacing, centre, dev)
    tx = _aperture(-(-ant // rx), 0.003, dev).repeat_interleave(rx, dim=0)[:ant].contiguous()
    rxo = _rx_offsets(rx, dev)
    rx_pos = tx.double() + rxo.double()[torch.arange(ant, device=dev) % rx]
    pts, rho = _scatterers(gen, spacing * min(shape), centre, dev)
    off = 0.15 if ti else 0.0
    meas = _samples(gen, tx.double(), rx_pos, pts, rho, freqs, off)
    return dict(x=x, y=y, z=z, ant=tx, rxo=rxo, meas=meas, wavelength=_f32(C / F_LO),
                slope=_f32((F_HI - F_LO) / (freqs - 1)), ti=ti, gen=gen, centre=centre)


def _shape(c):
    return c["nx"], c["ny"], c["nz"]


def _complex_normal(gen, shape, dev):
    return torch.view_as_complex(torch.randn(tuple(shape) + (2,), generator=gen,
                                             dtype=torch.float32, device=dev))


def _fft_spacing(freqs, bins):
    return _f32(3e8 / (2 * (F_HI - F_LO)) * freqs / bins)


def prepare(case, seed):
    from mmnorm_b200 import isosurface, ops
    kind = case["kind"]
    if kind == "batch":
        objs = _batch_objects(case, seed)
        keys = ("x", "y", "z", "ant", "rxo", "meas")
        names = ("x_locs", "y_locs", "z_locs", "antenna_locs", "rx_offsets", "meas")
        plan = ops.BatchPlan([dict({n: o[k] for n, k in zip(names, keys)},
                                   wavelength=o["wavelength"], slope=o["slope"]) for o in objs])
        return dict(case=case, plan=plan)
    if kind == "rsdf":
        return dict(case=case, **_cap(case, seed))
    if kind == "iso":
        sdf, bbox, vs, wl, loc, dirs, taus = _shell(case, seed)
        scene = isosurface.make_scene(sdf, bbox, vs, wl, case["rays"], case["rays"], 80, 80, True,
                                      device=loc.device)
        return dict(case=case, scene=scene, taus=taus, loc=loc, dirs=dirs)
    s = _scene(_shape(case), case["ant"] * (case["rx"] if kind == "stage1" else 1),
               case.get("rx", 1), case["freqs"], case.get("ti", False), seed)
    dev = s["ant"].device
    if case.get("pos") or kind in ("train", "adjoint"):
        s["pos"] = 5e-4 * torch.randn(s["ant"].shape, generator=s["gen"], device=dev)
    if kind == "interp":
        s["meas"] = torch.fft.fft(s["meas"], n=case["bins"], dim=1).contiguous()
    if kind == "stage1":
        r = case["rx"]
        s["tx"] = s["ant"][::r].double().contiguous()
        s["raw"] = s["meas"].reshape(case["ant"], r, case["freqs"]).permute(0, 2, 1).contiguous()
    if kind in ("train", "adjoint"):
        V = _shape(case)
        s["g_image"] = _complex_normal(s["gen"], V, dev)
        s["g_vote"] = _complex_normal(s["gen"], (3,) + V, dev) if kind == "train" else None
        if kind == "train":
            s["meas"].requires_grad_(True)
            s["pos"].requires_grad_(True)
    del s["gen"]
    return dict(s, case=case)


def _batch_objects(case, seed):
    g, a, f = ([int(t) for t in case[k].split(",")] for k in ("grids", "ants", "freqs"))
    return [_scene((n, n, n), m * m, 1, nf, False, 64 * seed + o + 1, spacing=0.15 / n)
            for o, (n, m, nf) in enumerate(zip(g, a, f))]


def _cap(case, seed):
    """Normals of a spherical cap's shell (float64, NaN outside), slightly perturbed."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = _shape(case)
    dx = case["spacing"]
    ax = [(np.arange(n) - (n - 1) / 2.0) * dx + c
          for n, c in zip((nx, ny, nz), rng.uniform(-0.002, 0.002, 3))]
    X, Y, Z = np.meshgrid(*ax, indexing="ij", sparse=True)
    r = np.sqrt(X ** 2 + Y ** 2 + Z ** 2)
    r0 = 0.42 * dx * min(nx, ny, nz)
    shell = (np.abs(r - r0) < 0.009) & (Z > -0.4 * r0)
    n = np.full((nx, ny, nz, 3), np.nan)
    v = np.stack(np.broadcast_arrays(X, Y, Z), axis=-1)[shell] / r[shell][:, None]
    v = v + 0.05 * rng.standard_normal(v.shape)
    n[shell] = v / np.linalg.norm(v, axis=1)[:, None]
    return dict(normals=n, x=ax[0], y=ax[1], z=ax[2])


def _shell(case, seed):
    """A sphere's signed distances in a +-8 mm shell on a 1 mm grid, antennas above it."""
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed + 5)
    n, vs = _shape(case), 1e-3
    jit = 2e-3 * (torch.rand(3, generator=gen, device=dev) - 0.5).cpu().numpy()
    lo = [-(m - 1) / 2.0 * vs for m in n[:2]] + [0.40]
    ax = [lo[k] + vs * torch.arange(n[k], device=dev) for k in range(3)]
    cz = lo[2] + 0.5 * vs * (n[2] - 1)
    r = torch.sqrt((ax[0] - jit[0])[:, None, None] ** 2 + (ax[1] - jit[1])[None, :, None] ** 2 +
                   (ax[2] - cz - jit[2])[None, None, :] ** 2) - 0.035
    sdf = torch.where(r.abs() < 0.008, r, torch.full_like(r, -50.0))
    bbox = lo + [lo[k] + vs * (n[k] - 1) for k in range(3)]
    K = case["wavelengths"]
    wl = C / (77.5e9 + np.arange(K) * 3e9 / max(1, K - 1))
    loc = 0.06 * (torch.rand((case["ant"], 3), generator=gen, dtype=torch.float64,
                             device=dev) - 0.5)
    loc[:, 2] = 0.0
    dirs = torch.zeros((case["ant"], 3), dtype=torch.float32, device=dev)
    dirs[:, 2] = -1.0   # the view direction's convention: rays leave against it
    taus = -0.003 + 0.006 * torch.rand((case["sets"], 1), generator=gen, device=dev)
    return sdf[..., None], bbox, vs, wl, loc, dirs, taus


# --------------------------------------------------------------------------------- passes

def run(state):
    from mmnorm_b200 import isosurface, ops, rsdf, stage1
    s, c = state, state["case"]
    kind = c["kind"]
    if kind == "batch":
        s["plan"].run()
        return [list(p) for p in s["plan"].results()]
    if kind == "rsdf":
        field, labels, _, _ = rsdf.compute_rsdf(s["normals"], s["x"], s["y"], s["z"])
        return field, labels
    if kind == "iso":
        return isosurface.simulate_channels_batch(s["scene"], s["taus"], s["loc"], s["dirs"])
    if kind == "stage1":
        out = stage1.image_and_normals(
            s["x"], s["y"], s["z"], s["tx"], s["raw"], s["rxo"], s["slope"], s["wavelength"],
            F_HI - F_LO, c["freqs"], is_ti_radar=c["ti"], use_interpolated_processing=True,
            precision="fast")
        return out["sum_image"], out["normals"], out["mask"], out["center_locs"]
    geo = (s["x"], s["y"], s["z"], s["ant"], s["rxo"], s["meas"], s["wavelength"], s["slope"])
    if kind == "interp":
        return ops.backproject(*geo, mode="interp", is_ti_radar=c["ti"],
                               fft_spacing=_fft_spacing(c["freqs"], c["bins"]))
    if kind == "train":
        image, vote = ops.backproject_differentiable(*geo, pos_offsets=s["pos"], mode="nufft")
        gm, gp = torch.autograd.grad((image, vote), (s["meas"], s["pos"]),
                                     (s["g_image"], s["g_vote"]))
        return image.detach(), vote.detach(), gm, gp
    if kind == "adjoint":
        return ops.backproject_backward(*geo, s["g_image"], None, pos_offsets=s["pos"])
    image, vote = ops.backproject(*geo, mode=c["mode"], is_ti_radar=c["ti"],
                                  pos_offsets=s.get("pos"))
    if not c["normals"]:
        return image, vote
    normals, mask = ops.surface_normals(image, vote, 0.05)
    return image, vote, normals, mask


# ----------------------------------------------------------------- least bytes and operations

def _image_work(V, A, F, mode, cell=8):
    # the recurrence needs 4 multiply-adds (8 flops) per voxel, antenna and sample; the
    # interpolated sums 8 complex cells with real weights, a range, a phasor and the vote
    per = {"mixed": 8.0 * F, "nufft": 2.0 * 2 * 8 + 60.0, "interp": 60.0}[mode]
    return dict(bytes=float(V) * 32 + float(A) * (F * cell + 24), flops=float(V) * A * per)


def work(case):
    k = case["kind"]
    if k == "batch":
        g, a, f = ([int(t) for t in case[q].split(",")] for q in ("grids", "ants", "freqs"))
        parts = [_image_work(n ** 3, m * m, nf, "mixed") for n, m, nf in zip(g, a, f)]
        return {q: sum(p[q] for p in parts) for q in ("bytes", "flops")}
    V = float(case["nx"]) * case["ny"] * case["nz"]
    if k == "rsdf":
        return dict(bytes=V * (24 + 8 + 8), flops=0.0)
    if k == "iso":
        rays = float(case["rays"]) ** 2 * case["ant"] * case["sets"]
        return dict(bytes=V * 4 + case["ant"] * case["sets"] * case["wavelengths"] * 8.0,
                    flops=rays * 100.0)
    if k == "image":
        w = _image_work(V, case["ant"], case["freqs"], case["mode"])
        if case["normals"]:
            w["bytes"] += V * 13
        return w
    if k == "interp":
        return _image_work(V, case["ant"], case["bins"], "interp")
    if k == "stage1":
        w = _image_work(V, case["ant"] * case["rx"], case["freqs"], "interp")
        w["bytes"] += V * 13
        return w
    A, F = case["ant"], case["freqs"]
    w = _image_work(V, A, F, "nufft")
    n = 3 if k == "train" else 2   # forward, position gradient, measurement gradient
    return dict(bytes=V * 32 * n + A * (F * 8.0 + 24) * n, flops=w["flops"] * n)


# ------------------------------------------------------------------------- 64-bit results

def _geometry(s, dev):
    x, y, z = (s[k].double() for k in ("x", "y", "z"))
    vox = torch.stack(torch.meshgrid(x, y, z, indexing="ij"), dim=-1).reshape(-1, 3)
    tx = s["ant"].double()
    if s.get("pos") is not None:
        tx = tx + s["pos"].detach().double()
    off = s["rxo"].double()[torch.arange(tx.shape[0], device=dev) % s["rxo"].shape[0]]
    return vox, tx, tx + off, tx + off / 2


def _blocks(V, A, per_pair, budget=1 << 31):
    vc = min(V, 16384)
    ac = max(1, min(A, budget // (vc * per_pair)))
    for v in range(0, V, vc):
        for a in range(0, A, ac):
            yield slice(v, min(V, v + vc)), slice(a, min(A, a + ac))


def _phasor(ph):
    return torch.polar(torch.ones_like(ph), ph)


def _adjoint_exact(s, sums, grads):
    """(image, vote) and, when ``grads``, (dL/dmeas, dL/dpos), all in 64 bits.

    A row's F samples are split as j = 16 q + r, so that exp(-i d kappa_j) is the product of
    one of 16 fine and one of F/16 coarse phasors."""
    dev = s["ant"].device
    vox, tx, rx, virt = _geometry(s, dev)
    V, A = vox.shape[0], tx.shape[0]
    m = s["meas"].detach().to(torch.complex128)
    F = m.shape[1]
    Q = -(-F // 16)
    m = torch.nn.functional.pad(torch.view_as_real(m), (0, 0, 0, 16 * Q - F))
    m = torch.view_as_complex(m.contiguous()).reshape(A, Q, 16)
    k0, kd = PI2 / s["wavelength"], PI2 * s["slope"] / C
    fine = kd * torch.arange(16, device=dev, dtype=torch.float64)
    coarse = k0 + kd * 16 * torch.arange(Q, device=dev, dtype=torch.float64)
    kap = (coarse[:, None] + fine[None, :])
    ti = 0.15 if s["ti"] else 0.0
    image = torch.zeros(V, dtype=torch.complex128, device=dev)
    vote = torch.zeros((3, V), dtype=torch.complex128, device=dev)
    if grads:
        gi = s["g_image"].reshape(V).to(torch.complex128)
        gw = s["g_vote"].reshape(3, V).to(torch.complex128) if s["g_vote"] is not None else None
        gm = torch.zeros((A, Q, 16), dtype=torch.complex128, device=dev)
        gp = torch.zeros((A, 3), dtype=torch.float64, device=dev)
    for vs, as_ in _blocks(V, A, 16 * (48 + 3 * Q)):
        e1, e2 = vox[vs][None] - tx[as_][:, None], vox[vs][None] - rx[as_][:, None]
        r1, r2 = e1.norm(dim=-1), e2.norm(dim=-1)
        d = r1 + r2 + ti
        Pf, Pq = _phasor(-d[..., None] * fine), _phasor(-d[..., None] * coarse)
        u = virt[as_][:, None] - vox[vs][None]
        c = None
        if sums or grads:
            c = (torch.bmm(Pf, m[as_].transpose(1, 2)) * Pq).sum(-1)
        if sums:
            image[vs] += c.sum(0)
            vote[:, vs] += torch.einsum("av,avk->kv", c, u.to(torch.complex128))
        if grads:
            G = gi[vs][None].expand_as(c)
            if gw is not None:
                G = G + torch.einsum("kv,avk->av", gw[:, vs], u.to(torch.complex128))
            gm[as_] += torch.bmm((G[..., None] * Pq.conj()).transpose(1, 2), Pf.conj())
            cp = (torch.bmm(Pf, (m[as_] * kap).transpose(1, 2)) * Pq).sum(-1)
            dd = -(e1 / r1[..., None] + e2 / r2[..., None])
            gp[as_] += torch.einsum("av,avk->ak", (G.conj() * cp).imag, dd)
            if gw is not None:
                gp[as_] += torch.einsum("kv,av->ak", gw[:, vs].conj(), c).real
    out = (image, vote)
    if grads:
        out += (gm.reshape(A, 16 * Q)[:, :F], gp)
    return out


def _interp_exact(s, fsp):
    dev = s["ant"].device
    vox, tx, rx, virt = _geometry(s, dev)
    V, A = vox.shape[0], tx.shape[0]
    m = s["meas"].to(torch.complex128)
    n = m.shape[1]
    image = torch.zeros(V, dtype=torch.complex128, device=dev)
    vote = torch.zeros((3, V), dtype=torch.complex128, device=dev)
    ti = 0.15 if s["ti"] else 0.0
    for vs, as_ in _blocks(V, A, 160):
        d = torch.cdist(tx[as_], vox[vs], compute_mode="donot_use_mm_for_euclid_dist") + \
            torch.cdist(rx[as_], vox[vs], compute_mode="donot_use_mm_for_euclid_dist") + ti
        b = torch.floor(d / fsp / 2).long()
        ok = d <= fsp * n
        c = torch.gather(m[as_], 1, b.clamp(0, n - 1)) * _phasor(-PI2 / s["wavelength"] * d)
        c = torch.where(ok, c, torch.zeros_like(c))
        image[vs] += c.sum(0)
        u = virt[as_][:, None] - vox[vs][None]
        vote[:, vs] += torch.einsum("av,avk->kv", c, u.to(torch.complex128))
    return image, vote


def _unit_normals(image, vote, percent=0.05):
    mag = image.abs()
    raw = (image.conj()[None] * vote).real / mag
    unit = (raw / raw.norm(dim=0, keepdim=True)).movedim(0, -1)
    return torch.where((mag > percent * mag.max())[..., None], unit,
                       torch.full_like(unit, float("nan")))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("rsdf", "iso"):
        return None   # a search order and ray hits: no closed 64-bit value
    if kind == "batch":
        out = []
        for o in _batch_objects(case, seed):
            n = (o["x"].numel(), o["y"].numel(), o["z"].numel())
            image, vote = _adjoint_exact(dict(o, pos=None), True, False)
            out.append([image.reshape(n), vote.reshape((3,) + n)])
        return out
    shape = _shape(case)
    s = prepare(case, seed)
    if kind == "stage1":
        rows = torch.fft.fft(s["raw"].to(torch.complex128), n=4096, dim=1)
        rows = rows.permute(0, 2, 1).reshape(case["ant"] * case["rx"], 4096)
        image, vote = _interp_exact(dict(s, meas=rows), _fft_spacing(case["freqs"], 4096))
        image, vote = (image / case["ant"]).reshape(shape), vote.reshape((3,) + shape)
        tx = s["tx"].repeat_interleave(case["rx"], dim=0)
        centres = (tx + tx + s["rxo"].double().repeat(case["ant"], 1)) / 2
        return image, _unit_normals(image, vote), None, centres
    if kind == "interp":
        image, vote = _interp_exact(s, _fft_spacing(case["freqs"], case["bins"]))
        return image.reshape(shape), vote.reshape((3,) + shape)
    if kind == "train":
        image, vote, gm, gp = _adjoint_exact(s, True, True)
        return image.reshape(shape), vote.reshape((3,) + shape), gm, gp
    if kind == "adjoint":
        return _adjoint_exact(s, False, True)[2:]
    image, vote = _adjoint_exact(s, True, False)
    image, vote = image.reshape(shape), vote.reshape((3,) + shape)
    if not case["normals"]:
        return image, vote
    return image, vote, _unit_normals(image, vote), None
