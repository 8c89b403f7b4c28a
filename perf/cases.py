"""Performance cases: the reconstructions a user of this package runs.

Every case is one call (or one short sequence of calls) of the package's
public functions at a size that tomography beamlines meet: detectors of 256
to 2560 pixels, 60 (sparse view) to 1801 angles, one slice up to a slab of
32.  ``listed()`` gives the fixed cases, ``draw()`` more of the same ranges.

Inputs are sinograms of random ellipses with photon noise, made on the GPU
from a seed.  ``exact()`` restates each call in plain float64 torch / numpy.
"""
import math

import numpy as np
import torch

DEV = "cuda"
PHOTONS = 1.0e4


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------
def listed():
    return [
        # preview of one slice of a small region of interest during a scan:
        # the smallest call, latency bound
        dict(name="fbp_slice_256", kind="fbp", nrow=181, nslice=0, ncol=256,
             storage="float32", log=True, pad_mode="edge"),
        # one slice of an ordinary scan, the interactive unit of work
        dict(name="fbp_slice_1024", kind="fbp", nrow=900, nslice=0, ncol=1024,
             storage="float32", log=False, pad_mode="edge"),
        # a slab of the full detector, resident on the GPU: the bulk of a
        # volume reconstruction
        dict(name="fbp_stack_2560", kind="fbp", nrow=1801, nslice=32,
             ncol=2560, storage="float32", log=False, pad_mode="edge"),
        # cropped detector, odd in every size, straight from transmission
        # data (-log), another padding
        dict(name="fbp_stack_ragged", kind="fbp", nrow=1201, nslice=19,
             ncol=1613, storage="float32", log=True, pad_mode="reflect"),
        # the same bulk work with the filtered sinogram stored in 16 bits
        dict(name="fbp_stack_f16", kind="fbp", nrow=1501, nslice=24,
             ncol=2048, storage="float16", log=False, pad_mode="edge"),
        # a stack in pinned host memory, streamed through the GPU
        dict(name="fbp_host_stack", kind="host", nrow=721, nslice=48,
             ncol=1536, log=False),
        # back-projection filtering of a stack
        dict(name="bpf_stack", kind="bpf", nrow=901, nslice=16, ncol=1280,
             log=False),
        # slices of uneven geometry (several scans, every eighth a widened
        # half-acquisition) in one captured batch
        dict(name="batch_uneven", kind="batch", items=12, wmin=512, wmax=1536,
             amin=361, amax=1201, geo=3000),
        # one iteration of sparse-view model-based reconstruction: forward
        # projection, least squares + total variation, its gradient
        dict(name="descent_2048", kind="descent", nrow=60, ncol=2048,
             center=False),
        # the candidates of a rotation-centre search on one slice
        dict(name="centers_1280", kind="centers", nrow=901, ncol=1280,
             count=41, step=0.5),
        # vertical slices through a stack of projections
        dict(name="vertical_1280", kind="vertical", nrow=901, height=96,
             ncol=1280, count=8),
        # direct Fourier inversion of one slice
        dict(name="dfi_1280", kind="dfi", nrow=901, nslice=0, ncol=1280),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case; never more updates than ``fbp_stack_2560``."""
    kind = rng.choice(["fbp", "fbp", "fbp", "fbp", "host", "bpf", "batch",
                       "descent", "centers", "vertical", "dfi"])
    if kind == "fbp":
        single = rng.random() < 0.4
        ncol = _log_int(rng, 200, 2560)
        return dict(kind=kind, nrow=_log_int(rng, 120, 1801),
                    nslice=0 if single else rng.randint(2, 32), ncol=ncol,
                    storage="float32" if single else rng.choice(
                        ["float32", "float32", "float16", "bfloat16"]),
                    log=rng.random() < 0.4,
                    pad_mode=rng.choice(["edge", "edge", "reflect",
                                         "constant"]))
    if kind == "host":
        return dict(kind=kind, nrow=_log_int(rng, 300, 901),
                    nslice=rng.randint(4, 64), ncol=_log_int(rng, 512, 1536),
                    log=rng.random() < 0.4)
    if kind == "bpf":
        return dict(kind=kind, nrow=_log_int(rng, 180, 1201),
                    nslice=rng.randint(1, 24), ncol=_log_int(rng, 256, 1536),
                    log=rng.random() < 0.4)
    if kind == "batch":
        return dict(kind=kind, items=rng.randint(3, 12), wmin=512, wmax=1536,
                    amin=361, amax=1201, geo=rng.randint(1, 1 << 20))
    if kind == "descent":
        return dict(kind=kind, nrow=rng.randint(30, 120),
                    ncol=_log_int(rng, 512, 2048), center=rng.random() < 0.3)
    if kind == "centers":
        return dict(kind=kind, nrow=_log_int(rng, 361, 901),
                    ncol=_log_int(rng, 512, 1536), count=rng.randint(9, 41),
                    step=rng.choice([0.25, 0.5, 1.0]))
    if kind == "vertical":
        return dict(kind=kind, nrow=_log_int(rng, 361, 901),
                    height=rng.randint(32, 160), ncol=_log_int(rng, 512, 1536),
                    count=rng.choice([1, 4, 8, 12]))
    return dict(kind=kind, nrow=_log_int(rng, 361, 1201),
                nslice=rng.choice([0, 2]), ncol=_log_int(rng, 512, 1801))


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _ellipses(rng, ncol, n=12):
    half, scale = 0.35 * ncol, min(1.0, ncol / 1024.0)
    return [(rng.uniform(-half, half), rng.uniform(-half, half),
             rng.uniform(20.0, 300.0) * scale, rng.uniform(20.0, 300.0) * scale,
             rng.uniform(0.0, math.pi)) for _ in range(n)]


def _sinogram(seed, nrow, nslice, ncol, center, angles, log=False,
              photons=PHOTONS):
    """float32 [nrow, nslice, ncol] on the GPU: attenuations of 12 ellipses
    (one shape per stack, another mixture per slice) with photon noise, or
    their transmissions (``log``)."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=DEV).manual_seed(int(seed) + 1)
    th = torch.as_tensor(np.asarray(angles), dtype=torch.float32,
                         device=DEV)[:, None]
    u = torch.arange(ncol, dtype=torch.float32, device=DEV)[None] - center
    chords = []
    for x0, y0, a, b, phi in _ellipses(rng, ncol):
        u0 = x0 * torch.cos(th) - y0 * torch.sin(th)
        a2 = (a * torch.cos(th + phi)) ** 2 + (b * torch.sin(th + phi)) ** 2
        chords.append(2.0 * a * b / ncol *
                      torch.sqrt((a2 - (u - u0) ** 2).clamp_(min=0.0)) / a2)
    mu = torch.rand((nslice, len(chords)), generator=gen, device=DEV) + 0.1
    out = torch.empty((nrow, nslice, ncol), dtype=torch.float32, device=DEV)
    for k in range(nslice):
        line = sum(float(m) * c for m, c in zip(mu[k].tolist(), chords))
        sd = torch.exp(0.5 * line) * photons ** -0.5
        noise = torch.randn((nrow, ncol), generator=gen, device=DEV)
        line = line + sd * noise.clamp_(-4.0, 4.0)
        out[:, k] = torch.exp(-line) if log else line
    return out


def _angles(nrow):
    return np.linspace(0.0, math.pi, nrow)


def _center(ncol):
    return (ncol - 1) / 2.0 - 1.2


def prepare(case, seed):
    kind, ncol = case["kind"], case["ncol"] if "ncol" in case else 0
    if kind == "batch":
        from algotom_b200.rec.batch import BatchedFBP
        geo = _geometry(case)
        sinos = [_sinogram(seed * 100 + k, g["nrow"], 1, g["ncol"],
                           g["center"], g["angles"])[:, 0].contiguous()
                 for k, g in enumerate(geo)]
        plan = BatchedFBP([(g["nrow"], g["ncol"]) for g in geo],
                          [g["center"] for g in geo],
                          [g["angles"] for g in geo])
        plan.capture()
        return dict(case, plan=plan, sinos=sinos)
    nrow, cen = case["nrow"], _center(ncol)
    ang = _angles(nrow)
    s = dict(case, ang=ang, cen=cen)
    if kind in ("fbp", "bpf", "dfi"):
        x = _sinogram(seed, nrow, max(1, case["nslice"]), ncol, cen, ang,
                      log=case.get("log", False))
        s["sino"] = x if case["nslice"] else x[:, 0].contiguous()
    elif kind == "host":
        x = _sinogram(seed, nrow, case["nslice"], ncol, cen, ang,
                      log=case["log"])
        s["sino"] = torch.empty(x.shape, pin_memory=True)
        s["sino"].copy_(x)
        s["out"] = torch.empty((ncol, case["nslice"], ncol), pin_memory=True)
    elif kind == "descent":
        s["ang"] = np.linspace(0.0, math.pi, nrow, endpoint=False)
        s["sino"] = _sinogram(seed, nrow, 1, ncol, cen, s["ang"])[:, 0] * ncol
        gen = torch.Generator(device=DEV).manual_seed(int(seed) + 2)
        coarse = torch.rand((1, 1, 17, 17), generator=gen, device=DEV)
        x = torch.nn.functional.interpolate(coarse, (ncol, ncol),
                                            mode="bicubic")[0, 0]
        x = x + 0.05 * torch.rand((ncol, ncol), generator=gen, device=DEV)
        s["x"] = x.contiguous().requires_grad_(True)
        s["c"] = torch.tensor(cen, dtype=torch.float64,
                              requires_grad=case["center"])
    elif kind == "centers":
        s["sino"] = _sinogram(seed, nrow, 1, ncol, cen,
                              ang)[:, 0].contiguous()
        s["centers"] = cen + case["step"] * (np.arange(case["count"])
                                             - case["count"] // 2)
    elif kind == "vertical":
        s["sino"] = _sinogram(seed, nrow, case["height"], ncol, cen, ang,
                              log=True)
    return s


def _geometry(case):
    from algotom_b200.rec.batch import uneven_batch_geometry
    return uneven_batch_geometry(case["geo"], case["items"], case["wmin"],
                                 case["wmax"], case["amin"], case["amax"])


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "batch":
        return s["plan"](s["sinos"])
    if kind == "descent":
        from algotom_b200.rec import autograd as ag
        r = ag.forward_projection(s["x"], s["c"], s["ang"]) - s["sino"]
        loss = 0.5 * (r * r).sum() + 1e-3 * ag.total_variation(s["x"])
        wrt = [s["x"], s["c"]] if s["center"] else [s["x"]]
        return [loss.detach(), r.detach(),
                list(torch.autograd.grad(loss, wrt))]
    from algotom_b200.rec import reconstruction as rec
    if kind == "fbp":
        return rec.fbp_reconstruction(
            s["sino"], s["cen"], angles=s["ang"], apply_log=s["log"],
            pad_mode=s["pad_mode"], storage=s["storage"])
    if kind == "host":
        return rec.fbp_reconstruction(s["sino"], s["cen"], angles=s["ang"],
                                      apply_log=s["log"], out=s["out"])
    if kind == "bpf":
        return rec.bpf_reconstruction(s["sino"], s["cen"], angles=s["ang"],
                                      apply_log=s["log"])
    if kind == "dfi":
        return rec.dfi_reconstruction(s["sino"], s["cen"], angles=s["ang"],
                                      apply_log=False)
    if kind == "centers":
        from algotom_b200.rec.center import reconstruct_centers
        return reconstruct_centers(s["sino"], s["centers"], angles=s["ang"])
    from algotom_b200.rec import vertrec
    mid, n = s["ncol"] // 2, s["count"]
    if n == 1:
        return vertrec.vertical_reconstruction(
            s["sino"], mid, s["cen"], alpha=30.0, angles=s["ang"],
            show_progress=False)
    return vertrec.vertical_reconstruction_multiple(
        s["sino"], mid - n // 2, mid - n // 2 + n - 1, s["cen"], alpha=30.0,
        angles=s["ang"], show_progress=False)


def work(case):
    """Each input read once, each output written once; 4 flops for every
    interpolated sample that is added, 5 n log2 n for a transform."""
    def fft(n, rows):
        return 2 * 2.5 * n * math.log2(n) * rows
    kind = case["kind"]
    if kind == "batch":
        geo = _geometry(case)
        return dict(bytes=sum(4 * g["nrow"] * g["ncol"] + 4 * g["ncol"] ** 2
                              for g in geo),
                    flops=sum(4 * g["nrow"] * g["ncol"] ** 2 +
                              fft(1.3 * g["ncol"], g["nrow"]) for g in geo))
    nrow, ncol = case["nrow"], case["ncol"]
    if kind == "descent":
        upd = nrow * ncol * ncol
        return dict(bytes=4 * (2 * nrow * ncol + 3 * ncol * ncol),
                    flops=(12 if case["center"] else 8) * upd)
    if kind == "centers":
        n = case["count"]
        return dict(bytes=4 * (nrow * ncol + n * ncol * ncol),
                    flops=4 * n * nrow * ncol * ncol + fft(1.3 * ncol, nrow))
    if kind == "vertical":
        n, h = case["count"], case["height"]
        return dict(bytes=4 * h * ncol * (nrow + n),
                    flops=4 * n * h * nrow * ncol)
    n = max(1, case["nslice"])
    size = 4 * n * (nrow * ncol + ncol * ncol)
    if kind == "dfi":
        w = 1.5 * ncol
        return dict(bytes=size + 4 * n * ncol * ncol,
                    flops=n * (fft(w, nrow) + 2 * fft(w, w)))
    flops = 4 * n * nrow * ncol * ncol
    if kind == "bpf":
        return dict(bytes=size, flops=flops + 4 * n * fft(1.3 * ncol, ncol))
    return dict(bytes=size, flops=flops + n * fft(1.3 * ncol, nrow))


# --------------------------------------------------------------------------
# the same in float64
# --------------------------------------------------------------------------
def _ramp_row(width):
    k = np.arange(width, dtype=np.float64) - math.ceil((width - 1.0) / 2)
    r = np.zeros(width)
    odd = np.abs(k) % 2 == 1
    r[odd] = -1.0 / (np.pi * k[odd]) ** 2
    r[k == 0] = 0.25
    return np.fft.fft(r), np.hanning(width)


def _ramp_filter(x, pad, pad_mode):
    """Padded ramp-and-hann filter of the last axis (float64)."""
    ncol = x.shape[-1]
    n = ncol + 2 * pad
    at = np.pad(np.arange(ncol), pad, mode="edge" if pad_mode == "constant"
                else pad_mode)
    p = x[..., torch.from_numpy(at).to(x.device)]
    if pad_mode == "constant":
        p[..., :pad] = 0.0
        p[..., pad + ncol:] = 0.0
    f, win = _ramp_row(n)
    h = torch.from_numpy(np.fft.ifftshift(np.fft.fftshift(f) * win))
    y = torch.fft.ifft(torch.fft.fft(p) * h.to(x.device)).real
    return torch.roll(y, -(n // 2), -1)[..., pad:pad + ncol].contiguous()


def _backproject(sino, angles, center, edge=False):
    """[nrow, S, ncol] float64 -> [S, ncol, ncol]: the linear interpolation
    of every slice at each pixel's position, summed over the angles of the
    float32-rounded geometry."""
    nrow, ns, ncol = sino.shape
    ang = np.float32(angles).astype(np.float64)
    cen = float(np.float32(center))
    ic = 0.5 * (ncol - 1)
    xc = torch.arange(ncol, dtype=torch.float64, device=DEV) - ic
    out = torch.zeros((ncol * ncol, ns), dtype=torch.float64, device=DEV)
    step = max(1, int(5e7 // (ncol * ncol)))
    for i0 in range(0, nrow, step):
        part = sino[i0:i0 + step]
        na = part.shape[0]
        tab = torch.zeros((na, ncol + 1, ns), dtype=torch.float64, device=DEV)
        tab[:, :ncol] = part.transpose(1, 2)
        idx = torch.empty((ncol, ncol, na, 2), dtype=torch.int32, device=DEV)
        wei = torch.empty((ncol, ncol, na, 2), dtype=torch.float64,
                          device=DEV)
        for k in range(na):
            a = ang[i0 + k]
            p = (xc[None, :] * math.cos(-a) + xc[:, None] * math.sin(-a)) + cen
            inside = (p >= 0.0) & (p <= ncol - 1)
            p = p.clamp_(0.0, ncol - 1)
            d = torch.floor(p)
            f = p - d
            live = 1.0 if edge else inside.double()
            wei[:, :, k, 0] = (1.0 - f) * live
            wei[:, :, k, 1] = f * live
            d = d.int() + k * (ncol + 1)
            idx[:, :, k, 0] = d
            idx[:, :, k, 1] = d + 1
        out += torch.nn.functional.embedding_bag(
            idx.view(ncol * ncol, 2 * na), tab.view(-1, ns), mode="sum",
            per_sample_weights=wei.view(ncol * ncol, 2 * na))
        del idx, wei, tab
    return out.t().reshape(ns, ncol, ncol)


def _disc(ncol):
    c = ncol // 2
    k = torch.arange(ncol, device=DEV) - c
    return (k[None] ** 2 + k[:, None] ** 2 <= c * c).double()


def _fbp(sino, ang, cen, pad_mode="edge"):
    """[nrow, S, ncol] attenuations -> [ncol, S, ncol]."""
    nrow, ncol = sino.shape[0], sino.shape[2]
    f = _ramp_filter(sino.double(), min(int(0.15 * ncol), 150), pad_mode)
    r = _backproject(f, ang, cen) * _disc(ncol) * (math.pi / (nrow - 1))
    return r.transpose(0, 1)


def _circular_filter(img, pad):
    """2-D circular ramp-and-hann filter of [S, ncol, ncol] images."""
    ncol = img.shape[-1]
    n = ncol + 2 * pad
    f, win = _ramp_row(n)
    prof = np.abs(np.fft.fftshift(f)) * win
    w = n + 1 if n % 2 == 0 else n
    c = w // 2
    x = np.arange(w)[::-1].astype(np.float64) - c
    y = np.arange(w).astype(np.float64) - c
    xm, ym = np.meshgrid(x, y)
    rad = np.float32(np.clip(np.sqrt(xm ** 2 + ym ** 2), 0, c))
    rad[np.arctan2(ym, xm) < 0] *= -1
    rad = np.float32(np.clip(rad + c, 0, w - 1))
    h = np.interp(rad.astype(np.float64), np.arange(n), prof)[:n, :n]
    h = torch.from_numpy(np.fft.ifftshift(h)).to(DEV)
    at = torch.from_numpy(np.pad(np.arange(ncol), pad, mode="edge")).to(DEV)
    out = torch.empty_like(img)
    for k in range(img.shape[0]):
        p = img[k][at][:, at]
        y = torch.fft.ifft2(torch.fft.fft2(p) * h).real
        out[k] = y[pad:pad + ncol, pad:pad + ncol]
    return out


def _positions(ncol, a, cen):
    xc = torch.arange(ncol, dtype=torch.float64, device=DEV) - 0.5 * (ncol - 1)
    p = xc[None, :] * math.cos(-a) + xc[:, None] * math.sin(-a) + cen
    live = ((p >= 0.0) & (p <= ncol - 1)).double()
    p = p.clamp_(0.0, ncol - 1)
    d = torch.floor(p)
    return d.long(), (p - d) * live, (1.0 - (p - d)) * live


def _vertical(sino, ang, cen, indices, alpha):
    """[nproj, height, ncol] transmissions -> [lines, height, ncol]: lines
    of points at ``alpha`` degrees (at most 45) through the columns
    ``indices``, edge samples outside the detector, zero-phase ramp filter
    afterwards."""
    nrow, height, ncol = sino.shape
    line = -torch.log(sino.double())
    mid, t = math.ceil(0.5 * (ncol - 1)), math.radians(alpha)
    res = []
    for index in indices:
        b = -(index - mid) / math.cos(t)
        x = -math.tan(t) * b / (1 + math.tan(t) ** 2) + \
            np.arange(-mid, ncol - mid) * math.cos(t)
        y = math.tan(t) * x + b
        x, y = (torch.from_numpy(np.float32(v).astype(np.float64)).to(DEV)
                for v in (x, y))
        acc = torch.zeros((height, ncol), dtype=torch.float64, device=DEV)
        for k, a in enumerate(np.float32(ang).astype(np.float64)):
            p = x * math.cos(a) + y * math.sin(a) + float(np.float32(cen))
            p = p.clamp_(0.0, ncol - 1)
            d = torch.floor(p).long()
            v = line[k][:, d]
            acc += v + (line[k][:, (d + 1).clamp_(max=ncol - 1)] - v) * (p - d)
        res.append(acc)
    pad = min(int(0.15 * ncol), 150)
    f, win = _ramp_row(ncol + 2 * pad)
    h = torch.from_numpy(np.fft.ifftshift(np.abs(np.fft.fftshift(f) * win)))
    p = torch.stack(res)
    p = p[..., torch.from_numpy(np.pad(np.arange(ncol), pad, "edge")).to(DEV)]
    y = torch.fft.ifft(torch.fft.fft(p) * h.to(DEV)).real
    return y[..., pad:pad + ncol] * (math.pi / (nrow - 1))


def exact(case, seed):
    kind = case["kind"]
    if kind == "dfi":  # float64 throughout already, held to its own type
        return None
    s = prepare(case, seed)
    if kind == "vertical":
        n, first = case["count"], case["ncol"] // 2 - case["count"] // 2
        r = _vertical(s["sino"], s["ang"], s["cen"], range(first, first + n),
                      30.0)
        return r[0] if n == 1 else r
    if kind == "batch":
        return [_fbp(x[:, None], g["angles"], g["center"])[:, 0]
                for x, g in zip(s["sinos"], _geometry(case))]
    ncol, nrow, ang, cen = case["ncol"], case["nrow"], s["ang"], s["cen"]
    if kind == "descent":
        x = s["x"].detach().double()
        r = torch.empty((nrow, ncol), dtype=torch.float64, device=DEV)
        for i in range(nrow):
            d, f, g = _positions(ncol, ang[i], cen)
            row = torch.bincount(d.flatten(), (g * x).flatten(), ncol + 1)
            row[1:] += torch.bincount(d.flatten(), (f * x).flatten(),
                                      ncol + 1)[:-1]
            r[i] = row[:ncol]
        r -= s["sino"].double()
        y = x.clone().requires_grad_(True)
        dx, dy = y[:-1, 1:] - y[:-1, :-1], y[1:, :-1] - y[:-1, :-1]
        tv = 1e-3 * torch.sqrt(dx * dx + dy * dy + 1e-8).sum()
        (grad,) = torch.autograd.grad(tv, [y])
        for i in range(nrow):
            d, f, g = _positions(ncol, ang[i], cen)
            row = torch.nn.functional.pad(r[i], (0, 1))
            grad += row[d] * g + row[d + 1] * f
        loss = 0.5 * (r * r).sum() + tv.detach()
        return [loss, r, [grad, None] if case["center"] else [grad]]
    sino = s["sino"]
    if kind == "centers":
        return torch.stack([_fbp(sino[:, None], ang, c)[:, 0]
                            for c in s["centers"]])
    if kind == "host":
        sino = sino.to(DEV)
    if case["log"]:
        sino = -torch.log(sino.double())
    two_d = sino.dim() == 2
    sino = (sino[:, None] if two_d else sino).double()
    if kind == "bpf":
        img = _backproject(sino, ang, cen, edge=True)
        img = _circular_filter(img, min(int(0.15 * ncol), 150)) * _disc(ncol)
        return (img * (math.pi / (nrow - 1))).transpose(0, 1)
    rec = _fbp(sino, ang, cen, case.get("pad_mode", "edge"))
    return rec[:, 0] if two_d else rec
