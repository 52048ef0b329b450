"""The work that users of this framework have it do, as timed cases.

Every case goes through the entry points a program calls: ``GPURec.recon_all``
on a scan, ``SinoPipeline.reconstruct`` on a chunk of rows (what the drivers
and the server run per chunk), the reference's own call sequence on the
drop-in operators, the laminography chain, ring removal, projection
pre-processing with phase retrieval, and the try-centre sweep.  Frames are
seeded ellipse phantoms with Beer-Lambert attenuation, photon noise, darks and
flats, in uint16 as detectors deliver them.
"""
import math

import numpy as np
import torch

from tomocupy_b200 import global_vars
from tomocupy_b200.dataio import ArrayReader, ArrayWriter
from tomocupy_b200.global_vars import params
from tomocupy_b200.pipeline import SinoPipeline
from tomocupy_b200.processing.proc_functions import ProcFunctions, darkflat_stats
from tomocupy_b200.processing.remove_stripe import remove_stripe_fw
from tomocupy_b200.rec import GPURec
from tomocupy_b200.reconstruction.backproj_functions import BackprojFunctions
from tomocupy_b200.reconstruction.backproj_lamfourier_parallel import BackprojLamFourierParallel
from tomocupy_b200.trycenter import TryCenterSweep

DEV = "cuda"


def _case(kind, **kw):
    return dict(kind=kind, **kw)


def listed():
    return [
        # a small scan through the full driver at the default chunk of 8 rows,
        # the size of the plain parallel-beam configuration: 16 rows x 360
        # angles x 512 columns; latency and launches count
        _case("scan", name="scan_512", n=512, nproj=360, nz=16, filter="parzen"),
        # the reference's own per-chunk sequence on the drop-in operators
        # (proc_sino, proc_proj, fbp_filter_center, backprojection), as a
        # program that switched its imports runs it
        _case("dropin", name="dropin_1024", n=1024, nproj=720, nz=16, filter="parzen"),
        # one chunk of the production scan, 2048 columns x 1500 angles, at the
        # production chunk of 128 rows: the largest case
        _case("chunk", name="fourierrec_2048", algorithm="fourierrec", precision="float32",
              n=2048, nproj=1500, nz=128, filter="shepp"),
        # a mixed-precision chunk with float16 slices out, as half of the
        # serving stream's requests: 1024 columns x 720 angles x 64 slices
        _case("chunk", name="mixed_1024", algorithm="fourierrec", precision="mixed",
              n=1024, nproj=720, nz=64, filter="shepp"),
        # a detector whose width is no power of two: 1500 angles x 2448 columns
        _case("chunk", name="fourierrec_2448", algorithm="fourierrec", precision="float32",
              n=2448, nproj=1500, nz=16, filter="parzen"),
        # the log-polar method
        _case("chunk", name="lprec_1024", algorithm="lprec", precision="float32",
              n=1024, nproj=900, nz=32, filter="shepp"),
        # the line-summation method
        _case("chunk", name="linerec_1024", algorithm="linerec", precision="float32",
              n=1024, nproj=720, nz=16, filter="shepp"),
        # Vo's ring removal in front of fourierrec
        _case("vo", name="vo_1024", n=1024, nproj=720, nz=16, filter="shepp"),
        # Fourier-wavelet ring removal of a production chunk (level 7, sigma 1)
        _case("fw", name="fw_2048", n=2048, nproj=1500, nz=16),
        # laminography, 30 degrees of tilt, at half the production size
        _case("lamino", name="lamino_512", n=512, nproj=600, deth=512, rh=256, filter="shepp"),
        # projections through dark/flat, phase retrieval and -log
        _case("phase", name="paganin_2048", n=2048, nproj=8, nz=2048),
        # a rotation-centre search: one row, 64 centres
        _case("try", name="try_1024", n=1024, nproj=720, centers=64, filter="parzen"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _even(v):
    return max(2, 2 * int(round(v / 2)))


FILTERS = ("ramp", "shepp", "hann", "parzen")


def draw(rng):
    """A case of the same ranges: widths 256-2448 (half of them powers of two,
    as detectors are), angles 90-1500, chunks of 2-128 rows."""
    kind = rng.choice(["scan", "dropin", "chunk", "chunk", "chunk", "chunk", "vo", "fw", "lamino",
                       "phase", "try"])
    filt = rng.choice(FILTERS)
    pow2 = rng.random() < 0.5

    def width(lo, hi):
        return 2 ** rng.randint(int(math.log2(lo)), int(math.log2(hi))) if pow2 \
            else _even(_log(rng, lo, hi))

    if kind == "scan":
        return _case("scan", n=width(256, 1024), nproj=int(_log(rng, 90, 720)),
                     nz=rng.randint(3, 40), filter=filt)
    if kind == "dropin":
        return _case("dropin", n=width(256, 1024), nproj=int(_log(rng, 90, 900)),
                     nz=_even(rng.uniform(2, 24)), filter=filt)
    if kind == "chunk":
        alg = rng.choice(["fourierrec", "fourierrec", "lprec", "linerec"])
        prec = rng.choice(["float32", "mixed"]) if alg == "fourierrec" else "float32"
        top = {"fourierrec": 2448, "lprec": 1200, "linerec": 1448}[alg]
        n, nproj = width(256, top), int(_log(rng, 180, 1500 if alg == "fourierrec" else 900))
        most = {"fourierrec": 64, "lprec": 40, "linerec": 24}[alg]
        nz = _even(_log(rng, 4, most)) if n <= 1024 else _even(_log(rng, 4, most / 4))
        return _case("chunk", algorithm=alg, precision=prec, n=n, nproj=nproj, nz=nz, filter=filt)
    if kind == "vo":
        return _case("vo", n=width(256, 1024), nproj=int(_log(rng, 180, 900)),
                     nz=_even(rng.uniform(2, 16)), filter=filt)
    if kind == "fw":
        return _case("fw", n=width(512, 2048), nproj=int(_log(rng, 360, 1500)),
                     nz=rng.randint(2, 16))
    if kind == "lamino":
        n = 4 * int(round(_log(rng, 128, 512) / 4))
        return _case("lamino", n=n, nproj=int(_log(rng, 120, 600)), deth=n,
                     rh=_even(n * rng.uniform(0.3, 0.6)), filter=filt)
    if kind == "phase":
        n = width(512, 2048)
        return _case("phase", n=n, nproj=rng.randint(3, 8), nz=_even(n * rng.uniform(0.3, 1.0)))
    return _case("try", n=width(512, 1024), nproj=int(_log(rng, 180, 720)),
                 centers=rng.randint(20, 64), filter=filt)


# ------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _theta(nproj, span=math.pi):
    return (np.arange(nproj) * span / nproj).astype(np.float32)


def _paths(seed, n, nproj, nz, count=16):
    """Line integrals [nproj, nz, n] float32 of ``count`` random ellipsoids."""
    rng = np.random.default_rng(int(seed))
    th = torch.as_tensor(_theta(nproj), device=DEV)[:, None, None]
    s = (torch.arange(n, device=DEV, dtype=torch.float32) + 0.5 - n / 2)[None, None, :]
    z = (torch.arange(nz, device=DEV, dtype=torch.float32))[None, :, None]
    out = torch.zeros((nproj, nz, n), dtype=torch.float32, device=DEV)
    for _ in range(count):
        rad, ang = 0.6 * n / 2 * math.sqrt(rng.uniform()), rng.uniform(0, 2 * math.pi)
        lim = n / 2 - rad
        a, b = rng.uniform(0.05, 0.5) * lim + 2, rng.uniform(0.05, 0.5) * lim + 2
        al, rho = rng.uniform(0, math.pi), rng.uniform(0, 3.0) / n
        cz, c = rng.uniform(0, nz), rng.uniform(0.7, 2.0) * max(nz, 8)
        k2 = torch.clamp(1 - ((z - cz) / c) ** 2, min=0.0)
        w2 = (a * torch.cos(th - al)) ** 2 + (b * torch.sin(th - al)) ** 2
        s0 = rad * torch.cos(th - ang)
        for p0 in range(0, nproj, 64):   # slabs of angles bound the temporaries
            p = slice(p0, p0 + 64)
            d2 = w2[p] * k2 - (s - s0[p]) ** 2
            out[p] += (2 * rho * a * b) / w2[p] * torch.sqrt(torch.clamp(d2, min=0.0))
    return out


def _u16(x):
    return x.round_().clamp_(0, 65535).to(torch.int32).to(torch.uint16)


def _frames(seed, n, nproj, nz, stripes=0):
    """(data, dark, flat) uint16 frames."""
    g = _gen(seed)
    t = _paths(seed, n, nproj, nz).neg_().exp_()
    gain = 1 + 0.02 * torch.randn((nz, n), generator=g, device=DEV)
    if stripes:
        cols = torch.randperm(n, generator=g, device=DEV)[:stripes]
        bad = torch.ones(n, device=DEV)
        bad[cols] = 0.9 + 0.2 * torch.rand(stripes, generator=g, device=DEV)
        t *= bad
    t *= 1e4 * gain
    t += torch.sqrt(t) * torch.randn(t.shape, generator=g, device=DEV)
    t += 100
    flat = 100 + 1e4 * gain + 100 * torch.randn((10, nz, n), generator=g, device=DEV)
    dark = 100 + 5 * torch.randn((10, nz, n), generator=g, device=DEV)
    return _u16(t), _u16(dark), _u16(flat)


def _norm_rows(seed, n, nproj, nz):
    """Normalised float32 projections [nproj, nz, n] with 30 stripe artefacts."""
    g = _gen(seed)
    t = _paths(seed, n, nproj, nz).neg_().exp_()
    bad = torch.ones(n, device=DEV)
    bad[torch.randperm(n, generator=g, device=DEV)[:30]] = \
        0.97 + 0.06 * torch.rand(30, generator=g, device=DEV)
    t *= bad
    t += 0.01 * torch.randn(t.shape, generator=g, device=DEV)
    return t


def _lam_rows(seed, n, nproj, deth):
    """Smooth float32 projections [nproj, deth, n] over [0, 2 pi)."""
    g = _gen(seed)
    f = torch.randn((4, 1, deth, n), generator=g, device=DEV)
    k = torch.exp(-0.5 * (torch.arange(-24, 25, device=DEV) / 8.0) ** 2)
    k = k / k.sum()
    f = torch.nn.functional.conv2d(f, k[None, None, None, :], padding=(0, 24))
    f = torch.nn.functional.conv2d(f, k[None, None, :, None], padding=(24, 0))[:, 0]
    f = f / f.std()
    th = torch.arange(nproj, device=DEV) * (2 * math.pi / nproj)
    c = torch.stack((1 + 0 * th, torch.cos(th), torch.sin(th), torch.cos(2 * th)), 1)
    return torch.tensordot(c, f, dims=1).contiguous()


def _center(c):
    return c["n"] / 2 + 2.25


def _shifts(c):
    return (0.375 * (np.arange(c["centers"]) - c["centers"] // 2)).astype(np.float32)


PHASE = dict(retrieve_phase_method="paganin", energy=20.0, propagation_distance=50.0,
             pixel_size=0.65, retrieve_phase_alpha=1e-3)


def _keep_globals(state):
    """The option namespaces as this program's scan set them."""
    state["args"], state["params"] = dict(vars(global_vars.args)), dict(vars(params))
    return state


def _use_globals(state):
    vars(global_vars.args).update(state["args"])
    vars(params).update(state["params"])


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "lamino":
        th = _theta(c["nproj"], 2 * math.pi)
        global_vars.reset(lamino_angle=30.0, reconstruction_algorithm="fourierrec",
                          nsino_per_chunk=32, nproj_per_chunk=60, fbp_filter=c["filter"])
        params.n, params.nz, params.nproj, params.ncproj, params.ncz = (
            c["n"], c["deth"], c["nproj"], min(60, c["nproj"]), 32)
        params.rh, params.center, params.theta, params.lamino_angle = c["rh"], c["n"] / 2, th, 30.0
        s = dict(kind=kind, data=_lam_rows(seed, c["n"], c["nproj"], c["deth"]),
                 bp=BackprojLamFourierParallel(device=DEV))
        return _keep_globals(s)
    if kind == "fw":
        return dict(kind=kind, data=_norm_rows(seed, c["n"], c["nproj"], c["nz"]))
    if kind == "phase":
        data, dark, flat = _frames(seed, c["n"], c["nproj"], c["nz"])
        global_vars.reset(**PHASE)
        params.nproj = c["nproj"]
        return _keep_globals(dict(kind=kind, data=data, dark=dark, flat=flat, proc=ProcFunctions()))
    if kind == "try":
        data, dark, flat = _frames(seed, c["n"], c["nproj"], 1)
        d0, f0, _ = darkflat_stats(dark, flat)
        sw = TryCenterSweep(c["n"], c["nproj"], _theta(c["nproj"]), _center(c), _shifts(c),
                            c["filter"], "float32", ncz=64, device=DEV)
        sw.load(data, d0, f0)
        sw.capture()
        return dict(kind=kind, data=data, d0=d0, f0=f0, sweep=sw)
    n, nproj, nz = c["n"], c["nproj"], c["nz"]
    data, dark, flat = _frames(seed, n, nproj, nz, stripes=30 if kind == "vo" else 0)
    th = _theta(nproj)
    if kind == "scan":
        global_vars.reset(fbp_filter=c["filter"], rotation_axis=_center(c))
        rec = GPURec(ArrayReader(data, dark, flat, theta=th), ArrayWriter(device=DEV), device=DEV)
        rec.pipe   # built once per scan
        return _keep_globals(dict(kind=kind, rec=rec))
    if kind == "dropin":
        global_vars.reset(fbp_filter=c["filter"], rotation_axis=_center(c), nsino_per_chunk=nz)
        ArrayReader(data, dark, flat, theta=th)   # sets the sizes of this scan
        s = dict(kind=kind, data=data, dark=dark, flat=flat, proc=ProcFunctions(),
                 bp=BackprojFunctions(device=DEV),
                 out=torch.empty((nz, n, n), dtype=torch.float32, device=DEV))
        return _keep_globals(s)
    d0, f0, _ = darkflat_stats(dark, flat)
    mixed = c.get("precision") == "mixed"
    pipe = SinoPipeline(n, nproj, nz, th, _center(c), c["filter"],
                        c.get("algorithm", "fourierrec"), device=DEV,
                        stripe=("vo-all", 3.0, 61, 21, 1) if kind == "vo" else None,
                        precision="mixed" if mixed else "float32",
                        out_dtype="float16" if mixed else "float32")
    out = torch.empty((nz, n, n), dtype=torch.float16 if mixed else torch.float32, device=DEV)
    return dict(kind=kind, data=data, d0=d0, f0=f0, pipe=pipe, out=out)


def run(state):
    s, kind = state, state["kind"]
    if kind in ("chunk", "vo"):
        return s["pipe"].reconstruct(s["out"], s["data"], s["d0"], s["f0"])
    if kind == "fw":
        return remove_stripe_fw(s["data"], 1.0, "sym16", 7)
    if kind == "try":
        s["sweep"].load(s["data"], s["d0"], s["f0"])
        return s["sweep"].run()
    _use_globals(s)
    if kind == "scan":
        return s["rec"].recon_all()
    if kind == "lamino":
        return s["bp"].rec_lam(s["data"])
    proj = s["proc"].proc_proj(s["proc"].proc_sino(s["data"], s["dark"], s["flat"]))
    if kind == "phase":
        return proj
    sino = s["bp"].fbp_filter_center(proj.permute(1, 0, 2).contiguous())
    s["bp"].cl_rec.backprojection(s["out"], sino, torch.cuda.current_stream())
    return s["out"]


# --------------------------------------------------------------------- work
def _fft(n):
    return 5.0 * n * math.log2(n)


def work(case):
    """Frames read once and slices written once; the flops of the method: rows
    filtered by real FFTs of twice their length, then fourierrec's gridding
    (81 cells of a complex value) and pruned inverse FFT, or a bilinear update
    per voxel and angle."""
    c, kind = case, case["kind"]
    n, P = c["n"], c["nproj"]
    if kind == "fw":
        px = P * c["nz"] * n
        return {"bytes": 8.0 * px, "flops": 4 / 3 * 2 * 4 * 32 * 2.0 * px * 1.125}
    if kind == "phase":
        pad = 4.0 * 2 ** (math.ceil(math.log2(n)) + math.ceil(math.log2(c["nz"])))
        return {"bytes": 6.0 * P * c["nz"] * n, "flops": P * 5.0 * pad * math.log2(pad)}
    if kind == "lamino":
        half = (c["deth"] // 2 + 1.0)
        flops = P * c["deth"] * 2 * _fft(2 * n) / 2 + P * _fft(n * c["deth"]) / 2
        flops += half * (P * n * 81 * 4 + 1.5 * _fft(4.0 * n * n))
        flops += n * n * (c["deth"] * 9 * 4 + _fft(2 * c["rh"]))
        return {"bytes": 4.0 * P * c["deth"] * n + 4.0 * c["rh"] * n * n, "flops": flops}
    nz = c["centers"] if kind == "try" else c["nz"]
    rows_in, ob = (1 if kind == "try" else nz), (2 if c.get("precision") == "mixed" else 4)
    nbytes = 2.0 * P * rows_in * n + ob * nz * n * n
    flops = P * nz * _fft(2 * n)
    alg = c.get("algorithm", "fourierrec")
    if alg == "linerec":
        flops += 8.0 * n * n * nz * P
    elif alg == "lprec":
        nth, nrho = 2 ** round(math.log2(P)), 2 * 2 ** round(math.log2(n))
        flops += 3 * nz * (_fft(nth * nrho) + 2 * 32 * (nth * nrho / 2 + n * n))
    else:
        flops += nz / 2 * (P * _fft(n) + P * n * 81 * 4 + 1.5 * _fft(4.0 * n * n))
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """About four times what is seen between two implementations of the same
    precision: the drop-in chain (padded cuFFT filter, register gridding)
    against the fused one (4e-6 relative, 1e-4 of the result's root mean square
    at 2448 x 1500), or against 64 bits where there is one implementation."""
    kind = case["kind"]
    if case.get("precision") == "mixed":
        return {"rel": 1e-3, "max": 2e-2}     # fp16 operands, fp16 slices
    if kind == "lamino":
        return {"rel": 5e-6, "max": 1e-4}
    if kind == "fw":
        return {"rel": 4e-6, "max": 1e-4}
    if kind == "phase":
        return {"rel": 2e-6, "max": 1e-4}
    if kind == "vo":
        # a pixel whose rank sits beside a tie may move to the next value
        return {"rel": 2e-5, "max": 5e-3}
    return {"rel": 2e-5, "max": 5e-4}


# -------------------------------------------------------------------- exact
def _wfilter64(ne, name):
    """The quadrature-corrected filter spectrum (float64)."""
    k, t = 12, np.arange(0, ne // 2 + 1) / ne
    N = len(t)
    s = np.linspace(1e-40, 1, k)
    iv = np.linalg.inv(np.exp(np.outer(np.arange(k), np.log(s))))
    q = np.arange(1, k + 2)
    u = np.diff(np.exp(np.outer(q, np.log(s))) / q[:, None])
    w1, w2 = iv @ u[1:k + 1], iv @ u[:k]
    p = 1 / np.concatenate((np.arange(1, k), (k - 1) * np.ones(N - 2 * (k - 1) - 1),
                            np.arange(k - 1, 0, -1)))
    w, nj = np.zeros(N), N - k + 1
    h = t[k - 1:] - t[:nj]
    for m in range(k - 1):
        wm = h[:, None] ** 2 * w1[None, :, m] + (h * t[:nj])[:, None] * w2[None, :, m]
        for i in range(k):
            w[i:i + nj] += p[m:m + nj] * wm[:, i]
    w[-40:] = w[-40] / (N - 40) * np.arange(N - 40, N)
    win = {"ramp": 1.0, "shepp": np.sinc(t), "hann": (1 + np.cos(2 * np.pi * t)) / 2,
           "parzen": (1 - 2 * t) ** 3}[name]
    w = ne * 0.5 * w * win
    w = 2 * w * (w >= 0)
    w[0] *= 2
    return w / ne


def _prep64(data, dark, flat, log=True):
    """Dark/flat correction and -log of frames [P, nz, n], float64."""
    d0 = dark.to(torch.float64).mean(0)
    f0 = flat.to(torch.float64).mean(0) * (1 + 1e-5) - d0
    x = (data.to(torch.float64) - d0) / f0
    return -torch.log(torch.where(x <= 0, torch.ones_like(x), x)) if log else x


def _filter64(rows, name, center, sht=0.0):
    """Edge-padded FBP filter of rows [nz, P, n] (float64, in place)."""
    nz, _, n = rows.shape
    ne, pad = 4 * n, 4 * n // 2 - n // 2
    w = torch.as_tensor(_wfilter64(ne, name), device=DEV)
    t = torch.arange(ne // 2 + 1, device=DEV, dtype=torch.float64) / ne
    sht = torch.as_tensor(np.broadcast_to(np.asarray(sht, np.float64), (nz,)).copy(), device=DEV)
    for z in range(nz):
        r = rows[z]
        r = torch.cat((r[:, :1].expand(-1, pad), r, r[:, -1:].expand(-1, ne - n - pad)), 1)
        ww = w * torch.exp(-2j * math.pi * (-center + float(sht[z]) + n / 2) * t)
        rows[z] = (torch.fft.irfft(torch.fft.rfft(r) * ww, n=ne) * ne)[:, pad:pad + n]
    return rows


def _sign(i):
    return (1 - 2 * ((i + 1) % 2)).to(torch.float64)


def _spread64(grid, x, y, vals, mu0, mu1, n0, n1, base=0):
    """grid [cells, comps] += Gaussian footprints (9 x 9 cells, periodic
    2 n1 x 2 n0) of vals [samples, comps] at x, y (cycles per cell)."""
    m = 4
    b0, b1 = torch.floor(2 * n0 * x).long() - m, torch.floor(2 * n1 * y).long() - m
    for i1 in range(2 * m + 1):
        w1 = torch.exp(-math.pi ** 2 / mu1 * ((b1 + i1) / (2.0 * n1) - y) ** 2)
        row = (n1 + b1 + i1) % (2 * n1)
        for i0 in range(2 * m + 1):
            w0 = torch.exp(-math.pi ** 2 / mu0 * ((b0 + i0) / (2.0 * n0) - x) ** 2)
            idx = base + row * (2 * n0) + (n0 + b0 + i0) % (2 * n0)
            grid.index_add_(0, idx, (w0 * w1)[:, None] * vals)


def _fourierrec64(rows, out):
    """out [nz, n, n] float64 <- fourierrec of filtered rows [nz, P, n]; slices
    k and k + nz/2 travel as one complex sinogram."""
    nz, P, n = rows.shape
    h, mu = nz // 2, math.log(1e3) / (2 * n * n)
    th = torch.as_tensor(_theta(P), device=DEV).to(torch.float64)
    r = ((torch.arange(n, device=DEV) - n // 2) / n).to(torch.float64)
    x, y = (r * torch.cos(th)[:, None]).reshape(-1), (-r * torch.sin(th)[:, None]).reshape(-1)
    x = torch.where(x >= 0.5, torch.full_like(x, 0.5 - 1e-5), x)
    y = torch.where(y >= 0.5, torch.full_like(y, 0.5 - 1e-5), y)
    s = _sign(torch.arange(n, device=DEV))
    s2 = _sign(torch.arange(4, 2 * n + 4, device=DEV))
    t = torch.arange(n, device=DEV)
    d = (t / n - 0.5).to(torch.float64)
    phi = torch.exp(mu * n * n * (d[None, :] ** 2 + d[:, None] ** 2)) / P * (1 - n % 4)
    c = ((t - n // 2) / n).to(torch.float64)
    phi = phi * ((4 * c[None, :] ** 2 + 4 * c[:, None] ** 2) < 1)
    step = max(1, min(h, int(2 ** 31 / (4 * n * n * 16))))
    for k0 in range(0, h, step):
        k1 = min(h, k0 + step)
        g = torch.complex(rows[k0:k1], rows[h + k0:h + k1])
        g = torch.fft.fft(g * s) * s * (4.0 / n * math.pi / (mu * 4 * n * n))
        vals = torch.view_as_real(g.reshape(k1 - k0, -1).t().contiguous()).reshape(P * n, -1)
        grid = torch.zeros((4 * n * n, vals.shape[1]), dtype=torch.float64, device=DEV)
        _spread64(grid, x, y, vals, mu, mu, n, n)
        grid = torch.view_as_complex(grid.view(2 * n, 2 * n, k1 - k0, 2))
        for k in range(k0, k1):
            f = grid[:, :, k - k0] * s2[:, None] * s2
            f = torch.fft.ifft2(f, norm="forward")
            f = (f * s2[:, None] * s2)[n // 2 + 1:n // 2 + 1 + n, n // 2:n // 2 + n] * phi
            out[k], out[h + k] = f.real, f.imag
    return out


def _linerec64(rows, out):
    """out [nz, n, n] <- bilinear line summation of rows [nz, P, n] (the voxel
    row z meets detector row z)."""
    nz, P, n = rows.shape
    th = torch.as_tensor(_theta(P), device=DEV).to(torch.float64)
    X = (torch.arange(n, device=DEV) - n // 2).to(torch.float64)
    out.zero_()
    for p in range(P):
        u = torch.cos(th[p]) * X[None, :] + torch.sin(th[p]) * X[:, None] + n // 2
        i = (u - 1e-5).trunc().long()
        ok = (i >= 0) & (i < n - 1)
        i = torch.where(ok, i, 0)
        w = u - i
        for z in range(nz):
            v = rows[z, p]
            out[z] += torch.where(ok, v[i] * (1 - w) + v[i + 1] * w, 0.0)
    out *= 4.0 / P
    return out.flip(1)


SYM16 = (
    5.764107394356608e-06, -4.418079054180866e-06, -0.0001011046640375809, 6.612766430523652e-05,
    0.000850728356483547, -0.0003755038256163555, -0.004381808863067106, 0.0007754538556196767,
    0.014174276451819888, 1.026142119842727e-05, -0.026075903837101934, 0.010176084591989107,
    0.028643708207463453, -0.09394878853561413, -0.08405148978060076, 0.3536233896498427,
    0.7532601221050154, 0.5154890124190248, -0.0029194240352577168, -0.13053811730498155,
    0.033833271475262855, 0.07200208133441333, -0.00665513643793778, -0.02531391691867016,
    0.0008761469298043955, 0.006229398424104775, -0.0004546791664901557, -0.001247791440191024,
    0.00011125575250768447, 0.0001751786877487489, -8.945414562934247e-06, -1.167075771969278e-05)


def _dwt64(x, lo, hi, axis):
    L, N = len(lo), x.shape[axis]
    out = (N + L - 1) // 2
    p = 2 * (out - 1) - N + L
    i = torch.arange(-(p // 2), N + (p + 1) // 2, device=DEV) % (2 * N)
    x = x.index_select(axis, torch.where(i >= N, 2 * N - 1 - i, i))
    a, b = 0, 0
    for j in range(L):
        t = x.narrow(axis, j, 2 * out - 1)[(slice(None),) * axis + (slice(None, None, 2),)]
        a, b = a + lo[j] * t, b + hi[j] * t
    return a, b


def _idwt64(lo, hi, g0, g1, axis):
    L, H = len(g0), lo.shape[axis]
    shape = list(lo.shape)
    shape[axis] = 2 * (H - 1) + L
    out = torch.zeros(shape, dtype=torch.float64, device=DEV)
    for j in range(L):
        out[(slice(None),) * axis + (slice(j, j + 2 * H - 1, 2),)] += g0[j] * lo + g1[j] * hi
    return out.narrow(axis, L - 2, shape[axis] - 2 * (L - 2))


def _fw64(data, level=7, sigma=1.0):
    """Fourier-wavelet ring removal of [P, nz, n] (float64)."""
    r0 = list(SYM16)
    d0 = r0[::-1]
    d1 = [(-1.0) ** (k + 1) * v for k, v in enumerate(r0)]
    h0, h1, g0, g1 = d0[::-1], d1[::-1], r0, d1[::-1]
    P, nz, n = data.shape
    npad = P + P // 8
    st = (npad - P) // 2
    x = torch.zeros((nz, npad, n), dtype=torch.float64, device=DEV)
    x[:, st:st + P] = data.to(torch.float64).permute(1, 0, 2)
    bands = []
    for _ in range(level):
        lo, hi = _dwt64(x, h0, h1, 2)
        x, lh = _dwt64(lo, h0, h1, 1)
        hl, hh = _dwt64(hi, h0, h1, 1)
        my = hl.shape[1]
        y = np.fft.ifftshift((np.arange(-my, my, 2) + 1) / 2)[:my // 2 + 1]
        damp = torch.as_tensor(-np.expm1(-y ** 2 / (2 * sigma ** 2)), device=DEV)[:, None]
        bands.append((lh, torch.fft.irfft(torch.fft.rfft(hl, dim=1) * damp, n=my, dim=1), hh))
    for lh, hl, hh in bands[::-1]:
        x = x[:, :hl.shape[1], :hl.shape[2]]
        x = _idwt64(_idwt64(x, lh, g0, g1, 1), _idwt64(hl, hh, g0, g1, 1), g0, g1, 2)
    return x[:, st:st + P, :n].permute(1, 0, 2).contiguous()


def _median64(x, size):
    """Running median along the last axis, mode reflect."""
    h, n = size // 2, x.shape[-1]
    i = torch.arange(-h, n + h, device=DEV) % (2 * n)
    x = x[..., torch.where(i >= n, 2 * n - 1 - i, i)]
    return torch.stack([r.unfold(-1, size, 1).median(-1).values for r in x])


def _vo_mask(fact, snr):
    """Stripe columns of the row statistics [nz, n], widened by one column."""
    n = fact.shape[1]
    s = fact.sort(1, descending=True).values
    x = torch.arange(n, device=DEV, dtype=torch.float64)
    nd = int(0.25 * n)
    xs, ys = x[nd:n - nd - 1], s[:, nd:n - nd - 1]
    dx = xs - xs.mean()
    slope = ((ys - ys.mean(1, keepdim=True)) * dx).sum(1) / (dx ** 2).sum()
    icpt = ys.mean(1) - slope * xs.mean()
    end = icpt + slope * (n - 1)
    noise = torch.clamp((end - icpt).abs(), min=1e-6)
    up = ((s[:, 0] - icpt).abs() / noise >= snr)[:, None] & (
        fact > (icpt + noise * snr * 0.5)[:, None])
    dn = ((s[:, -1] - end).abs() / noise >= snr)[:, None] & (
        fact <= (end - noise * snr * 0.5)[:, None])
    m = up | dn
    w = m.clone()
    w[:, 1:] |= m[:, :-1]
    w[:, :-1] |= m[:, 1:]
    return w


def _vo64(t, snr=3.0, la=61, sm=21):
    """Vo's all-stripe removal of rows [nz, P, n] (float64)."""
    nz, P, n = t.shape
    i = torch.arange(-5, P + 5, device=DEV) % (2 * P)
    cs = torch.cumsum(t[:, torch.where(i >= P, 2 * P - 1 - i, i)], 1)
    cs = torch.cat((torch.zeros_like(cs[:, :1]), cs), 1)
    diff = (t - (cs[:, 10:10 + P] - cs[:, :P]) / 10).abs().sum(1)
    mask = _vo_mask(diff / _median64(diff, la), snr)
    mask[:, :2] = False
    mask[:, -2:] = False
    for z in range(nz):
        good, miss = (~mask[z]).nonzero()[:, 0], mask[z].nonzero()[:, 0]
        if len(miss):
            k = torch.searchsorted(good, miss)
            a, b = good[k - 1], good[k]
            t[z][:, miss] = t[z][:, a] + (miss - a) * (t[z][:, b] - t[z][:, a]) / (b - a)
    drop = int(0.05 * P)
    srt, ids = t.sort(dim=1, stable=True)
    smooth = _median64(srt, la)
    fact = srt[:, drop:P - drop].mean(1) / smooth[:, drop:P - drop].mean(1)
    mask = _vo_mask(fact, snr)
    back = torch.empty_like(t).scatter_(1, ids, smooth)
    t = torch.where(mask[:, None, :], back, t / fact[:, None, :])
    srt, ids = t.sort(dim=1, stable=True)
    return torch.empty_like(t).scatter_(1, ids, _median64(srt, sm))


def _paganin64(x):
    """Paganin phase retrieval of projections [P, dy, dz] (float64)."""
    _, dy, dz = x.shape
    px, dist, alpha = 0.65e-4, 5.0, 1e-3
    wl = 2 * 3.14159265359 * 6.58211928e-19 * 299792458e+2 / 20.0

    def pad(d):
        return int((2 ** math.ceil(math.log2(d + math.ceil(3.14159265359 * wl * dist / px ** 2)))
                    - d) * 0.5)

    def coord(k):
        return torch.arange(-(k - 1), k, 2, device=DEV, dtype=torch.float64) * (0.5 / ((k - 1) * px))

    py, pz = pad(dy), pad(dz)
    w2 = coord(dy + 2 * py)[:, None] ** 2 + coord(dz + 2 * pz)[None, :] ** 2
    f = torch.fft.fftshift(1 / (wl * dist * w2 / (4 * 3.14159265359) + alpha))
    f = f / f.max()
    iy = torch.clamp(torch.arange(-py, dy + py, device=DEV), 0, dy - 1)
    iz = torch.clamp(torch.arange(-pz, dz + pz, device=DEV), 0, dz - 1)
    out = torch.empty_like(x)
    for k in range(x.shape[0]):
        g = torch.fft.ifft2(torch.fft.fft2(x[k][iy][:, iz].to(torch.complex128)) * f)
        out[k] = g.real[py:py + dy, pz:pz + dz]
    return out


def _lamino64(data, c):
    """The laminography chain of [P, deth, n] projections, float64."""
    n, P, deth, rh = c["n"], c["nproj"], c["deth"], c["rh"]
    phi = math.pi / 2 + 30.0 / 180 * math.pi
    rows = _filter64(data.to(torch.float64), c["filter"], n / 2)
    ck = _sign(torch.arange(max(n, deth), device=DEV))
    s1 = torch.fft.rfft2(rows * ck[:deth, None] * ck[:n]) * -(ck[:deth, None] * ck[:n // 2 + 1])
    s1 /= deth * n
    del rows
    mu = math.log(1e3) / (2 * n * n)
    th = torch.as_tensor(_theta(P, 2 * math.pi), device=DEV).to(torch.float64)[:, None, None]
    tx = torch.arange(n, device=DEV)
    ku = ((tx - n / 2) / n).to(torch.float64)
    s2s = _sign(torch.arange(4, 2 * n + 4, device=DEV))
    t = torch.arange(n, device=DEV)
    ker = torch.exp(-mu * ((t - n // 2) ** 2)[None, :] - mu * ((t - n // 2) ** 2)[:, None])
    nrow = deth // 2 + 1
    s2 = torch.empty((nrow, n, n), dtype=torch.complex128, device=DEV)
    step = max(1, int(2 ** 22 / (P * n)))
    for r0 in range(0, nrow, step):
        r = torch.arange(r0, min(nrow, r0 + step), device=DEV)
        kv = ((r - deth / 2) / deth).to(torch.float64)[None, :, None]
        x = ku * torch.cos(th) + kv * torch.sin(th) * math.cos(phi)
        y = ku * torch.sin(th) - kv * torch.cos(th) * math.cos(phi)
        x, y = (q.clamp(-0.5 + 1e-5, 0.5 - 1e-5).reshape(-1) for q in (x, y))
        v = torch.where(tx <= n // 2, s1[:, r][:, :, torch.clamp(tx, max=n // 2)],
                        s1[:, (deth - r) % deth][:, :, torch.clamp(n - tx, max=n // 2)].conj())
        v = torch.view_as_real((v * (math.pi / (mu * math.sqrt(P)))).contiguous()).reshape(-1, 2)
        base = ((r - r0) * (4 * n * n))[None, :, None].expand(P, -1, n).reshape(-1)
        g = torch.zeros((len(r) * 4 * n * n, 2), dtype=torch.float64, device=DEV)
        _spread64(g, x, y, v, mu, mu, n, n, base)
        g = torch.view_as_complex(g).view(-1, 2 * n, 2 * n) * s2s[:, None] * s2s
        g = torch.fft.ifft2(g, norm="forward") * s2s[:, None] * s2s
        g = g.flip(1)[:, 2 * n - 1 - (n - 1 + n // 2):, n // 2:n // 2 + n][:, :n]
        s2[r] = g / ker / (n * n)
    del s1, g
    n2 = rh
    mu2 = math.log(1e3) / (2.0 * n2 * n2)
    tz = torch.arange(deth, device=DEV)
    z = (((tz - deth / 2) / deth) * math.sin(phi)).to(torch.float64)
    grid = torch.zeros((2 * n2, n, n), dtype=torch.complex128, device=DEV)
    b = torch.floor(2 * n2 * z).long() - 4
    bl, zl = b.tolist(), z.tolist()
    for k in range(deth):
        v = s2[k] if k <= deth // 2 else s2[deth - k].conj()
        for j in range(9):
            w = math.sqrt(math.pi / (mu2 * n)) * math.exp(
                -math.pi ** 2 / mu2 * ((bl[k] + j) / (2.0 * n2) - zl[k]) ** 2)
            grid[(n2 + bl[k] + j) % (2 * n2)] += w * v
    s = _sign(torch.arange(4, 2 * n2 + 4, device=DEV))[:, None, None]
    grid = torch.fft.ifft(grid * s, dim=0, norm="forward") * s
    tz = torch.arange(n2, device=DEV)
    ker = torch.exp(-mu2 * ((tz - n2 // 2) ** 2).to(torch.float64))[:, None, None]
    return grid[n2 // 2:n2 // 2 + n2].real / ker / (2 * n2)


def exact(case, seed):
    c, kind = case, case["kind"]
    n, P = c["n"], c["nproj"]
    if kind == "lamino":
        return _lamino64(_lam_rows(seed, n, P, c["deth"]), c)
    if kind == "fw":
        return _fw64(_norm_rows(seed, n, P, c["nz"]))
    if kind == "phase":
        x = _paganin64(_prep64(*_frames(seed, n, P, c["nz"]), log=False))
        return -torch.log(torch.where(x <= 0, torch.ones_like(x), x))
    if c.get("algorithm") == "lprec":
        # lprec's value is defined by texture fetches with 8-bit fixed-point
        # weights between log-polar grids: it has no 64-bit counterpart
        return None
    if kind == "try":
        rows = _prep64(*_frames(seed, n, P, 1)).permute(1, 0, 2)
        S = c["centers"]
        sht = np.zeros(64, np.float32)
        sht[:S] = _shifts(c)
        rows = _filter64(rows.repeat(64, 1, 1), c["filter"], _center(c), sht)
        return _fourierrec64(rows, torch.empty((64, n, n), dtype=torch.float64, device=DEV))[:S]
    nz = c["nz"]
    data, dark, flat = _frames(seed, n, P, nz, stripes=30 if kind == "vo" else 0)
    ncz = 8 if kind == "scan" else nz
    out = torch.empty((nz, n, n), dtype=torch.float64, device=DEV)
    for z0 in range(0, nz, ncz):
        z1 = min(nz, z0 + ncz)
        if kind == "vo":
            rows = _vo64(_prep64(data, dark, flat, log=False).permute(1, 0, 2).contiguous())
            rows = -torch.log(torch.where(rows <= 0, torch.ones_like(rows), rows))
        else:
            rows = torch.zeros((ncz, P, n), dtype=torch.float64, device=DEV)
            rows[:z1 - z0] = _prep64(data[:, z0:z1], dark[:, z0:z1],
                                     flat[:, z0:z1]).permute(1, 0, 2)
        rows = _filter64(rows, c["filter"], _center(c))
        if c.get("algorithm") == "linerec":
            return _linerec64(rows, out)
        part = _fourierrec64(rows, torch.empty((ncz, n, n), dtype=torch.float64, device=DEV))
        out[z0:z1] = part[:z1 - z0]
    return out
