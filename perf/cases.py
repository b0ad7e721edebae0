"""The workloads that the framework's speed is judged on, one pass each through its public entry points.

A mapmaker's program does four things: it builds a noise model per TOD (``Tod.set_noise``), projects between maps and
timestreams (``SkyMap.map2tod`` / ``tod2map``, ``PolMap``), filters timestreams with the noise model
(``NoiseSmoothedSVD.apply_noise``) and iterates the operator that chains these (``TodVec.dot``, ``run_pcg``).  The
cases take each of them at the sizes of this repository's configurations (``minkasi_gb300.synth.CONFIGS``): the 64
detector TOD on a 256 x 256 map, the 256 detector TODs on a 1024 x 1024 map, the mixed-detector batch on a 2048 x 2048
map, and the small calls of its tests.

Inputs: daisy scans (petal period 22 s at 180 Hz) of a square detector grid, white plus 1/f timestreams with a common
mode, inverse spectra with a 1/f knee, all from the seed.
"""
import math

import numpy as np
import torch

from minkasi_gb300.maps import Mapset, SkyMap
from minkasi_gb300.noise import NoiseSmoothedSVD
from minkasi_gb300.pcg import run_pcg
from minkasi_gb300.polmap import PolMap
from minkasi_gb300.projections import jacobi_precon
from minkasi_gb300.synth import CONFIGS, tod_shapes
from minkasi_gb300.tods import Tod, TodVec
from minkasi_gb300.truncate import truncated_length

FSAMP, PETAL_S, KNEE_HZ = 180.0, 22.0, 1.0


def listed():
    return [
        # the smallest call: a test-sized TOD scattered onto a small map (launch and call cost)
        dict(name="tod2map_f64_small", kind="tod2map", dtype="f64", ntod=1, ndet=8, ndata=3001, side=64, pix=4.0),
        # the two projections at the 1024 x 1024 configuration, TOD by TOD, in double precision
        dict(name="map2tod_f64", kind="map2tod", dtype="f64", ntod=4, ndet=256, ndata=130978, side=1024, pix=1.0),
        dict(name="tod2map_f64", kind="tod2map", dtype="f64", ntod=4, ndet=256, ndata=130978, side=1024, pix=1.0),
        # polarised projections (IQU), both directions, on the 64 detector TOD
        dict(name="pol_f64", kind="pol", dtype="f64", ntod=1, ndet=64, ndata=65341, side=256, pix=2.0),
        # the noise model that every TOD needs before anything is solved
        dict(name="set_noise_f64", kind="build", dtype="f64", ntod=1, ndet=64, ndata=65341, side=0, pix=0.0),
        # the filter with default options on an odd detector count, double precision
        dict(name="noise_f64_odd", kind="noise", dtype="f64", ntod=1, ndet=53, ndata=20001, rot=0),
        # the filter at full size, double precision, on the sliced tensor-core rotation the operator selects
        dict(name="noise_f64", kind="noise", dtype="f64", ntod=1, ndet=256, ndata=130978, rot=4),
        # the filter at full size, single precision, tensor-core rotation; 2 (n - 1) has a large prime factor here,
        # as about a third of the truncated lengths do
        dict(name="noise_f32_prime", kind="noise", dtype="f32", ntod=1, ndet=256, ndata=144278, rot=2),
        # the operator of the mixed-precision solver's inner iteration: one small TOD, and a batch of TODs with
        # uneven lengths and detector counts on the 2048 x 2048 map
        dict(name="dot_f32_one", kind="dot", dtype="f32", ntod=1, ndet=64, ndata=65341, side=256, pix=2.0),
        dict(name="dot_f32_batch", kind="dot", dtype="f32", ntod=10, ndet=0, ndata=0, side=2048, pix=0.5),
        # the double-precision operator (plain solves, and the residual replacements of the mixed one)
        dict(name="dot_f64", kind="dot", dtype="f64", ntod=2, ndet=256, ndata=130978, side=1024, pix=1.0),
        # a whole solve of the plain method, a few iterations
        dict(name="pcg_f64", kind="pcg", dtype="f64", ntod=1, ndet=64, ndata=65341, side=256, pix=2.0),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["map2tod", "tod2map", "noise", "noise", "dot", "dot"])
    dtype = rng.choice(["f32", "f64"])
    if kind in ("map2tod", "tod2map"):
        side, pix = rng.choice([(64, 4.0), (256, 2.0), (1024, 1.0), (2048, 0.5)])
        return dict(kind=kind, dtype=dtype, ntod=rng.randint(1, 4), ndet=rng.randint(3, 256), ndata=log_int(1000, 130000),
                    side=side, pix=pix)
    if kind == "noise":
        rot = rng.choice([0, 4] if dtype == "f64" else [0, 2])
        ndet = rng.choice([32, 64, 128, 256]) if rot == 2 else rng.randint(2, 256)
        n = log_int(1000, 130000)
        return dict(kind=kind, dtype=dtype, ntod=1, ndet=ndet, ndata=rng.choice([n, truncated_length(n)]), rot=rot)
    side, pix = rng.choice([(256, 2.0), (1024, 1.0), (2048, 0.5)])
    return dict(kind=kind, dtype=dtype, ntod=rng.randint(1, 3), ndet=rng.choice([32, 64, 128, 256]),
                ndata=truncated_length(log_int(20000, 130000)), side=side, pix=pix)


# ---- inputs ------------------------------------------------------------------
def _dtype(case):
    return torch.float64 if case["dtype"] == "f64" else torch.float32


def _gen(seed, k):
    return torch.Generator(device="cuda").manual_seed((int(seed) * 1000003 + 7919 * k + 17) % (1 << 62))


def _shapes(case):
    """(ndet, ndata) per TOD; the mixed batch (ndet 0) takes consecutive TODs of the 200-TOD configuration: 32 to
    256 detectors, 51,451 to 563,201 samples, two of ten with a large prime factor in 2 (n - 1)."""
    if case["ndet"]:
        return [(case["ndet"], case["ndata"])] * case["ntod"]
    return tod_shapes(CONFIGS["c4"])[3:3 + case["ntod"]]


def _ipix(case, seed, k, ndet, n):
    """int32 pixel indices of a daisy scan of a square detector grid."""
    side, pix = case["side"], case["pix"]
    rng = np.random.default_rng([int(seed) % (1 << 31), k])
    t = torch.arange(n, device="cuda", dtype=torch.float64) / FSAMP
    w1 = 2 * math.pi / PETAL_S
    ph1, ph2, rr, aa = (float(v) for v in rng.uniform(0, 1, size=4))
    half = side * pix / 2  # arcsec from the map's centre to its edge
    r = 0.35 * half * torch.sin(w1 * t + 2 * math.pi * ph1)
    th = w1 / 1.6180339887 * t + 2 * math.pi * ph2
    cr = 0.25 * half * math.sqrt(rr)
    nr = max(1, int(math.isqrt(ndet)))
    d = torch.arange(ndet, device="cuda", dtype=torch.float64)
    pitch = min(10.0, 0.5 * half / nr)
    ox = (torch.remainder(d, nr) - (nr - 1) / 2) * pitch
    oy = (torch.div(d, nr, rounding_mode="floor") - (ndet / nr - 1) / 2) * pitch
    x = cr * math.cos(2 * math.pi * aa) + r * torch.cos(th)
    y = cr * math.sin(2 * math.pi * aa) + r * torch.sin(th)
    px = torch.round((x[None, :] + ox[:, None]) / pix + side / 2).clamp(0, side - 1)
    py = torch.round((y[None, :] + oy[:, None]) / pix + side / 2).clamp(0, side - 1)
    return (px * side + py).to(torch.int32).contiguous()


def _stream(seed, k, ndet, n):
    """White plus 1/f noise (1 mK) and a 3 mK common mode, double precision, (ndet, n)."""
    g = _gen(seed, 3 * k)
    f = torch.fft.rfftfreq(n, d=1.0 / FSAMP, device="cuda", dtype=torch.float64)
    f[0] = f[1] if n > 1 else 1.0
    amp = torch.sqrt(1.0 + (KNEE_HZ / f) ** 2)

    def rows(m):
        w = torch.randn((m, n), generator=g, device="cuda", dtype=torch.float64)
        return torch.fft.irfft(torch.fft.rfft(w) * amp, n=n)

    gains = 1 + 0.02 * torch.randn((ndet, 1), generator=g, device="cuda", dtype=torch.float64)
    cm = rows(1)
    return (1e-3 * rows(ndet) + 3e-3 * gains * cm / cm.std()).contiguous()


def _sky(case, seed, comps=1):
    side = case["side"]
    g = _gen(seed, 1001)
    x = (torch.arange(side, device="cuda", dtype=torch.float64) - side / 2) * case["pix"]
    r2 = x[:, None] ** 2 + x[None, :] ** 2
    m = (-1e-3 / torch.sqrt(1 + r2 / 900.0))[..., None].expand(side, side, comps)
    m = m + 1e-4 * torch.randn((side, side, comps), generator=g, device="cuda", dtype=torch.float64)
    return (m[..., 0] if comps == 1 else m).contiguous()


def _model(seed, k, ndet, n):
    """(v, vT, inverse spectra) of a noise model: an orthogonal rotation and 1/f-knee inverse spectra."""
    g = _gen(seed, 3 * k + 1)
    q = torch.linalg.qr(torch.randn((ndet, ndet), generator=g, device="cuda", dtype=torch.float64))[0]
    f = torch.arange(n, device="cuda", dtype=torch.float64) * (FSAMP / 2 / max(n - 1, 1))
    f[0] = f[1]
    knee = 0.2 + 2.0 * torch.rand((ndet, 1), generator=g, device="cuda", dtype=torch.float64)
    w = 1.0 / (2e-6 * n * (1.0 + (knee / f) ** 2))
    w[:, 0] = 0
    return q.T.contiguous(), q.contiguous(), w.contiguous()


def _tods(case, seed, models):
    tv = TodVec()
    for k, (nd, n) in enumerate(_shapes(case)):
        tod = Tod({"ipix": _ipix(case, seed, k, nd, n), "dat_calib": torch.empty((nd, n), dtype=torch.float64, device="meta")})
        if models:
            tod.noise = NoiseSmoothedSVD.from_arrays(*_model(seed, k, nd, n))
        tv.add_tod(tod)
    return tv


def prepare(case, seed):
    kind, dt = case["kind"], _dtype(case)
    s = {"case": case, "kind": kind}
    if kind in ("map2tod", "tod2map"):
        s["tods"] = _tods(case, seed, False)
        s["map"] = SkyMap.from_shape(case["side"], case["side"], dtype=dt)
        if kind == "map2tod":
            s["map"].assign(_sky(case, seed))
            s["dats"] = [torch.empty((nd, n), dtype=dt, device="cuda") for nd, n in _shapes(case)]
        else:
            s["dats"] = [_stream(seed, k, nd, n).to(dt) for k, (nd, n) in enumerate(_shapes(case))]
    elif kind == "pol":
        (nd, n), = _shapes(case)
        s["tods"] = _tods(case, seed, False)
        tg = torch.rand((nd, n), generator=_gen(seed, 5), device="cuda", dtype=torch.float64) * 2 * math.pi
        s["tods"].tods[0].info["twogamma_saved"] = tg
        lims = [0.0, 1e-3, 0.0, 1e-3]
        s["map"] = PolMap(lims, 1e-5, "IQU", nx=case["side"], ny=case["side"], dtype=dt)
        s["map"].assign(_sky(case, seed, 3))
        s["out"] = PolMap(lims, 1e-5, "IQU", nx=case["side"], ny=case["side"], dtype=dt)
        s["dat"] = torch.empty((nd, n), dtype=dt, device="cuda")
    elif kind == "build":
        (nd, n), = _shapes(case)
        s["tod"] = Tod({"dat_calib": _stream(seed, 0, nd, n)})
    elif kind == "noise":
        (nd, n), = _shapes(case)
        s["noise"] = NoiseSmoothedSVD.from_arrays(*_model(seed, 0, nd, n))
        s["dat"] = _stream(seed, 0, nd, n).to(dt)
    elif kind == "dot":
        s["tods"] = _tods(case, seed, True)
        m = SkyMap.from_shape(case["side"], case["side"], dtype=dt)
        m.assign(_sky(case, seed))
        s["x"] = Mapset()
        s["x"].add_map(m)
        s["tods"].engine(s["x"].maps[0])
    else:
        s["tods"] = _tods(case, seed, True)
        m = SkyMap.from_shape(case["side"], case["side"], dtype=dt)
        s["x0"] = Mapset()
        s["x0"].add_map(m)
        hits = SkyMap.from_shape(case["side"], case["side"], dtype=dt)
        for k, ((nd, n), tod) in enumerate(zip(_shapes(case), s["tods"].tods)):
            m.tod2map(tod, _rhs_stream(seed, k, nd, n).to(dt))
            hits.tod2map(tod, torch.ones((nd, n), dtype=dt, device="cuda"))
        s["b"] = Mapset()
        s["b"].add_map(m)
        s["precon"] = jacobi_precon(hits)
        s["tods"].engine(s["b"].maps[0])
    return s


def _rhs_stream(seed, k, ndet, n):
    """A filtered timestream for the right-hand side: zero-mean white noise at the filter's scale."""
    return torch.randn((ndet, n), generator=_gen(seed, 3 * k + 2), device="cuda", dtype=torch.float64)


PCG_ITERS = 10


def run(s):
    kind = s["kind"]
    if kind == "map2tod":
        for tod, dat in zip(s["tods"].tods, s["dats"]):
            s["map"].map2tod(tod, dat, do_add=False)
        return s["dats"]
    if kind == "tod2map":
        s["map"].clear()
        for tod, dat in zip(s["tods"].tods, s["dats"]):
            s["map"].tod2map(tod, dat)
        return s["map"].map
    if kind == "pol":
        tod = s["tods"].tods[0]
        s["map"].map2tod(tod, s["dat"], do_add=False)
        s["out"].clear()
        s["out"].tod2map(tod, s["dat"])
        return [s["dat"], s["out"].map]
    if kind == "build":
        s["tod"].set_noise(NoiseSmoothedSVD, fwhm=50.0)
        noise = s["tod"].noise
        return {"v": noise.v, "vT": noise.vT, "mywt": noise.mywt, "weights": noise.get_det_weights()}
    if kind == "noise":
        return s["noise"].apply_noise(s["dat"], rot_mode=s["case"]["rot"])
    if kind == "dot":
        return s["tods"].dot(s["x"]).maps[0].map
    x = run_pcg(s["b"], s["x0"], s["tods"], precon=s["precon"], maxiter=PCG_ITERS, verbose=False)
    return x.maps[0].map


# ---- what a pass cannot do without ---------------------------------------------
def work(case):
    es = 8 if case["dtype"] == "f64" else 4
    shapes = _shapes(case)
    S = sum(nd * n for nd, n in shapes)
    npix = case.get("side", 0) ** 2
    fft = sum(nd * 2.5 * n * math.log2(n) for nd, n in shapes)  # one DCT-I of each row
    rot = sum(2.0 * nd * nd * n for nd, n in shapes)
    ops = sum(2 * nd * nd * es for nd, n in shapes)
    kind = case["kind"]
    if kind in ("map2tod", "tod2map"):
        return {"bytes": S * (4 + es) + npix * es, "flops": float(S if kind == "tod2map" else 0)}
    if kind == "pol":  # both directions: index, angles' cosine and sine, sample; the three-component maps
        return {"bytes": 2 * S * (4 + 3 * es) + 2 * 3 * npix * es, "flops": 8.0 * S}
    if kind == "build":  # the Gram matrix, the rotation, the spectrum and its smoothing (three transforms)
        return {"bytes": 2 * S * es, "flops": 2 * rot + 3 * fft}
    if kind == "noise":
        return {"bytes": 3 * S * es + ops, "flops": 2 * rot + 2 * fft}
    one = {"bytes": 2 * 4 * S + S * es + ops + 2 * npix * es, "flops": 2 * rot + 2 * fft + S}
    if kind == "dot":
        return one
    return {k: v * (PCG_ITERS + 1) for k, v in one.items()}


# ---- the same in 64 bits by plain torch ------------------------------------------
def _dct1(x):
    """Unnormalised DCT-I of each row: the real DFT of its even extension."""
    out = torch.empty_like(x)
    for i in range(0, x.shape[0], 32):
        b = x[i:i + 32]
        out[i:i + 32] = torch.fft.rfft(torch.cat([b, b[:, 1:-1].flip(1)], dim=1)).real
    return out


def _filter(v, vT, w, d):
    x = _dct1(_dct1(v @ d) * w[:, :d.shape[1]])
    x[:, 0] *= 0.5
    x[:, -1] *= 0.5
    return vT @ x


def _apply(case, seed, parts, x):
    out = torch.zeros_like(x)
    for k, (nd, n) in enumerate(_shapes(case)):
        ip, mod = parts(k, nd, n)
        out.index_add_(0, ip, _filter(*mod, x[ip].view(nd, n)).reshape(-1))
    return out


def exact(case, seed):
    kind, dt = case["kind"], _dtype(case)
    shapes = _shapes(case)

    def parts(k, nd, n):
        return _ipix(case, seed, k, nd, n).reshape(-1).long(), _model(seed, k, nd, n)

    if kind == "map2tod":
        sky = _sky(case, seed).to(dt).double().reshape(-1)
        return [sky[_ipix(case, seed, k, nd, n).reshape(-1).long()].view(nd, n) for k, (nd, n) in enumerate(shapes)]
    if kind == "tod2map":
        m = torch.zeros(case["side"] ** 2, dtype=torch.float64, device="cuda")
        for k, (nd, n) in enumerate(shapes):
            ip = _ipix(case, seed, k, nd, n).reshape(-1).long()
            m.index_add_(0, ip, _stream(seed, k, nd, n).to(dt).double().reshape(-1))
        return m.view(case["side"], case["side"])
    if kind == "pol":
        (nd, n), = shapes
        ip = _ipix(case, seed, 0, nd, n).reshape(-1).long()
        tg = (torch.rand((nd, n), generator=_gen(seed, 5), device="cuda", dtype=torch.float64) * 2 * math.pi).reshape(-1)
        st = torch.stack([torch.ones_like(tg), torch.cos(tg), torch.sin(tg)], dim=1)
        sky = _sky(case, seed, 3).to(dt).double().reshape(-1, 3)
        dat = (sky[ip] * st).sum(1)
        m = torch.zeros_like(sky)
        m.index_add_(0, ip, st * dat[:, None])
        return [dat.view(nd, n), m.view(case["side"], case["side"], 3)]
    if kind == "build":
        # the rotation's rows are fixed up to sign, the spectra and weights altogether
        (nd, n), = shapes
        d = _stream(seed, 0, nd, n)
        u = torch.linalg.svd(d, full_matrices=False)[0]
        x = _dct1(u.T.contiguous() @ d) ** 2
        sig = 50.0 / math.sqrt(8 * math.log(2))
        ker = torch.exp(-0.5 * (torch.arange(n, device="cuda", dtype=torch.float64) / sig) ** 2)
        ker = ker / (ker[0] + ker[-1] + 2 * ker[1:-1].sum())
        w = _dct1(_dct1(x) * _dct1(ker[None, :])) / (2 * (n - 1))
        w[:, 1:] = 1.0 / w[:, 1:]
        w[:, 0] = 0
        wt = 2.0 * torch.diagonal(u @ (w.sum(1)[:, None] * u.T)).clone()
        return {"v": None, "vT": None, "mywt": w, "weights": wt}
    if kind == "noise":
        (nd, n), = shapes
        return _filter(*_model(seed, 0, nd, n), _stream(seed, 0, nd, n).to(dt).double())
    if kind == "dot":
        x = _sky(case, seed).to(dt).double().reshape(-1)
        return _apply(case, seed, parts, x).view(case["side"], case["side"])
    b = torch.zeros(case["side"] ** 2, dtype=torch.float64, device="cuda")
    hits = torch.zeros_like(b)
    for k, (nd, n) in enumerate(shapes):
        ip = _ipix(case, seed, k, nd, n).reshape(-1).long()
        b.index_add_(0, ip, _rhs_stream(seed, k, nd, n).to(dt).double().reshape(-1))
        hits.index_add_(0, ip, torch.ones(nd * n, dtype=torch.float64, device="cuda"))
    kept = [parts(k, nd, n) for k, (nd, n) in enumerate(shapes)]
    M = torch.where(hits > 0, 1.0 / hits.clamp(min=1.0), torch.zeros_like(hits))
    x, r = torch.zeros_like(b), b.clone()
    z = M * r
    p, zr = z.clone(), torch.dot(r, z)
    for _ in range(PCG_ITERS):
        ap = _apply(case, seed, lambda k, nd, n: kept[k], p)
        a = zr / torch.dot(p, ap)
        x, r = x + a * p, r - a * ap
        z = M * r
        new = torch.dot(r, z)
        p, zr = z + (new / zr) * p, new
    return x.view(case["side"], case["side"])
