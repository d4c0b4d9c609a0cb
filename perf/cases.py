"""The work that users of the transform engine have it do, as measurable cases.

A case names a kind of call, sizes and options.  The kinds are the public entry
points that programs built on libsharp (alm2map_cxx, anafast_cxx, smoothing_cxx,
conviqt) and the torch callers use:

    synth    healpix.alm2map / alm2map_spin / alm2map_pol
    anal     healpix.map2alm / map2alm_spin / map2alm_pol
    round    healpix.alm2map_pol, then healpix.map2alm_pol of its maps
    iter     healpix.map2alm_iter (Jacobi sweeps, the body of anafast_cxx)
    der1     healpix.alm2map_der1 (map and first derivatives)
    grad     autograd.alm2map: chi-square of T, Q, U maps and its a_lm gradient
    sets     execute_device, alm2map and map2alm of several T+QU sets per call
    batch    execute_batch, an uneven list of spin-0 and spin-2 jobs, both ways
    grid     execute_device on a Gauss-Legendre grid (odd rings, any spin, float I/O)
    host     execute on host arrays (the drop-in call of a C caller), both ways

The a_lm are drawn from C_l = (l+1)^-2 exp(-l(l+1) sigma^2) with sigma of about
a pixel, E 0.1 and B 0.01 of T; maps are noise with a large-scale signal.
"""
import functools
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "planck-levels_b200"))
import sharp_b200 as sb  # noqa: E402
from sharp_b200 import autograd as sa  # noqa: E402
from sharp_b200 import healpix as hp  # noqa: E402


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest transforms a program makes (masks, low-resolution maps, tests): one
        # temperature map each way at Nside 64, where the latency of a call counts
        {"name": "synth_t_n64", "kind": "synth", "nside": 64, "lmax": 128, "comps": "T"},
        {"name": "anal_t_n64", "kind": "anal", "nside": 64, "lmax": 128, "comps": "T"},
        # a C caller with a map and a_lm in host memory (anafast_cxx, alm2map_cxx through the
        # drop-in): alm2map and map2alm of one low-resolution map, copies included
        {"name": "host_t_n256", "kind": "host", "nside": 256, "lmax": 512},
        # point-source and lensing work: a map and its derivatives at l = 3 Nside - 1
        {"name": "der1_n256_l767", "kind": "der1", "nside": 256, "lmax": 767},
        # beam convolution on a Gauss-Legendre grid: odd rings, single-precision arrays,
        # three simultaneous spin-1 transforms, both directions
        {"name": "grid_f32_l500", "kind": "grid", "lmax": 500, "mmax": 500, "nrings": 501,
         "nphi": 1001, "spin": 1, "ntrans": 3, "double": False},
        # map-domain chi-square of a polarised map and its gradient (a sampler's step)
        {"name": "grad_pol_n512", "kind": "grad", "nside": 512, "lmax": 1024,
         "precision": "fp64"},
        # many maps of mixed resolution and spin in one call (simulations), reduced precision
        {"name": "batch_mixed_48_16", "kind": "batch", "nside": 1024, "spin0": 48, "spin2": 16,
         "mixed": True},
        # anafast with three Jacobi sweeps at Nside 1024
        {"name": "iter3_t_n1024", "kind": "iter", "nside": 1024, "lmax": 2048, "sweeps": 3},
        # a polarised full-resolution map, each way (synfast/anafast at Nside 2048)
        {"name": "synth_pol_n2048", "kind": "synth", "nside": 2048, "lmax": 4096,
         "comps": "TQU"},
        {"name": "anal_pol_n2048", "kind": "anal", "nside": 2048, "lmax": 4096, "comps": "TQU"},
        # twelve polarised simulations at full resolution in the reduced-precision form
        {"name": "sets_mixed_n2048", "kind": "sets", "nside": 2048, "lmax": 4096, "ntrans": 12,
         "mixed": True},
        # the largest: a polarised round trip at Nside 4096
        {"name": "round_pol_n4096", "kind": "round", "nside": 4096, "lmax": 8192},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _nside(rng, lo, hi):
    """Mostly powers of two, as maps are stored, sometimes any other Nside of the range."""
    if rng.random() < 0.65:
        k = rng.randint(math.ceil(math.log2(lo)), math.floor(math.log2(hi)))
        return 1 << k
    return _log_int(rng, lo, hi)


def _lmax(rng, nside):
    return max(8, min(8192, int(nside * rng.uniform(1.4, 3.0)) - rng.randint(0, 1)))


def draw(rng: random.Random):
    kind = rng.choice(["synth", "synth", "anal", "anal", "round", "iter", "der1", "grad", "sets",
                       "batch", "grid", "host"])
    if kind in ("synth", "anal"):
        nside = _nside(rng, 16, 2048)
        lmax = min(4500, _lmax(rng, nside))
        return {"kind": kind, "nside": nside, "lmax": lmax, "comps": rng.choice(["T", "QU", "TQU"])}
    if kind == "round":
        nside = _nside(rng, 64, 2048)
        return {"kind": kind, "nside": nside, "lmax": min(4500, _lmax(rng, nside))}
    if kind == "iter":
        nside = _nside(rng, 32, 1024)
        return {"kind": kind, "nside": nside, "lmax": _lmax(rng, nside),
                "sweeps": rng.randint(1, 3)}
    if kind == "der1":
        nside = _nside(rng, 32, 1024)
        return {"kind": kind, "nside": nside, "lmax": _lmax(rng, nside)}
    if kind == "grad":
        nside = _nside(rng, 32, 1024)
        return {"kind": kind, "nside": nside, "lmax": min(2500, _lmax(rng, nside)),
                "precision": rng.choice(["fp64", "mixed"])}
    if kind == "sets":
        nside = _nside(rng, 64, 1024)
        return {"kind": kind, "nside": nside, "lmax": min(2500, _lmax(rng, nside)),
                "ntrans": rng.randint(2, 13), "mixed": rng.random() < 0.6}
    if kind == "batch":
        nside = 1 << rng.randint(7, 10)
        return {"kind": kind, "nside": nside, "spin0": rng.randint(3, 48),
                "spin2": rng.randint(2, 16), "mixed": rng.random() < 0.5}
    if kind == "grid":
        lmax = _log_int(rng, 24, 2000)
        mmax = lmax if rng.random() < 0.6 else rng.randint(max(4, lmax // 8), lmax)
        return {"kind": kind, "lmax": lmax, "mmax": mmax, "nrings": lmax + rng.randint(1, 12),
                "nphi": 2 * mmax + rng.randint(1, 16), "spin": rng.choice([0, 0, 1, 2, 3]),
                "ntrans": rng.randint(1, 6), "double": rng.random() < 0.5}
    nside = _nside(rng, 16, 512)
    return {"kind": "host", "nside": nside, "lmax": _lmax(rng, nside)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
_EBSCALE = {"T": 1.0, "E": 0.1, "B": 0.01}


def _nalm(lmax, mmax=None):
    mmax = lmax if mmax is None else mmax
    return (mmax + 1) * (mmax + 2) // 2 + (mmax + 1) * (lmax - mmax)


@functools.lru_cache(maxsize=8)
def _lidx(lmax, mmax, device):
    """l of every entry of the triangular m-major a_lm layout."""
    l = torch.arange(lmax + 1, dtype=torch.int32, device=device)
    keep = l[None, :] >= torch.arange(mmax + 1, dtype=torch.int32, device=device)[:, None]
    return l.expand(mmax + 1, -1)[keep]


def _alm(lmax, mmax, scale, spin, gen):
    """One seeded a_lm set (complex128, m = 0 real, zero below l = max(2, spin))."""
    dev = gen.device
    l = torch.arange(lmax + 1, dtype=torch.float64, device=dev)
    sigma = 0.5 * math.pi / (lmax + 1)
    cl = scale * torch.exp(-l * (l + 1) * sigma * sigma) / (l + 1) ** 2
    cl[: max(2, spin)] = 0.0
    a = torch.randn(_nalm(lmax, mmax), 2, dtype=torch.float64, device=dev, generator=gen)
    a *= torch.sqrt(cl / 2)[_lidx(lmax, mmax, str(dev)).long()].unsqueeze(-1)
    a[: lmax + 1, 0] *= math.sqrt(2.0)
    a[: lmax + 1, 1] = 0.0
    return torch.view_as_complex(a)


def _map(npix, gen):
    """One seeded map: unit noise and a signal that is smooth along the pixel order."""
    m = torch.randn(npix, dtype=torch.float64, device=gen.device, generator=gen)
    x = torch.arange(npix, dtype=torch.float64, device=gen.device) * (2 * math.pi / npix)
    ph = torch.rand(3, dtype=torch.float64, device=gen.device, generator=gen) * (2 * math.pi)
    for k in range(3):
        m += torch.sin((k + 1) * x + ph[k])
    return m


@functools.lru_cache(maxsize=8)
def _gauss(nrings, nphi):
    """The grid a program keeps for its run."""
    return sb.Geometry.grid("gauss", nrings, nphi)


@functools.lru_cache(maxsize=8)
def _layout(lmax, mmax):
    return sb.AlmInfo.triangular(lmax, mmax)


def _batch_sizes(case):
    """(spin, nside) of the jobs of a batch: a seeded mix of three resolutions."""
    r = random.Random(case["nside"] * 10007 + case["spin0"] * 101 + case["spin2"])
    sides = [case["nside"] // 4, case["nside"] // 2, case["nside"]]
    return [(0, r.choice(sides)) for _ in range(case["spin0"])] + \
           [(2, r.choice(sides)) for _ in range(case["spin2"])]


def _inputs(case, seed, dev):
    """The seeded inputs of a case as tensors on `dev`."""
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    k = case["kind"]
    if k == "batch":
        out, groups = {}, {}
        for spin, nside in _batch_sizes(case):
            groups[spin, nside] = groups.get((spin, nside), 0) + 1
        for (spin, nside), n in sorted(groups.items()):
            out[spin, nside] = torch.stack(
                [_alm(2 * nside, 2 * nside, _EBSCALE[c], spin, gen)
                 for _ in range(n) for c in ("T" if spin == 0 else "EB")])
        return out
    lmax = case["lmax"]
    npix = 12 * case["nside"] ** 2 if "nside" in case else case["nrings"] * case["nphi"]
    if k in ("iter",):
        return {"T": _map(npix, gen)}
    if k == "anal":
        return {c: _map(npix, gen) for c in case["comps"]}
    if k == "grid":
        n = case["ntrans"] * (2 if case["spin"] else 1)
        return {"a": torch.stack([_alm(lmax, case["mmax"], 1.0, case["spin"], gen)
                                  for _ in range(n)])}
    if k == "sets":
        return {c: torch.stack([_alm(lmax, lmax, _EBSCALE[c], 2 * (c != "T"), gen)
                                for _ in range(case["ntrans"])]) for c in "TEB"}
    comps = {"T": "T", "QU": "EB", "TQU": "TEB"}[case.get("comps", "TQU")]
    if k in ("der1", "host"):
        comps = "T"
    out = {c: _alm(lmax, lmax, _EBSCALE[c], 2 * (c != "T"), gen) for c in comps}
    if k == "grad":
        out["d"] = torch.stack([_map(npix, gen) for _ in range(3)])
        out["W"] = 0.5 + 1.5 * torch.rand(3, npix, dtype=torch.float64, device=dev,
                                          generator=gen)
    return out


def prepare(case, seed):
    k = case["kind"]
    dev = torch.device("cuda")
    s = {"case": case, "in": _inputs(case, seed, dev)}
    f8, c16 = torch.float64, torch.complex128

    def zeros(*shape, dtype=f8):
        return torch.zeros(*shape, dtype=dtype, device=dev)

    if k == "batch":
        jobs, s["map"], s["alm"] = [], {}, {}
        flags = sb.SHARP_DP | (sb.SHARP_MIXED if case["mixed"] else 0)
        for (spin, nside), a in s["in"].items():
            s["map"][spin, nside] = zeros(a.shape[0], 12 * nside * nside)
            s["alm"][spin, nside] = torch.zeros_like(a)
        at = {key: 0 for key in s["in"]}
        back = []
        for spin, nside in _batch_sizes(case):
            g, ai = hp.geometry(nside), hp.alm_info(2 * nside)
            i, n = at[spin, nside], 2 if spin else 1
            at[spin, nside] += n
            a, m, o = (list(s[x][spin, nside][i:i + n]) for x in ("in", "map", "alm"))
            jobs.append((sb.SHARP_ALM2MAP, spin, a, m, g, ai, 1, flags))
            back.append((sb.SHARP_MAP2ALM, spin, o, m, g, ai, 1, flags))
        s["jobs"], s["back"] = jobs, back
        return s
    lmax = case["lmax"]
    npix = 12 * case["nside"] ** 2 if "nside" in case else 0
    n = _nalm(lmax)
    if k in ("synth", "round"):
        s["map"] = {c: zeros(npix) for c in case.get("comps", "TQU")}
    if k in ("anal", "iter"):
        s["alm"] = {c: zeros(n, dtype=c16)
                    for c in {"T": "T", "QU": "EB", "TQU": "TEB"}[case.get("comps", "T")]}
    if k == "round":
        s["alm"] = {c: zeros(n, dtype=c16) for c in "TEB"}
    if k == "der1":
        s["map"] = [zeros(npix) for _ in range(3)]
    if k == "grad":
        s["geom"], s["layout"] = hp.geometry(case["nside"]), hp.alm_info(lmax)
    if k == "sets":
        s["map"] = {c: zeros(case["ntrans"], npix) for c in "TQU"}
        s["alm"] = {c: zeros(case["ntrans"], n, dtype=c16) for c in "TEB"}
        s["geom"], s["layout"] = hp.geometry(case["nside"]), hp.alm_info(lmax)
        s["flags"] = sb.SHARP_DP | (sb.SHARP_MIXED if case["mixed"] else 0)
    if k == "grid":
        real = f8 if case["double"] else torch.float32
        a = torch.view_as_real(s["in"]["a"]).reshape(s["in"]["a"].shape[0], -1).to(real)
        s["a"] = a.contiguous()
        s["map"] = zeros(a.shape[0], case["nrings"] * case["nphi"], dtype=real)
        s["alm"] = torch.zeros_like(s["a"])
        s["geom"] = _gauss(case["nrings"], case["nphi"])
        s["layout"] = _layout(lmax, case["mmax"])
        s["flags"] = sb.SHARP_DP if case["double"] else 0
    if k == "host":
        s["a"] = s["in"]["T"].cpu().numpy()
        s["map"], s["alm"] = np.zeros(npix), np.zeros(n, np.complex128)
        s["geom"], s["layout"] = hp.geometry(case["nside"]), hp.alm_info(lmax)
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _interleave(*xs):
    """Rows of several stacks, one of each in turn (E0, B0, E1, B1, ...)."""
    return [r for rows in zip(*xs) for r in rows]


def run(s):
    case = s["case"]
    k, i = case["kind"], s["in"]
    if k == "synth":
        m, c, lmax = s["map"], case["comps"], case["lmax"]
        if c == "T":
            hp.alm2map(i["T"], m["T"], lmax)
        elif c == "QU":
            hp.alm2map_spin(i["E"], i["B"], m["Q"], m["U"], 2, lmax)
        else:
            hp.alm2map_pol(i["T"], i["E"], i["B"], m["T"], m["Q"], m["U"], lmax)
        return m
    if k == "anal":
        a, c, lmax = s["alm"], case["comps"], case["lmax"]
        if c == "T":
            hp.map2alm(i["T"], a["T"], lmax)
        elif c == "QU":
            hp.map2alm_spin(i["Q"], i["U"], a["E"], a["B"], 2, lmax)
        else:
            hp.map2alm_pol(i["T"], i["Q"], i["U"], a["T"], a["E"], a["B"], lmax)
        return a
    if k == "round":
        m, a, lmax = s["map"], s["alm"], case["lmax"]
        hp.alm2map_pol(i["T"], i["E"], i["B"], m["T"], m["Q"], m["U"], lmax)
        hp.map2alm_pol(m["T"], m["Q"], m["U"], a["T"], a["E"], a["B"], lmax)
        return {"map": m, "alm": a}
    if k == "iter":
        return hp.map2alm_iter(i["T"], s["alm"]["T"], case["lmax"], case["sweeps"])
    if k == "der1":
        return list(hp.alm2map_der1(i["T"], *s["map"], case["lmax"]))
    if k == "grad":
        g, ai, p = s["geom"], s["layout"], case["precision"]
        xs = [i[c].detach().requires_grad_(True) for c in "TEB"]
        maps = (sa.alm2map(g, ai, 0, xs[0], precision=p),
                *sa.alm2map(g, ai, 2, xs[1], xs[2], precision=p))
        loss = 0.5 * sum(((i["W"][j] * (maps[j] - i["d"][j])) ** 2).sum() for j in range(3))
        return {"loss": loss.detach(), "grad": list(torch.autograd.grad(loss, xs))}
    if k == "sets":
        n, g, ai, fl = case["ntrans"], s["geom"], s["layout"], s["flags"]
        m, a = s["map"], s["alm"]
        qu, eb = _interleave(m["Q"], m["U"]), _interleave(a["E"], a["B"])
        sb.execute_device(sb.SHARP_ALM2MAP, 0, list(i["T"]), list(m["T"]), g, ai, n, fl)
        sb.execute_device(sb.SHARP_ALM2MAP, 2, _interleave(i["E"], i["B"]), qu, g, ai, n, fl)
        sb.execute_device(sb.SHARP_MAP2ALM, 0, list(a["T"]), list(m["T"]), g, ai, n, fl)
        sb.execute_device(sb.SHARP_MAP2ALM, 2, eb, qu, g, ai, n, fl)
        return {"map": m, "alm": a}
    if k == "batch":
        sb.execute_batch(s["jobs"], device=True)
        sb.execute_batch(s["back"], device=True)
        return {"map": {str(x): v for x, v in s["map"].items()},
                "alm": {str(x): v for x, v in s["alm"].items()}}
    if k == "grid":
        args = (s["geom"], s["layout"], case["ntrans"], s["flags"])
        sb.execute_device(sb.SHARP_ALM2MAP, case["spin"], list(s["a"]), list(s["map"]), *args)
        sb.execute_device(sb.SHARP_MAP2ALM, case["spin"], list(s["alm"]), list(s["map"]), *args)
        return {"map": s["map"], "alm": s["alm"]}
    sb.execute(sb.SHARP_ALM2MAP, 0, [s["a"]], [s["map"]], s["geom"], s["layout"])
    sb.execute(sb.SHARP_MAP2ALM, 0, [s["alm"]], [s["map"]], s["geom"], s["layout"])
    return {"map": s["map"], "alm": s["alm"]}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _healpix_rings(nside):
    """theta, phi0, nph of the rings of a HEALPix RING map, north to south."""
    i = np.arange(1, 4 * nside)
    cap = np.minimum(i, 4 * nside - i)
    polar = cap < nside
    th = 2 * np.arcsin(np.minimum(cap, nside) / (math.sqrt(6.0) * nside))
    th = np.where(i > 2 * nside, math.pi - th, th)
    th = np.where(polar, th, np.arccos(np.clip((2 * nside - i) * (2.0 / (3 * nside)), -1, 1)))
    nph = 4 * np.where(polar, cap, nside)
    phi0 = np.where(polar | ((i - nside) % 2 == 0), math.pi / nph, 0.0)
    return th, phi0, nph


def _rings(case):
    if "nside" in case:
        th, phi0, nph = _healpix_rings(case["nside"])
        return th, phi0, nph, np.full(len(nph), 4 * math.pi / (12.0 * case["nside"] ** 2))
    x, w = np.polynomial.legendre.leggauss(case["nrings"])
    n = case["nrings"]
    return (np.arccos(-x), np.zeros(n), np.full(n, case["nphi"]),
            w * (2 * math.pi / case["nphi"]))


@functools.lru_cache(maxsize=64)
def _one_way(kind_key, spin, ntrans):
    """(bytes, flops) of one transform of `ntrans` maps (pairs) on a set of rings: the
    Legendre recurrence and sums over every (l, m) that reaches a pair of rings, the ring
    FFTs, and each map and a_lm once."""
    sizes = dict(kind_key)
    lmax, mmax = sizes["lmax"], sizes["mmax"]
    th, _, nph, _ = _rings(sizes)
    half = th <= math.pi / 2 + 1e-9
    mm = np.minimum(mmax, np.floor(lmax * np.sin(th[half])) + spin)
    triples = float(((mm + 1) * (lmax + 1) - mm * (mm + 1) / 2).sum())
    comps = ntrans * (2 if spin else 1)
    flops = triples * ((4 + 4 * ntrans) if spin == 0 else (8 + 16 * ntrans))
    flops += comps * float((2.5 * nph * np.log2(np.maximum(nph, 2))).sum())
    word = sizes["word"]
    return comps * word * (float(nph.sum()) + 2.0 * _nalm(lmax, mmax)), flops


def work(case):
    k = case["kind"]
    parts = []
    if k == "batch":
        n = {}
        for key in _batch_sizes(case):
            n[key] = n.get(key, 0) + 1
        for (spin, nside), cnt in n.items():
            key = (("lmax", 2 * nside), ("mmax", 2 * nside), ("nside", nside), ("word", 8))
            parts += [(2, _one_way(key, spin, cnt))]
    elif k == "grid":
        key = (("lmax", case["lmax"]), ("mmax", case["mmax"]), ("nrings", case["nrings"]),
               ("nphi", case["nphi"]), ("word", 8 if case["double"] else 4))
        parts = [(2, _one_way(key, case["spin"], case["ntrans"]))]
    else:
        key = (("lmax", case["lmax"]), ("mmax", case["lmax"]), ("nside", case["nside"]),
               ("word", 8))
        nt = case.get("ntrans", 1)
        t, p = _one_way(key, 0, nt), _one_way(key, 2, nt)
        times = {"synth": 1, "anal": 1, "round": 2, "iter": 1 + 2 * case.get("sweeps", 0),
                 "der1": 1, "grad": 2, "sets": 2, "host": 2}[k]
        comps = {"host": "T", "iter": "T", "der1": "T"}.get(k, case.get("comps", "TQU"))
        if "T" in comps:
            parts.append((times, t))
        if "Q" in comps or k == "der1":
            parts.append((times, p))
    return {"bytes": sum(n * x[0] for n, x in parts), "flops": sum(n * x[1] for n, x in parts)}


# ---------------------------------------------------------------------------
# the same in plain torch, 64 bits, ring by ring
# ---------------------------------------------------------------------------
_BIG = 2.0 ** 400


def _seeds(mmax, spin, x):
    """Value and exponent (powers of 2^800) of the functions at l = max(m, |spin|) for every
    m and ring: normalised P_mm for spin 0, d^l_{m,spin} (unnormalised) otherwise."""
    dev = x.device
    v = torch.zeros(mmax + 1, len(x), dtype=torch.float64, device=dev)
    e = torch.zeros_like(v, dtype=torch.int32)
    st = torch.sqrt((1 - x) * (1 + x))
    c, h = torch.sqrt((1 + x) / 2), torch.sqrt((1 - x) / 2)
    cur, ex = None, torch.zeros(len(x), dtype=torch.int32, device=dev)
    s = abs(spin)
    for m in range(mmax + 1):
        if m < s:
            # d^s_{m,s} up to the sign fixed below
            f = math.sqrt(math.comb(2 * s, s + m))
            v[m] = f * c ** (s + m) * h ** (s - m) if spin > 0 else f * c ** (s - m) * h ** (s + m)
            continue
        if s == 0:
            cur = torch.full_like(x, math.sqrt(1 / (4 * math.pi))) if m == 0 else \
                -cur * st * math.sqrt((2 * m + 1) / (2.0 * m))
        elif m == s:
            cur = c ** (2 * s) if spin > 0 else h ** (2 * s)
        else:
            cur = cur * (math.sqrt(2.0 * m * (2 * m - 1) / ((m + s) * (m - s)))) * c * h
        small = cur.abs() < 1 / _BIG
        cur = torch.where(small, cur * _BIG * _BIG, cur)
        ex = ex - small.to(torch.int32)
        v[m], e[m] = cur, ex
    if s:
        m = torch.arange(mmax + 1, device=dev)
        if spin > 0:   # (-1)^(m - s) above m = s, none below
            sign = torch.where((m >= s) & ((m - s) % 2 == 1), -1.0, 1.0)
        else:          # (-1)^(m + s) of d^l_{m,-s}, seen from m >= s and from m < s alike
            sign = torch.where((m + s) % 2 == 1, -1.0, 1.0)
        v *= sign.to(torch.float64)[:, None]
    return v, e


def _functions(lmax, mmax, spin, x, block=32):
    """Blocks (l0, f[m, l - l0, ring]) of the normalised functions sqrt((2l+1)/4pi) d^l_{m,spin}
    (spin 0: the associated Legendre functions), zero for l < max(m, |spin|)."""
    dev = x.device
    v, e = _seeds(mmax, spin, x)
    s = abs(spin)
    m = torch.arange(mmax + 1, dtype=torch.float64, device=dev)[:, None]
    cur, ex = torch.zeros_like(v), torch.zeros_like(e)
    prev = torch.zeros_like(v)
    for l0 in range(0, lmax + 1, block):
        out = torch.zeros(mmax + 1, min(block, lmax + 1 - l0), len(x), dtype=torch.float64,
                          device=dev)
        for l in range(l0, l0 + out.shape[1]):
            start = torch.clamp(m, min=float(s)) == l
            cur = torch.where(start, v, cur)
            ex = torch.where(start, e, ex)
            f = torch.where(ex == 0, cur, torch.zeros_like(cur))
            out[:, l - l0] = f if s == 0 else f * math.sqrt((2 * l + 1) / (4 * math.pi))
            live = torch.clamp(m, min=float(s)) <= l
            up = torch.where(live, (l + 1.0) ** 2 - m * m, torch.ones_like(m))
            dn = torch.where(live, float(l) ** 2 - m * m, torch.zeros_like(m))
            if s == 0:
                a = torch.sqrt((2 * l + 3.0) * (2 * l + 1.0) / up)
                b = torch.sqrt((2 * l + 3.0) * dn / (max(2 * l - 1.0, 1.0) * up))
                new = a * x * cur - b * prev
            else:
                up = torch.sqrt(up * max((l + 1.0) ** 2 - s * s, 1.0))
                a = (l + 1.0) * (2 * l + 1.0) / up
                t = m * (spin / (l * (l + 1.0))) if l else torch.zeros_like(m)
                b = torch.sqrt(dn * max(l * l - s * s, 0)) * ((l + 1.0) / l if l else 0.0) / up
                new = a * (x - t) * cur - b * prev
            new = torch.where(live, new, torch.zeros_like(new))
            prev, cur = torch.where(live, cur, torch.zeros_like(cur)), new
            # a value that outgrew its scale takes the next one, with its predecessor
            big = (cur.abs() > _BIG) & (ex < 0)
            cur = torch.where(big, cur / (_BIG * _BIG), cur)
            prev = torch.where(big, prev / (_BIG * _BIG), prev)
            ex = ex + big.to(torch.int32)
        yield l0, out


def _spin_pair(lmax, mmax, spin, x):
    """Blocks of (w, y): the sum and difference of the two spin functions, such that
    Q_m = sum w G + i y C and U_m = sum w C - i y G."""
    sg = -1.0 if spin % 2 == 0 else 1.0
    for (l0, p), (_, q) in zip(_functions(lmax, mmax, spin, x), _functions(lmax, mmax, -spin, x)):
        if spin % 2:
            p = -p
        yield l0, 0.5 * sg * (p + q), 0.5 * sg * (q - p)


def _square(a, lmax, mmax):
    """a_lm stacks [n, nalm] as [m, n, l]."""
    out = torch.zeros(a.shape[0], mmax + 1, lmax + 1, dtype=torch.complex128, device=a.device)
    keep = torch.arange(lmax + 1)[None, :] >= torch.arange(mmax + 1)[:, None]
    out[:, keep.to(a.device)] = a
    return out.permute(1, 0, 2)


def _packed(sq, lmax, mmax):
    keep = torch.arange(lmax + 1)[None, :] >= torch.arange(mmax + 1)[:, None]
    return sq.permute(1, 0, 2)[:, keep.to(sq.device)]


def _rmul(c, r):
    """Batched product of a complex stack with a real one, real and imaginary parts apart."""
    return torch.complex(torch.bmm(c.real.contiguous(), r), torch.bmm(c.imag.contiguous(), r))


def _to_rings(ph, phi0, nph):
    """ph[m, n, ring] -> maps [n, npix]: sum_m Re(...) on the pixels of each ring."""
    n = ph.shape[1]
    m = torch.arange(ph.shape[0], dtype=torch.float64, device=ph.device)
    out = []
    for r in range(len(nph)):
        c = ph[:, :, r].T * torch.exp(1j * m * float(phi0[r]))
        c = torch.cat([c[:, :1].real.to(c.dtype), 2 * c[:, 1:]], 1)
        k = int(nph[r])
        bins = torch.zeros(n, k, dtype=c.dtype, device=c.device)
        for j in range(0, c.shape[1], k):
            bins[:, : min(k, c.shape[1] - j)] += c[:, j:j + k]
        out.append((torch.fft.ifft(bins) * k).real)
    return torch.cat(out, 1)


def _from_rings(maps, mmax, phi0, nph, wgt):
    """Adjoint of _to_rings without its factor 2, times the ring weights: [m, n, ring]."""
    m = torch.arange(mmax + 1, device=maps.device)
    md = m.to(torch.float64)
    cols, at = [], 0
    for r in range(len(nph)):
        k = int(nph[r])
        f = torch.fft.fft(maps[:, at:at + k])
        at += k
        cols.append((f[:, m % k] * torch.exp(-1j * md * float(phi0[r])) * float(wgt[r])).T)
    return torch.stack(cols, 2)


def _synth(a, lmax, mmax, spin, rings):
    """a [n, nalm] (spin > 0: E, B in turn) -> maps [n, npix]."""
    th, phi0, nph, _ = rings
    x = torch.cos(torch.tensor(th, dtype=torch.float64)).to(a.device)
    sq = _square(a, lmax, mmax)
    sq[0] = sq[0].real.to(sq.dtype)
    ph = torch.zeros(mmax + 1, a.shape[0], len(x), dtype=torch.complex128, device=a.device)
    if spin == 0:
        for l0, f in _functions(lmax, mmax, 0, x):
            ph += _rmul(sq[:, :, l0:l0 + f.shape[1]], f)
    else:
        g, c = sq[:, 0::2], sq[:, 1::2]
        for l0, w, y in _spin_pair(lmax, mmax, spin, x):
            gg, cc = (t[:, :, l0:l0 + w.shape[1]] for t in (g, c))
            ph[:, 0::2] += _rmul(gg, w) + 1j * _rmul(cc, y)
            ph[:, 1::2] += _rmul(cc, w) - 1j * _rmul(gg, y)
    return _to_rings(ph, phi0, nph)


def _anal(maps, lmax, mmax, spin, rings, weighted=True):
    """maps [n, npix] (spin > 0: Q, U in turn) -> a [n, nalm]."""
    th, phi0, nph, wgt = rings
    x = torch.cos(torch.tensor(th, dtype=torch.float64)).to(maps.device)
    ph = _from_rings(maps, mmax, phi0, nph, wgt if weighted else np.ones(len(nph)))
    sq = torch.zeros(mmax + 1, maps.shape[0], lmax + 1, dtype=torch.complex128,
                     device=maps.device)
    if spin == 0:
        for l0, f in _functions(lmax, mmax, 0, x):
            sq[:, :, l0:l0 + f.shape[1]] = _rmul(ph, f.transpose(1, 2).contiguous())
    else:
        q, u = ph[:, 0::2], ph[:, 1::2]
        for l0, w, y in _spin_pair(lmax, mmax, spin, x):
            w, y = (t.transpose(1, 2).contiguous() for t in (w, y))
            at = slice(l0, l0 + w.shape[2])
            sq[:, 0::2, at] = _rmul(q, w) + 1j * _rmul(u, y)
            sq[:, 1::2, at] = _rmul(u, w) - 1j * _rmul(q, y)
    sq[0] = sq[0].real.to(sq.dtype)
    return _packed(sq, lmax, mmax)


def exact(case, seed):
    k = case["kind"]
    lmax = case.get("lmax", 2 * case.get("nside", 0))
    passes = {"iter": 1 + 2 * case.get("sweeps", 0), "grad": 2, "sets": 2, "grid": 2, "host": 2,
              "round": 2, "batch": 6}.get(k, 1)
    comps = max(case.get("ntrans", 1), case.get("spin0", 1))
    # larger ones take more than a few seconds
    if lmax > 1100 or passes * comps * (lmax / 1100.0) ** 3 > 8:
        return None
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    i = _inputs(case, seed, dev)
    if k == "batch":
        m, a = {}, {}
        for (spin, nside), x in i.items():
            rings = _rings({"nside": nside})
            m[str((spin, nside))] = mm = _synth(x, 2 * nside, 2 * nside, spin, rings)
            a[str((spin, nside))] = _anal(mm, 2 * nside, 2 * nside, spin, rings)
        return {"map": m, "alm": a}
    rings = _rings(case)
    both = lambda x, y: torch.stack(_interleave(x, y))  # noqa: E731
    if k == "grid":
        mmax, spin = case["mmax"], case["spin"]
        x = i["a"]
        if not case["double"]:
            x = x.to(torch.complex64).to(torch.complex128)
        m = _synth(x, lmax, mmax, spin, rings)
        a = _anal(m if case["double"] else m.to(torch.float32).to(torch.float64), lmax, mmax,
                  spin, rings)
        return {"map": m, "alm": torch.view_as_real(a).reshape(a.shape[0], -1)}
    if k == "synth" or k == "round" or k == "sets":
        m, lead = {}, (lambda x: x) if k == "sets" else (lambda x: x[None])
        if "T" in i:
            m["T"] = _synth(lead(i["T"]), lmax, lmax, 0, rings)
        if "E" in i:
            qu = _synth(both(lead(i["E"]), lead(i["B"])), lmax, lmax, 2, rings)
            m["Q"], m["U"] = qu[0::2], qu[1::2]
        if k == "synth":
            return {c: x[0] for c, x in m.items()}
        eb = _anal(both(m["Q"], m["U"]), lmax, lmax, 2, rings)
        a = {"T": _anal(m["T"], lmax, lmax, 0, rings), "E": eb[0::2], "B": eb[1::2]}
        if k == "round":
            m, a = ({c: x[0] for c, x in y.items()} for y in (m, a))
        return {"map": m, "alm": a}
    if k == "anal":
        a = {}
        if "T" in i:
            a["T"] = _anal(i["T"][None], lmax, lmax, 0, rings)[0]
        if "Q" in i:
            a["E"], a["B"] = _anal(torch.stack([i["Q"], i["U"]]), lmax, lmax, 2, rings)
        return a
    if k == "iter":
        t = i["T"][None]
        a = _anal(t, lmax, lmax, 0, rings)
        for _ in range(case["sweeps"]):
            a = a + _anal(t - _synth(a, lmax, lmax, 0, rings), lmax, lmax, 0, rings)
        return a[0]
    if k == "der1":
        x = i["T"][None]
        l = _lidx(lmax, lmax, str(dev)).to(torch.float64)
        d = torch.cat([x * torch.sqrt(l * (l + 1)), torch.zeros_like(x)])
        dth, dph = _synth(d, lmax, lmax, 1, rings)
        return [_synth(x, lmax, lmax, 0, rings)[0], dth, dph]
    if k == "grad":
        m = torch.cat([_synth(i["T"][None], lmax, lmax, 0, rings),
                       _synth(torch.stack([i["E"], i["B"]]), lmax, lmax, 2, rings)])
        r = i["W"] * (m - i["d"])
        g = torch.cat([_anal((i["W"] * r)[:1], lmax, lmax, 0, rings, False),
                       _anal((i["W"] * r)[1:], lmax, lmax, 2, rings, False)])
        g[:, lmax + 1:] *= 2
        return {"loss": 0.5 * (r * r).sum(), "grad": list(g)}
    m = _synth(i["T"][None], lmax, lmax, 0, rings)
    return {"map": m[0].cpu().numpy(),
            "alm": _anal(m, lmax, lmax, 0, rings)[0].cpu().numpy()}
