"""Workloads of the interferometer visibility path for measuring its speed.

Every case is work that a simulation built on this package has it do, through
the C entry points bound by ``oskar_b200.call``: whole dumps of a small array,
station beams, correlation of joined Jones matrices, and whole blocks of dumps
and channels with and without smearing. Sizes are those of the package's own
configurations (``oskar_b200.workloads``, ``bench.py``) and odd sizes around
them; skies and layouts have the same value distributions, made on the device
from a seed.

A case's ``kind`` selects the entry points:

  chain     one dump: station (u, v, w) -> Jones K -> J = K E -> correlation
            (FP64 direct), what a simulator without smearing runs per channel
  corr      oskb_cross_correlate_{d,f} on joined Jones (smearing and Gaussian
            sources optional), what a drop-in caller runs per sky chunk
  block     oskb_correlate_block_direct_{d,f}: dumps x channels with fused K,
            Gaussian sources and both smearings
  tc_block  oskb_correlate_block_tc: dumps x channels on the tensor cores
  tc64      oskb_cross_correlate_tc64_d on joined Jones (FP64-class)
  tc64_block  oskb_correlate_block_tc64_d
  beam      oskb_station_beam_aa_weighted_{d,f}: station beams of all stations
"""
import math

import torch

import oskar_b200 as ob

C0 = 299792458.0
OMEGA_EARTH = 7.272205217e-5
LAT = math.radians(-27.0)
LON = math.radians(116.76)
RA0, DEC0 = 0.0, math.radians(-30.0)
BANDWIDTH_HZ, TIME_AVERAGE_SEC = 1e5, 10.0


def listed():
    return [
        # A small array and sky (30 stations, 1,000 sources): a dump is a few
        # microseconds of work, so launches and latency count.
        dict(name="chain_30x1000", kind="chain", stations=30, sources=1000,
             extent_m=500.0),
        # An aperture-array simulation's correlation after the beam: one
        # channel of one dump, 12,000 sources.
        dict(name="chain_128x12000", kind="chain", stations=128,
             sources=12000, extent_m=40e3),
        # One odd-sized sky chunk of point sources with both smearings, as a
        # simulator calls the correlator per (dump, chunk, channel).
        dict(name="corr_f64_197x4001_smear", kind="corr", bits=64,
             stations=197, sources=4001, gaussian=False, bandwidth=True,
             time=True, extent_m=20e3),
        # The same call in single precision: a chunk of Gaussian sources with
        # bandwidth smearing only.
        dict(name="corr_f32_351x7013_gauss", kind="corr", bits=32,
             stations=351, sources=7013, gaussian=True, bandwidth=True,
             time=False, extent_m=2e3),
        # Blocks of a spectral simulation with 30 % Gaussian sources and both
        # smearings: 256 stations out to 65 km in double precision, ...
        dict(name="block_f64_256x20000", kind="block", bits=64, stations=256,
             sources=20000, times=1, channels=4, extent_m=65e3),
        # ... and a ragged one of a compact array in single precision.
        dict(name="block_f32_211x9001", kind="block", bits=32, stations=211,
             sources=9001, times=2, channels=3, extent_m=2e3),
        # The headline workload: one dump x 16 channels of 512 stations and
        # 100,000 point sources on the tensor cores.
        dict(name="tc_block_512x100000", kind="tc_block", stations=512,
             sources=100000, times=1, channels=16, extent_m=65e3),
        # A small block of the same kind (a prototype array).
        dict(name="tc_block_64x3000", kind="tc_block", stations=64,
             sources=3000, times=2, channels=4, extent_m=5e3),
        # FP64-class correlation of one channel, as the drop-in issues it per
        # (dump, chunk, channel).
        dict(name="tc64_256x20000", kind="tc64", stations=256, sources=20000,
             extent_m=65e3),
        # An FP64-class block of a ragged array.
        dict(name="tc64_block_300x15001", kind="tc64_block", stations=300,
             sources=15001, times=1, channels=8, extent_m=65e3),
        # Station beams of aperture arrays with 256 dipoles: planar stations
        # in double precision, ...
        dict(name="beam_f64_128x256x12000", kind="beam", bits=64,
             stations=128, elements=256, directions=12000, planar=True,
             weighted=False),
        # ... and a larger single-precision set on uneven ground with element
        # weights (errors or apodisation).
        dict(name="beam_f32_512x256x10001", kind="beam", bits=32,
             stations=512, elements=256, directions=10001, planar=False,
             weighted=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _log_float(rng, lo, hi):
    return round(math.exp(rng.uniform(math.log(lo), math.log(hi))), 1)


def _source_baselines(case):
    n = case["stations"]
    return (n * (n - 1) // 2 * case["sources"] * case.get("times", 1) *
            case.get("channels", 1))


def draw(rng):
    kind = rng.choice(["chain", "corr", "corr", "block", "block", "tc_block",
                       "tc64", "tc64_block", "beam", "beam"])
    if kind == "beam":
        while True:
            case = dict(kind=kind, bits=rng.choice([32, 64]),
                        stations=_log_int(rng, 1, 512),
                        elements=_log_int(rng, 16, 1024),
                        directions=_log_int(rng, 200, 30000),
                        planar=rng.random() < 0.5,
                        weighted=rng.random() < 0.5)
            if (case["stations"] * case["elements"] * case["directions"] <=
                    512 * 256 * 10001):
                return case
    limit = {"chain": 3e9, "corr": 1.5e9, "block": 2e9, "tc_block": 4e10,
             "tc64": 1e10, "tc64_block": 1e10}[kind]
    while True:
        case = dict(kind=kind, stations=_log_int(rng, 16, 512),
                    sources=_log_int(rng, 100, 50000))
        if kind in ("corr", "block"):
            case["bits"] = rng.choice([32, 64])
        if kind == "corr":
            case["gaussian"] = rng.random() < 0.5
            case["bandwidth"] = rng.random() < 0.6
            case["time"] = rng.random() < 0.5
        if kind in ("block", "tc_block", "tc64_block"):
            case["times"] = rng.randint(1, 4)
            case["channels"] = rng.randint(1, 16)
        # single precision holds the phases of a compact array only
        case["extent_m"] = _log_float(rng, 500.0, 3e3 if
                                      case.get("bits") == 32 else 65e3)
        if _source_baselines(case) <= limit:
            return case


# ------------------------------------------------------------------ inputs
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(g, lo, hi, *shape):
    u = torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)
    return lo + (hi - lo) * u


def _sky(g, num, gaussian_share=0.0):
    """Point sources in a 20 degree field, I ~ S^-1.5 on [0.01, 10] Jy,
    |Q|, |U|, |V| <= 0.1 I; a share of them Gaussian, 1 to 60 arcsec."""
    r = torch.sqrt(_uniform(g, 0, 1, num)) * math.sin(math.radians(10.0))
    th = _uniform(g, 0, 2 * math.pi, num)
    l, m = r * torch.cos(th), r * torch.sin(th)
    lo, hi = 0.01 ** -0.5, 10.0 ** -0.5
    flux = (lo + _uniform(g, 0, 1, num) * (hi - lo)) ** -2.0
    sky = dict(l=l, m=m, n=torch.sqrt(1.0 - l * l - m * m), I=flux)
    for k in "QUV":
        sky[k] = flux * _uniform(g, -0.1, 0.1, num)
    if gaussian_share:
        on = _uniform(g, 0, 1, num) < gaussian_share
        arcsec = math.pi / 180 / 3600
        major = _uniform(g, 1, 60, num) * arcsec
        minor = torch.minimum(major, _uniform(g, 1, 60, num) * arcsec)
        pa = _uniform(g, 0, math.pi, num)
        k = 0.5 * math.pi ** 2 / (2 * math.log(2))
        a2, b2 = k * major ** 2, k * minor ** 2
        c2, s2 = torch.cos(pa) ** 2, torch.sin(pa) ** 2
        sky["a"] = (c2 * b2 + s2 * a2) * on
        sky["b"] = 0.5 * torch.sin(2 * pa) * (a2 - b2) * on
        sky["c"] = (s2 * b2 + c2 * a2) * on
    return sky


def _stations(g, num, extent_m):
    """ECEF offsets [3][station] of a layout that is log-radial from 50 m out
    to the given extent."""
    r = torch.exp(_uniform(g, math.log(50.0), math.log(extent_m), num))
    th = _uniform(g, 0, 2 * math.pi, num)
    e, n = r * torch.cos(th), r * torch.sin(th)
    sl, cl, so, co = (math.sin(LAT), math.cos(LAT), math.sin(LON),
                      math.cos(LON))
    return torch.stack([-so * e - sl * co * n, co * e - sl * so * n, cl * n])


def _hour_angle(g, times):
    """Greenwich hour angle of the phase centre per dump, near transit."""
    start = -LON + float(_uniform(g, -0.5, 0.5, 1)[0])
    return [start + 7.3e-4 * t for t in range(times)]


def _uvw(ecef, hour_angle):
    """Station (u, v, w) [dump][3][station] in metres."""
    x, y, z = ecef
    sd, cd = math.sin(DEC0), math.cos(DEC0)
    out = []
    for ha in hour_angle:
        sh, ch = math.sin(ha), math.cos(ha)
        t = x * ch - y * sh
        out.append(torch.stack([x * sh + y * ch, z * cd - t * sd,
                                z * sd + t * cd]))
    return torch.stack(out)


def _jones(g, stations, sources, dtype):
    """Station beam per station-source: identity plus complex N(0, 0.1)."""
    e = torch.randn((stations, sources, 8), generator=g, device="cuda",
                    dtype=torch.float32)
    e.mul_(0.1)
    e[..., 0] += 1.0
    e[..., 6] += 1.0
    return e.to(dtype)


def _frequencies(case):
    return [100e6 + 1e6 * c for c in range(case.get("channels", 1))]


def _beam_inputs(case, g):
    n, ne, nd = case["stations"], case["elements"], case["directions"]
    dtype = torch.float64 if case["bits"] == 64 else torch.float32
    s = dict(frequency=110e6, wavelength=C0 / 110e6)
    # stations as dense as 256 dipoles in a 38 m disc
    radius = 19.0 * math.sqrt(ne / 256.0)
    r = radius * torch.sqrt(_uniform(g, 0, 1, n, ne))
    th = _uniform(g, 0, 2 * math.pi, n, ne)
    s["x"], s["y"] = (r * torch.cos(th)).to(dtype), \
        (r * torch.sin(th)).to(dtype)
    s["z"] = torch.zeros_like(s["x"]) if case["planar"] else \
        _uniform(g, -0.5, 0.5, n, ne).to(dtype)
    s["factors"] = None
    if case["weighted"]:
        gain = 1.0 + 0.05 * _uniform(g, -1, 1, n, ne)
        phase = _uniform(g, -0.1, 0.1, n, ne)
        s["factors"] = torch.stack([gain * torch.cos(phase),
                                    gain * torch.sin(phase)], -1).to(dtype)
    s["orientation"] = _uniform(g, 0, 2 * math.pi, n)
    el = _uniform(g, math.radians(45), math.radians(85), n)
    az = _uniform(g, 0, 2 * math.pi, n)
    point = torch.stack([torch.cos(el) * torch.sin(az),
                         torch.cos(el) * torch.cos(az), torch.sin(el)], 1)
    s["point"] = point.contiguous()
    # directions: most within 10 degrees of the pointing, a sixth anywhere in
    # the sky (some of them below the horizon)
    rr = math.sin(math.radians(10.0)) * torch.sqrt(_uniform(g, 0, 1, n, nd))
    tt = _uniform(g, 0, 2 * math.pi, n, nd)
    a, b = rr * torch.cos(tt), rr * torch.sin(tt)
    c = torch.sqrt(1 - a * a - b * b)
    east = torch.stack([torch.cos(az), -torch.sin(az), 0 * az], 1)
    north = torch.linalg.cross(point, east)
    d = (a[..., None] * east[:, None] + b[..., None] * north[:, None] +
         c[..., None] * point[:, None])
    far = torch.randn((n, nd, 3), generator=g, device="cuda",
                      dtype=torch.float64)
    far[..., 2] = far[..., 2].abs() * torch.where(
        _uniform(g, 0, 1, n, nd) < 0.1, -1.0, 1.0)
    far /= far.norm(dim=-1, keepdim=True)
    d = torch.where(_uniform(g, 0, 1, n, nd, 1) < 1 / 6, far, d).to(dtype)
    s["dirs"] = [d[..., k].contiguous() for k in range(3)]
    s["beam"] = torch.empty((n, nd, 8), dtype=dtype, device="cuda")
    return s


def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    if kind == "beam":
        return dict(_beam_inputs(case, g), case=case)
    f32 = case.get("bits") == 32
    dtype = torch.float32 if f32 else torch.float64
    n, ns = case["stations"], case["sources"]
    nt, nc = case.get("times", 1), case.get("channels", 1)
    share = 0.3 if kind == "block" else 1.0 if case.get("gaussian") else 0.0
    sky = {k: v.to(dtype).contiguous()
           for k, v in _sky(g, ns, share).items()}
    ecef = _stations(g, n, case["extent_m"])
    ha = _hour_angle(g, nt)
    uvw = _uvw(ecef, ha)
    freqs = _frequencies(case)
    s = dict(case=case, sky=sky, ha=ha, ecef=ecef.to(dtype),
             uvw=uvw.to(dtype), freqs=freqs,
             inv_wl=torch.tensor([f / C0 for f in freqs], device="cuda",
                                 dtype=torch.float64),
             ha_dev=torch.tensor(ha, device="cuda", dtype=torch.float64),
             vis=torch.empty((nt, nc, n * (n - 1) // 2, 8), device="cuda",
                             dtype=torch.float32 if f32 else torch.float64))
    e_type = torch.float32 if kind == "tc_block" else dtype
    s["E"] = _jones(g, n, ns, e_type)
    if kind == "chain":
        s["uvw"] = torch.empty((3, n), dtype=dtype, device="cuda")
        s["K"] = torch.empty((n, ns, 2), dtype=dtype, device="cuda")
        s["J"] = torch.empty_like(s["E"])
    if kind in ("corr", "tc64"):
        # joined Jones K E, as the step before leaves it
        u, v, w = uvw[0]
        phase = (2 * math.pi * freqs[0] / C0) * (
            u[:, None] * sky["l"].double() + v[:, None] * sky["m"].double() +
            w[:, None] * (sky["n"].double() - 1))
        k = torch.polar(torch.ones_like(phase), phase)
        e = torch.view_as_complex(s.pop("E").double().view(n, ns, 4, 2))
        s["J"] = torch.view_as_real(e * k[..., None]).to(dtype).reshape(
            n, ns, 8).contiguous()
    return s


# -------------------------------------------------------------------- runs
def _suffix(case):
    return "f" if case.get("bits") == 32 else "d"


def run(state):
    case = state["case"]
    stream = ob.stream_ptr()
    if case["kind"] == "beam":
        beam = state["beam"]
        ob.call("oskb_station_beam_aa_weighted_" + _suffix(case),
                case["stations"], case["elements"], state["x"], state["y"],
                state["z"], None, None, None, None, state["factors"],
                state["orientation"], state["orientation"],
                0.5 * state["wavelength"], 0, 1, 1, 0,
                0 if case["planar"] else 1, state["frequency"],
                state["point"], state["point"], case["directions"],
                *state["dirs"], 1, beam, stream)
        return beam
    n, ns = case["stations"], case["sources"]
    nt, nc = case.get("times", 1), case.get("channels", 1)
    sky, vis = state["sky"], state["vis"]
    flux = [sky[k] for k in "IQUV"]
    lmn = [sky[k] for k in "lmn"]
    shape = [sky.get(k) for k in "abc"]
    f = state["freqs"][0]
    vis.zero_()
    kind = case["kind"]
    if kind == "chain":
        u, v, w = state["uvw"]
        ob.call("oskb_convert_ecef_to_station_uvw_d", n, *state["ecef"], RA0,
                DEC0, state["ha"][0] + RA0, 0, 0, u, v, w, stream)
        ob.call("oskb_evaluate_jones_K_d", ns, *lmn, n, u, v, w,
                2 * math.pi * f / C0, sky["I"], 0.0, 1e300, 0, state["K"],
                stream)
        ob.call("oskb_mem_multiply_d", 3, 0, 0, 0, n * ns, state["K"],
                state["E"], state["J"], stream)
        ob.call("oskb_cross_correlate_d", 0, 0, ns, n, 0, state["J"], *flux,
                *lmn, None, None, None, u, v, w, None, None, 0.0, 3e38,
                f / C0, 0.0, 0.0, 0.0, 0.0, vis, stream)
    elif kind == "corr":
        u, v, w = state["uvw"][0]
        x, y, _ = state["ecef"]
        ob.call("oskb_cross_correlate_" + _suffix(case), 0,
                1 if case["gaussian"] else 0, ns, n, 0, state["J"], *flux,
                *lmn, *shape, u, v, w, x, y, 0.0, 3e38, f / C0,
                BANDWIDTH_HZ / f if case["bandwidth"] else 0.0,
                TIME_AVERAGE_SEC if case["time"] else 0.0, state["ha"][0],
                DEC0, vis, stream)
    elif kind == "block":
        x, y, _ = state["ecef"]
        ob.call("oskb_correlate_block_direct_" + _suffix(case), 0, ns, n, nt,
                nc, state["E"], 0, *flux, *lmn, *shape, state["uvw"], x, y,
                state["inv_wl"], BANDWIDTH_HZ, TIME_AVERAGE_SEC,
                state["ha_dev"], DEC0, 0.0, 3e38, 0, 0.0, 3e38, vis, stream)
    elif kind == "tc64":
        u, v, _ = state["uvw"][0]
        ob.call("oskb_cross_correlate_tc64_d", 0, ns, n, 0, state["J"],
                *flux, u, v, 0.0, 3e38, f / C0, vis, None, 0, stream)
    else:
        name = "oskb_correlate_block_tc" if kind == "tc_block" else \
            "oskb_correlate_block_tc64_d"
        ob.call(name, 0, ns, n, nt, nc, state["E"], *lmn, *flux,
                state["uvw"], state["inv_wl"], 0.0, 3e38, vis, None, 0,
                stream)
    return vis


def work(case):
    if case["kind"] == "beam":
        n, ne, nd = case["stations"], case["elements"], case["directions"]
        word = case["bits"] // 8
        per_el = 2 + (0 if case["planar"] else 1) + \
            (2 if case["weighted"] else 0)
        # per element-direction: the phase (two operations per coordinate),
        # one sine and one cosine, one complex multiply-add (8)
        dims = 2 if case["planar"] else 3
        return {"bytes": word * (n * ne * per_el + n * nd * (3 + 8)),
                "flops": n * ne * nd * (2 * dims + 2 + 8)}
    n, ns = case["stations"], case["sources"]
    nt, nc = case.get("times", 1), case.get("channels", 1)
    word = 4 if case.get("bits") == 32 else 8
    e_word = 4 if case["kind"] == "tc_block" else word
    return {"bytes": e_word * 8 * n * ns + word * 10 * ns +
            word * 8 * nt * nc * (n * (n - 1) // 2),
            # eight complex multiply-adds per source-baseline
            "flops": 64 * _source_baselines(case)}


def tolerance(case):
    # about four times the distance from the results in 64 bits (beyond 64
    # bits for the double-precision cases): phases of 1e4 radians carry
    # 1e-12 in double and those of a compact array 1e-5 in single precision
    kind = case["kind"]
    if kind == "beam":
        return {"rel": 5e-6} if case["bits"] == 32 else {"rel": 1e-14}
    if kind == "tc_block":
        return {"rel": 1.5e-6}  # 24-bit fixed point, bound 1e-6
    if case.get("bits") == 32:
        return {"rel": 1e-4 if kind == "block" else 1e-6}
    return {"rel": {"corr": 1e-13, "tc64": 2e-13}.get(kind, 4e-12)}


# ------------------------------------------------------- results in 64 bits
# Phases reach 1e4 radians, so their products are formed as unevaluated sums
# of two doubles (T. J. Dekker, "A floating-point technique for extending the
# available precision", 1971) and reduced before the sine and cosine.
def _two_prod(a, b):
    def split(v):
        t = 134217729.0 * v
        hi = t - (t - v)
        return hi, v - hi
    p = a * b
    ah, al = split(a)
    bh, bl = split(b)
    return p, ((ah * bh - p) + ah * bl + al * bh) + al * bl


def _two_sum(a, b):
    s = a + b
    t = s - a
    return s, (a - (s - t)) + (b - t)


def _dot(pairs):
    """Sum of the products of the pairs as two doubles."""
    hi = lo = None
    for a, b in pairs:
        p, e = _two_prod(a, b)
        if hi is None:
            hi, lo = p, e
        else:
            hi, d = _two_sum(hi, p)
            lo = lo + e + d
    return hi, lo


def _cis_turns(hi, lo, scale, scale_lo=0.0):
    """exp(2 pi i (hi + lo) (scale + scale_lo))."""
    p, e = _two_prod(hi, torch.as_tensor(scale, dtype=torch.float64,
                                         device=hi.device))
    turns = (p - torch.round(p)) + (e + lo * scale + hi * scale_lo)
    return torch.polar(torch.ones_like(turns), 2 * math.pi * turns)


def _baselines(n):
    """(q, p) station indices of every baseline, in the output's order."""
    i = torch.triu_indices(n, n, 1, device="cuda")
    return i[0], i[1]


def _phases(uvw, sky, scale, scale_lo=0.0):
    u, v, w = (c.double()[:, None] for c in uvw)
    n1 = sky["n"].double() - 1.0
    hi, lo = _dot([(u, sky["l"].double()), (v, sky["m"].double()), (w, n1)])
    return _cis_turns(hi, lo, scale, scale_lo)


def _factors(jones, phases, sky):
    """(J B, J) as [station][i][source][k] for J = K E."""
    n, ns = jones.shape[:2]
    j = torch.view_as_complex(jones.double().reshape(n, ns, 4, 2))
    j = j.reshape(n, ns, 2, 2)
    if phases is not None:
        j = j * phases[:, :, None, None]
    i, q, u, v = (sky[k].double() for k in "IQUV")
    b = torch.stack([torch.complex(i + q, 0 * i), torch.complex(u, v),
                     torch.complex(u, -v), torch.complex(i - q, 0 * i)], -1)
    jb = j @ b.reshape(ns, 2, 2)
    return jb.permute(0, 2, 1, 3).contiguous(), \
        j.permute(0, 2, 1, 3).contiguous()


def _correlate(jones, phases, sky, smear=None):
    """Visibilities [baseline][8] of J = K E; smear(q) gives the factors
    [station p > q][source]."""
    left, right = _factors(jones, phases, sky)
    n, _, ns, _ = left.shape
    if smear is None:
        g = left.reshape(2 * n, 2 * ns) @ right.reshape(2 * n, 2 * ns).mH
        q, p = _baselines(n)
        vis = g.reshape(n, 2, n, 2)[p, :, q, :]
    else:
        rows = []
        for q in range(n - 1):
            t = left[q + 1:] * smear(q)[:, None, :, None]
            t = t.reshape(-1, 2 * ns) @ right[q].reshape(2, 2 * ns).mH
            rows.append(t.reshape(-1, 2, 2))
        vis = torch.cat(rows)
    return torch.view_as_real(vis.contiguous()).reshape(-1, 8)


def _smear(case, state, sky, t, inv_wl):
    """The smearing factors of one dump and channel as a function of q."""
    bandwidth = case["kind"] == "block" or case["bandwidth"]
    time = case["kind"] == "block" or case["time"]
    gauss = case["kind"] == "block" or case["gaussian"]
    if not (bandwidth or time or gauss):
        return None
    u, v, w = state["uvw"][t].double()
    x, y = state["ecef"][0].double(), state["ecef"][1].double()
    l, m, n1 = (sky["l"].double(), sky["m"].double(),
                sky["n"].double() - 1.0)
    sh, ch = math.sin(state["ha"][t]), math.cos(state["ha"][t])
    xr, yr = x * ch - y * sh, x * sh + y * ch
    decl = math.sin(DEC0) * m - math.cos(DEC0) * n1

    def sinc(d):
        return torch.where(d == 0, 1.0, torch.sin(d) / d)

    def factors(q):
        uu, vv, ww = ((c[q + 1:] - c[q])[:, None] for c in (u, v, w))
        f = torch.ones((u.numel() - q - 1, l.numel()), device=l.device,
                       dtype=torch.float64)
        if gauss:
            a, b, c = (sky[k].double() for k in "abc")
            us, vs = uu * inv_wl, vv * inv_wl
            f = torch.exp(-(a * us * us + 2 * b * us * vs + c * vs * vs))
        if bandwidth:
            f = f * sinc((uu * l + vv * m + ww * n1) *
                         (math.pi * BANDWIDTH_HZ / C0))
        if time:
            dx, dy = ((c[q + 1:] - c[q])[:, None] for c in (xr, yr))
            f = f * sinc((dx * l + dy * decl) *
                         (math.pi * OMEGA_EARTH * TIME_AVERAGE_SEC * inv_wl))
        return f
    return factors


def _exact_beam(case, s):
    """Dipole pattern times array factor over the beam's amplitude at the
    pointing, in 64 bits."""
    n = case["stations"]
    out = torch.empty(s["beam"].shape, dtype=torch.float64, device="cuda")
    k_turns = s["frequency"] / C0
    kl = math.pi * 0.5 * s["wavelength"] * k_turns

    def pattern(x, y, z, orientation):
        p0, theta = torch.atan2(y, x), torch.atan2(torch.hypot(x, y), z)
        parts = []
        for phi in (p0 - orientation, p0 + math.pi / 2 - orientation):
            cp, sp, ct = torch.cos(phi), torch.sin(phi), torch.cos(theta)
            t = (torch.cos(kl * cp * torch.sin(theta)) - math.cos(kl)) / \
                (1 + cp * cp * (ct * ct - 1))
            parts += [-cp * ct * t, sp * t]
        return torch.stack(parts, -1)

    for st in range(n):
        el = [s[k][st].double()[:, None] for k in "xyz"]
        b = s["point"][st]
        d = [c[st].double() for c in s["dirs"]]
        if case["planar"]:
            # the array factor's plane has no z term in the direction
            el[2] = torch.zeros_like(el[2])
        weight = torch.ones(case["elements"], dtype=torch.complex128,
                            device="cuda")
        if s["factors"] is not None:
            weight = torch.view_as_complex(s["factors"][st].double())

        def array_factor(dx, dy, dz):
            hi, lo = _dot([(el[0], dx), (el[1], dy), (el[2], dz),
                           (el[0], -b[0]), (el[1], -b[1]), (el[2], -b[2])])
            e = _cis_turns(hi, lo, k_turns)
            return (weight @ e) / case["elements"]

        af = array_factor(*d)
        v = pattern(*d, s["orientation"][st]) * af[:, None]
        v = torch.where((d[2] < 0)[:, None], torch.zeros_like(v), v)
        bn = [c.reshape(1) for c in b]
        amp = pattern(*bn, s["orientation"][st]) * array_factor(*bn)[:, None]
        v = v / torch.sqrt((amp.abs() ** 2).sum() / 2)
        out[st] = torch.view_as_real(v).reshape(-1, 8)
    return out


def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]
    if kind == "beam":
        return _exact_beam(case, s)
    sky, freqs = s["sky"], s["freqs"]
    if kind == "chain":
        uvw = _uvw(s["ecef"], s["ha"])[0]
        # the phase is the given wavenumber's: turns through 1 / (2 pi) as
        # two doubles
        k = 2 * math.pi * freqs[0] / C0
        inv_2pi, inv_2pi_lo = 0.15915494309189535, -9.839338337591243e-18
        kt, kt_lo = _two_prod(*(torch.tensor(v, dtype=torch.float64)
                                for v in (k, inv_2pi)))
        phases = _phases(uvw, sky, float(kt), float(kt_lo) + k * inv_2pi_lo)
        return _correlate(s["E"], phases, sky).reshape(s["vis"].shape)
    if kind in ("corr", "tc64"):
        smear = _smear(case, s, sky, 0, freqs[0] / C0) if kind == "corr" \
            else None
        return _correlate(s["J"], None, sky, smear).reshape(s["vis"].shape)
    out = torch.empty(s["vis"].shape, dtype=torch.float64, device="cuda")
    for t in range(case["times"]):
        for c, f in enumerate(freqs):
            smear = _smear(case, s, sky, t, f / C0) if kind == "block" \
                else None
            out[t, c] = _correlate(s["E"], _phases(s["uvw"][t], sky, f / C0),
                                   sky, smear)
    return out
