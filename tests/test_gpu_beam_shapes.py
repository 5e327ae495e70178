"""The station beam's work split and phase tables at their limits: several
element types through the kernel of whole rounds (four or fewer directions per
thread, the rest in parts) and the one for few directions, the tables' phase
factors one by one against long double, and the largest number of directions.

Tolerances: as tests/test_gpu_beam.py; phase factors below."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(),
                                 reason="needs a CUDA device")]

import oskar_b200 as ob  # noqa: E402
from oracle_lib import oracle, suffix  # noqa: E402
from test_gpu_beam import TOL, dev, rel, stations  # noqa: E402

C0 = 299792458.0
PI_LD = np.arccos(np.longdouble(-1))


def types_beam(real, nst, n, nd, num_types, types, kinds, el, ori, freq, b,
               dirs, flags, scalar=False, meas=None, out=None):
    """oskb_station_beam_aa_types / _scalar of stations that share the
    directions; flags: normalise element, array, final; swap; 3-D."""
    tapers = np.zeros(num_types, np.int32)
    if out is None:
        out = torch.zeros((nst, nd, 2 if scalar else 8), device="cuda",
                          dtype=torch.float64 if real == np.float64 else
                          torch.float32)
    name = "scalar" if scalar else "types"
    ob.call("oskb_station_beam_aa_%s_%s" % (name, suffix(real)), nst, n, *el,
            *(meas or [None] * 3), None, None, num_types, types,
            np.array([1.5, 1.1, 2.0, 0.7][:num_types]), kinds, tapers,
            np.zeros(num_types), ori, ori, *flags, freq, b, b, nd, *dirs, 0,
            out, ob.stream_ptr())
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("real", [np.float64, np.float32])
@pytest.mark.parametrize("num_types", [1, 2, 3, 4])
@pytest.mark.parametrize("nst,num_dir", [(300, 1030), (300, 2047), (4, 65),
                                         (149, 257)])
def test_types_in_rounds_and_parts(real, num_types, nst, num_dir):
    """300 stations fill the device with blocks of 1,024 (FP64: 1,024, 512 or
    256) directions, whole rounds of which come first, and leave one direction
    to almost a block per station; the others are parts only."""
    flags = (1, 1, 1, 0, 1)
    n = 5
    base = stations(real, num_st=3, num_el=n, num_dir=num_dir)
    dirs = base[0]["dirs"]
    rng = np.random.default_rng(num_dir + num_types)
    types = rng.integers(0, num_types, (nst, n)).astype(np.int32)
    ori = rng.uniform(0, np.pi, (nst, num_types))
    cat = lambda i: dev(np.stack([base[s % 3]["el"][i] for s in range(nst)]))
    b = np.stack([base[0]["b"]] * nst)
    got = types_beam(real, nst, n, num_dir, num_types, dev(types),
                     np.zeros(num_types, np.int32), [cat(i) for i in range(3)],
                     dev(ori), 110e6, dev(b), [dev(d) for d in dirs],
                     flags).cpu().numpy()
    zero = np.zeros(num_types)
    for s in {0, 1, nst // 2, nst - 2, nst - 1}:
        c = base[s % 3]
        ref = np.zeros(8 * num_dir, real)
        oracle().call("station_beam_aa_types_" + suffix(real), np.float64, n,
                      1, *c["el"], *c["el"], np.zeros(n, real),
                      np.tile([1.0, 0.0], n).astype(real), num_types,
                      types[s].copy(),
                      np.array([1.5, 1.1, 2.0, 0.7][:num_types]),
                      np.zeros(num_types, np.int32),
                      np.zeros(num_types, np.int32), zero, ori[s].copy(),
                      ori[s].copy(), *flags[:4], 0, flags[4], 110e6, *b[s],
                      *b[s], num_dir, *dirs, ref)
        assert rel(got[s].ravel(), ref) <= TOL[real], s


@pytest.mark.parametrize("real,entries,steps,bound",
                         [(np.float64, 512, 81.48733086305042, 4e-16),
                          (np.float32, 256, 40.74366543152521, 1.5e-7)])
@pytest.mark.parametrize("reach", [1.0, 600.0, 1e5, 1e6, 5e9])
@pytest.mark.parametrize("num_dir", [300, 400000])
def test_table_phase_factors(real, entries, steps, bound, reach, num_dir):
    """One isotropic element at x = 1 m, no normalisation: the beam is the
    phase factor of u = k l in table steps, which float arithmetic here forms
    as the kernel does, so the factor is compared with that of exactly u. 300
    directions take one per thread, 400,000 four. Bound: entry, remainder and
    the last two roundings, a unit and a half of the type in all (with the
    FP32 remainder's 2e-10); beyond 2^32 (FP32: 2^21) steps the library's."""
    freq = 110e6
    k_steps = 2.0 * np.pi * freq / C0 * steps
    rng = np.random.default_rng(int(reach) % 1000)
    l = (rng.uniform(-reach, reach, num_dir) / k_steps).astype(real)
    l[:3] = 0
    u = (k_steps * l.astype(np.float64)).astype(real)
    z = lambda n: torch.zeros(n, device="cuda", dtype=torch.float64
                              if real == np.float64 else torch.float32)
    one = z(1) + 1
    got = types_beam(real, 1, 1, num_dir, 1, None, np.ones(1, np.int32),
                     [one, z(1), z(1)], torch.zeros(1, dtype=torch.float64,
                                                    device="cuda"), freq,
                     dev(np.array([[0.0, 0.0, 1.0]])),
                     [dev(l), z(num_dir), z(num_dir) + 1],
                     (0, 0, 0, 0, 0)).cpu().numpy()[0]
    x = np.fmod(u.astype(np.float64), entries).astype(np.longdouble) * \
        2 * PI_LD / entries
    assert np.max(np.abs(got[:, 0] - np.cos(x))) <= bound
    assert np.max(np.abs(got[:, 1] - np.sin(x))) <= bound
    assert np.all(got[:3, 0] == 1) and np.all(got[:3, 1] == 0)


@pytest.mark.parametrize("length", [0.7, 1.36, 2.9])
def test_pattern_towards_the_dipole_axis(length):
    """FP64: one dipole at the origin along x (its pattern is the beam), from
    across it down to 1e-7 rad from its axis, against long double. (cos(kL a)
    - cos kL) / (1 - a^2) is formed there as 2 sin(kL (1 + a) / 2) sin(kL (1 -
    a) / 2) / (1 - a^2) with 1 - a^2 = |(y, z)|^2 / |d|^2. The quotient's
    parts are a few roundings each: 2e-15, of the larger of the value and the
    two sines' product near the pattern's own zeros."""
    freq = 110e6
    rng = np.random.default_rng(8)
    off = 10.0 ** np.linspace(-7, 0.19, 4000)
    tilt = rng.uniform(0, 0.5 * np.pi, 4000)
    d = [np.cos(off) * np.where(rng.random(4000) < 0.5, -1, 1),
         np.sin(off) * np.cos(tilt) * np.where(rng.random(4000) < 0.5, -1, 1),
         np.sin(off) * np.sin(tilt)]
    z = torch.zeros(1, dtype=torch.float64, device="cuda")
    out = torch.zeros((1, 4000, 8), dtype=torch.float64, device="cuda")
    up = dev(np.array([[0.0, 0.0, 1.0]]))
    ob.call("oskb_station_beam_aa_d", 1, 1, z, z, z, None, None, None, None,
            z, z, length, 0, 0, 0, 0, 0, freq, up, up, 4000,
            *[dev(c) for c in d], 0, out, ob.stream_ptr())
    got = out.cpu().numpy()[0]
    kl = np.longdouble(length * (np.pi * freq / C0))
    x, y, w = (c.astype(np.longdouble) for c in d)
    h2 = x * x + y * y + w * w
    rho2 = x * x + y * y
    one_a2 = (y * y + w * w) / h2
    a = np.abs(x) / np.sqrt(h2)
    num = 2 * np.sin(kl * (1 + a) / 2) * np.sin(kl * one_a2 / (1 + a) / 2)
    theta = -x * w / np.sqrt(rho2 * h2) * num / one_a2
    phi = y / np.sqrt(rho2) * num / one_a2
    size = np.abs(2 * np.sin(kl * one_a2 / (1 + a) / 2) / one_a2)
    for col, want, scale in ((0, theta, x * w / np.sqrt(rho2 * h2)),
                             (2, phi, y / np.sqrt(rho2))):
        bound = 4e-15 * np.abs(scale) * size
        assert np.all(np.abs(got[:, col] - want) <= bound)


def test_largest_direction_count():
    """2^31 - 1 directions: the last block reaches past the largest int. The
    same direction throughout, so every output is the first one; 26 GB."""
    nd = 2 ** 31 - 1
    if torch.cuda.mem_get_info()[0] < 40 << 30:
        pytest.skip("needs 40 GB of free device memory")
    d = torch.full((nd,), 0.5, dtype=torch.float32, device="cuda")
    one = torch.ones(1, dtype=torch.float32, device="cuda")
    out = torch.full((nd + 2048, 2), 7.0, dtype=torch.float32, device="cuda")
    types_beam(np.float32, 1, 1, nd, 1, None, np.ones(1, np.int32),
               [one, one, one], torch.zeros(1, dtype=torch.float64,
                                            device="cuda"), 110e6,
               dev(np.array([[0.0, 0.0, 1.0]])), [d, d, d], (0, 0, 0, 0, 0),
               scalar=True, out=out)
    first = out[0].clone()
    assert 0.5 < float(first.norm()) < 2 and float(first[0]) != 7
    for start in range(0, nd, 1 << 28):
        part = out[start:min(nd, start + (1 << 28))]
        assert bool((part == first).all())
    assert bool((out[nd:] == 7).all())
    del d, out
    torch.cuda.empty_cache()
