"""FP64 smearing factors of stations far from the phase origin against long
double: station phases of up to hundreds of radians whose differences d are
small, as on the short baselines of an array's far arm. The factor
sin(d) / d comes from the stations' own sines and cosines, so it holds only
if those belong to the same phases as d.

One unpolarised source of 1 Jy on identity Jones makes every visibility its
baseline's factor. Bound per baseline: sine and cosine within 2.2e-16 each
(two ulp below 1), so the two products of the identity are within 1e-15
together with their roundings, over d; the phases are rounded once (their inputs are scaled
by powers of two), which moves d by up to |phi| 2^-52 and the factor by d / 3
of that; a few roundings of the quotient and the sum."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(),
                                 reason="needs a CUDA device")]

from test_gpu_direct import run_gpu_xcorr  # noqa: E402
from xcorr_cases import XcorrCase  # noqa: E402

OMEGA_EARTH = 7.272205217e-5
NUM_ST = 40
L = 0.25


@pytest.mark.parametrize("phase", [0.0, 12.0, 100.0, 700.0])
@pytest.mark.parametrize("kind", ["bandwidth", "time", "both"])
def test_factor_of_distant_stations(phase, kind):
    c = XcorrCase(NUM_ST, 1, ranges="physical", gaussian=False,
                  bandwidth_hz=0.0,
                  time_avg=0.0 if kind == "bandwidth" else 10.0)
    c.inv_wavelength = 1.0
    if kind != "time":
        c.frac_bandwidth = 1.0 / 1024
    rng = np.random.default_rng(int(phase) + len(kind))
    for k in ("st_u", "st_v", "st_w", "st_x", "st_y"):
        setattr(c, k, np.zeros(NUM_ST))
    q, p = np.triu_indices(NUM_ST, 1)
    want, bound = np.longdouble(1), 1e-15
    for name, on, scale in (
            ("st_u", kind != "time", np.pi / 1024),
            ("st_x", kind != "bandwidth", np.pi * OMEGA_EARTH * 10.0)):
        if not on:
            continue
        pos = (phase + rng.uniform(-0.3, 0.3, NUM_ST)) / (L * scale)
        setattr(c, name, pos)
        phi = np.longdouble(pos) * np.longdouble(scale) * np.longdouble(L)
        d = phi[p] - phi[q]
        ad = np.abs(d)
        assert np.sum(ad > 1 / 16) > 400
        want = want * np.where(d == 0, 1, np.sin(d) / np.where(d == 0, 1, d))
        bound = bound + 1e-15 / np.maximum(ad, 1 / 16) + \
            ad / 3 * float(np.max(np.abs(phi))) * 2.0 ** -52
    c.gha0 = 0.0
    c.jones = np.tile([1.0, 0, 0, 0, 0, 0, 1.0, 0], NUM_ST)
    c.I, c.l, c.n = np.ones(1), np.full(1, L), np.ones(1)
    c.Q = c.U = c.V = c.m = np.zeros(1)
    c.vis0 = np.zeros_like(c.vis0)
    got = run_gpu_xcorr(c, np.float64).reshape(-1, 8)
    for col in (0, 6):
        assert np.all(np.abs(got[:, col] - want) <= bound * np.abs(want))
    assert np.all(got[:, [1, 2, 3, 4, 5, 7]] == 0)
