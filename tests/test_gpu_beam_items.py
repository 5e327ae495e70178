"""The station beam at the edges of its work items against the CPU oracle:
direction counts around its blocks (256 threads, one to four directions
each), more stations than CTAs run at a time (whole rounds and the short
last one), more elements than one staged chunk, phases the tables do not
cover and non-finite input.

Tolerances as tests/test_gpu_beam.py (FP64 1e-12, FP32 2e-5) where the phases
are a station's. Huge phases: k r |phi| ulps of phase, 2.3e9 rad x 2^-53 x
about 8 roundings = 2e-6 (FP64) and 7e4 rad x 2^-24 x 8 = 3e-2 (FP32), the
FP32 result against the FP64 oracle on the same inputs."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(),
                                 reason="needs a CUDA device")]

from beam_cases import beam_case, oracle_beam  # noqa: E402
from test_gpu_beam import TOL, rel, run_gpu, stations  # noqa: E402


@pytest.mark.parametrize("real", [np.float64, np.float32])
@pytest.mark.parametrize("num_dir", [1, 255, 257, 1023, 1025, 2049])
def test_direction_blocks(real, num_dir):
    flags = (1, 1, 1, 0, num_dir % 2)
    cases = stations(real, num_st=2, num_el=20, num_dir=num_dir,
                     is_3d=flags[4])
    got = run_gpu(cases, real, flags)
    for s, c in enumerate(cases):
        assert rel(got[s], oracle_beam(c, real, flags)) <= TOL[real]


@pytest.mark.parametrize("real", [np.float64, np.float32])
@pytest.mark.parametrize("num_st", [295, 297, 310, 600])
def test_more_stations_than_ctas(real, num_st):
    flags = (0, 1, 1, 0, 1)
    cases = stations(real, num_st=num_st, num_el=6, num_dir=33)
    got = run_gpu(cases, real, flags)
    for s, c in enumerate(cases):
        assert rel(got[s], oracle_beam(c, real, flags)) <= TOL[real], s


@pytest.mark.parametrize("real", [np.float64, np.float32])
@pytest.mark.parametrize("num_el", [511, 512, 513, 1100])
def test_element_chunks(real, num_el):
    flags = (1, 1, 1, 1, 1)
    c = beam_case(real, seed=num_el, num_el=num_el, num_dir=300)
    assert rel(run_gpu([c], real, flags)[0],
               oracle_beam(c, real, flags)) <= TOL[real]


@pytest.mark.parametrize("real,scale,tol", [(np.float64, 1e9, 2e-6),
                                            (np.float32, 3e4, 3e-2)])
def test_phases_beyond_the_table(real, scale, tol):
    flags = (1, 1, 0, 0, 1)
    c = beam_case(real, seed=5, num_el=40, num_dir=200)
    for k in range(2):
        c["el"][k] = (c["el"][k] * real(scale / 19)).astype(real)
        c["meas"][k] = c["el"][k].copy()
    c["meas"][2] = c["el"][2].copy()
    wide = {k: ([a.astype(np.float64) for a in v] if isinstance(v, list)
                else v) for k, v in c.items()}
    wide["cable"] = c["cable"].astype(np.float64)
    assert rel(run_gpu([c], real, flags)[0],
               oracle_beam(wide, np.float64, flags)) <= tol


@pytest.mark.parametrize("real", [np.float64, np.float32])
def test_non_finite_input(real):
    flags = (1, 1, 1, 0, 1)
    cases = stations(real, num_st=2, num_el=30, num_dir=300)
    up = np.nonzero(cases[0]["dirs"][2] >= 0)[0]
    cases[1]["el"][0][7] = np.nan          # every direction of station 1
    cases[0]["dirs"][0][up[3]] = np.nan    # one direction (shared)
    got = run_gpu(cases, real, flags).reshape(2, 300, 8)
    assert np.isnan(got[1][up]).all()
    assert np.isnan(got[0][up[3]]).all()
    rest = np.delete(up, 3)
    assert np.isfinite(got[0][rest]).all()
