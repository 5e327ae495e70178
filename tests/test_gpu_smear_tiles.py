"""The smearing / Gaussian kernel at the edges of its tiles against the CPU
oracle: station counts around its 8 x 8 patches and 32 x 32 tiles (patches
above the diagonal or past the last station are skipped), source counts
around its chunks of 8, and skies whose Gaussian sources (a, b, c not all
zero) are mixed with points, which skip the exponential one by one.

Tolerances as the other direct kernels (tests/test_gpu_direct.py): FP64
1e-12; FP32 1e-5 (sums of at most 8 terms in FP32, unit round-off 6e-8,
each product a few roundings)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(),
                                 reason="needs a CUDA device")]

from test_gpu_direct import (assert_close, run_gpu_xcorr,  # noqa: E402
                             run_oracle_xcorr)
from xcorr_cases import XcorrCase  # noqa: E402


@pytest.mark.parametrize("num_st,num_src", [(8, 7), (9, 8), (25, 9),
                                            (32, 15), (40, 16), (64, 1),
                                            (71, 41)])
@pytest.mark.parametrize("real", [np.float64, np.float32])
@pytest.mark.parametrize("matrix", [True, False])
@pytest.mark.parametrize("bw,ts", [(0.0, 0.0), (100e3, 0.0), (0.0, 10.0),
                                   (100e3, 10.0)])
def test_patches_chunks_and_mixed_sources(num_st, num_src, real, matrix, bw,
                                          ts):
    c = XcorrCase(num_st, num_src, real=real, ranges="physical",
                  matrix=matrix, bandwidth_hz=bw, time_avg=ts, gaussian=True,
                  seed=num_st, casa=num_src % 2, offset_out=1)
    point = np.arange(num_src) % 3 != 0
    for k in "abc":
        getattr(c, k)[point] = 0
    assert_close(run_gpu_xcorr(c, real), run_oracle_xcorr(c, real), real)


@pytest.mark.parametrize("real", [np.float64, np.float32])
@pytest.mark.parametrize("bw,ts", [(100e3, 0.0), (0.0, 10.0), (100e3, 10.0)])
@pytest.mark.parametrize("core", [0, 8, 20, 70])
def test_short_and_long_baselines(real, bw, ts, core):
    """FP32 patches whose phase differences are all small take the series
    alone, the others (and FP64) select it per baseline: a core of stations
    within 60 m (FP64) or 400 m (FP32) and the rest up to 60 (6) km, from none
    of one to none of the other. FP32 phases of 0.02 x 6 km carry 120 x 6e-8 absolute error:
    1e-5 as above."""
    c = XcorrCase(70, 57, real=real, ranges="physical", bandwidth_hz=bw,
                  time_avg=ts, gaussian=False, seed=core + 1)
    near, far = (0.06, 60.0) if real == np.float64 else (0.4, 6.0)
    scale = np.where(np.arange(70) < core, near, far).astype(real)
    for k in ("st_u", "st_v", "st_w", "st_x", "st_y"):
        setattr(c, k, (getattr(c, k) * scale * real(2 if k[-1] in "uvw"
                                                    else 1)).astype(real))
    assert_close(run_gpu_xcorr(c, real), run_oracle_xcorr(c, real), real)
