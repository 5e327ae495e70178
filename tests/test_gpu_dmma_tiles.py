"""The FP64 tensor-pipe correlation (point sources without smearing) at the
edges of its tiles against the CPU oracle: station counts around its 8 x 16
warp tiles (those that hold no baseline are skipped) and one, two, three and
more chunks of 8 sources (its pipeline runs two chunks ahead). FP64 1e-12, as
tests/test_gpu_direct.py."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(),
                                 reason="needs a CUDA device")]

from test_gpu_direct import (assert_close, run_gpu_xcorr,  # noqa: E402
                             run_oracle_xcorr)
from xcorr_cases import XcorrCase  # noqa: E402


@pytest.mark.parametrize("num_st", [2, 8, 9, 16, 17, 25, 40, 49, 65])
@pytest.mark.parametrize("num_src", [1, 8, 9, 17, 25, 41])
def test_warp_tiles_and_chunks(num_st, num_src):
    c = XcorrCase(num_st, num_src, real=np.float64, ranges="physical",
                  seed=num_st, casa=num_src % 2, offset_out=2)
    assert_close(run_gpu_xcorr(c, np.float64),
                 run_oracle_xcorr(c, np.float64), np.float64)
