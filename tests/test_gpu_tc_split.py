"""Integer contractions whose last wave of tiles is split over the source
blocks: a call recorded into a CUDA graph runs every tile whole (it takes no
memory from the scratch pool), a plain call of these sizes splits them, and
the sums are exact integers, so the visibilities are the same bits. Both
forms: three limbs (oskb_cross_correlate_tc_d, and a block of problems) and
six (oskb_cross_correlate_tc64_d). One tile to a few dozen, source counts
around the 32-source blocks and the order kernel's runs of 1/32 of the
sources, fluxes over eight decades (several amplitude buckets)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(),
                                 reason="needs a CUDA device")]

import oskar_b200 as ob  # noqa: E402
from test_gpu_tc import dev, errors, oracle_vis  # noqa: E402
from test_gpu_tc64 import case  # noqa: E402


def both(call, size):
    """The outputs of call(vis) run plainly and replayed from a graph."""
    plain = torch.zeros(size, dtype=torch.float64, device="cuda")
    call(plain)
    torch.cuda.synchronize()
    captured = torch.zeros_like(plain)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call(captured)
    g.replay()
    torch.cuda.synchronize()
    out = plain.cpu().numpy(), captured.cpu().numpy()
    del g
    return out


@pytest.mark.parametrize("form", ["tc", "tc64"])
@pytest.mark.parametrize("nst,nsrc", [(2, 1), (31, 1023), (33, 1025),
                                      (64, 4097), (97, 3000), (257, 2049)])
def test_split_and_whole_tiles_same_bits(form, nst, nsrc):
    rng = np.random.default_rng(nst + nsrc)
    l, m, n, I, Q, U, V, u, v, w, J = case(rng, nst, nsrc, decades=8)
    name = "oskb_cross_correlate_%s_d" % form
    need = ob.call("oskb_cross_correlate_%s_workspace_bytes" % form, nsrc,
                   nst, check=False)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    d = [dev(x) for x in (J, I, Q, U, V, u, v)]
    plain, captured = both(
        lambda vis: ob.call(name, 0, nsrc, nst, 0, *d, 0.0, 3e38, 1.3, vis,
                            ws, need, ob.stream_ptr()),
        nst * (nst - 1) // 2 * 8)
    assert np.array_equal(plain, captured)
    ref = oracle_vis(nst, nsrc, J, I, Q, U, V, l, m, n, u, v, w, 1.3)
    l2, mx = errors(plain, ref)
    tol = 1e-12 if form == "tc64" else 1e-6
    assert l2 <= tol and mx <= tol, (l2, mx)


def test_split_block_same_bits():
    rng = np.random.default_rng(3)
    nst, nsrc, ntime, nchan = 40, 2500, 2, 3
    l, m, n, I, Q, U, V, u, v, w, J = case(rng, nst, nsrc)
    uvw = np.stack([np.stack([u, v, w])] * ntime)
    inv_wl = 0.3 + 0.01 * np.arange(nchan)
    need = ob.call("oskb_correlate_block_tc_workspace_bytes", nsrc, nst,
                   ntime * nchan, check=False)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    d = [dev(x) for x in (J.astype(np.float32), l, m, n, I, Q, U, V, uvw,
                          inv_wl)]
    plain, captured = both(
        lambda vis: ob.call("oskb_correlate_block_tc", 0, nsrc, nst, ntime,
                            nchan, *d, 0.0, 3e38, vis, ws, need,
                            ob.stream_ptr()),
        ntime * nchan * nst * (nst - 1) // 2 * 8)
    assert np.array_equal(plain, captured)
