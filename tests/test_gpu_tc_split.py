"""Integer contractions whose last wave of tiles is split over the source
blocks: a call recorded into a CUDA graph with a workspace of just the size
needed runs every tile whole (it takes no memory from the scratch pool), a
plain call splits them where that saves time, and the sums are exact
integers, so the visibilities are the same bits. Both forms: three limbs
(oskb_cross_correlate_tc_d, and a block of problems) and six
(oskb_cross_correlate_tc64_d). One tile to a few dozen, source counts around
the 32-source blocks and the order kernel's runs of 1/32 of the sources,
fluxes over eight decades (several amplitude buckets); 2 x 1 is too little
to split, and so is the last wave of 257 x 2,049 in the six-limb form.

The partial sums lie behind the operand images of a larger workspace, of the
library's own and of a block plan's, so those split in a graph too; a few
tiles more than the device has SMs run one whole wave first."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(),
                                 reason="needs a CUDA device")]

import oskar_b200 as ob  # noqa: E402
from test_gpu_tc import dev, errors, oracle_vis  # noqa: E402
from test_gpu_tc64 import case  # noqa: E402
from test_gpu_tc_plan import ENV_KEYS, make_case, run_plan  # noqa: E402

ROOM = 16 << 20   # more than the partial sums of any call take


def runs():
    return ob.call("oskb_tc_last_wave_runs", check=False)


def device_bytes(size):
    return torch.empty(size, dtype=torch.uint8, device="cuda")


def recorded(call, size, before=None):
    """call's output replayed from a graph; before(): run on the same stream
    ahead of the capture."""
    out = torch.zeros(size, dtype=torch.float64, device="cuda")
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        if before:
            before()
            s.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            call(out)
        g.replay()
        s.synchronize()
    got = out.cpu().numpy()
    del g
    return got


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


@pytest.mark.parametrize("form", ["tc", "tc64"])
def test_room_behind_the_images(form):
    """Recorded calls split with a larger workspace and with the library's
    own, as the plain call does from the pool."""
    nst, nsrc = 97, 3000
    l, m, n, I, Q, U, V, u, v, w, J = case(np.random.default_rng(5), nst,
                                           nsrc, decades=8)
    name = "oskb_cross_correlate_%s_d" % form
    need = ob.call("oskb_cross_correlate_%s_workspace_bytes" % form, nsrc,
                   nst, check=False)
    size = nst * (nst - 1) // 2 * 8
    d = [dev(x) for x in (J, I, Q, U, V, u, v)]

    def call(ws, ws_bytes):
        return lambda vis: ob.call(name, 0, nsrc, nst, 0, *d, 0.0, 3e38, 1.3,
                                   vis, ws, ws_bytes, ob.stream_ptr())

    exact = call(device_bytes(need), need)
    plain = torch.zeros(size, dtype=torch.float64, device="cuda")
    exact(plain)
    assert runs() > 1
    whole = recorded(exact, size)
    assert runs() == 1
    larger = recorded(call(device_bytes(need + ROOM), need + ROOM), size)
    assert runs() > 1
    scrap = torch.zeros_like(plain)
    kept = recorded(call(None, 0), size, before=lambda: call(None, 0)(scrap))
    assert runs() > 1
    assert np.array_equal(whole, plain.cpu().numpy())
    assert np.array_equal(whole, larger) and np.array_equal(whole, kept)


@pytest.mark.parametrize("form", ["tc", "tc64"])
def test_whole_wave_then_split_wave(form):
    """Ten tiles (six limbs: twice as many, half as wide) beyond the number
    of SMs, with auto-correlations: pool, workspace tail and whole tiles."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    nst, nsrc, ntime = 20, 1500, 2
    nchan = (sms + 10) // (2 if form == "tc" else 4)
    l, m, n, I, Q, U, V, u, v, w, J = case(np.random.default_rng(6), nst,
                                           nsrc, decades=4)
    uvw = np.stack([np.stack([u, v, w])] * ntime)
    inv_wl = 0.3 + 0.001 * np.arange(nchan)
    name = "oskb_correlate_block_" + {"tc": "tc", "tc64": "tc64"}[form]
    full = name + ("_auto" if form == "tc" else "_auto_d")
    need = ob.call(name + "_workspace_bytes", nsrc, nst, ntime * nchan,
                   check=False)
    e = J.astype(np.float32) if form == "tc" else J
    d = [dev(x) for x in (e, l, m, n, I, Q, U, V, uvw, inv_wl)]
    nvis = ntime * nchan * nst * (nst - 1) // 2 * 8
    size = nvis + ntime * nchan * nst * 8

    def call(ws_bytes):
        ws = device_bytes(ws_bytes)
        return lambda out: ob.call(full, 0, nsrc, nst, ntime, nchan, *d, 0.0,
                                   3e38, out, out[nvis:], ws, ws_bytes,
                                   ob.stream_ptr())

    plain = torch.zeros(size, dtype=torch.float64, device="cuda")
    call(need)(plain)
    assert runs() > 1
    plain = plain.cpu().numpy()
    assert np.all(np.abs(plain).reshape(-1, 8).max(axis=1) > 0)
    whole = recorded(call(need), size)
    if form == "tc64":   # (the FP16 image that tc is sized for is larger)
        assert runs() == 1
    larger = recorded(call(need + ROOM), size)
    assert runs() > 1
    assert np.array_equal(whole, plain) and np.array_equal(whole, larger)


def test_plan_graphs_split(monkeypatch):
    """A plan's graphs run the contraction as its tuning run timed it."""
    for k in ENV_KEYS:
        monkeypatch.delenv(k, raising=False)
    c = make_case(nst=64, nsrc=3000, nt=2, nch=4, nblocks=2)
    monkeypatch.setenv("OSKB_TC_PLAN_FORM", "1")
    outs, form, launches, _ = run_plan(c)
    assert form == 1 and launches == 2
    assert runs() > 1
    monkeypatch.setenv("OSKB_TC_PLAN_GRAPH", "0")
    eager, _, _, _ = run_plan(c)
    assert runs() > 1
    for a, b in zip(outs, eager):
        assert np.array_equal(a, b)
