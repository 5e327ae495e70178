"""Matrix products of oskb_mem_multiply on aligned arrays (one complex part
per thread), on arrays that start at an odd real (one matrix per thread), in
place on either operand, with element offsets and counts that are not whole
warps, against numpy in the working precision: two complex products and a sum
per part, at most 8 roundings."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(),
                                 reason="needs a CUDA device")]

import oskar_b200 as ob  # noqa: E402

CM_M, MC_M, MM_M = 3, 4, 5


@pytest.mark.parametrize("real", [np.float64, np.float32])
@pytest.mark.parametrize("kind", [CM_M, MC_M, MM_M])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 1001])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("where", ["out", "in_a", "in_b"])
def test_matrix_products(real, kind, n, shift, where):
    sa, sb = (2 if kind == CM_M else 8), (2 if kind == MC_M else 8)
    if (where == "in_a" and sa == 2) or (where == "in_b" and sb == 2):
        pytest.skip("the output does not fit the operand")
    rng = np.random.default_rng(n + kind)
    off = (3, 5, 2) if where == "out" else (3, 5, 3 if where == "in_a" else 5)
    x, y = (rng.normal(size=(n + o, s)).astype(real)
            for o, s in ((off[0], sa), (off[1], sb)))

    def put(v):
        t = torch.zeros(v.size + shift, dtype=torch.from_numpy(v).dtype,
                        device="cuda")
        t[shift:] = torch.from_numpy(v.ravel()).cuda()
        return t[shift:]
    a, b = put(x), put(y)
    c = a if where == "in_a" else b if where == "in_b" else \
        put(np.zeros((n + off[2], 8), real))
    ob.call("oskb_mem_multiply_" + ("d" if real == np.float64 else "f"),
            kind, *off, n, a, b, c, ob.stream_ptr())
    torch.cuda.synchronize()

    def cplx(v, o, s):
        z = v[o:].astype(np.float64).reshape(n, s // 2, 2)
        z = z[..., 0] + 1j * z[..., 1]
        return z.reshape(n, 2, 2) if s == 8 else z.reshape(n, 1, 1)
    p, q = cplx(x, off[0], sa), cplx(y, off[1], sb)
    want = p @ q if kind == MM_M else p * q
    got = c.cpu().numpy().reshape(-1, 8)[off[2]:].astype(np.float64)
    got = (got[:, 0::2] + 1j * got[:, 1::2]).reshape(n, 2, 2)
    bound = 8 * np.finfo(real).eps * (np.abs(p) @ np.abs(q) if kind == MM_M
                                      else np.abs(p) * np.abs(q))
    assert np.all(np.abs(got - want) <= 2 * bound + 1e-300)
