"""The cache's calls read FP32 rows where the caller has them, or stage them
where they cannot be read in 16-byte pieces; the transposed weights of the
backward pass follow every change of the weights."""
import numpy as np
import pytest

from nuray_gb300.nrc import INPUTS, NUM_PARAMS, Cache

pytestmark = pytest.mark.gpu


def _rows(n, seed):
    r = np.random.default_rng(seed)
    return r.uniform(-1, 1, (n, INPUTS)).astype(np.float32), r.gamma(1.0, 1.0, (n, 3)).astype(np.float32)


def _at(a, offset):
    """A copy of a that starts `offset` bytes past a 64-byte boundary."""
    buf = np.zeros(a.nbytes + 128, np.uint8)
    start = (-buf.ctypes.data) % 64 + offset
    v = buf[start:start + a.nbytes].view(np.float32).reshape(a.shape)
    v[...] = a
    return v


@pytest.mark.parametrize("tc", [0, 1])
@pytest.mark.parametrize("n", [1, 127, 128, 129, 384, 385, 5000, 116737])
def test_rows_at_any_address(gpu_lib, n, tc):
    x, y = _rows(n, n)
    c = Cache(f"seed=3 tc={tc}")
    out = c.infer(_at(x, 0))
    g, loss = c.gradient(_at(x, 0), _at(y, 0))
    assert np.all(np.isfinite(out)) and out.shape == (n, 3)
    for o in (4, 8, 16, 36):
        np.testing.assert_array_equal(c.infer(_at(x, o)), out)
        g2, loss2 = c.gradient(_at(x, o), _at(y, (o + 4) % 64))
        # float atomics in any order: sums of up to n terms of either sign
        np.testing.assert_allclose(g2, g, rtol=1e-4, atol=1e-5 * np.abs(g).max())
        assert loss2 == pytest.approx(loss, rel=1e-5)


def test_backward_weights_follow_every_change(gpu_lib):
    x, y = _rows(700, 1)
    a = Cache("seed=5 lr=0.01")
    for _ in range(3):
        a.train_step(x, y)

    def same(c):
        """c's gradient is that of the mma.sync kernels, which read the weights themselves, at the same weights."""
        d = Cache("tc=0")
        d.set_params(c.get_params())
        g, ref = c.gradient(x, y)[0], d.gradient(x, y)[0]
        # data gradients rounded to BF16 from sums taken in another order: a few flips of half a BF16 ulp (2^-9)
        assert np.linalg.norm(g - ref) <= 2.0 ** -8 * np.linalg.norm(ref)

    same(a)                                                 # after Adam steps
    b = Cache("seed=9")
    b.set_params(a.get_params())
    same(b)                                                 # after set_params
    e = Cache("seed=10")
    e.train_step(x, y)
    e.set_state("params", a.get_state("params"))
    same(e)                                                 # after set_state
    assert a.get_params().size == NUM_PARAMS
