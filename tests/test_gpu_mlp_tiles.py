"""Network kernels at the edges of their tiles: one to four tiles in flight per
CTA, the last tile partly filled, a second round of a CTA's tile slots, and
partial gradient rows that are not 16-byte aligned.  Tolerance of the forward
pass: tests/test_gpu_mlp.py's (bf16 operands, MUFU SiLU)."""
import numpy as np
import pytest

import zsph_b200 as z
from oracle import mlp_oracle as mo
from tests.test_gpu_mlp import FWD_TOL, _params, _rel

pytestmark = pytest.mark.gpu

SMS = 148


@pytest.mark.parametrize("n", [1, 128 * SMS, 128 * SMS + 1, 128 * 4 * SMS + 77])
def test_forward_at_tile_edges(n):
    rng = np.random.default_rng(n)
    net = z.Mlp(seed=1)
    p = _params(3)
    net.params = p
    X = rng.normal(size=(n, 32)).astype(np.float32)
    y = net.forward(z.Mlp.pack(z.DeviceArray.from_host(X), n), n)
    want = mo.forward(p, mo.standardize(X))
    assert y.shape[0] == n
    for rows in (slice(0, n), slice(max(n - 130, 0), n)):
        assert _rel(y[rows], want[rows]) < FWD_TOL
    net.close()


def test_partial_rows_of_any_alignment():
    rng = np.random.default_rng(4)
    n, nt = 128 * 5, 5
    net = z.Mlp(seed=3)
    tiles = z.Mlp.pack(z.DeviceArray.from_host(rng.normal(size=(n, 32)).astype(np.float32)), n)
    y = z.DeviceArray.from_host(rng.normal(size=(n, 4)).astype(np.float32))
    w = z.DeviceArray.from_host(np.ones(n, np.float32))
    buf = z.DeviceArray.from_host(np.zeros(nt * mo.NPARTIAL + 4, np.float32))
    got = []
    for off in (0, 1):
        parts = z.ctypes.c_int(0)
        z.check(z.lib.zsph_mlp_grad(net.h, tiles.ptr, y.ptr, w.ptr, None, nt, 1.0 / n, buf.ptr.value + 4 * off,
                                    z.ctypes.byref(parts), None))
        assert parts.value == nt
        got.append(buf.get()[off:off + nt * mo.NPARTIAL].copy())
    assert np.array_equal(got[0], got[1])
    net.close()
