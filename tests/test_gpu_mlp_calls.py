"""Concurrent calls on one network: more of them than it keeps status words."""
import threading

import numpy as np
import pytest
import torch

import zsph_b200 as z
from tests.test_gpu_mlp import _params

pytestmark = pytest.mark.gpu


def test_more_concurrent_calls_than_status_words():
    n, calls = 300000, 40
    net = z.Mlp(seed=1)
    net.params = _params(3)
    x = torch.randn(n, 32, device="cuda")
    tiles = torch.empty((n + z.MLP_TILE - 1) // z.MLP_TILE, 4096, dtype=torch.int16, device="cuda")
    z.check(z.lib.zsph_mlp_pack(x.data_ptr(), n, None, None, tiles.data_ptr(), None))
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(calls)]
    out = torch.zeros(calls + 1, n, 4, device="cuda")
    torch.cuda.synchronize()
    z.check(z.lib.zsph_mlp_forward(net.h, tiles.data_ptr(), n, out[calls].data_ptr(), None))
    gate, rc = threading.Barrier(calls), [None] * calls

    def call(k):
        gate.wait()
        for _ in range(3):
            rc[k] = z.lib.zsph_mlp_forward(net.h, tiles.data_ptr(), n, out[k].data_ptr(), streams[k].cuda_stream)

    threads = [threading.Thread(target=call, args=(k,)) for k in range(calls)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert rc == [0] * calls
    want = out[calls].cpu().numpy()
    assert np.isfinite(want).all()
    for k in range(calls):
        assert np.array_equal(out[k].cpu().numpy(), want), k
    net.close()
