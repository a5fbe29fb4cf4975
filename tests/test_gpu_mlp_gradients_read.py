"""Reading a handle's gradients is a read: it allocates no device memory (it
works when none is left), changes nothing, and may be done from several threads
at once."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "fp16", "bf16", "fp8"])
def test_reading_gradients(prec):
    from hairmsnn_gb300 import build, mlp
    build.build()
    net = mlp.TinyMLP("hairmsnn_cache.json", 12, 3, precision=prec, seed=3)
    x = torch.rand(3000, 12, generator=torch.Generator().manual_seed(1)).cuda()
    t = torch.rand(3000, 3, generator=torch.Generator().manual_seed(2)).cuda()
    net.training_step(x, t)
    net.params()  # the read-back path's own set-up
    other = mlp.TinyMLP("hairmsnn_cache.json", 12, 3, precision=prec, seed=3)
    other.training_step(x, t)
    other.gradients()  # loads what the read launches
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    first = net.gradients()
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] == free
    got = [None] * 4
    threads = [threading.Thread(target=lambda k=k: got.__setitem__(k, net.gradients())) for k in range(4)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert np.abs(first).max() > 0
    assert all(np.array_equal(g, first) for g in got)
