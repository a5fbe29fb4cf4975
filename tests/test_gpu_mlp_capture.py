"""Inference and training steps captured in a CUDA graph use the parameters of
the moment of the replay, whoever changed them since: the host, a training step
outside the graph, or one inside it.  Every comparison is with a direct call on
the same parameters: the same kernels, equal bit for bit."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

N = 700
PRECS = ["fp32", "fp16", "bf16", "fp8"]


@pytest.fixture(scope="module")
def mods():
    from hairmsnn_gb300 import _ffi, build, mlp
    build.build()
    L = _ffi.lib()
    L.hm_mlp_inference_noalloc.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int64, ctypes.c_void_p]
    return _ffi, mlp, L


def setup(mlp, prec, seed=3):
    net = mlp.TinyMLP("hairmsnn_cache.json", 12, 3, precision=prec, seed=seed)
    g = torch.Generator().manual_seed(seed)
    x = (torch.rand(N, 12, generator=g) - 0.5).cuda()
    t = torch.rand(N, 3, generator=g).cuda()
    net.set_params(net.params() + np.float32(0.01))
    return net, x, t


def call(mods, net, x, out, noalloc):
    ffi, _, L = mods
    f = L.hm_mlp_inference_noalloc if noalloc else L.hm_mlp_inference
    ffi.check(f(net._h, x.data_ptr(), out.data_ptr(), N, torch.cuda.current_stream().cuda_stream))


def direct(mods, net, x, noalloc):
    out = torch.full((N, 3), float("nan"), device="cuda")
    call(mods, net, x, out, noalloc)
    torch.cuda.synchronize()
    return out


def captured(mods, net, x, noalloc):
    out = torch.full((N, 3), float("nan"), device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call(mods, net, x, out, noalloc)
    torch.cuda.synchronize()
    return g, out


@pytest.mark.parametrize("noalloc", [False, True])
@pytest.mark.parametrize("prec", PRECS)
def test_replay_follows_the_parameters(mods, prec, noalloc):
    net, x, t = setup(mods[1], prec)
    first = direct(mods, net, x, noalloc)
    g, out = captured(mods, net, x, noalloc)
    changes = [lambda: net.set_params(net.params() * np.float32(1.5)), lambda: net.training_step(x, t),
               lambda: net.optimizer_step(), lambda: net.reset()]
    last = first
    for change in changes:
        change()
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        replayed = out.clone()
        now = direct(mods, net, x, noalloc)
        assert torch.equal(replayed, now)
        assert not torch.equal(now, last)
        last = now


@pytest.mark.parametrize("prec", PRECS)
def test_capture_before_the_first_use_of_new_parameters(mods, prec):
    net, x, _ = setup(mods[1], prec)
    direct(mods, net, x, False)
    net.set_params(net.params() * np.float32(1.5))
    captured(mods, net, x, False)  # never replayed
    fresh, _, _ = setup(mods[1], prec)
    fresh.set_params(fresh.params() * np.float32(1.5))
    assert torch.equal(direct(mods, net, x, False), direct(mods, fresh, x, False))


@pytest.mark.parametrize("prec", PRECS)
def test_replayed_training_steps_reach_later_calls(mods, prec):
    net, x, t = setup(mods[1], prec)
    net.training_step(x, t)
    direct(mods, net, x, False)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        net.training_step(x, t)
    last = direct(mods, net, x, False)
    for _ in range(2):
        g.replay()
        torch.cuda.synchronize()
        now = direct(mods, net, x, False)
        fresh, _, _ = setup(mods[1], prec)
        fresh.set_params(net.params())
        assert torch.equal(now, direct(mods, fresh, x, False))
        assert not torch.equal(now, last)
        last = now
