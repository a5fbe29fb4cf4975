"""What a training forward leaves for its backward outlives the calls that come
between them: inferences of other sizes, and calls refused for lack of memory
(asked for far more than any device holds, so that nothing is launched)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

N = 1500
HUGE = 1 << 31  # x 144 encoded inputs: more than a terabyte


@pytest.fixture(scope="module")
def mlp():
    from hairmsnn_gb300 import build, mlp
    build.build()
    return mlp


def setup(mlp, prec):
    net = mlp.TinyMLP("c1_cache_w128.json", 16, 3, precision=prec, seed=2)
    g = torch.Generator().manual_seed(1)
    return net, torch.rand(N, 16, generator=g).cuda(), torch.rand(N, 3, generator=g).cuda()


def gradients(mlp, prec):
    net, x, t = setup(mlp, prec)
    net.forward(x)
    net.backward(t)
    return net.gradients()


def call(mlp, name, net, x, out):
    torch.cuda.synchronize()
    return getattr(mlp.lib(), name)(net._h, x.data_ptr(), out, HUGE, torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("n", [1, N, 5000])
@pytest.mark.parametrize("prec", ["fp32", "fp16", "bf16", "fp8"])
def test_inference_between_forward_and_backward(mlp, prec, n):
    net, x, t = setup(mlp, prec)
    net.forward(x)
    net.inference(torch.rand(n, 16, device="cuda"))
    net.backward(t)
    assert np.array_equal(net.gradients(), gradients(mlp, prec))


def test_refused_inference_keeps_the_forward(mlp):
    net, x, t = setup(mlp, "fp32")
    net.inference(x)
    net.forward(x)
    assert call(mlp, "hm_mlp_inference", net, x, x.data_ptr()) != 0
    net.backward(t)
    assert np.array_equal(net.gradients(), gradients(mlp, "fp32"))
    net.inference(x)


@pytest.mark.parametrize("prec", ["fp32", "fp16", "bf16", "fp8"])
def test_refused_forward_leaves_nothing_to_go_back_through(mlp, prec):
    net, x, t = setup(mlp, prec)
    net.forward(x)
    assert call(mlp, "hm_mlp_forward", net, x, None) != 0
    with pytest.raises(mlp._ffi.HMError):
        net.backward(t)
    net.forward(x)
    net.backward(t)
    assert np.array_equal(net.gradients(), gradients(mlp, prec))
