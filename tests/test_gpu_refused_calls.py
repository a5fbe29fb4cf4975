"""A call refused for lack of memory reports it once: the next call on the same
thread starts clean."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

HUGE = 1 << 31  # x 144 encoded inputs: more than a terabyte, nothing is launched


def test_next_call_does_not_report_the_last_refusal():
    from hairmsnn_gb300 import build, mlp
    build.build()
    net = mlp.TinyMLP("c1_cache_w128.json", 16, 3, seed=2)
    x = torch.rand(1500, 16, device="cuda")
    first = net.inference(x)
    torch.cuda.synchronize()
    st = mlp.lib().hm_mlp_inference(net._h, x.data_ptr(), first.data_ptr(), HUGE,
                                    torch.cuda.current_stream().cuda_stream)
    assert st == 5  # HM_ENOMEM
    assert torch.equal(net.inference(x), first)
