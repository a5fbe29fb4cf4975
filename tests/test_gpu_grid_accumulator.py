"""Hash-grid gradients start from zero whatever became of the call before: here
a handle's first backward, recorded into a graph that never runs, with an
accumulator in memory that held something else (tables of a few kilobytes share
the allocator's blocks with the buffers of handles that are gone)."""
import json

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


CONFIG = json.dumps({
    "encoding": {"otype": "Composite", "nested": [
        {"otype": "HashGrid", "n_dims_to_encode": 3, "n_levels": 8, "log2_hashmap_size": 8, "base_resolution": 3,
         "per_level_scale": 1.7}, {"otype": "Identity"}]},
    "loss": {"otype": "L2"}, "optimizer": {"otype": "Adam"},
    "network": {"otype": "FullyFusedMLP", "n_neurons": 64, "n_hidden_layers": 2}})


@pytest.mark.parametrize("replays", [0, 2])
@pytest.mark.parametrize("prec", ["fp32", "fp16"])
def test_gradients_after_a_recorded_backward(prec, replays):
    from hairmsnn_gb300 import build, mlp
    build.build()
    x = (torch.rand(3000, 12, generator=torch.Generator().manual_seed(1)) - 0.5).cuda()
    t = torch.rand(3000, 3, generator=torch.Generator().manual_seed(2)).cuda()

    def step(net):
        net.forward(x)
        net.backward(t)

    ref = mlp.TinyMLP(CONFIG, 12, 3, precision=prec, seed=3)
    step(ref)
    expected = ref.gradients()
    net = mlp.TinyMLP(CONFIG, 12, 3, precision=prec, seed=3)
    net.forward(x)
    torch.cuda.synchronize()
    gone = [mlp.TinyMLP(CONFIG, 12, 3, precision=prec, seed=k) for k in range(8)]
    for k, other in enumerate(gone):
        other.set_params(np.full(other.n_params, 3.0 + k, np.float32))
        step(other)
        other.optimizer_step()
    torch.cuda.synchronize()
    for other in gone:
        other.close()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="relaxed"):  # the first backward allocates
        net.backward(t)
    torch.cuda.synchronize()
    for _ in range(replays):
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(net.gradients(), expected)
    for _ in range(2):
        step(net)
        assert np.array_equal(net.gradients(), expected)
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(net.gradients(), expected)
