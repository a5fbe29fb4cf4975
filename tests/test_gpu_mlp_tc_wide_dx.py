"""Tensor-core training of a network with hash tables behind more than 256
encoded inputs: the input gradients come in several matrix products, 256 columns
the widest, whose last one may be 16 or 32 wide.  Against the FP64 oracle as
test_gpu_train_shapes.py."""
import json

import numpy as np
import pytest

from oracle import mlp_oracle as mo

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp16", "fp8"])
@pytest.mark.parametrize("n,width,bins", [(129, 32, 27), (700, 64, 28), (300, 64, 56), (2111, 128, 60)])
def test_gradients(n, width, bins, prec):
    from hairmsnn_gb300 import build, mlp
    build.build()
    cfg = json.dumps({"loss": {"otype": "RelativeL2Luminance"}, "optimizer": {"otype": "Adam"},
                      "encoding": {"otype": "Composite", "nested": [
                          {"otype": "OneBlob", "n_dims_to_encode": 9, "n_bins": bins},
                          {"otype": "HashGrid", "n_dims_to_encode": 3, "n_levels": 5, "log2_hashmap_size": 10,
                           "base_resolution": 4, "per_level_scale": 2.0}]},
                      "network": {"otype": "FullyFusedMLP", "n_neurons": width, "n_hidden_layers": 1,
                                  "init": "he_normal"}})
    net = mlp.TinyMLP(cfg, 12, 3, precision=prec, seed=4)
    oc = mo.Config(net.config_text, 12, 3)
    assert oc.n_net_params == net.info().n_network_params and net.info().padded_input_width > 256 - 16
    rng = np.random.default_rng(n)
    p = net.params()
    p[oc.n_net_params:] = rng.uniform(-0.5, 0.5, oc.n_enc_params)
    net.set_params(p)
    x = rng.uniform(0, 1, (n, 12)).astype(np.float32)
    t = rng.lognormal(0.0, 1.0, (n, 3)).astype(np.float32)
    net.training_step(torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda())
    g = net.gradients().astype(np.float64)
    _, ref = mo.backward(oc, p.astype(np.float64), x, t)
    bound = 2.5e-2 if prec == "fp16" else 3e-1  # E4M3: as test_gpu_mlp_tc_train.py
    for lo, hi in [(off, off + fo * fi) for off, fo, fi in oc.layer_shapes] + [(oc.n_net_params, oc.n_params)]:
        d, r = g[lo:hi] - ref[lo:hi], ref[lo:hi]
        assert np.sqrt(np.mean(d ** 2)) <= bound * np.sqrt(np.mean(r ** 2)), lo
