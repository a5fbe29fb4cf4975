"""16-bit networks of width 16: inference and training, against the FP64 oracle
(outputs within 5e-3 of the rms for FP16 operands: a few roundings of 5e-4 each;
FP16 gradients within 2.5e-2 rms, as test_gpu_mlp_tc_train.py; BF16 eight times
both: three significand bits fewer)."""
import json

import numpy as np
import pytest

from oracle import mlp_oracle as mo

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def config(hidden, grid):
    nested = [{"otype": "HashGrid", "n_dims_to_encode": 3, "n_levels": 5, "log2_hashmap_size": 10,
               "base_resolution": 4, "per_level_scale": 2.0}] if grid else []
    return json.dumps({"loss": {"otype": "RelativeL2Luminance"}, "optimizer": {"otype": "Adam"},
                       "encoding": {"otype": "Composite", "nested": nested + [{"otype": "Identity"}]},
                       "network": {"otype": "FullyFusedMLP", "n_neurons": 16, "n_hidden_layers": hidden,
                                   "init": "he_normal"}})


@pytest.mark.parametrize("prec", ["fp16", "bf16"])
@pytest.mark.parametrize("n,hidden,grid", [(1, 1, False), (129, 2, False), (4159, 2, True), (70001, 4, True)])
def test_width_16(n, hidden, grid, prec):
    from hairmsnn_gb300 import build, mlp
    build.build()
    net = mlp.TinyMLP(config(hidden, grid), 12, 3, precision=prec, seed=4)
    oc = mo.Config(net.config_text, 12, 3)
    rng = np.random.default_rng(n)
    p = net.params()
    p[oc.n_net_params:] = rng.uniform(-0.5, 0.5, oc.n_enc_params)
    net.set_params(p)
    x = rng.uniform(0, 1, (n, 12)).astype(np.float32)
    t = rng.lognormal(0.0, 1.0, (n, 3)).astype(np.float32)
    d = torch.from_numpy(x).cuda()
    ref = mo.forward(oc, p.astype(np.float64), x)[0][:, :3]
    rms = np.sqrt(np.mean(ref ** 2))
    k = 1 if prec == "fp16" else 8
    out = net.inference(d).cpu().numpy()
    assert np.sqrt(np.mean((out - ref) ** 2)) <= 5e-3 * k * rms
    assert np.sqrt(np.mean((net.forward(d).cpu().numpy() - ref) ** 2)) <= 5e-3 * k * rms
    net.training_step(d, torch.from_numpy(t).cuda())
    g = net.gradients().astype(np.float64)
    _, gref = mo.backward(oc, p.astype(np.float64), x, t)
    parts = [(off, off + fo * fi) for off, fo, fi in oc.layer_shapes]
    if oc.n_enc_params:
        parts.append((oc.n_net_params, oc.n_params))
    for lo, hi in parts:
        e, r = g[lo:hi] - gref[lo:hi], gref[lo:hi]
        assert np.sqrt(np.mean(e ** 2)) <= 2.5e-2 * k * np.sqrt(np.mean(r ** 2)), lo
