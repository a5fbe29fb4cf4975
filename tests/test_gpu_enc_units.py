"""The tensor-core kernels' two encoders against each other, feature by
feature and bit for bit.

A network whose segments are made of whole 8-feature units is encoded a unit
at a time; the same segments behind one identity input start off a unit's
boundary and go through the general encoder.  One-hot weights pass three
features at a time through the network unchanged (out = relu(f) - relu(-f)),
so the outputs are the encoded operands themselves and must be equal.  Inputs
cover the period's ends, bin edges and values far outside [0, 1)."""
import json

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mlpmod():
    from hairmsnn_gb300 import build, mlp
    build.build()
    return mlp


def config(parts, width):
    return json.dumps({"encoding": {"otype": "Composite", "nested": parts}, "loss": {"otype": "L2"},
                       "optimizer": {"otype": "Adam"},
                       "network": {"otype": "FullyFusedMLP", "n_neurons": width, "n_hidden_layers": 1}})


SEGMENTS = {
    "frequency": ([{"otype": "Frequency", "n_dims_to_encode": 2, "n_frequencies": 6}], 24),
    "oneblob4": ([{"otype": "OneBlob", "n_dims_to_encode": 2, "n_bins": 4}], 8),
    "oneblob8": ([{"otype": "OneBlob", "n_dims_to_encode": 2, "n_bins": 8}], 16),
    "oneblob24": ([{"otype": "OneBlob", "n_dims_to_encode": 2, "n_bins": 24}], 48),
    "oneblob32": ([{"otype": "OneBlob", "n_dims_to_encode": 2, "n_bins": 32}], 64),
    "grid": ([{"otype": "HashGrid", "n_dims_to_encode": 3, "n_levels": 8, "log2_hashmap_size": 9,
               "base_resolution": 3, "per_level_scale": 1.7}], 16),
    "mixed": ([{"otype": "OneBlob", "n_dims_to_encode": 1, "n_bins": 8},
               {"otype": "Frequency", "n_dims_to_encode": 1, "n_frequencies": 4},
               {"otype": "OneBlob", "n_dims_to_encode": 1, "n_bins": 16}], 32),
}


@pytest.mark.parametrize("width", [64, 128])
@pytest.mark.parametrize("prec", ["fp16", "bf16", "fp8"])
@pytest.mark.parametrize("name", sorted(SEGMENTS))
def test_units_equal_general_encoder(mlpmod, name, prec, width):
    parts, n_feat = SEGMENTS[name]
    dims = sum(p["n_dims_to_encode"] for p in parts)
    ident = {"otype": "Identity", "n_dims_to_encode": 1}
    rng = np.random.default_rng(len(name))
    edges = np.array([0.0, 1.0, -1.0, 2.0, 0.5, 1.0 / 24, 23.0 / 24, 31.0 / 32, np.nextafter(np.float32(1), 0), -1e-7])
    x = np.concatenate([np.repeat(edges[:, None], dims, 1), rng.uniform(0, 1, (120, dims)),
                        rng.uniform(-1.5, 2.5, (150, dims))]).astype(np.float32)
    one = np.ones((len(x), 1), np.float32)
    nets = [(mlpmod.TinyMLP(config(parts + [ident], width), dims + 1, 3, precision=prec), np.hstack([x, one]), 0),
            (mlpmod.TinyMLP(config([ident] + parts, width), dims + 1, 3, precision=prec), np.hstack([one, x]), 1)]
    table = None
    for f0 in range(0, n_feat, 3):
        outs = []
        for net, xin, shift in nets:
            d = net.info()
            p = np.zeros(d.n_params, np.float32)
            w0, w1 = p[:width * d.padded_input_width], p[width * d.padded_input_width:d.n_network_params]
            for o in range(3):
                f = min(f0 + o, n_feat - 1) + shift
                w0.reshape(width, -1)[2 * o, f], w0.reshape(width, -1)[2 * o + 1, f] = 1.0, -1.0
                w1.reshape(16, width)[o, 2 * o], w1.reshape(16, width)[o, 2 * o + 1] = 1.0, -1.0
            n_table = d.n_params - d.n_network_params
            if n_table:
                table = rng.uniform(-0.5, 0.5, n_table).astype(np.float32) if table is None else table
                p[d.n_network_params:] = table
            net.set_params(p)
            outs.append(net.inference(torch.from_numpy(np.ascontiguousarray(xin)).cuda()).cpu().numpy())
        assert np.abs(outs[0]).max() > 0 or name.startswith("oneblob")
        assert np.array_equal(outs[0].view(np.int32) & 0x7fffffff, outs[1].view(np.int32) & 0x7fffffff), f0
        assert np.array_equal(outs[0], outs[1])
