"""Training gradients at the sizes where the weight-gradient kernels' tiles
and chunks end: batches around a stage (64 rows) and a chunk (2048 rows), one
and several input tiles, an encoding wider than 256 features, every network
width.  Against the FP64 oracle, per weight matrix and for the hash tables:
FP32 within 2e-4 of the largest gradient (as test_gpu_mlp.py), FP16 within
2.5e-2 rms (as test_gpu_mlp_tc_train.py; the operand rounding dominates)."""
import json

import numpy as np
import pytest

from oracle import mlp_oracle as mo

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mlpmod():
    from hairmsnn_gb300 import build, mlp
    build.build()
    return mlp


def config(width, hidden, encoding):
    nested = {"wide": [{"otype": "Frequency", "n_dims_to_encode": 12, "n_frequencies": 12}],
              "small": [{"otype": "OneBlob", "n_dims_to_encode": 4, "n_bins": 4}, {"otype": "Identity"}],
              "grid": [{"otype": "HashGrid", "n_dims_to_encode": 3, "n_levels": 5, "log2_hashmap_size": 10,
                        "base_resolution": 4, "per_level_scale": 2.0}, {"otype": "Identity"}]}[encoding]
    return json.dumps({"loss": {"otype": "RelativeL2Luminance"}, "optimizer": {"otype": "Adam"},
                       "encoding": {"otype": "Composite", "nested": nested},
                       "network": {"otype": "FullyFusedMLP", "n_neurons": width, "n_hidden_layers": hidden,
                                   "init": "he_normal"}})


@pytest.mark.parametrize("n,width,hidden,encoding,prec", [
    (*shape, prec) for shape in [
        (64, 64, 2, "small"), (65, 64, 2, "grid"), (191, 32, 1, "grid"), (2048, 64, 3, "grid"),
        (2049, 128, 2, "small"), (4159, 32, 2, "grid"), (2111, 64, 1, "wide"), (333, 128, 1, "wide")]
    for prec in ("fp32", "fp16")] + [(4159, 16, 2, "grid", "fp32"), (63, 16, 1, "wide", "fp32")])
def test_gradients_at_tile_edges(mlpmod, n, width, hidden, encoding, prec):
    net = mlpmod.TinyMLP(config(width, hidden, encoding), 12, 3, precision=prec, seed=4)
    oc = mo.Config(net.config_text, 12, 3)
    rng = np.random.default_rng(n)
    p = net.params()
    p[oc.n_net_params:] = rng.uniform(-0.5, 0.5, oc.n_enc_params)
    net.set_params(p)
    x = rng.uniform(0, 1, (n, 12)).astype(np.float32)
    t = rng.lognormal(0.0, 1.0, (n, 3)).astype(np.float32)
    loss = net.training_step(torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()).item()
    ref_loss, ref = mo.backward(oc, p.astype(np.float64), x, t)
    g = net.gradients().astype(np.float64)
    assert abs(loss - ref_loss) <= (1e-4 if prec == "fp32" else 2e-3) * abs(ref_loss)
    parts = [(off, off + fo * fi) for off, fo, fi in oc.layer_shapes]
    if oc.n_enc_params:
        parts.append((oc.n_net_params, oc.n_params))
    for lo, hi in parts:
        d, r = g[lo:hi] - ref[lo:hi], ref[lo:hi]
        if prec == "fp32":
            assert np.abs(d).max() <= 2e-4 * np.abs(r).max(), (lo, np.abs(d).max() / np.abs(r).max())
        else:
            assert np.sqrt(np.mean(d ** 2)) <= 2.5e-2 * np.sqrt(np.mean(r ** 2)), lo


@pytest.mark.parametrize("prec,n,encoding", [("fp32", 700001, "wide"), ("fp16", 2000001, "small")])
def test_gradients_of_a_batch_whose_partials_go_in_several_launches(mlpmod, prec, n, encoding):
    """More than 64 M floats of weight-gradient partials (104 k / 72 k per
    chunk of 1024 / 2048 rows): the sum of the gradients of two parts, each in
    one launch and cut at a chunk's end.  The partials are the same numbers;
    three sums of at most 980 of them, mostly of one sign, err by at most
    3 x 980 x 2^-24 = 1.8e-4 of the sum."""
    net = mlpmod.TinyMLP(config(128, 5, encoding), 12, 3, precision=prec, seed=4)
    gen = torch.Generator(device="cuda").manual_seed(n)
    x = torch.rand(n, 12, generator=gen, device="cuda")
    dy = torch.rand(n, 3, generator=gen, device="cuda") / n
    cut = n // 4096 * 2048

    def grads(rows):
        net.forward(x[rows])
        net.backward_output_grad(dy[rows])
        return net.gradients().astype(np.float64)

    whole = grads(slice(0, n))
    parts = grads(slice(0, cut)) + grads(slice(cut, n))
    for off, fo, fi in mo.Config(net.config_text, 12, 3).layer_shapes:
        d, r = whole[off:off + fo * fi] - parts[off:off + fo * fi], whole[off:off + fo * fi]
        assert np.abs(r).max() > 0
        assert np.abs(d).max() <= 2e-4 * np.abs(r).max(), (off, np.abs(d).max() / np.abs(r).max())
