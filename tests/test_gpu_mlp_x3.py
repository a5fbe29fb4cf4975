"""FP32 inference on the tensor cores (three BF16 planes per operand) at the
sizes where its tiles and chunks end, against the FP64 oracle and against the
FP32 multiply-add layers of the training forward.

  outputs   |gpu - ref| <= 2e-4 * rms(ref) + 1e-4 * |ref|  (as test_gpu_mlp.py)
  forward   |inference - forward| <= 2e-5 * (rms + |forward|): both are FP32
            results, each within a few 1e-6 of 64 bits
  rows with infinite or huge values are computed with the training forward's
  own arithmetic: equal bit for bit, infinities and NaNs included
"""
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


def config(width, hidden, in_ch, freqs):
    nested = [{"otype": "Frequency", "n_dims_to_encode": 1, "n_frequencies": freqs}] if freqs else []
    return json.dumps({"encoding": {"otype": "Composite", "nested": nested + [{"otype": "Identity"}]},
                       "loss": {"otype": "L2"}, "optimizer": {"otype": "Adam"},
                       "network": {"otype": "FullyFusedMLP", "n_neurons": width, "n_hidden_layers": hidden,
                                   "init": "he_normal"}})


@pytest.mark.parametrize("n,width,hidden,in_ch,freqs", [
    (1, 64, 2, 12, 0), (127, 16, 1, 3, 0), (128, 32, 14, 17, 0), (129, 64, 1, 40, 4), (1000, 128, 5, 12, 8),
    (333, 16, 3, 5, 40), (40961, 64, 2, 9, 12), (20011, 128, 1, 130, 10), (257, 32, 2, 12, 110)])
def test_inference_at_tile_edges(mlpmod, n, width, hidden, in_ch, freqs):
    net = mlpmod.TinyMLP(config(width, hidden, in_ch, freqs), in_ch, 3, seed=n % 1000)
    oc = mo.Config(net.config_text, in_ch, 3)
    x = np.random.default_rng(n).uniform(-1, 1, (n, in_ch)).astype(np.float32)
    d = torch.from_numpy(x).cuda()
    out = net.inference(d).cpu().numpy()
    m = min(n, 4096)
    ref = mo.forward(oc, net.params().astype(np.float64), x[-m:])[0][:, :3]
    rms = np.sqrt(np.mean(ref ** 2))
    assert (np.abs(out[-m:] - ref) <= 2e-4 * rms + 1e-4 * np.abs(ref)).all()
    fwd = net.forward(d).cpu().numpy()
    assert (np.abs(out - fwd) <= 2e-5 * (np.sqrt(np.mean(fwd.astype(np.float64) ** 2)) + np.abs(fwd))).all()


@pytest.mark.parametrize("width,hidden", [(16, 1), (64, 2), (128, 3)])
def test_huge_and_infinite_rows(mlpmod, width, hidden):
    net = mlpmod.TinyMLP(config(width, hidden, 6, 0), 6, 3, seed=5)
    x = np.random.default_rng(1).uniform(-1, 1, (300, 6)).astype(np.float32)
    x[3, 1], x[140, 0], x[141, 5], x[299, 2] = np.inf, -np.inf, 3.4e38, 1e33
    x[17, 4] = np.nan
    d = torch.from_numpy(x).cuda()
    out, fwd = net.inference(d).cpu().numpy(), net.forward(d).cpu().numpy()
    special = [3, 140, 141, 299]
    assert np.array_equal(out[special], fwd[special], equal_nan=True)
    rest = np.setdiff1d(np.arange(300), special)
    assert np.array_equal(np.isnan(out[rest]), np.isnan(fwd[rest]))
    a, b = out[rest][~np.isnan(fwd[rest])], fwd[rest][~np.isnan(fwd[rest])]
    assert (np.abs(a - b) <= 2e-5 * (np.sqrt(np.mean(b.astype(np.float64) ** 2)) + np.abs(b))).all()


def test_new_parameters_are_repacked(mlpmod):
    net = mlpmod.TinyMLP(config(64, 2, 6, 0), 6, 3, seed=5)
    d = torch.rand(200, 6, device="cuda")
    first = net.inference(d)
    net.set_params(net.params() * np.float32(2.0))
    assert torch.allclose(net.inference(d), 8.0 * first, rtol=1e-5, atol=1e-6)  # three matrices doubled
