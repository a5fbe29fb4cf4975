"""FP32 inference on the tensor cores at the ends of what its three BF16 planes
can carry.

  range     weights that are infinite or round to infinity in BF16, sums and
            outputs that overflow in one half of the K steps: rows with such a
            sum have the training forward's results (FP32 multiply-adds in
            input order), bit for bit, infinities and NaNs included
  depth     rows computed that way on the deepest and widest network do not
            run out the other warps' waits
  accuracy  rms error against 64 bits on the same inputs below 1e-6 of the
            outputs' rms, and not above the multiply-adds'.  FP32's rounding is
            6e-8 a step; leaving out any one of the six partial products costs
            2^-17 to 2^-18 of |a||w|, 4e-6 and more"""
import json

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mlp():
    from hairmsnn_gb300 import build, mlp
    build.build()
    return mlp


def config(width, hidden):
    return json.dumps({"encoding": {"otype": "Identity"}, "loss": {"otype": "L2"}, "optimizer": {"otype": "Adam"},
                       "network": {"otype": "FullyFusedMLP", "n_neurons": width, "n_hidden_layers": hidden,
                                   "init": "he_normal"}})


def matrices(p, in_pad, width, hidden):
    out, off = [], 0
    for k in range(hidden + 1):
        rows, cols = (16 if k == hidden else width), (in_pad if k == 0 else width)
        out.append(p[off:off + rows * cols].reshape(rows, cols))
        off += rows * cols
    return out


def infinite(m):
    m[1][2, 3] = np.inf


def rounds_to_infinity(m):
    m[0][5, 7] = 3.395e38


def negative(m):
    m[0][5, 7] = -3.4e38
    m[1][0, 1] = -np.inf


def halves_overflow(m):  # even K steps to +inf, odd ones to -inf: the multiply-adds stay at +inf
    m[0][4, :] = 0.0
    m[0][4, 0], m[0][4, 16] = 2e38, -2e38


def output_halves_overflow(m):
    m[0][0, :], m[0][16, :] = 2.0, 2.0
    for k in range(1, len(m) - 1):
        m[k][0, :], m[k][16, :] = 0.5, 0.5
    m[-1][0, :] = 0.0
    m[-1][0, 0], m[-1][0, 16] = 3e38, -3e38


@pytest.mark.parametrize("change", [infinite, rounds_to_infinity, negative, halves_overflow, output_halves_overflow])
@pytest.mark.parametrize("width,hidden", [(32, 2), (64, 2), (128, 5)])
def test_weights_and_sums_out_of_range(mlp, width, hidden, change):
    net = mlp.TinyMLP(config(width, hidden), 32, 3, seed=4)
    p = net.params()
    change(matrices(p, 32, width, hidden))
    net.set_params(p)
    x = torch.from_numpy(np.random.default_rng(2).uniform(3, 5, (300, 32)).astype(np.float32)).cuda()
    out, fwd = net.inference(x).cpu().numpy(), net.forward(x).cpu().numpy()
    if hidden == 2 and change is not negative:  # (ReLU turns NaNs into zeros on a longer way)
        assert not np.isfinite(fwd[:, 0]).all()
    assert np.array_equal(out, fwd, equal_nan=True)


@pytest.mark.parametrize("n,every", [(40000, 1), (40000, 37), (129, 1)])
@pytest.mark.parametrize("width", [16, 128])
def test_rows_out_of_range_on_the_deepest_network(mlp, width, n, every):
    net = mlp.TinyMLP(config(width, 14), 40, 3, seed=6)
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (n, 40)).astype(np.float32)
    x[::every, 11] = rng.choice(np.array([np.inf, -np.inf, 2e30, -3.4e38, np.nan], np.float32), len(x[::every]))
    d = torch.from_numpy(x).cuda()
    out = net.inference(d).cpu().numpy()
    fwd = net.forward(d).cpu().numpy()
    assert np.array_equal(out[::every], fwd[::every], equal_nan=True)
    again = net.inference(d).cpu().numpy()  # reports a wait that ran out in the call before
    assert np.array_equal(out, again, equal_nan=True)


@pytest.mark.parametrize("width,hidden,in_ch", [(16, 1, 16), (16, 3, 48), (32, 2, 32), (64, 1, 64), (64, 2, 64),
                                                (64, 5, 144), (64, 14, 64), (128, 1, 128), (128, 5, 144)])
def test_error_against_64_bits(mlp, width, hidden, in_ch):
    n = 8192
    net = mlp.TinyMLP(config(width, hidden), in_ch, 3, seed=9)
    x = np.random.default_rng(width + hidden).uniform(-1, 1, (n, in_ch)).astype(np.float32)
    d = torch.from_numpy(x).cuda()
    h = x.astype(np.float64)
    ms = matrices(net.params().astype(np.float64), in_ch, width, hidden)
    for k, m in enumerate(ms):
        h = h @ m.T
        if k < hidden:
            h = np.maximum(h, 0.0)
    ref = h[:, :3]
    rms = np.sqrt(np.mean(ref ** 2))
    err = [np.sqrt(np.mean((y.cpu().numpy() - ref) ** 2)) / rms for y in (net.inference(d), net.forward(d))]
    assert err[0] <= 1e-6 and err[0] <= err[1], err
