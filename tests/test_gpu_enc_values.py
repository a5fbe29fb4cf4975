"""The encoded operands of the tensor-core kernels, feature by feature, against
the 64-bit encoding: every inference form, the training forward, and the copies
that a training forward keeps for the weight gradients.

Inference and forward: one-hot weights pass three features at a time through the
network (out = relu(f) - relu(-f)).  The copies: with an output gradient on one
row only, the gradient of a first-layer weight is that row's feature times the
gradient at the hidden unit, which is made 1.

Bounds, derived: the operand's rounding (FP16 2^-11, BF16 2^-8 of the value; E4M3
2^-4 of the value with the row's scale, twice, as the hidden activation is
rounded again) plus 2e-5 for the FP32 evaluation (a OneBlob mass is a difference
of sums up to 3 at slopes up to 32 bins: 32 x 3 x 2^-24, twice)."""
import ctypes
import json

import numpy as np
import pytest

from oracle import mlp_oracle as mo

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

REL = {"fp16": 2.0 ** -11, "bf16": 2.0 ** -8, "fp8": 2.0 ** -3}
KEPT = {"fp16": 2.0 ** -11, "bf16": 2.0 ** -8, "fp8": 2.0 ** -11}  # E4M3 rows are kept as FP16
ABS = 2e-5
IDENT = {"otype": "Identity", "n_dims_to_encode": 1}
SEGMENTS = {
    "frequency": [{"otype": "Frequency", "n_dims_to_encode": 2, "n_frequencies": 6}],
    "oneblob4": [{"otype": "OneBlob", "n_dims_to_encode": 2, "n_bins": 4}],
    "oneblob8": [{"otype": "OneBlob", "n_dims_to_encode": 2, "n_bins": 8}],
    "oneblob24": [{"otype": "OneBlob", "n_dims_to_encode": 2, "n_bins": 24}],
    "oneblob32": [{"otype": "OneBlob", "n_dims_to_encode": 1, "n_bins": 32}],
    "oneblob5": [{"otype": "OneBlob", "n_dims_to_encode": 2, "n_bins": 5}],  # general encoder
    "grid": [{"otype": "HashGrid", "n_dims_to_encode": 3, "n_levels": 8, "log2_hashmap_size": 9,
              "base_resolution": 3, "per_level_scale": 1.7}],
    "mixed": [{"otype": "OneBlob", "n_dims_to_encode": 1, "n_bins": 8},
              {"otype": "Frequency", "n_dims_to_encode": 1, "n_frequencies": 4},
              {"otype": "OneBlob", "n_dims_to_encode": 1, "n_bins": 16}],
}


@pytest.fixture(scope="module")
def mods():
    from hairmsnn_gb300 import _ffi, build, mlp
    build.build()
    L = _ffi.lib()
    L.hm_debug_tc_path.argtypes = [ctypes.c_int]
    L.hm_mlp_inference_noalloc.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int64, ctypes.c_void_p]
    yield _ffi, mlp, L
    L.hm_debug_tc_path(0)


def setup(mlp, name, prec, width):
    """network, oracle, inputs (last one 1), hash tables, the encoding in 64 bits"""
    parts = SEGMENTS[name]
    dims = sum(p["n_dims_to_encode"] for p in parts)
    cfg = json.dumps({"encoding": {"otype": "Composite", "nested": parts + [IDENT]}, "loss": {"otype": "L2"},
                      "optimizer": {"otype": "Adam"},
                      "network": {"otype": "FullyFusedMLP", "n_neurons": width, "n_hidden_layers": 1}})
    net = mlp.TinyMLP(cfg, dims + 1, 3, precision=prec)
    oc = mo.Config(cfg, dims + 1, 3)
    rng = np.random.default_rng(len(name))
    edges = np.array([0.0, 0.5, 1.0 / 24, 23.0 / 24, 31.0 / 32, np.nextafter(np.float32(1), 0), -1e-7, -0.5])
    x = np.concatenate([np.repeat(edges[:, None], dims, 1), rng.uniform(0, 1, (133, dims)),
                        rng.uniform(-1, 1, (159, dims))]).astype(np.float32)
    x = np.hstack([x, np.ones((len(x), 1), np.float32)])
    p = np.zeros(oc.n_params, np.float32)
    p[oc.n_net_params:] = rng.uniform(-0.5, 0.5, oc.n_params - oc.n_net_params)
    return net, oc, x, p, mo.encode(oc, p.astype(np.float64), x, exact_phase=True)


def matrices(oc, p):
    return [p[off:off + fo * fi].reshape(fo, fi) for off, fo, fi in oc.layer_shapes]


@pytest.mark.parametrize("width", [32, 64, 128])
@pytest.mark.parametrize("prec", ["fp16", "bf16", "fp8"])
@pytest.mark.parametrize("name", sorted(SEGMENTS))
def test_operands(mods, name, prec, width):
    ffi, mlp, L = mods
    net, oc, x, p, ref = setup(mlp, name, prec, width)
    d = torch.from_numpy(x).cuda()
    n_feat = oc.segs[-1]["out_off"] + 1

    def noalloc():
        out = torch.empty(len(x), 3, device="cuda")
        ffi.check(L.hm_mlp_inference_noalloc(net._h, d.data_ptr(), out.data_ptr(), len(x),
                                             torch.cuda.current_stream().cuda_stream))
        return out

    forms = {"automatic": (0, lambda: net.inference(d)), "two kernels": (1, lambda: net.inference(d)),
             "one kernel": (1, noalloc), "training": (0, lambda: net.forward(d))}
    for f0 in range(0, n_feat, 3):
        feats = [min(f0 + o, n_feat - 1) for o in range(3)]
        w0, w1 = matrices(oc, p)
        w0[...], w1[...] = 0.0, 0.0
        for o, f in enumerate(feats):
            w0[2 * o, f], w0[2 * o + 1, f] = 1.0, -1.0
            w1[o, 2 * o], w1[o, 2 * o + 1] = 1.0, -1.0
        net.set_params(p)
        for form, (path, call) in forms.items():
            assert L.hm_debug_tc_path(path) == 0
            out = call().cpu().numpy()
            assert (np.abs(out - ref[:, feats]) <= REL[prec] * np.abs(ref[:, feats]) + ABS).all(), (form, feats)
    L.hm_debug_tc_path(0)


@pytest.mark.parametrize("prec", ["fp16", "bf16", "fp8"])
@pytest.mark.parametrize("name", sorted(SEGMENTS))
def test_kept_copies(mods, name, prec):
    _, mlp, _ = mods
    net, oc, x, p, ref = setup(mlp, name, prec, 64)
    w0, w1 = matrices(oc, p)
    w0[0, oc.segs[-1]["out_off"]] = 1.0  # a hidden unit that is 1 for every row
    w1[0, 0] = 1.0
    net.set_params(p)
    d = torch.from_numpy(x).cuda()
    net.forward(d)
    for row in (0, 5, 7, 130, 150, len(x) - 1):
        dy = torch.zeros(len(x), 3, device="cuda")
        dy[row, 0] = 1.0
        net.backward_output_grad(dy)
        got = net.gradients()[:oc.in_pad]
        assert (np.abs(got - ref[row]) <= KEPT[prec] * np.abs(ref[row]) + ABS).all(), row
