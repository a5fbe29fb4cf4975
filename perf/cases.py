"""The work that a user of hairmsnn_gb300 has it do, as timed cases.

Five kinds of work, each through the package's public calls:

  bsdf    a batch of hair vertices through bsdf_eval / bsdf_sample /
          bsdf_eval_grad
  infer   TinyMLP.inference: the radiance cache queried for a batch
  train   TinyMLP.training_step and the gradients of it
  trace   Scene.trace: a batch of rays against the hair and the head
  render  Renderer.frame: whole frames of path tracing or HairMSNN

listed() holds the sizes that are met most (the per-vertex batch, one frame's
cache queries, one frame's training records, the bench scene), draw() the
ranges around them.  Everything a case needs is made from its seed on the GPU.
"""
import json
import math
import os

import numpy as np
import torch

import hairmsnn_gb300 as hm
from hairmsnn_gb300 import mlp, render

# hair material of the benchmark: sigma_a, beta_m, beta_n, alpha (radians)
SIGMA_A = (0.06, 0.1, 0.2)
CONFIGS = {"c1_w64": "c1_cache_w64.json",    # Frequency + OneBlob, 5 x 64
           "c1_w128": "c1_cache_w128.json",  # Frequency + OneBlob, 5 x 128
           "grid": "hairmsnn_cache.json"}    # the renderer's: hash grid + OneBlob, 2 x 64
IN_CH = {"c1_w64": 16, "c1_w128": 16, "grid": 12}


def listed():
    return [
        # the per-vertex batch of the benchmark's vertex workload: BSDF values
        {"name": "bsdf_eval_262144", "kind": "bsdf", "op": "eval", "n": 262144, "beta_m": 0.3, "beta_n": 0.3},
        # importance sampling for a large wavefront of vertices, an odd count
        {"name": "bsdf_sample_8000003", "kind": "bsdf", "op": "sample", "n": 8000003, "beta_m": 0.3, "beta_n": 0.3},
        # appearance fitting: values and material derivatives of a vertex batch
        {"name": "bsdf_grad_100003", "kind": "bsdf", "op": "grad", "n": 100003, "beta_m": 0.3, "beta_n": 0.3},
        # the smallest calls: a handful of cache queries (a probe, a preview tile)
        {"name": "infer_grid_fp32_517", "kind": "infer", "config": "grid", "precision": "fp32", "n": 517},
        # the renderer's cache over every pixel of a 512x512 frame, default precision
        {"name": "infer_grid_fp32_262144", "kind": "infer", "config": "grid", "precision": "fp32", "n": 262144},
        # the large batch of the precision sweep, FP16 operands
        {"name": "infer_c1w64_fp16_1048576", "kind": "infer", "config": "c1_w64", "precision": "fp16", "n": 1048576},
        # the wide network with 8-bit operands on a ragged batch
        {"name": "infer_c1w128_fp8_300007", "kind": "infer", "config": "c1_w128", "precision": "fp8", "n": 300007},
        # one frame's training step of the renderer's cache, default precision
        {"name": "train_grid_fp32_16384", "kind": "train", "config": "grid", "precision": "fp32", "n": 16384},
        # the large training batch of the precision sweep
        {"name": "train_c1w64_fp16_65536", "kind": "train", "config": "c1_w64", "precision": "fp16", "n": 65536},
        # closest hits of a 512x512 camera image's rays
        {"name": "trace_closest_262144", "kind": "trace", "rays": "camera", "any_hit": False, "n": 262144,
         "hair": "straight", "strands": 10000, "control_points": 64},
        # the flagship: HairMSNN frames with online cache training at 512x512
        {"name": "render_msnn_512x512", "kind": "render", "mode": "msnn", "width": 512, "height": 512, "frames": 4,
         "beta": 1, "precision": "fp32", "hair": "straight", "strands": 10000, "control_points": 64},
        # a small plain path-traced preview
        {"name": "render_pt_160x120", "kind": "render", "mode": "pt", "width": 160, "height": 120, "frames": 2,
         "beta": 1, "precision": "fp32", "hair": "straight", "strands": 5000, "control_points": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bsdf", "infer", "infer", "train", "train", "trace", "render"])
    if kind == "bsdf":
        op = rng.choice(["eval", "sample", "grad"])
        return {"kind": kind, "op": op, "n": _log_int(rng, 1000, 1000000 if op == "grad" else 4000000),
                "beta_m": round(rng.uniform(0.15, 0.6), 3), "beta_n": round(rng.uniform(0.15, 0.6), 3)}
    if kind in ("infer", "train"):
        case = {"kind": kind, "config": rng.choice(sorted(CONFIGS)),
                "precision": rng.choice(["fp32", "fp16", "bf16", "fp8"])}
        case["n"] = _log_int(rng, 300, 1000000) if kind == "infer" else _log_int(rng, 2000, 70000)
        return case
    hair = {"hair": rng.choice(["straight", "curly"]), "strands": _log_int(rng, 2000, 12000),
            "control_points": rng.randint(48, 80)}
    if kind == "trace":
        return {"kind": kind, "rays": rng.choice(["camera", "scatter"]), "any_hit": rng.random() < 0.5,
                "n": _log_int(rng, 1000, 500000), **hair}
    return {"kind": kind, "mode": rng.choice(["msnn", "pt"]), "width": _log_int(rng, 96, 400),
            "height": _log_int(rng, 96, 400), "frames": rng.randint(1, 3), "beta": rng.randint(1, 3),
            "precision": "fp32", **hair}


# ------------------------------------------------------------------ inputs
def _gen(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * int(seed) + salt)
    return g


def _uniform(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float32)


def _unit(g, n):
    v = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float32)
    return v / v.norm(dim=1, keepdim=True)


def _hair_values(case):
    return [*SIGMA_A, case["beta_m"], case["beta_n"], 3.14159 * 2.0 / 180.0, 1.0, 1.0, 1.0, 1.0]


def _bsdf_inputs(case, seed):
    """Vertices with directions and fibre tangents uniform on the sphere, h and
    the sampling numbers uniform."""
    g, n = _gen(seed, 1), case["n"]
    wo, wi, t = (_unit(g, n).t().contiguous() for _ in range(3))
    h = 2.0 * _uniform(g, n) - 1.0
    u = _uniform(g, 4, n)
    return wo, wi, t, h, u


def _mlp_inputs(case, seed):
    """Cache queries: position, directions and (c1) the material, as the
    renderer and the vertex workload pack them."""
    g, n = _gen(seed, 2), case["n"]
    if case["config"] == "grid":
        x = torch.zeros(n, 12, device="cuda")
        x[:, 0:3] = _uniform(g, n, 3) - 0.5
        x[:, 3:6] = _unit(g, n)
        x[:, 6:9] = _unit(g, n)
        return x
    x = torch.zeros(n, 16, device="cuda")
    x[:, 0:3] = 2.0 * _uniform(g, n, 3) - 1.0
    x[:, 3:7] = _uniform(g, n, 4)
    x[:, 7] = 2.0 * _uniform(g, n) - 1.0
    x[:, 8:11] = torch.tensor(SIGMA_A, device="cuda")
    x[:, 11:13] = 0.3
    return x


def _targets(case, seed):
    """Radiance: positive, log-normal."""
    return torch.randn(case["n"], 3, generator=_gen(seed, 3), device="cuda").exp()


def _config(case):
    path = os.path.join(os.path.dirname(os.path.abspath(mlp.__file__)), "configs", CONFIGS[case["config"]])
    with open(path) as f:
        return json.load(f)


def _layout(case):
    """Encoding segments, weight matrices [(offset, rows, columns)], counts."""
    cfg = _config(case)
    segs, in_off, out_off, tables = [], 0, 0, 0
    for e in cfg["encoding"]["nested"]:
        dims = e.get("n_dims_to_encode", IN_CH[case["config"]] - in_off)
        s = {"type": e["otype"], "in": in_off, "dims": dims}
        if s["type"] == "Identity":
            width = dims
        elif s["type"] == "Frequency":
            s["freqs"] = e["n_frequencies"]
            width = dims * s["freqs"] * 2
        elif s["type"] == "OneBlob":
            s["bins"] = e["n_bins"]
            width = dims * s["bins"]
        else:
            s["levels"] = []
            for k in range(e["n_levels"]):
                scale = e["base_resolution"] * e["per_level_scale"] ** k - 1.0
                res = int(math.ceil(scale)) + 1
                size = min(2 ** e["log2_hashmap_size"], (res ** 3 + 7) // 8 * 8)
                s["levels"].append((scale, res, size, tables))
                tables += size
            width = 2 * e["n_levels"]
        segs.append(s)
        in_off, out_off = in_off + dims, out_off + width
    net = cfg["network"]
    width, hidden = net["n_neurons"], net["n_hidden_layers"]
    pad = (out_off + 15) // 16 * 16
    mats, off = [], 0
    for k in range(hidden + 1):
        rows, cols = (16 if k == hidden else width), (pad if k == 0 else width)
        mats.append((off, rows, cols))
        off += rows * cols
    return {"segs": segs, "encoded": out_off, "pad": pad, "mats": mats, "matrix": off, "params": off + 2 * tables,
            "width": width, "hidden": hidden}


def _weights(case, seed):
    """He-normal matrices; hash tables as training leaves them."""
    lay = _layout(case)
    rng = np.random.default_rng([int(seed), 4])
    p = np.empty(lay["params"], np.float32)
    for off, rows, cols in lay["mats"]:
        p[off:off + rows * cols] = rng.standard_normal(rows * cols, dtype=np.float32) * math.sqrt(2.0 / cols)
    p[lay["matrix"]:] = (rng.random(lay["params"] - lay["matrix"], dtype=np.float32) - 0.5) * 0.4
    return p


def _scene(case, seed):
    cfg = render.straight_hair_scene(case.get("width", 512), case.get("height", 512), strands=case["strands"],
                                     control_points=case["control_points"], seed=1 + int(seed))
    if case["hair"] == "curly":
        cfg["hair"]["procedural"].update(type="curly", helix_radius=0.04, helix_pitch=0.1)
    return render.Scene(cfg)


def _rays(case, seed, scene):
    """camera: one jittered ray for each point of a regular grid on the image
    plane; scatter: rays that leave points around the hair in any direction."""
    g, n = _gen(seed, 5), case["n"]
    if case["rays"] == "camera":
        pos, d00, du, dv = torch.from_numpy(scene.export("camera").reshape(4, 3).copy()).cuda()
        side = max(1, int(math.sqrt(n)))
        k = torch.arange(n, device="cuda")
        rows = (n + side - 1) // side
        jit = _uniform(g, n, 2)
        su = ((k % side).float() + jit[:, 0]) / side
        sv = ((k // side).float() + jit[:, 1]) / rows
        d = d00 + su[:, None] * du + sv[:, None] * dv
        org = pos.expand(n, 3).contiguous()
    else:
        org = _unit(g, n) * (0.9 + 0.6 * _uniform(g, n, 1))
        d = _unit(g, n)
    return org, (d / d.norm(dim=1, keepdim=True)).contiguous()


def prepare(case, seed):
    state = {"case": case}
    kind = case["kind"]
    if kind == "bsdf":
        state["in"] = _bsdf_inputs(case, seed)
        state["hair"] = _hair_values(case)
    elif kind in ("infer", "train"):
        state["x"] = _mlp_inputs(case, seed)
        state["net"] = mlp.TinyMLP(CONFIGS[case["config"]], IN_CH[case["config"]], 3, precision=case["precision"])
        state["net"].set_params(_weights(case, seed))
        if kind == "train":
            state["target"] = _targets(case, seed)
    else:
        state["scene"] = _scene(case, seed)
        state["scene"].build()
        if kind == "trace":
            state["rays"] = _rays(case, seed, state["scene"])
        else:
            mode = {"msnn": render.MSNN, "pt": render.PT}[case["mode"]]
            state["renderer"] = render.Renderer(state["scene"], mode=mode, beta=case["beta"],
                                                precision=mlp.PRECISIONS[case["precision"]])
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "bsdf":
        wo, wi, t, h, u = state["in"]
        if case["op"] == "eval":
            f, pdf = hm.bsdf_eval(wo, wi, t, h, state["hair"])
            return {"f": f, "pdf": pdf}
        if case["op"] == "sample":
            w, f, pdf = hm.bsdf_sample(wo, t, h, u, state["hair"])
            return {"wi": w, "f": f, "pdf": pdf}
        f, pdf, df, dpdf = hm.bsdf_eval_grad(wo, wi, t, h, state["hair"])
        return {"f": f, "pdf": pdf, "df": df, "dpdf": dpdf}
    if kind == "infer":
        return {"out": state["net"].inference(state["x"])}
    if kind == "train":
        loss = state["net"].training_step(state["x"], state["target"])
        return {"loss": loss, "gradients": state["net"].gradients()}
    if kind == "trace":
        hits = state["scene"].trace(*state["rays"], any_hit=case["any_hit"])
        if case["any_hit"]:  # which of a ray's occluders is reported depends on timing: the answer is whether there is one
            return {"occluded": hits.view(torch.int32)[:, 1] >= 0}
        return {"t": hits[:, 0], "prim": hits.view(torch.int32)[:, 1], "uv": hits[:, 2:4]}
    r = state["renderer"]
    r.reset()
    for _ in range(case["frames"]):
        r.frame()
    r.wait()
    return {"image": (r.device_sums() / case["frames"]).float()}


def work(case):
    kind = case["kind"]
    if kind == "bsdf":
        # floats read and written per vertex; arithmetic of the four lobes,
        # a transcendental counted as one operation
        floats = {"eval": 10 + 4, "sample": 11 + 7, "grad": 10 + 4 + 24}[case["op"]]
        flops = {"eval": 350, "sample": 500, "grad": 1500}[case["op"]]
        return {"bytes": 4.0 * floats * case["n"], "flops": float(flops) * case["n"]}
    if kind in ("infer", "train"):
        lay, n = _layout(case), case["n"]
        first, rest = lay["encoded"] * lay["width"], (lay["hidden"] - 1) * lay["width"] ** 2 + 3 * lay["width"]
        if kind == "infer":
            return {"bytes": 4.0 * (n * (IN_CH[case["config"]] + 3) + lay["params"]), "flops": 2.0 * n * (first + rest)}
        grid = lay["params"] > lay["matrix"]  # the encoding has parameters: gradients go through layer 0
        return {"bytes": 4.0 * (n * (IN_CH[case["config"]] + 3) + 8 * lay["params"]),
                "flops": 2.0 * n * ((3 if grid else 2) * first + 3 * rest)}
    curves = 16.0 * case["strands"] * case["control_points"]
    if kind == "trace":
        return {"bytes": 40.0 * case["n"] + curves, "flops": 1000.0 * case["n"]}
    pixels = case["width"] * case["height"]
    return {"bytes": 24.0 * pixels * case["frames"] + curves, "flops": 2.0e4 * pixels * case["frames"]}


# ------------------------------------------------------------------ 64 bits
def _dot(a, b):
    return (a * b).sum(0)


def _norm(a):
    return a / _dot(a, a).sqrt()


def _cross(a, b):
    return torch.stack([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]])


ETA = 1.55


class _Hair:
    """The hair BSDF (Chiang et al. 2016, four lobes) in 64 bits."""

    def __init__(self, m):
        bm, bn, alpha = m[3], m[4], m[5]
        v0 = (0.726 * bm + 0.812 * bm ** 2 + 3.7 * bm ** 20) ** 2
        self.sigma = m[0:3]
        self.v = [v0, 0.25 * v0, 4.0 * v0]
        self.s = 0.626657069 * (0.265 * bn + 1.194 * bn ** 2 + 5.372 * bn ** 22)
        sin2k, cos2k = [alpha.sin()], [alpha.cos()]
        for _ in range(2):
            sin2k.append(2.0 * cos2k[-1] * sin2k[-1])
            cos2k.append(cos2k[-1] ** 2 - sin2k[-2] ** 2)
        self.sin2k, self.cos2k = sin2k, cos2k
        self.lo = 1.0 / (1.0 + (math.pi / self.s).exp())
        self.span = 1.0 - 2.0 * self.lo

    def tilt(self, p, st, ct):
        if p == 0:
            return st * self.cos2k[1] - ct * self.sin2k[1], ct * self.cos2k[1] + st * self.sin2k[1]
        k = 0 if p == 1 else 2
        return st * self.cos2k[k] + ct * self.sin2k[k], ct * self.cos2k[k] - st * self.sin2k[k]

    def geometry(self, wo, h):
        st = wo[0]
        ct = (1.0 - st ** 2).clamp_min(0.0).sqrt()
        sin_gt = h * ct / (ETA ** 2 - st ** 2).sqrt()
        cos_gt = (1.0 - sin_gt ** 2).clamp_min(0.0).sqrt()
        go, gt = h.asin(), sin_gt.clamp(-1.0, 1.0).asin()
        fac = 2.0 * cos_gt / (1.0 - (st / ETA) ** 2).sqrt()
        T = torch.stack([(-s * fac).exp() for s in self.sigma])
        f0 = ((1.0 - ETA) / (1.0 + ETA)) ** 2
        fr = f0 + (1.0 - f0) * (1.0 - ct * go.cos()) ** 5
        a1 = (1.0 - fr) ** 2 * T
        a2 = a1 * T * fr
        a = [fr.expand_as(T), a1, a2, a2 * fr * T / (1.0 - T * fr)]
        mean = [x.mean(0) for x in a]
        total = mean[0] + mean[1] + mean[2] + mean[3]
        return st, ct, go, gt, a, [x / total for x in mean]

    def mp(self, cti, cto, sti, sto, v):
        a, b = cti * cto / v, sti * sto / v
        i0, term = torch.zeros_like(a), torch.ones_like(a)
        for k in range(10):
            i0 = i0 + term
            term = term * a * a / (4.0 * (k + 1) ** 2)
        if float(v) > 0.1:
            return (-b).exp() * i0 / ((1.0 / v).sinh() * 2.0 * v)
        big = a + 0.5 * (-math.log(2.0 * math.pi) - a.clamp_min(1e-30).log() + 1.0 / (8.0 * a.clamp_min(1e-30)))
        log_i0 = torch.where(a > 12.0, big, i0.log())
        return (log_i0 - b - 1.0 / v + 0.6931 + (1.0 / (2.0 * v)).log()).exp()

    def eval(self, wo, wi, h):
        st, ct, go, gt, a, ap = self.geometry(wo, h)
        sti = wi[0]
        cti = (1.0 - sti ** 2).clamp_min(0.0).sqrt()
        phi = torch.atan2(wi[2], wi[1]) - torch.atan2(wo[2], wo[1])
        f = torch.zeros_like(a[1])
        pdf = torch.zeros_like(st)
        for p in range(4):
            if p == 3:
                m, nn = self.mp(cti, ct, sti, st, self.v[2]), 1.0 / (2.0 * math.pi)
            else:
                sop, cop = self.tilt(p, st, ct)
                m = self.mp(cti, cop.abs(), sti, sop, self.v[p])
                d = phi - (2.0 * p * gt - 2.0 * go + p * math.pi)
                d = torch.remainder(d + math.pi, 2.0 * math.pi) - math.pi
                e = (-d.abs() / self.s).exp()
                nn = e / (self.s * (1.0 + e) ** 2) / self.span
            f = f + m * a[p] * nn
            pdf = pdf + m * ap[p] * nn
        return f, pdf

    def sample(self, wo, h, u):
        st, ct, go, gt, _, ap = self.geometry(wo, h)
        sin_gt = h * ct / (ETA ** 2 - st ** 2).sqrt()
        gt = sin_gt.clamp(-1.0, 1.0).asin()
        c0, c1, c2 = ap[0], ap[0] + ap[1], ap[0] + ap[1] + ap[2]
        p = (u[0] >= c0).long() + (u[0] >= c1).long() + (u[0] >= c2).long()
        pick = lambda xs: torch.stack([x.expand_as(st) for x in xs]).gather(0, p[None])[0]  # noqa: E731
        tilts = [self.tilt(k, st, ct) for k in range(3)] + [(st, ct)]
        sop, cop = pick([x[0] for x in tilts]), pick([x[1] for x in tilts])
        v = pick([*self.v, self.s])  # the last lobe takes s in the reference's layout
        e2 = u[1].clamp_min(1e-5)
        cos_th = 1.0 + v * (e2 + (1.0 - e2) * (-2.0 / v).exp()).log()
        sin_th = (1.0 - cos_th ** 2).clamp_min(0.0).sqrt()
        sti = -cos_th * sop + sin_th * (2.0 * math.pi * u[2]).cos() * cop
        cti = (1.0 - sti ** 2).clamp_min(0.0).sqrt()
        x = (-self.s * (1.0 / (u[3] * self.span + self.lo) - 1.0).log()).clamp(-math.pi, math.pi)
        lobe = p.double()
        dphi = torch.where(p < 3, 2.0 * lobe * gt - 2.0 * go + lobe * math.pi + x, 2.0 * math.pi * u[3])
        phi = torch.atan2(wo[2], wo[1]) + dphi
        return _norm(torch.stack([sti, cti * phi.cos(), cti * phi.sin()]))


def _exact_bsdf(case, seed):
    wo, wi, t, h, u = (x.double() for x in _bsdf_inputs(case, seed))
    y = _norm(_cross(wo, t))
    z = _norm(_cross(t, y))
    local = lambda w: _norm(torch.stack([_dot(t, w), _dot(y, w), _dot(z, w)]))  # noqa: E731
    material = torch.tensor(_hair_values(case)[:6], dtype=torch.float32).double().cuda()
    if case["op"] == "eval":
        f, pdf = _Hair(material).eval(local(wo), local(wi), h)
        return {"f": f, "pdf": pdf}
    if case["op"] == "sample":
        hair, lo = _Hair(material), local(wo)
        w = hair.sample(lo, h, u)
        f, pdf = hair.eval(lo, w, h)
        return {"wi": _norm(w[0] * t + w[1] * y + w[2] * z), "f": f, "pdf": pdf}
    lo, li = local(wo), local(wi)
    df, dpdf = [], []
    for k in range(6):
        e = torch.zeros_like(material)
        e[k] = 1.0
        (f, pdf), (d, dp) = torch.func.jvp(lambda m: _Hair(m).eval(lo, li, h), (material,), (e,))
        df.append(d)
        dpdf.append(dp)
    return {"f": f, "pdf": pdf, "df": torch.stack(df), "dpdf": torch.stack(dpdf)}


def _encode(lay, x, tables):
    cols = []
    for s in lay["segs"]:
        xs = x[:, s["in"]:s["in"] + s["dims"]]
        if s["type"] == "Identity":
            cols.append(xs)
        elif s["type"] == "Frequency":
            a = xs[:, :, None] * 2.0 ** torch.arange(s["freqs"], device=x.device)
            a = math.pi * torch.remainder(a, 2.0)
            cols.append(torch.stack([a.sin(), a.cos()], -1).flatten(1))
        elif s["type"] == "OneBlob":
            nb = s["bins"]
            edge = torch.arange(nb + 1, device=x.device, dtype=x.dtype) / nb
            cdf = 0.0
            for k in (-1.0, 0.0, 1.0):
                q = (edge - xs[:, :, None] + k) * nb
                cdf = cdf + (q * (15.0 - 10.0 * q ** 2 + 3.0 * q ** 4) / 16.0 + 0.5).clamp(0.0, 1.0)
            cdf = torch.cat([cdf[..., :nb], cdf[..., :1] + 1.0], -1)
            cols.append((cdf[..., 1:] - cdf[..., :-1]).flatten(1))
        else:
            for scale, res, size, off in s["levels"]:
                f = xs * scale + 0.5
                g = f.floor()
                w, g = f - g, g.long()
                acc = 0.0
                for c in range(8):
                    bit = [(c >> k) & 1 for k in range(3)]
                    i = [(g[:, k] + bit[k]) & 0xFFFFFFFF for k in range(3)]
                    stride, index = 1, 0
                    for k in range(3):
                        if stride > size:
                            break
                        index = (index + i[k] * stride) & 0xFFFFFFFF
                        stride *= res
                    if size < stride:
                        index = i[0] ^ (i[1] * 2654435761 & 0xFFFFFFFF) ^ (i[2] * 805459861 & 0xFFFFFFFF)
                    wt = 1.0
                    for k in range(3):
                        wt = wt * (w[:, k] if bit[k] else 1.0 - w[:, k])
                    acc = acc + wt[:, None] * tables[off + index % size]
                cols.append(acc)
    n_pad = lay["pad"] - lay["encoded"]
    return torch.cat([*cols, torch.ones(len(x), n_pad, device=x.device, dtype=x.dtype)], 1)


def _exact_mlp(case, seed):
    lay = _layout(case)
    params = torch.from_numpy(_weights(case, seed)).cuda().double()
    x = _mlp_inputs(case, seed).double()

    def forward(p, rows):
        h = _encode(lay, rows, p[lay["matrix"]:].view(-1, 2))
        for k, (off, r, c) in enumerate(lay["mats"]):
            h = h @ p[off:off + r * c].view(r, c).t()
            if k < lay["hidden"]:
                h = h.relu()
        return h[:, :3]

    step = 1 << 16
    if case["kind"] == "infer":
        return {"out": torch.cat([forward(params, x[k:k + step]) for k in range(0, len(x), step)])}
    target, params = _targets(case, seed).double(), params.requires_grad_(True)
    loss = 0.0
    for k in range(0, len(x), step):
        out = forward(params, x[k:k + step])
        lum = (out * torch.tensor([0.299, 0.587, 0.114], device="cuda", dtype=torch.float64)).sum(1, keepdim=True)
        part = ((out - target[k:k + step]) ** 2 / (lum ** 2 + 0.01).detach()).sum() / target.numel()
        part.backward()
        loss += float(part)
    return {"loss": torch.tensor([loss], dtype=torch.float64), "gradients": params.grad}


def exact(case, seed):
    if case["kind"] == "bsdf":
        return _exact_bsdf(case, seed)
    if case["kind"] in ("infer", "train"):
        return _exact_mlp(case, seed)
    # rays against half a million curves, and frames of a random walk through
    # them: no closed form, and far more than seconds in 64 bits
    return None
