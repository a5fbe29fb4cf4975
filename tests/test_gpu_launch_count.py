"""hm_render_timings.kernel_launches: the kernels of one frame, as replayed from
a graph or launched stage by stage, for every cache precision."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# forward, backward, weight gradients and their sum, hash-grid scatter and
# conversion, Adam; then the FP32 step encodes in a kernel of its own, the
# others pack their weights (E4M3: after the weights' maxima)
TRAIN = {"fp32": 8, "fp16": 8, "bf16": 8, "fp8": 9}
# encoder and layers in one kernel for the 16-bit types
INFER = {"fp32": 2, "fp16": 1, "bf16": 1, "fp8": 2}


@pytest.fixture(scope="module")
def scene():
    from hairmsnn_gb300 import build, render
    build.build()
    s = render.Scene(render.straight_hair_scene(64, 64, strands=200, control_points=16, path_v2=6, triangles=200))
    s.build()
    return s


@pytest.mark.parametrize("timing", [False, True])
@pytest.mark.parametrize("train", [False, True])
@pytest.mark.parametrize("prec", sorted(TRAIN))
def test_msnn_frame(scene, prec, train, timing):
    from hairmsnn_gb300 import mlp, render
    r = render.Renderer(scene, mode=render.MSNN, beta=1, precision=mlp.PRECISIONS[prec], train=train)
    r.instrument(timing=timing)
    for _ in range(2):  # captured in the first one, replayed in the second
        r.frame()
        r.wait()
        t = r.timings()
        # camera, five kernels a round, finalize, compose; a graph's frame number
        path = 1 + 5 * t.bounces + 2 + (0 if timing else 1)
        assert t.kernel_launches == path + INFER[prec] + (TRAIN[prec] if train else 0)


@pytest.mark.parametrize("timing", [False, True])
def test_path_traced_frame(scene, timing):
    from hairmsnn_gb300 import render
    r = render.Renderer(scene, mode=render.PT)
    r.instrument(timing=timing)
    for _ in range(2):
        r.frame()
        r.wait()
        t = r.timings()
        assert t.kernel_launches == 1 + 5 * t.bounces + 1 + (0 if timing else 1)
