"""A frame's traced rounds replayed from a graph, where rounds 16 to 31, 32 to
63 and so on lie in conditional nodes, against the same rounds launched one by
one: bit for bit, for path lengths around each node's first round and for the
longest a scene may ask for."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def R():
    from hairmsnn_gb300 import build, render
    build.build()
    return render


def scene(R, path_v2):
    cfg = R.straight_hair_scene(64, 64, strands=6000, path_v2=path_v2)
    cfg["hair"]["procedural"].update(type="curly", helix_radius=0.04, helix_pitch=0.1, radius=2e-3)
    cfg["hair"]["sigma_a"] = [0.01, 0.01, 0.01]
    return R.Scene(cfg)


def test_the_scene_has_paths_in_the_conditional_rounds(R):
    r = R.Renderer(scene(R, 40), R.PT)
    r.instrument(timing=True)
    r.frame()
    assert r.timings().paths_by_bounce[17] > 0
    r.close()


@pytest.mark.parametrize("path_v2", [1, 14, 15, 16, 30, 31, 32, 63, 1024])
def test_replayed_rounds_match_single_launches(R, path_v2):
    images = []
    for graphs in (True, False):
        r = R.Renderer(scene(R, path_v2), R.PT, frames_in_flight=2)
        r.set_graphs(graphs)
        for _ in range(4):
            r.frame()
        images.append(r.read(R.IMAGE_FINAL))
        r.close()
    assert np.isfinite(images[0]).all() and images[0].max() > 0
    assert np.array_equal(images[0], images[1])
