"""Any-hit rays where the traversal stops spreading them over its warps (five
rays for each lane of the grid: 486,400 at five blocks on each of 152 SMs): a ray
is occluded exactly where it has a closest hit.  Both walk the same tree with the
same intersectors."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene():
    from hairmsnn_gb300 import build, render
    build.build()
    s = render.Scene(render.straight_hair_scene(64, 64, strands=1500, control_points=24, path_v2=6, triangles=500))
    s.build()
    return s


@pytest.mark.parametrize("n", [1, 31, 97281, 486399, 486400, 486401, 1500007])
def test_occluded_where_there_is_a_closest_hit(scene, n):
    g = torch.Generator(device="cuda").manual_seed(n)
    o = torch.randn(n, 3, generator=g, device="cuda")
    o = (o / o.norm(dim=1, keepdim=True) * (0.9 + 0.6 * torch.rand(n, 1, generator=g, device="cuda"))).contiguous()
    d = torch.randn(n, 3, generator=g, device="cuda")
    d = (d / d.norm(dim=1, keepdim=True)).contiguous()
    closest = scene.trace(o, d).view(torch.int32)[:, 1] >= 0
    occluded = scene.trace(o, d, any_hit=True).view(torch.int32)[:, 1] >= 0
    assert torch.equal(closest, occluded)
    if n > 1000:
        assert 0.05 < closest.float().mean() < 0.95
