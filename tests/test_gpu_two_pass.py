"""The two-pass occlusion raster on caller geometry, GPU against the oracle bit
for bit: an occluder threshold set by the caller is taken as it is, in scenes of
any size, so near-plane-clipped occluders, ties, slivers, meshlets of a few
pixels and all three schedules go through occluders, hierarchical depth, filter
and survivors; the default draws scenes this small in one pass."""
import numpy as np
import pytest

from tests.parity import compare_frame
from tests.test_gpu_edge_geometry import _edge_mesh, _transforms
from tests.test_gpu_small_meshlets import _scene

pytestmark = pytest.mark.gpu


def _edge_scene(lh, camera):
    pos, tris = _edge_mesh()
    if camera == "front":
        u = lh.make_uniforms((0.0, 0.0, -2.4), 1.5707963, 0.0, 60.0, 640, 480, 3)
    else:
        u = lh.make_uniforms((0.05, -0.1, -0.012), 1.5707963, 0.35, 100.0, 640, 480, 3)
    return lh.Scene.from_mesh(pos, tris, _transforms(), u).upload(0)


def _check(lh, oracle, scene, w, h, shadow, cap, tunings):
    """The scene at its default tuning, in one pass, then at each of `tunings`, in two."""
    r = lh.Renderer(lh.Config(width=w, height=h, shadow_size=shadow, max_instances=1024, max_draws=cap))
    r.set_scene(scene)
    fr = oracle.run_scene(scene, shadow_size=shadow, max_instances=1024, max_draws=cap)
    r.frame(scene.uniforms)
    assert list(r.status().occlusion) == [0, 0, 0]
    seen = []
    for tuning in tunings:
        r.set_tuning(**dict({"schedule": 0, "small_px": 32, "medium_px": 32}, **tuning))
        r.frame(scene.uniforms)
        st = r.status()
        errors, stats = compare_frame(r, fr, cap, 1024)
        assert not errors, "%s: %s %s" % (tuning, "\n".join(errors), stats)
        assert st.flags == fr.flags
        assert r.tuning().occlusion_px == tuning["occlusion_px"]
        occ, opaque, alpha = (int(x) for x in st.occlusion)
        assert occ + opaque + alpha > 0 and occ + opaque <= st.visible_opaque[0], (tuning, occ, opaque, alpha)
        seen.append((occ, opaque, st))
    return seen


@pytest.mark.parametrize("camera", ["front", "near"])
def test_edge_geometry_in_two_passes(native, oracle, camera):
    scene = _edge_scene(native, camera)
    seen = _check(native, oracle, scene, 640, 480, 1024, 200000, [
        {"occlusion_px": 127},
        {"occlusion_px": 16},                                     # most meshlets are occluders
        {"occlusion_px": 1},
        {"occlusion_px": 65536},                                  # none but those at the camera plane
        {"occlusion_px": 16, "small_px": 0, "medium_px": 0},      # every triangle through the chunk queue, twice
        {"occlusion_px": 16, "schedule": native.SCHEDULE_PERSISTENT},
        {"occlusion_px": 16, "schedule": native.SCHEDULE_PER_VIEW},
    ])
    assert seen[1][0] > 10 and seen[2][0] >= seen[1][0] >= seen[0][0] >= seen[3][0]
    if camera == "near":
        # meshlets that reach the camera plane are occluders at any threshold
        assert seen[3][0] > 0


@pytest.mark.parametrize("scales,copies,window,pixels", [
    ((0.05, 1.0), 6, (333, 217), (1, 3)),
    ((0.3, 1.0), 130, (641, 359), (8, 32)),
    ((3.0, 4.0, 5.0), 5, (1279, 719), (32, 127)),
])
def test_small_meshlets_in_two_passes(native, oracle, scales, copies, window, pixels):
    scene, n = _scene(native, scales, copies, *window)
    seen = _check(native, oracle, scene, window[0], window[1], 512, 40000, [{"occlusion_px": p} for p in pixels])
    assert seen[0][0] > 0
    assert np.all([s[2].fragments[0] > 100 for s in seen])
