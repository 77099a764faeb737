"""The raster's packed path for small meshlets, GPU against the oracle bit
for bit, where it can go wrong: meshlets from a fraction of a pixel to past
the 127-pixel reach of its 16-bit offsets, over the edges of a window of odd
size, whole meshlets and quarters of them (few units), units by the hundred
with claims of 1, 8 and guided size, every bin, and the plain and occlusion
passes."""
import numpy as np
import pytest

from tests.parity import compare_frame

pytestmark = pytest.mark.gpu


def _grid(n):
    """An n x n grid of quads over [-1, 1]^2 with a wave across it (meshlets
    of about 60 vertices and 90 triangles, facing -z)."""
    t = np.linspace(-1.0, 1.0, n + 1)
    x, y = np.meshgrid(t, t)
    pos = np.stack([x, y, 0.05 * np.sin(5.0 * x) * np.cos(4.0 * y)], axis=-1).reshape(-1, 3).astype(np.float32)
    a = (np.arange(n)[:, None] * (n + 1) + np.arange(n)[None, :]).reshape(-1)
    tris = np.concatenate([np.stack([a, a + n + 1, a + 1], 1), np.stack([a + 1, a + n + 1, a + n + 2], 1)])
    return pos, tris.astype(np.uint32)


def _scene(lh, scales, copies, w, h):
    """Grids of the given scales side by side and behind one another, past
    the window's edges, seen from the origin along +z."""
    tr = []
    for k in range(copies):
        for i, s in enumerate(scales):
            m = np.eye(4) * s
            c, sn = np.cos(0.4 * k + i), np.sin(0.4 * k + i)
            m[:2, :2] = np.array([[c, -sn], [sn, c]]) * s
            m[:3, 3] = (2.3 * ((k * 7 + i * 3) % 9 - 4), 1.7 * ((k * 5 + i) % 7 - 3), 8.0 + 0.11 * k + 0.4 * i)
            m[3, 3] = 1.0
            tr.append(m)
    u = lh.make_uniforms((0.0, 0.0, 0.0), 1.5707963, 0.0, 70.0, w, h, len(tr))
    pos, tris = _grid(40)
    return lh.Scene.from_mesh(pos, tris, tr, u).upload(0), len(tr)


@pytest.mark.parametrize("case", [
    # (scales, copies, window, tuning)
    ((0.05, 0.2), 6, (333, 217), {}),                                   # sub-pixel meshlets, quarters of meshlets
    ((0.3, 1.0), 130, (641, 359), {}),                                  # thousands of units, guided claims
    ((0.3, 1.0), 130, (641, 359), {"raster_batch": 1, "occlusion_px": 0}),
    ((0.3, 1.0), 130, (641, 359), {"raster_batch": 64, "small_px": 4, "medium_px": 64}),
    ((3.0, 4.0, 5.0), 5, (1279, 719), {"occlusion_px": 0}),             # 60 to 250 pixels: both sides of the reach
    ((3.0, 4.0, 5.0), 5, (1279, 719), {"small_px": 0, "medium_px": 0}),  # every triangle through the chunk queue
])
def test_small_meshlets_match_the_oracle(native, oracle, case):
    lh = native
    scales, copies, (w, h), tuning = case
    scene, n = _scene(lh, scales, copies, w, h)
    r = lh.Renderer(lh.Config(width=w, height=h, shadow_size=512, max_instances=1024, max_draws=40000))
    r.set_scene(scene)
    r.set_tuning(**tuning)
    r.frame(scene.uniforms)
    st = r.status()
    fr = oracle.run_scene(scene, shadow_size=512, max_instances=1024, max_draws=40000)
    errors, stats = compare_frame(r, fr, 40000, 1024)
    assert not errors, "\n".join(errors) + " %s" % stats
    assert st.flags == fr.flags
    assert st.fragments[0] > 100 and stats["covered"] > 100
