"""Texel gradients of the resolve adjoint for textures of every shape the
scatter treats apart: one texel, one wide, one high, up to 64 texels (summed
in shared memory) and more.  With one colour everywhere the image does not
depend on a texture's size and a sample's four weights add to 1, so the
gradients of a texture's texels add to the gradient of the 1 x 1 texture.
Tolerance: ~15,000 pixels' terms of one sign in float32, their sums in any
order within 1e-5 of each other, the weights' sum within 2^-22 of 1; ten
times that."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _totals(lh, scene, w, h):
    import torch
    d = scene.desc
    texels = torch.tensor([180, 140, 90, 255], dtype=torch.uint8, device="cuda").repeat(w * h)
    table = (lh.Texture * d.n_textures)()
    for t in table:
        t.texels, t.width, t.height, t.srgb = texels.data_ptr(), w, h, 0
    r = lh.Renderer(lh.Config(width=d.width, height=d.height, shadow_size=256, max_instances=1024, max_draws=200000))
    r.set_scene(scene)
    lh._check(lh.lib().lh_set_scene(r.ctx, d.device_instances, d.n_instances, table, d.n_textures),
              "lh_set_scene", r.ctx)
    r.frame(scene.uniforms)
    grads = torch.zeros(d.n_textures, h, w, 4, device="cuda")
    where = torch.tensor([g.data_ptr() for g in grads], dtype=torch.int64, device="cuda")
    upstream = torch.ones(d.height, d.width, 4, device="cuda")
    targets = lh.GradTargets(texture_grads=where.data_ptr())
    lh._check(lh.lib().lh_resolve_backward(r.ctx, upstream.data_ptr(), C.byref(targets), None), "lh_resolve_backward",
              r.ctx)
    torch.cuda.synchronize()
    return grads.double().sum((1, 2)).cpu().numpy()


def test_texel_gradients_add_up(native):
    lh = native
    scene = lh.Scene(1, detail=0.3, width=160, height=96).upload(0)
    want = _totals(lh, scene, 1, 1)
    scale = np.abs(want).max()
    assert scale > 1.0
    for w, h in ((1, 5), (5, 1), (2, 2), (3, 7), (1, 97), (97, 1), (64, 2), (33, 31)):
        got = _totals(lh, scene, w, h)
        assert np.all(np.isfinite(got))
        assert np.abs(got - want).max() <= 1e-4 * scale, (w, h, np.abs(got - want).max() / scale)
