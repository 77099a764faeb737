"""Texel gradients where textures of different sizes share one gradient buffer:
gradients are added to what is there, so the shared buffer holds the sum of what
the textures' own buffers would.  Neighbouring pixels of different materials then
sample the same first address with different neighbours.  Tolerance: the same
terms, some 10,000, summed in another order in float32 (1e-5 of the largest sum),
ten times that."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = ((1, 1), (2, 2), (1, 4), (4, 2), (3, 3))


def _gradients(lh, r, where, upstream):
    import torch
    table = torch.tensor([t.data_ptr() for t in where], dtype=torch.int64, device="cuda")
    targets = lh.GradTargets(texture_grads=table.data_ptr())
    lh._check(lh.lib().lh_resolve_backward(r.ctx, upstream.data_ptr(), C.byref(targets), None), "lh_resolve_backward",
              r.ctx)
    torch.cuda.synchronize()


def test_shared_texel_targets(native):
    import torch
    lh = native
    scene = lh.Scene(2, seed=5, n_instances=400, detail=0.15, width=320, height=180).upload(0)
    d = scene.desc
    sizes = [SIZES[i % len(SIZES)] for i in range(d.n_textures)]
    assert d.n_textures > len(SIZES)
    texels = torch.tensor([180, 140, 90, 255], dtype=torch.uint8, device="cuda").repeat(64)
    table = (lh.Texture * d.n_textures)()
    for t, (w, h) in zip(table, sizes):
        t.texels, t.width, t.height, t.srgb = texels.data_ptr(), w, h, 0
    r = lh.Renderer(lh.Config(width=d.width, height=d.height, shadow_size=256, max_instances=1024, max_draws=200000))
    r.set_scene(scene)
    lh._check(lh.lib().lh_set_scene(r.ctx, d.device_instances, d.n_instances, table, d.n_textures), "lh_set_scene", r.ctx)
    r.frame(scene.uniforms)
    upstream = torch.rand(d.height, d.width, 4, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    own = [torch.zeros(16, 4, device="cuda") for _ in sizes]
    _gradients(lh, r, own, upstream)
    shared = torch.zeros(16, 4, device="cuda")
    _gradients(lh, r, [shared] * len(sizes), upstream)
    want = torch.stack(own).double().sum(0).cpu().numpy()
    got = shared.double().cpu().numpy()
    assert np.abs(want).max() > 1.0 and np.count_nonzero(want[:, 0]) >= 8
    assert np.abs(got - want).max() <= 1e-4 * np.abs(want).max(), (got[:, 0], want[:, 0])
