"""Bytes of the display transform on both sides of every rounding boundary of
the sRGB encoding.  The table holds one colour, so each channel is encoded from
a known value.  Rounding on the way (six blends of a value with itself, a power
of 2 ulp and the scaling, in float32) moves the code by less than 2e-4, so at
3e-4 and 3e-3 from a boundary, on both sides of the guard, the byte is certain."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_display_bytes_at_the_boundaries(native):
    import torch
    lh = native
    scene = lh.Scene(1, detail=0.05, width=64, height=36).upload(0)
    r = lh.Renderer(lh.Config(width=64, height=36, shadow_size=64, max_instances=1024, max_draws=200000))
    r.set_scene(scene)
    r.frame(scene.uniforms)
    steps = np.array([-3e-3, -3e-4, 3e-4, 3e-3])
    code = (np.arange(1, 256)[:, None] + steps[None, :]).reshape(-1)  # before floor, 255 x + 0.5
    encoded = (code - 0.5) / 255.0
    knee = 0.003130 * 12.92
    linear = np.where(encoded <= knee, encoded / 12.92, ((np.maximum(encoded, knee) + 0.055) / 1.055) ** 2.4)
    keep = np.abs(linear - 0.003130) > 1e-5  # the two branches do not meet exactly
    code, linear = code[keep], linear[keep].astype(np.float32)
    code, linear = code[:len(code) // 3 * 3].reshape(-1, 3), linear[:len(linear) // 3 * 3].reshape(-1, 3)
    special = np.array([[0.0, -1.0, np.nan], [1.0, 1.5, 2.0]], np.float32)
    out = torch.zeros(36 * 64 * 4, dtype=torch.uint8, device="cuda")
    rows = [(v, np.floor(c)) for v, c in zip(linear, code)]
    rows += [(special[0], np.zeros(3)), (special[1], np.full(3, 255.0))]
    for v, want in rows:
        lut = np.ones((48, 48, 48, 4), np.float32)
        lut[..., :3] = v
        lut_dev = torch.from_numpy(lut).cuda()
        r.display_transform(out.data_ptr(), lut_dev.data_ptr())
        torch.cuda.synchronize()
        got = out.cpu().numpy().reshape(-1, 4)
        assert np.all(got[:, :3] == want.astype(np.uint8)), (v, want, np.unique(got[:, :3], axis=0))
        assert np.all(got[:, 3] == 255)
