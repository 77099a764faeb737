"""Device memory a context takes per draw slot: two classes of slots in each of the
main view and the four cascades (draw command 16 B, reference 8 B, draw record
48 B), the main view's four raster lists and the cascades' one (4 B each)."""
import pytest

pytestmark = pytest.mark.gpu


def _taken(lh, max_draws):
    import torch
    before = torch.cuda.mem_get_info()[0]
    r = lh.Renderer(lh.Config(width=64, height=36, shadow_size=64, max_instances=1024, max_draws=max_draws))
    taken = before - torch.cuda.mem_get_info()[0]
    del r
    return taken


def test_bytes_per_draw_slot(native):
    import torch
    torch.zeros(1, device="cuda")
    _taken(native, 1 << 20)
    small, large = _taken(native, 1 << 20), _taken(native, 3 << 20)
    expected = 5 * 2 * (16 + 8 + 48) + (4 + 4) * 4
    # a few allocations, each rounded up to 2 MiB
    assert abs((large - small) - (2 << 20) * expected) <= 16 * (2 << 20), (large - small) / (2 << 20)
