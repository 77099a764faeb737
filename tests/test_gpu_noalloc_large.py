"""lh_cull_instances_noalloc past one look-back window (32 tiles of 1,024), past
two, past the tiles that are resident at once, and at the call's limit of 2^20
instances; one more is refused before any launch.  Entries stand in instance
order, so the sector of the first n instances is the beginning of that of all."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMIT = 1 << 20
SIZES = (31 * 1024, 32 * 1024, 32 * 1024 + 1, 33 * 1024 + 1, 64 * 1024, 65 * 1024 + 1, 311299, 700001, LIMIT - 1, LIMIT)


def test_noalloc_cull_to_its_limit(native):
    import torch
    lh = native
    L = lh.lib()
    L.lh_cull_instances_noalloc.argtypes = [C.c_void_p, C.c_uint32, C.c_void_p, C.c_void_p, C.c_uint32, C.c_void_p,
                                            C.c_void_p]
    L.lh_cull_instances_noalloc.restype = C.c_int32
    scene = lh.Scene(5, n_instances=LIMIT, detail=0.05, width=320, height=180).upload(0)
    d = scene.desc
    r = lh.Renderer(lh.Config(width=320, height=180, shadow_size=128, max_instances=LIMIT, max_draws=1 << 20))
    r.set_scene(scene)
    r.frame(scene.uniforms)
    ref = r.prefix_sector(0)
    count = int(ref[:8].view(np.uint64)[0]) >> 32
    entries = ref[8:8 + 8 * count].view(np.uint32).reshape(-1, 2)
    assert count > 10000 and np.all(np.diff(entries[:, 0].astype(np.int64)) > 0)
    flags = torch.zeros(1, dtype=torch.int32, device="cuda")
    sector = torch.empty(8 + 8 * LIMIT, dtype=torch.uint8, device="cuda")

    def call(n):
        sector.fill_(0xAB)
        return L.lh_cull_instances_noalloc(d.device_instances, n, C.addressof(scene.uniforms), sector.data_ptr(), LIMIT,
                                           flags.data_ptr(), None)

    for n in SIZES:
        assert call(n) == 0
        torch.cuda.synchronize()
        got = sector.cpu().numpy()
        want = entries[entries[:, 0] < n]
        assert int(got[:8].view(np.uint64)[0]) == (len(want) << 32) | int(want[-1, 1]), n
        assert np.array_equal(got[8:8 + 8 * len(want)].view(np.uint32).reshape(-1, 2), want), n
        assert np.all(got[8 + 8 * len(want):] == 0xAB), n
        assert int(flags.item()) == 0, n
    ERR_CAPACITY = 4
    assert call(LIMIT + 1) == ERR_CAPACITY
    torch.cuda.synchronize()
    assert bool((sector == 0xAB).all()) and int(flags.item()) == 0
