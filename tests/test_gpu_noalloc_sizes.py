"""lh_cull_instances_noalloc over the sizes where its two kernels and their
tiles end: one cluster of 8 blocks up to 4,096 instances, 1,024-instance tiles
with a look-back above.  Entries stand in instance order, so the sector of the
first n instances is the beginning of the sector of all of them."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOTAL = 20011
SIZES = (1, 31, 32, 33, 249, 255, 256, 257, 1023, 1024, 1025, 3073, 4095, 4096, 4097, 4351, 4352, 4353, 8191, 5119, 5120, 5121, 8191, 8193, 16641, TOTAL)


def test_noalloc_cull_sizes(native):
    import torch
    lh = native
    L = lh.lib()
    L.lh_cull_instances_noalloc.argtypes = [C.c_void_p, C.c_uint32, C.c_void_p, C.c_void_p, C.c_uint32, C.c_void_p,
                                            C.c_void_p]
    L.lh_cull_instances_noalloc.restype = C.c_int32
    scene = lh.Scene(5, n_instances=TOTAL, detail=0.05, width=320, height=180).upload(0)
    d = scene.desc
    r = lh.Renderer(lh.Config(width=320, height=180, shadow_size=128, max_instances=TOTAL, max_draws=2000000))
    r.set_scene(scene)
    r.frame(scene.uniforms)
    ref = r.prefix_sector(0)
    count = int(ref[:8].view(np.uint64)[0]) >> 32
    entries = ref[8:8 + 8 * count].view(np.uint32).reshape(-1, 2)
    assert count > 100 and np.all(np.diff(entries[:, 0].astype(np.int64)) > 0)
    flags = torch.zeros(1, dtype=torch.int32, device="cuda")
    for n in SIZES:
        sector = torch.full((8 + 8 * TOTAL,), 0xAB, dtype=torch.uint8, device="cuda")
        st = L.lh_cull_instances_noalloc(d.device_instances, n, C.addressof(scene.uniforms), sector.data_ptr(), n,
                                         flags.data_ptr(), None)
        assert st == 0
        torch.cuda.synchronize()
        got = sector.cpu().numpy()
        want = entries[entries[:, 0] < n]
        total = int(want[-1, 1]) if len(want) else 0
        assert int(got[:8].view(np.uint64)[0]) == (len(want) << 32) | total, n
        assert np.array_equal(got[8:8 + 8 * len(want)].view(np.uint32).reshape(-1, 2), want), n
        assert np.all(got[8 + 8 * len(want):] == 0xAB), n
        assert int(flags.item()) == 0, n
