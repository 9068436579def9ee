"""What a context keeps of freed device memory: a map's buffers, however large, for the next
map; of a call's temporaries at most 4 GiB; nothing once it is destroyed."""

import ctypes as C
import gc

import pytest

pytestmark = pytest.mark.gpu

GIB = 1 << 30


def _free():
    import torch

    return torch.cuda.mem_get_info()[0]


def _mesh(n):
    import torch

    t = torch.arange(n + 1, dtype=torch.float64, device="cuda") / n
    return torch.stack(torch.meshgrid(t, t, indexing="ij"), -1).reshape(-1, 2).contiguous()


def test_map_buffers_are_kept():
    import torch

    from otmap_b200 import native as N

    n = 12288
    xy, density = _mesh(n), torch.ones(n * n, dtype=torch.float64, device="cuda")
    size = 8 * (xy.numel() + density.numel())  # 3.6e9: above 4 GiB together with a second map's
    gc.collect()  # contexts of other tests
    torch.cuda.empty_cache()
    ctx = N.Context(0)
    free = _free()

    def create(count):
        maps = []
        for _ in range(count):
            h = C.c_void_p()
            N.check(N.lib().otm_map_create(ctx.handle, n, N.ptr(xy), N.ptr(density), C.byref(h)))
            maps.append(h)
        for h in maps:
            N.check(N.lib().otm_map_destroy(h))
        ctx.profile(0)  # synchronises

    create(3)
    assert free - _free() >= 3 * size
    create(3)
    assert 3 * size <= free - _free() <= 3 * size + GIB
    ctx.close()
    assert free - _free() <= GIB


def test_temporaries_are_given_back():
    import torch

    from otmap_b200 import native as N

    n, count = 8192, 6
    xy = _mesh(n)
    out = torch.empty_like(xy)
    gc.collect()  # contexts of other tests
    torch.cuda.empty_cache()
    ctx = N.Context(0)
    free = _free()
    meshes = (C.c_void_p * count)(*[xy.data_ptr()] * count)  # the call stages up to count + 1 meshes of 1 GiB
    weights = (C.c_double * count)(*[1.0 / count] * count)
    N.check(N.lib().otm_mesh_blend(ctx.handle, n, count, meshes, weights, C.c_void_p(out.data_ptr())))
    ctx.profile(0)
    assert free - _free() <= 4 * GIB + GIB
    assert float((out - xy).abs().max()) <= 1e-15
    ctx.close()
