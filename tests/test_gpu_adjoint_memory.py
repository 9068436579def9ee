"""The adjoint's workspaces of a context share one allocation: its memory is that of the largest
call, whatever numbers of maps and sizes came before, and a call's gradient does not depend on
what the others left there."""

import ctypes as C
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _loss(ctx, n, count, solves=6):
    import torch

    from otmap_b200 import native as N
    from otmap_b200 import workloads as W

    dens = [torch.from_numpy(np.ascontiguousarray(W.to_cells(W.gaussian_mixture(n, 20 + k)))).cuda()
            for k in range(count)]
    grads = [torch.empty_like(d) for d in dens]
    target = torch.ones(32 * 32, dtype=torch.float64, device="cuda")
    weights = (C.c_double * count)(*[1.0 / count] * count)
    opt, aopt = N.default_options(), N.AdjointOptionsC()
    opt.max_iter = 5
    N.lib().otm_default_adjoint_options(C.byref(aopt))
    aopt.max_iter = solves
    loss = C.c_double()
    arr = lambda ts: (C.c_void_p * count)(*[t.data_ptr() for t in ts])  # noqa: E731
    torch.cuda.synchronize()
    N.check(N.lib().otm_barycenter_loss(ctx.handle, n, count, arr(dens), weights, 32, C.c_void_p(target.data_ptr()),
                                        C.byref(opt), C.byref(aopt), None, C.byref(loss), arr(grads), None))
    return [g.cpu().numpy() for g in grads]


def test_memory_is_that_of_the_largest_call():
    import torch

    from otmap_b200 import native as N

    n = 512  # 41 basis vectors and 8 others of 2 MiB for each map
    gc.collect()  # contexts of other tests
    ctx = N.Context(0)
    _loss(ctx, n, 8)
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    for count in range(7, 0, -1):
        _loss(ctx, n, count)
    torch.cuda.empty_cache()
    # the solver keeps its own workspaces of six batches (23 MiB a map); 28 maps' bases are 2.8 GiB
    assert free - torch.cuda.mem_get_info()[0] <= 1 << 30
    ctx.close()


def test_gradients_do_not_depend_on_earlier_calls():
    from otmap_b200 import native as N

    calls = [(64, 2), (100, 3), (32, 8), (128, 1), (64, 2), (100, 1), (32, 8), (7, 4), (128, 1)]
    ctx = N.Context(0)
    got = [_loss(ctx, n, count, 60) for n, count in calls]
    ctx.close()
    for (n, count), grads in zip(calls, got):
        alone = N.Context(0)
        want = _loss(alone, n, count, 60)
        alone.close()
        for a, b in zip(grads, want):
            assert np.array_equal(a, b)
