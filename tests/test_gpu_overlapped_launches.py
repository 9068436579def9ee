"""Kernels whose launches overlap their predecessor's end (the solver's iteration and the
adjoint's step, unless a product kernel is among them) against the same kernels launched plainly,
as they are while per-kernel profiling is on: a read or write before the wait for the predecessor
would show as another value. The arithmetic is the same, so the results are equal bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# block and register transforms, FP64 and split, alone and in batches of several kernels per
# stage; size 5 brings the product kernels, beside which nothing overlaps
@pytest.mark.parametrize("sizes", [(32,), (64,), (100,), (256,), (513,), (1024,), (64, 100, 256, 512), (5, 64, 100),
                                   (512,) * 4, (1024,) * 3])
@pytest.mark.parametrize("precision", ["fp64", "split"])
def test_solve_equals_plain_launches(sizes, precision):
    from otmap_b200 import native as N
    from otmap_b200 import otmap as ot
    from otmap_b200 import workloads as W

    dens = [W.to_cells(W.gaussian_mixture(n, 7 + k)) for k, n in enumerate(sizes)]
    out = []
    for plain in (0, 1):
        ctx = N.Context(0)
        ctx.set_precision(N.PRECISION_SPLIT if precision == "split" else N.PRECISION_FP64)
        ctx.profile(plain)
        for _ in range(1 if plain else 3):
            out.append([(m.stats.iterations, m.fwd_mesh()) for m in ot.solve_batch(dens, context=ctx)])
        ctx.close()
    for other in out[1:]:
        for (ia, a), (ib, b) in zip(out[0], other):
            assert ia == ib and np.array_equal(a, b)


@pytest.mark.parametrize("n", [5, 64, 100, 256])
def test_gradient_equals_plain_launches(n):
    import torch

    from otmap_b200 import autograd as A
    from otmap_b200 import native as N
    from otmap_b200 import workloads as W

    dens = torch.tensor(W.to_cells(W.gaussian_mixture(n, 3)), device="cuda:0").flatten()
    out = []
    for plain in (0, 1, 0):
        ctx = N.Context(0)
        ctx.profile(plain)
        x = dens.clone().requires_grad_(True)
        y = A.transport_map(x, n, context=ctx)
        torch.sin(3.0 * y).sum().backward()
        out.append(x.grad.cpu().numpy())
        ctx.close()
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
