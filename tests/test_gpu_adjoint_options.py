"""Context options reach every adjoint, whatever the context has computed before: the adjoint of
a context that has changed an option equals, bit for bit, that of a new one with the option set
from the start."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inputs(n):
    from otmap_b200 import otmap as ot
    from otmap_b200 import workloads as W

    xy = ot.grid_vertices(n)
    x, y = xy[:, 0].copy(), xy[:, 1].copy()
    xy[:, 0] += 0.01 * np.sin(2 * np.pi * x) * np.cos(np.pi * y)
    xy[:, 1] += 0.01 * np.sin(2 * np.pi * y) * np.cos(np.pi * x)
    return W.to_cells(W.gaussian_mixture(n, 7)), xy, np.random.default_rng(3).standard_normal(((n + 1) ** 2, 2))


def _adjoint(ctx, n, mode, inputs):
    from otmap_b200 import native as N

    density, fwd, q = inputs
    ctx.init(n)
    g = np.empty(n * n)
    opt = N.AdjointOptionsC()
    N.lib().otm_default_adjoint_options(C.byref(opt))
    opt.mode = mode
    opt.max_iter = 120
    N.check(N.lib().otm_adjoint(ctx.handle, n, N.ptr(density), N.ptr(fwd), N.ptr(q), C.byref(opt), N.ptr(g), None))
    return g


@pytest.mark.parametrize("mode", [0, 1])  # one step, Krylov
@pytest.mark.parametrize("n", [32, 64, 100])
def test_poisson_option(n, mode):
    from otmap_b200 import native as N

    inputs = _inputs(n)
    alone = {}
    for poisson in (N.POISSON_AUTO, N.POISSON_DENSE):
        ctx = N.Context(0)
        ctx.set_poisson(poisson)
        alone[poisson] = _adjoint(ctx, n, mode, inputs)
        ctx.close()
    assert not np.array_equal(alone[N.POISSON_AUTO], alone[N.POISSON_DENSE])  # they round differently
    ctx = N.Context(0)
    for poisson in (N.POISSON_AUTO, N.POISSON_DENSE, N.POISSON_AUTO):
        ctx.set_poisson(poisson)
        assert np.array_equal(_adjoint(ctx, n, mode, inputs), alone[poisson])
    ctx.close()


@pytest.mark.parametrize("n", [64, 128])
def test_wait_test_option(n):
    """Adjoints first computed while the bounded waits are made to run out (an error, and the
    steps' launches captured with it) are right once the option is off; and the option takes
    effect after launches captured without it."""
    from otmap_b200 import native as N

    inputs = _inputs(n)
    clean = N.Context(0)
    good = _adjoint(clean, n, N.ADJOINT_KRYLOV, inputs)
    clean.close()
    ctx = N.Context(0)
    for _ in range(2):
        N.check(N.lib().otm_set_option(ctx.handle, N.OPT_WAIT_TEST, 1))
        with pytest.raises(N.OtmError) as e:
            _adjoint(ctx, n, N.ADJOINT_KRYLOV, inputs)
        assert e.value.code == N.ERR_TIMEOUT
        N.check(N.lib().otm_set_option(ctx.handle, N.OPT_WAIT_TEST, 0))
        assert np.array_equal(_adjoint(ctx, n, N.ADJOINT_KRYLOV, inputs), good)
    ctx.close()
