"""Small instances are solved by one thread-block cluster each instead of a loop of kernels. Both
run the same arithmetic in the same order, so the kernels (launched one by one while per-kernel
profiling is on) give the same iterations, outcomes and meshes bit for bit. Sizes around the
transform lengths' steps and the largest the cluster takes; batches whose instances may stop at
different iterations, of one more instance than fits, and loops that end at once, at a limit
and far beyond convergence."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _both(dens, opt):
    from otmap_b200 import native as N
    from otmap_b200 import otmap as ot

    out = []
    for plain in (0, 1):
        ctx = N.Context(0)
        ctx.profile(plain)
        maps = ot.solve_batch(dens, opt, context=ctx)
        out.append([(m.stats.iterations, m.stats.outcome, m.fwd_mesh()) for m in maps])
        ctx.close()
    for (ia, oa, a), (ib, ob, b) in zip(*out):
        assert ia == ib and oa == ob and np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("n", [8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 100, 127, 129])
def test_equals_the_kernels(n):
    from otmap_b200 import otmap as ot
    from otmap_b200 import workloads as W

    dens = [W.to_cells(W.gaussian_mixture(n, 11 + k)) for k in range(3)]
    _both(dens[:1], ot.SolverOptions())
    _both(dens, ot.SolverOptions(threshold=1e-10, max_iter=60))


@pytest.mark.parametrize("count", [2, 7, 10, 40])
@pytest.mark.parametrize("n", [24, 64])
def test_batches(n, count):
    from otmap_b200 import otmap as ot
    from otmap_b200 import workloads as W

    rng = np.random.default_rng(count)
    dens = [W.to_cells(W.gaussian_mixture(n, k)) + float(rng.uniform(0, 3)) for k in range(count)]
    _both(dens, ot.SolverOptions())


@pytest.mark.parametrize("n", [20, 64])
def test_loop_ends(n):
    from otmap_b200 import otmap as ot
    from otmap_b200 import workloads as W

    mix = W.to_cells(W.gaussian_mixture(n, 5))
    flat = np.ones_like(mix)
    for max_iter, threshold in ((0, 1e-7), (1, 1e-7), (3, 1e-7), (400, 0.0)):
        _both([mix, flat, mix], ot.SolverOptions(max_iter=max_iter, threshold=threshold))


def test_threads_on_sizes_of_one_kernel():
    """Contexts of their own on host threads, sizes that share a kernel with different shared-memory needs."""
    import threading

    from otmap_b200 import native as N
    from otmap_b200 import otmap as ot
    from otmap_b200 import workloads as W

    sizes = [66, 100, 127, 66]
    dens = [W.to_cells(W.gaussian_mixture(n, 40 + n)) for n in sizes]
    want = [ot.solve_batch([d])[0].fwd_mesh() for d in dens]
    wrong = []

    def work(k):
        try:
            for _ in range(15):
                ctx = N.Context(0)  # a new layout each time
                got = ot.solve_batch([dens[k]], context=ctx)[0].fwd_mesh()
                ctx.close()
                if not np.array_equal(got, want[k]):
                    wrong.append(k)
        except Exception as e:  # noqa: BLE001
            wrong.append((k, e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(sizes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
