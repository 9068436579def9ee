"""A batch of many sizes without a register transform: the sizes of one transform length share
their launches, whose number does not grow with that of the sizes, and an instance's map
depends neither on its place in the batch nor on the others beside it."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (sizes, families among them): powers of two without a register transform are one each, others
# share the chirp length from 2n - 1 on (9..15: 32, 17..31: 64, 33..63: 128, ...)
SIZES = {"one length": (list(range(40, 64)), 1), "lengths' ends": ([33, 63, 65, 127, 17, 31, 9, 15], 4),
         "with others": ([50, 64, 8, 51, 32, 33, 128, 7, 16, 200, 62, 50], 5)}


def _solve(sizes, opt):
    from otmap_b200 import native as N
    from otmap_b200 import otmap as ot
    from otmap_b200 import workloads as W

    ctx = N.Context(0)
    maps = ot.solve_batch([W.to_cells(W.gaussian_mixture(n, n)) for n in sizes], opt, context=ctx)
    out = {n: (m.stats.iterations, m.stats.outcome, m.fwd_mesh()) for n, m in zip(sizes, maps)}
    ctx.close()
    return out


@pytest.mark.parametrize("name", SIZES)
def test_sizes_of_one_length_share_launches(name):
    from otmap_b200 import native as N
    from otmap_b200 import otmap as ot
    from otmap_b200 import workloads as W

    sizes, families = SIZES[name]
    ctx = N.Context(0)
    ctx.profile(1)
    ot.solve_batch([W.to_cells(W.gaussian_mixture(n, n)) for n in sizes], ot.SolverOptions(max_iter=4, threshold=0.0),
                   context=ctx)
    totals = ctx.profile_totals()
    ctx.close()
    for kernel in ("fft_rows_fwd", "fft_cols", "fft_rows_inv"):
        assert totals[kernel][1] == 4 * families


@pytest.mark.parametrize("name", SIZES)
def test_place_in_the_batch(oracle_port, name):
    from otmap_b200 import otmap as ot
    from otmap_b200 import workloads as W

    sizes, _ = SIZES[name]
    opt = ot.SolverOptions()
    there, back = _solve(sizes, opt), _solve(sizes[::-1], opt)
    for n in set(sizes):
        assert there[n][:2] == back[n][:2] and np.array_equal(there[n][2], back[n][2])
        want = oracle_port.solve(W.to_cells(W.gaussian_mixture(n, n)), n)
        assert there[n][0] == want.iterations
        # both end within the threshold of one iteration's arithmetic: FP64 rounding through a solve
        assert np.abs(there[n][2].ravel() - want.fwd.ravel()).max() <= 1e-9
