"""Autotuning where the strip rule goes below 16 rows or one kernel runs the whole loop: the
rule's own heights are among the timed ones, and a one-kernel loop keeps the rule's height."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

K = 4  # iterations of a timed run: 4 set-up kernels and 5 per iteration, two runs per height


# the rule's height; heights that the first call times
@pytest.mark.parametrize("sizes,rule,tried", [([256], 4, 5), ([512], 16, 3), ([256, 128], 4, 5), ([64], None, 0),
                                              ([100], None, 0), ([50] * 4, None, 0), ([1024], 32, 3)])
def test_heights_tried(sizes, rule, tried):
    from otmap_b200 import native as N
    from otmap_b200 import otmap as ot
    from otmap_b200 import workloads as W

    dens = [W.to_cells(W.gaussian_mixture(n, 3 + k)) for k, n in enumerate(sizes)]
    plain = N.Context(0)
    ref = ot.solve_batch(dens, context=plain)
    if rule is not None:
        assert plain.strip_rows() == rule
    tuned = N.Context(0)
    tuned.set_autotune(True)
    counts, out = [], []
    for _ in range(2):
        before = tuned.launch_count()
        out.append(ot.solve_batch(dens, context=tuned))
        counts.append(tuned.launch_count() - before)
    transforms = sum(3 for _ in set(sizes))
    assert counts[0] - counts[1] == 2 * tried * (4 + K * (transforms + 2))
    if tried == 0:
        assert tuned.strip_rows() == plain.strip_rows()
        for a, b in zip(ref, out[0]):
            assert np.array_equal(a.fwd_mesh(), b.fwd_mesh())
    for a, b in zip(*out):
        assert np.array_equal(a.fwd_mesh(), b.fwd_mesh())
    plain.close()
    tuned.close()
