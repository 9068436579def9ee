"""Copies between pageable host memory and the device: below and above the size from which they
go through the context's pinned ring, whole and partial chunks, one and several turns of the
ring, unaligned starts. A blend with weights (1, 0) returns its first mesh bit for bit (finite
entries: x + 0 y = x)."""

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _roundtrip(ctx, n, offset):
    from otmap_b200 import otmap as ot

    rng = np.random.default_rng(n)
    count = 2 * (n + 1) ** 2
    raw = np.empty(count * 8 + 64, dtype=np.uint8)
    a = raw[offset:offset + count * 8].view(np.float64).reshape(-1, 2)
    a[:] = rng.uniform(0.5, 1.0, a.shape)
    b = rng.uniform(0.5, 1.0, a.shape)
    assert np.array_equal(ot.interpolate([a, b], 0.0, context=ctx), a)


@pytest.mark.parametrize("offset", [0, 8])
@pytest.mark.parametrize("n", [1, 300, 722, 723, 724, 1000, 1447, 2000])
def test_copies_round_trip(n, offset):
    from otmap_b200 import native as N

    ctx = N.Context(0)
    _roundtrip(ctx, n, offset)
    _roundtrip(ctx, n, offset)
    ctx.close()


def test_contexts_copy_from_their_own_threads():
    from otmap_b200 import native as N

    errors = []

    def work(k):
        try:
            ctx = N.Context(0)
            for n in (300 + k, 900 + k, 730 + k):
                _roundtrip(ctx, n, 0)
            ctx.close()
        except BaseException as e:  # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
