"""LU fallbacks of different sizes from several host threads at once: every call
has a context and a stream of its own, but what a kernel may have of an SM's
shared memory is set per function, for all of them. Each result is the one that
the same call gives alone, bit for bit."""
import threading

import numpy as np
import pytest

from sfmtory_gb300 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batched", [False, True], ids=["dense", "batch"])
def test_sizes_from_several_threads(batched):
    rng = np.random.default_rng(0)
    systems, alone, failed = [], [], []
    for n in (1500, 6, 700, 40):
        A, b = rng.standard_normal((n, n)), rng.standard_normal(n)
        systems.append(([A, A], [b, b]) if batched else ([A], [b]))
        alone.append(native.dense_lu(*systems[-1], batched=batched))
    start = threading.Barrier(len(systems))

    def work(k):
        try:
            start.wait()
            for _ in range(6 if k % 2 == 0 else 150):
                for x, y in zip(native.dense_lu(*systems[k], batched=batched), alone[k]):
                    assert np.array_equal(x, y)
        except BaseException as e:
            failed.append((k, e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(systems))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
