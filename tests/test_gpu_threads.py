"""Two contexts on two host threads, as the C header allows (one thread per
context): eigensolver batches whose kernels need different amounts of shared
memory, launched side by side many times.  Every call succeeds and gives the
bits of the same call made alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_eigensolver_of_two_contexts():
    import block_gb300

    rng = np.random.default_rng(4)

    def batch(orders):
        out = []
        for n in orders:
            X = rng.standard_normal((n, n))
            out.append(0.5 * (X + X.T))
        return out

    # the second thread's limits lie below the first's needs in every kernel
    batches = [batch([460]), batch([35])]
    ctxs = [block_gb300.Context(0) for _ in batches]
    alone = [c.diagonalise(b) for c, b in zip(ctxs, batches)]
    start = threading.Barrier(2)
    done = threading.Event()
    errors = []

    def work(i):
        start.wait()
        try:
            for _ in range(250 if i == 0 else 20000):
                if i == 1 and done.is_set():
                    break
                for (w, V), (w0, V0) in zip(ctxs[i].diagonalise(batches[i]), alone[i]):
                    assert np.array_equal(w, w0) and np.array_equal(V, V0)
        except BaseException as e:  # reported by the main thread
            errors.append(e)
        finally:
            done.set()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for c in ctxs:
        c.close()
    assert not errors, errors
