"""Tables computed by two threads at once, on handles whose quadratures need different
amounts of shared memory (degree 2: 22 KB, degree 10: 160 KB): the same tables as one
after the other, and no launch that another thread's setting makes fail."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_tables_of_two_degrees_at_once():
    import aifmm_ls_b200 as A
    handles = [A.LSKernel(n_cheb=n, kappa=10.0, degree=d, depth=2, q_kind="gauss_aw") for n, d in ((3, 2), (10, 10))]
    want = []
    for K in handles:
        K.tables_compute(round6=False)
        want.append(K.tables_get())
    failed = []

    def work(K, w):
        try:
            for _ in range(60):
                K.tables_compute(round6=False)
            for a, b in zip(K.tables_get(), w):
                assert np.array_equal(a, b, equal_nan=True)
        except Exception as e:
            failed.append(repr(e))

    # four threads of the small degree: their calls are short, and fall between the other's
    small = [handles[0]] + [A.LSKernel(n_cheb=3, kappa=10.0, degree=2, depth=2, q_kind="gauss_aw") for _ in range(3)]
    ts = [threading.Thread(target=work, args=(K, want[0])) for K in small]
    ts.append(threading.Thread(target=work, args=(handles[1], want[1])))
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not failed, failed
