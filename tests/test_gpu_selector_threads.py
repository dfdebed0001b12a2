"""Selector.infer keeps its device buffers between calls: threads that share a
selector get their own rows' results, and a large call's buffers are given
back."""

import threading

import numpy as np
import pytest

from mallard_gb300.selector import IN, Selector, default_weights_path

pytestmark = pytest.mark.gpu


def rows(n, seed):
    return np.random.default_rng(seed).uniform(-1, 1, (n, IN)).astype(np.float32)


def test_threads_share_a_selector():
    with Selector() as s:
        s.load(default_weights_path())
        # small and large in turn, so that the buffers grow under other calls
        X = [rows(n, i) for i, n in enumerate((40, 3000, 129, 20000, 1000, 50000))]
        alone = [s.infer(x) for x in X]
        with Selector() as fresh:
            fresh.load(default_weights_path())
            wrong, start = [], threading.Barrier(len(X))

            def work(i):
                start.wait()
                for _ in range(20):
                    L, P = fresh.infer(X[i])
                    if not (np.array_equal(L, alone[i][0]) and np.array_equal(P, alone[i][1])):
                        wrong.append(i)

            threads = [threading.Thread(target=work, args=(i,)) for i in range(len(X))]
            for t in threads:
                t.start()
            for t in threads:
                t.join()
    assert wrong == []


def test_large_call_gives_its_buffers_back():
    import torch
    with Selector() as s:
        s.load(default_weights_path())
        X = rows(600000, 3)
        a = s.infer(X[:100000])
        free = torch.cuda.mem_get_info()[0]
        L, P = s.infer(X)  # 310 MB of buffers
        assert torch.cuda.mem_get_info()[0] >= free - (64 << 20)
        np.testing.assert_array_equal(L[:100000], a[0])
        np.testing.assert_array_equal(P[:100000], a[1])
        b = s.infer(X[:100000])
        np.testing.assert_array_equal(b[0], a[0])
