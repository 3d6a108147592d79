"""Solvers of several host threads on the default stream, one handle per thread:
a solve whose pass is captured as a graph (the second and later ones) beside
another thread's setup, data updates, solves and its own work on the default
stream."""
import threading

import numpy as np
import pytest

from cuclarabel_b200 import BatchSolver, Solver, problems

pytestmark = pytest.mark.gpu


def test_captures_beside_other_threads_on_the_default_stream(cuda_device):
    import torch
    pbs = problems.mpc_batch(3, seed0=40)
    one = problems.portfolio(4, 20, 3)
    ref = BatchSolver(pbs).solve()
    ref_one = Solver(*one).solve()
    errors, done = [], threading.Event()

    def guard(f):
        def run():
            try:
                f()
            except BaseException as e:  # noqa: B902 -- reported by the main thread
                errors.append(repr(e))
            finally:
                done.set()
        return run

    def captures():
        for _ in range(25):  # every new solver captures in its second solve
            bs = BatchSolver(pbs)
            for _ in range(3):
                for a, b in zip(bs.solve(), ref):
                    assert a.status == b.status and np.array_equal(a.x, b.x)

    def others():
        x = torch.zeros(1000, device="cuda")
        n = 0
        while not done.is_set():
            for _ in range(20):
                x += 1  # the default stream
            n += 20
            assert float(x[0]) == n
            if n > 100000:
                x.zero_()
                n = 0

    def setups():
        while not done.is_set():
            s = Solver(*one)
            for _ in range(2):
                assert np.array_equal(s.solve().x, ref_one.x)
            s.update_q(one[1])
            assert s.solve().status == ref_one.status

    ths = [threading.Thread(target=guard(f)) for f in (captures, others, setups)]
    for t in ths:
        t.start()
    for t in ths:
        t.join(120)
    assert not errors, errors
    assert not any(t.is_alive() for t in ths)
