"""Contexts and solvers of different sizes driven from two host threads at once.  Kernels whose
shared memory grows with the problem share one limit per function: a thread must be able to launch
whatever another one has just launched.  Each thread's results are those of its run alone, bit for bit."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _together(jobs):
    out, errors = [None] * len(jobs), []
    gate = threading.Barrier(len(jobs))

    def run(i):
        try:
            gate.wait()
            out[i] = jobs[i]()
        except Exception as e:   # raised in the main thread below
            errors.append(e)
    threads = [threading.Thread(target=run, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]
    return out


def test_steps_of_two_radial_sizes():
    import oracle as O
    import rayleigh_b200 as rb
    from rayleigh_b200 import build as rbuild
    rbuild.build()
    contexts, states = [], []
    for n_r in (16, 128):
        cfg = dict(n_r=n_r, l_max=15, dt=1e-6, rayleigh=1e5, ekman=1e-3)
        oc = O.Config(**cfg)
        states.append(O.seeded_state(oc, amp=1e-3, lmax_pert=10))
        contexts.append(rb.Rayleigh(rb.Config(**cfg, use_graph=False)))

    def steps(i):
        contexts[i].put_state(*states[i], None, iteration=1)
        contexts[i].step(1500)
        return contexts[i].get_state()
    alone = [steps(i) for i in (0, 1)]
    for got, want in zip(_together([lambda: steps(0), lambda: steps(1)]), alone):
        for x, y in zip(got, want):
            assert np.array_equal(x, y)
    for g in contexts:
        g.close()


def test_solvers_of_two_orders():
    import rayleigh_b200 as rb
    rng = np.random.Generator(np.random.PCG64(5))
    solvers, mats, b = [], [], []
    for n in (64, 384):
        a = rng.standard_normal((4, n, n)) / np.sqrt(n) + 2.0 * np.eye(n)
        mats.append(a)
        b.append(rng.standard_normal((4, 16, n)))
        solvers.append(rb.BatchedLU(n, 4))

    def solve(i):
        for _ in range(200):
            solvers[i].factor(mats[i])
            x = [solvers[i].solve(b[i], mode)[0] for mode in (rb.SOLVE_FP64, rb.SOLVE_REFINE)]
        return x
    alone = [solve(i) for i in (0, 1)]
    for got, want in zip(_together([lambda: solve(0), lambda: solve(1)]), alone):
        for x, y in zip(got, want):
            assert np.array_equal(x, y)
    for lu in solvers:
        lu.close()


def test_row_ffts_of_two_lengths():
    import rayleigh_b200 as rb
    contexts = [rb.Rayleigh(rb.Config(n_r=8, n_theta=n, l_max=15, use_graph=False)) for n in (48, 1536)]
    rows = [np.random.Generator(np.random.PCG64(n)).standard_normal((8, 2 * n + 2)) for n in (48, 1536)]

    def transform(i):
        for _ in range(1500):
            x = contexts[i].fft_r2c(rows[i])
        return x
    alone = [transform(i) for i in (0, 1)]
    for got, want in zip(_together([lambda: transform(0), lambda: transform(1)]), alone):
        assert np.array_equal(got, want)
    for g in contexts:
        g.close()
