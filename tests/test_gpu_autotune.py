"""What the set-up autotuner times is the launch that the step makes.  On the dynamo set the implicit
solve has four systems; with N_r = 16 each of them is one 64-row block, so that a candidate timed
without C and A takes half of the step's own solve stage (device times of the same launches otherwise:
three quarters leaves room for the gaps between events).  The state is the same after the search."""
import numpy as np
import pytest

import test_gpu_mhd as M

pytestmark = pytest.mark.gpu


def test_every_system_of_the_solve_is_timed():
    cfg = dict(n_r=16, l_max=255, dt=1e-6, rayleigh=1e5, ekman=1e-3, magnetism=True, magnetic_prandtl=5.0)
    wpt, z, c, a = M._seed(M._ocfg(cfg))
    g = M._ctx(cfg)
    g.put_state(wpt, z, None, iteration=1)
    g.put_magnetic_state(c, a)
    g.step(3)
    before = g.get_state() + g.get_magnetic_state()
    choice, ms = g.autotune(5)["solve_nc"]
    for x, y in zip(before, g.get_state() + g.get_magnetic_state()):
        assert np.array_equal(x, y)
    stage = min(g.time_steps(5)[1]["solve"] / 5 for _ in range(3))
    print(choice, ms, stage)
    assert ms > 0.75 * stage, (choice, ms, stage)
    g.close()
