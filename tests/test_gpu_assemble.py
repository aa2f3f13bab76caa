"""The implicit matrices formed on the device against the host's (ra_build_matrices) bit for bit: a
context that assembled its own matrices and one that was given the host's through ra_load_matrices +
ra_factor step to identical states, at creation and after a change of dt."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BASE = dict(n_r=26, l_max=15, dt=1e-4, rayleigh=1e5, ekman=1e-3)
ANEL = dict(BASE, reference_type=3, poly_n=2.0, poly_nrho=5.0, modified_rayleigh=0.5, magnetic_prandtl=2.0,
            nu_type=2, nu_power=-0.5, kappa_type=2, kappa_power=-0.5)


@pytest.mark.parametrize("cfg", [
    BASE,
    dict(BASE, no_slip_top=False, no_slip_bottom=False, fix_tvar_top=False, dtdr_top=-1.0),
    dict(BASE, fix_tvar_bottom=False, dtdr_bottom=-1.0, no_slip_bottom=False),
    dict(BASE, chebyshev=False),
    dict(BASE, magnetism=True, magnetic_prandtl=5.0),
    dict(ANEL, magnetism=True, eta_type=2, eta_power=-0.5, no_slip_top=False),
])
def test_device_matrices_are_the_hosts(cfg):
    import dataclasses
    import rayleigh_b200 as rb
    from rayleigh_b200 import build as rbuild
    rbuild.build()
    mag = bool(cfg.get("magnetism"))
    rng = np.random.default_rng(7)
    states = []
    for loaded in (False, True):
        c = rb.Config(**cfg)
        with rb.Rayleigh(c) as g:
            if not states:
                wpt = rng.standard_normal((g.n_lm, 2, 3 * g.n_r)) * 1e-3
                z = rng.standard_normal((g.n_lm, 2, g.n_r)) * 1e-3
                b = rng.standard_normal((2, g.n_lm, 2, g.n_r)) * 1e-3
            out = []
            for k, dt in enumerate((c.dt, 0.7 * c.dt)):
                if loaded:
                    at = dataclasses.replace(c, dt=dt)
                    for sys in range(4 if mag else 2):
                        lhs, coefs = rb.build_matrices(at, sys, 0, c.l_max + 1, coefs=True)
                        g.load_matrices(sys, lhs, coefs)
                    g.factor(dt)
                elif k:
                    g.set_dt(dt)
                g.put_state(wpt, z, None, iteration=1)
                if mag:
                    g.put_magnetic_state(b[0], b[1])
                g.step(3)
                out += list(g.get_state()) + (list(g.get_magnetic_state()) if mag else [])
            states.append(out)
    for x, y in zip(*states):
        assert np.isfinite(x).all() and np.array_equal(x, y)
