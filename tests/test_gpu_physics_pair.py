"""The physical-space kernel on (theta, pi - theta) row pairs at every transform length it is
built for: each plan of the phi transform (n_phi = 48 .. 1536), with l_max = 2 n_theta / 3 - 1
and the largest accepted one, (2 n_theta) / 3, whose last wavenumber is the one that the
pruned first pass treats apart; n_r = 10 leaves a remainder for the CTAs of several radii.
Every stage of an AB2 step against the oracle (relative L2 per buffer).  The bound is 1e-12,
as for the other stage tests: a transform of length n rounds to about 2^-53 log2(n), and the
nonlinear terms carry that through differences of up to ~1e2 in size."""
import pytest

import test_gpu_mhd as M
import test_gpu_parity as H
from test_gpu_anelastic import ANEL, ANEL_MHD

pytestmark = pytest.mark.gpu
TOL = 1e-12


def _check(errs):
    print({k: f"{v:.2e}" for k, v in errs.items()})
    bad = {k: v for k, v in errs.items() if v > TOL}
    assert not bad, errs


@pytest.mark.parametrize("top", [0, 1])
@pytest.mark.parametrize("n_theta", [24, 32, 48, 64, 96, 128, 192, 256])
def test_hydro_stages(n_theta, top):
    l_max = (2 * n_theta) // 3 - 1 + top
    _check(H._stage_compare(dict(n_r=10, l_max=l_max, n_theta=n_theta, dt=1e-5, rayleigh=1e5, ekman=1e-3),
                            steps_before=1))


@pytest.mark.parametrize("n_theta,n_r", [(24, 10), (32, 10), (48, 10), (64, 10), (96, 10), (128, 8), (192, 8), (256, 8),
                                         (384, 8), (512, 8), (768, 8)])
def test_magnetic_stages(n_theta, n_r):
    _check(M._stage_compare(dict(n_r=n_r, l_max=(2 * n_theta) // 3 - 1, n_theta=n_theta, dt=1e-6, rayleigh=1e5,
                                 ekman=1e-3, magnetism=True, magnetic_prandtl=5.0), steps_before=1))


def test_hydro_stages_512():
    _check(H._stage_compare(dict(n_r=8, l_max=341, n_theta=512, dt=1e-6, rayleigh=1e5, ekman=1e-3), steps_before=1))


@pytest.mark.parametrize("n_theta,n_r", [(32, 10), (48, 10), (192, 16), (256, 16), (512, 8), (768, 8)])
@pytest.mark.parametrize("mag", [False, True])
def test_heating_stages(n_theta, n_r, mag):
    compare = M._stage_compare if mag else H._stage_compare
    _check(compare(dict(ANEL_MHD if mag else ANEL, n_r=n_r, l_max=(2 * n_theta) // 3 - 1, n_theta=n_theta),
                   steps_before=2 if n_theta < 512 else 1))
