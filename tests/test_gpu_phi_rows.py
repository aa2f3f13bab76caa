"""The device-resident transforms' row-pair kernels (unfold + c2r and r2c + fold in one pass) against
the separate operators on the same numbers: StP / PtS and the packed phi FFT of single rows
(ra_legendre_*, ra_fft_*), at every transform length they are built for and with column counts
around their groups of four.  Both sides round to about 2^-53 log2(n_phi) per transform and carry
the same Legendre products: 1e-13 of the largest value."""
import numpy as np
import pytest

from layouts import row_index

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("top", [0, 1])
@pytest.mark.parametrize("n_theta,cols", [(24, 1), (24, 70), (32, 33), (48, 5), (64, 4), (96, 37), (128, 6), (192, 3),
                                          (256, 9), (384, 7), (512, 5), (768, 6)])
def test_rows_match_the_separate_operators(n_theta, cols, top):
    import torch
    import rayleigh_b200 as rb
    from rayleigh_b200 import build as rbuild
    rbuild.build()
    if top and n_theta > 256:
        pytest.skip("the last wavenumber's case is covered by the smaller plans")
    L = (2 * n_theta) // 3 + top
    n_phi = 2 * n_theta
    rng = np.random.default_rng(n_theta + cols)
    dev = torch.device("cuda")
    with rb.Rayleigh(rb.Config(n_r=8, n_theta=n_theta, l_max=L - 1, use_graph=False)) as g:
        s2 = []
        for m in range(L):
            a = rng.standard_normal((1, 2, cols, L - m))
            if m == 0:
                a[:, 1] = 0.0
            s2.append(a)
        spec = np.zeros((L * (L + 1) // 2, cols, 2))
        for m in range(L):
            for l in range(m, L):
                spec[row_index(m, l, L)] = s2[m][0, :, :, l - m].T
        d_spec = torch.tensor(spec, device=dev)
        back = torch.full_like(d_spec, float("nan"))
        grid = torch.full((n_theta, cols, n_phi + 2), float("nan"), dtype=torch.float64, device=dev)
        work = torch.empty((L * n_theta * cols * 2,), dtype=torch.float64, device=dev)
        g.transform_dev(0, rb.PREC_FP64, d_spec.data_ptr(), grid.data_ptr(), work.data_ptr(), cols)
        p2 = g.legendre_s2p(s2)                                    # [m](1, 2, cols, n_theta)
        x = np.zeros((n_theta, cols, n_phi + 2))
        for m in range(L):
            x[:, :, 2 * m:2 * m + 2] = p2[m][0].transpose(2, 1, 0)
        ref = g.fft_c2r(x)
        got = grid.cpu().numpy()
        assert np.abs(got[..., :n_phi] - ref[..., :n_phi]).max() <= 1e-13 * np.abs(ref).max()
        assert not got[..., n_phi:].any()
        # back, from unrelated rows
        rows = rng.standard_normal((n_theta, cols, n_phi + 2))
        grid.copy_(torch.tensor(rows))
        g.transform_dev(1, rb.PREC_FP64, back.data_ptr(), grid.data_ptr(), work.data_ptr(), cols)
        X = g.fft_r2c(rows)
        assert np.abs(grid.cpu().numpy() - X).max() <= 1e-13 * np.abs(X).max()
        p2 = [np.ascontiguousarray(X[:, :, 2 * m:2 * m + 2].transpose(2, 1, 0))[None] for m in range(L)]
        s2 = g.legendre_p2s(p2)
        want = np.zeros_like(spec)
        for m in range(L):
            for l in range(m, L):
                want[row_index(m, l, L)] = s2[m][0, :, :, l - m].T
        assert np.abs(back.cpu().numpy() - want).max() <= 1e-13 * np.abs(want).max()
