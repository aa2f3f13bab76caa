"""What the performance of this framework is measured on: whole calls as a user's program makes them.

Five kinds of case, over the sizes that the tests, the benchmark and the published set-ups use
(n_theta from 24 to 768, l_max = 2 n_theta / 3 - 1, n_r from 24 to 192):

  step       a running simulation: n time steps, then the state read back into pinned host memory
             (ra_step + ra_get_state, ra_get_magnetic_state), in the FP64 and the mixed form
  change_dt  the same with two changes of the time step on the way (ra_set_dt: the implicit matrices
             are rebuilt and factored)
  output     an output iteration: a step, then slices, averages and spectra of the new state
  transform  a batch of fields resident on the device, spectral -> physical ("inverse"), or there, a
             pointwise product and back ("product"): the pseudo-spectral pattern
  solve      a batch of per-l implicit systems solved for host right-hand sides (BatchedLU)

All inputs are synthetic and made from the seed.
"""
import ctypes
import math

import numpy as np
import torch

import rayleigh_b200 as rb

# n_theta of the phi grids that the physical-space stage supports
N_THETA = (24, 32, 48, 64, 96, 128, 192, 256, 384, 512, 768)
PREC = {"fp64": rb.PREC_FP64, "mixed": rb.PREC_MIXED}


def listed():
    step = dict(kind="step", fd=False)
    return [
        # the hydrodynamic accuracy benchmark's grid (Christensen et al. 2001, case 0): the smallest calls,
        # a power-of-two phi grid and the odd l_max = 41
        dict(step, name="step_hydro_41", set="hydro", n_theta=64, n_r=48, precision="fp64", steps=50),
        # the same benchmark in the finite-difference radial mode
        dict(step, name="step_fd_41", set="hydro", n_theta=64, n_r=48, precision="mixed", steps=50, fd=True),
        # the dynamo accuracy benchmark's grid (case 1), which runs for 150 000 steps
        dict(step, name="step_dynamo_63", set="dynamo", n_theta=96, n_r=64, precision="fp64", steps=50),
        # the anelastic hydrodynamic benchmark (Jones et al. 2011): cgs polytrope, viscous heating
        dict(step, name="step_jones_127", set="jones", n_theta=192, n_r=128, precision="fp64", steps=10),
        # the anelastic MHD workload at its own size
        dict(step, name="step_anelastic_255", set="anelastic", n_theta=384, n_r=128, precision="mixed", steps=10),
        # the large Boussinesq dynamo's horizontal grid in both forms, on 96 of its 192 levels
        dict(step, name="step_dynamo_511", set="dynamo", n_theta=768, n_r=96, precision="fp64", steps=10),
        dict(step, name="step_dynamo_511_mixed", set="dynamo", n_theta=768, n_r=96, precision="mixed", steps=10),
        # a CFL-limited run whose dt has just moved down and up again
        dict(kind="change_dt", name="change_dt_85", set="dynamo", n_theta=128, n_r=64, precision="mixed", steps=5),
        # an output iteration of a medium dynamo
        dict(kind="output", name="output_127", set="dynamo", n_theta=192, n_r=64, precision="fp64"),
        # the transform sweep: 16 fields x 32 levels at l_max 255, and an odd count of columns at 511
        dict(kind="transform", name="inverse_255", way="inverse", n_theta=384, columns=512, precision="fp64"),
        dict(kind="transform", name="product_511", way="product", n_theta=768, columns=237, precision="mixed"),
        # W-P-T systems of a 64-level shell, 8 complex right-hand sides each
        dict(kind="solve", name="solve_192", n_r=64, count=256, columns=16, mode="fp64"),
    ]


def draw(rng):
    """One more case of the same ranges; none costs more than the largest listed one."""
    kind = rng.choice(["step", "step", "step", "step", "transform", "transform", "change_dt", "output", "solve"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "solve":
        # count x n^2 stays below 512 x 384^2
        n_r = 2 * int(round(math.exp(rng.uniform(math.log(12), math.log(64)))))
        count = int(round(math.exp(rng.uniform(math.log(16), math.log(256)))))
        return dict(kind=kind, n_r=n_r, count=count, columns=rng.choice([1, 2, 7, 16, 33, 64]),
                    mode=rng.choice(["fp64", "refine"]))
    if kind == "transform":
        n_theta = rng.choice(N_THETA[3:])
        most = min(2048, 512 * 384 * 384 // n_theta ** 2)
        columns = int(round(math.exp(rng.uniform(math.log(16), math.log(most)))))
        return dict(kind=kind, way=rng.choice(["inverse", "product"]), n_theta=n_theta, columns=columns,
                    precision=precision)
    top = {"step": 768, "change_dt": 192, "output": 256}[kind]
    n_theta = rng.choice([n for n in N_THETA if n <= top])
    most = max(32, min(192, 64 * (768 * 768) // (n_theta * n_theta)))
    n_r = 2 * int(round(math.exp(rng.uniform(math.log(12), math.log(most / 2)))))
    which = rng.choice(["hydro", "dynamo", "anelastic"])
    case = dict(kind=kind, set=which, n_theta=n_theta, n_r=n_r, precision=precision)
    if kind == "step":
        case["fd"] = which == "hydro" and rng.random() < 0.25
        case["steps"] = 40 if n_theta <= 96 else 10
    elif kind == "change_dt":
        case["steps"] = 5
    return case


# ---- set-ups ----------------------------------------------------------------------------------------

def config(case, dt=None):
    which, n_theta = case["set"], case["n_theta"]
    c = dict(n_r=case["n_r"], n_theta=n_theta, l_max=2 * n_theta // 3 - 1, aspect_ratio=0.35,
             precision=PREC[case["precision"]], use_graph=True, chebyshev=not case.get("fd", False))
    if which == "jones":
        c.update(shell_depth=4.55e9, reference_type=2, poly_n=2.0, poly_nrho=5.0, poly_mass=1.9e30, poly_rho_i=1.1,
                 pressure_specific_heat=1.0509e8, angular_velocity=1.76e-4, nu_top=3.64364e12,
                 kappa_top=3.64364e12, no_slip_top=False, no_slip_bottom=False, t_bottom=851225.7, dt=30.0,
                 alpha_implicit=0.50001)
    elif which == "anelastic":
        c.update(reference_type=3, poly_n=2.0, poly_nrho=5.0, modified_rayleigh=0.5, ekman=1.0e-3, prandtl=1.0,
                 magnetic_prandtl=2.0, magnetism=True, no_slip_top=False, no_slip_bottom=False, dt=1.0e-4)
    elif n_theta >= 512:    # the large rotating cases
        c.update(rayleigh=2.0e8, ekman=1.0e-5, magnetic_prandtl=1.0, magnetism=which == "dynamo", dt=1.0e-6)
    else:                   # the accuracy benchmarks' parameters; dt falls with the grid
        c.update(rayleigh=1.0e5, ekman=1.0e-3, magnetic_prandtl=5.0, magnetism=which == "dynamo",
                 dt=1.0e-4 if n_theta <= 96 else 2.0e-5)
    if dt is not None:
        c["dt"] = dt
    return rb.Config(**c)


def host(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True)


def seeded(case, g, seed):
    """A conductive T (or entropy) profile with perturbations on every l >= 1 that fall as (l + 1)^-2,
    and with magnetism B likewise; the velocity starts from rest, as in a run's own random start."""
    n_lm, n_r = g.n_lm, g.n_r
    gen = torch.Generator(device="cuda").manual_seed(seed)
    l = torch.repeat_interleave(torch.arange(g.l_max + 1), torch.arange(1, g.l_max + 2)).cuda()
    fall = torch.where(l > 0, (l + 1.0) ** -2, 0.0 * l).double()[:, None, None]
    m0 = torch.arange(g.l_max + 1) * torch.arange(1, g.l_max + 2) // 2
    r = g.radius()
    big = g.cfg.t_bottom

    def noise(amp):
        k = min(16, n_r // 2)
        a = torch.randn((n_lm, 2, k), generator=gen, dtype=torch.float64, device="cuda")
        a *= fall * (amp / (1.0 + torch.arange(k, device="cuda")) ** 2)
        a[m0.cuda(), 1] = 0.0
        if g.cfg.chebyshev:
            return torch.nn.functional.pad(a, (0, n_r - k))
        x = torch.as_tensor((r - r[-1]) / (r[0] - r[-1])).cuda()   # grid values that vanish at the boundaries
        return a @ torch.sin(math.pi * torch.arange(1, k + 1, device="cuda")[:, None] * x[None])

    cond = big * r[0] * r[-1] / (r[-1] - r[0]) * (1.0 / r[0] - 1.0 / r) * math.sqrt(4 * math.pi)
    t = noise(1e-3 * big)
    t[0, 0] += torch.as_tensor(g.cheby_to_spectral(cond[None])[0] if g.cfg.chebyshev else cond).cuda()
    wpt = host((n_lm, 2, 3 * n_r)).zero_()
    wpt[:, :, 2 * n_r:] = t.cpu()
    z = host((n_lm, 2, n_r)).zero_()
    mag = None
    if g.cfg.magnetism:
        mag = host((n_lm, 2, n_r)), host((n_lm, 2, n_r))
        for b in mag:
            b.copy_(noise(1e-3))
    torch.cuda.synchronize()
    return wpt, z, mag


def check(g, rc):
    if rc != rb.RA_OK:
        raise RuntimeError("call refused: %d" % rc)


def address(t):
    return ctypes.c_void_p(t.data_ptr())


def simulation(case, seed):
    g = rb.Rayleigh(config(case))
    wpt, z, mag = seeded(case, g, seed)
    check(g, g.lib.ra_put_state(g.h, address(wpt), address(z), None, 1))
    s = dict(case=case, g=g, wpt=wpt, z=z, ab=host((4, g.n_lm, 2, g.n_r)))
    if mag:
        check(g, g.lib.ra_put_magnetic_state(g.h, address(mag[0]), address(mag[1]), None))
        s.update(c=mag[0], a=mag[1], ab_mag=host((2, g.n_lm, 2, g.n_r)))
    return s


def read_state(s):
    """The whole state in the program's own pinned buffers, one output a field."""
    g = s["g"]
    check(g, g.lib.ra_get_state(g.h, address(s["wpt"]), address(s["z"]), address(s["ab"])))
    n = g.n_r
    out = dict(w=s["wpt"][:, :, :n], p=s["wpt"][:, :, n:2 * n], t=s["wpt"][:, :, 2 * n:], z=s["z"], ab=s["ab"])
    if "c" in s:
        check(g, g.lib.ra_get_magnetic_state(g.h, address(s["c"]), address(s["a"]), address(s["ab_mag"])))
        out.update(c=s["c"], a=s["a"], ab_mag=s["ab_mag"])
    return out


def row_degrees(L):
    """l and m of the rows of the device's spectral buffers (m-major, even l - m first)."""
    ls, ms = [], []
    for m in range(L):
        l = np.concatenate([np.arange(m, L, 2), np.arange(m + 1, L, 2)])
        ls.append(l)
        ms.append(np.full(l.size, m))
    return np.concatenate(ls), np.concatenate(ms)


def columns_of(case, seed):
    """Coefficients of a batch of complex columns, amplitude (l + 1)^-1.5."""
    l, m = (torch.as_tensor(a).cuda() for a in row_degrees(2 * case["n_theta"] // 3))
    gen = torch.Generator(device="cuda").manual_seed(seed)
    spec = torch.randn((l.numel(), case["columns"], 2), generator=gen, dtype=torch.float64, device="cuda")
    spec *= ((l + 1.0) ** -1.5).double()[:, None, None]
    spec[m == 0, :, 1] = 0.0
    return spec


def systems_of(case, seed):
    l_max = 4 * -(-case["count"] // 4) - 1       # n_theta = 3 (l_max + 1) / 2 is even
    cfg = rb.Config(n_r=case["n_r"], l_max=l_max, dt=1e-5, ekman=1e-4, rayleigh=1e5)
    mats = rb.build_matrices(cfg, 0, 0, case["count"])
    b = np.random.default_rng(seed).standard_normal((case["count"], case["columns"], 3 * case["n_r"]))
    return mats, b


# ---- the measured calls -----------------------------------------------------------------------------

def prepare(case, seed):
    if case["kind"] == "transform":
        n_theta = case["n_theta"]
        L, cols, n_phi = 2 * n_theta // 3, case["columns"], 2 * n_theta
        g = rb.Rayleigh(rb.Config(n_r=8, n_theta=n_theta, l_max=L - 1, use_graph=False))
        spec = columns_of(case, seed)
        return dict(case=case, g=g, spec=spec, back=torch.empty_like(spec),
                    grid=torch.empty((n_theta, cols, n_phi + 2), dtype=torch.float64, device="cuda"),
                    work=torch.empty((L * n_theta * cols * 2,), dtype=torch.float64, device="cuda"))
    if case["kind"] == "solve":
        mats, b = systems_of(case, seed)
        lu = rb.BatchedLU(3 * case["n_r"], case["count"])
        lu.factor(mats)
        return dict(case=case, lu=lu, b=b)
    return simulation(case, seed)


QUANTITIES = ["v_r", "v_theta", "v_phi", "entropy", "vort_r", "kinetic_energy", "enstrophy"]


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "step":
        s["g"].step(case["steps"])
        return read_state(s)
    if kind == "change_dt":
        g = s["g"]
        dt = g.cfg.dt
        g.set_dt(0.9 * dt)
        g.step(case["steps"])
        g.set_dt(dt)
        g.step(case["steps"])
        return read_state(s)
    if kind == "output":
        g = s["g"]
        n_r = g.n_r
        g.step(1)
        return dict(slices=g.shell_slices(QUANTITIES[:4], [1, n_r // 2, n_r - 2]),
                    shells=g.shell_averages(QUANTITIES), azimuthal=g.azimuthal_averages(QUANTITIES),
                    equator=g.equatorial_slices(QUANTITIES[:4]), globals=g.global_averages(QUANTITIES),
                    spectra=g.shell_spectra(QUANTITIES[:3], [n_r // 4, n_r // 2]))
    if kind == "transform":
        g, grid, cols, prec = s["g"], s["grid"], case["columns"], PREC[case["precision"]]
        g.transform_dev(0, prec, s["spec"].data_ptr(), grid.data_ptr(), s["work"].data_ptr(), cols)
        if case["way"] == "inverse":
            return grid[..., :-2]
        grid.square_()
        g.transform_dev(1, prec, s["back"].data_ptr(), grid.data_ptr(), s["work"].data_ptr(), cols)
        return s["back"]
    x, _, _ = s["lu"].solve(s["b"], rb.SOLVE_FP64 if case["mode"] == "fp64" else rb.SOLVE_REFINE)
    return x


# ---- what a call cannot do without, and what its outputs may differ by ------------------------------

def work(case):
    if case["kind"] == "solve":
        n = 3 * case["n_r"]
        return dict(bytes=8.0 * case["count"] * n * (n + 2 * case["columns"]),
                    flops=2.0 * case["count"] * case["columns"] * n * n)
    n_theta = case["n_theta"]
    L, n_phi = 2 * n_theta // 3, 2 * n_theta
    n_lm = L * (L + 1) // 2
    fft = 2.5 * n_phi * math.log2(n_phi)    # one real row
    if case["kind"] == "transform":
        cols = case["columns"]
        ways = 1 if case["way"] == "inverse" else 2
        coefficients, grid = n_lm * cols * 16.0, n_theta * cols * n_phi * 8.0
        # the product's grid is an intermediate: only coefficients go in and come out
        return dict(bytes=coefficients + grid if ways == 1 else 2 * coefficients,
                    flops=ways * (2.0 * n_theta * cols * n_lm + n_theta * cols * fft))
    n_r, mag = case["n_r"], case["set"] in ("dynamo", "anelastic")
    nfa, nfb, ng, nf = (17, 7, 18, 6) if mag else (11, 4, 12, 4)
    rows, cols = n_theta * n_r, 2 * n_lm
    legendre = 2.0 * (n_theta // 2) * 2 * n_r * n_lm
    flops = legendre * (nfa + nfb) + (nfa + 3 + nfb) * rows * fft
    flops += 2.0 * (12 if mag else 10) * n_r * n_r * cols
    flops += ng * (2.0 * (n_r // 2) * (2 * n_r // 3) if not case.get("fd") else 10.0 * n_r) * cols
    state = 2 * nf * cols * n_r * 8.0       # the solution and its Adams-Bashforth terms, in and out once a pass
    if case["kind"] == "step":
        return dict(bytes=2 * state, flops=flops * case["steps"])
    if case["kind"] == "change_dt":
        lu = 2.0 / 3.0 * (27 + (3 if mag else 1)) * n_r ** 3 * L
        return dict(bytes=2 * state, flops=2 * (flops * case["steps"] + lu))
    outputs = 8.0 * (4 * 3 * n_theta * n_phi + 7 * n_r * (4 + n_theta) + 4 * n_r * n_phi + 12 * L * L)
    return dict(bytes=2 * state + outputs, flops=flops + legendre * nfa + 7 * rows * fft)


def tolerance(case):
    """About four times what the outputs move by when every input value is off by one rounding, and in
    the mixed form also what the start's FP64 and mixed forms differ by. The largest movement is that of
    the magnetic Adams-Bashforth terms (differences of nearly equal terms); the cgs polytrope's matrices
    (jones) are badly conditioned."""
    mixed = case.get("precision") == "mixed"
    if case["kind"] == "solve":
        return dict(rel=1e-11)
    if case["kind"] == "transform":
        return dict(rel=5e-10 if mixed else 1e-13)
    if case["set"] == "jones":
        return dict(rel=5e-7, max=6e-5)
    if case["set"] == "anelastic":
        return dict(rel=2e-6, max=1e-3) if mixed else dict(rel=2e-11, max=2e-9)
    return dict(rel=2e-7, max=2e-5) if mixed else dict(rel=1e-11, max=1e-9)


# ---- the same in 64 bits, in plain torch and numpy --------------------------------------------------

def legendre(L, x, ms):
    """Normalised P_l^m(x), l = m .. L - 1, for one m at the nodes x, by the three-term recurrence with
    sin^m carried as a logarithm (each m's block as [l][x])."""
    s = np.sqrt(1.0 - x * x)
    for m in ms:
        i = np.arange(1, m + 1)
        log = 0.5 * np.log((m + 0.5) / (2 * math.pi)) + 0.5 * np.log((2 * i - 1.0) / (2 * i)).sum()
        log = log + m * np.log(s)
        p = np.zeros((L - m, x.size))
        scale = np.maximum(log, -600.0)                # values below e^-600 start from there
        a, b, e = np.zeros_like(x), (-1.0) ** m * np.exp(scale), log - scale
        p[0] = b * np.exp(np.maximum(e, -700.0)) * (e > -700.0)
        for l in range(m + 1, L):
            up = math.sqrt((4.0 * l * l - 1) / (l * l - m * m))
            down = math.sqrt(((l - 1.0) ** 2 - m * m) / (4.0 * (l - 1) ** 2 - 1)) if l > m + 1 else 0.0
            a, b = b, up * (x * b - down * a)
            grow = np.abs(b) > 1e200                   # keep the carried factor in range
            if grow.any():
                f = np.where(grow, 1e-200, 1.0)
                a, b, e = a * f, b * f, e - np.log(f)
            p[l - m] = b * np.exp(np.maximum(e, -700.0)) * (e > -700.0)
        yield p


def exact(case, seed):
    """None for the time stepping and its outputs: in 64 bits they take a second implementation of the
    whole model (the repository's own NumPy restatement needs minutes at these sizes)."""
    if case["kind"] == "solve":
        mats, b = systems_of(case, seed)
        a = torch.as_tensor(mats).cuda().transpose(1, 2)
        return torch.linalg.solve(a, torch.as_tensor(b).cuda().transpose(1, 2)).transpose(1, 2).contiguous()
    if case["kind"] != "transform":
        return None
    n_theta, cols = case["n_theta"], case["columns"]
    L, n_phi = 2 * n_theta // 3, 2 * n_theta
    x, w = np.polynomial.legendre.leggauss(n_theta)    # ascending: the grid's rows run from the south pole
    spec = columns_of(case, seed)
    fourier = torch.zeros((n_theta, cols, n_phi // 2 + 1), dtype=torch.complex128, device="cuda")
    starts = np.concatenate([[0], np.cumsum(np.arange(L, 0, -1))])
    order = [np.concatenate([np.arange(0, L - m, 2), np.arange(1, L - m, 2)]) for m in range(L)]
    for m, p in enumerate(legendre(L, x, range(L))):
        p = torch.as_tensor(p[order[m]]).cuda() * (1.0 if m == 0 else 0.5)
        rows = spec[starts[m]:starts[m + 1]].reshape(L - m, 2 * cols)
        fourier[:, :, m] = torch.view_as_complex((p.T @ rows).reshape(n_theta, cols, 2))
    grid = torch.fft.irfft(fourier, n=n_phi, norm="forward")
    del fourier
    if case["way"] == "inverse":
        return grid
    fourier = torch.fft.rfft(grid.square_())
    back = torch.empty_like(spec)
    weight = torch.as_tensor(2 * math.pi * w).cuda()[:, None]
    for m, p in enumerate(legendre(L, x, range(L))):
        p = torch.as_tensor(p[order[m]]).cuda() * ((0.5 if m == 0 else 1.0) / n_theta)
        f = torch.view_as_real(fourier[:, :, m].contiguous()).reshape(n_theta, 2 * cols)
        back[starts[m]:starts[m + 1]] = (p @ (weight * f)).reshape(L - m, cols, 2)
    return back

