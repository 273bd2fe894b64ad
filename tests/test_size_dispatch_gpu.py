"""The kernels chosen by size, at the sizes where they can go wrong.

Tolerances: FP64 rounding of the path times a small factor (WENO steps and
transforms 1e-11 as the parity tests), FP32-mixed 1e-5 against FP64.
"""
import numpy as np
import pytest

from aeolus_b200 import CoreSpec, regular_grid
from aeolus_b200.inputs import embed, taylor_green
from oracle.oracle import OracleSimulation

pytestmark = pytest.mark.gpu


def Sim(spec):
    from aeolus_b200.simulation import Simulation
    return Simulation(spec)


def rel(a, b):
    n = np.linalg.norm(b)
    return np.linalg.norm(a - b) / (n if n > 0 else 1.0)


def random_state(g, seed, amp=1.0):
    rng = np.random.default_rng(seed)
    f = [embed(g, amp * rng.standard_normal((g.nz, g.ny, g.nx))) for _ in range(4)]
    if g.bc_z == "wall":
        f[2][g.halo[2]] = 0.0
    return f


# ---- the tiled WENO sweeps: tiles of 32 x 8 cells, chunks of levels by the number of tiles ---------------------
@pytest.mark.parametrize("size,bc_z", [((16, 4, 5), "wall"), ((32, 8, 4), "periodic"), ((64, 16, 13), "wall"),
                                       ((32, 32, 64), "periodic")])
@pytest.mark.parametrize("scheme", ["weno_js5", "weno_z5"])
@pytest.mark.parametrize("c_s", [0.0, 0.17])
def test_weno_steps_at_tile_and_chunk_edges(size, bc_z, scheme, c_s):
    g = regular_grid(size, (2 * np.pi,) * 3, bc_z=bc_z)
    kw = dict(grid=g, advection=scheme, nu=1e-3, c_s=c_s, theta0=300.0 if bc_z == "wall" else 0.0)
    state = random_state(g, 5, 0.5)
    state[3][g.interior] += kw["theta0"]
    o = OracleSimulation(CoreSpec(**kw))
    s64, s32 = Sim(CoreSpec(**kw)), Sim(CoreSpec(precision="fp32_mixed", **kw))
    for s in (o, s64, s32):
        s.set_state(*state)
        s.project()
        s.step_rk3(1e-3, 3)
    for n in ("u", "v", "w", "theta", "p"):
        want = o.get_field(n)[g.interior]
        assert rel(s64.get_field(n)[g.interior], want) <= 1e-11, n
        # the pressure is phi / dt: the FP32 divergence's rounding over it
        assert rel(s32.get_field(n)[g.interior], want) <= (1e-5 if n != "p" else 1e-3), n


@pytest.mark.parametrize("scheme", ["weno_js5", "weno_z5"])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-13), ("fp32_mixed", 1e-6)])
def test_weno_keeps_a_uniform_field_and_scales(scheme, precision, tol):
    """A uniform wind carries a uniform scalar unchanged, whatever its size, and the reconstruction of a field
    scaled by a power of two is the scaled one where its indicators stand far above eps."""
    g = regular_grid((32, 16, 16), (1.0, 1.0, 1.0))
    one = np.ones(g.storage_shape)
    for scale in (1e-6, 1.0, 1e6):
        s = Sim(CoreSpec(grid=g, advection=scheme, precision=precision))
        s.set_state(one, 0.5 * one, -0.25 * one, scale * one)
        s.step_rk3(1e-3, 2)
        assert np.abs(s.get_field("theta")[g.interior] / scale - 1).max() <= tol
        assert np.abs(s.get_field("u")[g.interior] - 1).max() <= tol
    rng = np.random.default_rng(3)
    th = embed(g, rng.standard_normal((g.nz, g.ny, g.nx)))
    out = []
    for scale in (1.0, 2.0 ** 24):
        s = Sim(CoreSpec(grid=g, advection="weno_z5", precision=precision))
        s.set_state(one, 0.5 * one, -0.25 * one, scale * th)
        s.step_rk3(1e-3)
        out.append(s.get_field("theta")[g.interior] / scale)
    assert rel(out[1], out[0]) <= (1e-12 if precision == "fp64" else 1e-5)


# ---- the diagnostics' levels, shared by several CTAs -----------------------------------------------------------
@pytest.mark.parametrize("size", [(8, 4, 3), (64, 64, 5), (128, 64, 2), (256, 128, 4)])
@pytest.mark.parametrize("precision", ["fp64", "fp32_mixed"])
def test_cfl_and_guard_over_shared_levels(size, precision):
    from aeolus_b200.simulation import CFLConstraints
    g = regular_grid(size, (2.0, 1.0, 0.5), bc_z="wall")
    kw = dict(grid=g, theta0=300.0, c_s=0.17, nu=1e-3)
    state = random_state(g, 2, 0.1)
    # one fast cell in the last row of the middle level sets the rate
    k = g.halo[2] + g.nz // 2
    state[0][k, -1 - g.halo[1], -1 - g.halo[0]] = 7.0
    state[3] += 300.0 + np.arange(g.storage_shape[0])[:, None, None]
    o, s = OracleSimulation(CoreSpec(**kw)), Sim(CoreSpec(precision=precision, **kw))
    for q in (o, s):
        q.set_state(*state)
    c = CFLConstraints(divergence_tol=1e9, max_retries=0)
    want, got = o.adaptive_dt(c)[0], s.cfl_diagnostics(c)
    assert abs(got["dt"] - want) <= (1e-12 if precision == "fp64" else 1e-5) * want
    rate = 0.5 / got["advective_rate"]
    assert rate < 0.5 * g.dx / 6.9
    st = s.step_adaptive(c)
    u = [s.get_field(n)[g.interior] for n in ("u", "v", "w")]
    assert st["max_speed"] == max(np.abs(a).max() for a in u)
    assert abs(st["max_divergence"] - s.max_divergence()) <= 1e-12 * max(1.0, st["max_divergence"])
    bad = [a.copy() for a in state]
    bad[3][k, g.halo[1], g.halo[0]] = np.nan
    s.set_state(*bad)
    from aeolus_b200._lib import NumericalFailure
    with pytest.raises(NumericalFailure):
        s.step_adaptive(c)


# ---- the transforms: registers for 32 .. 512 points a line, shared memory otherwise ----------------------------
def poisson(g, b):
    """The FFT solver's answer in numpy (zero mean mode)."""
    k = [4 / h ** 2 * np.sin(np.pi * np.arange(n) / n) ** 2 for h, n in ((g.dz, g.nz), (g.dy, g.ny), (g.dx, g.nx))]
    lam = -(k[0][:, None, None] + k[1][None, :, None] + k[2][None, None, :])
    lam[0, 0, 0] = 1.0
    f = np.fft.fftn(b) / lam
    f[0, 0, 0] = 0
    return np.fft.ifftn(f).real


@pytest.mark.parametrize("size", [(32, 16, 16), (64, 32, 32), (128, 64, 8), (256, 128, 4), (512, 8, 64), (1024, 4, 128),
                                  (2048, 4, 4), (16, 256, 8), (8, 512, 4), (4, 1024, 8), (8, 4, 256), (4, 8, 512),
                                  (4, 4, 1024), (64, 64, 64)])
@pytest.mark.parametrize("precision,eps", [("fp64", 2.0 ** -53), ("fp32_mixed", 2.0 ** -24)])
def test_fft_pressure_solve_at_every_length(size, precision, eps):
    """Tolerance: the two transforms' rounding, eps log2(N) |b| each in the 2-norm, grows by the largest 1/lambda of the
    inverted operator; |b| max(1/lambda) / |x| makes that a relative error."""
    g = regular_grid(size, (1.0, 0.7, 1.3))
    b = np.random.default_rng(sum(size)).standard_normal((g.nz, g.ny, g.nx))
    s = Sim(CoreSpec(grid=g, precision=precision))
    x, want = s.pressure_solve(b), poisson(g, b)
    low = max(h * h / 4 / np.sin(np.pi / n) ** 2 for h, n in ((g.dx, g.nx), (g.dy, g.ny), (g.dz, g.nz)))
    assert rel(x, want) <= 2 * eps * np.log2(g.ncells) * low * np.linalg.norm(b) / np.linalg.norm(want)


@pytest.mark.parametrize("size", [(32, 8, 7), (64, 32, 5), (128, 16, 33), (256, 64, 3), (512, 4, 9), (16, 128, 6)])
@pytest.mark.parametrize("core", ["boussinesq", "anelastic"])
@pytest.mark.parametrize("stretched", [False, True])
def test_column_projection_at_every_row_length(size, core, stretched):
    """The divergence formed in the r2c's loads (plain, W-weighted, stretched), through the column solve: the
    projected velocity and phi match the oracle's, and a source array through the same transforms too."""
    from aeolus_b200 import stretched_grid, tanh_faces
    from aeolus_b200.reference_state import anelastic_profiles, exponential_density
    nz = size[2]
    if stretched:
        g = stretched_grid(size, (1000.0, 800.0, 600.0), tanh_faces(nz, 600.0, 0.8))
    else:
        g = regular_grid(size, (1000.0, 800.0, 600.0), bc_z="wall")
    kw = dict(grid=g)
    if core == "anelastic":
        prof = anelastic_profiles(g, exponential_density(g), np.full(nz, 300.0))
        kw.update(core=core, wc=prof["wc"], wf=prof["wf"], thf=prof["thf"])
    o, s64, s32 = OracleSimulation(CoreSpec(**kw)), Sim(CoreSpec(**kw)), Sim(CoreSpec(precision="fp32_mixed", **kw))
    for s in (o, s64, s32):
        s.set_state(*random_state(g, 9))
        s.project()
    for n in ("u", "v", "w"):
        want = o.get_field(n)[g.interior]
        assert rel(s64.get_field(n)[g.interior], want) <= 1e-12, n
        assert rel(s32.get_field(n)[g.interior], want) <= 1e-5, n
    b = np.random.default_rng(1).standard_normal((nz, g.ny, g.nx))
    assert rel(s64.pressure_solve(b), o.pressure_solve(b)) <= 1e-12


# ---- the column solve: depths below, at and above its ring of levels --------------------------------------------
@pytest.mark.parametrize("nz", [2, 3, 4, 5, 6, 7, 8, 9, 15, 16, 17, 31, 64, 93])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("fp32_mixed", 1e-4)])
def test_column_solve_of_every_depth(nz, precision, tol):
    g = regular_grid((16, 4, nz), (1.0, 1.0, 0.1 * nz), bc_z="wall")
    b = np.random.default_rng(nz).standard_normal((nz, 4, 16))
    b -= b.mean()
    s, o = Sim(CoreSpec(grid=g, precision=precision)), OracleSimulation(CoreSpec(grid=g))
    assert rel(s.pressure_solve(b), o.pressure_solve(b)) <= tol


# ---- the centred sweeps: FP32 persistent CTAs over (64 x 8 tile, level) items, FP64 32 x 8 tiles in chunks of levels
@pytest.mark.parametrize("size,wall", [((8, 4, 5), True), ((32, 8, 4), False), ((64, 16, 13), True), ((128, 4, 33), True),
                                       ((32, 32, 64), False)])
@pytest.mark.parametrize("sgs", [None, "smagorinsky", "vreman", "sigma", "dynamic", "amd"])
def test_centred_steps_at_tile_and_range_edges(size, wall, sgs):
    g = regular_grid(size, (2 * np.pi,) * 3, bc_z="wall" if wall else "periodic")
    kw = dict(grid=g, nu=1e-3, theta0=300.0 if wall else 0.0)
    if sgs:
        kw.update(sgs=sgs, c_s=0.5 if sgs == "dynamic" else 0.17)
    state = random_state(g, 7, 0.5)
    state[3] += kw["theta0"]
    o = OracleSimulation(CoreSpec(**kw))
    s64, s32 = Sim(CoreSpec(**kw)), Sim(CoreSpec(precision="fp32_mixed", **kw))
    for s in (o, s64, s32):
        s.set_state(*state)
        s.project()
        s.step_rk3(1e-3, 2)
    for n in ("u", "v", "w", "theta"):
        want = o.get_field(n)[g.interior]
        assert rel(s64.get_field(n)[g.interior], want) <= 1e-11, n
        # the dynamic coefficient is a quotient of differences, its FP32 form the pair tests'
        assert rel(s32.get_field(n)[g.interior], want) <= (1e-4 if sgs == "dynamic" else 1e-5), n


@pytest.mark.parametrize("size", [(16, 8, 5), (64, 16, 33)])
@pytest.mark.parametrize("core", ["boussinesq", "anelastic"])
@pytest.mark.parametrize("stretched", [False, True])
@pytest.mark.parametrize("c_s", [0.0, 0.17])
def test_centred_steps_of_every_column_form(size, core, stretched, c_s):
    from aeolus_b200 import stretched_grid, tanh_faces
    from aeolus_b200.reference_state import anelastic_profiles, exponential_density
    nz = size[2]
    if stretched:
        g = stretched_grid(size, (1000.0, 800.0, 600.0), tanh_faces(nz, 600.0, 0.8))
    else:
        g = regular_grid(size, (1000.0, 800.0, 600.0), bc_z="wall")
    kw = dict(grid=g, nu=0.1, c_s=c_s, theta0=300.0, g=9.81)
    if core == "anelastic":
        prof = anelastic_profiles(g, exponential_density(g), np.full(nz, 300.0))
        kw.update(core=core, wc=prof["wc"], wf=prof["wf"], thf=prof["thf"])
    state = random_state(g, 8)
    state[3] += 300.0
    o, s64, s32 = OracleSimulation(CoreSpec(**kw)), Sim(CoreSpec(**kw)), Sim(CoreSpec(precision="fp32_mixed", **kw))
    for s in (o, s64, s32):
        s.set_state(*state)
        s.project()
        s.step_rk3(0.1, 2)
    for n in ("u", "v", "w", "theta"):
        want = o.get_field(n)[g.interior]
        assert rel(s64.get_field(n)[g.interior], want) <= 1e-11, n
        assert rel(s32.get_field(n)[g.interior], want) <= 1e-5, n



# ---- the multigrid cycle and the CG loop -----------------------------------------------------------------------
def cut_coeffs(n, seed):
    nx, ny, nz = n
    rng = np.random.default_rng(seed)
    c = [rng.choice([0.0, 0.3, 0.7, 1.0], s, p=[0.1, 0.1, 0.1, 0.7]) for s in ((nz, ny, nx + 1), (nz, ny + 1, nx), (nz + 1, ny, nx))]
    c[0][:, :, -1], c[1][:, -1] = c[0][:, :, 0], c[1][:, 0]
    c[2][0] = c[2][-1] = 0.0
    return c


@pytest.mark.parametrize("n", [(4, 4, 4), (32, 16, 8), (66, 6, 4), (64, 8, 12), (120, 88, 40), (256, 128, 64)])
@pytest.mark.parametrize("form", ["constant", "codes", "values"])
def test_cycle_over_every_level_size(n, form):
    """One cycle against the oracle's: levels of one pass per plane and of marching columns, coefficient forms."""
    from aeolus_b200.multigrid import MGPreconditionedCG
    from oracle.mgpcg import OracleMGPCG
    c = None if form == "constant" else cut_coeffs(n, sum(n))
    if form == "values":
        c = [a * (1 + 0.1 * np.sin(np.arange(a.size).reshape(a.shape))) for a in c]
        c[0][:, :, -1], c[1][:, -1] = c[0][:, :, 0], c[1][:, 0]
    b = np.random.default_rng(3).standard_normal(n[::-1])
    h = (1.0, 1.3, 0.7)
    want = OracleMGPCG(n, h, coeffs=c).precondition(b)
    assert rel(MGPreconditionedCG(n, h, coeffs=c).precondition(b), want) <= 1e-11
    assert rel(MGPreconditionedCG(n, h, coeffs=c, precision="fp32_mixed").precondition(b), want) <= 1e-4


@pytest.mark.parametrize("precond", ["vcycle", "jacobi", "identity"])
@pytest.mark.parametrize("n", [(16, 8, 8), (40, 24, 12), (9, 7, 5)])
def test_cg_loop_counts_and_ends(n, precond):
    """The loop ends after the update that converged or at maxit, with the oracle's count, the residual it reports
    and the same iterates as the harvesting graph; a zero right-hand side and a huge tolerance end it before."""
    from aeolus_b200.multigrid import MGPreconditionedCG
    c = cut_coeffs(n, 11) if n[0] != 9 else None
    b = MGPreconditionedCG(n, (1.0,) * 3, coeffs=c).apply(np.random.default_rng(4).standard_normal(n[::-1]))
    make = lambda **k: MGPreconditionedCG(n, (1.0,) * 3, coeffs=c, precond=precond, **k)
    for maxit in (1, 2, 5):
        s = make(tol=1e-30, maxit=maxit)
        x, st = s.solve(b)
        assert st["iterations"] == maxit and st["status"] == "maxit", st
        y, sh, pairs = s.solve_harvest(b, cap=8)
        assert np.array_equal(x, y) and sh["iterations"] == maxit and len(pairs) == maxit + 1
        r = b - b.mean() - s.apply(x)
        assert abs(np.linalg.norm(r) - st["residual"]) <= 1e-10 * st["bnorm"]
    s = make(tol=1e-6, maxit=400)
    for _ in range(2):
        x, st = s.solve(b)
        assert st["status"] == "converged" and st["residual"] <= 1e-6 * st["bnorm"]
    x, st = s.solve(np.zeros_like(b))
    assert st["status"] == "zero_rhs" and st["iterations"] == 0 and not x.any()
    for tol, maxit, status in ((2.0, 5, "converged"), (1.0, 1, "converged"), (2.0, 0, "converged"), (0.5, 0, "maxit")):
        x, st = make(tol=tol, maxit=maxit).solve(b)
        assert st["status"] == status and st["iterations"] == 0 and not x.any(), (tol, maxit)
        assert st["residual"] == st["bnorm"] > 0


# ---- the positivity-preserving advection: tiles of 64 (FP32) or 32 columns by 8 rows, chunks of one level (few tiles)
# to a dozen, whole and ragged
@pytest.mark.parametrize("size", [(8, 4, 3), (16, 8, 9), (64, 8, 8), (32, 16, 33), (128, 32, 40), (64, 4, 70),
                                  (256, 4, 24), (128, 64, 25), (256, 128, 40), (256, 64, 100)])
@pytest.mark.parametrize("scheme", ["weno_z5", "weno_js5"])
def test_positive_tendency_over_ragged_tiles(size, scheme):
    g = regular_grid(size, (1.0, 0.8, 0.6), bc_z="wall")
    u, v, w, phi = random_state(g, 5)
    phi = np.where(np.abs(phi) < 0.3, 0.0, np.abs(phi))
    base = np.random.default_rng(6).standard_normal(g.storage_shape)
    dt = 0.05 * min(g.dx, g.dy, g.dz)
    o = OracleSimulation(CoreSpec(grid=g))
    for precision, tol in (("fp64", 1e-11), ("fp32_mixed", 1e-5)):
        s = Sim(CoreSpec(grid=g, precision=precision))
        for acc in (False, True):
            want = o.advect_positive(u, v, w, phi, dt, scheme=scheme, tend=base, accumulate=acc)
            got = s.advect_positive(u, v, w, phi, dt, scheme=scheme, tend=base, accumulate=acc)
            assert rel(got[g.interior], want[g.interior]) <= tol
            if not acc and precision == "fp64":
                assert (phi + dt * got)[g.interior].min() >= -1e-14


# ---- the halo fill where rows and columns have several images ----------------------------------------------------
@pytest.mark.parametrize("size,bc_z", [((4, 4, 4), "periodic"), ((4, 4, 4), "wall"), ((8, 4, 8), "periodic"),
                                       ((4, 8, 5), "wall"), ((16, 4, 3), "wall"), ((8, 8, 2), "wall"), ((64, 32, 7), "wall")])
@pytest.mark.parametrize("scheme", ["centred", "weno_z5"])
def test_halo_images_at_the_smallest_extents(size, bc_z, scheme):
    g = regular_grid(size, (1.0, 1.0, 1.0), bc_z=bc_z)
    kw = dict(grid=g, advection=scheme, nu=1e-3)
    state = random_state(g, 12, 0.5)
    o = OracleSimulation(CoreSpec(**kw))
    s64, s32 = Sim(CoreSpec(**kw)), Sim(CoreSpec(precision="fp32_mixed", **kw))
    for s in (o, s64, s32):
        s.set_state(*state)
        s.project()
        s.step_rk3(2e-3, 3)
    for n in ("u", "v", "w", "theta"):
        want = o.get_field(n)[g.interior]
        assert rel(s64.get_field(n)[g.interior], want) <= 1e-11, n
        assert rel(s32.get_field(n)[g.interior], want) <= 1e-5, n


# ---- the U-Net: weight gradients of x-segment tiles at every channel count, host arrays through pinned lanes ----
@pytest.mark.parametrize("shape", [(512, 24, 8), (256, 16, 12), (512, 8, 16)])
def test_unet_gradients_where_every_level_takes_x_segments(shape):
    import test_unet_gpu
    test_unet_gpu.test_gradients_match_the_oracle(shape)



@pytest.mark.parametrize("shape", [(128, 16, 8), (128, 64, 32), (256, 64, 56), (512, 64, 32), (256, 48, 92)])
def test_host_arrays_pageable_pinned_and_from_threads(shape):
    """Below and above the size that takes the pinned lanes, whole and ragged chunks, as often as it takes until a
    handle uses the lanes: the same bits as from pinned arrays, and from several handles at once."""
    import threading
    import torch
    from aeolus_b200.unet import UNet
    rng = np.random.default_rng(1)
    n = shape[::-1]
    mask = (rng.random(n) > 0.1).astype(np.float32)
    rs = [rng.standard_normal(n) * mask for _ in range(3)]
    e = rng.standard_normal(n) * mask
    nets = [UNet(shape, seed=5) for _ in range(3)]
    want = []
    for net, r in zip(nets, rs):
        net.set_mask(mask)
        pin = torch.from_numpy(r).pin_memory().numpy()
        want.append(np.array(net.apply(pin)))
    loss = nets[0].gradients(torch.from_numpy(rs[0]).pin_memory().numpy(), torch.from_numpy(e).pin_memory().numpy())
    assert abs(nets[0].gradients(rs[0], e) - loss) <= 1e-12 * abs(loss)
    got = [None] * 3

    def work(q):
        for _ in range(3 + (40 << 20) // (2 * rs[q].nbytes)):   # the lanes' buffers are worth 40 MiB of plain copies
            got[q] = np.array(nets[q].apply(rs[q]))
            assert np.array_equal(got[q], want[q])

    th = [threading.Thread(target=work, args=(q,)) for q in range(3)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("steps", [1, 2, 3, 5])
@pytest.mark.parametrize("kw", [{}, {"precision": "fp32_mixed"}, {"solver": "pcg"}], ids=lambda kw: "-".join(kw.values()))
def test_a_run_of_steps_against_the_oracle(steps, kw):
    """The direct solvers' graph a step and the PCG solver's graph of pairs: the state after a run of odd and even
    length, p included (written in a step's last substage only), is the oracle's."""
    g = regular_grid((16, 16, 8), (1.0, 1.0, 1.0), bc_z="wall")
    s, o = Sim(CoreSpec(grid=g, nu=1e-3, **kw)), OracleSimulation(CoreSpec(grid=g, nu=1e-3, solver=kw.get("solver")))
    for q in (s, o):
        if "solver" in kw:
            q.set_pcg(None, tol=1e-12, maxit=100)
        q.set_state(*random_state(g, 9, 0.3))
        q.project()
        q.step_rk3(1e-3, steps)
    fp64 = "precision" not in kw
    for n in ("u", "v", "w", "theta", "p"):
        want = o.get_field(n)[g.interior]
        # the pressure is phi / dt: the solve's tolerance (1e-12 of the divergence) or the FP32 divergence's rounding over it
        tol = (1e-11 if n != "p" else 1e-8) if fp64 else (1e-5 if n != "p" else 1e-3)
        assert rel(s.get_field(n)[g.interior], want) <= tol, n
