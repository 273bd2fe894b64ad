"""The work a user has this framework do, as timed cases through its public
entry points: runs of the projected SSP-RK3 step (a few steps and the read of
the state, which is how a driver uses them between two outputs), the cut-cell
pressure solve on device arrays, the positivity-preserving tracer advection,
and the learned preconditioner's forward pass and training step.

`exact` restates each path in plain torch at 64 bits from the discrete
operators (it shares nothing with the package).
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PACKAGE = os.path.join(ROOT, "aeolus.jl_b200")
if PACKAGE not in sys.path:
    sys.path.insert(0, PACKAGE)

F64 = torch.float64
FIELDS = ("u", "v", "w", "theta", "p")


# ---- the cases ---------------------------------------------------------------
def listed():
    return [
        # the plain verification run: small, so launches and latency are what it costs
        {"name": "tgv_64_fp64", "kind": "step", "flow": "tgv", "nx": 64, "ny": 64, "nz": 64, "precision": "fp64",
         "steps": 20},
        # the dry convective boundary layer, the headline workload, in both precisions
        {"name": "cbl_256x256x128_fp32", "kind": "step", "flow": "cbl", "nx": 256, "ny": 256, "nz": 128,
         "precision": "fp32_mixed", "steps": 20},
        {"name": "cbl_256x256x128_fp64", "kind": "step", "flow": "cbl", "nx": 256, "ny": 256, "nz": 128,
         "precision": "fp64", "steps": 10},
        # a smaller, elongated boundary layer with an odd number of levels (columns need no power of two)
        {"name": "cbl_128x64x93_fp32", "kind": "step", "flow": "cbl", "nx": 128, "ny": 64, "nz": 93,
         "precision": "fp32_mixed", "steps": 20},
        # decaying isotropic turbulence, WENO-Z5 and adaptive steps: the largest grid, and FP64
        {"name": "hit_512_fp32", "kind": "step", "flow": "hit", "nx": 512, "ny": 512, "nz": 512,
         "precision": "fp32_mixed", "steps": 8},
        {"name": "hit_256_fp64", "kind": "step", "flow": "hit", "nx": 256, "ny": 256, "nz": 256,
         "precision": "fp64", "steps": 4},
        # the heated urban flow: WENO-JS5, Smagorinsky, every projection a multigrid-preconditioned CG
        {"name": "urban_256x256x96_fp32", "kind": "step", "flow": "urban", "nx": 256, "ny": 256, "nz": 96,
         "precision": "fp32_mixed", "steps": 2},
        # the cut-cell pressure solve by itself: the urban problem, and a small grid that is no power of two
        {"name": "solve_256x256x96_fp32", "kind": "solve", "nx": 256, "ny": 256, "nz": 96, "precision": "fp32_mixed"},
        {"name": "solve_120x88x40_fp64", "kind": "solve", "nx": 120, "ny": 88, "nz": 40, "precision": "fp64"},
        # one tracer's limited WENO-Z5 tendency
        {"name": "tracer_256_fp32", "kind": "tracer", "nx": 256, "ny": 256, "nz": 256, "bc_z": "periodic",
         "scheme": "weno_z5", "precision": "fp32_mixed"},
        # the learned preconditioner: a training step's forward and backward pass at the urban grid (its Adam update
        # of 0.1 M parameters comes on top), a forward pass at the training grid
        {"name": "unet_train_256x256x96", "kind": "unet_train", "nx": 256, "ny": 256, "nz": 96},
        {"name": "unet_apply_128x128x48", "kind": "unet_apply", "nx": 128, "ny": 128, "nz": 48},
    ]


def draw(rng):
    def pow2(lo, hi):
        return 2 ** rng.randint(lo, hi)

    def spread(lo, hi, multiple=1):
        return max(lo, multiple * round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / multiple))

    kind = rng.choice(("tgv", "cbl", "cbl", "hit", "dns", "urban", "solve", "solve", "tracer", "unet_train",
                       "unet_apply"))
    precision = rng.choice(("fp64", "fp32_mixed"))
    if kind in ("tgv", "hit", "dns"):
        return {"kind": "step", "flow": kind, "nx": pow2(5, 8), "ny": pow2(5, 8), "nz": pow2(5, 8),
                "precision": precision, "steps": rng.randint(3, 6)}
    if kind == "cbl":
        return {"kind": "step", "flow": kind, "nx": pow2(5, 8), "ny": pow2(5, 8), "nz": spread(24, 192),
                "precision": precision, "steps": rng.randint(5, 20)}
    if kind == "urban":
        return {"kind": "step", "flow": kind, "nx": pow2(5, 8), "ny": pow2(5, 8), "nz": spread(24, 96, 8),
                "precision": precision, "steps": rng.randint(1, 2)}
    if kind == "solve":
        return {"kind": kind, "nx": spread(48, 320, 16), "ny": spread(48, 320, 16), "nz": spread(24, 120, 8),
                "precision": precision}
    if kind == "tracer":
        bc_z = rng.choice(("periodic", "wall"))
        return {"kind": kind, "nx": pow2(5, 8), "ny": pow2(5, 8),
                "nz": pow2(5, 8) if bc_z == "periodic" else spread(24, 240), "bc_z": bc_z,
                "scheme": rng.choice(("weno_z5", "weno_js5")), "precision": precision}
    return {"kind": kind, "nx": rng.choice((128, 256)), "ny": spread(32, 256, 16), "nz": spread(16, 96, 4)}


def work(case):
    n = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] == "step":
        word = 8 if case["precision"] == "fp64" else 4
        # a substage's sweep reads u, v, w, theta and writes the predictor and theta, the pressure solve reads
        # the predictor and writes phi, the correction reads both and writes u, v, w; substages 2 and 3 also
        # read the four step-start fields; p once per step, and the five fields are read out at the end
        passes = 3 * (8 + 4 + 7) + 2 * 4 + 1
        points = n * case["steps"]
        # operations a cell and substage: 12 reconstructions of ~75 and their fluxes for WENO, ~130 centred,
        # ~170 with the closure, and the two transforms' 5 log2 N
        flops = 1000.0 if case["flow"] in ("tgv", "hit", "urban") else 130.0
        if case["flow"] in ("cbl", "urban"):
            flops += 170.0
        flops += 5.0 * math.log2(n)
        return {"bytes": float(word * (passes * points + 5 * n)), "flops": 3.0 * flops * points}
    if case["kind"] == "solve":
        # the solution cannot be had without reading b and the three faces' coefficients (one-byte codes) and
        # writing x; iterations come on top
        return {"bytes": n * (8.0 + 3.0 + 8.0), "flops": n * 30.0}
    if case["kind"] == "tracer":
        word = 8 if case["precision"] == "fp64" else 4
        return {"bytes": 5.0 * n * word, "flops": n * (3 * 75.0 + 80.0)}
    # U-Net: 3x3x3 convolutions of 16/32/32 channels, 2 * 27 * c_in * c_out a cell at the layer's level
    fwd = 2 * 27 * (4 * 256 + (512 + 1024 + 512) / 8 + 2 * 1024 / 64)
    if case["kind"] == "unet_apply":
        return {"bytes": n * 16.0, "flops": n * fwd}
    return {"bytes": n * 16.0, "flops": 3.0 * n * fwd}


def tolerance(case):
    """About four times what the paths are off from `exact`, over the ranges (the largest of the outputs)."""
    if case["kind"] == "unet_apply":
        return {"rel": 0.03, "max": 0.4}      # bf16 weights and activations: 0.010
    if case["kind"] == "unet_train":
        return {"rel": 0.03, "max": 0.9}      # the same through the backward pass, every parameter's gradient
    if case["kind"] == "solve":
        return {"rel": 1e-7, "max": 1e-5}     # residuals of 1e-8 of the right-hand side: 1e-9 to 2e-8
    if case["kind"] == "tracer":
        return {"rel": 2e-14, "max": 1e-10} if case["precision"] == "fp64" else {"rel": 1e-6, "max": 1e-3}
    if case["flow"] == "urban":
        return {"rel": 1e-6, "max": 1e-3} if case["precision"] == "fp64" else {"rel": 2e-6, "max": 2e-3}
    if case["precision"] == "fp64":
        return {"rel": 6e-12, "max": 1e-9}    # the pressure of the stretched anelastic column: 1.3e-12
    return {"rel": 3e-5, "max": 3e-3}         # the vertical velocity of the boundary layer: 7e-6


# ---- inputs, made on the device in 64 bits and handed over as host arrays --------
def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _generator(seed, stream):
    g = torch.Generator(device=_device())
    g.manual_seed(1000003 * int(seed) + stream)
    return g


def _spectral_noise(shape, gen, k_peak=4.0):
    """A random-phase field of energy spectrum k^4 exp(-2 (k / k_peak)^2) and unit rms."""
    nz, ny, nx = shape
    f = torch.fft.rfftn(torch.randn(shape, generator=gen, device=_device(), dtype=F64))
    kz = torch.fft.fftfreq(nz, 1.0 / nz, device=f.device, dtype=F64)[:, None, None]
    ky = torch.fft.fftfreq(ny, 1.0 / ny, device=f.device, dtype=F64)[None, :, None]
    kx = torch.fft.rfftfreq(nx, 1.0 / nx, device=f.device, dtype=F64)[None, None, :]
    k2 = kx * kx + ky * ky + kz * kz
    f *= k2.sqrt() * torch.exp(-k2 / k_peak ** 2)
    f[0, 0, 0] = 0
    out = torch.fft.irfftn(f, s=shape)
    return out / out.square().mean().sqrt()


def _uniform(shape, gen, amp):
    return amp * (2.0 * torch.rand(shape, generator=gen, device=_device(), dtype=F64) - 1.0)


def _layout(case):
    """Extents, faces and physical constants of a flow: plain numbers both sides build from."""
    flow, nx, ny, nz = case["flow"], case["nx"], case["ny"], case["nz"]
    d = {"halo": 3, "zf": None, "nu": 0.0, "c_s": 0.0, "theta0": 0.0, "flux_bot": 0.0, "g": 9.81, "pr_t": 1.0 / 3.0,
         "core": "boussinesq", "advection": "centred", "adaptive": False, "bc_z": "periodic"}
    if flow in ("tgv", "hit", "dns"):
        d["extent"] = tuple(2 * math.pi * m / max(nx, ny, nz) for m in (nx, ny, nz))
        if flow == "tgv":
            d.update(advection="weno_js5", nu=1.0 / 1600, dt=0.01 * 64 / max(nx, ny, nz))
        elif flow == "hit":
            d.update(advection="weno_z5", adaptive=True)
        else:
            d.update(nu=1e-3, dt=0.2 * d["extent"][0] / nx / 4.0)
    elif flow == "cbl":
        # 2 km deep, first cell about half of the uniform one, 20 m horizontally
        lz, beta = 2000.0, 1.0735
        xi = np.arange(nz + 1) / nz
        zf = lz * (1 - np.tanh(beta * (1 - xi)) / np.tanh(beta))
        zf[0], zf[-1] = 0.0, lz
        d.update(extent=(20.0 * nx, 20.0 * ny, lz), zf=zf, core="anelastic", c_s=0.17, flux_bot=0.1, bc_z="wall",
                 dt=min(1.0, 0.1 * (zf[1] - zf[0])))
    else:
        d.update(extent=(2.0 * nx, 2.0 * ny, 2.0 * nz), advection="weno_js5", c_s=0.17, theta0=300.0, flux_bot=0.15,
                 bc_z="wall", dt=0.1)
    return d


def _boxes(case, seed):
    """Floor-standing boxes of 10 to 40 m footprint and 10 to 60 m height on 2 m cells, as many per area as 40 on
    512 m x 512 m: (i0, i1, j0, j1, k1) in cell units, real numbers."""
    rng = np.random.default_rng(77000 + int(seed))
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    out = []
    for _ in range(max(2, round(40 * nx * ny / 65536))):
        cx, cy = rng.uniform(0, nx), rng.uniform(0, ny)
        wx, wy, h = rng.uniform(5, 20), rng.uniform(5, 20), rng.uniform(5, 30)
        wx, wy, h = min(wx, 0.4 * nx), min(wy, 0.4 * ny), min(h, 0.6 * nz)
        out.append((cx - wx / 2, cx + wx / 2, cy - wy / 2, cy + wy / 2, h))
    return out


def _staircase(case, seed):
    """0/1 apertures of the cells whose centre lies in a box (periodic in x and y), and the fluid mask."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    solid = np.zeros((nz, ny, nx), bool)
    x, y, z = np.arange(nx) + 0.5, np.arange(ny) + 0.5, np.arange(nz) + 0.5
    for i0, i1, j0, j1, h in _boxes(case, seed):
        inx = ((x - i0) % nx) < i1 - i0
        iny = ((y - j0) % ny) < j1 - j0
        solid |= (z < h)[:, None, None] & iny[None, :, None] & inx[None, None, :]
    open_ = (~solid).astype(np.float64)
    ax, ay, az = np.ones((nz, ny, nx + 1)), np.ones((nz, ny + 1, nx)), np.zeros((nz + 1, ny, nx))
    ax[:, :, :nx] = open_ * np.roll(open_, 1, axis=2)
    ax[:, :, nx] = ax[:, :, 0]
    ay[:, :ny, :] = open_ * np.roll(open_, 1, axis=1)
    ay[:, ny, :] = ay[:, 0, :]
    az[1:nz] = open_[1:] * open_[:-1]
    return (ax, ay, az), ~solid


def _fractions(case, seed):
    """Face apertures of the boxes with their sides cutting through cells (multiples of 1/16, as a 4 x 4 sampling of
    each face gives), and the mask of the cells that hold fluid."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]

    def samples(n, face):
        base = np.arange(n, dtype=np.float64)
        return base[:, None] + (np.zeros(1) if face else (np.arange(4) + 0.5) / 4)[None, :]

    def covered(fx, fy, fz):
        xs, ys, zs = samples(nx, fx), samples(ny, fy), samples(nz, fz)
        hit = np.zeros((nz, zs.shape[1], ny, ys.shape[1], nx, xs.shape[1]), bool)
        for i0, i1, j0, j1, h in _boxes(case, seed):
            inx, iny, inz = ((xs - i0) % nx) < i1 - i0, ((ys - j0) % ny) < j1 - j0, zs < h
            i, j, k = np.flatnonzero(inx.any(1)), np.flatnonzero(iny.any(1)), np.flatnonzero(inz.any(1))
            block = inz[k][:, :, None, None, None, None] & iny[j][None, None, :, :, None, None] & inx[i][None, None, None, None, :, :]
            hit[np.ix_(k, range(zs.shape[1]), j, range(ys.shape[1]), i, range(xs.shape[1]))] |= block
        return 1.0 - hit.mean(axis=(1, 3, 5))

    ax, ay, az = np.ones((nz, ny, nx + 1)), np.ones((nz, ny + 1, nx)), np.zeros((nz + 1, ny, nx))
    ax[:, :, :nx] = covered(True, False, False)
    ax[:, :, nx] = ax[:, :, 0]
    ay[:, :ny, :] = covered(False, True, False)
    ay[:, ny, :] = ay[:, 0, :]
    az[1:nz] = covered(False, False, True)[1:]
    # a cell whose six faces are all closed holds no fluid
    fluid = (ax[:, :, :-1] + ax[:, :, 1:] + ay[:, :-1, :] + ay[:, 1:, :] + az[:-1] + az[1:]) > 0
    return (ax, ay, az), fluid


def _initial(case, seed):
    """The interior state at the start of a run, (u, v, w, theta) in 64 bits on the device, before its projection."""
    d = _layout(case)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    shape, dev = (nz, ny, nx), _device()
    gens = [_generator(seed, s) for s in range(4)]
    flow = case["flow"]
    if flow == "tgv":
        lx, ly, lz = d["extent"]
        k = 2 * math.pi
        x = torch.arange(nx, device=dev, dtype=F64) / nx * k
        y = torch.arange(ny, device=dev, dtype=F64) / ny * k
        z = (torch.arange(nz, device=dev, dtype=F64) + 0.5) / nz * k
        xc, yc = x + math.pi / nx, y + math.pi / ny
        u = torch.sin(x)[None, None, :] * torch.cos(yc)[None, :, None] * torch.cos(z)[:, None, None]
        v = -torch.cos(xc)[None, None, :] * torch.sin(y)[None, :, None] * torch.cos(z)[:, None, None]
        return (u + _uniform(shape, gens[0], 1e-3), v + _uniform(shape, gens[1], 1e-3),
                _uniform(shape, gens[2], 1e-3), _uniform(shape, gens[3], 1.0))
    if flow in ("hit", "dns"):
        return tuple(_spectral_noise(shape, g) for g in gens)
    if flow == "cbl":
        # thermals of about 1 m/s below the inversion at 1 km, and the mixed-layer profile with +-0.1 K noise
        zf = torch.as_tensor(d["zf"], device=dev)
        zc = 0.5 * (zf[1:] + zf[:-1])
        env = torch.exp(-((zc - 500.0) / 500.0) ** 2)[:, None, None]
        u, v, w = (env * _spectral_noise(shape, g) for g in gens[:3])
        prof = torch.where(zc < 1000.0, 300.0 + 0 * zc, 303.0 + 3e-3 * (zc - 1000.0))
        return u, v, w, prof[:, None, None] + env * _uniform(shape, gens[3], 0.1)
    # urban: the log-profile wind with 0.5 m/s of turbulence, 300 K with +-0.1 K noise
    z = 2.0 * (torch.arange(nz, device=dev, dtype=F64) + 0.5)
    wind = 5.0 * torch.log(z / 0.1) / math.log(10.0 / 0.1)
    u, v, w = (0.5 * _spectral_noise(shape, g, 8.0) for g in gens[:3])
    return wind[:, None, None] + u, v, w, 300.0 + _uniform(shape, gens[3], 0.1)


def _solve_inputs(case, seed):
    """Face coefficients a^2, the right-hand side (the aperture divergence of a noisy log-profile wind: it vanishes in
    the solid and sums to zero) and the fluid mask."""
    (ax, ay, az), fluid = _fractions(case, seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dev = _device()
    gens = [_generator(seed, s) for s in range(3)]
    z = 2.0 * (torch.arange(nz, device=dev, dtype=F64) + 0.5)
    wind = (5.0 * torch.log(z / 0.1) / math.log(10.0 / 0.1))[:, None, None]
    u = wind + _uniform((nz, ny, nx), gens[0], 0.5)
    v = _uniform((nz, ny, nx), gens[1], 0.5)
    w = _uniform((nz, ny, nx), gens[2], 0.5)
    b = _aperture_divergence(u, v, w, [torch.as_tensor(a, device=dev) for a in (ax, ay, az)], (2.0, 2.0, 2.0))
    return (ax, ay, az), b, fluid


def _tracer_inputs(case, seed):
    """Padded u, v, w, phi: a divergent noisy wind at a first-order CFL of 0.9 and a non-negative field with empty
    regions, where the limiter acts."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    shape = (nz, ny, nx)
    gens = [_generator(seed, s) for s in range(5)]
    vel = [torch.randn(shape, generator=g, device=_device(), dtype=F64) for g in gens[:3]]
    if case["bc_z"] == "wall":
        vel[2][0] = 0
    rate = sum(float(a.abs().max()) * n for a, n in zip(vel, (nx, ny, nz)))
    vel = [a * (0.9 / rate) for a in vel]
    phi = 1.5 + 0.5 * _spectral_noise(shape, gens[3])
    phi = phi.clamp_min(0.0)
    phi = torch.where(torch.rand(shape, generator=gens[4], device=_device()) < 0.15, 0.0 * phi, phi)
    phi[:, :, : nx // 8] = 0
    wall = case["bc_z"] == "wall"
    return [_pad(vel[0], wall, "c"), _pad(vel[1], wall, "c"), _pad(vel[2], wall, "fz"), _pad(phi, wall, "c")]


def _unet_inputs(case, seed):
    """Random residuals and errors on the fluid, the mask of the boxes, and He-normal weights."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    _, fluid = _staircase(case, seed)
    rng = np.random.default_rng(int(seed))
    gens = [_generator(seed, s) for s in range(2)]
    mask = torch.as_tensor(fluid, device=_device())
    r = torch.randn((nz, ny, nx), generator=gens[0], device=_device(), dtype=F64) * mask
    e = _spectral_noise((nz, ny, nx), gens[1]) * mask
    params = []
    for name, ci, co in UNET_LAYERS:
        w = rng.standard_normal((27, co, ci)) * math.sqrt(2.0 / (27 * ci)) * (0.1 if name == "out" else 1.0)
        if name == "e1a":
            w[:, :, 2:] = 0.0
        if name == "out":
            w[:, 1:, :] = 0.0
        params += [w.ravel(), np.zeros(co)]
    return r.cpu().numpy(), e.cpu().numpy(), fluid.astype(np.float32), np.concatenate(params).astype(np.float32)


# ---- prepare and run: the framework ------------------------------------------------
def _embed(grid, interior, dtype):
    out = torch.zeros(grid.storage_shape, dtype=dtype, pin_memory=True)
    out.numpy()[grid.interior] = interior.to(dtype).cpu().numpy()
    return out.numpy()


def _simulation(case, seed):
    from aeolus_b200 import CoreSpec, regular_grid, stretched_grid
    from aeolus_b200.reference_state import anelastic_profiles
    from aeolus_b200.simulation import CFLConstraints, Simulation
    d = _layout(case)
    size = (case["nx"], case["ny"], case["nz"])
    if d["zf"] is not None:
        g = stretched_grid(size, d["extent"], d["zf"])
    else:
        g = regular_grid(size, d["extent"], bc_z=d["bc_z"])
    kw = {"advection": d["advection"], "nu": d["nu"], "c_s": d["c_s"], "theta0": d["theta0"], "g": d["g"],
          "flux_bot": d["flux_bot"], "precision": case["precision"]}
    if d["core"] == "anelastic":
        rho, theta = _profiles(d)
        prof = anelastic_profiles(g, rho, theta)
        kw.update(core="anelastic", wc=prof["wc"], wf=prof["wf"], thf=prof["thf"])
    if case["flow"] == "urban":
        kw.update(solver="pcg")
    sim = Simulation(CoreSpec(grid=g, **kw))
    if case["flow"] == "urban":
        sim.set_pcg(_staircase(case, seed)[0], tol=1e-8, maxit=200)
    single = case["precision"] != "fp64"
    dtype = torch.float32 if single else F64
    for name, f in zip(FIELDS, _initial(case, seed)):
        (sim.set_field_f32 if single else sim.set_field)(name, _embed(g, f, dtype))
    sim.project()
    # the pressure of the cut-cell step is defined up to a constant in each pocket of fluid: not read
    names = FIELDS[:4] if case["flow"] == "urban" else FIELDS
    out = {n: torch.empty(g.storage_shape, dtype=dtype, pin_memory=True).numpy() for n in names}
    c = CFLConstraints(C_advective=0.5, growth_max=1.1, divergence_tol=1e-2) if d["adaptive"] else None
    return {"kind": "step", "sim": sim, "out": out, "single": single, "steps": case["steps"], "dt": d.get("dt"),
            "constraints": c, "interior": g.interior}


def prepare(case, seed):
    if case["kind"] == "step":
        return _simulation(case, seed)
    if case["kind"] == "solve":
        from aeolus_b200.multigrid import MGPreconditionedCG
        a, b, fluid = _solve_inputs(case, seed)
        s = MGPreconditionedCG((case["nx"], case["ny"], case["nz"]), (2.0, 2.0, 2.0), coeffs=[x * x for x in a],
                               tol=1e-8, precision=case["precision"])
        m = torch.as_tensor(fluid, device=b.device).to(F64)
        return {"kind": "solve", "solver": s, "b": b.contiguous(), "x": torch.empty_like(b), "fluid": m,
                "nfluid": float(m.sum())}
    if case["kind"] == "tracer":
        from aeolus_b200 import CoreSpec, regular_grid
        from aeolus_b200.simulation import Simulation
        g = regular_grid((case["nx"], case["ny"], case["nz"]), (1.0, 1.0, 1.0), bc_z=case["bc_z"])
        sim = Simulation(CoreSpec(grid=g, advection=case["scheme"], precision=case["precision"]))
        dtype = F64 if case["precision"] == "fp64" else torch.float32
        arrays = [a.to(dtype).contiguous() for a in _tracer_inputs(case, seed)]
        return {"kind": "tracer", "sim": sim, "arrays": arrays, "tend": torch.zeros_like(arrays[0]),
                "scheme": case["scheme"]}
    from aeolus_b200.unet import UNet
    r, e, fluid, params = _unet_inputs(case, seed)
    net = UNet((case["nx"], case["ny"], case["nz"]))
    net.set_params(params)
    net.set_mask(fluid)
    net.set_out_scale(3.0)
    return {"kind": case["kind"], "net": net, "r": r, "e": e}


def run(state):
    if state["kind"] == "step":
        sim = state["sim"]
        if state["constraints"] is not None:
            sim.step_adaptive(state["constraints"], state["steps"])
        else:
            sim.step_rk3(state["dt"], state["steps"])
        for name, out in state["out"].items():
            (sim.get_field_f32 if state["single"] else sim.get_field)(name, out)
        return {name: out[state["interior"]] for name, out in state["out"].items()}
    if state["kind"] == "solve":
        state["solver"].solve_device(state["b"].data_ptr(), state["x"].data_ptr())
        # the solution is defined up to a constant and not in the solid: as its user takes it, relative to the
        # fluid's mean
        x, m = state["x"], state["fluid"]
        return (x - (x * m).sum() / state["nfluid"]) * m
    if state["kind"] == "tracer":
        state["sim"].advect_positive_device(*state["arrays"], state["tend"], 1.0, state["scheme"], accumulate=False)
        return state["tend"]
    if state["kind"] == "unet_apply":
        return state["net"].apply(state["r"])
    loss = state["net"].gradients(state["r"], state["e"])
    return {"loss": loss, "grads": state["net"].grads()}


# ---- the same in plain torch, 64 bits -------------------------------------------------
def _profiles(d):
    zc = 0.5 * (d["zf"][1:] + d["zf"][:-1])
    return 1.2 * np.exp(-zc / 8000.0), np.where(zc < 1000.0, 300.0, 303.0 + 3e-3 * (zc - 1000.0))


def _pad(f, wall, loc):
    """f with three halo layers: periodic in x and y, and in z periodic, mirrored, or (bottom faces) odd about the
    zero wall faces."""
    f = torch.cat([f[:, :, -3:], f, f[:, :, :3]], 2)
    f = torch.cat([f[:, -3:], f, f[:, :3]], 1)
    if not wall:
        return torch.cat([f[-3:], f, f[:3]], 0)
    if loc != "fz":
        return torch.cat([f[:3].flip(0), f, f[-3:].flip(0)], 0)
    zero = torch.zeros_like(f[:1])
    return torch.cat([-f[1:4].flip(0), zero, f[1:], zero, -f[-2:].flip(0)], 0)


class _At:
    """Neighbours of every interior point of a padded array; `more` adds a layer at the high end of one axis."""

    def __init__(self, padded, more=(0, 0, 0)):
        self.f = padded
        self.n = [padded.shape[2 - a] - 6 + more[a] for a in range(3)]

    def __call__(self, di, dj, dk):
        (nx, ny, nz) = self.n
        return self.f[3 + dk:3 + dk + nz, 3 + dj:3 + dj + ny, 3 + di:3 + di + nx]


def _weno(scheme, vel, f):
    """The upwinded fifth-order face value from the six cells around a face."""
    pos = vel >= 0
    v1, v2, v3, v4, v5 = (torch.where(pos, f[a], f[5 - a]) for a in range(5))
    q0 = (2 * v1 - 7 * v2 + 11 * v3) / 6
    q1 = (-v2 + 5 * v3 + 2 * v4) / 6
    q2 = (2 * v3 + 5 * v4 - v5) / 6
    b0 = ((v1 - 4 * v2 + 3 * v3) / 2) ** 2 + 13.0 / 3.0 * ((v1 - 2 * v2 + v3) / 2) ** 2
    b1 = ((v4 - v2) / 2) ** 2 + 13.0 / 3.0 * ((v2 - 2 * v3 + v4) / 2) ** 2
    b2 = ((-3 * v3 + 4 * v4 - v5) / 2) ** 2 + 13.0 / 3.0 * ((v3 - 2 * v4 + v5) / 2) ** 2
    if scheme == "weno_z5":
        eps, tau = 2.0 ** -104, (b0 - b2).abs()
        a0, a1, a2 = (c * (1 + (tau / (b + eps)) ** 2) for c, b in ((0.1, b0), (0.6, b1), (0.3, b2)))
    else:
        a0, a1, a2 = (c / (b + 1e-6) ** 2 for c, b in ((0.1, b0), (0.6, b1), (0.3, b2)))
    return (a0 * q0 + a1 * q1 + a2 * q2) / (a0 + a1 + a2)


def _face(scheme, F, axis, vel):
    step = [tuple(c if a == axis else 0 for a in range(3)) for c in range(-3, 3)]
    return _weno(scheme, vel, [F(*s) for s in step])


def _low(axis):
    return tuple(-1 if a == axis else 0 for a in range(3))


class _Flow:
    """The projected RK3 step of one case in plain torch."""

    def __init__(self, case, seed):
        self.case, self.d = case, _layout(case)
        d, dev = self.d, _device()
        self.n = (case["nx"], case["ny"], case["nz"])
        self.wall = d["bc_z"] == "wall"
        self.dx, self.dy = d["extent"][0] / self.n[0], d["extent"][1] / self.n[1]
        nz = self.n[2]
        dz = np.full(nz, d["extent"][2] / nz) if d["zf"] is None else np.diff(d["zf"])
        e = np.concatenate([[dz[0]], dz, [dz[-1]]])          # one ghost level each way
        self.dzmin = dz.min()

        def col(a):
            return torch.as_tensor(np.ascontiguousarray(a), device=dev, dtype=F64)[:, None, None]

        self.dz, self.dzf_np = dz, 0.5 * (e[1:] + e[:-1])    # nz + 1 face distances
        self.idz, self.idz_lo = col(1 / dz), col(1 / e[:-2])
        self.idzf, self.idzf_up = col(1 / self.dzf_np[:-1]), col(1 / self.dzf_np[1:])
        self.idz_off = col(2 / (self.dzf_np[:-1] + self.dzf_np[1:]))
        s = e[:-2] + e[1:-1]
        # centre -> face interpolation, and the area weighting of a w volume's side faces
        self.wlo, self.whi = col(e[1:-1] / s), col(e[:-2] / s)
        self.alo, self.ahi = col(e[:-2] / s), col(e[1:-1] / s)
        self.filter = col((self.dx * self.dy * dz) ** (1.0 / 3.0))
        self.anel = d["core"] == "anelastic"
        wc, wf, th = np.ones(nz), np.ones(nz + 1), np.zeros(nz)
        if self.anel:
            rho, theta = _profiles(d)
            a, b = rho[:-1], rho[1:]
            x = (a - b) / (a + b)
            # the logarithmic mean, by its series where the two are close
            lm = np.where(np.abs(x) < 1e-3, (a + b) / 2 * (1 - x * x / 3 - 4 * x ** 4 / 45), (a - b) / np.log(a / b))
            wc, wf = rho, np.concatenate([rho[:1], lm, rho[-1:]])
            wlo = dz[1:] / (dz[:-1] + dz[1:])
            th = np.concatenate([theta[:1], wlo * theta[:-1] + (1 - wlo) * theta[1:]])
        self.wc_np, self.wf_np = wc, wf
        self.wc, self.wc_lo = col(wc), col(np.concatenate([wc[:1] * wc[:1] / wc[1:2], wc[:-1]]))
        self.wfb, self.wft, self.thf = col(wf[:-1]), col(wf[1:]), col(th)
        self.masks = None
        if case["flow"] == "urban":
            self.ap = [torch.as_tensor(a, device=dev) for a in _staircase(case, seed)[0]]
        elif self.wall:
            self._columns(dev)
        self.state = list(_initial(case, seed))
        if self.wall:
            self.state[2][0] = 0
        self.p = None

    # the direct solvers
    def _columns(self, dev):
        nx, ny, nz = self.n
        lo = np.concatenate([[0.0], self.wf_np[1:-1] / (self.dz[1:] * self.dzf_np[1:-1])])
        up = np.concatenate([self.wf_np[1:-1] / (self.dz[:-1] * self.dzf_np[1:-1]), [0.0]])
        kx = 4 / self.dx ** 2 * torch.sin(math.pi * torch.arange(nx // 2 + 1, device=dev, dtype=F64) / nx) ** 2
        ky = 4 / self.dy ** 2 * torch.sin(math.pi * torch.arange(ny, device=dev, dtype=F64) / ny) ** 2
        lam = kx[None, :] + ky[:, None]
        lam[0, 0] = 1.0                                       # the mean mode is integrated instead
        self.lo, self.inv, self.cp = lo, [], []
        cp = torch.zeros_like(lam)
        for k in range(nz):
            den = -(lo[k] + up[k]) - lam * self.wc_np[k] - lo[k] * cp
            cp = up[k] / den
            self.inv.append(1 / den)
            self.cp.append(cp)

    def _solve(self, src):
        nx, ny, nz = self.n
        if not self.wall:
            S = torch.fft.rfftn(src)
            dev = src.device
            k = [4 / h ** 2 * torch.sin(math.pi * torch.arange(m, device=dev, dtype=F64) / n) ** 2
                 for h, m, n in ((self.dx, nx // 2 + 1, nx), (self.dy, ny, ny), (self.dz[0], nz, nz))]
            lam = -(k[0][None, None, :] + k[1][None, :, None] + k[2][:, None, None])
            lam[0, 0, 0] = 1.0
            S /= lam
            S[0, 0, 0] = 0
            return torch.fft.irfftn(S, s=src.shape)
        S = torch.fft.rfft2(src)
        mean = S[:, 0, 0].real.cpu().numpy()
        S[0] *= self.inv[0]
        for k in range(1, nz):
            S[k] = (S[k] - self.lo[k] * S[k - 1]) * self.inv[k]
        for k in range(nz - 2, -1, -1):
            S[k] -= self.cp[k] * S[k + 1]
        r = mean - (mean * self.dz).sum() / self.dz.sum()
        flux = np.cumsum(r * self.dz)
        col = np.concatenate([[0.0], np.cumsum(flux[:-1] * self.dzf_np[1:-1] / self.wf_np[1:-1])])
        col -= (col * self.dz).sum() / self.dz.sum()
        S[:, 0, 0] = torch.as_tensor(col, device=S.device).to(S.dtype)
        return torch.fft.irfft2(S, s=src.shape[1:])

    # one substage
    def _tendencies(self):
        d, P = self.d, [_pad(f, self.wall, loc) for f, loc in zip(self.state, ("c", "c", "fz", "c"))]
        U, V, W, T = (_At(p) for p in P)
        ix, iy = 1 / self.dx, 1 / self.dy
        iz, izf = self.idz, self.idzf
        h = 0.5
        if d["advection"] != "centred":
            t = []
            for f in range(4):
                s = 0
                for axis, i in ((0, ix), (1, iy), (2, iz)):
                    more = tuple(1 if a == axis else 0 for a in range(3))
                    A, F = _At(P[axis], more), _At(P[f], more)
                    vel = A(0, 0, 0) if f == 3 else (A(*_low(f)) + A(0, 0, 0)) / 2
                    flux = vel * _face(d["advection"], F, axis, vel)
                    s = s + torch.diff(flux, dim=2 - axis) * i
                t.append(-s)
        else:
            iwc, iwf = 1 / self.wc, 1 / self.wfb
            wft, wfb, wct, wcb = self.wft, self.wfb, self.wc, self.wc_lo

            def side(A, *at):
                lo, hi = A(at[0], at[1], -1), A(at[0], at[1], 0)
                return self.alo * lo + self.ahi * hi

            tu = -(((h * (U(0, 0, 0) + U(1, 0, 0))) ** 2 - (h * (U(-1, 0, 0) + U(0, 0, 0))) ** 2) * ix
                   + (h * (V(-1, 1, 0) + V(0, 1, 0)) * h * (U(0, 0, 0) + U(0, 1, 0))
                      - h * (V(-1, 0, 0) + V(0, 0, 0)) * h * (U(0, -1, 0) + U(0, 0, 0))) * iy
                   + (wft * h * (W(-1, 0, 1) + W(0, 0, 1)) * h * (U(0, 0, 0) + U(0, 0, 1))
                      - wfb * h * (W(-1, 0, 0) + W(0, 0, 0)) * h * (U(0, 0, -1) + U(0, 0, 0))) * iz * iwc)
            tv = -((h * (U(1, -1, 0) + U(1, 0, 0)) * h * (V(0, 0, 0) + V(1, 0, 0))
                    - h * (U(0, -1, 0) + U(0, 0, 0)) * h * (V(-1, 0, 0) + V(0, 0, 0))) * ix
                   + ((h * (V(0, 0, 0) + V(0, 1, 0))) ** 2 - (h * (V(0, -1, 0) + V(0, 0, 0))) ** 2) * iy
                   + (wft * h * (W(0, -1, 1) + W(0, 0, 1)) * h * (V(0, 0, 0) + V(0, 0, 1))
                      - wfb * h * (W(0, -1, 0) + W(0, 0, 0)) * h * (V(0, 0, -1) + V(0, 0, 0))) * iz * iwc)
            tw = -((side(U, 1, 0) * h * (W(0, 0, 0) + W(1, 0, 0)) - side(U, 0, 0) * h * (W(-1, 0, 0) + W(0, 0, 0))) * ix
                   + (side(V, 0, 1) * h * (W(0, 0, 0) + W(0, 1, 0)) - side(V, 0, 0) * h * (W(0, -1, 0) + W(0, 0, 0))) * iy
                   + (wct * (h * (W(0, 0, 0) + W(0, 0, 1))) ** 2 - wcb * (h * (W(0, 0, -1) + W(0, 0, 0))) ** 2) * izf * iwf)
            tt = -((U(1, 0, 0) * h * (T(0, 0, 0) + T(1, 0, 0)) - U(0, 0, 0) * h * (T(-1, 0, 0) + T(0, 0, 0))) * ix
                   + (V(0, 1, 0) * h * (T(0, 0, 0) + T(0, 1, 0)) - V(0, 0, 0) * h * (T(0, -1, 0) + T(0, 0, 0))) * iy
                   + (wft * W(0, 0, 1) * h * (T(0, 0, 0) + T(0, 0, 1))
                      - wfb * W(0, 0, 0) * h * (T(0, 0, -1) + T(0, 0, 0))) * iz * iwc)
            t = [tu, tv, tw, tt]
        if d["nu"]:
            for f, A in enumerate((U, V, W, T)):
                c2 = 2 * A(0, 0, 0)
                t[f] = t[f] + d["nu"] * ((A(1, 0, 0) - c2 + A(-1, 0, 0)) * ix ** 2 + (A(0, 1, 0) - c2 + A(0, -1, 0)) * iy ** 2
                                         + (A(0, 0, 1) - c2 + A(0, 0, -1)) * iz ** 2)
        if d["c_s"]:
            self._eddy(t, U, V, W, T)
        if self.anel or d["theta0"]:
            face = self.wlo * T(0, 0, -1) + self.whi * T(0, 0, 0)
            ref = self.thf if self.anel else d["theta0"]
            t[2] = t[2] + d["g"] / ref * (face - ref)
        t[3][0] += d["flux_bot"] / self.dz[0]
        return t

    def _eddy(self, t, U, V, W, T):
        d, ix, iy, iz, izf, izu = self.d, 1 / self.dx, 1 / self.dy, self.idz, self.idzf, self.idzf_up
        ux, vy, wz = (U(1, 0, 0) - U(0, 0, 0)) * ix, (V(0, 1, 0) - V(0, 0, 0)) * iy, (W(0, 0, 1) - W(0, 0, 0)) * iz

        def mid(A, a, b, i):     # the centred gradient along b at the cell centre of a component staggered along a
            s = [tuple(1 if q == a else 0 for q in range(3)), tuple(1 if q == b else 0 for q in range(3))]
            hi = A(*s[1]) + A(*(s[0][q] + s[1][q] for q in range(3)))
            lo = A(*(-s[1][q] for q in range(3))) + A(*(s[0][q] - s[1][q] for q in range(3)))
            return (hi - lo) * (0.25 * i)

        s12 = 0.5 * (mid(U, 0, 1, iy) + mid(V, 1, 0, ix))
        s13 = 0.5 * (mid(U, 0, 2, self.idz_off) + mid(W, 2, 0, ix))
        s23 = 0.5 * (mid(V, 1, 2, self.idz_off) + mid(W, 2, 1, iy))
        S2 = 2 * (ux ** 2 + vy ** 2 + wz ** 2) + 4 * (s12 ** 2 + s13 ** 2 + s23 ** 2)
        N = _At(_pad((d["c_s"] * self.filter) ** 2 * S2.sqrt(), self.wall, "c"))
        q = 0.25
        edge_z = (self.wft / self.wc, self.wfb / self.wc) if self.anel else (1.0, 1.0)

        def grad(A, *hi_lo):
            return A(*hi_lo[0]) - A(*hi_lo[1])

        o, x1, y1, z1, xm, ym, zm = (0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (-1, 0, 0), (0, -1, 0), (0, 0, -1)
        vert = (edge_z[0] * q * (N(-1, 0, 0) + N(0, 0, 0) + N(-1, 0, 1) + N(0, 0, 1)) * grad(U, z1, o) * izu
                - edge_z[1] * q * (N(-1, 0, -1) + N(0, 0, -1) + N(-1, 0, 0) + N(0, 0, 0)) * grad(U, o, zm) * izf) * iz
        t[0] = t[0] + (N(0, 0, 0) * grad(U, x1, o) - N(-1, 0, 0) * grad(U, o, xm)) * ix ** 2 + vert + (
            q * (N(-1, 0, 0) + N(0, 0, 0) + N(-1, 1, 0) + N(0, 1, 0)) * grad(U, y1, o)
            - q * (N(-1, -1, 0) + N(0, -1, 0) + N(-1, 0, 0) + N(0, 0, 0)) * grad(U, o, ym)) * iy ** 2
        vert = (edge_z[0] * q * (N(0, -1, 0) + N(0, 0, 0) + N(0, -1, 1) + N(0, 0, 1)) * grad(V, z1, o) * izu
                - edge_z[1] * q * (N(0, -1, -1) + N(0, 0, -1) + N(0, -1, 0) + N(0, 0, 0)) * grad(V, o, zm) * izf) * iz
        t[1] = t[1] + (N(0, 0, 0) * grad(V, y1, o) - N(0, -1, 0) * grad(V, o, ym)) * iy ** 2 + vert + (
            q * (N(0, -1, 0) + N(1, -1, 0) + N(0, 0, 0) + N(1, 0, 0)) * grad(V, x1, o)
            - q * (N(-1, -1, 0) + N(0, -1, 0) + N(-1, 0, 0) + N(0, 0, 0)) * grad(V, o, xm)) * ix ** 2
        we = (self.wc / self.wfb, self.wc_lo / self.wfb) if self.anel else (1.0, 1.0)
        t[2] = t[2] + (we[0] * N(0, 0, 0) * grad(W, z1, o) * iz - we[1] * N(0, 0, -1) * grad(W, o, zm) * self.idz_lo) * izf + (
            q * (N(0, 0, -1) + N(1, 0, -1) + N(0, 0, 0) + N(1, 0, 0)) * grad(W, x1, o)
            - q * (N(-1, 0, -1) + N(0, 0, -1) + N(-1, 0, 0) + N(0, 0, 0)) * grad(W, o, xm)) * ix ** 2 + (
            q * (N(0, 0, -1) + N(0, 1, -1) + N(0, 0, 0) + N(0, 1, 0)) * grad(W, y1, o)
            - q * (N(0, -1, -1) + N(0, 0, -1) + N(0, -1, 0) + N(0, 0, 0)) * grad(W, o, ym)) * iy ** 2
        k = 0.5 / d["pr_t"]
        t[3] = t[3] + k * (
            ((N(0, 0, 0) + N(1, 0, 0)) * grad(T, x1, o) - (N(-1, 0, 0) + N(0, 0, 0)) * grad(T, o, xm)) * ix ** 2
            + ((N(0, 0, 0) + N(0, 1, 0)) * grad(T, y1, o) - (N(0, -1, 0) + N(0, 0, 0)) * grad(T, o, ym)) * iy ** 2
            + (edge_z[0] * (N(0, 0, 0) + N(0, 0, 1)) * grad(T, z1, o) * izu
               - edge_z[1] * (N(0, 0, -1) + N(0, 0, 0)) * grad(T, o, zm) * izf) * iz)

    def _project(self, vel):
        """(corrected velocity, phi)"""
        u, v, w = vel
        if self.case["flow"] == "urban":
            h = (self.dx, self.dy, self.dz[0])
            b = _aperture_divergence(u, v, w, self.ap, h)
            phi = -_masked_poisson(b, [a * a for a in self.ap], h)
        else:
            wt = torch.cat([w[1:], torch.zeros_like(w[:1]) if self.wall else w[:1]])
            b = self.wc * ((u.roll(-1, 2) - u) / self.dx + (v.roll(-1, 1) - v) / self.dy) + (self.wft * wt - self.wfb * w) * self.idz
            phi = self._solve(b)
        down = torch.cat([phi[:1] if self.wall else phi[-1:], phi[:-1]])
        g = [(phi - phi.roll(1, 2)) / self.dx, (phi - phi.roll(1, 1)) / self.dy, (phi - down) * self.idzf]
        if self.case["flow"] == "urban":
            a = (self.ap[0][:, :, :-1], self.ap[1][:, :-1], self.ap[2][:-1])
            return [torch.where(q > 0, s - q * r, 0.0 * s) for q, s, r in zip(a, vel, g)], phi
        return [s - r for s, r in zip(vel, g)], phi

    def project(self):
        self.state[:3], _ = self._project(self.state[:3])

    def step(self, dt):
        start = list(self.state)
        for a, b in ((0.0, 1.0), (0.75, 0.25), (1.0 / 3.0, 2.0 / 3.0)):
            t = self._tendencies()
            new = [f + dt * s for f, s in zip(self.state, t)]
            if self.wall:
                new[2][0] = 0
            new[:3], phi = self._project(new[:3])
            self.state = new if a == 0 else [a * x + b * y for x, y in zip(start, new)]
            self.p = phi / dt

    def pick(self, previous):
        u, v, w = self.state[:3]
        rate = sum(torch.maximum(f.abs(), f.roll(-1, a).abs()) / h for f, a, h in ((u, 2, self.dx), (v, 1, self.dy), (w, 0, self.dz[0])))
        dt = 0.5 / float(rate.max())
        return dt if previous is None else min(dt, 1.1 * previous)


def _aperture_divergence(u, v, w, ap, h):
    fx = ap[0] * torch.cat([u, u[:, :, :1]], 2)
    fy = ap[1] * torch.cat([v, v[:, :1]], 1)
    fz = ap[2] * torch.cat([w, w[:1]], 0)
    return torch.diff(fx, dim=2) / h[0] + torch.diff(fy, dim=1) / h[1] + torch.diff(fz, dim=0) / h[2]


def _masked_poisson(b, c, h, tol=1e-13, most=400):
    """x with -div(c grad x) = b on the cells that a face is open to (0 elsewhere, zero mean): CG preconditioned by
    the open box's Poisson problem in the eigenvectors of its axes."""
    nz, ny, nx = b.shape
    dev = b.device
    diag = (c[0][:, :, :-1] + c[0][:, :, 1:]) / h[0] ** 2 + (c[1][:, :-1] + c[1][:, 1:]) / h[1] ** 2 + (c[2][:-1] + c[2][1:]) / h[2] ** 2
    m = (diag > 0).to(F64)
    count = m.sum()

    def apply(x):
        gx = c[0] * torch.cat([x[:, :, :1] - x[:, :, -1:], torch.diff(x, dim=2), x[:, :, :1] - x[:, :, -1:]], 2) / h[0] ** 2
        gy = c[1] * torch.cat([x[:, :1] - x[:, -1:], torch.diff(x, dim=1), x[:, :1] - x[:, -1:]], 1) / h[1] ** 2
        gz = c[2] * torch.cat([torch.zeros_like(x[:1]), torch.diff(x, dim=0), torch.zeros_like(x[:1])], 0) / h[2] ** 2
        return -(torch.diff(gx, dim=2) + torch.diff(gy, dim=1) + torch.diff(gz, dim=0))

    k = [4 / q ** 2 * torch.sin(math.pi * torch.arange(mm, device=dev, dtype=F64) / n) ** 2
         for q, mm, n in ((h[0], nx // 2 + 1, nx), (h[1], ny, ny), (h[2], 2 * nz, 2 * nz))]
    lam = k[0][None, None, :] + k[1][None, :, None] + k[2][:, None, None]
    lam[0, 0, 0] = 1.0

    def precondition(r):
        S = torch.fft.rfftn(torch.cat([r, r.flip(0)])) / lam
        S[0, 0, 0] = 0
        z = torch.fft.irfftn(S, s=(2 * nz, ny, nx))[:nz] * m
        return z - (z.sum() / count) * m

    r = (b - ((b * m).sum() / count)) * m
    x, p, rz, norm = torch.zeros_like(b), None, None, float(r.norm())
    best = float("inf")
    for it in range(most):
        z = precondition(r)
        new = (r * z).sum()
        p = z if p is None else z + (new / rz) * p
        rz = new
        q = apply(p)
        a = rz / (p * q).sum()
        x = x + a * p
        r = r - a * q
        now = float(r.norm())
        if now <= tol * norm or (it > 60 and now > 0.9 * best and now < 1e-12 * norm):
            break
        best = min(best, now)
    return (x - (x * m).sum() / count) * m


def _exact_step(case, seed):
    n = case["nx"] * case["ny"] * case["nz"]
    if n > 20_000_000:
        return None
    flow = _Flow(case, seed)
    flow.project()
    dt = None
    for _ in range(case["steps"]):
        dt = flow.pick(dt) if flow.d["adaptive"] else flow.d["dt"]
        flow.step(dt)
    out = dict(zip(FIELDS, flow.state))
    if case["flow"] != "urban":
        out["p"] = flow.p
    return out


def _exact_tracer(case, seed):
    P = _tracer_inputs(case, seed)
    if case["precision"] != "fp64":
        P = [p.float().double() for p in P]
    n = (case["nx"], case["ny"], case["nz"])
    phi = P[3]
    flux, low = [], []
    for axis in range(3):
        more = tuple(1 if a == axis else 0 for a in range(3))
        vel, F = _At(P[axis], more)(0, 0, 0), _At(phi, more)
        flux.append(vel * _face(case["scheme"], F, axis, vel))
        low.append(vel * torch.where(vel >= 0, F(*_low(axis)), F(0, 0, 0)))
    anti = [f - g for f, g in zip(flux, low)]

    def ends(f, axis):
        return f.narrow(2 - axis, 0, n[axis]), f.narrow(2 - axis, 1, n[axis])

    out = sum((ends(a, i)[1].clamp_min(0) + (-ends(a, i)[0]).clamp_min(0)) * n[i] for i, a in enumerate(anti))
    div = sum((ends(a, i)[1] - ends(a, i)[0]) * n[i] for i, a in enumerate(low))
    q = (_At(phi)(0, 0, 0) - div).clamp_min(0)
    ratio = torch.where(out > 0, (q / out).clamp_max(1.0), torch.ones_like(out))
    s = 0
    for i in range(3):
        dim = 2 - i
        before = torch.cat([ratio.narrow(dim, n[i] - 1, 1), ratio], dim)
        after = torch.cat([ratio, ratio.narrow(dim, 0, 1)], dim)
        f = low[i] + torch.where(anti[i] >= 0, before, after) * anti[i]
        s = s + (ends(f, i)[1] - ends(f, i)[0]) * n[i]
    tend = torch.zeros_like(phi)
    tend[3:-3, 3:-3, 3:-3] = -s
    return tend


UNET_LAYERS = (("e1a", 16, 16), ("e1", 16, 16), ("e2a", 16, 32), ("e2", 32, 32), ("e3a", 32, 32), ("e3", 32, 32),
               ("d2", 32, 16), ("d1", 16, 16), ("out", 16, 16))


def _shift(x, dz, dy, dx):
    y = x.roll((-dy, -dx), (1, 2))
    if dz == 0:
        return y
    zero = torch.zeros_like(y[:1])
    return torch.cat([y[1:], zero]) if dz > 0 else torch.cat([zero, y[:-1]])


TAPS = [(dz, dy, dx) for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1)]


def _conv(x, w, b):
    return sum(_shift(x, *t) @ w[q].T for q, t in enumerate(TAPS)) + b


def _conv_back(x, w, g):
    gx, gw = 0, []
    for q, (dz, dy, dx) in enumerate(TAPS):
        gw.append(g.reshape(-1, g.shape[-1]).T @ _shift(x, dz, dy, dx).reshape(-1, x.shape[-1]))
        gx = gx + _shift(g @ w[q], -dz, -dy, -dx)
    return gx, torch.stack(gw), g.sum((0, 1, 2))


def _pool(x):
    nz, ny, nx, c = x.shape
    return x.reshape(nz // 2, 2, ny // 2, 2, nx // 2, 2, c).mean((1, 3, 5))


def _up(x):
    return x.repeat_interleave(2, 0).repeat_interleave(2, 1).repeat_interleave(2, 2)


def _unet_forward(case, seed):
    r, e, fluid, flat = _unet_inputs(case, seed)
    dev = _device()
    r, e, m = (torch.as_tensor(a, device=dev).to(F64) for a in (r, e, fluid))
    flat, at, P = torch.as_tensor(flat, device=dev).to(F64), 0, {}
    for name, ci, co in UNET_LAYERS:
        P[name] = (flat[at:at + 27 * ci * co].reshape(27, co, ci), flat[at + 27 * ci * co:at + 27 * ci * co + co])
        at += 27 * ci * co + co
    scale = (m.sum() / (r * m).square().sum()).sqrt()
    x = torch.zeros(r.shape + (16,), device=dev, dtype=F64)
    x[..., 0], x[..., 1] = r * scale, m
    A = {"x": x}
    for name, src in (("e1a", "x"), ("e1", "e1a"), ("e2a", "p1"), ("e2", "e2a"), ("e3a", "p2"), ("e3", "e3a"), ("d2", "u2"), ("d1", "u1")):
        if src == "p1":
            A[src] = _pool(A["e1"])
        elif src == "p2":
            A[src] = _pool(A["e2"])
        elif src == "u2":
            A[src] = _up(A["e3"]) + A["e2"]
        elif src == "u1":
            A[src] = _up(A["d2"]) + A["e1"]
        A[name] = _conv(A[src], *P[name]).clamp_min(0)
    A["out"] = _conv(A["d1"], *P["out"])[..., 0]
    return A, P, m, e, scale


def _exact_unet(case, seed):
    A, P, m, e, scale = _unet_forward(case, seed)
    if case["kind"] == "unet_apply":
        return A["out"] * (3.0 / scale) * m
    nf = m.sum()
    target = e * (nf / (e * m).square().sum()).sqrt()
    d = ((A["out"] - (A["out"] * m).sum() / nf) - (target - (target * m).sum() / nf)) * m
    loss = d.square().sum() / nf
    g0 = 2 * d / nf
    g0 = (g0 - (g0 * m).sum() / nf) * m
    g = torch.zeros_like(A["d1"])
    g[..., 0] = g0
    G = {}

    def back(name, src, g):
        gx, gw, gb = _conv_back(A[src], P[name][0], g)
        G[name] = torch.cat([gw.reshape(-1), gb])
        return gx

    def gate(g, name):
        return g * (A[name] > 0)

    def down(g):
        nz, ny, nx, c = g.shape
        return g.reshape(nz // 2, 2, ny // 2, 2, nx // 2, 2, c).sum((1, 3, 5))

    gx = back("out", "d1", g)
    g_e1 = back("d1", "u1", gate(gx, "d1"))
    g_e2 = back("d2", "u2", gate(down(g_e1), "d2"))
    gx = back("e3", "e3a", gate(down(g_e2), "e3"))
    gx = back("e3a", "p2", gate(gx, "e3a"))
    gx = back("e2", "e2a", gate(g_e2 + _up(gx) / 8, "e2"))
    gx = back("e2a", "p1", gate(gx, "e2a"))
    gx = back("e1", "e1a", gate(g_e1 + _up(gx) / 8, "e1"))
    back("e1a", "x", gate(gx, "e1a"))
    return {"loss": loss, "grads": torch.cat([G[name] for name, _, _ in UNET_LAYERS])}


def exact(case, seed):
    if case["kind"] == "step":
        return _exact_step(case, seed)
    if case["kind"] == "solve":
        a, b, fluid = _solve_inputs(case, seed)
        x = -_masked_poisson(b, [torch.as_tensor(q, device=b.device) ** 2 for q in a], (2.0, 2.0, 2.0))
        m = torch.as_tensor(fluid, device=b.device).to(F64)
        return (x - (x * m).sum() / m.sum()) * m
    if case["kind"] == "tracer":
        return _exact_tracer(case, seed)
    return _exact_unet(case, seed)
