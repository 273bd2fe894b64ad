"""launches_per_step, and what bench.py counts for a solve and a tracer, against the kernels that the runtime's trace of a step holds."""
import numpy as np
import pytest

from aeolus_b200 import CoreSpec, regular_grid
from aeolus_b200.inputs import embed

pytestmark = pytest.mark.gpu


def traced(step):
    import torch
    from torch.autograd import DeviceType
    from torch.profiler import ProfilerActivity, profile
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        step()
        torch.cuda.synchronize()
    names = [e.name for e in p.events() if e.device_type == DeviceType.CUDA]
    return [n for n in names if not n.startswith(("Memcpy", "Memset"))
            and "set_scalar_kernel" not in n and "finite_check_kernel" not in n]


@pytest.mark.parametrize("kw", [{}, {"precision": "fp32_mixed", "c_s": 0.17}, {"advection": "weno_z5"},
                                {"sgs": "dynamic", "c_s": 0.5}, {"sgs": "lagrangian", "c_s": 0.16},
                                {"sgs": "tke", "c_s": 0.17}, {"solver": "pcg"}, {"solver": "pcg", "c_s": 0.17}],
                         ids=lambda kw: "-".join(str(v) for v in kw.values()) or "plain")
@pytest.mark.parametrize("size", [(64, 32, 16), (16, 16, 8)])
def test_launches_of_a_step_are_the_traced_ones(kw, size):
    import torch
    from aeolus_b200.simulation import Simulation
    torch.zeros(1, device="cuda")
    g = regular_grid(size, (1.0, 1.0, 1.0), bc_z="wall")
    s = Simulation(CoreSpec(grid=g, nu=1e-3, theta0=300.0, **kw))
    if "solver" in kw:
        s.set_pcg(None, tol=1e-30, maxit=3)   # as many iterations in every substage
    rng = np.random.default_rng(4)
    u, v, w, th = (embed(g, 0.1 * rng.standard_normal((g.nz, g.ny, g.nx))) for _ in range(4))
    w[g.halo[2]] = 0
    s.set_state(u, v, w, 300.0 + th)
    count = s.launches_per_step() if "solver" not in kw else None   # without a step before it too
    s.step_rk3(1e-4)
    got = traced(lambda: s.step_rk3(1e-4))
    assert len(got) == s.launches_per_step(), sorted(got)
    assert count in (None, len(got))


@pytest.mark.parametrize("precond", ["vcycle", "jacobi", "identity"])
def test_launches_of_a_solve(precond):
    """Two kernels to begin with, two for the mean's shift, and the iterations between them."""
    import torch
    from aeolus_b200.multigrid import MGPreconditionedCG
    n = (32, 16, 8)
    s = MGPreconditionedCG(n, (1.0,) * 3, tol=1e-8, maxit=200, precond=precond)
    b = torch.randn(n[::-1], dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    x = torch.empty_like(b)
    s.solve_device(b.data_ptr(), x.data_ptr())
    stats = []
    got = traced(lambda: stats.append(s.solve_device(b.data_ptr(), x.data_ptr())))
    assert len(got) == 4 + stats[0]["iterations"] * s.launches_per_iteration, sorted(got)


def test_launches_of_a_tracer():
    import torch
    from aeolus_b200.simulation import Simulation
    g = regular_grid((64, 16, 16), (1.0, 1.0, 1.0))
    s = Simulation(CoreSpec(grid=g))
    a = [torch.rand(g.storage_shape, dtype=torch.float64, device="cuda") for _ in range(4)]
    t = torch.zeros_like(a[0])
    go = lambda: (s.advect_positive_device(*a, t, 1e-3, "weno_z5", accumulate=False), s.synchronize())
    go()
    got = traced(go)
    assert len(got) == 2, got
