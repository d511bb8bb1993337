"""Per-cell flux forms: several pseudo-steps in one call (inner steps leave the next step's ghosts and
no norms) against one call per step, one and four threads per cell; every download and every scalar has
the same bits."""
import numpy as np
import pytest

import cfd_solver_withcuda_b200 as cb
from conftest import assert_bits_equal

pytestmark = pytest.mark.gpu


def _run(m, kw, U, opts, calls):
    s = cb.Solver(m, cb.default_config(**kw))
    for k, v in opts.items():
        s.set_option(k, v)
    s.upload_state(U)
    for n, t_end in calls:
        i = s.step(n, t_end)
    out = s.download(), (i.iterations, i.min_dt, i.total_time, tuple(i.error[:]), tuple(i.res_l2[:]))
    s.close()
    return out


@pytest.mark.parametrize("nx,ny,reorder", [(2, 1, 0), (33, 17, 4), (160, 150, 0)])  # 24,000: one thread per cell
@pytest.mark.parametrize("diss,order,integrator,time_accurate,lts", [
    (3, 1, 0, 1, 0), (3, 2, 0, 1, 1), (1, 1, 0, 0, 0), (2, 2, 1, 1, 1), (4, 2, 2, 1, 0), (5, 1, 3, 1, 1),
    (7, 1, 4, 1, 1), (6, 1, 0, 1, 1)])
def test_steps_in_one_call_equal_single_steps(nx, ny, reorder, diss, order, integrator, time_accurate, lts):
    m = cb.Mesh.ramp(nx, ny, open_top=True)
    rng = np.random.default_rng(nx)
    NP = m.n_physical
    f = lambda: 1.0 + 0.02 * rng.normal(size=NP)
    U = np.zeros((m.n_total, 4))
    U[:NP] = cb.conserved_from_primitive(f(), 2.0 * f(), 0.02 * rng.normal(size=NP), f() / 1.4)
    U[m.boundary[:, 3]] = U[m.boundary[:, 1]]
    kw = dict(dissipation_type=diss, is_second_order=order - 1, integrator=integrator, time_accurate=time_accurate,
              local_time_stepping=lts, cfl=0.1, inlet_rho=1.0, inlet_p=1.0 / 1.4, inlet_u=2.0, reorder=reorder)
    a, ia = _run(m, kw, U, {}, [(1, 0.0)] * 7)
    for opts, calls in (({}, [(7, 0.0)]), (dict(use_graph=0), [(4, 0.0), (3, 0.0)]), (dict(flux_lanes=4), [(7, 0.0)]),
                        (dict(flux_lanes=1), [(5, 0.0), (2, 1e9)])):
        b, ib = _run(m, kw, U, opts, calls)
        for k in ("U", "prim", "dt", "net_flux", "delU"):
            assert_bits_equal(a[k], b[k], k)
        assert ia == ib


@pytest.mark.parametrize("nx,ny,steps", [(2, 2, 300), (148, 128, 5), (149, 128, 5)])
@pytest.mark.parametrize("diss,order,lts", [(3, 2, 0), (1, 1, 1)])
def test_one_launch_limits(nx, ny, steps, diss, order, lts):
    """More steps than one launch holds; the largest mesh whose four lanes per cell are resident on 148 SMs
    (18,944 cells) and one beyond it.  Against the separate kernels in the same calls."""
    m = cb.Mesh.ramp(nx, ny, open_top=True)
    NP = m.n_physical
    U = np.zeros((m.n_total, 4))
    x = m.centers[:NP]
    U[:NP] = cb.conserved_from_primitive(1 + 0.02 * np.sin(7 * x[:, 0]), 2 + 0.02 * np.cos(5 * x[:, 1]), 0 * x[:, 0],
                                         (1 + 0.01 * np.sin(9 * x[:, 1])) / 1.4)
    U[m.boundary[:, 3]] = U[m.boundary[:, 1]]
    kw = dict(dissipation_type=diss, is_second_order=order - 1, integrator=0, time_accurate=1, local_time_stepping=lts,
              cfl=0.1, inlet_rho=1.0, inlet_p=1.0 / 1.4, inlet_u=2.0, reorder=4)
    a, ia = _run(m, kw, U, dict(one_launch_steps=0), [(steps, 0.0), (3, 0.0)])
    b, ib = _run(m, kw, U, {}, [(steps, 0.0), (3, 0.0)])
    for k in ("U", "prim", "dt", "net_flux", "delU"):
        assert_bits_equal(a[k], b[k], k)
    assert ia == ib
