"""What a call of several pseudo-steps does when it goes wrong, in the cooperative many-step kernels as in the
separate ones: a barrier wait that runs out ends the call with a status, a state that becomes non-physical
in the middle is reported with the same cell."""
import numpy as np
import pytest

import cfd_solver_withcuda_b200 as cb

pytestmark = pytest.mark.gpu

GRAD = dict(is_second_order=1, time_accurate=1, local_time_stepping=1, cfl=0.4, muscl=1, integrator=2, inlet_bc=3,
            dissipation_type=3, limiter=2, inlet_rho=1.0, inlet_p=1.0 / 1.4, inlet_u=2.0)
CELL = dict(time_accurate=1, cfl=0.3, dissipation_type=3, is_second_order=1, inlet_rho=1.0, inlet_p=1.0 / 1.4,
            inlet_u=2.0)


def _uniform(m):
    NP = m.n_physical
    o = np.ones(NP)
    U = np.zeros((m.n_total, 4))
    U[:NP] = cb.conserved_from_primitive(o, 2.0 * o, 0.0 * o, o / 1.4)
    U[m.boundary[:, 3]] = U[m.boundary[:, 1]]
    return U


@pytest.mark.parametrize("form", ["gradient", "per_cell", "batch"])
def test_barrier_wait_runs_out_with_a_status(form):
    """With one arrival that never comes the first wait runs out (about half a second), no later one waits,
    the call reports CFD_ERR_TIMEOUT, and a fresh context runs normally."""
    m = cb.Mesh.ramp(24, 12, open_top=True)
    kw = dict(CELL if form == "per_cell" else GRAD, reorder=0)
    inflow = (1.0, 2.0, 0.0, 1.0 / 1.4)
    for waits in (1, 0):
        if form == "batch":
            s = cb.Batch([m, m, m], cb.default_config(**kw), inflow=[inflow] * 3)
            s.upload_state([_uniform(m)] * 3)
            run = lambda: s.run(max_steps=8, tol=0.0, check_every=4)
        else:
            s = cb.Solver(m, cb.default_config(**kw))
            s.upload_state(_uniform(m))
            run = lambda: s.step(8)
        s.set_option("barrier_timeout_test", waits)
        if waits:
            with pytest.raises(cb.CfdError) as e:
                run()
            assert e.value.status == cb.CFD_ERR_TIMEOUT
        else:
            run()
        s.close()


@pytest.mark.parametrize("form", ["gradient", "gradient_fp32", "per_cell", "per_cell_lts"])
@pytest.mark.parametrize("steps", [12, 150])
def test_state_that_becomes_non_physical_in_the_middle(form, steps):
    """A cell of high pressure and too large a time step: after four to eight steps sound speeds become NaN.  The status and the reported cell are those of the separate kernels in the same call."""
    m = cb.Mesh.ramp(40, 20, open_top=True)
    kw, p = (dict(GRAD, cfl=3.5), 3.0) if form.startswith("gradient") else (dict(CELL, cfl=2.2), 10.0)
    if form == "gradient_fp32":
        kw.update(precision=cb.PREC_FP32_FLUX)
    if form == "per_cell_lts":
        kw.update(integrator=2, local_time_stepping=1, cfl=1.4)
    U = _uniform(m)
    NP = m.n_physical
    k = NP // 2 + 7
    U[k] = cb.conserved_from_primitive(np.array([1.0]), np.array([0.0]), np.array([0.0]), np.array([p]))[0]
    got = []
    for on in (1, 0):
        s = cb.Solver(m, cb.default_config(**dict(kw, reorder=0)))
        s.set_option("one_launch_steps", on)
        s.upload_state(U)
        s.step(1)
        with pytest.raises(cb.CfdError) as e:
            s.step(steps)
        got.append((e.value.status, str(e.value), np.isnan(s.download_U())))
        s.close()
    assert got[0][0] == got[1][0] == cb.CFD_ERR_NONPHYSICAL
    assert got[0][1] == got[1][1]
    assert np.array_equal(got[0][2], got[1][2])
