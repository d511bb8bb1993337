"""The forms a call of several pseudo-steps can take, each forced by its options and compared with the others:
the many-step kernels, the separate kernels with what the next step overwrites left out, single full steps,
and the persistent stage kernel; every boundary kind through every source of boundary values."""
import numpy as np
import pytest

import cfd_solver_withcuda_b200 as cb
from cases import CASES, initial_state, make_mesh, solver_config
from conftest import assert_bits_equal
from test_gpu_batch import config, ramp_case
from test_gpu_parity import ADDITIVE, OPTION_SETS

pytestmark = pytest.mark.gpu

SEPARATE = dict(one_launch_steps=0)
FORMS = {"gradient": dict(muscl=1, is_second_order=1, dissipation_type=3, limiter=2, integrator=2,
                          local_time_stepping=1),
         "gradient_fp32_hllc": dict(muscl=1, is_second_order=1, dissipation_type=7, limiter=1, integrator=3,
                                    local_time_stepping=1, precision=cb.PREC_FP32_FLUX),
         "per_cell": dict(is_second_order=1, dissipation_type=3),
         "per_cell_lts": dict(is_second_order=0, dissipation_type=1, integrator=2, local_time_stepping=1)}


@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("inlet,outlet", [(1, 1), (1, 3), (4, 3), (4, 1), (2, 2), (3, 0)])
def test_boundary_kinds_in_every_form(form, inlet, outlet):
    m = cb.Mesh.bump(31, 14, 3.0, 1.0, 0.1, 4, 0.3, 7, True)
    NP = m.n_physical
    rng = np.random.default_rng(4)
    f = lambda: 1.0 + 0.01 * rng.normal(size=NP)
    U = np.zeros((m.n_total, 4))
    U[:NP] = cb.conserved_from_primitive(f(), 0.6 * f(), 0.01 * rng.normal(size=NP), f() / 1.4)
    U[m.boundary[:, 3]] = U[m.boundary[:, 1]]
    kw = dict(FORMS[form], time_accurate=1, cfl=0.3, reorder=1, inlet_bc=inlet, exit_bc=outlet, inlet_rho=1.0,
              inlet_u=0.6, inlet_v=0.01, inlet_p=1.0 / 1.4, inlet_p0=0.97, inlet_t0=0.0027, exit_p=0.99 / 1.4, r_gas=287.0)
    got = []
    for opts, calls in (({}, (9, 2)), (SEPARATE, (9, 2)), (dict(SEPARATE, use_graph=0), (1,) * 11)):
        s = cb.Solver(m, cb.default_config(**kw))
        for k, v in opts.items():
            s.set_option(k, v)
        s.upload_state(U)
        for n in calls:
            i = s.step(n)
        got.append((s.download(), (i.iterations, i.min_dt, i.total_time), s.kernel_launches))
        s.close()
    assert got[0][2] < got[1][2]  # the many-step kernel ran
    for d, i, _ in got[1:]:
        assert i == got[0][1]
        for k in ("U", "prim", "dt", "net_flux", "delU"):
            assert_bits_equal(got[0][0][k], d[k], k)


@pytest.mark.parametrize("form", ["grad_muscl_minmod_ssp_lts", "grad_muscl_ausm_fp32_ssp_lts", "grad_muscl_hllc_minmod"])
def test_launch_options_of_the_separate_kernels(form):
    """Fused gather, face-kernel shapes, graphs, programmatic launch and the L2 window, with the many-step
    kernel off: the bits of the default options, which take that kernel where the form allows it."""
    case = CASES["cyl_roe2_lts"]
    m = make_mesh(case)
    U0 = initial_state(case, m)
    want, launches = None, []
    for opts in [{}, SEPARATE] + [dict(o, **SEPARATE) for o in OPTION_SETS]:
        s = cb.Solver(m, solver_config(case, **ADDITIVE[form]))
        for k, v in opts.items():
            s.set_option(k, v)
        s.upload_state(U0)
        n0 = s.kernel_launches
        s.step(12)
        launches.append(s.kernel_launches - n0)
        d = s.download()
        s.close()
        want = want or d
        for k in ("U", "prim", "dt", "net_flux", "delU"):
            assert_bits_equal(d[k], want[k], "%s %s" % (k, opts))
    assert min(launches[1:]) >= 12 * 3 * 3  # three kernels per stage at least
    if "ssp_lts" in form:
        assert launches[0] < 12


@pytest.mark.parametrize("minb", [0, 4, 6, 8])
@pytest.mark.parametrize("precision", [cb.PREC_FP64, cb.PREC_FP32_FLUX])
def test_persistent_stage_kernel_of_a_batch(precision, minb):
    """The persistent stage kernel (many-step kernel off) with every register budget: the bits of the
    separate kernels, instances freezing in the middle of the run."""
    specs = [(24, 12, 1.5), (64, 32, 2.2), (16, 8, 3.0), (40, 24, 2.6), (12, 6, 2.0)]
    cases = [ramp_case(*sp) for sp in specs]
    out = []
    for persistent in (0, 1):
        b = cb.Batch([c[0] for c in cases], config(precision=precision, limiter=cb.LIM_MINMOD),
                     inflow=[c[2] for c in cases])
        for k, v in dict(SEPARATE, persistent=persistent, persist_minb=minb).items():
            b.set_option(k, v)
        b.upload_state([c[1] for c in cases])
        res = b.run(max_steps=1500, tol=1e-4, check_every=50)
        out.append((res, b.download_state()))
        b.close()
    (r0, u0), (r1, u1) = out
    assert np.array_equal(r0["steps_to_tol"], r1["steps_to_tol"]) and (r0["steps_to_tol"] > 0).any()
    assert np.array_equal(r0["res_ratio"].view(np.int64), r1["res_ratio"].view(np.int64))
    for a, b_ in zip(u0, u1):
        assert_bits_equal(b_, a, "instance")


def test_autotune_times_the_separate_kernels_and_the_many_step_kernel():
    """The candidates of a small frozen-dt solve differ in options the many-step kernel ignores: each runs as
    separate kernels, and the many-step kernel has its own line."""
    case = CASES["cyl_roe2_lts"]
    m = make_mesh(case)
    s = cb.Solver(m, solver_config(case, **ADDITIVE["grad_muscl_minmod_ssp_lts"]))
    s.upload_state(initial_state(case, m))
    steps, n0 = 10, s.kernel_launches
    report = s.autotune(steps=steps)
    assert report.count("ms/step") == 20 and report.count("(chosen)") == 1
    assert s.kernel_launches - n0 >= 20 * (2 + steps) * 9
    kept = "kept for calls of several steps" in report
    assert kept or "one_launch_steps=1" in report and "turned off" in report
    n0 = s.kernel_launches
    s.step(steps)
    assert (s.kernel_launches - n0 < steps) == kept


@pytest.mark.parametrize("nx,fits", [(395, True), (400, False)])
def test_capacity_of_the_many_step_kernel(nx, fits):
    """The largest shares that fit 148 blocks' shared memory (101,120 cells) and the first that do not."""
    m = cb.Mesh.box(nx, 256, 0.0, 2.0, 0.0, 1.0)
    NP = m.n_physical
    x = m.centers[:NP]
    U = np.zeros((m.n_total, 4))
    U[:NP] = cb.conserved_from_primitive(1 + 0.02 * np.sin(7 * x[:, 0]), 2 + 0.02 * np.cos(5 * x[:, 1]), 0 * x[:, 0],
                                         (1 + 0.01 * np.sin(9 * x[:, 1])) / 1.4)
    U[m.boundary[:, 3]] = U[m.boundary[:, 1]]
    kw = dict(FORMS["gradient"], time_accurate=1, cfl=0.4, inlet_bc=3, inlet_rho=1.0, inlet_u=2.0, inlet_p=1.0 / 1.4,
              reorder=4)
    got = []
    for on in (1, 0):
        s = cb.Solver(m, cb.default_config(**kw))
        s.set_option("one_launch_steps", on)
        s.upload_state(U)
        n0 = s.kernel_launches
        s.step(6)
        got.append((s.download(), s.kernel_launches - n0))
        s.close()
    assert (got[0][1] < 6) == fits and got[1][1] >= 6 * 9
    for k in ("U", "prim", "dt", "net_flux", "delU"):
        assert_bits_equal(got[0][0][k], got[1][0][k], k)


def test_batch_up_to_the_capacity():
    """49 channels of 64 x 32 cells (100,352) run in one launch, 50 (two blocks each, too large a share) do
    not; every instance has the separate kernels' bits."""
    m, U0, q = ramp_case(64, 32, 2.2)
    for n in (49, 50):
        out = []
        for on in (1, 0):
            b = cb.Batch([m] * n, config(limiter=cb.LIM_MINMOD), inflow=[q] * n)
            b.set_option("one_launch_steps", on)
            b.upload_state([U0 * (1.0 + 0.001 * i) for i in range(n)])
            b.run(max_steps=9, tol=0.0, check_every=8)
            out.append(b.download_state())
            b.close()
        for x, y in zip(*out):
            assert_bits_equal(x, y, "instance")


@pytest.mark.parametrize("forms", [("gradient", "gradient", "gradient_fp32_hllc"), ("per_cell", "gradient", "per_cell_lts")])
def test_many_step_kernels_of_several_contexts_at_once(forms):
    """Three contexts on their own streams, their many-step launches queued side by side: no wait runs out
    and every context has the bits it has alone."""
    import torch
    sizes = ((160, 100), (150, 110), (170, 90))  # each takes most or all of the SMs
    runs = []
    for form, (nx, ny) in zip(forms, sizes):
        m = cb.Mesh.box(nx, ny, 0.0, 2.0, 0.0, 1.0)
        NP = m.n_physical
        x = m.centers[:NP]
        U = np.zeros((m.n_total, 4))
        U[:NP] = cb.conserved_from_primitive(1 + 0.02 * np.sin(7 * x[:, 0]), 2 + 0.02 * np.cos(5 * x[:, 1]), 0 * x[:, 0],
                                             (1 + 0.01 * np.sin(9 * x[:, 1])) / 1.4)
        U[m.boundary[:, 3]] = U[m.boundary[:, 1]]
        kw = dict(FORMS[form], time_accurate=1, cfl=0.3, inlet_bc=3, inlet_rho=1.0, inlet_u=2.0, inlet_p=1.0 / 1.4,
                  reorder=4)
        runs.append((m, kw, U))

    def make(run):
        m, kw, U = run
        stream = torch.cuda.Stream()
        s = cb.Solver(m, cb.default_config(stream=stream.cuda_stream, **kw))
        s.upload_state(U)
        return s, stream
    alone = []
    for run in runs:
        s, _ = make(run)
        n0 = s.kernel_launches
        s.step_async(400)
        s.step_async(150)
        s.sync()
        assert s.kernel_launches - n0 < 100  # the many-step kernels ran
        alone.append(s.download())
        s.close()
    together = [make(run) for run in runs]
    for n in (400, 150):
        for s, _ in together:
            s.step_async(n)
    for (s, _), want in zip(together, alone):
        s.sync()
        got = s.download()
        s.close()
        for k in ("U", "prim", "dt", "net_flux", "delU"):
            assert_bits_equal(got[k], want[k], k)


@pytest.mark.parametrize("nx,ny", [(512, 443), (512, 445)])  # 226,816 and 227,840 cells: two waves on 148 SMs
@pytest.mark.parametrize("kw", [dict(is_second_order=0, dissipation_type=1),
                                dict(is_second_order=1, dissipation_type=3, integrator=2, local_time_stepping=1)])
def test_per_cell_forms_around_two_waves(nx, ny, kw, oracle_lib):
    """Below two waves the stage kernel writes the ghosts, from there on the boundary kernel: steps in one call,
    single steps and the reference's entry points against the C restatement."""
    m = cb.Mesh.box(nx, ny, 0.0, 2.0, 0.0, 1.0)
    NP = m.n_physical
    x = m.centers[:NP]
    U = np.zeros((m.n_total, 4))
    U[:NP] = cb.conserved_from_primitive(1 + 0.02 * np.sin(7 * x[:, 0]), 2 + 0.02 * np.cos(5 * x[:, 1]), 0 * x[:, 0],
                                         (1 + 0.01 * np.sin(9 * x[:, 1])) / 1.4)
    U[m.boundary[:, 3]] = U[m.boundary[:, 1]]
    kw = dict(kw, time_accurate=1, cfl=0.3, inlet_rho=1.0, inlet_u=2.0, inlet_p=1.0 / 1.4)
    o = oracle_lib.OracleRun(m, **kw)
    o.set_state(U)
    o.iterate(2)
    want = o.state()
    for calls in ((2,), (1, 1), None):
        s = cb.Solver(m, cb.default_config(reorder=4, **kw))
        s.upload_state(U)
        for n in calls or ():
            s.step(n)
        if calls is None:
            for _ in range(2):
                s.Apply_Boundary_Conditions()
                s.Runge_Kutta_Method()
                s.Estimate_Error()
                s.Update()
        got = s.download()
        s.close()
        for k in ("U", "net_flux", "delU"):
            assert_bits_equal(got[k], want[k], "%s %s" % (k, calls))
