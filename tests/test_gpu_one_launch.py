"""Whole pseudo-steps in one launch (option "one_launch_steps") against the separate kernels: the same
state bits, Min_dt and Total_Time for every scheme, precision and frozen-dt integrator, at sizes
around the blocks' shares and the size limit; the norms are summed in another order (1e-12 relative)."""
import numpy as np
import pytest

import cfd_solver_withcuda_b200 as cb
from conftest import assert_bits_equal

pytestmark = pytest.mark.gpu

BASE = dict(is_second_order=1, time_accurate=1, local_time_stepping=1, cfl=0.4, muscl=1, inlet_bc=3, inlet_rho=1.0,
            inlet_p=1.0 / 1.4, inlet_u=2.0)


def _start(m, seed, mach=2.0):
    rng = np.random.default_rng(seed)
    NP = m.n_physical
    f = lambda: 1.0 + 0.02 * rng.normal(size=NP)
    U = np.zeros((m.n_total, 4))
    U[:NP] = cb.conserved_from_primitive(f(), mach * f(), 0.02 * rng.normal(size=NP), f() / 1.4)
    U[m.boundary[:, 3]] = U[m.boundary[:, 1]]
    return U


def _pair(m, kw, calls, U):
    out = []
    for on in (1, 0):
        s = cb.Solver(m, cb.default_config(**kw))
        s.set_option("one_launch_steps", on)
        s.upload_state(U)
        infos = []
        for n, t_end in calls:
            i = s.step(n, t_end)
            infos.append((i.iterations, i.min_dt, i.total_time, np.array(i.error[:]), np.array(i.res_l2[:])))
        launches = s.kernel_launches
        out.append((s.download(), infos, launches))
        s.close()
    (a, ia, la), (b, ib, lb) = out
    assert la < lb  # the one-launch form was taken
    for k in ("U", "prim", "dt", "net_flux", "delU"):
        assert_bits_equal(a[k], b[k], k)
    for x, y in zip(ia, ib):
        assert x[:3] == y[:3]
        np.testing.assert_allclose(x[3], y[3], rtol=1e-12)
        np.testing.assert_allclose(x[4], y[4], rtol=1e-12)


@pytest.mark.parametrize("diss,limiter,integrator,precision,extra", [
    (3, 2, 2, 0, {}), (3, 1, 2, 1, {}), (7, 1, 2, 0, {}), (6, 4, 2, 0, {}), (8, 3, 2, 1, {}), (3, 2, 1, 0, {}),
    (3, 2, 3, 0, {}), (7, 2, 4, 1, {}), (3, 1, 2, 0, dict(entropy_fix_linear=0.3, shock_fix=0.1))])
@pytest.mark.parametrize("nx,ny", [(3, 2), (33, 16), (91, 91)])
def test_one_launch_equals_separate_kernels(nx, ny, diss, limiter, integrator, precision, extra):
    m = cb.Mesh.ramp(nx, ny, open_top=True)  # 6, 528 and 8,281 cells
    kw = dict(BASE, dissipation_type=diss, limiter=limiter, integrator=integrator, precision=precision, **extra)
    _pair(m, kw, [(7, 0.0), (2, 0.0), (1, 0.0), (3, 0.0)], _start(m, nx))


@pytest.mark.parametrize("nx,ny", [(6144, 1), (33, 1), (384, 256), (49, 127)])
def test_one_launch_size_limits(nx, ny):
    """Long strips (two boundary entries per cell), the largest one-launch solve (98,304 cells) and a
    ragged size."""
    m = cb.Mesh.box(nx, ny, 0.0, 2.0, 0.0, 1.0)
    kw = dict(BASE, dissipation_type=3, limiter=2, integrator=2, reorder=0)
    _pair(m, kw, [(5, 0.0)], _start(m, ny))


def test_one_launch_mixed_mesh_and_t_end():
    """Triangles and quads with total-pressure inflow and static-pressure outflow; more steps than one
    launch holds; Total_Time passing t_end inside a launch."""
    m = cb.Mesh.bump(63, 24, 3.0, 1.0, 0.1, 4, 0.3, 7, True)
    kw = dict(BASE, dissipation_type=7, limiter=1, integrator=2, inlet_bc=2, exit_bc=2, inlet_p0=0.97, inlet_t0=0.0027,
              exit_p=1.0 / 1.4, r_gas=287.0, reorder=1)
    U = _start(m, 3, mach=0.6)
    _pair(m, kw, [(300, 0.0), (150, 0.0)], U)
    s = cb.Solver(m, cb.default_config(**kw))
    s.set_option("one_launch_steps", 0)
    s.upload_state(U)
    t_end = s.step(40).total_time
    s.close()
    _pair(m, kw, [(100, t_end)], U)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("persistent", [0, 1])
def test_batch_blocks_per_instance(precision, persistent):
    """Uneven instances, some freezing at the tolerance in the middle of the run."""
    meshes = [cb.Mesh.ramp(nx, ny, open_top=True) for nx, ny in ((24, 12), (90, 45), (16, 8), (40, 24), (3, 2))]
    machs = [1.5, 2.2, 3.0, 2.6, 2.0]
    inflow = [(1.0, M, 0.0, 1.0 / 1.4) for M in machs]
    out = []
    for on in (1, 0):
        b = cb.Batch(meshes, cb.default_config(**dict(BASE, dissipation_type=3, limiter=1, integrator=2, reorder=0,
                                                      precision=precision)), inflow=inflow)
        b.set_option("persistent", persistent)
        b.set_option("one_launch_steps", on)
        b.upload_state([_start(m, i, M) for i, (m, M) in enumerate(zip(meshes, machs))])
        r = b.run(max_steps=1200, tol=1e-3, check_every=50)
        out.append((r, b.download_state()))
        b.close()
    (ra, ua), (rb, ub) = out
    assert np.array_equal(ra["steps_to_tol"], rb["steps_to_tol"]) and (ra["steps_to_tol"] > 0).any()
    assert np.array_equal(ra["res_ratio"].view(np.int64), rb["res_ratio"].view(np.int64))
    for x, y in zip(ua, ub):
        assert_bits_equal(x, y, "instance")
