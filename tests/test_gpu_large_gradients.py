"""Gradient pass of meshes of two waves and more (inputs brought into L2 ahead) against the tile form,
which forms the gradients in shared memory: the same bits, at a ragged and at a full last block."""
import numpy as np
import pytest

import cfd_solver_withcuda_b200 as cb
from conftest import assert_bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("nx,ny", [(512, 448), (479, 481)])  # 229,376 = 896 x 256 and 230,399 cells
def test_gradients_equal_tile_form(nx, ny, precision):
    m = cb.Mesh.ramp(nx, ny, open_top=True)
    NP = m.n_physical
    x = m.centers[:NP]
    U = np.zeros((m.n_total, 4))
    U[:NP] = cb.conserved_from_primitive(1 + 0.02 * np.sin(7 * x[:, 0]), 2 + 0.02 * np.cos(5 * x[:, 1]), 0 * x[:, 0],
                                         (1 + 0.01 * np.sin(9 * x[:, 1])) / 1.4)
    U[m.boundary[:, 3]] = U[m.boundary[:, 1]]
    kw = dict(dissipation_type=3, is_second_order=1, muscl=1, limiter=2, integrator=2, time_accurate=1,
              local_time_stepping=1, cfl=0.3, inlet_bc=3, inlet_rho=1.0, inlet_p=1.0 / 1.4, inlet_u=2.0, reorder=4,
              precision=precision)
    out = []
    for tile in (0, 1):
        s = cb.Solver(m, cb.default_config(**kw))
        s.set_option("tile_stage", tile)
        s.upload_state(U)
        s.step(4)
        out.append(s.download())
        s.close()
    for k in ("U", "prim", "dt", "net_flux"):
        assert_bits_equal(out[0][k], out[1][k], k)
