"""Long thin meshes, up to the most rows of cells that the launches' grids
hold (65535 blocks of four rows of nodes), bit for bit against the C
restatement."""
from __future__ import annotations

import pytest

from conftest import CELL_FIELDS, EUC_FIELDS, NODE_FIELDS, assert_bitwise, get_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme", ["vnr", "euc"])
@pytest.mark.parametrize("nx,ny", [(2, 262139), (33, 247000), (262139, 2)])
def test_thin_mesh(scheme, nx, ny, port_lib):
    import mahyco_gb300 as M
    s = M.default_spec()
    s.scheme = M.SCHEME_VNR if scheme == "vnr" else M.SCHEME_EUCCLHYD
    s.test_case, s.nbmat, s.nx, s.ny = (16 if ny > nx else 15), 2, nx, ny
    s.dx, s.dy = 1.0 / max(nx, ny), 1.0 / max(nx, ny)
    s.final_time, s.dt_init, s.dt_min = 100.0, 1e-7, 1e-14
    s.projection, s.projection_order = 1, 2
    s.limiter, s.energy_limit, s.max_cycles = M.LIMITERS["minmod"], 0.0, 100
    g, c = M.Run(s), port_lib.PortRun(s)
    for n in (1, 1):
        assert g.step(n) == c.step(n)
        assert g.time() == c.time() and g.error() == c.error()
    for f in EUC_FIELDS if scheme == "euc" else CELL_FIELDS + NODE_FIELDS:
        assert_bitwise(f, get_field(g, f, s.nbmat), get_field(c, f, s.nbmat))
