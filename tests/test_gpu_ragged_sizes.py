"""Plain runs on meshes at the edges of the kernels' blocks (32-cell rows,
one or four rows a block, two cells across, long thin meshes), over the
remap's options and one to three materials, bit for bit against the C
restatement."""
from __future__ import annotations

import pytest

from conftest import CELL_FIELDS, EUC_FIELDS, NODE_FIELDS, assert_bitwise, get_field

pytestmark = pytest.mark.gpu

# (scheme, test case, materials, remap order, PenteBorne, mixte, complet, dual, limiter)
OPTIONS = {
    "vnr_pb": ("vnr", 16, 2, 2, 1, 0, 0, 0, "superBee"),
    "vnr_pb_mixte_x": ("vnr", 15, 2, 2, 1, 1, 0, 1, "minmod"),
    "vnr_pb_dual_complet": ("vnr", 15, 2, 2, 1, 1, 1, 2, "superBee"),
    "vnr_mono": ("vnr", 4, 1, 2, 0, 0, 0, 0, "vanLeer"),
    "vnr_o1": ("vnr", 16, 2, 1, 0, 0, 0, 0, "minmod"),
    "vnr_o3": ("vnr", 15, 2, 3, 0, 0, 0, 1, "minmod"),
    "vnr_sedov": ("vnr", 1, 1, 2, 1, 1, 0, 0, "minmodG"),
    "euc_pb_mixte": ("euc", 13, 3, 2, 1, 1, 0, 0, "superBee"),
    "euc_pb_complet": ("euc", 13, 3, 2, 1, 0, 1, 0, "vanLeer"),
    "euc_o3": ("euc", 13, 3, 3, 0, 0, 0, 0, "superBee"),
    "euc_mono": ("euc", 4, 1, 2, 0, 0, 0, 0, "minmod"),
    "euc_conservative": ("euc", 16, 2, 2, 1, 0, 0, 0, "superBee"),
}
SIZES = [(2, 2), (3, 2), (2, 5), (31, 4), (33, 5), (64, 37), (5, 131), (97, 301), (650, 17)]


def _spec(M, name, nx, ny, cycles):
    scheme, case, nbmat, order, pb, mixte, complet, dual, limiter = OPTIONS[name]
    s = M.default_spec()
    s.scheme = M.SCHEME_VNR if scheme == "vnr" else M.SCHEME_EUCCLHYD
    s.test_case, s.nbmat, s.nx, s.ny = case, nbmat, nx, ny
    if case == 13:
        s.dx, s.dy, s.init_variant = 7.0 / nx, 3.0 / ny, 3
    else:
        s.dx, s.dy, s.init_variant = 1.0 / nx, 1.1 / ny, 1 if case in (15, 16) and scheme == "vnr" else 0
    for m in range(3):
        s.eos[m], s.gamma[m] = 101, 1.4 + 0.05 * m
    s.gamma_scalar, s.cfl = 1.4, 0.4
    s.final_time, s.dt_init, s.dt_min = 100.0, 1e-4, 1e-12
    s.space_order, s.projection, s.projection_order = 2, 1, order
    s.projection_conservative = int(name == "euc_conservative")
    s.limiter, s.limiter_pure = M.LIMITERS[limiter], M.LIMITERS["arithmeticG"]
    s.pb, s.pb_mixte, s.pb_complet, s.dual_mass_flux = pb, mixte, complet, dual
    s.threshold, s.energy_limit, s.max_cycles = 1e-16, 0.0, cycles
    return s


@pytest.mark.parametrize("name", list(OPTIONS))
@pytest.mark.parametrize("nx,ny", SIZES)
def test_ragged_sizes(name, nx, ny, port_lib):
    import mahyco_gb300 as M
    spec = _spec(M, name, nx, ny, 40)
    g, c = M.Run(spec), port_lib.PortRun(spec)
    # past the time step's ramp: most of the mesh moves, mixed cells appear
    for n in (1, 2, 37):
        assert g.step(n) == c.step(n)
        assert g.time() == c.time()
        assert g.error() == c.error()
        for f in EUC_FIELDS if spec.scheme == M.SCHEME_EUCCLHYD else CELL_FIELDS + NODE_FIELDS:
            assert_bitwise(f, get_field(g, f, spec.nbmat), get_field(c, f, spec.nbmat))
