"""Order-3 remap next to a side with a boundary flux: the flux through the
side's face carries the value of the cell's opposite face, also where that
face is at rest.  Shock bubbles whose gas starts at rest at the right side
(the domain ends left of the moving gas) and the unit tests' left side, plain
and batched, bit for bit against the C restatement."""
from __future__ import annotations

import pytest

from conftest import GOLDEN, assert_bitwise, fields_of, get_field, load_golden

pytestmark = pytest.mark.gpu


def _spec(case, nx, ny, dx, dy):
    spec, _, _ = load_golden(GOLDEN / f"{case}.npz")
    spec.nx, spec.ny, spec.dx, spec.dy = nx, ny, dx, dy
    spec.projection_order, spec.pb = 3, 0
    spec.energy_limit, spec.max_cycles, spec.final_time = 0.0, 60, 10.0
    return spec


def _check(run, ref, spec):
    assert run.time() == ref.time()
    assert run.error() == ref.error()
    for f in fields_of(spec):
        assert_bitwise(f, get_field(run, f, spec.nbmat), get_field(ref, f, spec.nbmat))


@pytest.mark.parametrize("case,nx,ny,dx,dy", [
    ("SHOCK_BUBBLE_MinMod_o2", 8, 8, 0.07, 0.01),
    ("SHOCK_BUBBLE_MinMod_o2", 2, 3, 0.07, 0.01),
    ("SHOCK_BUBBLE_MinMod_o2", 3, 2, 0.07, 0.01),
    ("SHOCK_BUBBLE_MinMod_o2", 100, 16, 0.005, 0.005),
    ("BIUNIT_vnr_init", 8, 8, 0.1, 0.1),
    ("BIUNIT_vnr_init", 2, 5, 0.1, 0.1),
])
@pytest.mark.parametrize("batched", [False, True])
def test_order3_flux_side(case, nx, ny, dx, dy, batched, port_lib):
    import mahyco_gb300 as M
    spec = _spec(case, nx, ny, dx, dy)
    ctx = M.Context(0)
    run, ref = M.Run(spec, ctx), port_lib.PortRun(spec)
    batch = M.Batch([run], ctx) if batched else None
    for n in (1, 1, 28):
        (batch or run).step(n)
        ref.step(n)
        _check(run, ref, spec)
