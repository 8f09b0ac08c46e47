"""Fetching results while the server works: each result is taken as soon as
its request completes, while other requests join and leave (which makes the
worker capture its launches anew), and the client steps a run of its own in
the same context.  Every result equals the same run advanced alone, bit for
bit."""
from __future__ import annotations

import time

import pytest

from conftest import CELL_FIELDS, NODE_FIELDS, assert_bitwise, get_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tick", [4, 8])
def test_fetch_while_serving(tick):
    import mahyco_gb300 as M
    from mahyco_gb300.workloads import Instance, request_stream
    ctx = M.Context(0)
    srv = M.Server(ctx, max_resident=6, tick_cycles=tick)
    own_spec = Instance("sod", 48, 32, 2, "minmod", 400, "X").spec(M)
    own = M.Run(own_spec, ctx)
    specs, got, own_steps = {}, {}, 0
    for r in request_stream(1000.0, 60, seed=31, size_range=(12, 128), cycle_range=(8, 90)):
        spec = r.inst.spec(M)
        specs[srv.submit(spec, keep=True)] = spec
    t0 = time.time()
    while len(got) < len(specs):
        d = srv.poll(1.0)
        assert time.time() - t0 < 120.0, "serving did not finish"
        if d is None:
            continue
        assert d.status & ~M.ERR_NEGATIVE == 0
        run = srv.result(d.req_id)
        nb = specs[d.req_id].nbmat
        got[d.req_id] = ({f: get_field(run, f, nb) for f in CELL_FIELDS + NODE_FIELDS}, run.time())
        srv.release(d.req_id)
        if own_steps < 300:
            own.step(9)
            own_steps += 9
    srv.stop()
    other = M.Context(0)
    for rid, spec in specs.items():
        alone = M.Run(spec, other)
        alone.simulate()
        fields, at = got[rid]
        for f in CELL_FIELDS + NODE_FIELDS:
            assert_bitwise(f"req{rid}:{f}", fields[f], get_field(alone, f, spec.nbmat))
        assert at == alone.time(), rid
    alone = M.Run(own_spec, other)
    alone.step(own_steps)
    for f in CELL_FIELDS + NODE_FIELDS:
        assert_bitwise(f, get_field(own, f, 2), get_field(alone, f, 2))
