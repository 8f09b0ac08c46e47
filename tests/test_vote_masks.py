"""Warp votes and shuffles of the kernels name lanes that are known to arrive
there: __activemask() tells which lanes happen to run together, not which
ones reach the next instruction together."""
from __future__ import annotations

from conftest import ROOT


def test_no_vote_over_the_active_mask():
    sources = sorted((ROOT / "mahyco_gb300" / "csrc").rglob("*.cu*"))
    assert len(sources) > 10
    assert [p.name for p in sources if "__activemask" in p.read_text()] == []
