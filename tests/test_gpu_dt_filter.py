"""hydro_vnr_dt_noalloc at the edges of its filter: the single-block and the
two-launch form, ragged warps (31 columns, 8 rows a warp), uniform fields
where every cell ties, and values that the FP32 filter does not order
(zero, negative, tiny, huge, infinite, NaN), bit for bit against the cell
candidates in numpy."""
from __future__ import annotations

import numpy as np
import pytest

from test_zz_no_alloc import _call, _candidates, _entry, _want

pytestmark = pytest.mark.gpu

SIZES = [(2, 2), (31, 8), (32, 9), (30, 7), (124, 64), (125, 64), (62, 129), (2, 5000), (5000, 2),
         (333, 257), (2, 524288)]


def _fields(kind, nx, ny):
    rng = np.random.default_rng(nx * 7919 + ny)
    nn, nc = (nx + 1) * (ny + 1), nx * ny
    u, v = rng.uniform(-1, 1, nn), rng.uniform(-1, 1, nn)
    c = rng.uniform(0.5, 2.0, nc)
    if kind == "uniform":
        u[:], v[:], c[:] = 0.0, 0.0, 1.18
    elif kind == "odd":
        for x in (u, v):
            k = rng.integers(0, nn, 6)
            x[k] = [np.nan, np.inf, 1e300, 1e25, 1e-300, 0.0]
        k = rng.integers(0, nc, 8)
        c[k] = [0.0, np.nan, np.inf, 1e-300, 1e-40, 1e30, 1e200, -0.75]
    elif kind == "small":
        u, v, c = u * 1e-60, v * 1e-60, c * 1e-12
    return u, v, c


@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("kind", ["mixed", "uniform", "odd", "small"])
def test_dt_filter(nx, ny, kind):
    torch = pytest.importorskip("torch")
    import mahyco_gb300 as M
    L, f = _entry(M)
    u, v, c = _fields(kind, nx, ny)
    for dx, dy in ((1.0 / nx, 0.7 / ny), (3e-120, 2.5)):
        with np.errstate(all="ignore"):
            want = _want(_candidates(nx, ny, dx, dy, u, v, c), 1e3)
        got = _call(torch, L, f, nx, ny, dx, dy, u, v, c, 1e3)
        assert got == want, (dx, got, want)
