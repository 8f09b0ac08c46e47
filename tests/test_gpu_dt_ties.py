"""hydro_vnr_dt_noalloc where its filter decides: denominators that tie or
nearly tie, one odd value in the cell that holds the minimum, sound speeds
around the filter's lower bound, over its launch shapes (1 to 8 rows a warp,
ragged and narrow meshes), bit for bit against the cell candidates in numpy;
and a state at rest, where every cell ties, costs no multiple of an ordinary
one."""
from __future__ import annotations

import numpy as np
import pytest

from test_zz_no_alloc import _call, _candidates, _entry, _want

pytestmark = pytest.mark.gpu

# rows a warp: 1 1 1 1 1 2 4 4 8 8
SIZES = [(2, 2), (31, 8), (32, 9), (64, 48), (125, 64), (300, 300), (2, 5000), (512, 511), (1023, 1000),
         (2, 524288)]


def _check(nx, ny, fields):
    torch = pytest.importorskip("torch")
    import mahyco_gb300 as M
    L, f = _entry(M)
    dx, dy = 1.0 / nx, 0.7 / ny
    for name, (u, v, c) in fields:
        with np.errstate(all="ignore"):
            want = _want(_candidates(nx, ny, dx, dy, u, v, c), 1e300)
        got = _call(torch, L, f, nx, ny, dx, dy, u, v, c, 1e300)
        assert got == want, (name, got, want)


@pytest.mark.parametrize("nx,ny", SIZES)
def test_near_ties(nx, ny):
    rng = np.random.default_rng(nx * 7919 + ny)
    nn, nc = (nx + 1) * (ny + 1), nx * ny

    def fields():
        z = np.zeros(nn)
        yield "at rest", (z, z, np.full(nc, 1.18))
        yield "moving", (z + 0.75, z - 0.3, np.full(nc, 1.18))
        for eps in (1e-2, 1e-4, 1e-6, 1e-12):
            yield f"c {eps}", (z, z, 1.18 * (1 + eps * rng.uniform(-1, 1, nc)))
            yield f"u {eps}", (0.75 + eps * rng.uniform(-1, 1, nn), -0.3 + eps * rng.uniform(-1, 1, nn),
                               np.full(nc, 1.18))
        # around 2^-30, below which a sound speed is not ordered in FP32
        for lo, hi in ((1.0, 1.01), (0.99, 1.0), (0.9999, 1.0001), (0.5, 2.0)):
            u, v = rng.uniform(-1, 1, nn) * 1e-9, rng.uniform(-1, 1, nn) * 1e-9
            yield f"low {lo}", (u, v, 2.0 ** -30 * rng.uniform(lo, hi, nc))

    _check(nx, ny, fields())


@pytest.mark.parametrize("nx,ny", [(31, 8), (64, 48), (300, 300), (2, 5000), (512, 511)])
def test_one_odd_value(nx, ny):
    """The odd value sits in the cell that has the largest denominator
    without it, or is that largest one itself."""
    rng = np.random.default_rng(nx * 31 + ny)
    nn, nc = (nx + 1) * (ny + 1), nx * ny
    odd = [0.0, 5e-324, 1e-300, 1e-40, 2.0 ** -30, 2.0 ** -31, 1e18, 2.0 ** 61, 1e25, 1e200, 1e300,
           np.inf, np.nan]

    def fields():
        for k, x in enumerate(odd + [-0.75, -3.0, -1e-40]):
            u, v, c = rng.uniform(-1, 1, nn), rng.uniform(-1, 1, nn), rng.uniform(0.5, 2.0, nc)
            cell = (nc - 1, 0, int(rng.integers(nc)))[k % 3]
            i, j = divmod(cell, nx)
            n0 = i * (nx + 1) + j
            for nd in (n0, n0 + 1, n0 + nx + 2, n0 + nx + 1):
                u[nd] = 4.0 + 0.25 * (nd - n0 > 1)
            c[cell] = x
            yield f"c {x}", (u, v, c)
        for k, x in enumerate(odd):
            u, v, c = rng.uniform(-1, 1, nn), rng.uniform(-1, 1, nn), rng.uniform(0.5, 2.0, nc)
            cell = (0, int(rng.integers(nc)), nc - 1)[k % 3]
            i, j = divmod(cell, nx)
            c[cell] = 40.0
            (u, v)[k % 2][i * (nx + 1) + j + (nx + 2) * (k % 2)] = x
            yield f"u {x}", (u, v, c)

    _check(nx, ny, fields())


@pytest.mark.parametrize("nx,ny", [(64, 48), (90, 80), (128, 120), (2, 5000)])
def test_at_rest_costs_no_multiple(nx, ny):
    """Every cell's candidate is formed at rest: spread over the SMs that is
    under half a microsecond of FP64 work a thousand cells (at most 15 360
    here) on top of an ordinary call's latency; on a few SMs it was 5 to 15
    times the ordinary call."""
    torch = pytest.importorskip("torch")
    import mahyco_gb300 as M
    _, f = _entry(M)
    g = torch.Generator(device="cuda").manual_seed(7)

    def rand(*shape):
        return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)

    out = torch.empty(1, device="cuda", dtype=torch.float64)
    s = torch.cuda.current_stream().cuda_stream
    took = {}
    for name, u, c in (("ordinary", rand(ny + 1, nx + 1), 0.5 + rand(ny, nx)),
                       ("rest", 0.0 * rand(ny + 1, nx + 1), 0.0 * rand(ny, nx) + 1.18)):
        best = float("inf")
        for _ in range(8):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            for _ in range(50):
                assert f(nx, ny, 1.0 / nx, 0.7 / ny, u.data_ptr(), u.data_ptr(), c.data_ptr(), 1.0,
                         out.data_ptr(), s) == 0
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1))
        took[name] = best
    assert took["rest"] < 2.5 * took["ordinary"], took
