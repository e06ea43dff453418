"""A call with so many tables that its uv tiles (times tables) stay below the limit
of 2^30 for tiles that start at the grid, but not for the register tiles, which start
before it: gridded by the general kernel.  All tables are the same, so the grid is
that of a single one."""
import numpy as np
import pytest

import gpugrid as gg
import oracle as O
import synth
from helpers import planar_from_grid, rel_err

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_below_the_limit_by_the_general_tiles_only():
    N, S, G, n, tables = 2048, 8, 1, 500, 16_383  # (2048 / 8)^2 * 16383 < 2^30 < 258^2 * 16383
    rng = np.random.default_rng(2)
    uv = synth.fr(rng.uniform(-S, N + S, size=(n, 2)))
    vals = synth.normal_vals(rng, n, np.complex64)
    one = rng.uniform(0.5, 1, size=(G * G, S, S)).astype(np.complex64)
    index = rng.integers(tables, size=n).astype(np.int32)
    dev = [torch.from_numpy(a).cuda() for a in (uv, vals)]
    tab = torch.from_numpy(one.reshape(-1)).cuda().repeat(tables)
    out = torch.full((N * N,), float("nan"), device="cuda", dtype=torch.complex64)
    ctx = gg.Context(0)
    ctx.grid_job(gg.Options(mode=gg.MODE_WINDOW, accum=gg.ACC_COMPENSATED, oversample=G,
                            layout=gg.LAYOUT_INTERLEAVED),
                 gg.Context.make_job(out, *dev, tab, N, S, npts=n,
                                     gcf_index=torch.from_numpy(index).cuda(), n_gcf=tables))
    torch.cuda.synchronize()
    assert ctx.read_flags() == [0, 0, 0, 0]
    got = planar_from_grid(torch.view_as_real(out).reshape(-1).cpu().numpy(), 1, N, False)
    ctx.close()
    pairs = lambda c: np.stack([c.real, c.imag], -1).reshape(-1, 2).astype(np.float64)
    ref = O.grid_pz(uv, pairs(vals), pairs(one), N, S, gcf_grid=G)
    assert rel_err(got, ref) <= 1e-6
