"""Support 32 with the on-the-fly Gaussian, summed by 16x16 output block, at the
sizes where it can go wrong: grids around one block and one tile, coordinates
on every side, blocks shared by a CTA's warps and not, groups of records
around 32, dense tiles, layouts, grid types, polarisations, accumulation,
batches (also jobs that share a grid, which keep the adding kernel) and values
that are not finite.  Against the CPU oracle with the FP64 table; tolerances as
for every on-the-fly Gaussian: 1e-6 normwise, per cell 1e-6 compensated and
1e-5 plain.
"""
import numpy as np
import pytest

import gpugrid as gg
import oracle as O
import synth
from helpers import cell_err, planar_from_grid, rel_err

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
S = 32


@pytest.fixture(scope="module")
def ctx():
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    c = gg.Context(0)
    yield c
    c.close()


def pairs(c):
    c = np.asarray(c).reshape(-1)
    return np.stack([c.real, c.imag], -1).astype(np.float64)


def opts(comp=True, **kw):
    kw.setdefault("layout", gg.LAYOUT_INTERLEAVED)
    return gg.Options(mode=gg.MODE_WINDOW, accum=gg.ACC_COMPENSATED if comp else gg.ACC_PLAIN,
                      gcf_kind=gg.GCF_GAUSSIAN, **kw)


def device(uv, vals, cells, out=torch.complex64, fill=float("nan")):
    return (torch.from_numpy(np.ascontiguousarray(uv)).cuda(),
            torch.from_numpy(np.ascontiguousarray(vals)).cuda(),
            torch.full((cells,), fill, dtype=out, device="cuda"))


def planar(g, P, N, o):
    host = torch.view_as_real(g).reshape(-1).cpu().numpy()
    return planar_from_grid(host, P, N, o.layout == gg.LAYOUT_PLANAR)


def check(got, uv, vals, N, P=1, G=8, comp=True):
    gcf = synth.gcf_table(synth.gaussian_gcf_1d(S, G))
    ref = O.grid_pz(uv, pairs(vals), pairs(gcf), N, S, pols=P, gcf_grid=G, nthreads=8)
    mag = O.grid_mag(uv, pairs(vals), pairs(gcf), N, S, pols=P, gcf_grid=G, nthreads=8)
    assert rel_err(got, ref) <= 1e-6
    assert cell_err(got, ref, mag)[0] <= (1e-6 if comp else 1e-5)


@pytest.mark.parametrize("N,n,G,P,layout,out,comp", [
    (1, 40, 8, 1, gg.LAYOUT_INTERLEAVED, torch.complex64, True),
    (15, 300, 8, 2, gg.LAYOUT_PLANAR, torch.complex64, True),
    (16, 33, 1, 1, gg.LAYOUT_INTERLEAVED, torch.complex64, False),
    (17, 31, 16, 1, gg.LAYOUT_INTERLEAVED, torch.complex128, True),
    (95, 5000, 8, 3, gg.LAYOUT_INTERLEAVED, torch.complex64, True),
    (200, 20000, 4, 1, gg.LAYOUT_PLANAR, torch.complex128, False),
    # more blocks than shared ones are used for
    (2000, 30000, 8, 1, gg.LAYOUT_INTERLEAVED, torch.complex64, True),
    (2000, 30000, 8, 1, gg.LAYOUT_PLANAR, torch.complex64, False)])
def test_sizes_and_edges(ctx, N, n, G, P, layout, out, comp):
    rng = np.random.default_rng(N)
    uv = synth.fr(rng.uniform(-S, N + S, size=(n, 2)))
    uv[:6] = [[-16, 0], [N + 14, N - 1], [0, N + 15], [-15.5, -15.5], [N - 0.125, 3], [7.875, 8]]
    vals = synth.normal_vals(rng, n * P)
    o = opts(comp, layout=layout, oversample=G, polarizations=P)
    d_uv, d_v, g = device(uv, vals, P * N * N, out)
    ctx.grid(o, g, d_uv, d_v, None, N, S)
    torch.cuda.synchronize()
    assert ctx.read_flags() == [0, 0, 0, 0]
    check(planar(g, P, N, o), uv, vals, N, P, G, comp)


def test_dense_tile_and_empty_blocks(ctx):
    N, n, rng = 300, 40000, np.random.default_rng(5)
    uv = synth.fr(rng.uniform(96, 104, size=(n, 2)))
    vals = (1 + 0.5 * synth.normal_vals(rng, n)).astype(np.complex64)
    o = opts()
    d_uv, d_v, g = device(uv, vals, N * N)
    ctx.grid(o, g, d_uv, d_v, None, N, S)
    torch.cuda.synchronize()
    check(planar(g, 1, N, o), uv, vals, N)


def test_accumulate_and_batch(ctx):
    """two jobs of a batch into grids of their own, and into one grid"""
    rng, N, n = np.random.default_rng(8), 70, 2000
    sets = [(synth.fr(rng.uniform(0, N, size=(n, 2))), synth.normal_vals(rng, n))
            for _ in range(2)]
    o = opts(accumulate=True)
    dev = [device(uv, v, N * N, fill=0.0) for uv, v in sets]
    own = [gg.Context.make_job(d[2], d[0], d[1], None, N, S) for d in dev]
    ctx.grid_batch(o, own)
    ctx.grid_batch(o, own)  # twice: every sum doubled
    one = torch.zeros(N * N, dtype=torch.complex64, device="cuda")
    ctx.grid_batch(o, [gg.Context.make_job(one, d[0], d[1], None, N, S) for d in dev])
    torch.cuda.synchronize()
    for (uv, v), d in zip(sets, dev):
        check(planar(d[2], 1, N, o) / 2, uv, v, N)
    check(planar(one, 1, N, o), np.concatenate([s[0] for s in sets]),
          np.concatenate([s[1] for s in sets]), N)


@pytest.mark.parametrize("N", [64, 2000])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("comp", [True, False])
def test_values_that_are_not_finite_stay_in_their_footprint(ctx, N, comp, bad):
    n, rng = 500, np.random.default_rng(3)
    uv = synth.fr(rng.uniform(10, 60, size=(n, 2)))
    vals = synth.normal_vals(rng, n)
    odd = vals.copy()
    odd[7] = bad
    vals[7] = 0
    o = opts(comp)
    d_uv, d_v, g = device(uv, odd, N * N)
    ctx.grid(o, g, d_uv, d_v, None, N, S)
    torch.cuda.synchronize()
    got = planar(g, 1, N, o)[:, 0]
    ref = O.grid_pz(uv, pairs(vals), pairs(synth.gcf_table(synth.gaussian_gcf_1d(S))), N, S,
                    nthreads=8)[:, 0]
    x0, y0 = np.floor(uv[7]).astype(int) - S // 2 + 1
    inside = np.zeros((N, N), bool)
    inside[max(0, y0):y0 + S, max(0, x0):x0 + S] = True
    assert not np.isfinite(got[0][inside]).any()
    assert np.isfinite(got[:, ~inside]).all()
    assert rel_err(got[:, ~inside], ref[:, ~inside]) <= 1e-6
