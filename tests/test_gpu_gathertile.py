"""Gather by 16x16 output block (supports 8 and 16, FP32 values) at the sizes where
it can go wrong: grids around one block and one tile, coordinates on every
side, groups of records around 32, dense tiles, blocks shared by a CTA's warps
and not, real, complex and Gaussian factors, oversamplings, layouts, grid types,
polarisations, accumulation, batches with a support that keeps the 32-cell
tiles, and values that are not finite.  Against the CPU oracle; tolerances as
for every FP32 path: compensated 1e-6, plain 2e-6 (normwise), per cell 1e-6
and 1e-5.
"""
import numpy as np
import pytest

import gpugrid as gg
import oracle as O
import synth
from helpers import cell_err, planar_from_grid, rel_err

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


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
    return gg.Options(mode=gg.MODE_GATHER, accum=gg.ACC_COMPENSATED if comp else gg.ACC_PLAIN,
                      **kw)


def table(S, G, kind, rng):
    t = synth.gcf_table(synth.gaussian_gcf_1d(S, G))
    if kind == "complex":
        t = t * np.exp(1j * rng.uniform(0, 6, t.shape))
    return t.astype(np.complex64)


def device(uv, vals, gcf, cells, out=torch.complex64, fill=float("nan")):
    return (torch.from_numpy(np.ascontiguousarray(uv)).cuda(),
            torch.from_numpy(np.ascontiguousarray(vals)).cuda(),
            None if gcf is None else torch.from_numpy(gcf.reshape(-1)).cuda(),
            torch.full((cells,), fill, dtype=out, device="cuda"))


def check(g, o, uv, vals, gcf, N, S, P=1, G=8, comp=True, scale=1.0):
    host = torch.view_as_real(g).reshape(-1).cpu().numpy() / scale
    got = planar_from_grid(host, P, N, o.layout == gg.LAYOUT_PLANAR)
    ref = O.grid_pz(uv, pairs(vals), pairs(gcf), N, S, pols=P, gcf_grid=G, nthreads=8)
    mag = O.grid_mag(uv, pairs(vals), pairs(gcf), N, S, pols=P, gcf_grid=G, nthreads=8)
    assert rel_err(got, ref) <= (1e-6 if comp else 2e-6)
    assert cell_err(got, ref, mag)[0] <= (1e-6 if comp else 1e-5)


@pytest.mark.parametrize("kind", ["real", "complex"])
@pytest.mark.parametrize("S", [8, 16])
@pytest.mark.parametrize("N,n,G,P,layout,out,comp", [
    (1, 40, 8, 1, gg.LAYOUT_INTERLEAVED, torch.complex64, True),
    (15, 33, 4, 2, gg.LAYOUT_PLANAR, torch.complex64, True),
    (16, 31, 1, 1, gg.LAYOUT_INTERLEAVED, torch.complex64, False),
    (17, 300, 8, 1, gg.LAYOUT_INTERLEAVED, torch.complex128, True),
    (95, 5000, 2, 3, gg.LAYOUT_INTERLEAVED, torch.complex64, True),
    (200, 20000, 8, 1, gg.LAYOUT_PLANAR, torch.complex128, False),
    # more blocks than shared ones are used for
    (1200, 30000, 8, 1, gg.LAYOUT_INTERLEAVED, torch.complex64, True)])
def test_sizes_and_edges(ctx, N, n, G, P, layout, out, comp, S, kind):
    rng = np.random.default_rng(N + S)
    uv = synth.fr(rng.uniform(-S, N + S, size=(n, 2)))
    uv[:6] = [[-S / 2, 0], [N + S / 2 - 2, N - 1], [0, N + S / 2 - 1], [-S / 2 + .5, -S / 2],
              [N - 0.125, 3], [7.875, 8]]
    vals = synth.normal_vals(rng, n * P)
    gcf = table(S, G, kind, rng)
    o = opts(comp, layout=layout, oversample=G, polarizations=P)
    d = device(uv, vals, gcf, P * N * N, out)
    ctx.grid(o, d[3], *d[:3], N, S)
    torch.cuda.synchronize()
    assert ctx.read_flags() == [0, 0, 0, 0]
    check(d[3], o, uv, vals, gcf, N, S, P, G, comp)


@pytest.mark.parametrize("N", [150, 1200])
def test_dense_tile_empty_blocks_and_gaussian(ctx, N):
    n, S, rng = 30000, 16, np.random.default_rng(5)
    uv = synth.fr(rng.uniform(96, 104, size=(n, 2)))
    vals = (1 + 0.5 * synth.normal_vals(rng, n)).astype(np.complex64)
    o = opts(gcf_kind=gg.GCF_GAUSSIAN)
    d = device(uv, vals, None, N * N)
    ctx.grid(o, d[3], *d[:3], N, S)
    torch.cuda.synchronize()
    check(d[3], o, uv, vals, synth.gcf_table(synth.gaussian_gcf_1d(S)), N, S)


@pytest.mark.parametrize("layout", [gg.LAYOUT_INTERLEAVED, gg.LAYOUT_PLANAR])
def test_grid_aligned_to_one_float(ctx, layout):
    N, n, S, rng = 60, 3000, 8, np.random.default_rng(12)
    uv, vals = synth.fr(rng.uniform(0, N, size=(n, 2))), synth.normal_vals(rng, n)
    gcf, o = table(S, 8, "complex", rng), opts(layout=layout)
    d_uv, d_vals, d_gcf, g = device(uv, vals, gcf, N * N + 1)
    job = gg.Context.make_job(g, d_uv, d_vals, d_gcf, N, S)
    job.out += 4
    ctx.grid_job(o, job)
    torch.cuda.synchronize()
    cells = torch.view_as_real(g).reshape(-1)[1:-1].clone()
    check(torch.view_as_complex(cells.reshape(-1, 2)), o, uv, vals, gcf, N, S)


def test_accumulate_and_mixed_batch(ctx):
    """twice into the same grids; support 32 keeps the 32-cell tiles"""
    rng, n = np.random.default_rng(8), 2000
    o = opts(accumulate=True)
    tabs = {S: table(S, 8, "real", rng) for S in (8, 16, 32)}
    sets, jobs = [], []
    for N, S in ((70, 8), (45, 32), (90, 16), (33, 8)):
        uv = synth.fr(rng.uniform(0, N, size=(n, 2)))
        vals = synth.normal_vals(rng, n)
        d = device(uv, vals, tabs[S], N * N, fill=0.0)
        if any(s[3] == S for s in sets):  # one table per support
            d = (d[0], d[1], next(s[4][2] for s in sets if s[3] == S), d[3])
        sets.append((uv, vals, N, S, d))
        jobs.append(gg.Context.make_job(d[3], d[0], d[1], d[2], N, S))
    ctx.grid_batch(o, jobs)
    ctx.grid_batch(o, jobs)
    torch.cuda.synchronize()
    for uv, vals, N, S, d in sets:
        check(d[3], o, uv, vals, tabs[S], N, S, scale=2.0)


@pytest.mark.parametrize("N", [64, 1200])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("S", [8, 16])
def test_values_that_are_not_finite_stay_in_their_footprint(ctx, S, N, bad):
    n, rng = 500, np.random.default_rng(3)
    uv = synth.fr(rng.uniform(10, 60, size=(n, 2)))
    vals = synth.normal_vals(rng, n)
    odd = vals.copy()
    odd[7] = bad
    vals[7] = 0
    gcf = table(S, 8, "real", rng)
    o = opts()
    d = device(uv, odd, gcf, N * N)
    ctx.grid(o, d[3], *d[:3], N, S)
    torch.cuda.synchronize()
    got = planar_from_grid(torch.view_as_real(d[3]).reshape(-1).cpu().numpy(), 1, N, False)[:, 0]
    ref = O.grid_pz(uv, pairs(vals), pairs(gcf), N, S, nthreads=8)[:, 0]
    x0, y0 = np.floor(uv[7]).astype(int) - S // 2 + 1
    inside = np.zeros((N, N), bool)
    inside[max(0, y0):y0 + S, max(0, x0):x0 + S] = True
    assert not np.isfinite(got[0][inside]).any()
    assert np.isfinite(got[:, ~inside]).all()
    assert rel_err(got[:, ~inside], ref[:, ~inside]) <= 1e-6
