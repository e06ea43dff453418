"""The register-tile moving window (8-cell uv tiles, supports 8 and 16, FP32
values) at the sizes where it can go wrong: blocks of records around its
sorting block of 128 and its runs of 16, every footprint position in a tile,
tiles cut into several items, grids smaller than a tile, coordinates around
the grid's edges, real, complex and per-CTA Gaussian tables, oversamplings,
polarisations, and values that are not finite.  Against the CPU oracle on the
GPU's inputs; tolerances as for every FP32 path: compensated 1e-6, plain 2e-6
(normwise), per cell 1e-6 and 1e-5.
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


def table(S, G, kind, rng):
    if kind == "real":
        return synth.gcf_table(synth.gaussian_gcf_1d(S, G)).astype(np.complex64)
    t = rng.standard_normal((G * G, S, S)) + 1j * rng.standard_normal((G * G, S, S))
    return t.astype(np.complex64)


def grid(ctx, o, uv, vals, gcf, N, S, out=torch.complex64):
    P = o.polarizations
    d_uv = torch.from_numpy(np.ascontiguousarray(uv)).cuda()
    d_v = torch.from_numpy(np.ascontiguousarray(vals)).cuda()
    d_g = None if gcf is None else torch.from_numpy(gcf.reshape(-1)).cuda()
    g = torch.full((P * N * N,), float("nan"), dtype=out, device="cuda")
    ctx.grid(o, g, d_uv, d_v, d_g, N, S)
    torch.cuda.synchronize()
    assert ctx.read_flags() == [0, 0, 0, 0]
    host = torch.view_as_real(g).reshape(-1).cpu().numpy()
    return planar_from_grid(host, P, N, o.layout == gg.LAYOUT_PLANAR)


def check(got, uv, vals, gcf, N, S, P, G, comp):
    ref = O.grid_pz(uv, pairs(vals), pairs(gcf), N, S, pols=P, gcf_grid=G, nthreads=8)
    mag = O.grid_mag(uv, pairs(vals), pairs(gcf), N, S, pols=P, gcf_grid=G, nthreads=8)
    assert rel_err(got, ref) <= (1e-6 if comp else 2e-6)
    assert cell_err(got, ref, mag)[0] <= (1e-6 if comp else 1e-5)


@pytest.mark.parametrize("comp", [True, False])
@pytest.mark.parametrize("kind", ["real", "complex"])
@pytest.mark.parametrize("S", [8, 16])
@pytest.mark.parametrize("n", [1, 2, 15, 17, 33, 127, 128, 129, 257, 1500])
def test_one_tile_block_sizes(ctx, n, S, kind, comp):
    """n records of one tile: blocks, runs and read-ahead at their edges"""
    N, rng = 48, np.random.default_rng(n)
    uv = synth.fr(rng.uniform(16, 24, size=(n, 2)))
    vals = synth.normal_vals(rng, n)
    gcf = table(S, 8, kind, rng)
    o = gg.Options(mode=gg.MODE_WINDOW, accum=gg.ACC_COMPENSATED if comp else gg.ACC_PLAIN,
                   layout=gg.LAYOUT_INTERLEAVED)
    check(grid(ctx, o, uv, vals, gcf, N, S), uv, vals, gcf, N, S, 1, 8, comp)


@pytest.mark.parametrize("chunk", [0, 32, 100])
@pytest.mark.parametrize("S", [8, 16])
@pytest.mark.parametrize("N,G,P,layout,out", [
    (3, 8, 1, gg.LAYOUT_INTERLEAVED, torch.complex64),
    (8, 4, 2, gg.LAYOUT_PLANAR, torch.complex64),
    (61, 8, 3, gg.LAYOUT_INTERLEAVED, torch.complex64),
    (64, 1, 1, gg.LAYOUT_INTERLEAVED, torch.complex128),
    (131, 2, 1, gg.LAYOUT_PLANAR, torch.complex128)])
def test_edges_layouts_and_items(ctx, N, G, P, layout, out, S, chunk):
    """coordinates on every side of the grid, items of a few records"""
    rng = np.random.default_rng(N + S)
    uv = synth.fr(rng.uniform(-S, N + S, size=(3000, 2)))
    uv[:9] = [[0, 0], [N - 1, N - 1], [-S / 2, 1], [1, -S / 2], [N + S / 2 - 1, 0],
              [0, N + S / 2 - 1], [N - 0.5, 0.25], [-0.5, N], [7.875, 8]]
    vals = synth.normal_vals(rng, 3000 * P)
    gcf = table(S, G, "real" if P == 1 else "complex", rng)
    o = gg.Options(mode=gg.MODE_WINDOW, accum=gg.ACC_COMPENSATED, layout=layout,
                   oversample=G, polarizations=P, window_chunk=chunk)
    check(grid(ctx, o, uv, vals, gcf, N, S, out), uv, vals, gcf, N, S, P, G, True)


@pytest.mark.parametrize("kind", ["real", "complex"])
@pytest.mark.parametrize("S,G,P,ntab,n", [(8, 8, 1, 3, 4000), (16, 8, 2, 5, 3000),
                                          (16, 16, 1, 1, 900), (8, 16, 3, 2, 2000),
                                          (16, 8, 4, 2, 40000), (16, 4, 3, 7, 5000),
                                          (8, 8, 4, 4, 30000), (16, 8, 5, 2, 1500)])
def test_tables_in_global_memory(ctx, S, G, P, ntab, n, kind):
    """per-visibility tables, one too large for shared memory, and (below) a
    table for each job of a batch"""
    N, rng = 90, np.random.default_rng(S + G)
    uv = synth.fr(rng.uniform(-S, N + S, size=(n, 2)))
    vals = synth.normal_vals(rng, n * P)
    tabs = np.concatenate([table(S, G, kind, rng) * np.float32(1 + t) for t in range(ntab)])
    idx = rng.integers(0, ntab, n).astype(np.int32)
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (uv, vals, tabs.reshape(-1), idx)]
    out = torch.full((P * N * N,), float("nan"), dtype=torch.complex64, device="cuda")
    o = gg.Options(mode=gg.MODE_WINDOW, accum=gg.ACC_COMPENSATED, layout=gg.LAYOUT_INTERLEAVED,
                   oversample=G, polarizations=P)
    ctx.grid_job(o, gg.Context.make_job(out, d[0], d[1], d[2], N, S,
                                        gcf_index=d[3] if ntab > 1 else None, n_gcf=ntab))
    torch.cuda.synchronize()
    assert ctx.read_flags() == [0, 0, 0, 0]
    got = planar_from_grid(torch.view_as_real(out).reshape(-1).cpu().numpy(), P, N, False)
    for p in range(P):
        v = vals.reshape(n, P)[:, p].copy()
        ref = O.grid_pz_gcfinx(uv, v, idx, tabs.reshape(-1), N, S, gcf_grid=G, nthreads=8)
        mag = O.grid_mag(uv, pairs(v), pairs(tabs), N, S, gcf_grid=G, gcfinx=idx, nthreads=8)
        assert rel_err(got[:, p:p + 1], ref) <= 1e-6
        assert cell_err(got[:, p:p + 1], ref, mag)[0] <= 1e-6


def test_a_table_for_each_job(ctx):
    S, n, rng = 16, 2500, np.random.default_rng(2)
    o = gg.Options(mode=gg.MODE_WINDOW, accum=gg.ACC_COMPENSATED, layout=gg.LAYOUT_INTERLEAVED)
    sets, jobs = [], []
    for N in (40, 77, 120):
        uv = synth.fr(rng.uniform(0, N, size=(n, 2)))
        vals, gcf = synth.normal_vals(rng, n), table(S, 8, "complex", rng)
        d = [torch.from_numpy(a).cuda() for a in (uv, vals, gcf.reshape(-1))]
        g = torch.full((N * N,), float("nan"), dtype=torch.complex64, device="cuda")
        sets.append((uv, vals, gcf, N, d, g))
        jobs.append(gg.Context.make_job(g, *d, N, S))
    ctx.grid_batch(o, jobs)
    torch.cuda.synchronize()
    for uv, vals, gcf, N, d, g in sets:
        host = torch.view_as_real(g).reshape(-1).cpu().numpy()
        check(planar_from_grid(host, 1, N, False), uv, vals, gcf, N, S, 1, 8, True)


@pytest.mark.parametrize("kind", [gg.GCF_TABLE, gg.GCF_GAUSSIAN])
def test_reserved_workspace_holds_smaller_jobs(kind):
    """items get shorter with the job, so a smaller job has more of them for
    its records: none of these may outgrow the workspace reserved for the largest"""
    N, nmax = 2048, 3_000_000
    o = gg.Options(mode=gg.MODE_WINDOW, accum=gg.ACC_COMPENSATED, gcf_kind=kind,
                   layout=gg.LAYOUT_INTERLEAVED)
    uv = torch.zeros(2 * nmax, dtype=torch.float32, device="cuda")   # inside: tile 0 only
    vals = torch.zeros(nmax, dtype=torch.complex64, device="cuda")
    gcf = torch.zeros(64 * 256, dtype=torch.complex64, device="cuda")
    out = torch.empty(N * N, dtype=torch.complex64, device="cuda")
    with gg.Context(0) as c:
        c.reserve(o, nmax, N, 32 if kind == gg.GCF_GAUSSIAN else 16)
        held = c.workspace_bytes()
        for S in (16, 8, 4):
            for n in (nmax, 2_000_000, 1_245_185, 700_001, 622_593, 400_000, 50_000, 777, 1):
                kw = {"gcf_sigma": S / 6.0} if kind == gg.GCF_GAUSSIAN else {}
                c.grid_job(o, gg.Context.make_job(out, uv[:2 * n], vals[:n],
                                                  None if kw else gcf, N, S, **kw))
                assert c.workspace_bytes() == held, (S, n)
        torch.cuda.synchronize()


@pytest.mark.parametrize("S", [8, 16])
def test_gaussian(ctx, S):
    N, rng = 200, np.random.default_rng(S)
    uv = synth.fr(rng.uniform(0, N, size=(20000, 2)))
    vals = synth.normal_vals(rng, 20000)
    o = gg.Options(mode=gg.MODE_WINDOW, accum=gg.ACC_COMPENSATED, layout=gg.LAYOUT_INTERLEAVED,
                   gcf_kind=gg.GCF_GAUSSIAN)
    got = grid(ctx, o, uv, vals, None, N, S)
    check(got, uv, vals, synth.gcf_table(synth.gaussian_gcf_1d(S)), N, S, 1, 8, True)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("comp", [True, False])
@pytest.mark.parametrize("S", [8, 16])
def test_values_that_are_not_finite_stay_in_their_footprint(ctx, S, comp, bad):
    """a NaN or infinite value reaches the cells of its footprint only; the
    others hold the sums without it"""
    N, n, rng = 64, 400, np.random.default_rng(3)
    uv = synth.fr(rng.uniform(16, 40, size=(n, 2)))
    vals = synth.normal_vals(rng, n)
    gcf = table(S, 8, "real", rng)
    o = gg.Options(mode=gg.MODE_WINDOW, accum=gg.ACC_COMPENSATED if comp else gg.ACC_PLAIN,
                   layout=gg.LAYOUT_INTERLEAVED)
    odd = vals.copy()
    odd[7] = bad
    vals[7] = 0
    got = grid(ctx, o, uv, odd, gcf, N, S)[:, 0]
    ref = O.grid_pz(uv, pairs(vals), pairs(gcf), N, S, nthreads=8)[:, 0]
    x0, y0 = (np.floor(uv[7]).astype(int) - S // 2 + 1)
    inside = np.zeros((N, N), bool)
    inside[y0:y0 + S, x0:x0 + S] = True
    assert not np.isfinite(got[0][inside]).any()
    assert np.isfinite(got[:, ~inside]).all()
    assert rel_err(got[:, ~inside], ref[:, ~inside]) <= (1e-6 if comp else 2e-6)
