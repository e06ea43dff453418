"""The moving window with several tables, of which those without imaginary parts
take real products (as a single one does): a component of a value that is not
finite stays in its own component of the grid, and tables of both kinds in one
call, given by index or by job, each take their own way.  Against the CPU oracle:
compensated 1e-6, plain 2e-6, normwise, as for every moving window."""
import numpy as np
import pytest

import gpugrid as gg
import oracle as O
import synth
from helpers import planar_from_grid, rel_err

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


def stack(S, kinds, rng):
    """tables scaled apart by powers of two, so that a mixed-up one shows"""
    out = []
    for k, kind in enumerate(kinds):
        t = synth.gcf_table(synth.gaussian_gcf_1d(S)).astype(complex) * 2.0 ** (3 * k)
        if kind == "complex":
            t = t * np.exp(1j * rng.uniform(0, 6, t.shape))
        elif kind == "one":
            t[5, S - 1, S // 2] += 0.25j * 2.0 ** (3 * k)
        out.append(t.astype(np.complex64))
    return np.stack(out)


@pytest.mark.parametrize("accum,tol", [(gg.ACC_COMPENSATED, 1e-6), (gg.ACC_PLAIN, 2e-6)])
@pytest.mark.parametrize("S,P,N,n", [(8, 1, 70, 900), (8, 2, 300, 5000), (16, 1, 90, 700),
                                     (16, 4, 60, 4000), (16, 3, 200, 300)])
def test_tables_of_both_kinds(ctx, S, P, N, n, accum, tol):
    rng = np.random.default_rng(S + n)
    kinds = ["real", "complex", "one", "real"]
    tabs = stack(S, kinds, rng)
    uv = synth.fr(rng.uniform(-S, N + S, size=(n, 2)))
    vals = synth.normal_vals(rng, n * P, np.complex64)
    index = rng.integers(len(kinds), size=n).astype(np.int32)
    out = torch.full((P * N * N,), float("nan"), device="cuda", dtype=torch.complex64)
    o = gg.Options(mode=gg.MODE_WINDOW, accum=accum, layout=gg.LAYOUT_INTERLEAVED, polarizations=P)
    dev = [torch.from_numpy(a).cuda() for a in (uv, vals, tabs.reshape(-1), index)]
    ctx.grid_job(o, gg.Context.make_job(out, *dev[:3], N, S, npts=n, gcf_index=dev[3],
                                        n_gcf=len(kinds)))
    torch.cuda.synchronize()
    got = planar_from_grid(torch.view_as_real(out).reshape(-1).cpu().numpy(), P, N, False)
    v = vals.reshape(n, P)
    ref = sum(O.grid_pz(uv[index == k], pairs(v[index == k]), pairs(tabs[k]), N, S, pols=P)
              for k in range(len(kinds)))
    assert rel_err(got, ref) <= tol


@pytest.mark.parametrize("S", [8, 16])
def test_a_table_of_its_own_for_every_job(ctx, S):
    rng = np.random.default_rng(S)
    kinds = ["complex", "real", "one"]
    tabs = stack(S, kinds, rng)
    todo, keep = [], []
    for k, N in enumerate((50, 200, 90)):
        uv = synth.fr(rng.uniform(-S, N + S, size=(700, 2)))
        vals = synth.normal_vals(rng, 700, np.complex64)
        d = [torch.from_numpy(a).cuda() for a in (uv, vals, tabs[k].reshape(-1))]
        out = torch.full((N * N,), float("nan"), device="cuda", dtype=torch.complex64)
        todo.append(gg.Context.make_job(out, *d, N, S))
        keep.append((out, d, uv, vals, N))
    ctx.grid_batch(gg.Options(mode=gg.MODE_WINDOW, accum=gg.ACC_COMPENSATED,
                              layout=gg.LAYOUT_INTERLEAVED), todo)
    torch.cuda.synchronize()
    for k, (out, _, uv, vals, N) in enumerate(keep):
        got = planar_from_grid(torch.view_as_real(out).reshape(-1).cpu().numpy(), 1, N, False)
        assert rel_err(got, O.grid_pz(uv, pairs(vals), pairs(tabs[k]), N, S)) <= 1e-6


@pytest.mark.parametrize("accum", [gg.ACC_COMPENSATED, gg.ACC_PLAIN])
@pytest.mark.parametrize("S", [8, 16])
def test_components_that_are_not_finite_stay_apart(ctx, S, accum):
    N, n = 120, 300
    rng = np.random.default_rng(S)
    tabs = stack(S, ["real", "real"], rng)
    uv = synth.fr(rng.uniform(40, 80, size=(n, 2)))
    vals = synth.normal_vals(rng, n, np.complex64)
    vals[3], vals[7] = complex(1.0, np.inf), complex(np.nan, -2.0)
    index = rng.integers(2, size=n).astype(np.int32)
    out = torch.full((N, N), float("nan"), device="cuda", dtype=torch.complex64)
    o = gg.Options(mode=gg.MODE_WINDOW, accum=accum, layout=gg.LAYOUT_INTERLEAVED)
    dev = [torch.from_numpy(a).cuda() for a in (uv, vals, tabs.reshape(-1), index)]
    ctx.grid_job(o, gg.Context.make_job(out, *dev[:3], N, S, npts=n, gcf_index=dev[3], n_gcf=2))
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    for part, q in ((got.imag, 3), (got.real, 7)):
        x0, y0 = np.floor(uv[q]).astype(int) - S // 2 + 1
        bad = np.zeros((N, N), bool)
        bad[y0:y0 + S, x0:x0 + S] = True
        assert not np.isfinite(part[bad]).any() and np.isfinite(part[~bad]).all()
