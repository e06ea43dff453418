"""Compensated gridding loses no more than a two-sum of single taps would.

Into a complex128 grid nothing is rounded but the taps and their sums.  Errors are
rounding errors of random sign, so their variances add: a product rounded to
nearest has a relative error of rms 0.425 u, u = 2^-24 (uniform within half a unit
in the last place, significand with density 1/m).  Call its square one unit.  A tap
by a real factor rounds once: 1 unit of its square; by a complex factor it is two
products, the first rounded to half the tap's square on average and the tap
itself: 1.5; by the Gaussian the product of the factors of both axes and the tap:
2.  Exact sums add nothing; runs of sixteen plainly summed taps would take 8.5.  The statistic is
over the cells, relative to the sum of the squares of the taps of each, and within
2 % of its mean.
"""
import numpy as np
import pytest

import gpugrid as gg
import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
G = 8


@pytest.fixture(scope="module")
def ctx():
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    c = gg.Context(0)
    yield c
    c.close()


def sums(uv, vals, tabs, index, N, S):
    """exact sums of the taps, and of their squares, by cell"""
    fl = np.floor(uv)
    sub = np.floor(G * (uv - fl)).astype(int)
    first = fl.astype(int) - S // 2 + 1
    k = np.arange(S)
    cell = (first[:, 1, None, None] + k[:, None]) * N + first[:, 0, None, None] + k
    t = vals.astype(complex)[:, None, None] * tabs.astype(complex)[index, sub[:, 1] * G + sub[:, 0]]
    c = cell.reshape(-1)
    add = lambda w: np.bincount(c, weights=w.reshape(-1), minlength=N * N)
    return add(t.real) + 1j * add(t.imag), add(np.abs(t) ** 2)


def statistic(got, exact, squares):
    hit = squares > 0
    return np.sqrt((np.abs(got.reshape(-1) - exact)[hit] ** 2 / squares[hit]).mean())


def run(ctx, S, n, tabs, index, uv, vals, N, **opts):
    out = torch.full((N * N,), float("nan"), device="cuda", dtype=torch.complex128)
    o = gg.Options(accum=gg.ACC_COMPENSATED, layout=gg.LAYOUT_INTERLEAVED, **opts)
    dev = [torch.from_numpy(uv).cuda(), torch.from_numpy(vals).cuda()]
    tab = None if tabs is None else torch.from_numpy(tabs.reshape(-1)).cuda()
    ix = None if index is None else torch.from_numpy(index.astype(np.int32)).cuda()
    ctx.grid_job(o, gg.Context.make_job(out, *dev, tab, N, S, npts=n, gcf_index=ix,
                                        n_gcf=1 if tabs is None else len(tabs)))
    torch.cuda.synchronize()
    return out.cpu().numpy()


def observation(S, n, N, seed):
    rng = np.random.default_rng(seed)
    uv = synth.fr(rng.uniform(S, N - S, size=(n, 2)))
    return rng, uv, synth.normal_vals(rng, n, np.complex64)


def tables(rng, k, S, kind):
    # factors of one size: all taps count
    t = rng.uniform(1, 2, size=(k, G * G, S, S)) * rng.choice([-1, 1], size=(k, G * G, S, S))
    if kind == "complex":
        t = t * np.exp(1j * rng.uniform(0, 2 * np.pi, t.shape))
    return t.astype(np.complex64)


@pytest.mark.parametrize("several", [False, True])
@pytest.mark.parametrize("kind,units", [("real", 1.0), ("complex", 1.5)])
@pytest.mark.parametrize("S,N,n", [(8, 120, 40_000), (8, 300, 9_000), (16, 120, 20_000)])
def test_error_of_register_tiles(ctx, S, N, n, kind, units, several):
    rng, uv, vals = observation(S, n, N, S + N)
    k = 3 if several else 1
    tabs = tables(rng, k, S, kind)
    index = rng.integers(k, size=n)
    got = run(ctx, S, n, tabs, index if several else None, uv, vals, N, mode=gg.MODE_WINDOW)
    assert statistic(got, *sums(uv, vals, tabs, index, N, S)) <= 1.03 * np.sqrt(units) * 0.425 * 2.0 ** -24


@pytest.mark.parametrize("S", [8, 16])
def test_values_that_grow_within_an_item(ctx, S):
    """values that double every 128 visibilities, all in one uv tile and item"""
    N, n = 200, 2000
    rng, uv, vals = observation(S, n, N, 3)
    uv = synth.fr(np.stack([rng.uniform(96, 104, n), rng.uniform(96, 104, n)], 1))
    vals *= np.exp2(np.arange(n) // 128).astype(np.float32)
    tabs = tables(rng, 1, S, "real")
    got = run(ctx, S, n, tabs, None, uv, vals, N, mode=gg.MODE_WINDOW, window_chunk=4096)
    # few large taps in every cell: the mean of fewer independent errors
    assert statistic(got, *sums(uv, vals, tabs, np.zeros(n, int), N, S)) <= 1.5 * 0.425 * 2.0 ** -24
