"""Degridding by tables without imaginary parts, with a single one and with all,
at counts of visibilities around a warp's 32 and a step's 32/S, on grids where
some or all footprints leave the grid, and from grids that are not finite.
Against the CPU oracle on the GPU's inputs; tolerances as for every degridding:
FP64 1e-12, compensated FP32 1e-6.
"""
import numpy as np
import pytest

import gpugrid as gg
import oracle as O
import synth

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


def degrid(ctx, uv, grid, tab, N, S):
    vals = torch.zeros(len(uv), dtype=torch.complex128 if tab.dtype == np.complex128
                       else torch.complex64, device="cuda")
    o = gg.Options(accum=gg.ACC_COMPENSATED, layout=gg.LAYOUT_INTERLEAVED)
    ctx.degrid(o, torch.from_numpy(grid).cuda(), torch.from_numpy(uv).cuda(), vals,
               torch.from_numpy(tab.reshape(-1)).cuda(), N, S)
    torch.cuda.synchronize()
    return vals.cpu().numpy()


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("kind", ["real", "one", "complex"])
@pytest.mark.parametrize("S,N,n", [(4, 10, 7), (4, 60, 33), (8, 7, 31), (8, 64, 32), (8, 90, 65),
                                   (16, 40, 1), (16, 120, 97), (32, 31, 33), (32, 130, 64)])
def test_tables_and_remainders(ctx, S, N, n, kind, dtype):
    rng = np.random.default_rng(n + S)
    uv = synth.fr(rng.uniform(-S / 2, N + S / 2, size=(n, 2)))
    uv[: n // 2] = synth.fr(rng.uniform(min(S, N / 2), max(N - S, N / 2), size=(n // 2, 2)))
    tab = synth.gcf_table(synth.gaussian_gcf_1d(S))
    if kind == "one":
        tab[:, S // 2, S - 1] += 0.25j
    elif kind == "complex":
        tab = tab * np.exp(1j * rng.uniform(0, 6, tab.shape))
    tab = tab.astype(dtype)
    grid = (rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))).astype(dtype)
    got = degrid(ctx, uv, grid, tab, N, S)
    planar = np.stack([grid.real, grid.imag]).astype(np.float64).reshape(2, 1, N, N)
    ref = O.degrid_pz(uv, planar, pairs(tab), N, S)
    ref = np.asarray(ref).reshape(n, -1)
    ref = ref[:, 0] + 1j * ref[:, 1] if ref.shape[1] == 2 else ref.reshape(-1)
    tol = 1e-12 if dtype == np.complex128 else 1e-6
    assert np.abs(got - ref).max() <= tol * np.abs(ref).max()


def test_grid_that_is_not_finite(ctx):
    """an infinite imaginary part times the zero imaginary part of a factor is
    NaN in the real part, as the complex product gives it"""
    N, S, n, rng = 48, 8, 40, np.random.default_rng(1)
    uv = synth.fr(rng.uniform(S, N - S, size=(n, 2)))
    uv[0] = [24.25, 24.5]
    tab = synth.gcf_table(synth.gaussian_gcf_1d(S)).astype(np.complex64)
    grid = np.ones((N, N), np.complex64)
    grid[24, 24] = complex(1, np.inf)
    got = degrid(ctx, uv, grid, tab, N, S)
    m = np.floor(uv).astype(int)
    hit = ((m[:, 0] - 3 <= 24) & (24 <= m[:, 0] + 4) & (m[:, 1] - 3 <= 24) & (24 <= m[:, 1] + 4))
    assert hit.any() and not hit.all()
    assert np.isnan(got.real[hit]).all() and not np.isfinite(got.imag[hit]).any()
    assert np.isfinite(got[~hit]).all()


@pytest.mark.parametrize("S,n", [(4, 1), (4, 640_001), (8, 5), (8, 4_999), (8, 622_592 + 3),
                                 (16, 9_731), (16, 40_003), (32, 4_865), (32, 1_217)])
def test_shares_of_the_warps(ctx, S, n):
    """a step or less for a warp, shares of several groups of 32, and groups dealt out"""
    N, rng = 70, np.random.default_rng(n)
    uv = synth.fr(rng.uniform(0, N, size=(n, 2)))
    tab = synth.gcf_table(synth.gaussian_gcf_1d(S)).astype(np.complex64)
    grid = (rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))).astype(np.complex64)
    got = degrid(ctx, uv, grid, tab, N, S)
    planar = np.stack([grid.real, grid.imag]).astype(np.float64).reshape(2, 1, N, N)
    ref = np.asarray(O.degrid_pz(uv, planar, pairs(tab), N, S, nthreads=8)).reshape(n, -1)
    ref = ref[:, 0] + 1j * ref[:, 1] if ref.shape[1] == 2 else ref.reshape(-1)
    assert np.abs(got - ref).max() <= 1e-6 * np.abs(ref).max()
