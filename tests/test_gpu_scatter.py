"""The scatter kernel's two ways through a tap, at every support: complex64 taps a
lane each, complex128 ones a component a lane, products by tables without
imaginary parts and with (also with a single one), coordinates on every side of
grids smaller and larger than a footprint, polarisations, batches whose jobs
change within a block of visibilities, and values that are not finite.
Against the CPU oracle on the GPU's inputs: FP64 1e-12, plain FP32 2e-6
(normwise; per cell 1e-5), as for every scatter.
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


def case(S, N, n, kind, f64, P=1, seed=0):
    rng = np.random.default_rng(seed + 7 * S + N)
    uv = synth.fr(rng.uniform(-S, N + S, size=(n, 2)))
    vals = synth.normal_vals(rng, n * P, np.complex128 if f64 else np.complex64)
    gcf = synth.gcf_table(synth.gaussian_gcf_1d(S))
    if kind == "complex":
        gcf = gcf * np.exp(1j * rng.uniform(0, 6, gcf.shape))
    elif kind == "one":
        gcf[9, S - 1, S // 2] += 0.25j
    return uv, vals, gcf.astype(vals.dtype)


def device(uv, vals, gcf, cells):
    return (torch.from_numpy(uv).cuda(), torch.from_numpy(vals).cuda(),
            torch.from_numpy(gcf.reshape(-1)).cuda(),
            torch.full((cells,), float("nan"), device="cuda",
                       dtype=torch.complex128 if vals.dtype == np.complex128 else torch.complex64))


def check(g, uv, vals, gcf, N, S, P):
    host = torch.view_as_real(g).reshape(-1).cpu().numpy()
    got = planar_from_grid(host, P, N, False)
    ref = O.grid_pz(uv, pairs(vals), pairs(gcf), N, S, pols=P, nthreads=8)
    mag = O.grid_mag(uv, pairs(vals), pairs(gcf), N, S, pols=P, nthreads=8)
    f64 = vals.dtype == np.complex128
    assert rel_err(got, ref) <= (1e-12 if f64 else 2e-6)
    assert cell_err(got, ref, mag)[0] <= (1e-12 if f64 else 1e-5)


@pytest.mark.parametrize("f64", [True, False])
@pytest.mark.parametrize("kind", ["real", "complex", "one"])
@pytest.mark.parametrize("S,N,P", [(4, 3, 1), (4, 50, 2), (8, 9, 1), (8, 70, 3), (16, 15, 1),
                                   (16, 77, 1), (32, 33, 2), (32, 101, 1)])
def test_supports_edges_and_tables(ctx, S, N, P, kind, f64):
    uv, vals, gcf = case(S, N, 700, kind, f64, P)
    d = device(uv, vals, gcf, P * N * N)
    o = gg.Options(mode=gg.MODE_SCATTER, layout=gg.LAYOUT_INTERLEAVED, polarizations=P)
    ctx.grid(o, d[3], *d[:3], N, S)
    torch.cuda.synchronize()
    assert ctx.read_flags() == [0, 0, 0, 0]
    check(d[3], uv, vals, gcf, N, S, P)


@pytest.mark.parametrize("f64", [True, False])
@pytest.mark.parametrize("n", [1, 31, 33, 1217, 19457, 40001])
def test_shares_of_the_warps(ctx, n, f64):
    """fewer visibilities than warps, shares of one or two groups of 32, uneven ones"""
    S, N, P = 8, 60, 1
    uv, vals, gcf = case(S, N, n, "real", f64, P)
    d = device(uv, vals, gcf, P * N * N)
    o = gg.Options(mode=gg.MODE_SCATTER, layout=gg.LAYOUT_INTERLEAVED, polarizations=P)
    ctx.grid(o, d[3], *d[:3], N, S)
    torch.cuda.synchronize()
    assert ctx.read_flags() == [0, 0, 0, 0]
    check(d[3], uv, vals, gcf, N, S, P)


@pytest.mark.parametrize("f64", [True, False])
def test_jobs_change_within_a_block(ctx, f64):
    sets = [case(8, N, n, kind, f64, seed=k)
            for k, (N, n, kind) in enumerate([(20, 30, "real"), (64, 5, "complex"),
                                              (33, 400, "one"), (90, 61, "real")])]
    sizes = [20, 64, 33, 90]
    dev = [device(*s, N * N) for s, N in zip(sets, sizes)]
    jobs = [gg.Context.make_job(d[3], d[0], d[1], d[2], N, 8) for d, N in zip(dev, sizes)]
    ctx.grid_batch(gg.Options(mode=gg.MODE_SCATTER, layout=gg.LAYOUT_INTERLEAVED), jobs)
    torch.cuda.synchronize()
    for (uv, vals, gcf), d, N in zip(sets, dev, sizes):
        check(d[3], uv, vals, gcf, N, 8, 1)


def test_fp64_values_that_are_not_finite(ctx):
    """an infinite component times a zero imaginary part is NaN, as in the
    reference's product, also with a table without imaginary parts"""
    N, S = 40, 16
    uv, vals, gcf = case(S, N, 50, "real", True)
    uv = synth.fr(np.clip(uv, 12, 28))
    vals[5] = complex(1.0, np.inf)
    d = device(uv, vals, gcf, N * N)
    ctx.grid(gg.Options(mode=gg.MODE_SCATTER, layout=gg.LAYOUT_INTERLEAVED), d[3], *d[:3], N, S)
    torch.cuda.synchronize()
    got = d[3].cpu().numpy().reshape(N, N)
    x0, y0 = np.floor(uv[5]).astype(int) - S // 2 + 1
    inside = np.zeros((N, N), bool)
    inside[y0:y0 + S, x0:x0 + S] = True
    assert np.isnan(got.real[inside]).all() and not np.isfinite(got.imag[inside]).any()
    assert np.isfinite(got.real[~inside]).all() and np.isfinite(got.imag[~inside]).all()


@pytest.mark.parametrize("n", [3_001, (1 << 21) - 1, 1 << 21])
def test_compensated_on_both_sides_of_the_large_calls(ctx, n):
    S, N, P = 4, 300, 1
    uv, vals, gcf = case(S, N, n, "real", False, P)
    d = device(uv, vals, gcf, N * N)
    o = gg.Options(mode=gg.MODE_SCATTER, accum=gg.ACC_COMPENSATED,
                   layout=gg.LAYOUT_INTERLEAVED)
    ctx.grid(o, d[3], *d[:3], N, S)
    torch.cuda.synchronize()
    got = planar_from_grid(torch.view_as_real(d[3]).reshape(-1).cpu().numpy(), P, N, False)
    ref = O.grid_pz(uv, pairs(vals), pairs(gcf), N, S, nthreads=8)
    assert rel_err(got, ref) <= 1e-6
