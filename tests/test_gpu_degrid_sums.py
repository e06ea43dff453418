"""Compensated degridding loses no more than a two-sum of single taps would.

Errors are rounding errors of random sign, so their variances add.  A result
rounded to nearest has a relative error of rms 0.425 u, u = 2^-24 (uniform
within half a unit in the last place, significand with density 1/m); call its
square one unit.  In units, relative to the sum of the taps' squares:
 * every tap's product rounded, exact sums, result rounded: 1 + 1;
 * by a table with imaginary parts a tap is two products, the first rounded to
   half the tap's square on average and the tap itself: 0.5 + 1, and 1.
Runs of four plainly summed taps: 1 + 2 + 3 + 4 over four taps, and 1 (3.5).  The
statistic over 20,000 visibilities is within 2 % of its mean.
"""
import numpy as np
import pytest

import gpugrid as gg
import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def ctx():
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    c = gg.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("kind,units", [("real", 2.0), ("complex", 2.5)])
@pytest.mark.parametrize("S", [4, 8, 16])
def test_error_of_compensated_sums(ctx, S, kind, units):
    N, n, G = 200, 20_000, 8
    rng = np.random.default_rng(S)
    uv = synth.fr(rng.uniform(S, N - S, size=(n, 2)))
    # factors of one size: all taps count
    gcf = rng.uniform(1, 2, size=(G * G, S, S)) * rng.choice([-1, 1], size=(G * G, S, S))
    if kind == "complex":
        gcf = gcf * np.exp(1j * rng.uniform(0, 2 * np.pi, gcf.shape))
    gcf = gcf.astype(np.complex64)
    grid = synth.normal_vals(rng, N * N, np.complex64).reshape(N, N)
    out = torch.full((n,), float("nan"), device="cuda", dtype=torch.complex64)
    ctx.degrid(gg.Options(accum=gg.ACC_COMPENSATED), torch.from_numpy(grid).cuda(),
               torch.from_numpy(uv).cuda(), out, torch.from_numpy(gcf.reshape(-1)).cuda(), N, S)
    torch.cuda.synchronize()
    fl = np.floor(uv)
    sub = np.floor(G * (uv - fl)).astype(int)
    first = fl.astype(int) - S // 2 + 1
    k = np.arange(S)
    c = grid[first[:, 1, None, None] + k[:, None], first[:, 0, None, None] + k].astype(complex)
    t = c * np.conj(gcf[sub[:, 1] * G + sub[:, 0]].astype(complex))
    err = np.abs(out.cpu().numpy() - t.sum((1, 2))) ** 2 / (np.abs(t) ** 2).sum((1, 2))
    assert np.sqrt(err.mean()) <= 1.03 * np.sqrt(units) * 0.425 * 2.0 ** -24
