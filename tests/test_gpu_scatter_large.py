"""Compensated scatter by support 16 on both sides of the count from which its launch
holds more CTAs.  Against the CPU oracle, normwise 1e-6."""
import numpy as np
import pytest

import gpugrid as gg
import oracle as O
import synth
from helpers import planar_from_grid, rel_err

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [(1 << 21) - 1, 1 << 21])
def test_support_16(n):
    S, N = 16, 200
    rng = np.random.default_rng(n)
    uv = synth.fr(rng.uniform(-S, N + S, size=(n, 2)))
    vals = synth.normal_vals(rng, n, np.complex64)
    gcf = synth.gcf_table(synth.gaussian_gcf_1d(S)).astype(np.complex64)
    pairs = lambda c: np.stack([c.real, c.imag], -1).reshape(-1, 2).astype(np.float64)
    out = torch.full((N * N,), float("nan"), device="cuda", dtype=torch.complex64)
    ctx = gg.Context(0)
    ctx.grid(gg.Options(mode=gg.MODE_SCATTER, accum=gg.ACC_COMPENSATED,
                        layout=gg.LAYOUT_INTERLEAVED), out,
             *(torch.from_numpy(a).cuda() for a in (uv, vals, gcf.reshape(-1))), N, S)
    torch.cuda.synchronize()
    got = planar_from_grid(torch.view_as_real(out).reshape(-1).cpu().numpy(), 1, N, False)
    ctx.close()
    assert rel_err(got, O.grid_pz(uv, pairs(vals), pairs(gcf), N, S, nthreads=8)) <= 1e-6
