"""Compensated scatter by support 16 on both sides of the count from which its launch
holds more CTAs.  Against FP64 sums of the same values, normwise 1e-6."""
import numpy as np
import pytest

import gpugrid as gg
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
    ctx, grids = gg.Context(0), []
    for accum, ct in ((gg.ACC_COMPENSATED, np.complex64), (gg.ACC_PLAIN, np.complex128)):
        out = torch.full((N * N,), float("nan"), device="cuda",
                         dtype=torch.complex64 if ct == np.complex64 else torch.complex128)
        dev = [torch.from_numpy(a).cuda() for a in (uv, vals.astype(ct), gcf.reshape(-1).astype(ct))]
        ctx.grid(gg.Options(mode=gg.MODE_SCATTER, accum=accum, layout=gg.LAYOUT_INTERLEAVED), out,
                 *dev, N, S)
        torch.cuda.synchronize()
        grids.append(planar_from_grid(torch.view_as_real(out).reshape(-1).cpu().numpy(), 1, N, False))
    ctx.close()
    assert rel_err(*grids) <= 1e-6
