"""Reserving for gather covers grids aligned to one float, which take the general
kernel with a workspace of its own: the call allocates nothing."""
import numpy as np
import pytest

import gpugrid as gg
import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("S", [8, 16])
@pytest.mark.parametrize("first", [0, 1])
def test_reserved_workspace_holds(S, first):
    N, n = 64, 300
    rng = np.random.default_rng(S)
    ctx = gg.Context(0)
    o = gg.Options(mode=gg.MODE_GATHER, accum=gg.ACC_COMPENSATED, layout=gg.LAYOUT_INTERLEAVED)
    ctx.reserve(o, n, N, S, gg.C64)
    before = ctx.workspace_bytes()
    uv = torch.from_numpy(synth.fr(rng.uniform(0, N, size=(n, 2)))).cuda()
    vals = torch.from_numpy(synth.normal_vals(rng, n, np.complex64)).cuda()
    gcf = torch.from_numpy(synth.gcf_table(synth.gaussian_gcf_1d(S)).astype(np.complex64)).cuda()
    out = torch.empty(2 * N * N + 2, device="cuda")[first:first + 2 * N * N]
    ctx.grid(o, out, uv, vals, gcf.reshape(-1), N, S)
    torch.cuda.synchronize()
    assert ctx.workspace_bytes() == before
    ctx.close()
