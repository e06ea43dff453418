"""Support 32 with the on-the-fly Gaussian into a grid that holds values: the cells
that no footprint covers stay as they are, to the bit (a negative zero, a NaN with a
payload), and the others have the sums added.  Against the CPU oracle."""
import numpy as np
import pytest

import gpugrid as gg
import oracle as O
import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
S = 32


@pytest.fixture(scope="module")
def ctx():
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    c = gg.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("accum", [gg.ACC_PLAIN, gg.ACC_COMPENSATED])
@pytest.mark.parametrize("layout", [gg.LAYOUT_INTERLEAVED, gg.LAYOUT_PLANAR])
@pytest.mark.parametrize("real,P", [(torch.float32, 1), (torch.float32, 2), (torch.float64, 1)])
@pytest.mark.parametrize("N,n", [(200, 3), (2000, 40)])
def test_untouched_cells_keep_their_bits(ctx, N, n, real, P, layout, accum):
    rng = np.random.default_rng(n)
    uv = synth.fr(rng.uniform(S, N - S, size=(n, 2)))
    vals = synth.normal_vals(rng, n * P, np.complex64)
    dtype, bits = (np.float32, np.uint32) if real == torch.float32 else (np.float64, np.uint64)
    nan = np.array([0x7fc01234], np.uint32).view(np.float32) if dtype == np.float32 else \
        np.array([0x7ff8000000001234], np.uint64).view(np.float64)
    before = np.full(2 * P * N * N, -0.0, dtype)
    before[::3] = nan[0]
    cell = np.zeros((N, N), bool)
    for x, y in np.floor(uv).astype(int) - S // 2 + 1:
        cell[y:y + S, x:x + S] = True
    hit = (np.broadcast_to(cell, (2, P, N, N)) if layout == gg.LAYOUT_PLANAR
           else np.broadcast_to(cell[None, :, :, None], (P, N, N, 2))).reshape(-1)
    before[hit] = 0.5
    out = torch.from_numpy(before.copy()).cuda()
    o = gg.Options(mode=gg.MODE_WINDOW, accum=accum, gcf_kind=gg.GCF_GAUSSIAN, layout=layout,
                   polarizations=P, accumulate=True)
    job = gg.Context.make_job(out, torch.from_numpy(uv).cuda(), torch.from_numpy(vals).cuda(), None,
                              N, S, npts=n)
    job.out_type = gg.C64 if real == torch.float32 else gg.C128
    ctx.grid_job(o, job)
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    assert np.array_equal(got[~hit].view(bits), before[~hit].view(bits))
    g = synth.gcf_table(synth.gaussian_gcf_1d(S))
    pairs = lambda c: np.stack([c.real, c.imag], -1).reshape(-1, 2).astype(np.float64)
    ref = O.grid_pz(uv, pairs(vals), pairs(g.astype(complex)), N, S, pols=P)  # planar
    if layout == gg.LAYOUT_INTERLEAVED:
        ref = np.moveaxis(ref, 0, -1)
    err = np.abs(got.astype(np.float64) - 0.5 - np.ascontiguousarray(ref).reshape(-1))[hit].max()
    assert err <= 2e-6 * max(1.0, np.abs(ref).max())
