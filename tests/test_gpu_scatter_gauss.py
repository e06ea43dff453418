"""The on-the-fly Gaussian's factors are real: by the scatter method too, an
infinite or NaN component of a value reaches only its own component of the grid,
and no cell outside the footprint, whatever the types, sums and layout."""
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


@pytest.mark.parametrize("layout", [gg.LAYOUT_INTERLEAVED, gg.LAYOUT_PLANAR])
@pytest.mark.parametrize("accum", [gg.ACC_PLAIN, gg.ACC_COMPENSATED])
@pytest.mark.parametrize("vals_t,out_t", [(np.complex64, torch.complex64),
                                          (np.complex64, torch.complex128),
                                          (np.complex128, torch.complex128)])
@pytest.mark.parametrize("S", [4, 16, 32])
def test_components_that_are_not_finite_stay_apart(ctx, S, vals_t, out_t, accum, layout):
    N, n = 90, 40
    rng = np.random.default_rng(S)
    uv = synth.fr(rng.uniform(S, N - S, size=(n, 2)))
    vals = synth.normal_vals(rng, n, vals_t)
    vals[3], vals[7] = complex(1.0, np.inf), complex(np.nan, -2.0)
    out = torch.full((N * N,), float("nan"), device="cuda", dtype=out_t)
    o = gg.Options(mode=gg.MODE_SCATTER, accum=accum, gcf_kind=gg.GCF_GAUSSIAN, layout=layout)
    ctx.grid(o, out, torch.from_numpy(uv).cuda(), torch.from_numpy(vals).cuda(), None, N, S)
    torch.cuda.synchronize()
    got = torch.view_as_real(out).reshape(-1).cpu().numpy()
    re, im = (got.reshape(2, N, N) if layout == gg.LAYOUT_PLANAR
              else np.moveaxis(got.reshape(N, N, 2), -1, 0))
    for part, q in ((im, 3), (re, 7)):
        x0, y0 = np.floor(uv[q]).astype(int) - S // 2 + 1
        bad = np.zeros((N, N), bool)
        bad[y0:y0 + S, x0:x0 + S] = True
        assert not np.isfinite(part[bad]).any()
        assert np.isfinite(part[~bad]).all()
