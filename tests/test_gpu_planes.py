"""Several polarisations of an odd number of visibilities: the sorted values of
the planes then start at odd multiples of 8 bytes unless the distance between
planes is rounded up, and the bulk copies of window_kernel and gather_kernel
need 16-byte boundaries.  Against the CPU oracle; tolerances as for every FP32
path (compensated, normwise 1e-6).
"""
import numpy as np
import pytest

import gpugrid as gg
import oracle as O
import synth
from helpers import planar_from_grid, rel_err

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def pairs(c):
    c = np.asarray(c).reshape(-1)
    return np.stack([c.real, c.imag], -1).astype(np.float64)


@pytest.mark.parametrize("mode", [gg.MODE_WINDOW, gg.MODE_GATHER])
@pytest.mark.parametrize("S,P,n", [(4, 2, 1001), (4, 3, 777), (8, 2, 1501), (16, 3, 501),
                                   (32, 2, 301), (32, 4, 65)])
def test_odd_counts(S, P, n, mode):
    N, rng = 70, np.random.default_rng(S + P)
    uv = synth.fr(rng.uniform(0, N, size=(n, 2)))
    vals = synth.normal_vals(rng, n * P)
    gcf = synth.gcf_table(synth.gaussian_gcf_1d(S)).astype(np.complex64)
    o = gg.Options(mode=mode, accum=gg.ACC_COMPENSATED, layout=gg.LAYOUT_INTERLEAVED,
                   polarizations=P, tile=32)   # the general kernels
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (uv, vals, gcf.reshape(-1))]
    out = torch.full((P * N * N,), float("nan"), dtype=torch.complex64, device="cuda")
    with gg.Context(0) as c:
        c.grid_job(o, gg.Context.make_job(out, *d, N, S))
        torch.cuda.synchronize()
        assert c.read_flags() == [0, 0, 0, 0]
    got = planar_from_grid(torch.view_as_real(out).reshape(-1).cpu().numpy(), P, N, False)
    ref = O.grid_pz(uv, pairs(vals), pairs(gcf), N, S, pols=P, nthreads=8)
    assert rel_err(got, ref) <= 1e-6
