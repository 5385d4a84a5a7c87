"""Denoising with several iterations per launch (pdt_denoise.cu): image sizes around the edges of a block's region, of
its inner part and of the rules that choose the iterations per launch and the region; iteration counts that leave a
short last launch or are shorter than one. Against the FP64 oracle.

Tolerance: each FP32 iteration adds a relative rounding error of a few 2^-24 to every variable and the iteration does
not amplify it (steps tau sigma |K|^2 <= 1), so 25 iterations stay within 25 x 4 x 6e-8 = 6e-6.
"""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

TOL = 1e-5
# one block (32 x 32 and less); 8 iterations a launch (inner part 16 x 16); 6 (20 x 20); 3 on the three regions
SIZES = [(32, 32), (33, 32), (1, 33), (16, 48), (17, 49), (31, 65), (181, 182), (200, 200), (363, 362), (640, 625), (633, 641)]


@pytest.mark.parametrize("tgv", [False, True])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("H,W", SIZES)
def test_regions_match_oracle(pdt, oracle, H, W, cplx, tgv):
    rng = np.random.default_rng(H * 1000 + W)
    f = rng.random((H, W)).astype(np.float32)
    if cplx:
        f = (f + 1j * rng.random((H, W))).astype(np.complex64)
    d = pdt.denoising
    o = (d.TgvOptimizer_2c if cplx else d.TgvOptimizer_2f)() if tgv else (d.TvOptimizer_2c if cplx else d.TvOptimizer_2f)()
    o.setNoisyData(f)
    p = o.getParameters()
    p.Lambda = 8.0
    kw = dict(alpha0=0.2, alpha1=0.1) if tgv else {}
    for k, v in kw.items():
        setattr(p, k, v)
    for iters in (25, 5, 1) if H * W < 40000 else (10,):
        p.max_iter = iters - 1
        o.setInput0UV(f)
        o.solve()
        ref = (oracle.tgv_solve if tgv else oracle.tv_solve)(f, lam=8.0, max_iter=iters - 1, prec=64, **kw)
        assert rel_l2(o.getResult(), ref) <= TOL
        # u-bar = 2 u - u of one iteration earlier, written by the last launch alone
        if iters > 1:
            p.max_iter = iters - 2
            q = o.getField("ubar")
            o.setInput0UV(f)
            o.solve()
            assert rel_l2(q, 2 * np.asarray(ref) - o.getResult()) <= TOL


def test_projection_of_overflowing_duals(pdt, oracle):
    """|p|^2 beyond FP32's range and alpha^2 too: 1 / max(1, inf / alpha) = 0. The FP32 oracle evaluates the same
    expression; four iterations of a few roundings of 2^-24 each stay within 1e-6."""
    rng = np.random.default_rng(5)
    f = (1e21 * rng.standard_normal((40, 48))).astype(np.float32)
    opt = pdt.denoising.TgvOptimizer_2f()
    prm = opt.getParameters()
    prm.max_iter, prm.Lambda, prm.alpha0, prm.alpha1 = 3, 10.0, 1e20, 1e20
    opt.setNoisyData(f)
    opt.solve()
    ref = oracle.tgv_solve(f, lam=10.0, alpha0=1e20, alpha1=1e20, max_iter=3, prec=32)
    assert np.isfinite(ref).all()
    assert rel_l2(opt.getResult(), ref) <= 1e-6
