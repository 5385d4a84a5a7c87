"""Masks of whole phase-encode lines: the solvers run K^H K row by row (pdt_gram.h) instead of the three
operator passes. Image and k-space dual against the FP64 oracle of the iteration, at transform lengths with a
compiled split of their own and at padded ones, one to many coils, mask values other than one.

Tolerance: an FP32 transform pair of length n <= 768 is off by at most about log2(n) 2^-23 = 1.2e-6 relative,
and the prox forgets it at rate 1 / (1 + sigma lambda), so r and K^H r stay within 9 x 1.2e-6 of |f| (sigma
1/8, lambda 1); u integrates tau times that over the iterations here, below 1e-5 of |u|.
"""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

TOL = 1e-5

# (C, H, W, roos, optimizer): W with a split of its own (48 .. 512), then padded rows (W odd, prime, tiny)
SHAPES = [(3, 24, 48, True, "tgv_mri"), (4, 16, 176, False, "tv_op"), (2, 12, 208, False, "tgv_op"),
          (1, 20, 272, False, "tgv_mri"), (5, 10, 304, False, "tgv_mri"), (33, 8, 368, False, "tgv_mri"),
          (2, 8, 512, False, "tgv_mri"), (3, 24, 32, False, "tgv_mri"),
          (2, 30, 7, False, "tgv_mri"), (3, 18, 23, False, "tv_op"), (4, 14, 50, True, "tgv_op"),
          (17, 9, 175, False, "tgv_mri"), (2, 6, 341, False, "tgv_mri"), (2, 321, 33, False, "tgv_mri")]


def _problem(C, H, W, roos, oracle, seed):
    rng = np.random.default_rng(seed)
    c = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    sens = c(C, H, W)
    sens /= np.linalg.norm(sens, axis=0, keepdims=True)
    mask = np.zeros((H, W), np.float32)
    cols = np.nonzero(rng.random(W) < 0.4)[0]
    mask[:, cols] = rng.choice([1.0, 0.5], len(cols)).astype(np.float32)
    mask[:, W // 2] = 1
    kind = "cartesian_roos" if roos else "cartesian"
    f = oracle.op_apply(kind, sens, mask, c(H // 2 if roos else H, W)).astype(np.complex64)
    return kind, sens, mask, f + 0.01 * c(C, H, W)


@pytest.mark.parametrize("C,H,W,roos,opt", SHAPES)
def test_line_mask_solves_match_oracle(pdt, oracle, C, H, W, roos, opt):
    kind, sens, mask, f = _problem(C, H, W, roos, oracle, C + H + W)
    op = (pdt.mri.MriCartesianRemoveROOSOperator if roos else pdt.mri.MriCartesianOperator)()
    op.setCoilSens(sens)
    op.setMask(mask)
    assert "solver=line_gram" in op.tuning()
    o = {"tgv_mri": pdt.mri.TgvMriOptimizer_2c3c, "tgv_op": pdt.mri.TgvOptimizer_2c3c,
         "tv_op": pdt.mri.TvOptimizerWithOp_2c3c}[opt]()
    prm = o.getParameters()
    kw = dict(alpha0=0.125, alpha1=0.0625, reduction=1.0, lam=1.0)
    if opt != "tv_op":
        prm.alpha0, prm.alpha1 = kw["alpha0"], kw["alpha1"]
    if opt != "tgv_mri":
        prm.Lambda = 1.0
    o.setOperator(op)
    o.setNoisyData(f)
    state = None
    for n in (24, 9):  # even and odd; the second continues, so the k-space dual of the first enters it
        prm.max_iter = n - 1
        o.solve()
        ref, state = oracle.op_solve(kind, sens, mask, f, opt, max_iter=n - 1, prec=64, state=state, return_state=True,
                                     **kw)
        assert rel_l2(o.getResult(), ref) <= TOL
    sampled = (mask != 0).any(axis=0)
    r = state["r"].reshape(f.shape)
    assert np.linalg.norm((o.getField("r") - r)[:, :, sampled]) <= 1e-5 * np.linalg.norm(f)
    for k in ("ubar", "px", "py") + (() if opt == "tv_op" else ("vbarx", "qxy")):
        ref = state[{"vbarx": "vbx"}.get(k, k)].reshape(o.getField(k).shape)
        assert np.linalg.norm(o.getField(k) - ref) <= TOL * max(np.linalg.norm(ref), np.linalg.norm(state["u"])), k


def test_other_masks_keep_the_three_passes(pdt):
    rng = np.random.default_rng(0)
    mask = (rng.random((20, 24)) < 0.5).astype(np.float32)
    op = pdt.mri.MriCartesianOperator()
    op.setCoilSens(np.ones((2, 20, 24), np.complex64))
    op.setMask(mask)
    assert "solver=line_gram" not in op.tuning()


# rows and columns whose transforms have radices 2 to 5, a prime of their own and a padded row; 256 iterations are the
# first number with K^H f as a pair of FP32 images
@pytest.mark.parametrize("C,H,W,roos,n", [(8, 96, 92, False, 1001), (3, 58, 31, False, 256), (5, 80, 48, True, 400)])
def test_long_solves_keep_the_k_space_duals_accuracy(pdt, oracle, C, H, W, roos, n):
    from primaldualtoolbox import synthetic

    case = synthetic.cartesian_case(C=C, H=H, W=W, roos=roos, seed=0)
    op = (pdt.mri.MriCartesianRemoveROOSOperator if roos else pdt.mri.MriCartesianOperator)()
    op.setCoilSens(case["sens"])
    op.setMask(case["mask"])
    assert "solver=line_gram" in op.tuning()
    o = pdt.mri.TgvMriOptimizer_2c3c()
    prm = o.getParameters()
    prm.max_iter, prm.reduction, prm.alpha1 = n - 1, 0.01, case["alpha1"]
    prm.alpha0 = 2 * prm.alpha1
    o.setOperator(op)
    o.setNoisyData(case["rawdata"])
    o.solve()
    ref = oracle.op_solve("cartesian_roos" if roos else "cartesian", case["sens"], case["mask"], case["rawdata"], "tgv_mri",
                          alpha0=float(prm.alpha0), alpha1=float(prm.alpha1), reduction=0.01, max_iter=n - 1, prec=64)
    # a NumPy model of the first case's 1001 iterations in FP32 ends 3.0e-7 off with the k-space dual, 3.3e-7 with the
    # row operator and K^H f in 64 bits, 1.2e-6 with K^H f in FP32; twice the middle one
    assert rel_l2(o.getResult(), ref) <= 6.6e-7
