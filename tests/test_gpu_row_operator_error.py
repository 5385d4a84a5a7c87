"""Error of line-sampled solves against FP64 where K^H r is the small difference of large terms: data weights far below
one, coil maps whose squares do not add up to one, solves of some hundred iterations and solves continued in short calls.

Tolerance: a NumPy model of the iteration in FP32 with the k-space dual r itself (complex64 pocketfft transforms) gives
`model` for each case; twice that.
"""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

# (C, H, W, seed, map scale, optimizer, Lambda, reduction, calls), model
CASES = [((8, 64, 72, 0, 2.5, "tgv_mri", 1.0, 0.01, [101]), 1.63e-7),
         ((1, 64, 64, 0, 2.5, "tgv_mri", 1.0, 0.01, [101]), 1.76e-7),
         ((3, 58, 31, 0, 2.5, "tgv_mri", 1.0, 0.01, [255]), 6.7e-8),  # padded rows, a prime length
         ((8, 96, 92, 0, 1.0, "tgv_mri", 1.0, 0.01, [255]), 2.07e-7),
         ((8, 64, 72, 0, 2.5, "tgv_mri", 1.0, 1.0, [100] * 4), 9.3e-8),
         ((4, 48, 48, 4, 1.0, "tgv_op", 0.25, 1.0, [1001]), 1.60e-7),
         ((4, 48, 48, 4, 1.0, "tgv_op", 0.1, 1.0, [1001]), 2.50e-7),
         ((4, 48, 48, 4, 1.0, "tgv_op", 0.0, 1.0, [1001]), 1.39e-7),
         ((4, 48, 48, 3, 1.0, "tv_op", 0.0, 1.0, [1001]), 2.47e-7)]


@pytest.mark.parametrize("case,model", CASES)
def test_error_is_that_of_the_k_space_dual(pdt, oracle, case, model):
    from primaldualtoolbox import synthetic

    C, H, W, seed, scale, opt, lam, red, calls = case
    d = synthetic.cartesian_case(C=C, H=H, W=W, roos=False, seed=seed, accel=4)
    sens, f = (d["sens"] * scale).astype(np.complex64), (d["rawdata"] * scale).astype(np.complex64)
    ax = (-2, -1)
    img = np.fft.ifft2(np.fft.ifftshift(f.astype(np.complex128) * d["mask"], axes=ax), axes=ax, norm="ortho")
    u0 = (np.conj(sens) * np.fft.fftshift(img, axes=ax)).sum(0).astype(np.complex64)
    op = pdt.mri.MriCartesianOperator()
    op.setCoilSens(sens)
    op.setMask(d["mask"])
    assert "solver=line_gram" in op.tuning()
    o = {"tgv_mri": pdt.mri.TgvMriOptimizer_2c3c, "tgv_op": pdt.mri.TgvOptimizer_2c3c,
         "tv_op": pdt.mri.TvOptimizerWithOp_2c3c}[opt]()
    prm = o.getParameters()
    a1 = float(np.float32(d["alpha1"]))
    if opt == "tgv_mri":
        prm.reduction = red
    else:
        prm.Lambda = lam
    if opt != "tv_op":
        prm.alpha1, prm.alpha0 = a1, 2 * a1
    o.setOperator(op)
    o.setNoisyData(f)
    getattr(o, "setInput0", getattr(o, "setInput0UV", None))(u0)
    for n in calls:
        prm.max_iter = n - 1
        o.solve()
    ref, state = oracle.op_solve("cartesian", sens, d["mask"], f, opt, alpha0=2 * a1, alpha1=a1, reduction=red, lam=lam,
                                 max_iter=sum(calls) - 1, u0=u0, prec=64, return_state=True)
    assert rel_l2(o.getResult(), ref) <= 2 * model
    # r carries the transforms' rounding of K u: relative to the data, and summed up to 1 / Lambda where it is not
    # drawn back by u
    sampled = (d["mask"] != 0).any(axis=0)
    r = state["r"].reshape(f.shape)
    assert np.linalg.norm((o.getField("r") - r)[:, :, sampled]) <= 1e-5 * np.linalg.norm(f)


def test_k_space_dual_at_the_end_has_fp32_rows(pdt, oracle):
    """Where the tuner keeps the tensor-core forward rows (TF32 triples, about 1e-6 off), r = K U - c f must not take
    them. The NumPy model's r is 1.23e-7 of |f| off after these 40 iterations; twice that."""
    from primaldualtoolbox import synthetic

    C, H, W = 8, 320, 250
    d = synthetic.cartesian_case(C=C, H=H, W=W, roos=False, seed=0, accel=4)
    op = pdt.mri.MriCartesianOperator()
    op.setCoilSens(d["sens"])
    op.setMask(d["mask"])
    if "rows_fwd=tensor_dft" not in op.tuning():
        pytest.skip("the tuner chose FP32 rows")
    o = pdt.mri.TgvMriOptimizer_2c3c()
    prm = o.getParameters()
    a1 = float(np.float32(d["alpha1"]))
    prm.max_iter, prm.reduction, prm.alpha1, prm.alpha0 = 39, 1.0, a1, 2 * a1
    o.setOperator(op)
    o.setNoisyData(d["rawdata"])
    u0 = op.adjoint(d["rawdata"])
    o.setInput0(u0)
    o.solve()
    _, state = oracle.op_solve("cartesian", d["sens"], d["mask"], d["rawdata"], "tgv_mri", alpha0=2 * a1, alpha1=a1,
                               reduction=1.0, max_iter=39, u0=u0, prec=64, return_state=True)
    sampled = (d["mask"] != 0).any(axis=0)
    diff = (o.getField("r") - state["r"].reshape(C, H, W))[:, :, sampled]
    assert np.linalg.norm(diff) <= 2.5e-7 * np.linalg.norm(d["rawdata"])
