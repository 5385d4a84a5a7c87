"""The Cartesian operators' row passes on register transforms: row lengths of each kind against NumPy in double
precision, with ragged row blocks, one and many coils, and 2-D masks."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

# sizes of each kind of split (powers of two, primes 7 ... 23, Q = 8, 16, 24, 32), the smallest and the largest
WIDTHS = [48, 64, 80, 112, 176, 208, 240, 256, 272, 304, 336, 352, 368, 416, 480, 512, 576, 640]


def _reference(u, sens, mask):
    # kspace = mask . fftshift(FFT2(ifftshift(u . sens))) / sqrt(n); an odd or even length shifts by int((n + 1) / 2)
    axes = (-2, -1)
    x = np.fft.ifftshift(u[None] * sens, axes=axes) if sens is not None else np.fft.ifftshift(u[None], axes=axes)
    k = np.fft.fftshift(np.fft.fft2(x, axes=axes, norm="ortho"), axes=axes)
    return k * mask[None]


@pytest.mark.parametrize("W", WIDTHS)
@pytest.mark.parametrize("C,H,kind", [(1, 9, "lines"), (11, 20, "points")])
def test_operator_matches_numpy(pdt, W, C, H, kind):
    rng = np.random.default_rng(W + C)
    c = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    sens = c(C, H, W)
    mask = (rng.random((H, W)) < 0.3).astype(np.float32) if kind == "points" else np.zeros((H, W), np.float32)
    if kind == "lines":
        mask[:, ::3] = 1.0
    op = pdt.mri.MriCartesianOperator()
    op.setCoilSens(sens)
    op.setMask(mask)
    u, k = c(H, W), c(C, H, W)
    fwd, adj = op.forward(u), op.adjoint(k)
    want = _reference(u.astype(np.complex128), sens.astype(np.complex128), mask)
    # FP32 transforms of n = H W points: relative error below log2(n) 2^-23 a value in the norm, doubled for the
    # products with the maps and the mask; where the tensor-core rows were chosen, 22-bit operands: 2^-20
    tol = 2 * np.log2(H * W) * 2.0**-23 + 2.0**-20
    assert rel_l2(fwd, want) <= tol
    assert (fwd[:, mask == 0] == 0).all()
    kk = np.fft.ifftshift(k.astype(np.complex128) * mask[None], axes=(-2, -1))
    img = np.fft.fftshift(np.fft.ifft2(kk, axes=(-2, -1), norm="ortho"), axes=(-2, -1))
    assert rel_l2(adj, (np.conj(sens.astype(np.complex128)) * img).sum(0)) <= tol
