"""The Cartesian operators' row passes on register transforms, chosen by PDT_REGISTER_ROWS whatever the tuner measured:
every compiled row length against NumPy in double precision, with ragged row blocks, one to many coils (up to eight form a
cluster), the readout-oversampling operator's row offset, and a k-space that does not start on a 16-byte boundary."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

WIDTHS = [48, 64, 80, 96, 112, 128, 144, 160, 176, 192, 208, 224, 240, 256, 272, 288, 304, 320, 336, 352, 368, 384, 416, 448,
          480, 512, 576, 640]


def _tol(H, W):
    # FP32 transforms of n = H W points: relative error below log2(n) 2^-23 in the norm, doubled for the products with
    # the maps and the mask
    return 2 * np.log2(H * W) * 2.0**-23


def _case(pdt, monkeypatch, kind, C, H, W, seed):
    monkeypatch.setenv("PDT_REGISTER_ROWS", "1")
    rng = np.random.default_rng(seed)
    c = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    mask = (rng.random((H, W)) < 0.3).astype(np.float32)
    op = (pdt.mri.MriCartesianRemoveROOSOperator if kind == "roos" else pdt.mri.MriCartesianOperator)()
    sens = c(C, H, W)
    op.setCoilSens(sens)
    op.setMask(mask)
    report = op.tuning()
    assert "rows_fwd=register_fft" in report and "rows_adj=register_fft" in report
    Hi = H // 2 if kind == "roos" else H
    y0 = int(np.float32(2 * Hi) * np.float32(0.25) + np.float32(1)) if kind == "roos" else 0
    u, k = c(Hi, W), c(C, H, W)
    full = np.zeros((H, W), np.complex128)
    full[y0:y0 + Hi] = u
    ax, s = (-2, -1), sens.astype(np.complex128)
    want_k = np.fft.fftshift(np.fft.fft2(np.fft.ifftshift(full[None] * s, axes=ax), axes=ax, norm="ortho"), axes=ax) * mask
    img = np.fft.fftshift(np.fft.ifft2(np.fft.ifftshift(k.astype(np.complex128) * mask, axes=ax), axes=ax, norm="ortho"), axes=ax)
    want_u = (np.conj(s) * img).sum(0)[y0:y0 + Hi]
    return op, mask, u, k, want_k, want_u


@pytest.mark.parametrize("W", WIDTHS)
@pytest.mark.parametrize("kind,C,H", [("plain", 1, 9), ("plain", 3, 16), ("plain", 11, 20), ("roos", 5, 44)])
def test_operator_matches_numpy(pdt, monkeypatch, kind, C, H, W):
    op, mask, u, k, want_k, want_u = _case(pdt, monkeypatch, kind, C, H, W, W + C)
    got = op.forward(u)
    assert rel_l2(got, want_k) <= _tol(H, W)
    assert (got[:, mask == 0] == 0).all()
    assert rel_l2(op.adjoint(k), want_u) <= _tol(H, W)


@pytest.mark.parametrize("H,offset", [(20, 0), (20, 1), (21, 1), (21, 2)])  # even and odd numbers of values from each start
def test_k_space_off_a_16_byte_boundary(pdt, monkeypatch, H, offset):
    torch = pytest.importorskip("torch")
    C, W = 3, 304
    op, _, u, _, want_k, _ = _case(pdt, monkeypatch, "plain", C, H, W, H)
    n = C * H * W
    buf = torch.full((n + offset + 4,), 7.0 + 7.0j, dtype=torch.complex64, device="cuda")
    out = buf[offset:offset + n].view(C, H, W)
    op.forward(torch.from_numpy(u).cuda(), out=out)
    torch.cuda.synchronize()
    assert rel_l2(out.cpu().numpy(), want_k) <= _tol(H, W)
    rest = torch.cat([buf[:offset], buf[offset + n:]])
    assert (rest == 7.0 + 7.0j).all()  # nothing outside
