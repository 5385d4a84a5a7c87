"""Radial operators on grid lengths with a compiled transform split and on others, one to many coils (chunks of 16 in
the row passes), kernel widths and sample lists with cells gridded by a block of their own, against the FP64 oracle.

Tolerance: two FP32 transforms of length G <= 320 (about log2(G) 2^-23 relative each), deapodisation and up to 64
taps: below 5e-6; the bar of the operators is 1e-5.
"""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

# (N, osf, kernel width, coils, spokes): G = 32, 60, 96, 130, 144, 220, 270, 320 compiled; 34, 46, 122 not
CASES = [(16, 2.0, 3, 1, 9), (48, 1.25, 4, 5, 20), (64, 1.5, 3, 17, 40), (104, 1.25, 3, 2, 16), (96, 1.5, 5, 33, 8),
         (176, 1.25, 3, 3, 12), (180, 1.5, 6, 1, 10), (160, 2.0, 3, 12, 24), (17, 2.0, 3, 3, 9), (23, 2.0, 8, 2, 7),
         (81, 1.5, 3, 16, 13)]


@pytest.mark.parametrize("N,osf,kw,C,spokes", CASES)
def test_radial_operator_matches_oracle(pdt, oracle, N, osf, kw, C, spokes):
    rng = np.random.default_rng(N + C)
    c = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    ang = np.arange(spokes) * np.pi * (np.sqrt(5) - 1) / 2
    r = (np.arange(2 * N) - N) / (2 * N)
    k = (r[:, None] * np.exp(1j * ang[None, :])).ravel()
    traj = np.array([k.imag, k.real]).astype(np.float32)
    dcf = np.sqrt(np.abs(k)).astype(np.float32)[None, :]
    sens = c(C, N, N)
    op = pdt.mri.MriRadialOperator({"osf": osf, "sector_width": 8, "kernel_width": kw, "img_dim": N})
    op.setTrajectory(traj)
    op.setDcf(dcf)
    op.setCoilSens(sens)
    u, f = c(N, N), c(C, traj.shape[1])
    assert rel_l2(op.forward(u), oracle.radial_apply(traj, dcf, sens, u, N, osf, kw)) <= 1e-5
    assert rel_l2(op.adjoint(f), oracle.radial_apply(traj, dcf, sens, f, N, osf, kw, mode="adjoint")) <= 1e-5


@pytest.mark.parametrize("C", [1, 2, 5])
def test_gridding_of_many_samples_per_cell(pdt, oracle, C):
    # a smooth image's samples add up coherently in the cells near k = 0, which hold hundreds of entries each; one
    # coil leaves the block that grids such a cell 256 partial sums
    N, osf, kw, spokes = 64, 1.25, 5, 59
    ang = np.arange(spokes) * np.pi * (np.sqrt(5) - 1) / 2
    r = (np.arange(2 * N) - N) / (2 * N)
    k = (r[:, None] * np.exp(1j * ang[None, :])).ravel()
    traj = np.array([k.imag, k.real]).astype(np.float32)
    dcf = np.sqrt(np.abs(k)).astype(np.float32)[None, :]
    y, x = np.mgrid[:N, :N] / N - 0.5
    sens = np.stack([np.exp(-((x - 0.1 * c) ** 2 + y**2) + 1j * c * x) for c in range(C)]).astype(np.complex64)
    f = oracle.radial_apply(traj, dcf, sens, (x**2 + y**2 < 0.16).astype(np.complex64), N, osf, kw).astype(np.complex64)
    op = pdt.mri.MriRadialOperator({"osf": osf, "sector_width": 8, "kernel_width": kw, "img_dim": N})
    op.setTrajectory(traj)
    op.setDcf(dcf)
    op.setCoilSens(sens)
    # a cell of n entries: ceil(n / 256) + 8 additions and a product in a chain, 11 2^-24 = 6.6e-7 at worst, and two
    # transforms of 80 points, 2 log2(80) 2^-25 = 3.8e-7
    assert rel_l2(op.adjoint(f), oracle.radial_apply(traj, dcf, sens, f, N, osf, kw, mode="adjoint")) <= 1.04e-6
