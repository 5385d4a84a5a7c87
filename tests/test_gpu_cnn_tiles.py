"""Gradients of the warm-start network at the edges of its kernels' pixel tiles (16 x 8 and 8 x 16), against the oracle's
FP64 restatement with BF16 rounding at the same storage points."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


# one pixel, exactly one tile, one pixel more than a tile both ways, several ragged tiles in a batch
@pytest.mark.parametrize("B,H,W", [(1, 1, 1), (1, 8, 16), (2, 9, 17), (3, 33, 7)])
def test_gradients_at_tile_edges(pdt, oracle, B, H, W):
    torch = pytest.importorskip("torch")
    from primaldualtoolbox.warmstart import WarmStartNet

    rng = np.random.default_rng(B * 1000 + H * 10 + W)
    c = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    u0, ut, vt = c(B, H, W), c(B, H, W), c(B, 2, H, W)
    net = WarmStartNet(seed=5)
    net.set_params(net.get_params() * 2.0)
    p = net.get_params()
    loss = net.train_step(*(torch.from_numpy(a).cuda() for a in (u0, ut, vt)), lr=0.0)
    g = net.grads()
    ref_loss, ref_g, _ = oracle.cnn_grad(p, u0, ut, vt)
    # Both sides round to BF16 (2^-9 relative) at the same points, so they differ where an FP32 sum lands on the
    # other side of a rounding boundary: 2^-8 of one value through at most 14 roundings in a chain, 14 2^-8 = 5.5e-2
    # of that value if every one flipped the same way, sqrt(14) 2^-8 = 1.5e-2 with random signs.
    tol = 2e-2
    assert abs(loss - ref_loss) <= tol * ref_loss
    o = 0
    for n in [9 * 32 * 2, 32] + [9 * 32 * 32, 32] * 6 + [9 * 8 * 32, 8]:
        ref = ref_g[o:o + n]
        if np.linalg.norm(ref) > 0:
            assert rel_l2(g[o:o + n], ref) <= tol
        o += n
