"""The denoiser's tiling: 16x8-pixel tiles, or runs of 128 pixels where the images' edges
would waste too many, two tiles per block in training, and tiles of background. Training and
inference against the FP64 restatement at sizes where the last tiles are partial."""
import numpy as np
import pytest

import luz_gb300 as L
from luz_gb300 import _abi, denoiser as D
from oracle import denoiser as OD

pytestmark = pytest.mark.gpu


def _batch(n, h, w, seed, background):
    rng = np.random.default_rng(seed)
    depth = (5.0 + 3.0 * rng.random((n, h, w))).astype(np.float32)
    depth[rng.random((n, h, w)) < 0.1] = 0.0
    if background:
        depth[:, : h // 2] = 0.0                      # whole tiles of background
    lit = (depth > 0)[..., None]
    feat = OD.bf16_round((rng.random((n, h, w, 8)) * 2 - 1).astype(np.float32)) * lit
    uns = (rng.random((n, h, w, 4)) * lit).astype(np.float32)
    noisy = (uns * rng.random((n, h, w, 4))).astype(np.float32)
    target = rng.random((n, h, w, 4)).astype(np.float32)
    bits = (np.ascontiguousarray(feat, np.float32).view(np.uint32) >> 16).astype(np.uint16)
    return bits, depth, noisy, uns, target


@pytest.mark.parametrize("n,h,w,background", [(1, 1, 1, False), (3, 5, 7, False), (2, 16, 16, True), (1, 33, 130, False),
                                              (2, 48, 64, True), (1, 128, 1, False)])
def test_tiles_match_fp64_restatement(n, h, w, background):
    torch = pytest.importorskip("torch")
    bits, depth, noisy, uns, target = _batch(n, h, w, 7 * h + w, background)
    ctx = L.Context(0)
    try:
        den = D.Denoiser(ctx)
        den.load()
        dev = [torch.from_numpy(a).cuda() for a in (bits.view(np.int16), depth, noisy, uns, target)]
        b = _abi.DenoiseBatch()
        b.features, b.lin_depth, b.noisy, b.unshadowed, b.target = (t.data_ptr() for t in dev)
        b.weight = None
        b.width, b.height, b.images = w, h, n
        out = torch.full((n, h, w, 4), 7.0, device="cuda")
        torch.cuda.synchronize()
        den.infer(b, out.data_ptr())
        grad, loss = den.gradient(b)
        ctx.synchronize()
        assert ctx.device_status() == 0
        y, loss64, g64 = OD.forward_backward(den.weights(), bits, depth, noisy, uns, target)
        # BF16 activations: the bounds of the other denoiser tests
        assert np.abs(out.cpu().numpy() - y).max() < 2e-2
        assert abs(loss - loss64) <= 2e-2 * max(loss64, 1e-12)
        cos = float(np.dot(grad, g64) / max(np.linalg.norm(grad) * np.linalg.norm(g64), 1e-30))
        assert not g64.any() or cos > 0.995, cos
        again, loss2 = den.gradient(b)
        assert loss2 == loss and np.array_equal(again.view(np.uint32), grad.view(np.uint32))
    finally:
        ctx.close()
