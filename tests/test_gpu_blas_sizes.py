"""BLAS builds at the edges of the hierarchy kernel's spans of leaves (they start at the
shortest prefix of windows of 256 leaves around the multiples of 256, so at 128 leaves there
is a second one), of the sort's tiles (2048 keys) and of the bounds' rows, with random
triangles, runs of equal Morton codes (split by index) and clusters far apart; several sizes
in one batch, empty meshes among them. Nodes, triangles, codes and order are the oracle's
bit for bit, and those of the build without allocations are the same."""
import ctypes as C

import numpy as np
import pytest

import luz_gb300 as L
import oracle as O

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 33, 127, 128, 129, 130, 255, 256, 257, 383, 385, 511, 512, 513, 640, 1025, 2047, 2049, 4097, 9001]


def _mesh(n, kind, rng):
    p = rng.uniform(-1, 1, (n, 1, 3)) + rng.uniform(-0.05, 0.05, (n, 3, 3))
    if kind == "equal" and n:
        k = max(n // 2, 1)
        p[:k] = p[0]                                   # equal codes
        p[k:] = p[k + rng.integers(0, max((n - k) // 7, 1), n - k)] if n > k else p[k:]
    if kind == "clusters":
        p += 40.0 * rng.integers(-2, 3, (n, 1, 3))
    v = np.zeros((3 * n, 12), np.float32)
    v[:, :3] = p.reshape(-1, 3)
    return v, np.arange(3 * n, dtype=np.uint32)


def _same(got, want):
    for name, a, b in zip(("nodes", "triangles", "codes", "order"), got, want):
        assert np.array_equal(np.ascontiguousarray(a).view(np.uint32), np.ascontiguousarray(b).view(np.uint32)), name


@pytest.mark.parametrize("kind", ["random", "equal", "clusters"])
def test_sizes(kind):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(len(kind))
    meshes = [_mesh(n, kind, rng) for n in SIZES]
    want = []
    for v, i in meshes:
        on, ot, om, oo = O.OracleBlas(v, i).arrays()
        want.append((on, ot, om, oo))
    ctx = L.Context(0)
    try:
        for batch in (list(range(len(SIZES))), list(range(len(SIZES)))[::-3]):
            parts = [meshes[k] for k in batch]
            empty = (np.zeros((1, 12), np.float32), np.zeros(0, np.uint32))
            built = ctx.build_blas([empty] + parts[:3] + [empty] + parts[3:] + [empty])
            built = built[1:4] + built[5:-1]
            for k, b in zip(batch, built):
                gn, gt, gm, go = b.download()
                _same((gn, gt, gm, go), want[k])
        stream = torch.cuda.Stream()
        for (v, i), w in zip(meshes, want):
            n = i.size // 3
            dv, di = torch.from_numpy(v).cuda(), torch.from_numpy(i.view(np.int32)).cuda()
            out = [torch.zeros(s, dtype=torch.int32, device="cuda") for s in ((max(n, 2) - 1, 16), (n, 12), (n,), (n,))]
            torch.cuda.synchronize()
            p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
            assert L.lib.luz_blas_build_noalloc(p(dv), v.shape[0], p(di), i.size, *(p(t) for t in out),
                                                C.c_void_p(stream.cuda_stream)) == 0
            _same([t.cpu().numpy() for t in out], w)
    finally:
        ctx.close()
