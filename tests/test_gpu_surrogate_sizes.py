"""The surrogate's gradients over node counts at the edges of the tensor-core
products, against the CPU oracle: 40 and 64 nodes are one slice of K (weight
gradients without a split, bias gradients by their own kernel), 65 the first
split, 127 to 129 the edge of a 128-row tile, 1000 several splits whose last
slice is partial.

Bound: a gradient block differs from the oracle's by BF16 values and ReLU
branches that fall on the other side of a boundary.  A flipped branch changes
one of (nodes x 128) terms, so at 40 nodes some ten flips (10 / 5120 of the
terms, uncorrelated: sqrt(10 / 5120) = 4.4e-2) are the most that is expected:
5e-2 of the block's norm.  A dropped or repeated node at 129 nodes is 9e-2."""
import numpy as np
import pytest

from oracle import surrogate_oracle as SO
from uph_b200 import surrogate as SG

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [40, 64, 65, 127, 128, 129, 1000])
def test_gradients_at_tile_edges(n):
    rng = np.random.default_rng(n)
    side = int(np.ceil(np.sqrt(n)))
    ij = np.stack(np.meshgrid(np.arange(side), np.arange(side)), -1).reshape(-1, 2)[:n]
    pos = (ij + rng.uniform(-0.2, 0.2, ij.shape)) * 0.02
    vel = rng.normal(0, 0.05, (n, 2))
    rho = 1000.0 * (1 + rng.normal(0, 1e-3, n))
    nf = n - n // 8
    itype = np.where(np.arange(n) < nf, 1, -1).astype(np.int32)
    cfg = SG.NetConfig(radius=0.05, dt=1e-4, rho0=1000.0, vel_scale=0.1, rho_scale=0.01, macro_steps=5)
    flat = SG.init_params(n, 3).astype(np.float64)
    W = SO.unpack(flat, 3)
    W["dec2.w"][:SO.NOUT] *= 10.0
    for r in range(3):
        W[f"r{r}.n2.w"] *= 10.0
    flat = flat.astype(np.float32)
    dev = lambda a, dt=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device="cuda")
    nodes = SG.Nodes(dev(pos[:, 0]), dev(pos[:, 1]), dev(vel[:, 0]), dev(vel[:, 1]), dev(rho),
                     dev(itype, torch.int32), nf, (-0.1, -0.1, side * 0.02 + 0.1, side * 0.02 + 0.1))
    tgt = rng.normal(0, 1, (nf, SO.NOUT))
    sur = SG.Surrogate(cfg, n, flat)
    loss, grad = sur.gradients(nodes, dev(tgt, torch.float32))
    grad = grad.cpu().numpy().astype(np.float64)
    sur.close()
    g = SO.Graph(pos[:, 0], pos[:, 1], cfg.radius, rho, cfg.rho0 * cfg.edge_rho_scale)
    F = SO.node_features(vel[:, 0], vel[:, 1], rho, itype, cfg.vel_scale, cfg.rho0, cfg.rho_scale)
    out, cache = SO.forward(flat, F, g, 3, emulate=True)
    ref_loss, dout = SO.loss_and_grad(out, tgt, nf)
    ref = SO.backward(cache, dout)
    assert loss == pytest.approx(ref_loss, rel=1e-3)
    off, _ = SO.offsets(3)
    for name, (o, shape) in off.items():
        sz = int(np.prod(shape))
        rn = np.linalg.norm(ref[o:o + sz])
        if rn == 0:
            assert np.all(grad[o:o + sz] == 0), name
            continue
        e = np.linalg.norm(grad[o:o + sz] - ref[o:o + sz]) / rn
        assert e <= 5e-2, (name, e)


@pytest.mark.parametrize("M,splits,accumulate,skew", [(200, 5, 0, 0), (200, 5, 1, 0), (256, 3, 1, 0), (77, 1, 1, 0),
                                                      (200, 5, 1, 1)])
def test_split_products_of_partial_tiles(M, splits, accumulate, skew):
    """M off the 128-row tile (partials are not whole boxes), 11 slices of K
    over splits that do not divide them, a sum added to what is there, a
    result off the 16-byte boundary; the bound is the summation order's, 1e-3
    of the largest value."""
    import ctypes as C

    from test_gpu_tc_gemm import _lib
    lib = _lib()
    N, K = 128, 11 * 64
    gen = torch.Generator(device="cuda").manual_seed(M)
    A = torch.randn(M, K, device="cuda", generator=gen).to(torch.bfloat16)
    B = torch.randn(N, K, device="cuda", generator=gen).to(torch.bfloat16)
    c = torch.randn((M + 8) * N + 4, device="cuda", generator=gen)[skew:skew + (M + 8) * N].view(M + 8, N)
    before = c.clone()
    part = torch.empty(splits * M * N, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    st = lib.uph_tc_gemm_bf16(A.data_ptr(), K, B.data_ptr(), K, M, N, K, None, 0, c.data_ptr(), None, N, splits,
                              part.data_ptr() if splits > 1 else None, accumulate, err.data_ptr(),
                              C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0, lib.uph_last_error()
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    ref = A.float() @ B.float().T + (before[:M] if accumulate else 0)
    assert (c[:M] - ref).abs().max().item() <= 1e-3 * ref.abs().max().item() + 1e-3
    assert torch.equal(c[M:], before[M:])  # rows beyond the result are left alone
