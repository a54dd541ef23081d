"""The row products' epilogue in every combination of what it reads (a residual,
the old result, a mask) and writes (FP32, BF16, both), against FP32 torch.

Bound: both sides add at most K + 3 exact or FP32-rounded terms in FP32, so
they differ by less than (K + 3) 2^-23 times the sum of the terms' magnitudes.
The BF16 result is exactly the FP32 result rounded, whether that is written too
or not.  A masked entry is zero exactly."""
import itertools

import pytest

from uph_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,ldc", [(1, 128, 64, 128), (200, 256, 128, 264), (384, 128, 256, 128)])
def test_epilogue_combinations(M, N, K, ldc):
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda").manual_seed(M + N + K)

    def rnd(*shape):
        return torch.randn(*shape, device="cuda", generator=g)

    A, B, bias = rnd(M, K).bfloat16(), rnd(N, K).bfloat16(), rnd(N)
    residual, mask, old = rnd(M, ldc).bfloat16(), rnd(M, ldc).bfloat16(), rnd(M, ldc)
    mask[:, ::5] = 0.0
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    product = A.float() @ B.float().T
    size = A.float().abs() @ B.float().abs().T + bias.abs() + residual[:, :N].float().abs() + old[:, :N].abs()
    tol = (K + 3) * 2.0 ** -23 * size
    for res, acc, msk, relu, out in itertools.product((0, 1), (0, 1), (0, 1), (0, 1), ("32", "both", "16")):
        if acc and out == "16":
            continue  # there is no old result to add
        c32 = old.clone() if out != "16" else None
        c16 = torch.full((M, ldc), 7.0, device="cuda", dtype=torch.bfloat16) if out != "32" else None
        at = [None if t is None else t.data_ptr() for t in (c32, c16)]
        st = _lib.lib().uph_tc_gemm_bf16_epilogue(A.data_ptr(), K, B.data_ptr(), K, M, N, K, bias.data_ptr(),
                                                  residual.data_ptr() if res else None, acc, relu,
                                                  mask.data_ptr() if msk else None, *at, ldc, err.data_ptr(),
                                                  torch.cuda.current_stream().cuda_stream)
        assert st == 0, _lib.lib().uph_last_error()
        torch.cuda.synchronize()
        assert int(err.item()) == 0
        want = product + bias
        if res:
            want = want + residual[:, :N].float()
        if acc:
            want = want + old[:, :N]
        if relu:
            want = torch.relu(want)
        if msk:
            want = torch.where(mask[:, :N].float() > 0, want, torch.zeros_like(want))
        what = (res, acc, msk, relu, out)
        if c32 is not None:
            got = c32[:, :N]
            assert bool(((got - want).abs() <= tol).all()), what
            if msk:
                assert bool((got[mask[:, :N].float() <= 0] == 0).all()), what
        if c16 is not None:
            # "16": the FP32 result of "both", just before it
            assert torch.equal(c16[:, :N], got.bfloat16()), what
        # what lies beyond the columns stays
        if c32 is not None:
            assert torch.equal(c32[:, N:], old[:, N:])
        if c16 is not None:
            assert bool((c16[:, N:] == 7.0).all())
