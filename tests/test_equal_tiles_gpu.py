"""Prompt products in equal tiles of rows (pairs of CTAs, weights on the wide side)."""
import math

import pytest
import torch

from test_kernels_gpu import stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [129, 160, 255, 257, 372, 905])
@pytest.mark.parametrize("N,K_", [(256, 64), (301, 72), (520, 1032), (2048, 512)])
def test_products_in_equal_tiles_of_rows(M, N, K_):
    """Row tiles that end inside the last one, columns that end inside a panel, an odd number of columns, K that ends inside a block."""
    from titan_b200 import kernels as K
    g = torch.Generator().manual_seed(M + N)
    x = torch.randn(M, K_, generator=g).to(torch.bfloat16).cuda()
    w = (torch.randn(N, K_, generator=g) / math.sqrt(K_)).to(torch.bfloat16).cuda()
    z, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    err = size * K_ * 2.0 ** -23                          # float32 sums of exact products
    try:
        K.set_gemm_plain_tile(4)
        room = torch.full((M + 1, -(-N // 8) * 8 + 8), 7.0, dtype=torch.bfloat16, device="cuda")
        out = room[:M, :N]
        K.gemm_tc(x, w, out, K.EPI_STORE, stream())
        assert bool(((out.double() - z).abs() <= err + z.abs() * 2.0 ** -8).all())
        assert bool((room[M:] == 7.0).all()) and bool((room[:, N:] == 7.0).all())
        K.gemm_tc(x, w, out, K.EPI_STORE, stream(), gate=K.UNARY_RELU2)
        want = z.clamp_min(0) ** 2
        assert bool(((out.double() - want).abs() <= 2.1 * err * z.abs() + err * err + want * 2.0 ** -8).all())
        if N % 2 == 0:
            room.fill_(7.0)
            act, gate, up = room[:M, :N // 2], z[:, 0::2], z[:, 1::2]
            K.gemm_tc(x, w, act, K.EPI_SWIGLU, stream())
            want = torch.nn.functional.silu(gate) * up
            bound = 1.1 * err[:, 0::2] * up.abs() + torch.nn.functional.silu(gate).abs() * err[:, 1::2] + want.abs() * (2.0 ** -8 + 2.0 ** -18) + 1e-30
            assert bool(((act.double() - want).abs() <= bound).all())
            assert bool((room[M:] == 7.0).all()) and bool((room[:, N // 2:] == 7.0).all())
    finally:
        K.set_gemm_plain_tile(0)
    assert K.wait_errors() == {}
