"""A prompt's sublayers started by one call each."""
import math

import pytest
import torch

from test_kernels_gpu import stream

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K():
    from titan_b200 import kernels
    kernels.lib()
    return kernels


@pytest.mark.parametrize("T", [9, 17, 130, 300])
@pytest.mark.parametrize("H,F", [(64, 72), (256, 320)])
def test_a_prompts_feed_forward_started_by_one_call(K, T, H, F):
    """The same kernels in the same order as the norm and the two products one by one: the same bits where no tile is cut along K."""
    g = torch.Generator().manual_seed(T + F)
    x = torch.randn(T, H, generator=g).cuda()
    nw = (1 + 0.1 * torch.randn(H, generator=g)).cuda()
    gu, down = ((torch.randn(n, k, generator=g) / math.sqrt(k)).to(torch.bfloat16).cuda() for n, k in ((2 * F, H), (H, F)))
    h, act = torch.empty(T, H, dtype=torch.bfloat16, device="cuda"), torch.empty(T, F, dtype=torch.bfloat16, device="cuda")
    one, many = x.clone(), x.clone()
    assert K.norm_gated_mlp(one, nw, 1e-6, gu, down, h, act, stream(), ordered=True)
    h2, act2 = torch.empty_like(h), torch.empty_like(act)
    K.rmsnorm(many, nw, h2, 1e-6, stream())
    K.gemm_tc(h2, gu, act2, K.EPI_SWIGLU, stream(), ordered=True)
    K.gemm_tc(act2, down, many, K.EPI_ADD, stream(), ordered=True)
    assert torch.equal(h, h2) and torch.equal(act, act2) and torch.equal(one, many)
    assert K.wait_errors() == {}
    # sizes that the tensor-core kernel does not take (F no multiple of 8) are refused before anything is launched
    odd = x.clone()
    assert not K.norm_gated_mlp(odd, nw, 1e-6, gu[:2 * (F - 4)].contiguous(), down[:, :F - 4].contiguous(), h, torch.empty(T, F - 4, dtype=torch.bfloat16, device="cuda"), stream())
    assert torch.equal(odd, x)
