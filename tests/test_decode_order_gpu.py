"""Decode attention that works its sequences off from the longest down, and that reads older rows before the kernels before it have ended."""
import math

import pytest
import torch

from test_kernels_gpu import Paged, layout_for, stream
from test_paired_units_gpu import K, attention  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,nkv,hd", [(38, 8, 128), (160, 2, 64), (161, 2, 128)])
def test_decode_attention_from_the_longest_sequence_down(K, B, nkv, hd):
    """More blocks than places: the order in which sequences are worked off changes nothing; equal lengths among them; one more sequence than a block has threads."""
    g = torch.Generator().manual_seed(B)
    lens = [1 + (37 * i * i) % 200 for i in range(B)]
    lens[5] = lens[6] = lens[7]
    slots, nh = list(range(B)), 2 * nkv
    lay = layout_for(slots, [n - 1 for n in lens], [1] * B)
    cache = Paged(K, slots, lens, nkv, hd, torch.bfloat16)
    q = torch.randn(B, nh * hd, generator=g).to(torch.bfloat16).cuda()
    out = torch.full((B, nh * hd), float("nan"), dtype=torch.bfloat16, device="cuda")
    scratch = torch.empty(B * nh * (hd + 2), device="cuda")
    a = K.AttnArgs()
    a.q, a.q_stride, a.out, a.out_stride = q.data_ptr(), nh * hd, out.data_ptr(), nh * hd
    a.cache, a.batch, a.nh, a.nkv, a.hd, a.scale = cache.view, lay.c_struct(), nh, nkv, hd, 0.02 / math.sqrt(hd)
    a.chunk, a.n_splits, a.scratch = 128, 1, scratch.data_ptr()
    K.attn_decode_mma(a, stream())
    assert K.wait_errors() == {}
    for i, n in enumerate(lens):
        rows = [cache.get(i, p) for p in range(n)]
        k, v = torch.stack([r[0] for r in rows]).cuda(), torch.stack([r[1] for r in rows]).cuda()
        want, weight = attention(q[i:i + 1].reshape(1, nh, hd), k, v, n - 1, 0, 0, a.scale, None)
        bound = weight * (2.0 ** -8 + 2.0 ** -14) + want.abs() * 2.0 ** -8 * 1.01 + 1e-30
        assert bool(((out[i].double().reshape(1, nh, hd) - want).abs() <= bound).all()), i
