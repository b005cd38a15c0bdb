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


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nh,nkv,hd,window,keep,ring", [(16, 8, 64, 0, 0, 0), (6, 3, 32, 100, 0, 0), (4, 2, 8, 100, 5, 0), (4, 4, 128, 64, 0, 128)])
def test_any_size_decode_attention_that_reads_older_rows_early(K, dtype, nh, nkv, hd, window, keep, ring):
    """With lengths known before the step (by sequence, or by slot) the same bits as without."""
    g = torch.Generator().manual_seed(nh + hd)
    lens = [1, 2, 31, 256, 257, 513, 700]
    B, slots = len(lens), [6, 2, 0, 5, 1, 3, 4]
    lay = layout_for(slots, [n - 1 for n in lens], [1] * B)
    cache = Paged(K, slots, lens, nkv, hd, dtype, ring_rows=ring)
    q = torch.randn(B, nh * hd, generator=g).to(dtype).cuda()
    committed = torch.zeros(8, dtype=torch.int32)
    for s, n in zip(slots, lens):
        committed[s] = n - 1
    committed = committed.cuda()
    outs = []
    for mode in (0, 1, 2):
        out, scratch = torch.full((B, nh * hd), float("nan"), dtype=dtype, device="cuda"), torch.full((B * nh * 3 * (hd + 2),), float("nan"), device="cuda")
        a = K.AttnArgs()
        a.q, a.q_stride, a.out, a.out_stride = q.data_ptr(), nh * hd, out.data_ptr(), nh * hd
        a.cache, a.batch, a.nh, a.nkv, a.hd, a.scale, a.window, a.keep_first = cache.view, lay.c_struct(), nh, nkv, hd, 0.002, window, keep
        a.chunk, a.n_splits, a.scratch = 256, 3, scratch.data_ptr()
        a.early_mode, a.early_len = mode, (None if mode == 0 else lay.kv_len.data_ptr() if mode == 1 else committed.data_ptr())
        K.attn_decode(a, dtype, stream())
        outs.append(out)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2]) and not bool(torch.isnan(outs[0]).any())
