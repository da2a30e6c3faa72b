"""Decode attention over split sequences: the merge of the partial results, from two splits to more than one block of them, with splits
that hold no page."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("G,R", [(1, 1), (4, 1), (7, 2), (16, 1)])
@pytest.mark.parametrize("splits", [2, 7, 8, 9, 64, 65, 130])
def test_merge(D, G, R, splits):
    from llaminar_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(splits)
    Hk, lens = 2, [700, 5, 64]
    B, P = len(lens), 11
    kv = torch.randn(B * P, 2, Hk, 64, D, device=DEV, generator=g).bfloat16()
    table = torch.randperm(B * P, generator=torch.Generator().manual_seed(1)).view(B, P).to(torch.int32).to(DEV)
    q = torch.randn(B * R, Hk * G, D, device=DEV, generator=g).bfloat16()
    out, sc = torch.full_like(q, float("nan")), ops.scratch_for(DEV)
    ops.attn_decode(q, kv, out, table, torch.tensor(lens, dtype=torch.int32, device=DEV), Hk * G, Hk, D, R, 1 / math.sqrt(D), splits, sc)
    assert int(sc.attn_tickets.abs().sum()) == 0
    for b, n in enumerate(lens):
        k, v = (kv[table[b].long(), i].transpose(1, 2).reshape(P * 64, Hk, D)[:n].double().repeat_interleave(G, 1) for i in (0, 1))
        for r in range(R):
            m = n - (R - 1 - r)
            s = torch.einsum("hd,shd->hs", q[b * R + r].double(), k[:m]) / math.sqrt(D)
            want = torch.einsum("hs,shd->hd", torch.softmax(s, -1), v[:m])
            # probabilities and the output are rounded to bf16, sums are fp32
            assert (out[b * R + r].double() - want).norm() <= 6e-3 * want.norm(), (b, r)


@pytest.mark.parametrize("B,Hk,splits", [(111, 3, 1), (112, 3, 1), (100, 4, 1), (42, 4, 2)])
def test_8_bit_cache_around_two_ctas_an_sm(B, Hk, splits):
    """333 CTAs, and more: the form of three CTAs an SM."""
    from llaminar_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(B)
    D, G, P = 128, 4, 4
    codes = torch.randint(-127, 128, (B * P, 2, Hk, 64, D), device=DEV, generator=g, dtype=torch.int8)
    # scales of seven mantissa bits, as the cache keeps them
    scales = torch.randint(64, 128, (B * P, 2, Hk, 64, D // 32), device=DEV, generator=g).half() * 2.0 ** -12
    kv = torch.cat([codes.view(B * P, -1).view(torch.uint8), scales.view(B * P, -1).view(torch.uint8)], 1).contiguous()
    table = torch.randperm(B * P, generator=torch.Generator().manual_seed(1)).view(B, P).to(torch.int32).to(DEV)
    lens = torch.randint(1, P * 64 + 1, (B,), generator=torch.Generator().manual_seed(2)).to(torch.int32).to(DEV)
    q = torch.randn(B, Hk * G, D, device=DEV, generator=g).bfloat16()
    out, sc = torch.full_like(q, float("nan")), ops.scratch_for(DEV)
    ops.attn_decode(q, kv, out, table, lens, Hk * G, Hk, D, 1, 1 / math.sqrt(D), splits, sc)
    values = codes.double() * scales.double().repeat_interleave(32, -1)
    for b in range(B):
        n = int(lens[b])
        k, v = (values[table[b].long(), i].transpose(1, 2).reshape(P * 64, Hk, D)[:n].repeat_interleave(G, 1) for i in (0, 1))
        s = torch.einsum("hd,shd->hs", q[b].double(), k) / math.sqrt(D)
        want = torch.einsum("hs,shd->hd", torch.softmax(s, -1), v)
        # probabilities and queries are rounded to fp16, the output to bf16; sums are fp32
        assert (out[b].double() - want).norm() <= 6e-3 * want.norm(), b
