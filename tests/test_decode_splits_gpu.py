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
