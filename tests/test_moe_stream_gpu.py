"""Streaming expert kernels of a decode step."""
import pytest
import torch

from llaminar_b200.gguf import GGMLType, dequantize, quantize

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("qt", [GGMLType.Q4_K, GGMLType.Q5_K, GGMLType.Q6_K, GGMLType.Q8_0, GGMLType.Q4_0, GGMLType.IQ3_S])
@pytest.mark.parametrize("tokens,E,k,d,ff", [(1, 8, 2, 256, 256), (9, 8, 8, 512, 256), (40, 20, 3, 1280, 512)])
def test_experts(qt, tokens, E, k, d, ff):
    """One item for the whole GPU, one chunk per row, many items per CTA, experts of another rank; against 32 bits."""
    from llaminar_b200 import ops
    from llaminar_b200.ops.layout import interleave_gate_up, pack_experts
    g = torch.Generator(device=DEV).manual_seed(tokens)
    e0, n_local = (0, E) if tokens < 40 else (3, E - 5)
    mats = [[torch.randn(*s, device=DEV, generator=g) * 0.05 for s in ((ff, d), (ff, d), (d, ff))] for _ in range(n_local)]
    raw = [[quantize(m, qt) for m in ms] for ms in mats]
    deq = [[dequantize(r, qt, tuple(m.shape)) for r, m in zip(rs, ms)] for rs, ms in zip(raw, mats)]
    gu = pack_experts(torch.cat([interleave_gate_up(r[0], r[1], qt, ff, d)[0] for r in raw]), qt, n_local, 2 * ff, d)
    dn = pack_experts(torch.cat([r[2] for r in raw]), qt, n_local, d, ff)
    h = torch.randn(tokens, d, device=DEV, generator=g)
    norm_w = 1.0 + 0.1 * torch.randn(d, device=DEV, generator=g)
    router = (torch.randn(E, d, device=DEV, generator=g) * 0.05).bfloat16()
    i32 = lambda *s: torch.zeros(*s, dtype=torch.int32, device=DEV)
    z_max = n_local + (tokens * k + 3) // 4
    ids, wts, items, n_items, ticket = i32(tokens, k), torch.zeros(tokens, k, device=DEV), i32(z_max * ops.MOE_ITEM_INTS), i32(1), i32(1)
    act, y, tt, sc = torch.zeros(tokens * k, ff, dtype=torch.bfloat16, device=DEV), torch.zeros(tokens * k, d, device=DEV), i32((d + 127) // 128), ops.scratch_for(DEV)
    sc.status.zero_()
    ops.moe_route(h, norm_w, 1e-6, router, k, True, e0, n_local, ids, wts, items, n_items, ticket)
    out = []
    for _ in range(2):
        hh = h.clone()
        ops.moe_gate_up(gu, hh, norm_w, 1e-6, act, items, n_items, k, z_max, scratch=sc)
        ops.moe_down_combine(dn, act, y, items, n_items, z_max, ids, wts, k, e0, n_local, hh, tt, scratch=sc)
        out.append(hh)
    assert torch.equal(*out) and int(sc.status[0]) == 0 and int(sc.tickets.abs().sum()) == 0
    xn, want = h * torch.rsqrt((h * h).mean(-1, keepdim=True) + 1e-6) * norm_w, torch.zeros_like(h)
    for t in range(tokens):
        for j in range(k):
            e = int(ids[t, j]) - e0
            if 0 <= e < n_local:
                G, U, D = deq[e]
                want[t] += wts[t, j] * (D @ (torch.nn.functional.silu(G @ xn[t]) * (U @ xn[t])))
    # activations are rounded to 8 bits per 32 values in both products (about 0.4 % each), the hidden rows to bf16 between them
    assert (out[0] - h - want).norm() <= 1.5e-2 * want.norm()
