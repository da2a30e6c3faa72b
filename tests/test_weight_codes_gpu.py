"""The weights that the tensor-core kernels multiply are, bit for bit, those of `dequant`: rows of the identity pick them out."""
import pytest
import torch

from llaminar_b200.gguf import GGMLType, dequantize, quantize

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("qt", [GGMLType.Q4_K, GGMLType.Q5_K, GGMLType.Q6_K, GGMLType.Q8_0, GGMLType.Q4_0, GGMLType.IQ3_S])
@pytest.mark.parametrize("rows", [32, 64, 128, 256])
@pytest.mark.parametrize("most", [3.0, 1e9])
def test_weights_are_those_of_dequant(qt, rows, most):
    """Scales of trained models, of zero, and (without the bound) too large for the short conversions of 4 and 5 bits, in one matrix."""
    from llaminar_b200 import ops
    n, k = 256, 768
    g = torch.Generator(device=DEV).manual_seed(rows)
    w = torch.randn(n, k, device=DEV, generator=g) * 0.05
    w[32:64] *= 30.0
    w[64:80, ::3] *= 100.0
    w[80:84] = 0.0
    w = w.clamp(-most, most)
    pw, sc = ops.pack_matrix(quantize(w, qt), qt, n, k), ops.scratch_for(DEV)
    want, eye, out = ops.dequant(pw).float(), torch.eye(k, device=DEV).bfloat16(), torch.empty(rows, n, device=DEV)
    for c in range(0, k, rows):
        ops.gemm(pw, eye[c:c + rows].contiguous(), out, scratch=sc)
        assert torch.equal(out, want[:, c:c + rows].T), c


def test_scale_that_is_no_number():
    """The outputs of its own weight row become NaN and no others."""
    from llaminar_b200 import ops
    n, k = 128, 512
    raw = quantize(torch.randn(n, k, device=DEV) * 0.05, GGMLType.Q4_K).view(n, 2, 144)
    raw[5, 1, 1] = 0x7e                                     # high byte of the block's fp16 scale
    pw, sc = ops.pack_matrix(raw.reshape(-1), GGMLType.Q4_K, n, k), ops.scratch_for(DEV)
    eye, out = torch.eye(k, device=DEV).bfloat16(), torch.empty(k, n, device=DEV)
    ops.gemm(pw, eye, out, scratch=sc)
    bad = out.isnan().sum(0)
    assert int(bad[5]) == k and int(bad.sum()) == k         # a row times NaN anywhere is NaN
    part = torch.empty(64, n, device=DEV)
    ops.gemm(pw, eye[:64].contiguous(), part, scratch=sc)
    assert int(part.isnan().sum()) == 64


def test_experts_with_large_scales():
    """Scales of 0.4 to 4 (4 bits): the grouped products of a prompt and the streaming kernels of a decode step, both against 64 bits."""
    from llaminar_b200 import ops
    from llaminar_b200.ops.layout import interleave_gate_up, pack_experts
    qt, E, k, d, ff, T = GGMLType.Q4_K, 4, 2, 512, 256, 40
    g = torch.Generator(device=DEV).manual_seed(7)
    std = lambda e, rows: torch.linspace(1.0, 10.0, rows, device=DEV)[:, None] * (1.0 if e else 0.1)      # one expert of ordinary scales
    raw = [[quantize(torch.randn(*s, device=DEV, generator=g) * std(e, s[0]), qt) for s in ((ff, d), (ff, d), (d, ff))] for e in range(E)]
    deq = [[dequantize(r, qt, s).double() for r, s in zip(rs, ((ff, d), (ff, d), (d, ff)))] for rs in raw]
    assert max(float(m.abs().max()) for ms in deq for m in ms) > 30
    gu = pack_experts(torch.cat([interleave_gate_up(r[0], r[1], qt, ff, d)[0] for r in raw]), qt, E, 2 * ff, d)
    dn = pack_experts(torch.cat([r[2] for r in raw]), qt, E, d, ff)
    h, norm_w = torch.randn(T, d, device=DEV, generator=g), torch.full((d,), 0.01, device=DEV)
    router = (torch.randn(E, d, device=DEV, generator=g) * 3).bfloat16()
    i32 = lambda *s: torch.zeros(*s, dtype=torch.int32, device=DEV)
    ids, wts, xn, sc = i32(T, k), torch.zeros(T, k, device=DEV), torch.zeros(T, d, dtype=torch.bfloat16, device=DEV), ops.scratch_for(DEV)
    act, y = torch.zeros(T * k, ff, dtype=torch.bfloat16, device=DEV), torch.zeros(T * k, d, device=DEV)
    # prompt
    ops.moe_route_only(h, norm_w, 1e-6, router, k, True, ids, wts, xn)
    pos, rows, tiles, xg, prompt = i32(T, k), i32(E + 1), i32(E + 1), torch.zeros(T * k, d, dtype=torch.bfloat16, device=DEV), h.clone()
    ops.moe_sort(ids, wts, 0, E, 256, pos, rows, tiles, xn, xg)
    ops.gemm_grouped(gu, xg, act, rows, tiles, 256, epi=ops.EPI_SWIGLU, scratch=sc)
    ops.gemm_grouped(dn, act, y, rows, tiles, 256, scratch=sc)
    ops.moe_combine_sorted(prompt, y, pos, wts, k)
    # decode step
    z_max = E + (T * k + 3) // 4
    items, n_items, step, ids2, wts2 = i32(z_max * ops.MOE_ITEM_INTS), i32(1), h.clone(), i32(T, k), torch.zeros(T, k, device=DEV)
    ops.moe_route(h, norm_w, 1e-6, router, k, True, 0, E, ids2, wts2, items, n_items, i32(1))
    ops.moe_gate_up(gu, step, norm_w, 1e-6, act, items, n_items, k, z_max, scratch=sc)
    ops.moe_down_combine(dn, act, y, items, n_items, z_max, ids2, wts2, k, 0, E, step, i32((d + 127) // 128), scratch=sc)
    x = h.double() * torch.rsqrt(h.double().square().mean(-1, keepdim=True) + 1e-6) * 0.01
    want = torch.zeros_like(x)
    for t in range(T):
        for j in range(k):
            G, U, D = deq[int(ids[t, j])]
            want[t] += wts[t, j].double() * (D @ (torch.nn.functional.silu(G @ x[t]) * (U @ x[t])))
    # rows, weights and hidden rows are rounded to bf16 (prompt), rows and hidden rows to 8 bits per 32 values, about 0.4 % each (step)
    assert int(sc.status[0]) == 0
    for got in (prompt, step):
        assert (got.double() - h.double() - want).norm() <= 1.5e-2 * want.norm()
