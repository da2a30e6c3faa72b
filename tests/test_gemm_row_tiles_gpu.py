"""The persistent dequantising GEMM at the edges of its 32-, 64- and 128-row tiles."""
import pytest
import torch

from llaminar_b200.gguf import GGMLType, dequantize, quantize

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp(min=1e-12)).item()


@pytest.mark.parametrize("qt", [GGMLType.Q4_K, GGMLType.Q5_K, GGMLType.Q6_K, GGMLType.Q8_0, GGMLType.Q4_0, GGMLType.IQ3_S])
@pytest.mark.parametrize("m", [32, 33, 64, 65, 127, 128, 129])
@pytest.mark.parametrize("n,k", [(200, 256), (4096, 1792), (1280, 9472)])
def test_row_tile_edges(qt, m, n, k):
    """One ragged tile; more tiles than SMs share evenly; tiles split between several CTAs.  Operands are rounded to bf16 (2^-9 of a
    value at most, 2^-9 / sqrt(3) on average, twice): 1.2e-2 leaves room for the formats whose scale and minimum are rounded too."""
    from llaminar_b200 import ops
    from llaminar_b200.ops.layout import interleave_gate_up
    g = torch.Generator(device=DEV).manual_seed(m)
    raw = quantize(torch.randn(n, k, generator=g, device=DEV) * 0.05, qt)
    wf = dequantize(raw, qt, (n, k))
    pw = ops.pack_matrix(raw, qt, n, k)
    sc = ops.scratch_for(DEV)
    sc.status.zero_()
    x = torch.randn(m, k, generator=g, device=DEV).to(torch.bfloat16)
    ref = x.float() @ wf.T
    wide = torch.full((m + 1, n + 8), 7.0, dtype=torch.bfloat16, device=DEV)
    out = wide[:m, :n]                                   # rows and columns behind the result must stay as they are
    ops.gemm(pw, x, out, scratch=sc)
    whole = torch.empty(m, n, dtype=torch.float32, device=DEV)
    ops.gemm(pw, x, whole, scratch=sc, ksplit=1)         # no tile is split
    bias, h0 = torch.randn(n, generator=g, device=DEV), torch.randn(m, n, generator=g, device=DEV)
    h = h0.clone()
    ops.gemm(pw, x, h, epi=ops.EPI_RESID, bias=bias, scratch=sc)
    again = h0.clone()
    ops.gemm(pw, x, again, epi=ops.EPI_RESID, bias=bias, scratch=sc)
    gu = n // 32 * 16
    raw2, _, n2, _ = interleave_gate_up(raw[:raw.numel() // n * gu], raw[raw.numel() // n * gu:raw.numel() // n * 2 * gu], qt, gu, k)
    act = torch.empty(m, gu, dtype=torch.bfloat16, device=DEV)
    ops.gemm(ops.pack_matrix(raw2, qt, n2, k), x, act, epi=ops.EPI_SWIGLU, scratch=sc)
    torch.cuda.synchronize()
    assert int(sc.status[0]) == 0 and int(sc.tickets.abs().sum()) == 0
    assert _rel(out, ref) < 1.2e-2 and _rel(whole, ref) < 1.2e-2 and _rel(h - h0 - bias, ref) < 1.2e-2
    if m <= 128:
        assert torch.equal(h, again)                     # partial sums meet in CTA order
    assert bool((wide[m:] == 7.0).all()) and bool((wide[:, n:] == 7.0).all())
    gate, up = ref[:, :gu], ref[:, gu:2 * gu]
    assert _rel(act, torch.nn.functional.silu(gate) * up) < 2.4e-2


@pytest.mark.parametrize("qt", [GGMLType.Q4_K, GGMLType.Q8_0])
@pytest.mark.parametrize("n,k", [(640, 16384), (2000, 9728), (300, 4096)])
@pytest.mark.parametrize("m", [129, 160, 256, 300])
def test_long_and_narrow(qt, n, k, m):
    """Shapes around the line where K is split between CTAs whose sums meet by atomics: values, and counters and sums back at zero."""
    from llaminar_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(m)
    raw = quantize(torch.randn(n, k, generator=g, device=DEV) * 0.05, qt)
    pw, sc = ops.pack_matrix(raw, qt, n, k), ops.scratch_for(DEV)
    sc.status.zero_()
    x = torch.randn(m, k, generator=g, device=DEV).to(torch.bfloat16)
    ref = x.float() @ dequantize(raw, qt, (n, k)).T
    out, h0 = torch.empty(m, n, dtype=torch.bfloat16, device=DEV), torch.randn(m, n, generator=g, device=DEV)
    h = h0.clone()
    ops.gemm(pw, x, out, scratch=sc)
    ops.gemm(pw, x, h, epi=ops.EPI_RESID, scratch=sc)
    torch.cuda.synchronize()
    assert int(sc.status[0]) == 0 and int(sc.tickets.abs().sum()) == 0 and float(sc.accum.abs().max()) == 0
    assert _rel(out, ref) < 1.2e-2 and _rel(h - h0, ref) < 1.2e-2
