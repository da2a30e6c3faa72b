"""The dequantising GEMM of CTA pairs at the edges of its tiles: 256 weight rows (two tiles of 128), up to 256 tokens in steps of 32,
chunks of 256 columns that two sets of warps take in turn."""
import pytest
import torch

from llaminar_b200.gguf import GGMLType, dequantize, quantize

pytestmark = pytest.mark.gpu
DEV = "cuda"
FORMATS = [GGMLType.Q4_K, GGMLType.Q5_K, GGMLType.Q6_K, GGMLType.Q8_0, GGMLType.Q4_0, GGMLType.IQ3_S]
# operands are rounded to bf16 (2^-9 of a value at most, 2^-9 / sqrt(3) on average, twice); 1.2e-2 leaves room for the formats whose
# scale and minimum are rounded too
REL = 1.2e-2


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp(min=1e-12)).item()


@pytest.mark.parametrize("qt", FORMATS)
@pytest.mark.parametrize("m,n,k", [(129, 100, 256), (160, 128, 512), (257, 384, 768), (500, 1000, 1792), (300, 19200, 256), (1031, 4224, 1280)])
def test_pair_edges(qt, m, n, k):
    """One tile and many per pair, an odd number of weight tiles and of chunks, one chunk per tile, ragged rows and columns."""
    from llaminar_b200 import ops
    from llaminar_b200.ops.layout import interleave_gate_up
    g = torch.Generator(device=DEV).manual_seed(m)
    raw = quantize(torch.randn(n, k, generator=g, device=DEV) * 0.05, qt)
    pw, sc = ops.pack_matrix(raw, qt, n, k), ops.scratch_for(DEV)
    sc.status.zero_()
    x = torch.randn(m, k, generator=g, device=DEV).to(torch.bfloat16)
    ref = x.float() @ dequantize(raw, qt, (n, k)).T
    wide = torch.full((m + 1, n + 8), 7.0, dtype=torch.bfloat16, device=DEV)
    out = wide[:m, :n]                                   # rows and columns behind the result must stay as they are
    ops.gemm(pw, x, out, scratch=sc)
    bias, h0 = torch.randn(n, generator=g, device=DEV), torch.randn(m, n, generator=g, device=DEV)
    h = h0.clone()
    ops.gemm(pw, x, h, epi=ops.EPI_RESID, bias=bias, scratch=sc)
    whole, bare, added = torch.empty(m, n, dtype=torch.float32, device=DEV), torch.empty(m, n, dtype=torch.float32, device=DEV), h0.clone()
    ops.gemm(pw, x, whole, bias=bias, scratch=sc)
    ops.gemm(pw, x, bare, scratch=sc)
    ops.gemm(pw, x, added, epi=ops.EPI_RESID, scratch=sc)
    gu = n // 32 * 16
    row = raw.numel() // n
    raw2, _, n2, _ = interleave_gate_up(raw[:row * gu], raw[row * gu:row * 2 * gu], qt, gu, k)
    act = torch.empty(m, gu, dtype=torch.bfloat16, device=DEV)
    ops.gemm(ops.pack_matrix(raw2, qt, n2, k), x, act, epi=ops.EPI_SWIGLU, scratch=sc)
    torch.cuda.synchronize()
    assert int(sc.status[0]) == 0
    assert _rel(out, ref) < REL and _rel(h - h0 - bias, ref) < REL and _rel(whole - bias, ref) < REL
    assert torch.equal(added, h0 + bare)                 # the same sums, and one rounded addition
    assert bool((wide[m:] == 7.0).all()) and bool((wide[:, n:] == 7.0).all())
    assert _rel(act, torch.nn.functional.silu(ref[:, :gu]) * ref[:, gu:2 * gu]) < 2 * REL


@pytest.mark.parametrize("qt", [GGMLType.Q4_K, GGMLType.Q6_K])
@pytest.mark.parametrize("bm", [64, 128, 256])
def test_groups(qt, bm):
    """Groups without rows, of one row, of whole tiles and beyond; rows behind the last group stay as they are."""
    from llaminar_b200 import ops
    sizes, n, k = [0, 1, bm, bm + 1, 0, 31, 33, 3 * bm - 5, 0], 384, 768
    g = torch.Generator(device=DEV).manual_seed(bm)
    E, P = len(sizes), sum(sizes)
    raw = [quantize(torch.randn(n, k, generator=g, device=DEV) * 0.05, qt) for _ in sizes]
    pw, sc = ops.pack_experts(torch.cat(raw), qt, E, n, k), ops.scratch_for(DEV)
    sc.status.zero_()
    x = torch.randn(P + 3, k, generator=g, device=DEV).to(torch.bfloat16)
    out = torch.full((P + 3, n), 7.0, device=DEV)
    rows = torch.tensor([0] + sizes).cumsum(0).to(torch.int32).to(DEV)
    tiles = torch.tensor([0] + [(s + bm - 1) // bm for s in sizes]).cumsum(0).to(torch.int32).to(DEV)
    ops.gemm_grouped(pw, x, out, rows, tiles, bm, scratch=sc)
    torch.cuda.synchronize()
    assert int(sc.status[0]) == 0 and bool((out[P:] == 7.0).all())
    at = 0
    for s, r in zip(sizes, raw):
        if s:
            assert _rel(out[at:at + s], x[at:at + s].float() @ dequantize(r, qt, (n, k)).T) < REL
        at += s
