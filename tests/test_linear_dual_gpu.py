"""Two matrices of different block formats in one launch, against 32 bits and against one launch each."""
import pytest
import torch

from llaminar_b200.gguf import GGMLType, dequantize, quantize

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm()).item()


@pytest.mark.parametrize("fa,fb", [(GGMLType.Q4_K, GGMLType.Q6_K), (GGMLType.Q4_K, GGMLType.Q5_K), (GGMLType.Q5_K, GGMLType.Q6_K)])
@pytest.mark.parametrize("rows", [1, 2, 3, 4, 5, 32, 33, 64, 100, 128])
@pytest.mark.parametrize("na,nb,k", [(256, 128, 256), (200, 100, 768), (5120, 1024, 2048), (128, 4096, 1024), (128, 128 * 500, 1024)])
def test_dual(fa, fb, rows, na, nb, k):
    """A tile or less each, more CTAs than chunks, ragged columns, the second matrix the larger one, and all but a five hundredth."""
    from llaminar_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(rows)
    raw = [quantize(torch.randn(n, k, device=DEV, generator=g) * 0.05, f) for n, f in ((na, fa), (nb, fb))]
    a, b = (ops.pack_matrix(r, f, n, k) for r, f, n in zip(raw, (fa, fb), (na, nb)))
    sc = ops.scratch_for(DEV)
    sc.status.zero_()
    x, gain, bias = torch.randn(rows, k, device=DEV, generator=g), torch.rand(k, device=DEV, generator=g) + 0.5, torch.randn(na + nb, device=DEV, generator=g)
    out, apart = (torch.full((rows + 1, na + nb + 8), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    parts = lambda o: (o[:rows, :na], o[:rows, na:na + nb])
    if rows <= ops.GEMV_MAX_ROWS:
        how, ref = dict(norm_w=gain), x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * gain
        for w, o, bi in zip((a, b), parts(apart), (bias[:na], bias[na:])):
            ops.gemv(w, x, o, norm_w=gain, bias=bi, scratch=sc)
    else:
        x = x.bfloat16()
        how, ref = {}, x.float()
        for w, o, bi in zip((a, b), parts(apart), (bias[:na], bias[na:])):
            ops.gemm(w, x, o, bias=bi, scratch=sc)
    assert ops.linear_dual(a, b, x, *parts(out), sc, bias_a=bias[:na], bias_b=bias[na:], **how)
    assert int(sc.status[0]) == 0 and int(sc.tickets.abs().sum()) == 0
    assert bool((out[rows:] == 7.0).all()) and bool((out[:, na + nb:] == 7.0).all())
    want = torch.cat([ref @ dequantize(r, f, (n, k)).T for r, f, n in zip(raw, (fa, fb), (na, nb))], 1) + bias
    # 8-bit activation blocks (rms 1 / 254 / sqrt(3) of the largest of 32 values) or bf16 operands; the two ways only order their sums differently
    assert _rel(out[:rows, :na + nb], want) < 1.5e-2 and _rel(out[:rows], apart[:rows]) < 3e-3


def test_other_mixes_are_left_alone():
    from llaminar_b200 import ops
    ws = [ops.pack_matrix(quantize(torch.randn(128, 256, device=DEV), f), f, 128, 256) for f in (GGMLType.Q6_K, GGMLType.Q4_K)]
    out = torch.full((8, 256), 7.0, dtype=torch.bfloat16, device=DEV)
    assert not ops.linear_dual(*ws, torch.randn(8, 256, device=DEV).bfloat16(), out[:, :128], out[:, 128:], ops.scratch_for(DEV))
    assert bool((out == 7.0).all())
