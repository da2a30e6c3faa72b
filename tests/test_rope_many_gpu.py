"""Rotation, norms and cache append of long chunks: a warp takes eight heads of a token, the last one of a token fewer."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("heads,kv_heads", [(16, 4), (7, 1), (1, 1), (12, 2)])
@pytest.mark.parametrize("q8", [False, True])
@pytest.mark.parametrize("odd", [0, 1])
def test_chunk_equals_its_tokens(D, heads, kv_heads, q8, odd):
    """The values of a chunk are, bit for bit, those of its tokens in portions that a warp per head takes; rows that start between two
    words too."""
    from llaminar_b200 import ops
    total = heads + 2 * kv_heads
    T = 4736 // ((total + 7) // 8) + 5
    g = torch.Generator(device=DEV).manual_seed(heads)
    qkv = torch.randn(T, total * D, device=DEV, generator=g).bfloat16()
    qn, kn = (torch.rand(D, device=DEV, generator=g) + 0.5 for _ in range(2))
    pages = (T + 63) // 64
    data = 2 * kv_heads * 64 * D
    i32 = lambda x: x.to(torch.int32).to(DEV)
    pos, table, sid = i32(torch.arange(T)), i32(torch.randperm(pages)).view(1, pages), torch.zeros(T, dtype=torch.int32, device=DEV)

    def run(step):
        kv = torch.zeros(pages, data + data // 16, dtype=torch.uint8, device=DEV) if q8 else torch.zeros(pages, 2, kv_heads, 64, D, dtype=torch.bfloat16, device=DEV)
        q = torch.zeros(T, heads, D, dtype=torch.bfloat16, device=DEV)
        for t in range(0, T, step):
            s = slice(t, min(t + step, T))
            rows = torch.empty(qkv[s].numel() + odd, dtype=torch.bfloat16, device=DEV)[odd if step == T else 0:][:qkv[s].numel()].view_as(qkv[s]).copy_(qkv[s])
            ops.rope_kv(rows, q[s], kv, qn, kn, pos[s], sid[s], table, heads, kv_heads, D, 1e6, 1e-6)
        return q, kv

    (q, kv), (q1, kv1) = run(T), run(300)
    assert torch.equal(q, q1) and torch.equal(kv, kv1) and bool((q != 0).any())
