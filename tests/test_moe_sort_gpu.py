"""Routing of a prompt and the order of its rows by expert."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("tokens,k,E,e0,n_local,bm", [(1, 8, 128, 0, 128, 256), (700, 8, 128, 0, 128, 256), (333, 3, 256, 0, 256, 64), (1000, 8, 128, 32, 48, 128), (50, 2, 8, 6, 2, 256)])
def test_sort(tokens, k, E, e0, n_local, bm):
    from llaminar_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(tokens)
    ids = torch.stack([torch.randperm(E, device=DEV, generator=g)[:k] for _ in range(tokens)]).to(torch.int32)
    wts = torch.rand(tokens, k, device=DEV, generator=g) + 0.1
    xn = torch.randn(tokens, 512, device=DEV, generator=g).bfloat16()
    i32 = lambda *s: torch.full(s, -1, dtype=torch.int32, device=DEV)
    pos, rows, tiles, xg, w = i32(tokens, k), i32(n_local + 1), i32(n_local + 1), torch.zeros(tokens * k, 512, dtype=torch.bfloat16, device=DEV), wts.clone()
    ops.moe_sort(ids, w, e0, n_local, bm, pos, rows, tiles, xn, xg)
    local = (ids >= e0) & (ids < e0 + n_local)
    key = torch.where(local, ids - e0, torch.full_like(ids, n_local)).view(-1).long()
    order = torch.argsort(key, stable=True)
    want = torch.empty_like(order)
    want[order] = torch.arange(tokens * k, device=DEV)
    counts = torch.bincount(key, minlength=n_local + 1)[:n_local]
    zero = torch.zeros(1, dtype=torch.long, device=DEV)
    assert torch.equal(pos.view(-1).long(), want)
    assert torch.equal(rows.long(), torch.cat([zero, counts.cumsum(0)])) and torch.equal(tiles.long(), torch.cat([zero, ((counts + bm - 1) // bm).cumsum(0)]))
    assert torch.equal(w, torch.where(local, wts, torch.zeros_like(wts))) and torch.equal(xg, xn[order // k])


def test_route_of_many_tokens_equals_route_of_few():
    """Eight tokens per CTA and one: the same numbers in the same order."""
    from llaminar_b200 import ops
    T, E, k, d = 445, 100, 6, 1024
    g = torch.Generator(device=DEV).manual_seed(0)
    h, w = torch.randn(T, d, device=DEV, generator=g), torch.rand(d, device=DEV, generator=g) + 0.5
    router = (torch.randn(E, d, device=DEV, generator=g) * 0.1).bfloat16()

    def run(step):
        ids, wts, xn = torch.zeros(T, k, dtype=torch.int32, device=DEV), torch.zeros(T, k, device=DEV), torch.zeros(T, d, dtype=torch.bfloat16, device=DEV)
        for t in range(0, T, step):
            s = slice(t, min(T, t + step))
            ops.moe_route_only(h[s], w, 1e-6, router, k, True, ids[s], wts[s], xn[s])
        return ids, wts, xn

    for a, b in zip(run(T), run(100)):
        assert torch.equal(a, b)
