"""The tcgen05 prefill attention at the edges of its tiles: 128 query rows and 128 keys, two slots (heads of a group, or query tiles
where the group is odd) per CTA."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
# P is rounded to bf16 (2^-9 of each term at most, zero mean), the output once more; the sums are fp32
REL = 6e-3


def _reference(q, k, v, ctx, window=0, softcap=0.0, sink=None):
    """q [L, H, D] behind ctx keys, k / v [ctx + L, Hk, D]; 64-bit."""
    L, H, D = q.shape
    k, v = (x.double().repeat_interleave(H // x.shape[1], 1) for x in (k, v))
    s = torch.einsum("lhd,shd->hls", q.double(), k) / math.sqrt(D)
    if softcap:
        s = softcap * torch.tanh(s / softcap)
    row, col = torch.arange(L, device=DEV)[:, None] + ctx, torch.arange(ctx + L, device=DEV)[None]
    s = s.masked_fill((col > row) | (window > 0) & (col <= row - window), -math.inf)
    if sink is not None:
        s = torch.cat([s, sink.double()[:, None, None].expand(H, L, 1)], 2)
        v = torch.cat([v, torch.zeros_like(v[:1])])
    return torch.einsum("hls,shd->lhd", torch.softmax(s, -1), v)


def _case(heads, kv_heads, lens, ctx, rising, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    D, B = 128, len(lens)
    pages = max((c + n + 63) // 64 for c, n in zip(ctx, lens)) + 1
    table = torch.randperm(B * pages, generator=torch.Generator().manual_seed(seed)).view(B, pages).to(torch.int32).to(DEV)
    kv = torch.zeros(B * pages, 2, kv_heads, 64, D, dtype=torch.bfloat16, device=DEV)
    q = torch.randn(sum(lens), heads, D, device=DEV, generator=g)
    if rising:
        q[..., 0] = 4.0                                          # scores grow with the key's place: the running maximum rises tile by tile
    q, keys, values = q.bfloat16(), [], []
    for b, (c, n) in enumerate(zip(ctx, lens)):
        k, v = torch.randn(2, c + n, kv_heads, D, device=DEV, generator=g).bfloat16()
        if rising:
            k[..., 0] = (torch.arange(c + n, device=DEV) * 0.05)[:, None]
        keys.append(k)
        values.append(v)
        for t in range(0, c + n, 64):
            part = slice(t, min(t + 64, c + n))
            for i, x in enumerate((k, v)):
                kv[table[b, t // 64], i, :, :part.stop - t] = x[part].transpose(0, 1)
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    return q, kv, table, cu, torch.tensor(ctx, dtype=torch.int32, device=DEV), keys, values


def _check(out, q, cu, ctx, keys, values, **how):
    for b, (k, v) in enumerate(zip(keys, values)):
        rows = slice(int(cu[b]), int(cu[b + 1]))
        want = _reference(q[rows], k, v, int(ctx[b]), **how)
        assert (out[rows].double() - want).norm() <= REL * want.norm(), b


@pytest.mark.parametrize("rising", [False, True])
@pytest.mark.parametrize("heads,kv_heads,lens,ctx", [
    (8, 2, [1, 127, 128], [0, 0, 0]), (8, 2, [129, 257], [63, 0]), (7, 1, [130, 3, 385], [0, 128, 1]), (14, 2, [255, 64], [1000, 65]),
    (3, 3, [129, 300], [0, 127]), (1, 1, [1], [0]), (16, 1, [17], [2500]), (28, 4, [37], [0])])
def test_tiles(heads, kv_heads, lens, ctx, rising):
    from llaminar_b200 import ops
    q, kv, table, cu, c, keys, values = _case(heads, kv_heads, lens, ctx, rising)
    out, sc = torch.full_like(q, float("nan")), ops.scratch_for(DEV)
    ops.attn_prefill(q, kv, out, table, cu, c, heads, kv_heads, 128, 1 / math.sqrt(128), max(lens), tensor_core=True, scratch=sc)
    assert int(sc.status[0]) == 0
    _check(out, q, cu, c, keys, values)


@pytest.mark.parametrize("heads,kv_heads,lens,ctx", [(8, 2, [1], [4000]), (7, 1, [130, 3], [1100, 2000]), (4, 4, [17, 250], [513, 0]), (32, 8, [40], [5000])])
def test_keys_shared_out(heads, kv_heads, lens, ctx):
    """Few query rows behind many keys: splits of equal tiles, a ragged last one, sequences with fewer tiles than splits."""
    from llaminar_b200 import ops
    q, kv, table, cu, c, keys, values = _case(heads, kv_heads, lens, ctx, True, 2)
    sc, outs = ops.scratch_for(DEV), []
    for longest in (0, max(n + m for n, m in zip(lens, ctx))):
        outs.append(torch.full_like(q, float("nan")))
        before = ops.launch_count()
        ops.attn_prefill(q, kv, outs[-1], table, cu, c, heads, kv_heads, 128, 1 / math.sqrt(128), max(lens), scratch=sc, max_kv_len=longest)
        assert ops.launch_count() - before == (2 if longest >= 1024 else 1)      # a split has four tiles of 128 keys at least
        _check(outs[-1], q, cu, c, keys, values)
    assert int(sc.status[0]) == 0


def test_many_short_prompts():
    """More CTAs than SMs and few keys each: the other kernel, by the sizes alone."""
    from llaminar_b200 import ops
    lens = [1 + i % 10 for i in range(40)]
    ctx = [i % 7 for i in range(40)]
    q, kv, table, cu, c, keys, values = _case(16, 16, lens, ctx, False, 4)
    out, sc = torch.full_like(q, float("nan")), ops.scratch_for(DEV)
    assert ops._few_keys_many_ctas(40, 16, 16, 10, 16)
    ops.attn_prefill(q, kv, out, table, cu, c, 16, 16, 128, 1 / math.sqrt(128), max(lens), scratch=sc, max_kv_len=16)
    _check(out, q, cu, c, keys, values)


@pytest.mark.parametrize("window,softcap,sink", [(1, 0.0, False), (100, 0.0, True), (129, 20.0, False), (0, 30.0, True)])
def test_masks(window, softcap, sink):
    from llaminar_b200.ops import grouped
    heads, kv_heads, lens, ctx = 7, 1, [140, 300], [200, 0]
    q, kv, table, cu, c, keys, values = _case(heads, kv_heads, lens, ctx, False, 1)
    logits = torch.randn(heads, device=DEV) if sink else None
    out, status = torch.full_like(q, float("nan")), torch.zeros(4, dtype=torch.int32, device=DEV)
    grouped.attn_prefill(q, kv, out, table, cu, c, 1 / math.sqrt(128), max(lens), window, logits, None, status, softcap=softcap)
    assert int(status[0]) == 0
    _check(out, q, cu, c, keys, values, window=window, softcap=softcap, sink=logits)


@pytest.mark.parametrize("window,softcap", [(0, 0.0), (100, 20.0)])
@pytest.mark.parametrize("bad", [math.inf, math.nan])
@pytest.mark.parametrize("heads,kv_heads,lens,ctx,late", [(8, 2, [200, 64, 1], [0, 100, 63], 130), (7, 1, [140, 300], [200, 0], 60), (4, 4, [17, 250], [513, 0], 9), (32, 8, [40], [2000], 30)])
def test_values_behind_the_mask(heads, kv_heads, lens, ctx, late, bad, window, softcap):
    """V rows that are not finite, of a later token and in what a page held before, reach no row that does not see them; rows that do
    are not finite in those columns and right in the others."""
    from llaminar_b200 import ops
    from llaminar_b200.ops import grouped
    q, kv, table, cu, c, keys, values = _case(heads, kv_heads, lens, ctx, False, 3)
    for b, (n, m) in enumerate(zip(lens, ctx)):
        end = n + m
        if end % 64:
            kv[table[b, end // 64], 1, :, end % 64:] = bad
        kv[table[b, end // 64 + 1], 1] = bad
        if n > late:
            at = m + late
            kv[table[b, at // 64], 1, :, at % 64, 5:9] = bad
            values[b][at, :, 5:9] = 0
    out, sc = torch.full_like(q, 7.0), ops.scratch_for(DEV)
    if window or softcap:
        grouped.attn_prefill(q, kv, out, table, cu, c, 1 / math.sqrt(128), max(lens), window, None, None, sc.status, softcap=softcap)
    else:
        ops.attn_prefill(q, kv, out, table, cu, c, heads, kv_heads, 128, 1 / math.sqrt(128), max(lens), tensor_core=True, scratch=sc, max_kv_len=max(n + m for n, m in zip(lens, ctx)))
    assert int(sc.status[0]) == 0
    for b, (k, v) in enumerate(zip(keys, values)):
        rows = slice(int(cu[b]), int(cu[b + 1]))
        want, got = _reference(q[rows], k, v, int(ctx[b]), window=window, softcap=softcap), out[rows].double()
        place = torch.arange(lens[b], device=DEV)
        sees = (place >= late) & ((place < late + window) if window else (place >= 0)) if lens[b] > late else torch.zeros_like(place, dtype=torch.bool)
        assert not bool(got[sees][..., 5:9].isfinite().any())
        got[sees.nonzero()[:, 0], :, 5:9] = want[sees.nonzero()[:, 0], :, 5:9]
        assert (got - want).norm() <= REL * want.norm(), b
