"""Prompt attention with two query heads a block (many query tiles, an even number of heads a key/value head): against 64-bit
attention at the edges of query tiles, pages and key blocks, with a cache before the prompt, a window and sinks."""
import math

import pytest
import torch

BF = torch.bfloat16


@pytest.mark.gpu
@pytest.mark.parametrize("nh,nkv", [(32, 8), (16, 8), (24, 2)])
@pytest.mark.parametrize("new,past", [([1, 127, 128, 129, 257, 300] * 3, [0, 0, 0, 0, 0, 0] * 3),
                                      ([64, 65, 130, 385] * 5, [1, 63, 127, 500] * 5), ([1700, 1411], [0, 33])])
@pytest.mark.parametrize("window,sink", [(None, False), (100, True)])
def test_against_64_bit(nh, nkv, new, past, window, sink):
    from synaptix_b200.ops.attention import attn_prefill_tc, attn_tc_status
    hd, g = 128, torch.Generator().manual_seed(nh + sum(new))
    T, lens = sum(new), [a + b for a, b in zip(new, past)]
    need = [(n + 63) // 64 for n in lens]
    order = torch.randperm(sum(need), generator=g).add(1).tolist()        # page 0 belongs to nobody
    table = torch.zeros(len(new), max(need), dtype=torch.int32)
    k = torch.full((sum(need) + 1, nkv, 64, hd), float("nan"), dtype=BF)
    v = k.clone()
    keys, values = [], []
    for s, n in enumerate(lens):
        keys.append(torch.randn(n, nkv, hd, generator=g).to(BF))
        values.append(torch.randn(n, nkv, hd, generator=g).to(BF))
        for i in range(need[s]):
            page = table[s, i] = order.pop()
            m = min(64, n - 64 * i)
            k[page, :, :m] = keys[s][64 * i:64 * i + m].transpose(0, 1)
            v[page, :, :m] = values[s][64 * i:64 * i + m].transpose(0, 1)
    q = (torch.randn(T, nh * hd, generator=g) * 2).to(BF)
    sinks = torch.randn(nh, generator=g) if sink else None
    tiles = [(s, t) for t in range(0, max(new), 128) for s in range(len(new)) if t < new[s]]
    assert 4 * (nh // 2) * len(tiles) >= 5 * torch.cuda.get_device_properties(0).multi_processor_count
    i32 = lambda x: torch.tensor(x, dtype=torch.int32).cuda()
    cu = [sum(new[:i]) for i in range(len(new) + 1)]
    out = attn_prefill_tc(q.cuda(), k.cuda(), v.cuda(), i32([s for s, _ in tiles]), i32([t for _, t in tiles]), i32(cu), i32(past),
                          i32(lens), table.cuda(), nh, nkv, hd, 1 / math.sqrt(hd), window, sinks=None if sinks is None else sinks.cuda())
    out = out.view(T, nh, hd).double()
    for s in range(len(new)):
        qs = q[cu[s]:cu[s + 1]].view(-1, nh, hd).cuda().double()
        pos, at = torch.arange(past[s], lens[s]).cuda()[:, None], torch.arange(lens[s]).cuda()[None]
        seen = (at <= pos) & ((at > pos - window) if window else True)
        for h in range(nh):
            sc = (qs[:, h] @ keys[s][:, h // (nh // nkv)].cuda().double().T / math.sqrt(hd)).masked_fill(~seen, -math.inf)
            if sink:
                sc = torch.cat([sc, sinks[h].double().cuda().expand(new[s], 1)], 1)
            p = torch.softmax(sc, -1)[:, :lens[s]]
            val = values[s][:, h // (nh // nkv)].cuda().double()
            want = p @ val
            # P is rounded to bfloat16 (2^-9 of every term; as much again for the scores, the exponentials and the sums), the result too
            bound = 2.0 ** -8 * (p @ val.abs()) + 2.0 ** -8 * want.abs() + 1e-6
            assert ((out[cu[s]:cu[s + 1], h] - want).abs() <= bound).all(), (s, h)
    assert attn_tc_status() == 0
