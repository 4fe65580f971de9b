"""Decode attention of many sequences, one share each: blocks of two compute warps where three of them an SM hold all, of three else."""
import math

import pytest
import torch


def _plain(q, k, v, lens, table, nh, nkv, hd):
    out = torch.empty(len(lens), nh, hd, dtype=torch.float64, device=q.device)
    for s, n in enumerate(lens):
        pages = table[s, :(n + 63) // 64].long()
        for h in range(nkv):
            kk, vv = (t[pages, h].reshape(-1, hd)[:n].double() for t in (k, v))
            g = nh // nkv
            w = torch.softmax(q.view(len(lens), nh, hd)[s, h * g:(h + 1) * g].double() @ kk.T / math.sqrt(hd), -1)
            out[s, h * g:(h + 1) * g] = w @ vv
    return out.view(len(lens), -1)


@pytest.mark.gpu
@pytest.mark.parametrize("nh,nkv,hd", [(8, 2, 128), (12, 4, 64), (16, 1, 128)])
@pytest.mark.parametrize("over", [0, 1, 40])          # blocks: two an SM and none, a few, many more; at 40 with one kv head three and more
def test_blocks_between_two_and_three_an_sm(nh, nkv, hd, over):
    from synaptix_b200.ops.attention import attn_decode_status, attn_decode_tma
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    S = 2 * sms // nkv + over + (sms if over == 40 and nkv == 1 else 0)
    lens = [(1, 63, 64, 65, 127, 129, 200, 257)[i % 8] + (i % 5) * (i % 8 > 5) for i in range(S)]
    need = [(n + 63) // 64 for n in lens]
    table, at = torch.zeros(S, max(need), dtype=torch.int32), 1
    for s, n in enumerate(need):
        table[s, :n] = torch.arange(at, at + n)
        at += n
    g = torch.Generator().manual_seed(S)
    k, v = (torch.randn(at, nkv, 64, hd, generator=g).to(torch.bfloat16).cuda() for _ in range(2))
    for t in (k, v):
        for s, n in enumerate(lens):
            t[table[s, need[s] - 1].item(), :, (n - 1) % 64 + 1:] = float("nan")       # (what no step wrote)
    q = torch.randn(S, nh * hd, generator=g).to(torch.bfloat16).cuda()
    got = attn_decode_tma(q, k, v, torch.tensor(lens, dtype=torch.int32).cuda(), table.cuda(), nh, nkv, hd, 1 / math.sqrt(hd), None, 1)
    want = _plain(q, k, v, lens, table, nh, nkv, hd)
    # weights and results are rounded to bfloat16 (2^-9 each) and values are about 1: 4 units of that, times the largest value
    assert (got.double() - want).abs().max() <= 4 * 2 ** -9 * v[~v.isnan()].abs().max()
    assert attn_decode_status() == 0
