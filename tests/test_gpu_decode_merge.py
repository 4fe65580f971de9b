"""Decode attention's results and partial results written four at a time: the same bits where the output starts at an odd place."""
import math

import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("nh,nkv,hd", [(32, 8, 128), (5, 1, 64), (16, 1, 128), (3, 3, 128)])
@pytest.mark.parametrize("splits,cluster", [(1, None), (2, True), (4, True), (8, True), (16, True), (3, None), (4, False)])
def test_output_at_an_odd_place(nh, nkv, hd, splits, cluster):
    from synaptix_b200.ops.attention import attn_decode_status, attn_decode_tma
    g = torch.Generator().manual_seed(nh)
    lens = [1, 63, 64, 65, 700]
    need = [(n + 63) // 64 for n in lens]
    table, at = torch.zeros(len(lens), max(need), dtype=torch.int32), 1
    for s, n in enumerate(need):
        table[s, :n] = torch.arange(at, at + n)
        at += n
    k, v = (torch.randn(at, nkv, 64, hd, generator=g).to(torch.bfloat16).cuda() for _ in range(2))
    q = torch.randn(len(lens), nh * hd, generator=g).to(torch.bfloat16).cuda()
    run = lambda out: attn_decode_tma(q, k, v, torch.tensor(lens, dtype=torch.int32).cuda(), table.cuda(), nh, nkv, hd,
                                      1 / math.sqrt(hd), None, splits, out=out, cluster=cluster)
    n = len(lens) * nh * hd
    buf = torch.full((n + 2,), float("nan"), dtype=torch.bfloat16, device="cuda")
    want = run(torch.full((len(lens), nh * hd), float("nan"), dtype=torch.bfloat16, device="cuda"))
    got = run(buf[1:n + 1].view(len(lens), -1))
    assert torch.equal(got, want) and not torch.isnan(want.float()).any()
    assert torch.isnan(buf[0].float()) and torch.isnan(buf[-1].float())          # and nothing beside it
    assert attn_decode_status() == 0
