"""Single-token attention whose splits meet in a thread-block cluster or through scratch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 3])
@pytest.mark.parametrize("n_splits", [2, 3, 5, 6, 7, 8, 9, 13])
def test_attention_splits_that_meet_in_a_cluster_or_through_scratch(n_splits, T):
    """One round of chunks a block: up to 8 splits of a (row, key/value head) merge as a cluster while the grid has at most 32
    blocks, others through scratch; rows whose sequences end inside the first, a middle and the last split; with and
    without the sink."""
    from tinyllama_c_b200 import ops
    g = torch.Generator().manual_seed(n_splits)
    H, KV, hd = 6, 2, 64
    lens = [128 * n_splits, 1 + 5, 128 * ((n_splits + 1) // 2) - 3][:T]
    max_keys = 128 * n_splits
    pages = [(n + 63) // 64 for n in lens]
    table = torch.zeros(T, max(pages), dtype=torch.int32)
    at = 1
    for t, n in enumerate(pages):
        table[t, :n] = torch.arange(at, at + n)
        at += n
    k, v = (torch.randn(at, KV, 64, hd, generator=g).bfloat16() for _ in range(2))
    qkv = torch.randn(T, (H + 2 * KV) * hd, generator=g)
    pos = torch.tensor([n - 1 for n in lens], dtype=torch.int32)
    ar = torch.arange(T, dtype=torch.int32)
    none = torch.zeros(0)
    try:
        ops.attention_decode_fused_passes(1)
        for sink in (False, True):
            kd, vd, out = k.cuda(), v.cuda(), torch.empty(T, H * hd, device="cuda", dtype=torch.bfloat16)
            arrivals = ops.new_arrival_counters(torch.device("cuda"))
            for _ in range(2):
                ops.attention_decode_fused(qkv.cuda(), 0, H * hd, (H + KV) * hd, kd, vd, none.cuda(), True, table.cuda(), pos.cuda(), ar.cuda(),
                                           ar.cuda(), out, H, KV, hd, 0.125, 0, max_keys, arrivals, sink=sink)
            torch.cuda.synchronize()
            for t, n in enumerate(lens):
                q = qkv[t, :H * hd].bfloat16().double().view(H, hd)
                rows = [x[table[t].long()].permute(1, 0, 2, 3).reshape(KV, -1, hd)[:, :n].double().clone() for x in (k, v)]
                rows[0][:, n - 1] = qkv[t, H * hd:(H + KV) * hd].bfloat16().double().view(KV, hd)
                rows[1][:, n - 1] = qkv[t, (H + KV) * hd:].bfloat16().double().view(KV, hd)
                kk, vv = (x.repeat_interleave(H // KV, 0) for x in rows)
                s = torch.einsum("hd,hnd->hn", q, kk) * 0.125
                if sink:
                    s = torch.cat([s, torch.zeros(H, 1, dtype=torch.float64)], 1)
                p = s.softmax(-1)[:, :n]
                ref = torch.einsum("hn,hnd->hd", p, vv).reshape(-1)
                # weights and result are rounded to 8 bits of mantissa
                assert (out[t].cpu().double() - ref).abs().max().item() <= 2.0 ** -8 * (ref.abs().max().item() + vv.abs().max().item() * 2.0 ** -1), (t, sink)
    finally:
        ops.attention_decode_fused_passes(0)


@pytest.mark.parametrize("T", [1, 9])
@pytest.mark.parametrize("n_splits", [1, 3])
@pytest.mark.parametrize("what", ["one key", "every key of a split"])
def test_a_nan_among_the_scores_reaches_the_result_by_every_route(n_splits, T, what):
    """One block a (row, head), a cluster (T 1) and scratch (T 9): the heads whose keys hold a NaN are NaN in the row that sees
    them, everything else is finite."""
    from tinyllama_c_b200 import ops
    g = torch.Generator().manual_seed(3)
    H, KV, hd, n = 6, 2, 64, 128 * n_splits
    table = (1 + torch.arange(T * 2 * n_splits, dtype=torch.int32)).view(T, 2 * n_splits)
    k, v = (torch.randn(1 + T * 2 * n_splits, KV, 64, hd, generator=g).bfloat16() for _ in range(2))
    if what == "one key":
        k[table[0, 0], 1, 17, 3] = float("nan")
    else:
        k[table[0, :2].long(), 1] = float("nan")
    qkv = torch.randn(T, (H + 2 * KV) * hd, generator=g).cuda()
    pos, ar = torch.full((T,), n - 1, dtype=torch.int32).cuda(), torch.arange(T, dtype=torch.int32).cuda()
    kd, vd, out, table = k.cuda(), v.cuda(), torch.empty(T, H * hd, device="cuda", dtype=torch.bfloat16), table.cuda()
    try:
        ops.attention_decode_fused_passes(1)
        ops.attention_decode_fused(qkv, 0, H * hd, (H + KV) * hd, kd, vd, torch.zeros(0).cuda(), True, table, pos, ar, ar, out, H, KV, hd, 0.125,
                                   0, n, ops.new_arrival_counters(torch.device("cuda")))
        torch.cuda.synchronize()
    finally:
        ops.attention_decode_fused_passes(0)
    bad = out.float().isnan().view(T, H, hd)
    assert bad[0, 3:].all() and not bad[0, :3].any() and not bad[1:].any()
