"""The row-by-row scan fetches four rows at a time, into two buffers in turn."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("aligned", [True, False])
@pytest.mark.parametrize("N,P", [(3, 5), (32, 16), (68, 20), (130, 12), (256, 64)])
@pytest.mark.parametrize("lens", [(1,), (7, 8, 9), (23, 1, 16)])
def test_scan_rows_staged_in_batches(lens, N, P, aligned):
    """Sequences that end before, at and after a batch, rows that are laid out in 16-byte pieces and rows that are not,
    states that start on a 16-byte boundary or 4 bytes past one; against the recurrence in 64 bits."""
    from tinyllama_c_b200 import ops
    g = torch.Generator().manual_seed(sum(lens) * 31 + N)
    Hs, G = 4, 2
    T, B, Di = sum(lens), len(lens), Hs * P
    Cd = Di + 2 * G * N
    xbc, dt = torch.randn(T, Cd, generator=g), torch.rand(T, Hs, generator=g)
    dA, D, state = torch.rand(T, Hs, generator=g), torch.randn(Hs, generator=g), torch.randn(B, Hs, P, N, generator=g)
    start = torch.tensor([3 if b % 2 else 0 for b in range(B)], dtype=torch.int32)
    cu = torch.tensor([sum(lens[:b]) for b in range(B + 1)], dtype=torch.int32)
    y_ref, S_ref = torch.empty(T, Di, dtype=torch.float64), state.double()
    for b in range(B):
        S = S_ref[b] if start[b] else torch.zeros(Hs, P, N, dtype=torch.float64)
        for t in range(cu[b], cu[b + 1]):
            x = xbc[t, :Di].double().view(Hs, P)
            Bm = xbc[t, Di:Di + G * N].double().view(G, N).repeat_interleave(Hs // G, 0)
            Cm = xbc[t, Di + G * N:].double().view(G, N).repeat_interleave(Hs // G, 0)
            S = S * dA[t].double()[:, None, None] + (x * dt[t].double()[:, None])[..., None] * Bm[:, None]
            y_ref[t] = ((S * Cm[:, None]).sum(-1) + x * D.double()[:, None]).reshape(-1)
        S_ref[b] = S
    y, off = torch.empty(T, Di, device="cuda"), 0 if aligned else 1
    st = torch.empty(state.numel() + off, device="cuda")[off:].view(state.shape)
    st.copy_(state)
    ops.ssm_scan(xbc.cuda(), dt.cuda(), dA.cuda(), D.cuda(), st, cu.cuda(), torch.arange(B, dtype=torch.int32).cuda(), start.cuda(), y, Hs, P, N, G)
    torch.cuda.synchronize()
    # products and sums of N terms in 32 bits over at most 23 rows
    assert (y.cpu().double() - y_ref).abs().max().item() <= (N + 40) * 2.0 ** -23 * 16 * N ** 0.5 * 4
    assert (st.cpu().double() - S_ref).abs().max().item() <= 60 * 2.0 ** -23 * S_ref.abs().max().item()
