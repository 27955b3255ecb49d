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


@pytest.mark.parametrize("N,P", [(68, 4), (128, 20), (132, 64), (256, 12)])
@pytest.mark.parametrize("lens,chunk", [((1,), 0), ((4, 5, 1), 0), ((23, 8), 0), ((1, 70, 33), 32)])
def test_rows_in_16_byte_pieces_give_the_general_kernels_bits(N, P, lens, chunk):
    """The same outputs and states, row by row; in chunks the general kernel multiplies a chunk's decays in another order."""
    from tinyllama_c_b200 import ops
    g = torch.Generator().manual_seed(sum(lens) + N)
    Hs, G = 6, 2
    T, B, Di = sum(lens), len(lens), Hs * P
    xbc, dt, dA = torch.randn(T, Di + 2 * G * N, generator=g).cuda(), torch.rand(T, Hs, generator=g).cuda(), torch.rand(T, Hs, generator=g).cuda()
    D, state = torch.randn(Hs, generator=g).cuda(), torch.randn(B, Hs, P, N, generator=g).cuda()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    cu = [sum(lens[:b]) for b in range(B + 1)]
    chunks = None
    if chunk:
        firsts = [[c for c in range(cu[b], cu[b + 1], chunk)] for b in range(B)]
        chunks = (i32(sum(firsts, []) + [T]), i32([b for b in range(B) for _ in firsts[b]]),
                  i32([sum(len(f) for f in firsts[:b]) for b in range(B + 1)]))
    got = []
    for own in (True, False):
        ops.ssm_scan_rows(own)
        try:
            y, st = torch.full((T, Di), float("nan"), device="cuda"), state.clone()
            ops.ssm_scan(xbc, dt, dA, D, st, i32(cu), i32(range(B)), i32([3 if b % 2 else 0 for b in range(B)]), y, Hs, P, N, G, chunks)
            torch.cuda.synchronize()
        finally:
            ops.ssm_scan_rows(True)
        got.append((y, st))
    for a, b in zip(*got):
        assert torch.equal(a, b) if not chunk else (a - b).abs().max() <= 70 * 2.0 ** -23 * b.abs().max()


@pytest.mark.parametrize("B,Hs,P,N", [(3, 4, 8, 72), (64, 8, 64, 72), (65, 8, 64, 128), (65, 8, 64, 132)])
def test_one_row_a_sequence_gives_the_same_bits_by_either_kernel(B, Hs, P, N):
    """12, 2,048 and 2,080 blocks of up to 128 columns, and more columns; steps of one row each, and the same number of rows otherwise
    divided (two of one sequence, none of another)."""
    from tinyllama_c_b200 import ops
    g = torch.Generator().manual_seed(B + N)
    Di = Hs * P
    xbc, dt, dA = torch.randn(B, Di + 2 * N, generator=g).cuda(), torch.rand(B, Hs, generator=g).cuda(), torch.rand(B, Hs, generator=g).cuda()
    D, state = torch.randn(Hs, generator=g).cuda(), torch.randn(B, Hs, P, N, generator=g).cuda()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    for cu in (list(range(B + 1)), [0, 2, 2] + list(range(3, B + 1))):
        got = []
        for own in (True, False):
            ops.ssm_scan_rows(own)
            try:
                y, st = torch.full((B, Di), float("nan"), device="cuda"), state.clone()
                ops.ssm_scan(xbc, dt, dA, D, st, i32(cu), i32(range(B)), i32([3 if b % 2 else 0 for b in range(B)]), y, Hs, P, N, 1, None)
                torch.cuda.synchronize()
            finally:
                ops.ssm_scan_rows(True)
            got.append((y, st))
        assert all(torch.equal(a, b) for a, b in zip(*got))
