"""The scan of prompts in matrix form: first chunks of new sequences in a kernel of their own, the same bits as in the walk."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Hs,P,N,G", [(4, 64, 256, 1), (6, 32, 128, 2), (2, 96, 256, 1), (4, 128, 128, 4)])
@pytest.mark.parametrize("apart", [False, True])
def test_first_chunks_give_the_bits_of_the_walk(Hs, P, N, G, apart):
    """Sequences that start in the step and ones that continue; one row, less than a chunk, exactly one, one row more and
    several chunks; heads of 32, 64, 96 and 128 rows; the outputs in one sum and in two; twice."""
    from tinyllama_c_b200 import ops
    from tinyllama_c_b200.engine.step import chunk_table
    g = torch.Generator().manual_seed(Hs * 1000 + N + P)
    lens, begins = [1, 50, 128, 129, 300, 128, 40, 257], [0, 0, 0, 0, 0, 70, 9, 0]
    T, B, Di = sum(lens), len(lens), Hs * P
    Cd = Di + 2 * G * N
    xbc = (torch.randn(T, Cd, generator=g) * 0.5).bfloat16().cuda()
    dt = torch.rand(T, Hs, generator=g).cuda() * 0.1
    A, D = -torch.rand(Hs, generator=g).cuda() * 4, torch.randn(Hs, generator=g).cuda()
    state0 = torch.randn(B + 2, Hs, P, N, generator=g).cuda()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32).cuda()  # noqa: E731
    cu, slots, start = i32([sum(lens[:b]) for b in range(B + 1)]), i32([3, 0, 9, 2, 5, 1, 7, 4]), i32(begins)
    chunks = tuple(i32(t) for t in chunk_table(lens, ops.SSD_CHUNK, 0))
    got = []
    try:
        for mode in (1, 2, 2):
            ops.ssd_first_chunks(mode)
            y, part, state = torch.full((T, Di), 5.0, device="cuda"), torch.empty(T, Di, device="cuda"), state0.clone()
            two = ops.ssm_scan(xbc, dt, torch.exp(dt * A), D, state, cu, slots, start, y, Hs, P, N, G, chunks, A, part if apart else None)
            torch.cuda.synchronize()
            ops.check_errors()
            assert two == apart
            got.append((y + part if apart else y, state))
    finally:
        ops.ssd_first_chunks(0)
    for other in got[1:]:
        assert torch.equal(got[0][1], other[1]), "states"
        assert torch.equal(got[0][0], other[0]), "outputs"
