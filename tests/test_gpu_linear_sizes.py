"""Products at the sizes where their kernels change: against 64-bit sums, with the bound that 32-bit sums of K terms have."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(out, a, w, scale, bias, before, round16=False):
    """|out - exact| <= (K + 8) 2^-24 sum |a||w| (any order of the sum), scaled, plus the epilogue's own roundings."""
    a64, w64 = a.double(), w.double()
    ref, mag = a64 @ w64.T, a64.abs() @ w64.abs().T
    bound = (a.shape[1] + 8) * 2.0 ** -24 * mag
    if scale is not None:
        ref, bound = ref * scale.double(), bound * scale.double().abs()
    if bias is not None:
        ref = ref + bias.double()
    if before is not None:
        ref = ref + before.double()
    bound = bound + 4 * 2.0 ** -24 * (ref.abs() + (0 if before is None else before.double().abs())) + (2.0 ** -8 * ref.abs() if round16 else 0) + 1e-30
    over = ((out.double() - ref).abs() - bound).max().item()
    assert over <= 0, f"{over} over the bound"


def _run(M, N, K, dtype, pad=4):
    from tinyllama_c_b200 import ops
    g = torch.Generator().manual_seed(M * 1000003 + N * 1009 + K)
    rnd = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    a, w = rnd(M, K).to(dtype).cuda(), (rnd(N, K) * 0.05).to(dtype).cuda()
    cs, cb, start = (1 + 0.3 * rnd(N)).cuda(), rnd(N).cuda(), rnd(M, N + pad).cuda()
    for accumulate, scale, bias, o_dt in ((False, None, None, torch.float32), (True, cs, None, torch.float32), (False, cs, cb, torch.bfloat16)):
        outs = []
        for _ in range(2):
            buf = start.to(o_dt, copy=True)
            ops.linear(a, w, buf[:, :N], scale, bias, accumulate)
            outs.append(buf)
        torch.cuda.synchronize()
        ops.check_errors()
        assert torch.equal(outs[0], outs[1]), "two runs of the same product differ"
        assert torch.equal(outs[0][:, N:], start.to(o_dt)[:, N:]), "wrote past N"
        _check(outs[0][:, :N], a, w, scale, bias, start[:, :N] if accumulate else None, o_dt == torch.bfloat16)


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8, 9, 16, 17, 64, 65, 131])
@pytest.mark.parametrize("N,K", [(1, 4), (67, 36), (130, 1028), (4740, 132), (2048, 68)])
def test_linear_of_32_bit_rows_in_pieces_of_16_bytes(M, N, K):
    """Few rows (one or two columns a warp, two or four from five rows on; more than eight rows in two launches), then
    tiles of 64 x 128 or of 64 x 64 with K in four parts: K shorter than a step, parts without a step, edges in M and N."""
    _run(M, N, K, torch.float32)
