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
    tiles of 64 x 64 with K in four parts: K shorter than a step, parts without a step, edges in M and N."""
    _run(M, N, K, torch.float32)


@pytest.mark.parametrize("M,N,K", [(449, 4740, 132), (1211, 2050, 36), (577, 4096, 4), (2368, 1028, 68)])
def test_linear_of_32_bit_rows_in_tiles_of_64_by_128(M, N, K):
    """As many tiles as two an SM (296 on 148 SMs): one K-step or several, the last one shorter, edges in M and N or none."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert -(-M // 64) * -(-N // 128) >= 2 * min(sms, 148)
    _run(M, N, K, torch.float32)


@pytest.mark.parametrize("M,N,K", [(1, 16424, 72), (4, 16500, 2056), (5, 16384, 4096), (8, 18950, 136), (9, 16390, 520), (16, 16400, 264), (17, 16385, 200), (32, 20000, 72)])
def test_linear_of_a_vocabulary_with_few_rows(M, N, K):
    """Outputs of 128 tiles of 128 weight rows and more: 16 or 32 activation rows on the narrow side, last tiles past N."""
    _run(M, N, K, torch.bfloat16)


@pytest.mark.parametrize("split", [1, 2, 4, 8])
@pytest.mark.parametrize("M,N,K", [(9, 300, 520), (16, 1000, 1096), (13, 128, 136), (24, 2064, 328)])
def test_linear_with_16_or_32_rows_on_the_narrow_side_and_a_fixed_split(M, N, K, split):
    """The sums of 1 to 8 blocks: fewer K-steps than blocks, a share of the rows that some blocks do not have; the gated form."""
    from tinyllama_c_b200 import ops
    ops.linear_few_rows(True, split)
    try:
        _run(M, N, K, torch.bfloat16, pad=3)
        if N % 16 == 0:
            g = torch.Generator().manual_seed(N + M)
            a, w = torch.randn(M, K, generator=g).bfloat16().cuda(), (torch.randn(N, K, generator=g) * 0.05).bfloat16().cuda()
            out = torch.empty(M, N // 2, device="cuda")
            ops.linear_swiglu(a, w, out)
            gu = (a.double() @ w.double().T).view(M, N // 16, 2, 8)
            ref = (torch.nn.functional.silu(gu[:, :, 0]) * gu[:, :, 1]).reshape(M, N // 2)
            # sums of K terms (relative 2^-13 at the most here) through a product and a SiLU of slope at most 1.1
            assert (out.double() - ref).abs().max().item() <= 3 * (K + 8) * 2.0 ** -24 * 8 * (1 + gu.abs().max().item()) ** 2
            ops.check_errors()
    finally:
        ops.linear_few_rows(True, 0)


_WITHOUT_SET_UP = """
import ctypes, sys, torch
from tinyllama_c_b200 import ops
from tinyllama_c_b200.csrc import build
lib = build.load()
lib.tlc_linear.restype, lib.tlc_linear.argtypes = ops._SIGNATURES["tlc_linear"]
lib.tlc_last_error.restype = ctypes.c_char_p
a, w, out = torch.randn(64, 64).cuda(), torch.randn(64, 64).cuda(), torch.empty(64, 64, device="cuda")
rc = lib.tlc_linear(a.data_ptr(), 0, 64, w.data_ptr(), 0, 64, out.data_ptr(), 0, 64, None, None, 0, 64, 64, 64, 33, None)
torch.cuda.synchronize()
assert rc == 0, lib.tlc_last_error()
assert (out.double() - a.double() @ w.double().T).abs().max().item() < 72 * 2.0 ** -24 * 64 * 16
"""


def test_32_bit_products_without_the_set_up_of_the_tensor_core_kernels():
    """A process that has not called tlc_linear_init: the 32-bit products need none (tiles with shared K-steps take more
    shared memory than a kernel has unasked)."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    run = subprocess.run([sys.executable, "-c", _WITHOUT_SET_UP], cwd=root, capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]


@pytest.mark.parametrize("M", [1, 4, 8, 9, 16, 17, 100])
def test_32_bit_products_of_what_the_kernel_before_them_writes(M):
    """w comes from the kernel in front of the product (here a norm's rows): the product reads it after that kernel's end."""
    from tinyllama_c_b200 import ops
    g = torch.Generator().manual_seed(M)
    N, K = 4100, 1028
    a, x, gain = torch.randn(M, K, generator=g).cuda(), torch.randn(N, K, generator=g).cuda(), torch.ones(K, device="cuda")
    w, out = torch.full((N, K), float("nan"), device="cuda"), torch.empty(M, N, device="cuda")
    torch.cuda.synchronize()
    ops.rmsnorm(x, gain, 1e-5, w)
    ops.linear(a, w, out)
    torch.cuda.synchronize()
    _check(out, a, w, None, None, None)


@pytest.mark.parametrize("M", [1, 5, 8])
@pytest.mark.parametrize("N,K", [(4752, 2048), (8240, 2048), (8244, 1032), (9472, 2040), (4768, 1160)])
def test_products_of_up_to_8_rows_with_two_tiles_a_block(M, N, K):
    """297, 515 and 516 tiles (an odd number, a part of one), 592; K of a whole round and of parts of one: the bits of a tile a
    block, and the oracle's values."""
    from tinyllama_c_b200 import ops
    g = torch.Generator().manual_seed(N + K + M)
    a, w = torch.randn(M, K, generator=g).bfloat16().cuda(), torch.randn(N, K, generator=g).bfloat16().cuda()
    scale, bias, before = torch.randn(N, generator=g).cuda(), torch.randn(N, generator=g).cuda(), torch.randn(M, N, generator=g).cuda()
    got = []
    for two in (True, False):
        ops.linear_skinny_two(two)
        try:
            out = [before.clone(), before.clone(), torch.full((M, N), float("nan"), device="cuda").bfloat16()]
            ops.linear(a, w, out[0], scale, bias, True)
            ops.linear(a, w, out[1])
            ops.linear(a, w, out[2], scale)
            if N % 16 == 0:
                out.append(torch.full((M, N // 2), float("nan"), device="cuda").bfloat16())
                ops.linear_swiglu(a, w, out[3], scale, bias)
            torch.cuda.synchronize()
        finally:
            ops.linear_skinny_two(True)
        got.append(out)
    assert all(torch.equal(x, y) for x, y in zip(*got))
    _check(got[0][1], a.float(), w.float(), None, None, None)


@pytest.mark.parametrize("M", [17, 24, 31, 32])
@pytest.mark.parametrize("N,K", [(2384, 4096), (2572, 5384), (3072, 12288), (4092, 4104)])
def test_products_of_17_to_32_rows_shared_among_clusters_of_four(M, N, K):
    """149, 161, 192 and 256 tiles of 16 columns (an odd number, a part of one), whole rounds of K and parts of one: the bits of the
    kernel with a tile a block, and the oracle's values."""
    from tinyllama_c_b200 import ops
    g = torch.Generator().manual_seed(N + K + M)
    a, w = torch.randn(M, K, generator=g).bfloat16().cuda(), torch.randn(N, K, generator=g).bfloat16().cuda()
    scale, bias, before = torch.randn(N, generator=g).cuda(), torch.randn(N, generator=g).cuda(), torch.randn(M, N + 4, generator=g).cuda()
    got = []
    for ring in (True, False):
        ops.linear_skinny_ring(ring)
        try:
            out = [before.clone() for _ in range(3)] + [torch.full((M, N), float("nan"), device="cuda").bfloat16()]
            ops.linear(a, w, out[0][:, :N], scale, bias, True)
            ops.linear(a, w, out[1][:, :N], scale, None, True)
            ops.linear(a, w, out[2][:, :N])
            ops.linear(a, w, out[3], None, bias)
            torch.cuda.synchronize()
        finally:
            ops.linear_skinny_ring(True)
        got.append(out)
    assert all(torch.equal(x, y) for x, y in zip(*got))
    assert torch.equal(got[0][0][:, N:], before[:, N:])
    _check(got[0][2][:, :N], a.float(), w.float(), None, None, None)


@pytest.mark.parametrize("rows,split", [(32, 1), (32, 2), (32, 8), (64, 0), (64, 1), (64, 4), (64, 8)])
@pytest.mark.parametrize("M,N,K", [(17, 132, 36), (33, 516, 260), (70, 1030, 132), (129, 257, 1028)])
def test_32_bit_tiles_with_their_k_steps_shared(M, N, K, rows, split):
    """Every tile with one block, some and eight (fewer K-steps than blocks, too), edges in part in both directions; sums added into
    the output, overwritten, in 16 bits, into rows that are not on 16-byte boundaries."""
    from tinyllama_c_b200 import ops
    g = torch.Generator().manual_seed(M + N + K)
    a, w = torch.randn(M, K, generator=g).cuda(), torch.randn(N, K, generator=g).cuda()
    scale, bias, before = torch.randn(N, generator=g).cuda(), torch.randn(N, generator=g).cuda(), torch.randn(M + 1, N + 3, generator=g).cuda()
    ops.linear_f32_tiles(rows, split)
    try:
        out, once, half = before.clone(), torch.full((M, N), float("nan"), device="cuda"), torch.full((M, N), float("nan"), device="cuda").bfloat16()
        ops.linear(a, w, out[:M, :N], scale, bias, True)
        ops.linear(a, w, once)
        ops.linear(a, w, half, scale)
        torch.cuda.synchronize()
    finally:
        ops.linear_f32_tiles(0)
    _check(out[:M, :N], a, w, scale, bias, before[:M, :N])
    _check(once, a, w, None, None, None)
    _check(half, a, w, scale, None, None, True)
    assert torch.equal(out[M], before[M]) and torch.equal(out[:, N:], before[:, N:])


@pytest.mark.parametrize("M,N,K", [(17, 60, 4), (33, 132, 36), (70, 1030, 132), (129, 257, 1028)])
def test_32_bit_tiles_with_k_in_four_parts(M, N, K):
    """Fewer K-steps than parts, parts of unequal length, edges in part; sums added into the output, overwritten, in 16 bits."""
    from tinyllama_c_b200 import ops
    g = torch.Generator().manual_seed(M + N + K)
    a, w = torch.randn(M, K, generator=g).cuda(), torch.randn(N, K, generator=g).cuda()
    scale, bias, before = torch.randn(N, generator=g).cuda(), torch.randn(N, generator=g).cuda(), torch.randn(M + 1, N + 3, generator=g).cuda()
    ops.linear_f32_tiles(64, -4)
    try:
        out, once, half = before.clone(), torch.full((M, N), float("nan"), device="cuda"), torch.full((M, N), float("nan"), device="cuda").bfloat16()
        ops.linear(a, w, out[:M, :N], scale, bias, True)
        ops.linear(a, w, once)
        ops.linear(a, w, half, scale)
        torch.cuda.synchronize()
    finally:
        ops.linear_f32_tiles(0)
    _check(out[:M, :N], a, w, scale, bias, before[:M, :N])
    _check(once, a, w, None, None, None)
    _check(half, a, w, scale, None, None, True)
    assert torch.equal(out[M], before[M]) and torch.equal(out[:, N:], before[:, N:])
