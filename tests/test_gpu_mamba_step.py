"""One-token steps of the Mamba2 mixer in one kernel: the same bits as the convolution and the scan as two kernels."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bf16_run", [False, True])
@pytest.mark.parametrize("Hs,P,N,G,K,bias", [(4, 16, 68, 1, 4, True), (2, 20, 128, 2, 3, False), (6, 4, 132, 3, 2, True), (3, 64, 256, 1, 4, True),
                                             (8, 36, 72, 4, 4, False), (120, 36, 72, 4, 4, False), (64, 64, 256, 1, 4, True),
                                             (416, 36, 72, 4, 4, False), (416, 64, 128, 1, 3, True), (820, 4, 68, 2, 2, True),
                                             (280, 68, 132, 4, 4, True), (416, 64, 256, 1, 3, False), (210, 100, 136, 3, 2, True)])
def test_step_kernel_against_convolution_and_scan(Hs, P, N, G, K, bias, bf16_run):
    """State columns that fill a warp's loads or not, rows of a head that end inside a block (of 16 rows; in the last
    six sets, 4,096 blocks and more, of 32), several groups, sequences at position 0 (zero window, zero state) beside ones
    that continue, slots in any order; y, the states and, after the norm that follows, all windows.  In 32 bits the
    recurrence in 64 bits too."""
    from tinyllama_c_b200 import ops
    g = torch.Generator().manual_seed(Hs * 1009 + N)
    B, Di = 5, Hs * P
    Cd = Di + 2 * G * N
    rnd = lambda *s: torch.randn(*s, generator=g).cuda()  # noqa: E731
    width = (Di + Cd + Hs + 11) // 4 * 4
    proj = rnd(B, width)
    w, cb = rnd(Cd, K), rnd(Cd) if bias else None
    dt_bias, A, D, norm_w = rnd(Hs), -rnd(Hs).abs() - 0.1, rnd(Hs), rnd(Di)
    conv0, state0 = rnd(7, K - 1, Cd), rnd(7, Hs, P, N)
    slots = torch.tensor([3, 0, 6, 2, 5], dtype=torch.int32).cuda()
    start = torch.tensor([9, 0, 130, 1, 0], dtype=torch.int32).cuda()
    ar = torch.arange(B + 1, dtype=torch.int32).cuda()
    z, eps = proj[:, :Di], 1e-5
    got = []
    for fused in (False, True):
        conv, state, y = conv0.clone(), state0.clone(), torch.full((B, Di), 7.0, device="cuda")
        out = torch.empty(B, Di, device="cuda", dtype=torch.bfloat16 if bf16_run else torch.float32)
        if fused:
            assert ops.mamba_step_ok(proj, Di, Hs, P, N, G, K)
            ops.mamba_step(proj, Di, Di + Cd, w, cb, dt_bias, A, D, conv, state, slots, start, y, Hs, P, N, G, bf16_run)
            ops.gated_rmsnorm(y, z, norm_w, eps, G, False, out, 0.5, window=(proj, Di, conv, slots, start, Di, Cd - Di))
        else:
            xbc, dt, dA = torch.empty(B, Cd, device="cuda"), torch.empty(B, Hs, device="cuda"), torch.empty(B, Hs, device="cuda")
            ops.mamba_conv(proj, Di, Di + Cd, w, cb, dt_bias, A, conv, ar, ar[:B].contiguous(), slots, start, xbc, dt, dA, True, bf16_run)
            ops.ssm_scan(xbc, dt, dA, D, state, ar, slots, start, y, Hs, P, N, G)
            ops.gated_rmsnorm(y, z, norm_w, eps, G, False, out, 0.5)
        torch.cuda.synchronize()
        ops.check_errors()
        got.append((y, state, conv, out))
    for a, b, name in zip(got[0], got[1], ("y", "states", "windows", "gated output")):
        assert torch.equal(a, b), name
    if bf16_run:
        return
    # the convolution of the last K - 1 stored rows and the new one, the time step, one step of the recurrence, with bounds on
    # the magnitudes that the roundings of a convolution, a SiLU of slope at most 1.1 and a sum of N terms are relative to
    live, at = start > 0, slots.long()
    ulp = 2.0 ** -24
    taps = torch.cat([conv0[at].double() * live[:, None, None], proj[:, None, Di:Di + Cd].double()], 1)      # [B, K, Cd]
    u, mag = (taps * w.double().T).sum(1), (taps.abs() * w.double().abs().T).sum(1)
    if bias:
        u, mag = u + cb.double(), mag + cb.double().abs()
    v = torch.nn.functional.silu(u)
    x, Bm, Cm = v[:, :Di].view(B, Hs, P), v[:, Di:Di + G * N], v[:, Di + G * N:]
    xm, bm, cm = (1.1 * mag[:, :Di]).view(B, Hs, P), 1.1 * mag[:, Di:Di + G * N], 1.1 * mag[:, Di + G * N:]
    by_head = lambda t: t.reshape(B, G, N).repeat_interleave(Hs // G, 1)[:, :, None]  # noqa: E731
    dt = torch.nn.functional.softplus(proj[:, Di + Cd:Di + Cd + Hs].double() + dt_bias.double())[:, :, None, None]
    dA = torch.exp(dt * A.double()[:, None, None])
    S0 = state0[at].double() * live[:, None, None, None] * dA
    S = S0 + x[..., None] * dt * by_head(Bm)
    size = S0.abs() + xm[..., None] * dt * by_head(bm)
    y = (S * by_head(Cm)).sum(-1) + x * D.double()[:, None]
    y_size = (size * by_head(cm)).sum(-1) + xm * D.double().abs()[:, None]
    # (the decay's exponent, of up to 4 |dt A| units, and a dozen products and functions of a few units each)
    steps = 64 + 4 * float((dt * A.double()[:, None, None]).abs().max())
    assert ((got[1][1][at].double() - S).abs() <= steps * ulp * size + 1e-30).all(), "states against 64 bits"
    assert ((got[1][0].view(B, Hs, P).double() - y).abs() <= (N + steps) * ulp * y_size + 1e-30).all(), "y against 64 bits"


def test_step_whose_waits_run_out_leaves_whole_states():
    """With a limit of one clock cycle a block whose state has not landed at once gives up: every block of rows keeps the
    state that it had or gets the new one, never a part of it, and check_errors raises if one was kept."""
    from tinyllama_c_b200 import ops
    Hs, P, N, G, K, B = 64, 64, 256, 1, 4, 5
    Di, Cd = Hs * P, Hs * P + 2 * G * N
    g = torch.Generator().manual_seed(41)
    rnd = lambda *s: torch.randn(*s, generator=g).cuda()  # noqa: E731
    proj, w, dt_bias, A, D = rnd(B, Di + Cd + Hs), rnd(Cd, K), rnd(Hs), -rnd(Hs).abs() - 0.1, rnd(Hs)
    conv0, state0 = rnd(B, K - 1, Cd), rnd(B, Hs, P, N)
    slots = torch.arange(B, dtype=torch.int32).cuda()
    start = torch.full((B,), 9, dtype=torch.int32).cuda()

    def step(state):
        conv, y = conv0.clone(), torch.empty(B, Di, device="cuda")
        ops.mamba_step(proj, Di, Di + Cd, w, None, dt_bias, A, D, conv, state, slots, start, y, Hs, P, N, G)
        torch.cuda.synchronize()
        return state.view(-1, 16, N)

    old, new = state0.view(-1, 16, N), step(state0.clone())
    ops.check_errors()
    try:
        ops.wait_limit_cycles(1)
        for _ in range(5):
            got = step(state0.clone())
            kept = (got == old).flatten(1).all(1)
            assert ((got == new).flatten(1).all(1) | kept).all(), "a state in parts"
            if kept.any():
                with pytest.raises(ops.KernelError, match="41"):
                    ops.check_errors()
            else:
                ops.check_errors()
    finally:
        ops.wait_limit_cycles(0)


def test_a_mixer_whose_convolution_weights_lie_at_any_address():
    """Weights bound as slices of one flat buffer, 4 bytes past a 16-byte boundary: a prompt, then one-token steps, give the
    bits of a mixer with weights of their own (the two kernels take the steps)."""
    from tinyllama_c_b200 import ops
    from tinyllama_c_b200.cache import Cache
    from tinyllama_c_b200.engine.step import StepEntry, pack
    from tinyllama_c_b200.parts.mixers.mamba2 import Mamba2Mixer
    g = torch.Generator().manual_seed(5)
    got = []
    for off in (None, 1):
        mixer = Mamba2Mixer(64, 64, 4, 16, 1, 128, 4, "", 1e-5)
        tensors = {spec.name: torch.randn(spec.shape, generator=g).cuda() * 0.2 for spec in mixer.weight_specs()}
        if off is not None:
            tensors = first                        # the same values
            for name in ("conv1d.weight", "conv1d.bias"):
                flat = torch.empty(tensors[name].numel() + off, device="cuda")[off:]
                tensors[name] = flat.view(tensors[name].shape).copy_(tensors[name])
        first = dict(tensors)
        mixer.bind(tensors, torch.float32, torch.device("cuda"))
        cache = Cache({0: mixer.cache_requests()}, 64, 3, torch.float32, "cuda")
        assert (mixer.conv_w.data_ptr() % 16 == 0) == (off is None)
        slots, outs = [cache.acquire() for _ in range(2)], []
        for lens in ((5, 3), (1, 1), (1, 1)):
            entries = [StepEntry(s, [0] * n) for s, n in zip(slots, lens)]
            step, _, _ = pack(entries, [cache.reserve(s, n) for s, n in zip(slots, lens)], 1, torch.device("cuda"))
            x = torch.randn(sum(lens), 64, generator=torch.Generator().manual_seed(sum(lens))).cuda()
            out = torch.zeros(sum(lens), 64, device="cuda")
            mixer.forward(x, step, cache.layer_view(0), out)
            outs.append(out)
            for s, n in zip(slots, lens):
                cache.commit(s, n)
        torch.cuda.synchronize()
        ops.check_errors()
        got.append(outs + [grp.data for grp in cache.state_groups])
    for a, b in zip(*got):
        assert torch.equal(a, b)
