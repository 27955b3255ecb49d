"""Mamba2 (selective state-space) mixer with a per-sequence conv window and state.

CodeClaper/tinyllama.c: in_proj of width d_ssm + conv_dim + n_heads laid out
z | x | B | C | dt (falcon_h1.c:342-343; cpu_op.c:849, 865, 925-929); causal depthwise
convolution + SiLU over x|B|C with a window of d_conv-1 raw samples (cpu_op.c:836-889);
dt = softplus(dt + dt_bias), dA = exp(dt * A) with A = -exp(A_log) (cpu_op.c:933-934,
806-808); S = S*dA + B*(x*dt), y = S.C + x*D (cpu_op.c:939-951); gate by silu(z) and
grouped RMSNorm (cpu_op.c:950-958); out_proj (falcon_h1.c:367-368).  The reference keeps
one window and one state per layer for its single sequence (falcon_h1.c:136-147); here
they are fixed-size per-sequence cache entries.  The five multipliers on the in_proj
slices, the in/out multipliers, the projection biases and norm-before-gate have no
counterpart in the reference.
"""
from __future__ import annotations

from typing import Callable, Dict, List, Optional, Sequence

import torch

from ... import ops
from ..base import ChunkRequest, LayerCache, Part, StateRequest, StepInfo, WeightSpec, register_mixer, scratch_buf, to_vec
from ..linear import StackedLinear


@register_mixer("mamba2")
class Mamba2Mixer(Part):
    single_token_launches = 3      # convolution, scan (or both in one), gated norm: what a one-token step launches in mix(), at most

    def __init__(self, hidden: int, d_ssm: int, n_heads: int, d_head: int, n_groups: int, d_state: int, d_conv: int,
                 prefix: str, eps: float, conv_bias: bool = True, proj_bias: bool = False, rms_norm: bool = True,
                 norm_before_gate: bool = False, slice_scales: Sequence[float] = (1.0,) * 5, in_scale: float = 1.0,
                 out_scale: float = 1.0, cache_key: str = "mamba", scan_chunk: int = ops.SSD_CHUNK,
                 names: Optional[Dict[str, str]] = None, norm_groups: Optional[int] = None):
        """names: tensor names after the prefix of in_proj, out_proj, conv, conv_bias, A_log, D, dt_bias, norm where they are
        not the in_proj.weight ... of the architecture's checkpoints (the convolution's weight is then [channels, taps]).
        norm_groups: into how many equal parts the gated norm cuts a row (default: n_groups)."""
        if n_heads * d_head != d_ssm or n_heads % n_groups or d_ssm % n_groups:
            raise ValueError("mamba2: n_heads*d_head must equal d_ssm and both be multiples of n_groups")
        if not (1 <= int(d_state) <= ops.MAX_STATE_SIZE):
            raise ValueError(f"mamba2: state size {d_state} is outside what the kernels are built for "
                             f"(1..{ops.MAX_STATE_SIZE})")
        if not (1 <= int(d_conv) <= ops.MAX_CONV_TAPS):
            raise ValueError(f"mamba2: {d_conv} convolution taps are outside what the kernels are built for "
                             f"(1..{ops.MAX_CONV_TAPS})")
        if int(n_heads) > ops.MAX_HEADS:
            raise ValueError(f"mamba2: {n_heads} heads exceed the kernels' limit of {ops.MAX_HEADS}")
        self.hidden, self.Di, self.Hs, self.P = int(hidden), int(d_ssm), int(n_heads), int(d_head)
        self.G, self.N, self.K = int(n_groups), int(d_state), int(d_conv)
        self.norm_groups = int(norm_groups) if norm_groups else self.G
        if self.norm_groups < 1 or int(d_ssm) % self.norm_groups:
            raise ValueError(f"mamba2: the gated norm cannot cut {d_ssm} values into {self.norm_groups} equal parts")
        self.own_names = names is not None
        self.nm = dict(in_proj="in_proj.weight", in_bias="in_proj.bias", out_proj="out_proj.weight", out_bias="out_proj.bias",
                       conv="conv1d.weight", conv_bias="conv1d.bias", A_log="A_log", D="D", dt_bias="dt_bias", norm="norm.weight")
        self.nm.update(names or {})
        self.Cd = self.Di + 2 * self.G * self.N                      # falcon_h1.c:124
        self.eps, self.rms_norm, self.norm_before_gate = float(eps), bool(rms_norm), bool(norm_before_gate)
        self.prefix, self.cache_key = prefix, cache_key
        # rows of a chunk of the parallel scan of prompts: the result does not depend on it (the state is
        # linear in its initial value); the tensor-core form takes chunks of ops.SSD_CHUNK rows only
        self.scan_chunk = int(scan_chunk)
        if self.scan_chunk < 1:
            raise ValueError(f"mamba2: a scan chunk of {scan_chunk} rows")
        self.conv_bias = bool(conv_bias)
        mz, mx, mb, mc, mdt = [float(v) for v in slice_scales]
        rows = [mz] * self.Di + [mx] * self.Di + [mb] * (self.G * self.N) + [mc] * (self.G * self.N) + [mdt] * self.Hs
        self.in_proj = StackedLinear(hidden)
        self.in_proj.add(prefix + self.nm["in_proj"], self.Di + self.Cd + self.Hs,
                         prefix + self.nm["in_bias"] if proj_bias else None, in_scale, rows)
        self.out_proj = StackedLinear(self.Di)
        self.out_proj.add(prefix + self.nm["out_proj"], hidden, prefix + self.nm["out_bias"] if proj_bias else None,
                          1.0, out_scale)
        self.conv_w = self.conv_b = self.A = self.D = self.dt_bias = self.norm_w = None
        self.dtype = None

    # ---- declarations ------------------------------------------------------------------
    def weight_specs(self) -> List[WeightSpec]:
        p = self.prefix
        specs = self.in_proj.weight_specs() + self.out_proj.weight_specs()
        nm = self.nm
        specs.append(WeightSpec(p + nm["conv"], (self.Cd, self.K) if self.own_names else (self.Cd, 1, self.K), "conv"))
        if self.conv_bias:
            specs.append(WeightSpec(p + nm["conv_bias"], (self.Cd,), "normal"))
        specs += [WeightSpec(p + nm["A_log"], (self.Hs,), "a_log"), WeightSpec(p + nm["D"], (self.Hs,), "d_skip"),
                  WeightSpec(p + nm["dt_bias"], (self.Hs,), "dt_bias")]
        if self.rms_norm:
            specs.append(WeightSpec(p + nm["norm"], (self.Di,), "ones"))
        return specs

    def cache_requests(self) -> list:
        return [StateRequest(self.cache_key + ".conv", (self.K - 1, self.Cd)),
                StateRequest(self.cache_key + ".ssm", (self.Hs, self.P, self.N))]

    # The row-by-row scan of a sequence takes 1 to 2 us a row and layer, more in a batch (a 128-token prompt of the
    # 1.5B sizes: 9.5 ms against 4.8 ms as one chunk in matrix form; 32 prompts of 128 tokens: 55 ms against 14.8;
    # 64 of 20 tokens: 20.4 against 11.8).  So the step's chunk table is asked for as soon as a sequence brings
    # more than CHUNKS_FROM_ROWS rows, and used when a sequence has more than 32 rows or the step has at least
    # 128: a few short sequences are quicker row by row (one prompt of 30 tokens: 4.0 ms against 4.5, the chunked
    # form's extra launches).
    CHUNKS_FROM_ROWS = 8
    CHUNKS_WORTH_ROWS, CHUNKS_WORTH_STEP = 32, 128

    # In 32 bits the chunks run row by row, one beside the other, and a chunk's rows are what a step of few chunks waits for: such steps
    # are cut into chunks of SHORT_CHUNK.  More chunks fill the GPU whatever their length, and every chunk costs a state of
    # scratch that three passes read and write: the blocks of a pass (16 head rows of a head of a chunk each) may be as many as
    # 22 chunks of 48 heads of 64 make, 28 where a sequence is cut by scan_chunk too, and sequences of no more than SHORT_ROWS gain
    # nothing.  Microseconds for the three passes with 256 columns, chunks of 128 and of 32 rows: 60 rows 64 / 54, 128 115 / 75,
    # 500 240 / 210, 800 (25 short chunks) 344 / 330, 900 (29) 370 / 376; sequences of 60 rows, 2 / 4 / 6 of them 101 / 145 / 187
    # and 79 / 136 / 192; of 100 rows, 4 / 6 / 9 (16 / 24 / 36 short chunks) 217 / 275 / 403 and 198 / 293 / 470; of 200, 3 / 4 (21 / 28)
    # 303 / 371 and 263 / 359; 20 of 33 (40) 399 / 511; 4 of 40 110 / 114.  (So the rounding of a sequence's rows in 32 bits depends
    # on what else a step brings, as CHUNKS_WORTH_STEP lets it in any type.)
    SHORT_CHUNK, SHORT_ROWS, SHORT_CHUNKS_STEP = 32, 48, 1024
    SHORT_BLOCKS, SHORT_BLOCKS_CUT = 22 * 48 * 4, 28 * 48 * 4

    def _chunks(self, step: StepInfo):
        """The table that cuts this step's sequences into chunks (None: row by row)."""
        if step.max_new <= self.CHUNKS_WORTH_ROWS and step.n_rows < self.CHUNKS_WORTH_STEP:
            return None
        short = step.chunks.get(self.SHORT_CHUNK) if self.dtype == torch.float32 and self.SHORT_CHUNK < self.scan_chunk else None
        if short is not None and step.max_new > self.SHORT_ROWS and step.n_rows <= self.SHORT_CHUNKS_STEP:
            blocks = short[1].numel() * self.Hs * ((self.P + 15) // 16)
            if blocks <= (self.SHORT_BLOCKS_CUT if step.max_new > self.scan_chunk else self.SHORT_BLOCKS):
                return short
        return step.chunks.get(self.scan_chunk)

    def step_requests(self) -> list:
        """(asked for again once the run's type is known)"""
        rows = [self.scan_chunk] + ([self.SHORT_CHUNK] if self.dtype == torch.float32 and self.SHORT_CHUNK < self.scan_chunk else [])
        return [ChunkRequest(n, min(n, self.CHUNKS_FROM_ROWS)) for n in rows]

    def bind(self, tensors: Dict[str, torch.Tensor], dtype, device) -> None:
        p = self.prefix
        self.dtype = dtype
        self.in_proj.bind(tensors, dtype, device)
        self.out_proj.bind(tensors, dtype, device)
        nm = self.nm
        self.conv_w = to_vec(tensors[p + nm["conv"]].reshape(self.Cd, self.K), device)
        self.conv_b = to_vec(tensors[p + nm["conv_bias"]], device) if self.conv_bias else None
        self.A = (-torch.exp(tensors[p + nm["A_log"]].to(torch.float32))).to(device).contiguous()    # cpu_op.c:806-808
        self.D = to_vec(tensors[p + nm["D"]], device)
        self.dt_bias = to_vec(tensors[p + nm["dt_bias"]], device)
        self.norm_w = to_vec(tensors[p + nm["norm"]], device) if self.rms_norm else None

    # ---- one step --------------------------------------------------------------------------
    def repeats(self):
        return frozenset(("prefix",))

    def input_projection(self) -> StackedLinear:
        return self.in_proj

    def forward(self, normed: torch.Tensor, step: StepInfo, cache: LayerCache, residual: torch.Tensor) -> None:
        proj = scratch_buf(f"mamba2.{self.cache_key}.proj", (step.n_rows, self.in_proj.out_features), torch.float32, normed.device)
        self.in_proj.forward(normed, proj)
        self.forward_projected(proj, step, cache, residual)

    def forward_projected(self, proj: torch.Tensor, step: StepInfo, cache: LayerCache, residual: torch.Tensor) -> None:
        """proj: this mixer's input projection, float32 [T, z|x|B|C|dt] (rows may be strided)."""
        self.output(self.mix(proj, step, cache), residual)

    def output_projection(self) -> StackedLinear:
        return self.out_proj

    mix_takes_scale = True         # mix() can multiply its result by a number on the way out
    mix_takes_join = True          # mix() calls `join` once, before its last kernel

    def mix(self, proj: torch.Tensor, step: StepInfo, cache: LayerCache, out: Optional[torch.Tensor] = None,
            out_scale: float = 1.0, join: Optional[Callable[[], None]] = None) -> torch.Tensor:
        """Everything between the input projection and the output projection: [T, d_ssm] times
        out_scale, written to `out` (rows may be strided) where one is given.  (A block that runs
        several output projections as one product moves a part of this one's multiplier here.)
        `join`, where given, is called once on the current stream before the last kernel: a block that runs
        other mixers on other streams waits for them there, where this stream waits for another one anyway
        (the scan's second stream), so that the kernel after this mixer follows its last one directly."""
        if not cache.writes:
            raise ValueError("mamba2: a recurrent mixer cannot run on another layer's cache without storing "
                             "(its window and state would advance twice in one step)")
        T, f32 = step.n_rows, torch.float32
        conv_state = cache.state[self.cache_key + ".conv"]
        ssm_state = cache.state[self.cache_key + ".ssm"]
        new = lambda tag, shape, dtype: scratch_buf(f"mamba2.{self.cache_key}.{tag}", shape, dtype, proj.device)   # (two mixers of a layer have two keys)
        y = new("y", (T, self.Di), f32)
        if step.max_new == 1 and T == step.n_seqs and ops.mamba_step_ok(proj, self.Di, self.Hs, self.P, self.N, self.G, self.K,
                                                                        self.conv_w, self.conv_b, conv_state, ssm_state):
            # one token per sequence: convolution and scan in one kernel
            ops.mamba_step(proj, self.Di, self.Di + self.Cd, self.conv_w, self.conv_b, self.dt_bias, self.A, self.D, conv_state,
                           ssm_state, step.slots, step.start_pos, y, self.Hs, self.P, self.N, self.G, self.dtype == torch.bfloat16)
            return self._gate(y, proj, None, out, out_scale, join, new,
                              (proj, self.Di, conv_state, step.slots, step.start_pos, self.Di, self.Cd - self.Di))
        # prompts cut into chunks of a bfloat16 run: the scan in matrix form, whose operands x|B|C the convolution
        # writes in bfloat16 at once; everything else scans 32-bit values
        chunks = self._chunks(step)
        matrix_form = chunks is not None and self.dtype == torch.bfloat16 and self.scan_chunk <= ops.SSD_CHUNK \
            and ops.ssd_ok(self.Hs, self.P, self.N, self.G)
        xbc = new("xbc", (T, self.Cd), torch.bfloat16 if matrix_form else f32)
        dt, dA = new("dt", (T, self.Hs), f32), new("dA", (T, self.Hs), f32)
        ops.mamba_conv(proj, self.Di, self.Di + self.Cd, self.conv_w, self.conv_b, self.dt_bias, self.A, conv_state,
                       step.cu_seqlens, step.row_seq, step.slots, step.start_pos, xbc, dt, dA,
                       step.max_new == 1, self.dtype == torch.bfloat16,
                       len(step.host_start) == step.n_seqs and not any(step.host_start))
        # in matrix form the outputs may come as two summands, the one that needs no state computed beside the walk
        # over the chunks; the gated norm adds them
        y_part = new("y_part", (T, self.Di), f32) if matrix_form else None
        in_two = ops.ssm_scan(xbc, dt, dA, self.D, ssm_state, step.cu_seqlens, step.slots, step.start_pos, y, self.Hs,
                              self.P, self.N, self.G, chunks, self.A if matrix_form else None, y_part)
        return self._gate(y, proj, y_part if in_two else None, out, out_scale, join, new)

    def _gate(self, y: torch.Tensor, proj: torch.Tensor, y_part: Optional[torch.Tensor], out: Optional[torch.Tensor], out_scale: float,
              join: Optional[Callable[[], None]], new: Callable, window=None) -> torch.Tensor:
        """The mixer's last kernel: the gate and the grouped norm of y (+ y_part); after mamba_step it also advances the
        windows of `window`."""
        gated = out if out is not None else new("gated", (y.shape[0], self.Di), self.dtype)
        if join is not None:
            join()
        more = {} if window is None else {"window": window}
        ops.gated_rmsnorm(y, proj[:, :self.Di], self.norm_w, self.eps, self.norm_groups, self.norm_before_gate, gated,
                          out_scale, y_part, **more)
        return gated

    def output(self, gated: torch.Tensor, residual: torch.Tensor) -> None:
        """Adds the output projection of `gated` into the residual stream."""
        self.out_proj.forward(gated, residual, accumulate=True)
