// Mamba2 mixer kernels: causal depthwise convolution with its per-sequence window,
// the time-step transform, and the selective state scan with its per-sequence state.
//
// CodeClaper/tinyllama.c states the math on the CPU only: convolution over the last K
// raw samples, tap K-1 on the newest, bias, SiLU, then the window shifts and stores the
// raw sample (cpu_op.c:836-889); dt = softplus(dt + bias), dA = exp(dt*A),
// S = S*dA + B*(x*dt), y = sum_n S*C + x*D (cpu_op.c:924-951).  Here a step carries
// several sequences of unequal length packed back to back; a sequence that starts at
// position 0 starts from a zero window and a zero state, any other continues from its
// slot.  Convolution, dt, the decay and the state are 32-bit.
#include "common.cuh"
#include "mbarrier.cuh"

#define CONV_MAX_TAPS 16

// ---- convolution + SiLU over packed rows, and softplus / decay of dt ---------------------
// In a bfloat16 run (QUICK) x|B|C are operands of the scan's matrix products: they are rounded to bfloat16
// here, whatever type they are stored in, so that a row's values do not depend on which scan reads them (the
// matrix form of long prompts, the row-by-row scan of short ones and of single-token steps).
template <bool BF16_RUN> __device__ __forceinline__ float as_operand(float v) {
  return BF16_RUN ? __bfloat162float(__float2bfloat16_rn(v)) : v;
}

// grid (ceil(T / 8), ceil(Cd/256)): a thread owns one channel of 8 consecutive rows.  It reads the
// raw samples of those rows and of the K-1 rows before them once (all loads issued together), and
// takes a tap from the sequence's stored window only where the row is among the first K-1 of a
// sequence that continues from a slot.  Also writes dt and dA of the rows (first blocks along y).
// With write_state (every sequence of the step starts at position 0, so that no block reads a stored window)
// the block that holds a sequence's last row also leaves the sequence's new window: its last K-1 raw samples,
// zeros before its first row.  A step with a sequence that continues leaves that to mamba_conv_state_kernel,
// which runs when every reader of the old windows has finished.
#define CONV_ROWS 8
template <typename T, typename TO, int K, bool QUICK>
__global__ void __launch_bounds__(256)
mamba_conv_rows_kernel(const T* __restrict__ proj, int ld, int xbc_off, int dt_off,
                  const float* __restrict__ w, const float* __restrict__ bias,
                  const float* __restrict__ dt_bias, const float* __restrict__ A,
                  const float* __restrict__ conv_state, const int* __restrict__ cu_seqlens,
                  const int* __restrict__ row_seq, const int* __restrict__ slots,
                  const int* __restrict__ start_pos, TO* __restrict__ xbc_out,
                  float* __restrict__ dt_out, float* __restrict__ dA_out, int n_rows, int Cd, int Hs,
                  float* state_out, int write_state) {   // state_out is conv_state, written only when nothing reads it
  tlc_pdl(proj, conv_state, xbc_out, dt_out, dA_out, state_out);
  __shared__ int s_i[CONV_ROWS], s_has[CONV_ROWS], s_slot[CONV_ROWS], s_last[CONV_ROWS], s_plain, s_any_last;
  const int t0 = blockIdx.x * CONV_ROWS;
  if (threadIdx.x == 0) { s_plain = 1; s_any_last = 0; }
  __syncthreads();
  if (threadIdx.x < CONV_ROWS) {
    const int t = t0 + threadIdx.x;
    int i = 0, has = 0, slot = 0, last = 0;
    if (t < n_rows) {
      const int b = row_seq[t];
      i = t - cu_seqlens[b];                          // index of the row inside its sequence's new tokens
      has = start_pos[b] > 0;
      slot = slots[b];
      last = write_state && t == cu_seqlens[b + 1] - 1;
    }
    s_i[threadIdx.x] = i;
    s_has[threadIdx.x] = has;
    s_slot[threadIdx.x] = slot;
    s_last[threadIdx.x] = last;
    if (last) s_any_last = 1;
    // plain: all of the block's rows exist and every tap of every row reads a row of this step
    if (t >= n_rows || i < K - 1) s_plain = 0;
  }
  __syncthreads();
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  // The common block is kept free of the window's address arithmetic and of per-row branches: the kernel is bound by
  // its instruction count, not by memory.  Row t0 + r reads raw rows r .. r + K - 1 (raw[0] is row t0 - (K-1)).
  if (c < Cd && s_plain) {
    const T* src = proj + (size_t)(t0 - (K - 1)) * ld + xbc_off + c;
    float raw[CONV_ROWS + K - 1], wk[K];
#pragma unroll
    for (int q = 0; q < CONV_ROWS + K - 1; q++) raw[q] = to_f32(src[(size_t)q * ld]);
#pragma unroll
    for (int k = 0; k < K; k++) wk[k] = w[(size_t)c * K + k];
    const float bv = bias ? bias[c] : 0.f;
    TO* dst = xbc_out + (size_t)t0 * Cd + c;
#pragma unroll
    for (int r = 0; r < CONV_ROWS; r++) {
      float sum = 0.f;
#pragma unroll
      for (int k = 0; k < K; k++) sum = fmaf(raw[r + k], wk[k], sum);
      dst[(size_t)r * Cd] = from_f32<TO>(as_operand<QUICK>(silu_of<QUICK>(sum + bv)));
    }
  } else if (c < Cd) {
    // raw[q] is the sample of packed row t0 - (K-1) + q; rows before the step's first are never used
    float raw[CONV_ROWS + K - 1], wk[K];
#pragma unroll
    for (int q = 0; q < CONV_ROWS + K - 1; q++) {
      const int t = t0 - (K - 1) + q;
      raw[q] = (t >= 0 && t < n_rows) ? to_f32(proj[(size_t)t * ld + xbc_off + c]) : 0.f;
    }
#pragma unroll
    for (int k = 0; k < K; k++) wk[k] = w[(size_t)c * K + k];
    const float bv = bias ? bias[c] : 0.f;
#pragma unroll
    for (int r = 0; r < CONV_ROWS; r++) {
      const int t = t0 + r;
      if (t >= n_rows) break;
      const int i = s_i[r];
      float sum = 0.f;
      if (i >= K - 1) {
        // every tap reads a row of this step: row t - (K-1-k) is raw row r + k (the common case, kept free of the
        // window's address arithmetic: the kernel is bound by its instruction count, not by memory)
#pragma unroll
        for (int k = 0; k < K; k++) sum = fmaf(raw[r + k], wk[k], sum);
      } else {
#pragma unroll
        for (int k = 0; k < K; k++) {
          const int j = i - (K - 1 - k);              // new-token index that tap k reads
          float x;
          if (j >= 0) x = raw[r + k];
          else x = s_has[r] ? conv_state[((size_t)s_slot[r] * (K - 1) + (K - 1 + j)) * Cd + c] : 0.f;
          sum = fmaf(x, wk[k], sum);
        }
      }
      xbc_out[(size_t)t * Cd + c] = from_f32<TO>(as_operand<QUICK>(silu_of<QUICK>(sum + bv)));
    }
  }
  if (s_any_last && c < Cd) {
    for (int r = 0; r < CONV_ROWS; r++) {
      if (!s_last[r]) continue;
      const int t = t0 + r, n = s_i[r] + 1;           // the sequence's last row and its number of rows
      float* st = state_out + (size_t)s_slot[r] * (K - 1) * Cd + c;
#pragma unroll
      for (int j = 0; j < K - 1; j++)                 // window row j is the sequence's row n - (K-1) + j
        st[(size_t)j * Cd] = j >= K - 1 - n ? to_f32(proj[(size_t)(t - (K - 2) + j) * ld + xbc_off + c]) : 0.f;
    }
  }
  if (c < Hs) {
    const float db = dt_bias[c], Ac = A[c];
#pragma unroll
    for (int r = 0; r < CONV_ROWS; r++) {
      const int t = t0 + r;
      if (t >= n_rows) break;
      const float dtv = softplus_f(to_f32(proj[(size_t)t * ld + dt_off + c]) + db);
      dt_out[(size_t)t * Hs + c] = dtv;
      dA_out[(size_t)t * Hs + c] = expf(dtv * Ac);
    }
  }
}

// Any number of taps: grid (T, ceil(Cd/256)), a thread per (row, channel).
template <typename T, typename TO>
__global__ void mamba_conv_kernel(const T* __restrict__ proj, int ld, int xbc_off, int dt_off,
                                  const float* __restrict__ w, const float* __restrict__ bias,
                                  const float* __restrict__ dt_bias, const float* __restrict__ A,
                                  const float* __restrict__ conv_state, const int* __restrict__ cu_seqlens,
                                  const int* __restrict__ row_seq, const int* __restrict__ slots,
                                  const int* __restrict__ start_pos, TO* __restrict__ xbc_out,
                                  float* __restrict__ dt_out, float* __restrict__ dA_out, int Cd, int K, int Hs,
                                  int bf16_run) {
  tlc_pdl(proj, conv_state, xbc_out, dt_out, dA_out);
  const int t = blockIdx.x;
  const int b = row_seq[t];
  const int i = t - cu_seqlens[b];                  // index of this row inside its sequence's new tokens
  const bool has_state = start_pos[b] > 0;
  const float* st = conv_state + (size_t)slots[b] * (K - 1) * Cd;
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  if (c < Cd) {
    float sum = 0.f;
    for (int k = 0; k < K; k++) {
      const int j = i - (K - 1 - k);                // new-token index that tap k reads
      float x;
      if (j >= 0) x = to_f32(proj[(size_t)(t - (K - 1 - k)) * ld + xbc_off + c]);
      else x = has_state ? st[(size_t)(K - 1 + j) * Cd + c] : 0.f;
      sum = fmaf(x, w[(size_t)c * K + k], sum);
    }
    if (bias) sum += bias[c];
    const float v = silu_f(sum);
    xbc_out[(size_t)t * Cd + c] = from_f32<TO>(bf16_run ? as_operand<true>(v) : v);
  }
  if (c < Hs) {
    const float dtv = softplus_f(to_f32(proj[(size_t)t * ld + dt_off + c]) + dt_bias[c]);
    dt_out[(size_t)t * Hs + c] = dtv;
    dA_out[(size_t)t * Hs + c] = expf(dtv * A[c]);
  }
}

// New window of each sequence: its last K-1 raw samples (old window rows where the step
// brought fewer).  One thread owns one (sequence, channel), reads all it needs, then writes.
template <typename T>
__global__ void mamba_conv_state_kernel(const T* __restrict__ proj, int ld, int xbc_off, float* __restrict__ conv_state,
                                        const int* __restrict__ cu_seqlens, const int* __restrict__ slots,
                                        const int* __restrict__ start_pos, int Cd, int K) {
  tlc_pdl(proj, conv_state);
  const int b = blockIdx.x;
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  if (c >= Cd) return;
  const int t0 = cu_seqlens[b], n = cu_seqlens[b + 1] - t0;
  if (n == 0) return;
  const bool has_state = start_pos[b] > 0;
  float* st = conv_state + (size_t)slots[b] * (K - 1) * Cd;
  float v[CONV_MAX_TAPS];
#pragma unroll
  for (int j = 0; j < CONV_MAX_TAPS; j++) {
    if (j < K - 1) {
      const int idx = n - (K - 1) + j;              // new-token index that lands in window row j
      if (idx >= 0) v[j] = to_f32(proj[(size_t)(t0 + idx) * ld + xbc_off + c]);
      else v[j] = has_state ? st[(size_t)(K - 1 + idx) * Cd + c] : 0.f;
    }
  }
#pragma unroll
  for (int j = 0; j < CONV_MAX_TAPS; j++)
    if (j < K - 1) st[(size_t)j * Cd + c] = v[j];
}

// One-token steps: every sequence brings exactly one row, so a thread owns one (sequence, channel):
// it reads the window, convolves, and writes the shifted window back -- one kernel instead of two.
// KT: the number of taps when it is 2, 3 or 4 (the window then takes KT - 1 registers instead of the limit's 16),
// else 0 and K is read at run time.
template <typename T, int KT>
__global__ void mamba_conv_decode_kernel(const T* __restrict__ proj, int ld, int xbc_off, int dt_off,
                                         const float* __restrict__ w, const float* __restrict__ bias,
                                         const float* __restrict__ dt_bias, const float* __restrict__ A,
                                         float* __restrict__ conv_state, const int* __restrict__ slots,
                                         const int* __restrict__ start_pos, float* __restrict__ xbc_out,
                                         float* __restrict__ dt_out, float* __restrict__ dA_out, int Cd, int K, int Hs,
                                         int bf16_run) {
  constexpr int TAPS = KT > 0 ? KT - 1 : CONV_MAX_TAPS;     // window rows held in registers
  if (KT > 0) K = KT;
  // The window was stored by the step before and the weights never change: both are fetched before the
  // wait on the previous kernel; only the row's projection is read after it.
  asm volatile("griddepcontrol.launch_dependents;");
  const int b = blockIdx.x;                          // row b belongs to sequence b
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  const bool has_state = start_pos[b] > 0;
  float* st = conv_state + (size_t)slots[b] * (K - 1) * Cd;
  float prev[TAPS], wk[TAPS + 1];
  float bv = 0.f, db = 0.f, Ac = 0.f;
  if (c < Cd) {
#pragma unroll
    for (int k = 0; k < TAPS; k++) {
      prev[k] = (k < K - 1 && has_state) ? st[(size_t)k * Cd + c] : 0.f;
      wk[k] = k < K ? w[(size_t)c * K + k] : 0.f;
    }
    wk[TAPS] = TAPS < K ? w[(size_t)c * K + TAPS] : 0.f;
    if (bias) bv = bias[c];
  }
  if (c < Hs) { db = dt_bias[c]; Ac = A[c]; }
  tlc_wait(proj, xbc_out, dt_out, dA_out);
  if (c < Cd) {
    const float cur = to_f32(proj[(size_t)b * ld + xbc_off + c]);
    float sum = bv;
#pragma unroll
    for (int k = 0; k < TAPS; k++)
      if (k < K - 1) sum = fmaf(prev[k], wk[k], sum);
    float wl = 0.f;
#pragma unroll
    for (int k = 0; k <= TAPS; k++) if (k == K - 1) wl = wk[k];
    sum = fmaf(cur, wl, sum);
    const float v = silu_f(sum);
    xbc_out[(size_t)b * Cd + c] = bf16_run ? as_operand<true>(v) : v;
#pragma unroll
    for (int k = 0; k < TAPS; k++) {
      if (k < K - 2) st[(size_t)k * Cd + c] = prev[k + 1];
      else if (k == K - 2) st[(size_t)k * Cd + c] = cur;
    }
  }
  if (c < Hs) {
    const float dtv = softplus_f(to_f32(proj[(size_t)b * ld + dt_off + c]) + db);
    dt_out[(size_t)b * Hs + c] = dtv;
    dA_out[(size_t)b * Hs + c] = expf(dtv * Ac);
  }
}

#define TLC_CONV_ROWS_Q(KT, QK)                                                                                        \
  tlc_launch(mamba_conv_rows_kernel<TT, TO, KT, QK>, dim3(grid8), dim3(256), 0, stream, (const TT*)proj, ld, xbc_off,  \
             dt_off, w, bias, dt_bias, A, conv_state, cu_seqlens, row_seq, slots, start_pos, (TO*)xbc_out, dt_out,     \
             dA_out, T, Cd, Hs, conv_state, fused_state)
#define TLC_CONV_ROWS(KT) do { if (quick) TLC_CONV_ROWS_Q(KT, true); else TLC_CONV_ROWS_Q(KT, false); } while (0)
// xbc_dtype: the element type of xbc_out [T, Cd].  Single-token steps and the 32-bit scans take float; the scan
// of prompts in matrix form takes its operands in bfloat16 and gets them in that type at once.
extern "C" int tlc_mamba_conv(const void* proj, int dtype, int ld, int xbc_off, int dt_off, const float* w,
                              const float* bias, const float* dt_bias, const float* A, float* conv_state,
                              const int* cu_seqlens, const int* row_seq, const int* slots, const int* start_pos,
                              void* xbc_out, int xbc_dtype, float* dt_out, float* dA_out, int T, int B, int Cd, int K,
                              int Hs, int single_rows, int quick, int all_fresh, cudaStream_t stream) {
  if (T == 0) return 0;
  // every sequence starts at position 0: nothing reads a stored window, and the rows' kernel writes the new ones
  const int fused_state = all_fresh && K >= 2 && K <= 4;
  TLC_REQUIRE(K >= 1 && K - 1 <= CONV_MAX_TAPS, "mamba_conv: %d taps exceed the kernel's limit of %d", K, CONV_MAX_TAPS + 1);
  TLC_REQUIRE(Hs <= Cd, "mamba_conv: more heads (%d) than conv channels (%d)", Hs, Cd);
  dim3 grid(T, (Cd + 255) / 256);
  dim3 grid8((T + CONV_ROWS - 1) / CONV_ROWS, (Cd + 255) / 256);
  dim3 grid2(B, (Cd + 255) / 256);
  if (single_rows && T == B) {
    TLC_REQUIRE(xbc_dtype == TLC_F32, "mamba_conv: single-token steps write 32-bit x|B|C");
#define TLC_CONV_DECODE(KT)                                                                                          \
  tlc_launch(mamba_conv_decode_kernel<TT, KT>, dim3(grid2), dim3(256), 0, stream, (const TT*)proj, ld, xbc_off, dt_off, w,  \
             bias, dt_bias, A, conv_state, slots, start_pos, (float*)xbc_out, dt_out, dA_out, Cd, K, Hs, quick)
    TLC_DISPATCH_DTYPE(dtype, TT, {
      if (K == 4) TLC_CONV_DECODE(4);
      else if (K == 3) TLC_CONV_DECODE(3);
      else if (K == 2) TLC_CONV_DECODE(2);
      else TLC_CONV_DECODE(0);
    });
#undef TLC_CONV_DECODE
    TLC_CHECK_LAUNCH("mamba_conv(decode)");
    return 0;
  }
  TLC_DISPATCH_DTYPE(dtype, TT, TLC_DISPATCH_DTYPE(xbc_dtype, TO, {
    if (K == 4) TLC_CONV_ROWS(4);
    else if (K == 3) TLC_CONV_ROWS(3);
    else if (K == 2) TLC_CONV_ROWS(2);
    else
      tlc_launch(mamba_conv_kernel<TT, TO>, dim3(grid), dim3(256), 0, stream, (const TT*)proj, ld, xbc_off, dt_off, w, bias,
                 dt_bias, A, conv_state, cu_seqlens, row_seq, slots, start_pos, (TO*)xbc_out, dt_out, dA_out, Cd, K, Hs, quick);
    if (K > 1 && !fused_state)
      tlc_launch(mamba_conv_state_kernel<TT>, dim3(grid2), dim3(256), 0, stream, (const TT*)proj, ld, xbc_off, conv_state,
                 cu_seqlens, slots, start_pos, Cd, K);
  }));
  TLC_CHECK_LAUNCH("mamba_conv");
  return 0;
}

// ---- selective scan ---------------------------------------------------------------------------
// The scan runs over *segments* of consecutive rows.  In the plain mode a segment is a whole
// sequence: it starts from its slot's state (zero at position 0) and leaves its final state there.
// Long prompts are cut into chunks that run in parallel, in three passes:
//   1. every chunk from a zero state, keeping only its final state  S_c           (mode 1)
//   2. per sequence, in chunk order: S_in[c] = S_in[c-1] * decay[c-1] + S_[c-1]    (state pass)
//   3. every chunk again from its true incoming state S_in[c], now writing y      (mode 3)
// which is the same recurrence, because the state is linear in its initial value.
//
// grid (segment, Hs, ceil(P / (4*RP))), 128 threads: each warp owns RP rows p of one head's state
// [P, N], each lane the columns lane, lane+32, ... (NPL of them) in registers.  Rows run in
// order; the inputs of SCAN_TT rows are staged in shared memory at a time.
#define SCAN_TT 4
#define SCAN_PLAIN 0
#define SCAN_CHUNK_STATE 1
#define SCAN_CHUNK_OUT 3
__device__ __forceinline__ void scan_copy16(float* dst, const float* src, bool on) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(on ? 16 : 0) : "memory");   // (0: zeros)
}
__device__ __forceinline__ void scan_copy4(float* dst, const float* src, bool on = true) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(on ? 4 : 0) : "memory");
}
// Blocks an SM: the registers that the state needs leave room for these, and what the compiler takes beyond them costs more than it
// gives (seven for every size: 64 sequences of one row, 48 heads of 64, 32 columns 26.7 us and not 24.1, 64 columns 31.5 and
// 28.2; a prompt of 1,500 rows in chunks, 128 columns 659 and 523, 130 columns 1215 and 878).
template <int NPL, int RP, bool VEC>
__global__ void __launch_bounds__(128, NPL == 1 ? 11 : NPL == 2 ? 9 : NPL == 4 ? 8 : VEC ? 7 : 6)
ssm_scan_kernel(const float* __restrict__ xbc, const float* __restrict__ dt, const float* __restrict__ dA,
                const float* __restrict__ Dskip, float* __restrict__ state, float* __restrict__ chunk_state,
                const int* __restrict__ seg_start, const int* __restrict__ seg_seq,
                const int* __restrict__ seq_seg_start, const int* __restrict__ slots,
                const int* __restrict__ start_pos, float* __restrict__ y, float* __restrict__ chunk_decay, int mode,
                int Hs, int P, int N, int G, int Cd) {
  // In the plain mode the state this block starts from was written by an earlier step, not by
  // the kernel before this one: it is fetched before the wait on that kernel (see tlc_pdl).
  asm volatile("griddepcontrol.launch_dependents;");
  if (mode != SCAN_PLAIN) tlc_wait(xbc, dt, dA, state, chunk_state, y, chunk_decay);
  extern __shared__ float sm[];
  const int seg = blockIdx.x, h = blockIdx.y;
  const int b = seg_seq ? seg_seq[seg] : seg;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rows_per_block = 4 * RP;
  const int p_blk = blockIdx.z * rows_per_block;
  const int p_base = p_blk + warp * RP;
  const int Di = Hs * P;
  const int g = h / (Hs / G);
  const int t0 = seg_start[seg], n_tok = seg_start[seg + 1] - t0;
  if (n_tok == 0) return;
  float* S_slot = state + (((size_t)slots[b] * Hs + h) * P) * N;
  float* S_chunk = chunk_state ? chunk_state + (((size_t)seg * Hs + h) * P) * N : nullptr;
  const float* S_init = nullptr;
  if (mode == SCAN_PLAIN) { if (start_pos[b] > 0) S_init = S_slot; }
  else if (mode == SCAN_CHUNK_OUT) S_init = S_chunk;
  float* S_final = nullptr;
  if (mode == SCAN_PLAIN) S_final = S_slot;
  else if (mode == SCAN_CHUNK_STATE) S_final = S_chunk;
  else if (seg + 1 == seq_seg_start[b + 1]) S_final = S_slot;        // the sequence's last chunk
  const bool want_y = mode != SCAN_CHUNK_STATE;
  // A lane owns the columns lane, lane + 32, ... of its rows, or (VEC: more than 64 columns, a multiple of 4, in states that
  // start on 16-byte boundaries) four consecutive columns 4 lane + 128 jj, which it loads and stores 16 bytes at a time.
  auto col = [&](int j) { return VEC ? 4 * lane + 128 * (j >> 2) + (j & 3) : lane + 32 * j; };
  float s[RP][NPL];
#pragma unroll
  for (int r = 0; r < RP; r++) {
    const int p = p_base + r;
    if (VEC) {
#pragma unroll
      for (int jj = 0; jj < NPL / 4; jj++) {
        const int n = 4 * lane + 128 * jj;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (S_init && p < P && n < N) v = *reinterpret_cast<const float4*>(S_init + (size_t)p * N + n);
        s[r][4 * jj] = v.x; s[r][4 * jj + 1] = v.y; s[r][4 * jj + 2] = v.z; s[r][4 * jj + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int j = 0; j < NPL; j++) {
        const int n = lane + 32 * j;
        s[r][j] = (S_init && p < P && n < N) ? S_init[(size_t)p * N + n] : 0.f;
      }
    }
  }
  if (mode == SCAN_PLAIN) tlc_wait(xbc, dt, dA, y);
  // Shared staging: per row  B[N] | C[N] | x[rows_per_block] | dt | dA, the rows SCAN_TT at a time, in two buffers: the
  // copies of a batch, in pieces of 16 bytes where the rows are laid out in them, are on their way while the batch
  // before it is worked on, so that a row costs its arithmetic and not a trip to memory.  Eight rows at a time in one
  // buffer, each row's loads in a loop of their own, before: 23 rows of the 1.5B sizes (48 heads of 64, 256 columns) 56.7 us,
  // so 46.8; eight sequences of 10 rows 53.0 and 38.5, one of 32 77.3 and 64.1, a single row 5.3 and 4.7; rows that are not in
  // pieces of 16 bytes (130 columns) 34.0 and 29.0, 36.4 and 34.6.  A prompt of 23 tokens is bound by the host and takes what
  // it took.
  const int per_tok = 2 * N + rows_per_block + 4;            // (a multiple of 4 where N is one)
  const float Dh = Dskip[h];
  const bool quads = N % 4 == 0 && P % 4 == 0 && Cd % 4 == 0 && ((uintptr_t)xbc & 15) == 0;
  const int nq = N >> 2, row_q = 2 * nq + RP;                // pieces of a row: B, C, x (4 RP values)
  auto fetch = [&](int tt0, float* buf) {
    const int nt = min(SCAN_TT, n_tok - tt0);
    if (quads) {
      for (int idx = threadIdx.x; idx < nt * row_q; idx += 128) {
        const int k = idx / row_q, q = idx - k * row_q;
        const float* row = xbc + (size_t)(t0 + tt0 + k) * Cd;
        const int p = p_blk + 4 * (q - 2 * nq);
        const float* src = row;
        bool on = true;
        if (q < nq) src = row + Di + (size_t)g * N + 4 * q;
        else if (q < 2 * nq) { src = row + Di + (size_t)G * N + (size_t)g * N + 4 * (q - nq); on = want_y; }
        else { on = p < P; if (on) src = row + (size_t)h * P + p; }
        scan_copy16(buf + (size_t)k * per_tok + 4 * q, src, on);
      }
    } else {
#pragma unroll 1
      for (int k = 0; k < nt; k++) {
        const float* row = xbc + (size_t)(t0 + tt0 + k) * Cd;
        const float* Bg = row + Di + (size_t)g * N;
        float* dst = buf + (size_t)k * per_tok;
#pragma unroll 1
        for (int e = threadIdx.x; e < N; e += 128) {
          scan_copy4(dst + e, Bg + e);
          scan_copy4(dst + N + e, Bg + (size_t)G * N + e, want_y);
        }
        if (threadIdx.x < rows_per_block) {
          const bool on = p_blk + threadIdx.x < P;
          scan_copy4(dst + 2 * N + threadIdx.x, on ? row + (size_t)h * P + p_blk + threadIdx.x : row, on);
        }
      }
    }
    if (threadIdx.x < 2 * SCAN_TT && (threadIdx.x >> 1) < nt)
      scan_copy4(buf + (size_t)(threadIdx.x >> 1) * per_tok + 2 * N + rows_per_block + (threadIdx.x & 1),
                 ((threadIdx.x & 1) ? dA : dt) + (size_t)(t0 + tt0 + (threadIdx.x >> 1)) * Hs + h);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(0, sm);
  for (int tt0 = 0, turn = 0; tt0 < n_tok; tt0 += SCAN_TT, turn ^= 1) {
    const int nt = min(SCAN_TT, n_tok - tt0);
    float* smb = sm + (size_t)turn * SCAN_TT * per_tok;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                         // this batch is here, and every warp is done with the one before it
    if (tt0 + SCAN_TT < n_tok) fetch(tt0 + SCAN_TT, sm + (size_t)(turn ^ 1) * SCAN_TT * per_tok);
    for (int k = 0; k < nt; k++) {
      const float* tk = smb + (size_t)k * per_tok;
      const float dtv = tk[2 * N + rows_per_block], dAv = tk[2 * N + rows_per_block + 1];
      float Bv[NPL], Cv[NPL];
#pragma unroll
      for (int j = 0; j < NPL; j++) {
        const int n = col(j);
        Bv[j] = n < N ? tk[n] : 0.f;
        Cv[j] = n < N ? tk[N + n] : 0.f;
      }
      if (want_y) {
#pragma unroll
        for (int r = 0; r < RP; r++) {
          const float xv = tk[2 * N + warp * RP + r];
          const float xdt = xv * dtv;
          float sum = 0.f;
#pragma unroll
          for (int j = 0; j < NPL; j++) {
            const float sv = fmaf(s[r][j], dAv, Bv[j] * xdt);
            s[r][j] = sv;
            sum = fmaf(sv, Cv[j], sum);
          }
          sum = warp_sum(sum);
          const int p = p_base + r;
          if (lane == 0 && p < P) y[(size_t)(t0 + tt0 + k) * Di + (size_t)h * P + p] = sum + xv * Dh;
        }
      } else {
#pragma unroll
        for (int r = 0; r < RP; r++) {
          const float xdt = tk[2 * N + warp * RP + r] * dtv;
#pragma unroll
          for (int j = 0; j < NPL; j++) s[r][j] = fmaf(s[r][j], dAv, Bv[j] * xdt);
        }
      }
    }
  }
  if (mode == SCAN_CHUNK_STATE && blockIdx.z == 0 && threadIdx.x == 0) {
    float d = 1.f;                         // decay of the whole chunk: the product of its rows' decays
    for (int k = 0; k < n_tok; k++) d *= dA[(size_t)(t0 + k) * Hs + h];
    chunk_decay[(size_t)seg * Hs + h] = d;
  }
  if (S_final) {
#pragma unroll
    for (int r = 0; r < RP; r++) {
      const int p = p_base + r;
      if (VEC) {
#pragma unroll
        for (int jj = 0; jj < NPL / 4; jj++) {
          const int n = 4 * lane + 128 * jj;
          if (p < P && n < N)
            *reinterpret_cast<float4*>(S_final + (size_t)p * N + n) =
                make_float4(s[r][4 * jj], s[r][4 * jj + 1], s[r][4 * jj + 2], s[r][4 * jj + 3]);
        }
      } else {
#pragma unroll
        for (int j = 0; j < NPL; j++) {
          const int n = lane + 32 * j;
          if (p < P && n < N) S_final[(size_t)p * N + n] = s[r][j];
        }
      }
    }
  }
}

// The same for states of more than 64 columns where everything lies in pieces of 16 bytes (columns and head rows multiples of 4,
// xbc, its rows and the states on 16-byte boundaries): row by row the state's values and the order of every sum are those of the
// kernel above, a row costs less.  (In chunks the decays of a chunk's rows are multiplied in another order: a lane's rows first,
// then the lanes.)  What a row cost there: four sums over a warp of five shuffles each, one after the other, B and C
// read value by value with a stride of four (bank conflicts), and a division and an address from scratch for every piece that
// is copied.  Here the sums of SCAN_TT rows x RP head rows, which every lane holds a share of, go through the same tree together:
// at each of the first steps a lane hands half of its values to its partner and keeps the other half (16 values: 16 shuffles
// and not 80), which leaves every pair of lanes with one value to store; B and C are read 16 bytes at a time; a thread copies the
// same pieces of every row and only moves its pointers on.  48 heads of 64, 256 columns, before and now, microseconds: one row 4.4
// and 3.7, 23 rows 30.3 and 13.0, eight sequences of 10 rows 40.0 and 23.4; in chunks (three passes) 310 rows of 128 353 and 188,
// of 32 212 and 140.  (Two head rows a warp, twice the warps: 23 rows 14.8, eight of 10 29.1.)
template <int NPL>
__global__ void __launch_bounds__(128, NPL == 4 ? 6 : 5)
ssm_scan_rows_kernel(const float* __restrict__ xbc, const float* __restrict__ dt, const float* __restrict__ dA,
                     const float* __restrict__ Dskip, float* __restrict__ state, float* __restrict__ chunk_state,
                     const int* __restrict__ seg_start, const int* __restrict__ seg_seq,
                     const int* __restrict__ seq_seg_start, const int* __restrict__ slots,
                     const int* __restrict__ start_pos, float* __restrict__ y, float* __restrict__ chunk_decay, int mode,
                     int Hs, int P, int N, int G, int Cd) {
  asm volatile("griddepcontrol.launch_dependents;");
  if (mode != SCAN_PLAIN) tlc_wait(xbc, dt, dA, state, chunk_state, y, chunk_decay);
  static_assert(NPL % 4 == 0, "four columns a lane at a time");
  constexpr int RP = 4, TT = SCAN_TT, PB = 4 * RP, V = TT * RP, NQ = NPL / 4;
  extern __shared__ __align__(16) float sm[];
  const int seg = blockIdx.x, h = blockIdx.y;
  const int b = seg_seq ? seg_seq[seg] : seg;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int p_blk = blockIdx.z * PB, p_base = p_blk + warp * RP;
  const int Di = Hs * P, g = h / (Hs / G);
  const int t0 = seg_start[seg], n_tok = seg_start[seg + 1] - t0;
  if (n_tok == 0) return;
  float* S_slot = state + (((size_t)slots[b] * Hs + h) * P) * N;
  float* S_chunk = chunk_state ? chunk_state + (((size_t)seg * Hs + h) * P) * N : nullptr;
  const float* S_init = mode == SCAN_PLAIN ? (start_pos[b] > 0 ? S_slot : nullptr) : mode == SCAN_CHUNK_OUT ? S_chunk : nullptr;
  float* S_final = mode == SCAN_PLAIN ? S_slot : mode == SCAN_CHUNK_STATE ? S_chunk : seg + 1 == seq_seg_start[b + 1] ? S_slot : nullptr;
  const bool want_y = mode != SCAN_CHUNK_STATE;
  float4 s[RP][NQ];                                          // columns 4 lane + 128 jj of the warp's head rows
#pragma unroll
  for (int r = 0; r < RP; r++)
#pragma unroll
    for (int jj = 0; jj < NQ; jj++) {
      const int n = 4 * lane + 128 * jj;
      s[r][jj] = S_init && p_base + r < P && n < N ? *reinterpret_cast<const float4*>(S_init + (size_t)(p_base + r) * N + n)
                                                    : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  if (mode == SCAN_PLAIN) tlc_wait(xbc, dt, dA, y);
  // a row in shared memory: B[N] | C[N] | x[PB] | dt | dA
  const int per_tok = 2 * N + PB + 4, nq = N >> 2, row_q = 2 * nq + RP;
  const float Dh = Dskip[h];
  // this thread's pieces of a row: where they come from (of the segment's first row), and whether they are copied at all
  const float* src[2];
  bool on[2];
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const int q = tid + 128 * i, p = p_blk + 4 * (q - 2 * nq);
    const float* row = xbc + (size_t)t0 * Cd;
    src[i] = row;
    on[i] = true;
    if (q < nq) src[i] = row + Di + (size_t)g * N + 4 * q;
    else if (q < 2 * nq) { src[i] = row + Di + (size_t)G * N + (size_t)g * N + 4 * (q - nq); on[i] = want_y; }
    else { on[i] = p < P; if (on[i]) src[i] = row + (size_t)h * P + p; }
  }
  const float* src_dt = ((tid & 1) ? dA : dt) + (size_t)(t0 + (tid >> 1)) * Hs + h;      // (threads 0 .. 2 TT - 1)
  auto fetch = [&](int tt0, float* buf) {
    const int nt = min(TT, n_tok - tt0);
#pragma unroll
    for (int k = 0; k < TT; k++) {
      if (k < nt) {
#pragma unroll
        for (int i = 0; i < 2; i++)
          if (tid + 128 * i < row_q) {
            scan_copy16(buf + k * per_tok + 4 * (tid + 128 * i), src[i], on[i]);
            src[i] += Cd;
          }
      }
    }
    if (tid < 2 * TT && (tid >> 1) < nt) scan_copy4(buf + (tid >> 1) * per_tok + 2 * N + PB + (tid & 1), src_dt + (size_t)tt0 * Hs);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(0, sm);
#pragma unroll 1
  for (int tt0 = 0, turn = 0; tt0 < n_tok; tt0 += TT, turn ^= 1) {
    const int nt = min(TT, n_tok - tt0);
    const float* smb = sm + turn * TT * per_tok;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                         // this batch is here, and every warp is done with the one before it
    if (tt0 + TT < n_tok) fetch(tt0 + TT, sm + (turn ^ 1) * TT * per_tok);
    float v[V];
#pragma unroll
    for (int k = 0; k < TT; k++) {
      if (k < nt) {
        const float* tk = smb + k * per_tok;
        const float2 dd = *reinterpret_cast<const float2*>(tk + 2 * N + PB);
        float x[RP];
#pragma unroll
        for (int r = 0; r < RP; r += 2) {
          const float2 u = *reinterpret_cast<const float2*>(tk + 2 * N + warp * RP + r);
          x[r] = u.x * dd.x;
          x[r + 1] = u.y * dd.x;
        }
#pragma unroll
        for (int r = 0; r < RP; r++) v[k * RP + r] = 0.f;
#pragma unroll
        for (int jj = 0; jj < NQ; jj++) {
          const int n = 4 * lane + 128 * jj;
          const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
          const float4 B = n < N ? *reinterpret_cast<const float4*>(tk + n) : z;
          const float4 C = want_y && n < N ? *reinterpret_cast<const float4*>(tk + N + n) : z;
#pragma unroll
          for (int r = 0; r < RP; r++) {
            float4& u = s[r][jj];
            float& a = v[k * RP + r];
            u.x = fmaf(u.x, dd.y, B.x * x[r]); a = fmaf(u.x, C.x, a);
            u.y = fmaf(u.y, dd.y, B.y * x[r]); a = fmaf(u.y, C.y, a);
            u.z = fmaf(u.z, dd.y, B.z * x[r]); a = fmaf(u.z, C.z, a);
            u.w = fmaf(u.w, dd.y, B.w * x[r]); a = fmaf(u.w, C.w, a);
          }
        }
      } else {
#pragma unroll
        for (int r = 0; r < RP; r++) v[k * RP + r] = 0.f;
      }
    }
    if (want_y) {
      // the tree of warp_sum for all values at once; bit by bit a lane keeps the half that its number names
#pragma unroll
      for (int o = 16, m = V / 2; o > 0; o >>= 1, m >>= 1) {
        if (m > 0) {
          const bool upper = lane & o;
#pragma unroll
          for (int i = 0; i < m; i++) {
            const float mine = upper ? v[i + m] : v[i], theirs = upper ? v[i] : v[i + m];
            v[i] = mine + __shfl_xor_sync(0xffffffffu, theirs, o);
          }
        } else {
          v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        }
      }
      constexpr int SPARE = 32 / V;                          // lanes that hold the same value
      const int idx = lane / SPARE, k = idx / RP, r = idx % RP, p = p_base + r;
      if (lane % SPARE == 0 && k < nt && p < P)
        y[(size_t)(t0 + tt0 + k) * Di + (size_t)h * P + p] = v[0] + smb[k * per_tok + 2 * N + warp * RP + r] * Dh;
    }
  }
  if (mode == SCAN_CHUNK_STATE && blockIdx.z == 0 && warp == 0) {
    float d = 1.f;                         // decay of the whole chunk: the product of its rows' decays
    for (int k = lane; k < n_tok; k += 32) d *= dA[(size_t)(t0 + k) * Hs + h];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) d *= __shfl_xor_sync(0xffffffffu, d, o);
    if (lane == 0) chunk_decay[(size_t)seg * Hs + h] = d;
  }
  if (S_final) {
#pragma unroll
    for (int r = 0; r < RP; r++)
#pragma unroll
      for (int jj = 0; jj < NQ; jj++) {
        const int n = 4 * lane + 128 * jj;
        if (p_base + r < P && n < N) *reinterpret_cast<float4*>(S_final + (size_t)(p_base + r) * N + n) = s[r][jj];
      }
  }
}
static int g_scan_rows = 1;                // test hook: 0 = the general kernel everywhere
extern "C" void tlc_ssm_scan_rows(int on) { g_scan_rows = on; }

// Pass 2: carries the state through a sequence's chunks.  chunk_state[c] holds the chunk's own
// contribution on entry and the state *before* the chunk on exit.  grid (B, Hs, blocks over P*N).
// With write_final the state after the last chunk goes to the sequence's slot.
__global__ void __launch_bounds__(256)
ssm_state_pass_kernel(const float* __restrict__ chunk_decay, float* __restrict__ state,
                      float* __restrict__ chunk_state, const int* __restrict__ seq_seg_start,
                      const int* __restrict__ slots, const int* __restrict__ start_pos, int Hs, int PN, int write_final) {
  tlc_pdl(chunk_decay, state, chunk_state);
  const int b = blockIdx.x, h = blockIdx.y;
  const int e = blockIdx.z * blockDim.x + threadIdx.x;
  const int c0 = seq_seg_start[b], c1 = seq_seg_start[b + 1];
  if (c1 - c0 <= 0 || e >= PN) return;
  float* slot = state + ((size_t)slots[b] * Hs + h) * PN + e;
  float s = start_pos[b] > 0 ? *slot : 0.f;
  constexpr int BATCH = 16;                // chunks whose values are fetched together
  for (int cb = c0; cb < c1; cb += BATCH) {
    float own[BATCH], decay[BATCH];
#pragma unroll
    for (int i = 0; i < BATCH; i++) {
      const int c = cb + i;
      own[i] = c < c1 ? chunk_state[((size_t)c * Hs + h) * PN + e] : 0.f;
      decay[i] = c < c1 ? chunk_decay[(size_t)c * Hs + h] : 1.f;
    }
#pragma unroll
    for (int i = 0; i < BATCH; i++) {
      const int c = cb + i;
      if (c < c1) {
        chunk_state[((size_t)c * Hs + h) * PN + e] = s;
        s = fmaf(s, decay[i], own[i]);
      }
    }
  }
  if (write_final) *slot = s;
}

// The same with four state elements a thread (16-byte loads and stores), for state sizes that are multiples of 4.
__global__ void __launch_bounds__(256)
ssm_state_pass_vec_kernel(const float* __restrict__ chunk_decay, float* __restrict__ state,
                          float* __restrict__ chunk_state, const int* __restrict__ seq_seg_start,
                          const int* __restrict__ slots, const int* __restrict__ start_pos, int Hs, int PN, int write_final) {
  tlc_pdl(chunk_decay, state, chunk_state);
  const int b = blockIdx.x, h = blockIdx.y;
  const int e = 4 * (blockIdx.z * blockDim.x + threadIdx.x);
  const int c0 = seq_seg_start[b], c1 = seq_seg_start[b + 1];
  if (c1 - c0 <= 0 || e >= PN) return;
  float4* slot = reinterpret_cast<float4*>(state + ((size_t)slots[b] * Hs + h) * PN + e);
  float4 s = start_pos[b] > 0 ? *slot : make_float4(0.f, 0.f, 0.f, 0.f);
  constexpr int BATCH = 16;                // chunks whose values are fetched together
  for (int cb = c0; cb < c1; cb += BATCH) {
    float4 own[BATCH];
    float decay[BATCH];
#pragma unroll
    for (int i = 0; i < BATCH; i++) {
      const int c = cb + i;
      own[i] = c < c1 ? *reinterpret_cast<const float4*>(chunk_state + ((size_t)c * Hs + h) * PN + e) : make_float4(0.f, 0.f, 0.f, 0.f);
      decay[i] = c < c1 ? chunk_decay[(size_t)c * Hs + h] : 1.f;
    }
#pragma unroll
    for (int i = 0; i < BATCH; i++) {
      const int c = cb + i;
      if (c < c1) {
        *reinterpret_cast<float4*>(chunk_state + ((size_t)c * Hs + h) * PN + e) = s;
        s = make_float4(fmaf(s.x, decay[i], own[i].x), fmaf(s.y, decay[i], own[i].y), fmaf(s.z, decay[i], own[i].z),
                        fmaf(s.w, decay[i], own[i].w));
      }
    }
  }
  if (write_final) *slot = s;
}

int tlc_ssm_state_pass_launch(const float* chunk_decay, float* state, float* chunk_state, const int* seq_seg_start,
                              const int* slots, const int* start_pos, int B, int Hs, int PN, int write_final,
                              cudaStream_t stream) {
  if (PN % 4 == 0 && ((uintptr_t)state % 16) == 0 && ((uintptr_t)chunk_state % 16) == 0) {
    dim3 grid(B, Hs, (PN / 4 + 255) / 256);
    tlc_launch(ssm_state_pass_vec_kernel, grid, dim3(256), 0, stream, chunk_decay, state, chunk_state, seq_seg_start, slots,
               start_pos, Hs, PN, write_final);
    TLC_CHECK_LAUNCH("ssm_state_pass");
    return 0;
  }
  dim3 grid(B, Hs, (PN + 255) / 256);
  tlc_launch(ssm_state_pass_kernel, grid, dim3(256), 0, stream, chunk_decay, state, chunk_state, seq_seg_start, slots,
             start_pos, Hs, PN, write_final);
  TLC_CHECK_LAUNCH("ssm_state_pass");
  return 0;
}

template <int NPL>
static int launch_scan(const float* xbc, const float* dt, const float* dA, const float* Dskip, float* state,
                       float* chunk_state, const int* seg_start, const int* seg_seq, const int* seq_seg_start,
                       const int* slots, const int* start_pos, float* y, float* chunk_decay, int mode, int n_seg, int Hs,
                       int P, int N, int G, int Cd, bool one_row, cudaStream_t stream) {
  constexpr int RP = 4;
  if constexpr (NPL % 4 == 0) {
    // A row a sequence, up to 128 columns and many blocks: states in and out are all there is, and the general kernel has eight blocks
    // an SM for that and not six.  Microseconds, by rows in 16-byte pieces and by the general kernel: 64 sequences of 24 heads of 64
    // and 128 columns (6,144 blocks) 20.3 and 19.1, of 80 heads 59.5 and 54.5, 16 of 48 heads and 68 columns (3,072) 10.8 and 10.0;
    // but 16 of 24 heads and 128 columns (1,536) 6.9 and 7.6, one sequence 3.0 and 3.2, and with two rows each 64 of 24 heads 22.6
    // and 25.6.
    const bool short_rows = one_row && NPL == 4 && (long long)n_seg * Hs * ((P + 15) / 16) > 2048;
    if (g_scan_rows && !short_rows && N % 4 == 0 && P % 4 == 0 && Cd % 4 == 0 && (((uintptr_t)state | (uintptr_t)chunk_state | (uintptr_t)xbc) & 15) == 0) {
      tlc_launch(ssm_scan_rows_kernel<NPL>, dim3(n_seg, Hs, (P + 15) / 16), dim3(128), (size_t)2 * SCAN_TT * (2 * N + 20) * sizeof(float), stream,
                 xbc, dt, dA, Dskip, state, chunk_state, seg_start, seg_seq, seq_seg_start, slots, start_pos, y, chunk_decay, mode, Hs, P, N, G, Cd);
      TLC_CHECK_LAUNCH("ssm_scan");
      return 0;
    }
  }
  dim3 grid(n_seg, Hs, (P + 4 * RP - 1) / (4 * RP));
  const size_t smem = (size_t)2 * SCAN_TT * (2 * N + 4 * RP + 4) * sizeof(float);
  auto run = [&](auto kernel) {
    tlc_launch(kernel, dim3(grid), dim3(128), smem, stream, xbc, dt, dA, Dskip, state, chunk_state, seg_start, seg_seq, seq_seg_start,
               slots, start_pos, y, chunk_decay, mode, Hs, P, N, G, Cd);
  };
  if constexpr (NPL % 4 == 0) {
    if (N % 4 == 0 && (((uintptr_t)state | (uintptr_t)chunk_state) & 15) == 0) run(ssm_scan_kernel<NPL, RP, true>);
    else run(ssm_scan_kernel<NPL, RP, false>);
  } else {
    run(ssm_scan_kernel<NPL, RP, false>);
  }
  TLC_CHECK_LAUNCH("ssm_scan");
  return 0;
}

static int scan_dispatch(const float* xbc, const float* dt, const float* dA, const float* Dskip, float* state,
                         float* chunk_state, const int* seg_start, const int* seg_seq, const int* seq_seg_start,
                         const int* slots, const int* start_pos, float* y, float* chunk_decay, int mode, int n_seg,
                         int Hs, int P, int N, int G, int Cd, cudaStream_t stream, bool one_row = false) {
#define TLC_SCAN(NPL) launch_scan<NPL>(xbc, dt, dA, Dskip, state, chunk_state, seg_start, seg_seq, seq_seg_start, slots, start_pos, y, chunk_decay, mode, n_seg, Hs, P, N, G, Cd, one_row, stream)
  if (N <= 32) return TLC_SCAN(1);
  if (N <= 64) return TLC_SCAN(2);
  if (N <= 128) return TLC_SCAN(4);
  return TLC_SCAN(8);
#undef TLC_SCAN
}

static int scan_checks(int Hs, int N, int G) {
  TLC_REQUIRE(G > 0 && Hs % G == 0, "ssm_scan: %d heads are not a multiple of %d groups", Hs, G);
  TLC_REQUIRE(N >= 1 && N <= 256, "ssm_scan: state size %d is outside the kernel's range 1..256", N);
  TLC_REQUIRE(Hs <= 65535, "ssm_scan: too many heads (%d)", Hs);
  return 0;
}

extern "C" int tlc_ssm_scan(const float* xbc, const float* dt, const float* dA, const float* Dskip, float* state,
                            const int* cu_seqlens, const int* slots, const int* start_pos, float* y, int B, int Hs,
                            int P, int N, int G, int Cd, cudaStream_t stream) {
  if (B == 0) return 0;
  if (int rc = scan_checks(Hs, N, G)) return rc;
  return scan_dispatch(xbc, dt, dA, Dskip, state, nullptr, cu_seqlens, nullptr, nullptr, slots, start_pos, y, nullptr,
                       SCAN_PLAIN, B, Hs, P, N, G, Cd, stream);
}

// The same for a step that brings one row of every sequence (a hint: the result does not depend on it).
extern "C" int tlc_ssm_scan_one_row(const float* xbc, const float* dt, const float* dA, const float* Dskip, float* state,
                                    const int* cu_seqlens, const int* slots, const int* start_pos, float* y, int B, int Hs,
                                    int P, int N, int G, int Cd, cudaStream_t stream) {
  if (B == 0) return 0;
  if (int rc = scan_checks(Hs, N, G)) return rc;
  return scan_dispatch(xbc, dt, dA, Dskip, state, nullptr, cu_seqlens, nullptr, nullptr, slots, start_pos, y, nullptr,
                       SCAN_PLAIN, B, Hs, P, N, G, Cd, stream, true);
}

// The same scan with every sequence cut into chunks that run in parallel.  seg_start [n_seg + 1]:
// first row of every chunk; seg_seq [n_seg]: its sequence; seq_seg_start [B + 1]: first chunk of
// every sequence; chunk_state: scratch [n_seg, Hs, P, N] + [n_seg, Hs] floats.
extern "C" int tlc_ssm_scan_chunked(const float* xbc, const float* dt, const float* dA, const float* Dskip,
                                    float* state, float* chunk_state, const int* seg_start, const int* seg_seq,
                                    const int* seq_seg_start, const int* slots, const int* start_pos, float* y,
                                    int B, int n_seg, int Hs, int P, int N, int G, int Cd, cudaStream_t stream) {
  if (B == 0 || n_seg == 0) return 0;
  if (int rc = scan_checks(Hs, N, G)) return rc;
  float* chunk_decay = chunk_state + (size_t)n_seg * Hs * P * N;
  if (int rc = scan_dispatch(xbc, dt, dA, Dskip, state, chunk_state, seg_start, seg_seq, seq_seg_start, slots, start_pos,
                             y, chunk_decay, SCAN_CHUNK_STATE, n_seg, Hs, P, N, G, Cd, stream)) return rc;
  if (int rc = tlc_ssm_state_pass_launch(chunk_decay, state, chunk_state, seq_seg_start, slots, start_pos, B, Hs, P * N, 0,
                                         stream)) return rc;
  return scan_dispatch(xbc, dt, dA, Dskip, state, chunk_state, seg_start, seg_seq, seq_seg_start, slots, start_pos, y,
                       chunk_decay, SCAN_CHUNK_OUT, n_seg, Hs, P, N, G, Cd, stream);
}

// ---- one-token steps: convolution and scan in one kernel ---------------------------------------------------------------
// Every sequence brings one row.  A block owns ROWS rows p of a head's state, which lie side by side in memory: one bulk
// copy brings them into shared memory, the threads update them there, one bulk copy takes them back.  The state, the
// stored windows of the channels that the block needs and the convolution's weights do not depend on the kernel before
// this one and are asked for ahead of the wait on it; after it come the row's projection, the convolution of the
// block's channels (B and C of the head's group, a thread four channels; x of its rows, the fifth warp), dt and the decay.
// B and C are convolved by every block of the group: 512 channels of L2 reads beside 16 or 32 KB of state, instead of a
// kernel of their own (2 to 5 us a layer) and a trip through memory.
//
// The windows of the x channels are the block's own to advance.  Those of B and C are read by all the blocks of (sequence,
// group), so the mixer's next kernel advances them (tlc_gated_rmsnorm_step).
// What bounds it: at batch 64 of the 1.5B sizes the state, 201 MB of a layer read and 201 MB written in 63 us (6.4 TB/s, the
// copy bandwidth measured here is 6.5); at batch 8 (25 + 25 MB in 13 us) the trip to memory and back of 1.5 waves of blocks.
// A step of the 1.5B sizes at batch 64 takes 2.97 ms, with the two kernels 3.45; at batch 8 and contexts of up to 512 1.18 and
// 1.27; of the 3B sizes at batch 16 3.29 and 3.41; of the 7B sizes at batch 32 7.01 and 7.27.
template <int NPL, int ROWS>
struct StepSmem {
  static constexpr int STATE = ROWS * 32 * NPL * 4;                       // at most
  static constexpr int OPS = (2 * 32 * NPL + ROWS + 4) * 4;               // B[N] | C[N] | x[ROWS] | dt | dA | whether a wait ran out
  static constexpr int TOTAL = STATE + OPS + 16;                          // + the mbarrier
};
template <int NPL, int ROWS, int KT>
__global__ void __launch_bounds__(160)
mamba_step_kernel(const float* __restrict__ proj, int ld, int xbc_off, int dt_off, const float* __restrict__ w,
                  const float* __restrict__ bias, const float* __restrict__ dt_bias, const float* __restrict__ A,
                  const float* __restrict__ Dskip, float* conv_state, float* state, const int* __restrict__ slots,
                  const int* __restrict__ start_pos, float* __restrict__ y, int Hs, int P, int N, int G, int Cd, int bf16_run,
                  ErrWords* err) {
  asm volatile("griddepcontrol.launch_dependents;");
  constexpr int RP = ROWS / 4;                       // rows of a warp
  extern __shared__ __align__(128) unsigned char step_sm[];
  float* ss = reinterpret_cast<float*>(step_sm);                                        // [rows][N]
  float* sm = reinterpret_cast<float*>(step_sm + StepSmem<NPL, ROWS>::STATE);
  const uint32_t bar = smem_u32(step_sm + StepSmem<NPL, ROWS>::STATE + StepSmem<NPL, ROWS>::OPS);
  int* ran_out = reinterpret_cast<int*>(sm + 2 * N + ROWS + 2);
  const int b = blockIdx.x, h = blockIdx.y, p_blk = blockIdx.z * ROWS;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int Di = Hs * P, g = h / (Hs / G), nq = N >> 2;
  const int rows = min(ROWS, P - p_blk);
  const bool has_state = start_pos[b] > 0;
  const int slot = slots[b];
  float* win = conv_state + (size_t)slot * (KT - 1) * Cd;
  float* S = state + (((size_t)slot * Hs + h) * P + p_blk) * N;
  const uint32_t bytes = (uint32_t)(rows * N * 4);
  if (threadIdx.x == 0 && has_state) {
    mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_expect_tx(bar, bytes);
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(ss)), "l"(S),
                 "r"(bytes), "r"(bar) : "memory");
  }
  // the four channels this thread convolves (-1: none), and where their values go
  int c = -1, dst = 0;
  if (warp < 4) {
    const int q = threadIdx.x;
    if (q < nq) c = Di + g * N + 4 * q;
    else if (q < 2 * nq) c = Di + G * N + g * N + 4 * (q - nq);
    dst = 4 * q;
  } else if (lane < RP && 4 * lane < rows) {
    c = h * P + p_blk + 4 * lane;
    dst = 2 * N + 4 * lane;
  }
  float4 prev[KT - 1], wk[KT], bv = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int k = 0; k < KT - 1; k++)
    prev[k] = c >= 0 && has_state ? *reinterpret_cast<const float4*>(win + (size_t)k * Cd + c) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int k = 0; k < KT; k++) wk[k] = c >= 0 ? __ldg(reinterpret_cast<const float4*>(w + (size_t)c * KT) + k) : make_float4(0.f, 0.f, 0.f, 0.f);
  if (bias && c >= 0) bv = __ldg(reinterpret_cast<const float4*>(bias + c));
  const float db = dt_bias[h], Ah = A[h], Dh = Dskip[h];
  const long long wait_limit = mbar_wait_limit(err);
  tlc_wait(proj, y);
  const float* row = proj + (size_t)b * ld;
  if (c >= 0) {
    const float4 cur = *reinterpret_cast<const float4*>(row + xbc_off + c);
    // the taps of channel c + i are the KT weights from (c + i) * KT on
    float wf[4 * KT];
#pragma unroll
    for (int k = 0; k < KT; k++) { wf[4 * k] = wk[k].x; wf[4 * k + 1] = wk[k].y; wf[4 * k + 2] = wk[k].z; wf[4 * k + 3] = wk[k].w; }
    auto conv1 = [&](int i, float b0, auto get) {
      float sum = b0;
#pragma unroll
      for (int k = 0; k < KT - 1; k++) sum = fmaf(get(prev[k]), wf[i * KT + k], sum);
      sum = silu_f(fmaf(get(cur), wf[i * KT + KT - 1], sum));
      return bf16_run ? as_operand<true>(sum) : sum;
    };
    float4 v;
    v.x = conv1(0, bv.x, [](const float4& u) { return u.x; });
    v.y = conv1(1, bv.y, [](const float4& u) { return u.y; });
    v.z = conv1(2, bv.z, [](const float4& u) { return u.z; });
    v.w = conv1(3, bv.w, [](const float4& u) { return u.w; });
    *reinterpret_cast<float4*>(sm + dst) = v;
    if (warp == 4) {                                 // x of this block's rows: nobody else reads that window
#pragma unroll
      for (int k = 0; k < KT - 1; k++) *reinterpret_cast<float4*>(win + (size_t)k * Cd + c) = k < KT - 2 ? prev[k < KT - 2 ? k + 1 : 0] : cur;
    }
  }
  if (warp == 4 && lane == 31) {
    const float dtv = softplus_f(row[dt_off + h] + db);
    sm[2 * N + ROWS] = dtv;
    sm[2 * N + ROWS + 1] = expf(dtv * Ah);
    *ran_out = 0;
  }
  __syncthreads();                                   // (also behind the mbarrier's initialisation)
  if (warp < 4) {
    // A wait that ran out is reported (the host raises): its warp leaves its rows alone and the block stores none, so that the
    // slot keeps the state it had.
    bool landed = !has_state || mbar_wait(bar, 0, err, 41, wait_limit);
    if (!landed) *ran_out = 1;
    landed = __all_sync(0xffffffffu, landed);
    const float dtv = sm[2 * N + ROWS], dAv = sm[2 * N + ROWS + 1];
    float4 Bv[NPL / 4], Cv[NPL / 4];
#pragma unroll
    for (int j = 0; j < NPL / 4; j++) {
      const int n = 4 * lane + 128 * j;
      Bv[j] = n < N ? *reinterpret_cast<const float4*>(sm + n) : make_float4(0.f, 0.f, 0.f, 0.f);
      Cv[j] = n < N ? *reinterpret_cast<const float4*>(sm + N + n) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float sum[RP];
#pragma unroll
    for (int r = 0; r < RP; r++) {
      const int p = warp * RP + r;
      const float xdt = p < rows ? sm[2 * N + p] * dtv : 0.f;
      float a = 0.f;
#pragma unroll
      for (int j = 0; j < NPL / 4; j++) {
        const int n = 4 * lane + 128 * j;
        if (n < N && p < rows && landed) {
          float4* at = reinterpret_cast<float4*>(ss + p * N + n);
          float4 u = has_state ? *at : make_float4(0.f, 0.f, 0.f, 0.f);
          u.x = fmaf(u.x, dAv, Bv[j].x * xdt); u.y = fmaf(u.y, dAv, Bv[j].y * xdt);
          u.z = fmaf(u.z, dAv, Bv[j].z * xdt); u.w = fmaf(u.w, dAv, Bv[j].w * xdt);
          a = fmaf(u.x, Cv[j].x, a); a = fmaf(u.y, Cv[j].y, a); a = fmaf(u.z, Cv[j].z, a); a = fmaf(u.w, Cv[j].w, a);
          *at = u;
        }
      }
      sum[r] = a;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // the threads' stores, before the copy reads them
    __syncwarp();                                                    // (bar.sync wants whole warps)
    asm volatile("bar.sync 1, 128;" ::: "memory");
    const bool store = *(volatile int*)ran_out == 0;
    if (threadIdx.x == 0 && store) {
      asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(S), "r"(smem_u32(ss)), "r"(bytes) : "memory");
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
#pragma unroll
    for (int r = 0; r < RP; r++) sum[r] = warp_sum(sum[r]);
    if (lane < RP) {
      float v = sum[0];
#pragma unroll
      for (int r = 1; r < RP; r++) if (lane == r) v = sum[r];
      const int p = warp * RP + lane;
      if (p < rows) y[(size_t)b * Di + (size_t)h * P + p_blk + p] = v + sm[2 * N + p] * Dh;
    }
    // complete, not only read: the next step's copy of this state starts when this kernel has ended
    if (threadIdx.x == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    // the copy that was waited for in vain is still on its way into this block's memory: it gets the default limit once more
    if (threadIdx.x == 0 && !store) mbar_wait(bar, 0, err, 41, wait_limit > TLC_WAIT_LIMIT_CYCLES ? wait_limit : TLC_WAIT_LIMIT_CYCLES);
  }
}

constexpr int STEP_BLOCKS = 4096;

// Whether mamba_step_kernel takes these sizes: 65..256 state columns and the other sizes in pieces of 16 bytes, 2 to 4 taps, on the
// device that the library is set up on.  Smaller states keep the two kernels, although measured the one would be about as
// quick or quicker there too (with the norm behind them, 48 heads of 64: 64 columns, batch 1 / 8 / 64 5.6 / 9.2 / 36.9 us with
// the two, 4.5 / 9.0 / 30.3 with the one; 16 columns 5.3 / 8.4 / 31.1 and 4.4 / 8.5 / 27.0); at 128 columns 6.2 / 11.2 / 49.3
// and 4.6 / 10.4 / 39.5, at 256 7.7 / 16.7 / 77.1 and 5.2 / 13.5 / 70.3.
extern "C" int tlc_mamba_step_ok(int Hs, int P, int N, int G, int Cd, int K) {
  return N > 64 && N <= 256 && N % 4 == 0 && P % 4 == 0 && Cd % 4 == 0 && K >= 2 && K <= 4 && G > 0 && Hs % G == 0 && Hs <= 65535 && Hs * P + 2 * G * N == Cd && tlc_error_words_here() != nullptr;
}

extern "C" int tlc_mamba_step(const float* proj, int ld, int xbc_off, int dt_off, const float* w, const float* bias,
                              const float* dt_bias, const float* A, const float* Dskip, float* conv_state, float* state,
                              const int* slots, const int* start_pos, float* y, int B, int Hs, int P, int N, int G, int Cd, int K,
                              int bf16_run, cudaStream_t stream) {
  if (B == 0) return 0;
  TLC_REQUIRE(tlc_error_words_here() != nullptr, "mamba_step: the library is not set up on this device (tlc_linear_init)");
  TLC_REQUIRE(tlc_mamba_step_ok(Hs, P, N, G, Cd, K), "mamba_step: %d heads of %d, state %d, %d groups, %d taps are outside the kernel's range", Hs, P, N, G, K);
  const void* aligned[] = {proj, w, bias, conv_state, state};
  for (const void* p : aligned) TLC_REQUIRE(((uintptr_t)p & 15) == 0, "mamba_step: operands must start on 16-byte boundaries");
  TLC_REQUIRE(ld % 4 == 0 && xbc_off % 4 == 0, "mamba_step: rows of the projection must start on 16-byte boundaries");
  // 16 rows a block (18.6 KB of shared memory), and 32 where that still makes STEP_BLOCKS blocks: then the convolution that every
  // block makes for itself counts, and the kernels beside this one no longer do.  A step of the 1.5B sizes at batch 64 (6,144 blocks
  // of 32 rows): 2.96 ms, with 16 rows 3.12; of the 7B sizes at batch 32 (3,072): 7.17 and 7.03; of 1.5B at batch 8 (768): 1.51 and
  // 1.18; of 3B at batch 16 (2,048): 4.71 and 3.29, blocks of 35 KB leave the attention kernel, which runs beside this one and
  // needs 131 KB of an SM's shared memory, no room until the last of them has started, and the products too little of
  // the first-level cache that their weight loads are in flight through.
#define TLC_STEP(NPL_, ROWS_, KT_)                                                                                                       \
  tlc_launch(mamba_step_kernel<NPL_, ROWS_, KT_>, dim3(B, Hs, (P + ROWS_ - 1) / ROWS_), dim3(160), StepSmem<NPL_, ROWS_>::TOTAL, stream,  \
             proj, ld, xbc_off, dt_off, w, bias, dt_bias, A, Dskip, conv_state, state, slots, start_pos, y, Hs, P, N, G, Cd, bf16_run,     \
             tlc_error_words())
#define TLC_STEP_K(NPL_, ROWS_) do { if (K == 4) TLC_STEP(NPL_, ROWS_, 4); else if (K == 3) TLC_STEP(NPL_, ROWS_, 3); else TLC_STEP(NPL_, ROWS_, 2); } while (0)
  const bool wide = (long long)B * Hs * ((P + 31) / 32) >= STEP_BLOCKS;
  if (N <= 128) { if (wide) TLC_STEP_K(4, 32); else TLC_STEP_K(4, 16); }
  else { if (wide) TLC_STEP_K(8, 32); else TLC_STEP_K(8, 16); }
#undef TLC_STEP_K
#undef TLC_STEP
  TLC_CHECK_LAUNCH("mamba_step");
  return 0;
}
