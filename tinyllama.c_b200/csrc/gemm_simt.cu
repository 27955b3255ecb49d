// Linear layers on the CUDA cores: out[m,n] = (sum_k a[m,k] * w[n,k]) * colscale[n] + colbias[n].
//
// y[r] = sum_c W[r,c] x[c] with W stored [out, in] is the reference's matmul
// (cpu_op.c:121-189 for one row, 253-328 for a batch).  These kernels are the true
// 32-bit path (FFMA, 32-bit accumulation, no tensor cores, no reduced matrix mode) and the
// fall-back for bfloat16 shapes the tensor-core kernel refuses.
// Two shapes: tiles for many rows, and a warp for one to four columns for the few rows of a
// decode step, where the weight matrix is streamed once.  The order of a sum follows from the
// kernel, and so from M, N and K: a lane's shares of K in order and then the lanes, K in order,
// or K in four parts that are each in order and then added.
#include "common.cuh"

// ---- tiled kernel ---------------------------------------------------------------------
#define BM 64
#define BN 64
#define BK 16

template <typename TA, typename TW, typename TO>
__global__ void __launch_bounds__(256)
gemm_tiled_kernel(const TA* __restrict__ a, int lda, const TW* __restrict__ w, int ldw, TO* __restrict__ out, int ldo,
                  const float* __restrict__ colscale, const float* __restrict__ colbias, TlcEpi accumulate, int M, int N,
                  int K) {
  tlc_pdl(a, w, out);
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[BK][BN + 4];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int tm = (tid / 16) * 4, tn = (tid % 16) * 4;
  float acc[4][4] = {};
  // each thread loads 4 elements of each tile: row = tid/4 (0..63), k = (tid%4)*4 .. +3
  const int lr = tid >> 2, lk = (tid & 3) * 4;
  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int k = k0 + lk + i;
      const int m = m0 + lr, n = n0 + lr;
      As[lk + i][lr] = (m < M && k < K) ? to_f32(a[(size_t)m * lda + k]) : 0.f;
      Ws[lk + i][lr] = (n < N && k < K) ? to_f32(w[(size_t)n * ldw + k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; k++) {
      float av[4], wv[4];
#pragma unroll
      for (int i = 0; i < 4; i++) { av[i] = As[k][tm + i]; wv[i] = Ws[k][tn + i]; }
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int m = m0 + tm + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int n = n0 + tn + j;
      if (n >= N) continue;
      float v = acc[i][j];
      if (colscale) v *= colscale[n];
      if (colbias) v += colbias[n];
      TO* o = out + (size_t)m * ldo + n;
      if (accumulate) v += to_f32(*o);
      *o = from_f32<TO>(v);
    }
  }
}

// ---- few rows: one warp per output column, the weight row read once ----------------------
template <typename TA, typename TW, typename TO, int MT>
__global__ void __launch_bounds__(256)
gemm_skinny_kernel(const TA* __restrict__ a, int lda, const TW* __restrict__ w, int ldw, TO* __restrict__ out, int ldo,
                   const float* __restrict__ colscale, const float* __restrict__ colbias, TlcEpi accumulate, int M, int N,
                   int K, int m_base) {
  tlc_pdl(a, w, out);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = blockIdx.x * (blockDim.x >> 5) + warp;
  if (n >= N) return;
  const TW* wr = w + (size_t)n * ldw;
  float acc[MT];
#pragma unroll
  for (int m = 0; m < MT; m++) acc[m] = 0.f;
  for (int k = lane; k < K; k += 32) {
    const float wv = to_f32(wr[k]);
#pragma unroll
    for (int m = 0; m < MT; m++)
      if (m_base + m < M) acc[m] = fmaf(to_f32(a[(size_t)(m_base + m) * lda + k]), wv, acc[m]);
  }
#pragma unroll
  for (int m = 0; m < MT; m++) {
    float v = warp_sum(acc[m]);
    if (lane == 0 && m_base + m < M) {
      if (colscale) v *= colscale[n];
      if (colbias) v += colbias[n];
      TO* o = out + (size_t)(m_base + m) * ldo + n;
      if (accumulate) v += to_f32(*o);
      *o = from_f32<TO>(v);
    }
  }
}

// bfloat16 weights and activations, K a multiple of 8 and 16-byte aligned rows: 128-bit loads.
template <typename TO, int MT>
__global__ void __launch_bounds__(256)
gemm_skinny_bf16x8_kernel(const __nv_bfloat16* __restrict__ a, int lda, const __nv_bfloat16* __restrict__ w, int ldw,
                          TO* __restrict__ out, int ldo, const float* __restrict__ colscale,
                          const float* __restrict__ colbias, TlcEpi accumulate, int M, int N, int K, int m_base) {
  tlc_pdl(a, out);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = blockIdx.x * (blockDim.x >> 5) + warp;
  if (n >= N) return;
  const uint4* wr = reinterpret_cast<const uint4*>(w + (size_t)n * ldw);
  float acc[MT];
#pragma unroll
  for (int m = 0; m < MT; m++) acc[m] = 0.f;
  const int K8 = K >> 3;
  for (int k8 = lane; k8 < K8; k8 += 32) {
    const uint4 wq = __ldg(wr + k8);
    const __nv_bfloat162* wp = reinterpret_cast<const __nv_bfloat162*>(&wq);
    float wf[8];
#pragma unroll
    for (int i = 0; i < 4; i++) { float2 f = __bfloat1622float2(wp[i]); wf[2 * i] = f.x; wf[2 * i + 1] = f.y; }
#pragma unroll
    for (int m = 0; m < MT; m++) {
      if (m_base + m < M) {
        const uint4 aq = *reinterpret_cast<const uint4*>(a + (size_t)(m_base + m) * lda + (size_t)k8 * 8);
        const __nv_bfloat162* ap = reinterpret_cast<const __nv_bfloat162*>(&aq);
#pragma unroll
        for (int i = 0; i < 4; i++) {
          float2 f = __bfloat1622float2(ap[i]);
          acc[m] = fmaf(f.x, wf[2 * i], acc[m]);
          acc[m] = fmaf(f.y, wf[2 * i + 1], acc[m]);
        }
      }
    }
  }
#pragma unroll
  for (int m = 0; m < MT; m++) {
    float v = warp_sum(acc[m]);
    if (lane == 0 && m_base + m < M) {
      if (colscale) v *= colscale[n];
      if (colbias) v += colbias[n];
      TO* o = out + (size_t)(m_base + m) * ldo + n;
      if (accumulate) v += to_f32(*o);
      *o = from_f32<TO>(v);
    }
  }
}

// ---- 32-bit operands in 16-byte pieces (rows of a multiple of 4 values on 16-byte boundaries) -----------------------
// Two kernels that do what the two general ones above do, in true 32-bit arithmetic with the sums in the same number of
// terms.  What bounded the general ones was loads: one 4-byte load a lane in flight (a one-token step of two
// sequences read its weights at 0.75 TB/s), and shared-memory reads a product (4 x 4 results a thread: 17 TFLOP/s).

// 16 bytes that this kernel reads once: they leave the first-level cache to the activations.
__device__ __forceinline__ float4 load_once(const float4* p) {
  float4 v;
  asm("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}

// Few rows: a warp takes COLS output columns and reads their weight rows 512 bytes at a time, U pieces a column in flight; an
// activation piece serves COLS columns.  Nothing is read before the wait on the previous kernel: in this arithmetic w may be
// what that kernel wrote (weights asked for ahead of the wait: 2 rows 13.4 us and not 14.1, 8 rows 44.9 and not 42.1).
// 2 rows, 2048 -> 8240 (67 MB): 90 -> 14.1 us, 4096 -> 2048 (34 MB): 95 -> 13.0 us; 8 rows 216 -> 20.6 and 237 -> 42 us.
template <typename TO, int MT, int COLS, int U>
__global__ void __launch_bounds__(256)
gemm_skinny_f32x4_kernel(const float* __restrict__ a, int lda, const float* __restrict__ w, int ldw, TO* __restrict__ out,
                         int ldo, const float* __restrict__ colscale, const float* __restrict__ colbias, TlcEpi accumulate,
                         int M, int N, int K, int m_base) {
  tlc_pdl(a, w, out);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = (blockIdx.x * 8 + warp) * COLS;
  const int K4 = K >> 2;
  const float4* wr[COLS];
#pragma unroll
  for (int c = 0; c < COLS; c++) wr[c] = reinterpret_cast<const float4*>(w + (size_t)min(n0 + c, N - 1) * ldw);   // clamped rows are never stored
  float acc[MT][COLS];
#pragma unroll
  for (int m = 0; m < MT; m++)
#pragma unroll
    for (int c = 0; c < COLS; c++) acc[m][c] = 0.f;
  for (int i0 = lane; i0 - lane < K4; i0 += 32 * U) {
    float4 wv[COLS][U];
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int c = 0; c < COLS; c++) wv[c][u] = i0 + 32 * u < K4 ? load_once(wr[c] + i0 + 32 * u) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int u = 0; u < U; u++) {
      if (i0 + 32 * u < K4) {
#pragma unroll
        for (int m = 0; m < MT; m++) {
          if (m_base + m < M) {
            const float4 x = *(reinterpret_cast<const float4*>(a + (size_t)(m_base + m) * lda) + i0 + 32 * u);
#pragma unroll
            for (int c = 0; c < COLS; c++) {
              acc[m][c] = fmaf(x.x, wv[c][u].x, acc[m][c]);
              acc[m][c] = fmaf(x.y, wv[c][u].y, acc[m][c]);
              acc[m][c] = fmaf(x.z, wv[c][u].z, acc[m][c]);
              acc[m][c] = fmaf(x.w, wv[c][u].w, acc[m][c]);
            }
          }
        }
      }
    }
  }
#pragma unroll
  for (int m = 0; m < MT; m++) {
#pragma unroll
    for (int c = 0; c < COLS; c++) {
      float v = warp_sum(acc[m][c]);
      const int n = n0 + c;
      if (lane == 0 && m_base + m < M && n < N) {
        if (colscale) v *= colscale[n];
        if (colbias) v += colbias[n];
        TO* o = out + (size_t)(m_base + m) * ldo + n;
        if (accumulate) v += to_f32(*o);
        *o = from_f32<TO>(v);
      }
    }
  }
}

// Two products of a pair of accumulators in one instruction, each rounded as fmaf rounds it.
__device__ __forceinline__ void fma_pair(float2& d, float2 a, float2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;"
      : "+l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)));
}

// A tile of 64 rows x 16 CT columns, 128 threads with 8 x CT results each; two K-steps of 16 in shared memory, the next one in
// registers.  CT = 8 for outputs of many tiles: 600 rows of 2048 -> 8192 500 us (41 TFLOP/s), 1,200 879 us (46).  CT = 4 with KG = 4,
// four groups of 128 threads that take a quarter of K each, for outputs of few tiles and a K so short that the meetings of a
// cluster (below) would cost more than its blocks bring: f32_plan has both sides.
constexpr int FT_M = 64, FT_K = 16, FT_LD = 4;
template <typename TO, int CT, int KG>
__global__ void __launch_bounds__(128 * KG)
gemm_tiled_f32x4_kernel(const float* __restrict__ a, int lda, const float* __restrict__ w, int ldw, TO* __restrict__ out,
                        int ldo, const float* __restrict__ colscale, const float* __restrict__ colbias, TlcEpi accumulate,
                        int M, int N, int K) {
  tlc_pdl(a, w, out);
  constexpr int TN = 16 * CT, LA = FT_M + FT_LD, LW = TN + FT_LD;
  constexpr int PA = FT_M * FT_K / 4 / 128, PW = TN * FT_K / 4 / 128;   // 16-byte pieces a thread brings of each operand
  extern __shared__ __align__(16) float ft_sm[];
  const int grp = threadIdx.x >> 7, tid = threadIdx.x & 127;
  float* As = ft_sm + grp * 2 * FT_K * (LA + LW);            // [2][FT_K][LA]
  float* Ws = As + 2 * FT_K * LA;                            // [2][FT_K][LW]
  const int m0 = blockIdx.y * FT_M, n0 = blockIdx.x * TN;
  const int tx = tid & 15, ty = tid >> 4;
  const int steps = (K + FT_K - 1) / FT_K, per = (steps + KG - 1) / KG;
  const int s_begin = min(steps, grp * per), s_end = min(steps, s_begin + per);
  float4 ra[PA], rw[PW];
  auto load = [&](int s) {
#pragma unroll
    for (int i = 0; i < PA; i++) {
      const int q = tid + 128 * i, r = m0 + (q >> 2), k = s * FT_K + (q & 3) * 4;
      ra[i] = (r < M && k < K) ? *reinterpret_cast<const float4*>(a + (size_t)r * lda + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < PW; i++) {
      const int q = tid + 128 * i, r = n0 + (q >> 2), k = s * FT_K + (q & 3) * 4;
      rw[i] = (r < N && k < K) ? __ldg(reinterpret_cast<const float4*>(w + (size_t)r * ldw + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int i = 0; i < PA; i++) {
      const int q = tid + 128 * i;
      float* d = As + buf * FT_K * LA + (q & 3) * 4 * LA + (q >> 2);
      d[0] = ra[i].x; d[LA] = ra[i].y; d[2 * LA] = ra[i].z; d[3 * LA] = ra[i].w;
    }
#pragma unroll
    for (int i = 0; i < PW; i++) {
      const int q = tid + 128 * i;
      float* d = Ws + buf * FT_K * LW + (q & 3) * 4 * LW + (q >> 2);
      d[0] = rw[i].x; d[LW] = rw[i].y; d[2 * LW] = rw[i].z; d[3 * LW] = rw[i].w;
    }
  };
  float2 acc[8][CT / 2];
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < CT / 2; j++) acc[i][j] = make_float2(0.f, 0.f);
  // all groups go through the same number of barriers
  if (s_begin < s_end) { load(s_begin); store(0); }
  __syncthreads();
#pragma unroll 1
  for (int i = 0; i < per; i++) {
    const int s = s_begin + i, buf = i & 1;
    if (s + 1 < s_end) load(s + 1);
    if (s < s_end) {
      const float* Ab = As + buf * FT_K * LA + ty * 8;
      const float* Wb = Ws + buf * FT_K * LW + tx * 4;
#pragma unroll
      for (int k = 0; k < FT_K; k++) {
        const float4 a0 = *reinterpret_cast<const float4*>(Ab + k * LA), a1 = *reinterpret_cast<const float4*>(Ab + k * LA + 4);
        const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
        float2 wv[CT / 2];
#pragma unroll
        for (int h = 0; h < CT / 4; h++) {
          const float4 b = *reinterpret_cast<const float4*>(Wb + k * LW + h * 64);
          wv[2 * h] = make_float2(b.x, b.y);
          wv[2 * h + 1] = make_float2(b.z, b.w);
        }
#pragma unroll
        for (int r = 0; r < 8; r++)
#pragma unroll
          for (int j = 0; j < CT / 2; j++) fma_pair(acc[r][j], make_float2(av[r], av[r]), wv[j]);
      }
    }
    if (s + 1 < s_end) store(buf ^ 1);
    __syncthreads();
  }
  if constexpr (KG > 1) {
    float* part = ft_sm;                                     // the other groups' sums, [KG - 1][8 * CT][128]
    if (grp > 0) {
      float* mine = part + (grp - 1) * 8 * CT * 128 + tid;
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < CT / 2; j++) {
          mine[((i * CT) + 2 * j) * 128] = acc[i][j].x;
          mine[((i * CT) + 2 * j + 1) * 128] = acc[i][j].y;
        }
    }
    __syncthreads();
    if (grp > 0) return;
#pragma unroll
    for (int q = 0; q < KG - 1; q++) {                       // in the order of K
      const float* other = part + q * 8 * CT * 128 + tid;
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < CT / 2; j++) {
          acc[i][j].x += other[((i * CT) + 2 * j) * 128];
          acc[i][j].y += other[((i * CT) + 2 * j + 1) * 128];
        }
    }
  }
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int m = m0 + ty * 8 + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < CT; j++) {
      const int n = n0 + tx * 4 + (j >> 2) * 64 + (j & 3);
      if (n >= N) continue;
      float v = (j & 1) ? acc[i][j >> 1].y : acc[i][j >> 1].x;
      if (colscale) v *= colscale[n];
      if (colbias) v += colbias[n];
      TO* o = out + (size_t)m * ldo + n;
      if (accumulate) v += to_f32(*o);
      *o = from_f32<TO>(v);
    }
  }
}
constexpr int ft_smem(int CT, int KG) { return KG * 2 * FT_K * (FT_M + 16 * CT + 2 * FT_LD) * 4; }
static_assert(ft_smem(4, 4) >= 3 * 8 * 4 * 128 * 4 && ft_smem(8, 1) <= 48 * 1024, "the other groups' sums reuse the operands' memory");

// The same where the tiles are too few for the SMs, or fill their last round badly, and K is long enough: a tile of 8 TM rows x 64 NC columns, 128 threads
// with TM x 4 NC results each, K-steps of KS.  Rows of both operands lie turned by 32 / (KS / 4) values for every four of K,
// which keeps the stores of the transposed pieces clear of bank conflicts.  `split` blocks of a thread-block cluster share a tile's
// K-steps: each leaves its sums in its own shared memory, the cluster meets, and block r adds up its share of the rows over
// all ranks, in their order, through distributed shared memory (the order follows from M, N and K alone).  K in four parts
// within a block of 64 x 64 (or the tiles of 64 x 128), before, and this, microseconds: 4096 -> 2048 at 17 / 64 / 128 / 200 / 310 / 600 /
// 1,200 rows 125 / 134 / 135 / 136 / 263 / 392 / 621 and 47 / 60 / 71 / 116 / 180 / 306 / 533, 2048 -> 8192 at 17 / 64 / 128 / 200 / 310
// rows 66 / 71 / 138 / 267 / 313 and 40 / 67 / 119 / 240 / 296.  What bounds all of these tiles is a rate of about 42 TFLOP/s of the 74 that the FP32 lanes have: more
// warps an SM (sixteen, 64 x 128), more results a thread (8 x 16) and operands stored twice so that no register
// has to be doubled all came to 38 to 42.
template <int TM, int NC, int KS> constexpr int fs_smem(int split) {
  constexpr int FS_N = 64 * NC;
  return (int)sizeof(float) * (split > 1 && 8 * TM * FS_N > 2 * KS * (8 * TM + FS_N) ? 8 * TM * FS_N : 2 * KS * (8 * TM + FS_N));   // (the sums reuse the operands' memory)
}
template <typename TO, int TM, int NC, int KS>
__global__ void __launch_bounds__(128, TM == 8 ? 2 : 4)
gemm_split_f32x4_kernel(const float* __restrict__ a, int lda, const float* __restrict__ w, int ldw, TO* __restrict__ out,
                        int ldo, const float* __restrict__ colscale, const float* __restrict__ colbias, TlcEpi accumulate,
                        int M, int N, int K, int split) {
  tlc_pdl(a, w, out);
  constexpr int FS_N = 64 * NC, ROWS = 8 * TM, PK = KS / 4, PW = FS_N * PK / 128;   // 16-byte pieces of a row; of the weights, a thread (of the activations one)
  extern __shared__ __align__(16) float fs_sm[];
  float* As = fs_sm;                                         // [2][KS][ROWS]
  float* Ws = fs_sm + 2 * KS * ROWS;                       // [2][KS][FS_N]
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int rank = (int)blockIdx.x % split;                  // clusters are runs of `split` consecutive blocks
  const int m0 = blockIdx.y * ROWS, n0 = (int)blockIdx.x / split * FS_N;
  const int steps = (K + KS - 1) / KS;
  const int s_begin = (int)((long long)steps * rank / split), s_end = (int)((long long)steps * (rank + 1) / split);
  // this thread's pieces: rows past the matrices are clamped (what they make is not stored), K past its end reads as zero
  static_assert(ROWS * PK == 128, "one piece of the activations a thread");
  constexpr int TURN = 32 / PK;                              // by how much rows are turned for every four of K
  const int q = tid / PK, kq = tid % PK * 4;
  const float* pa = a + (size_t)min(m0 + q, M - 1) * lda + kq;
  const float* pw[PW];
#pragma unroll
  for (int i = 0; i < PW; i++) pw[i] = w + (size_t)min(n0 + q + 128 / PK * i, N - 1) * ldw + kq;
  float4 ra, rw[PW];
  auto load = [&](int s) {
    const bool in = s * KS + kq < K;                       // (K is a multiple of 4)
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    ra = in ? *reinterpret_cast<const float4*>(pa + s * KS) : z;
#pragma unroll
    for (int i = 0; i < PW; i++) rw[i] = in ? *reinterpret_cast<const float4*>(pw[i] + s * KS) : z;
  };
  auto store = [&](int buf) {
    float* d = As + buf * KS * ROWS + kq * ROWS + ((q + TURN * (kq / 4)) & (ROWS - 1));
    d[0] = ra.x; d[ROWS] = ra.y; d[2 * ROWS] = ra.z; d[3 * ROWS] = ra.w;
#pragma unroll
    for (int i = 0; i < PW; i++) {
      const int c = q + 128 / PK * i;
      d = Ws + buf * KS * FS_N + kq * FS_N + (c & ~63) + ((c + TURN * (kq / 4)) & 63);
      d[0] = rw[i].x; d[FS_N] = rw[i].y; d[2 * FS_N] = rw[i].z; d[3 * FS_N] = rw[i].w;
    }
  };
  float2 acc[TM][2 * NC];
#pragma unroll
  for (int i = 0; i < TM; i++)
#pragma unroll
    for (int j = 0; j < 2 * NC; j++) acc[i][j] = make_float2(0.f, 0.f);
  if (s_begin < s_end) { load(s_begin); store(0); }
  __syncthreads();
#pragma unroll 1
  for (int s = s_begin; s < s_end; s++) {
    const int buf = (s - s_begin) & 1;
    if (s + 1 < s_end) load(s + 1);
#pragma unroll
    for (int k = 0; k < KS; k++) {
      const int turn = TURN * (k >> 2);
      const float* Ab = As + (buf * KS + k) * ROWS + ((TM * ty + turn) & (ROWS - 1));
      const float* Wb = Ws + (buf * KS + k) * FS_N + ((4 * tx + turn) & 63);
      float av[TM];
#pragma unroll
      for (int h = 0; h < TM / 4; h++) {
        const float4 v = *reinterpret_cast<const float4*>(Ab + 4 * h);
        av[4 * h] = v.x; av[4 * h + 1] = v.y; av[4 * h + 2] = v.z; av[4 * h + 3] = v.w;
      }
#pragma unroll
      for (int h = 0; h < NC; h++) {
        const float4 v = *reinterpret_cast<const float4*>(Wb + 64 * h);
#pragma unroll
        for (int r = 0; r < TM; r++) {
          fma_pair(acc[r][2 * h], make_float2(av[r], av[r]), make_float2(v.x, v.y));
          fma_pair(acc[r][2 * h + 1], make_float2(av[r], av[r]), make_float2(v.z, v.w));
        }
      }
    }
    if (s + 1 < s_end) store(buf ^ 1);
    __syncthreads();
  }
  // four columns of a row from their sum to the output
  const bool vec = ldo % 4 == 0 && (uintptr_t)out % (4 * sizeof(TO)) == 0;
  auto finish = [&](int m, int n, float4 v) {
    const float x[4] = {v.x, v.y, v.z, v.w};
    float y[4];
    TO* o = out + (size_t)m * ldo + n;
#pragma unroll
    for (int c = 0; c < 4; c++) {
      y[c] = x[c];
      if (n + c < N) {
        if (colscale) y[c] *= colscale[n + c];
        if (colbias) y[c] += colbias[n + c];
        if (accumulate) y[c] += to_f32(o[c]);
      }
    }
    if (std::is_same<TO, float>::value && vec && n + 4 <= N) {
      *reinterpret_cast<float4*>(o) = make_float4(y[0], y[1], y[2], y[3]);
    } else {
#pragma unroll
      for (int c = 0; c < 4; c++)
        if (n + c < N) o[c] = from_f32<TO>(y[c]);
    }
  };
  if (split == 1) {
#pragma unroll
    for (int i = 0; i < TM; i++) {
      const int m = m0 + ty * TM + i;
      if (m >= M) break;
#pragma unroll
      for (int h = 0; h < NC; h++)
        finish(m, n0 + 4 * tx + 64 * h, make_float4(acc[i][2 * h].x, acc[i][2 * h].y, acc[i][2 * h + 1].x, acc[i][2 * h + 1].y));
    }
    return;
  }
  // (the last barrier of the loop is behind every read of the operands)
#pragma unroll
  for (int i = 0; i < TM; i++)
#pragma unroll
    for (int h = 0; h < NC; h++)
      *reinterpret_cast<float4*>(fs_sm + (ty * TM + i) * FS_N + 4 * tx + 64 * h) =
          make_float4(acc[i][2 * h].x, acc[i][2 * h].y, acc[i][2 * h + 1].x, acc[i][2 * h + 1].y);
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  const int rows_per = ROWS / split, lane4 = (tid & 31) * 4;
  const float* src[8];
#pragma unroll
  for (int r = 0; r < 8; r++) {
    unsigned long long at;                                   // the same word in the block of rank r, for ordinary loads
    asm("mapa.u64 %0, %1, %2;" : "=l"(at) : "l"((unsigned long long)(uintptr_t)fs_sm), "r"(min(r, split - 1)));
    src[r] = reinterpret_cast<const float*>((uintptr_t)at);
  }
#pragma unroll 1
  for (int i = tid >> 5; i < NC / 2 * rows_per; i += 4) {    // (128 columns of a row a warp)
    const int row = rank * rows_per + i / (NC / 2), col = 128 * (i % (NC / 2)) + lane4;
    if (m0 + row >= M) break;
    float4 x[8];
#pragma unroll
    for (int r = 0; r < 8; r++)
      x[r] = r < split ? *reinterpret_cast<const float4*>(src[r] + row * FS_N + col) : make_float4(0.f, 0.f, 0.f, 0.f);
    float4 v = x[0];
#pragma unroll
    for (int r = 1; r < 8; r++) { v.x += x[r].x; v.y += x[r].y; v.z += x[r].z; v.w += x[r].w; }   // absent ranks add zero
    finish(m0 + row, n0 + col, v);
  }
  // no block leaves while another may still read its sums
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

static int g_f32_tile_rows = 0, g_f32_split = 0;             // test hooks: rows of a tile (32 or 64), blocks a tile; 0: chosen
extern "C" void tlc_linear_f32_tiles(int rows, int split) {
  // (a cluster adds up to eight blocks' sums, each a whole share of the rows; the other two kinds of tiles have one block)
  const bool there = (rows == 32 || rows == 64) && (split == 1 || split == 2 || split == 4 || split == 8 || (rows == 64 && (split == 0 || split == -4)));
  g_f32_tile_rows = there ? rows : 0;
  g_f32_split = there ? split : 0;
}

template <typename TO, int TM, int NC, int KS>
static void launch_split_f32x4(const float* a, int lda, const float* w, int ldw, TO* out, int ldo, const float* colscale, const float* colbias,
                               TlcEpi accumulate, int M, int N, int K, int split, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((N + 64 * NC - 1) / (64 * NC) * split, (M + 8 * TM - 1) / (8 * TM));
  cfg.blockDim = dim3(128);
  cfg.dynamicSmemBytes = fs_smem<TM, NC, KS>(split);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = g_tlc_pdl ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = split;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = split > 1 ? 2 : 1;
  cudaLaunchKernelEx(&cfg, gemm_split_f32x4_kernel<TO, TM, NC, KS>, a, lda, w, ldw, out, ldo, colscale, colbias, accumulate, M, N, K, split);
}

// Which tiles 17 and more rows take, by how much work lands on the fullest SM (so the order of a sum follows from the sizes and
// the number of SMs).  For a K of some thousand, in units of the time that a block of 64 x 256 columns with all of K takes beside a
// second one on its SM: n blocks cost 1, 1, 1.6, 2, 2.6, ... (a block alone is no quicker than two: the schedulers wait), a
// cluster 0.012 for each of its blocks, and the tiles of 64 x 128, at two and more blocks an SM, 0.71, 0.935, 1.16, ... for 3,
// 4, 5, ... (fitted to 17 to 1,200 rows of 2048 -> 8192 and 4096 -> 2048).  No split below four: a block's
// sums would be longer, and further off, than those of K in four parts are.  Tiles of 32 rows, eight blocks each, where
// that makes no more than four blocks an SM.
//
// What a cluster costs whatever K is (its meetings, and a tile's sums through shared memory) is more than it brings where K is
// short, and tiles of 256 columns are where the output has 64: there one block a tile, of 64 x 128 or with K in four parts
// within the block.  f32_us is a time in microseconds of each kind, fitted to 905 products of K 32 to 12288, N 64 to 16384 and
// 17 to 3,000 rows; of the two candidates the better one by it is within 6 % of the better one as measured in all but 7 of them
// (15 % at most).  Cluster and one block a tile, microseconds: 1,200 rows of 32 -> 2048 39.5 and 9.4, of 256 -> 2048 58.6
// and 43.1, of 1024 -> 2048 153 and 159; 310 rows of 128 -> 8192 49.2 and 24.1, of 1024 -> 8192 162 and 159; 48 rows of 64 -> 2048 6.2
// and 5.0, of 128 -> 2048 6.3 and 7.0, of 1024 -> 2048 19.7 and 35.3; 3,000 rows of 1024 -> 64 57 and 37.
struct F32Plan { int rows, split; };                         // split 0: the tiles of 64 x 128; -4: of 64 x 64, K in four parts
static int f32_blocks(int rows, int cols, int split, int M, int N, int sms) {   // on the fullest SM
  const long long tiles = (long long)((M + rows - 1) / rows) * ((N + cols - 1) / cols);
  return (int)((tiles * split + sms - 1) / sms);
}
static double f32_pairs(int f) { return f <= 2 ? 1.0 : f / 2 + (f & 1 ? 0.6 : 0.0); }   // f blocks of 64 x 256 columns
static double f32_us(F32Plan p, int M, int N, int K, int sms) {
  if (p.rows == 32) {
    const int f = f32_blocks(32, 128, p.split, M, N, sms);
    return 3.0 + f + K * (0.0031 + 0.003 * f);
  }
  if (p.split > 0) {
    const int f = f32_blocks(64, 256, p.split, M, N, sms);
    return 1.2 + 4.5 * f + 0.162 * K / p.split * f32_pairs(f);
  }
  if (p.split == 0) {
    const int f = f32_blocks(64, 128, 1, M, N, sms);
    return 2.5 + 0.85 * f + K * (0.0126 + 0.0458 * (f < 3 ? 3 : f));
  }
  return 1.1 + f32_blocks(64, 64, 1, M, N, sms) * (2.44 + 0.0315 * K);
}
static F32Plan f32_plan(int M, int N, int K, int sms) {
  if (g_f32_tile_rows) return F32Plan{g_f32_tile_rows == 32 ? 32 : 64, g_f32_split};
  auto over = [](long long x, long long y) { return (x + y - 1) / y; };
  const long long whole = over(N, 128) * over(M, 64);
  const F32Plan alone{64, whole >= 2 * sms ? 0 : -4};
  F32Plan best = alone;
  if (over(N, 128) * over(M, 32) * 8 <= 4 * sms) {
    best = F32Plan{32, 8};
  } else {
    double cost = whole >= 2 * sms ? 0.225 * over(whole, sms) + 0.035 : 1e30;
    for (int split = 4; split <= 8; split *= 2) {
      const double c = f32_pairs(f32_blocks(64, 256, split, M, N, sms)) / split + 0.012 * split;
      if (c < cost) { cost = c; best = F32Plan{64, split}; }
    }
  }
  return best.split > 0 && f32_us(alone, M, N, K, sms) < f32_us(best, M, N, K, sms) ? alone : best;
}
// 256 * rows + split (its low byte)
extern "C" int tlc_linear_f32_plan(int M, int N, int K, int sms) {
  const F32Plan plan = f32_plan(M, N, K, sms);
  return plan.rows * 256 + (plan.split & 255);
}

int tlc_linear_simt_init();

template <typename TO>
static int launch_simt_f32x4(const float* a, int lda, const float* w, int ldw, TO* out, int ldo, const float* colscale,
                              const float* colbias, TlcEpi accumulate, int M, int N, int K, cudaStream_t stream) {
  static int sms = 0;
  if (sms == 0) { int dev = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev); }
  if (M > 16) {
    if (int rc = tlc_linear_simt_init()) return rc;
    const F32Plan plan = f32_plan(M, N, K, sms);
#define TLC_FS(TM_, NC_, KS_) launch_split_f32x4<TO, TM_, NC_, KS_>(a, lda, w, ldw, out, ldo, colscale, colbias, accumulate, M, N, K, plan.split, stream)
    if (plan.rows == 32) TLC_FS(4, 2, 16);
    else if (plan.split > 0) TLC_FS(8, 4, 8);
    else if (plan.split == 0)
      tlc_launch(gemm_tiled_f32x4_kernel<TO, 8, 1>, dim3((N + 127) / 128, (M + 63) / 64), dim3(128), ft_smem(8, 1), stream, a, lda, w, ldw, out, ldo, colscale, colbias, accumulate, M, N, K);
    else
      tlc_launch(gemm_tiled_f32x4_kernel<TO, 4, 4>, dim3((N + 63) / 64, (M + 63) / 64), dim3(512), ft_smem(4, 4), stream, a, lda, w, ldw, out, ldo, colscale, colbias, accumulate, M, N, K);
#undef TLC_FS
    TLC_CHECK_LAUNCH("linear(simt)");
    return 0;
  }
  // A warp's columns share its activations: a read of them costs as much as one of the weights, so up to 2 rows take two
  // columns and more rows four, where that still makes two blocks an SM.  9 to 16 rows are two launches, each of which reads the
  // weights: 12 rows of 2048 -> 8240 40 us, of 4096 -> 2048 62 us; as tiles 66 and 126.
  auto blocks_of = [&](int cols) { return (unsigned)((N + 8 * cols - 1) / (8 * cols)); };
#define TLC_SK4(MT_, C_, U_) tlc_launch(gemm_skinny_f32x4_kernel<TO, MT_, C_, U_>, dim3(blocks_of(C_)), dim3(256), 0, stream, a, lda, w, ldw, out, ldo, \
                                        colscale, colbias, accumulate, M, N, K, mb)
  for (int mb = 0; mb < M; mb += 8) {
    const int rows = M - mb;
    const bool two = blocks_of(2) >= 2 * (unsigned)sms;
    if (rows <= 2) { if (two) TLC_SK4(2, 2, 4); else TLC_SK4(2, 1, 8); }
    else if (rows <= 4) { if (two) TLC_SK4(4, 2, 4); else TLC_SK4(4, 2, 2); }
    else { if (two) TLC_SK4(8, 4, 2); else TLC_SK4(8, 2, 2); }
  }
#undef TLC_SK4
  TLC_CHECK_LAUNCH("linear(simt)");
  return 0;
}

template <typename TA, typename TW, typename TO>
static int launch_simt(const void* a, int lda, const void* w, int ldw, void* out, int ldo, const float* colscale,
                       const float* colbias, TlcEpi accumulate, int M, int N, int K, cudaStream_t stream) {
  constexpr int MT = 8;
  if constexpr (std::is_same<TA, float>::value && std::is_same<TW, float>::value) {
    if (K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)a % 16 == 0) && ((uintptr_t)w % 16 == 0))
      return launch_simt_f32x4<TO>((const float*)a, lda, (const float*)w, ldw, (TO*)out, ldo, colscale, colbias, accumulate, M, N, K, stream);
  }
  if (M <= 16) {
    const bool vec = std::is_same<TA, __nv_bfloat16>::value && std::is_same<TW, __nv_bfloat16>::value && (K % 8 == 0) &&
                     (lda % 8 == 0) && (ldw % 8 == 0) && ((uintptr_t)a % 16 == 0) && ((uintptr_t)w % 16 == 0);
    const unsigned blocks = (unsigned)((N + 7) / 8);
    for (int mb = 0; mb < M; mb += MT) {
      if (vec)
        tlc_launch(gemm_skinny_bf16x8_kernel<TO, MT>, dim3(blocks), dim3(256), 0, stream, 
            (const __nv_bfloat16*)a, lda, (const __nv_bfloat16*)w, ldw, (TO*)out, ldo, colscale, colbias, accumulate, M,
            N, K, mb);
      else
        tlc_launch(gemm_skinny_kernel<TA, TW, TO, MT>, dim3(blocks), dim3(256), 0, stream, (const TA*)a, lda, (const TW*)w, ldw, (TO*)out,
                                                                       ldo, colscale, colbias, accumulate, M, N, K, mb);
    }
  } else {
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    tlc_launch(gemm_tiled_kernel<TA, TW, TO>, dim3(grid), dim3(256), 0, stream, (const TA*)a, lda, (const TW*)w, ldw, (TO*)out, ldo,
                                                            colscale, colbias, accumulate, M, N, K);
  }
  TLC_CHECK_LAUNCH("linear(simt)");
  return 0;
}

extern "C" int tlc_linear_simt(const void* a, int a_dtype, int lda, const void* w, int w_dtype, int ldw, void* out,
                               int out_dtype, int ldo, const float* colscale, const float* colbias, int accumulate,
                               int M, int N, int K, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  TLC_REQUIRE(K > 0 && lda >= K && ldw >= K && ldo >= N, "linear: bad sizes M=%d N=%d K=%d lda=%d ldw=%d ldo=%d", M, N, K,
              lda, ldw, ldo);
  TLC_DISPATCH_DTYPE(a_dtype, TA, TLC_DISPATCH_DTYPE(w_dtype, TW, TLC_DISPATCH_DTYPE(out_dtype, TO,
      return (launch_simt<TA, TW, TO>(a, lda, w, ldw, out, ldo, colscale, colbias, accumulate, M, N, K, stream)))));
  return 0;
}

// ---- few rows, bfloat16, tensor cores as the reducer ----------------------------------------
// A decode step multiplies up to a few dozen rows by every weight matrix; the time is the time
// to stream the weights once.  One block owns 16 output columns (= 16 weight rows); its four
// warps take interleaved 32-wide slices of K.  Each lane reads 16 contiguous bytes of two
// weight rows (g, g+8) and of one activation row per group of 8 rows, and feeds them to
// mma.sync.m16n8k16 with the weight rows as the M side and the activation rows as the N side.
// The contraction index is permuted the same way on both sides (a lane's 8 contiguous values
// serve two instructions), which a dot product does not notice.  Accumulators stay in
// registers; the four warps' partial sums meet in shared memory.
template <int MG> struct SkinnyAcc { float d[MG][2][4]; };

__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                               uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// A sum on its way out: scaled, with its bias, added to what is there.  The products that fuse into a sum are named, so that
// every kernel of this file that makes a value rounds it alike.
__device__ __forceinline__ float skinny_scaled(float v, int n, const float* __restrict__ colscale, const float* __restrict__ colbias) {
  if (colbias) return colscale ? fmaf(v, colscale[n], colbias[n]) : v + colbias[n];
  return colscale ? v * colscale[n] : v;
}
template <typename TO>
__device__ __forceinline__ void skinny_store(float v, int n, TO* o, const float* __restrict__ colscale, const float* __restrict__ colbias, bool accumulate) {
  if (accumulate && colscale && !colbias) v = fmaf(v, colscale[n], to_f32(*o));
  else {
    v = skinny_scaled(v, n, colscale, colbias);
    if (accumulate) v += to_f32(*o);
  }
  *o = from_f32<TO>(v);
}

constexpr int SK_WARPS = 16;          // warps per block, each with its own slices of K
static int g_skinny_pairs = 1;        // 0: never two blocks a tile (for comparisons)

// With SWIGLU a block's 16 weight rows are 8 gate rows followed by their 8 up rows, and the block
// writes silu(gate) * up for its 8 features (out is [M, N/2]).
//
// With PAIR two blocks of a cluster share a tile of 16 columns, each with one half of K: a matrix with few
// rows (N / 16 tiles for 148 SMs that hold two blocks each) and a long K otherwise needs several trips to
// memory on half of the SMs' load slots.  The second block leaves its sums in the first block's shared memory
// (distributed shared memory); the first adds them to its own, always in this order, and stores.
template <typename TO, int MG, int U, bool SWIGLU, bool PAIR>
__global__ void __launch_bounds__(SK_WARPS * 32, ((MG == 1 && U <= 4) || (MG == 2 && U <= 2) || (MG == 4 && U == 1)) ? 2 : 1)
gemm_skinny_mma_kernel(const __nv_bfloat16* __restrict__ a, int lda, const __nv_bfloat16* __restrict__ w, int ldw,
                       TO* __restrict__ out, int ldo, const float* __restrict__ colscale,
                       const float* __restrict__ colbias, TlcEpi accumulate, int M, int N, int K) {
  static_assert(!(PAIR && SWIGLU), "the paired form has no SwiGLU epilogue");
  // The weights do not depend on the previous kernel of the stream, the activations do: when this
  // kernel is launched early (programmatic dependent launch), the first round of weight loads is
  // in flight while the previous kernel is still finishing; only then does it wait for it.
  asm volatile("griddepcontrol.launch_dependents;");
  __shared__ float red[SK_WARPS][MG < 4 ? MG : 4][32][4];
  __shared__ float other[PAIR ? MG * 128 : 1];                       // the second block's sums, by output value
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int rank = PAIR ? (int)(blockIdx.x & 1) : 0;                 // clusters are pairs of consecutive blocks
  const int n0 = (PAIR ? blockIdx.x >> 1 : blockIdx.x) * 16;
  const int r0 = min(n0 + g, N - 1), r1 = min(n0 + g + 8, N - 1);     // clamped rows are never stored
  const uint4* w0 = reinterpret_cast<const uint4*>(w + (size_t)r0 * ldw);
  const uint4* w1 = reinterpret_cast<const uint4*>(w + (size_t)r1 * ldw);
  float acc[MG][4];
#pragma unroll
  for (int i = 0; i < MG; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
  const int K8 = K >> 3;                                             // 16-byte chunks per row
  const int all_steps = (K8 + 3) >> 2;                               // a step is 4 chunks = 32 values of K
  const int half_steps = (all_steps + 1) >> 1;
  const int s_first = PAIR ? rank * half_steps : 0;                  // this block's steps
  const int n_steps = PAIR ? min(all_steps, s_first + half_steps) : all_steps;
  // all of a warp's loads of one round are issued before the first multiply: one trip to memory
  for (int s0 = s_first + warp * U; s0 < n_steps; s0 += SK_WARPS * U) {
    uint4 wa[U], wb[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int c = (s0 + u) * 4 + t;
      const bool in = (s0 + u) < n_steps && c < K8;
      wa[u] = in ? __ldg(w0 + c) : make_uint4(0, 0, 0, 0);
      wb[u] = in ? __ldg(w1 + c) : make_uint4(0, 0, 0, 0);
    }
    if (s0 == s_first + warp * U) tlc_wait(a, out);                            // first round only
    // the activations of every row group, too, before the first multiply
    uint4 xq[MG][U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int c = (s0 + u) * 4 + t;
      const bool in = (s0 + u) < n_steps && c < K8;
#pragma unroll
      for (int mg = 0; mg < MG; mg++) {
        const int row = mg * 8 + g;
        xq[mg][u] = (in && row < M) ? *(reinterpret_cast<const uint4*>(a + (size_t)row * lda) + c) : make_uint4(0, 0, 0, 0);
      }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
#pragma unroll
      for (int mg = 0; mg < MG; mg++) {
        mma_bf16_16816(acc[mg], wa[u].x, wb[u].x, wa[u].y, wb[u].y, xq[mg][u].x, xq[mg][u].y);
        mma_bf16_16816(acc[mg], wa[u].z, wb[u].z, wa[u].w, wb[u].w, xq[mg][u].z, xq[mg][u].w);
      }
    }
  }
  if (s_first + warp * U >= n_steps) tlc_wait(a, out);                         // warps without a round of their own
  // the warps' partial sums meet in shared memory, at most four row groups at a time
  constexpr int RG = MG < 4 ? MG : 4;
#pragma unroll 1
  for (int g0 = 0; g0 < MG; g0 += RG) {
    if (g0 > 0) __syncthreads();
#pragma unroll
    for (int mg = 0; mg < MG; mg++)
      if (mg >= g0 && mg < g0 + RG)
#pragma unroll
        for (int j = 0; j < 4; j++) red[warp][mg - g0][lane][j] = acc[mg][j];
    __syncthreads();
    if (SWIGLU) {
      // one thread per output value: gate (rows 0..7 of the tile) and up (rows 8..15) of one feature and row
      for (int idx = threadIdx.x; idx < RG * 64; idx += blockDim.x) {
        const int mg = idx >> 6, ln = (idx & 63) >> 1, j = idx & 1;
        float vg = 0.f, vu = 0.f;
#pragma unroll
        for (int ww = 0; ww < SK_WARPS; ww++) { vg += red[ww][mg][ln][j]; vu += red[ww][mg][ln][j + 2]; }
        const int ng = n0 + (ln >> 2), nu = ng + 8;
        const int m = (g0 + mg) * 8 + 2 * (ln & 3) + j;
        if (nu < N && m < M) {
          vg = skinny_scaled(vg, ng, colscale, colbias);
          vu = skinny_scaled(vu, nu, colscale, colbias);
          out[(size_t)m * ldo + (n0 >> 1) + (ln >> 2)] = from_f32<TO>(glu_epilogue<false>(accumulate, vg, vu));   // (the activation's code)
        }
      }
      continue;
    }
    // one thread per output value: sum the warps' partial sums in warp order, epilogue, store
    if constexpr (PAIR) {
      if (rank == 1) {
        for (int idx = threadIdx.x; idx < RG * 128; idx += blockDim.x) {
          const int mg = idx >> 7, ln = (idx & 127) >> 2, j = idx & 3;
          float v = 0.f;
#pragma unroll
          for (int ww = 0; ww < SK_WARPS; ww++) v += red[ww][mg][ln][j];
          uint32_t dst;                                              // the same word of block 0's `other`
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"((uint32_t)__cvta_generic_to_shared(&other[g0 * 128 + idx])), "r"(0));
          asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst), "f"(v) : "memory");
        }
      }
      asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
      if (rank == 1) continue;
    }
    for (int idx = threadIdx.x; idx < RG * 128; idx += blockDim.x) {
      const int mg = idx >> 7, ln = (idx & 127) >> 2, j = idx & 3;
      float v = 0.f;
#pragma unroll
      for (int ww = 0; ww < SK_WARPS; ww++) v += red[ww][mg][ln][j];
      if constexpr (PAIR) v += other[g0 * 128 + idx];
      const int n = n0 + (ln >> 2) + (j >= 2 ? 8 : 0);
      const int m = (g0 + mg) * 8 + 2 * (ln & 3) + (j & 1);
      if (n < N && m < M) {
        skinny_store(v, n, out + (size_t)m * ldo + n, colscale, colbias, accumulate);
      }
    }
  }
}

// Up to 8 rows, K of one round, and more tiles than the SMs hold blocks but not more than twice as many: two tiles of 16 columns a
// block, so that all of the matrix is on its way before the wait on the previous kernel.  (With a tile a block, the blocks past
// the first two of an SM ask for their weights when others have gone through the wait, the products and the sums: the
// 33.7 MB of 2048 -> 8240 took 7.6 us behind the wait where the two narrow products of a layer, all of whose blocks are resident
// at once, take 4.4.)  The second tile's weights come by cp.async into shared memory, every thread its own pieces, and take
// neither registers nor lines of the first-level cache while they travel, which is what bounds the first tile's; the sums
// are those of a tile a block, in the same order.  A captured step of the 1.5B sizes, contexts of up to 512, microseconds,
// a tile a block and two: batch 1 925 and 855, 2 941 and 880, 4 998 and 931, 8 1186 and 1105.
template <typename TO, bool SWIGLU>
__global__ void __launch_bounds__(SK_WARPS * 32, 2)
gemm_skinny_two_kernel(const __nv_bfloat16* __restrict__ a, int lda, const __nv_bfloat16* __restrict__ w, int ldw,
                       TO* __restrict__ out, int ldo, const float* __restrict__ colscale, const float* __restrict__ colbias,
                       TlcEpi accumulate, int M, int N, int K) {
  asm volatile("griddepcontrol.launch_dependents;");
  constexpr int U = 4, NT = SK_WARPS * 32;
  extern __shared__ __align__(16) uint4 second[];                    // [U][2][NT]
  __shared__ float red[2][SK_WARPS][32][4];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int K8 = K >> 3, n_steps = (K8 + 3) >> 2;
  const int tiles[2] = {(int)blockIdx.x * 16, (int)(blockIdx.x + gridDim.x) * 16};
  const bool two = tiles[1] < N;
  const uint4* rows[2][2];
#pragma unroll
  for (int i = 0; i < 2; i++) {
    rows[i][0] = reinterpret_cast<const uint4*>(w + (size_t)min(tiles[i] + g, N - 1) * ldw);         // clamped rows are never stored
    rows[i][1] = reinterpret_cast<const uint4*>(w + (size_t)min(tiles[i] + g + 8, N - 1) * ldw);
  }
  if (two) {
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int c = (warp * U + u) * 4 + t;
      const bool in = warp * U + u < n_steps && c < K8;
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const unsigned dst = (unsigned)__cvta_generic_to_shared(second + (u * 2 + r) * NT + threadIdx.x);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(rows[1][r] + (in ? c : 0)), "r"(in ? 16 : 0) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  uint4 wv[U][2];
#pragma unroll
  for (int u = 0; u < U; u++) {
    const int c = (warp * U + u) * 4 + t;
    const bool in = warp * U + u < n_steps && c < K8;
#pragma unroll
    for (int r = 0; r < 2; r++) wv[u][r] = in ? __ldg(rows[0][r] + c) : make_uint4(0, 0, 0, 0);
  }
  tlc_wait(a, out);
  uint4 xq[U];
#pragma unroll
  for (int u = 0; u < U; u++) {
    const int c = (warp * U + u) * 4 + t;
    const bool in = warp * U + u < n_steps && c < K8;
    xq[u] = (in && g < M) ? *(reinterpret_cast<const uint4*>(a + (size_t)g * lda) + c) : make_uint4(0, 0, 0, 0);
  }
#pragma unroll
  for (int i = 0; i < 2; i++) {
    if (i == 1) {
      if (!two) break;
      asm volatile("cp.async.wait_all;" ::: "memory");               // (a thread reads its own pieces alone)
    }
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int u = 0; u < U; u++) {
      const uint4 p = i == 0 ? wv[u][0] : second[(u * 2) * NT + threadIdx.x], q = i == 0 ? wv[u][1] : second[(u * 2 + 1) * NT + threadIdx.x];
      mma_bf16_16816(acc, p.x, q.x, p.y, q.y, xq[u].x, xq[u].y);
      mma_bf16_16816(acc, p.z, q.z, p.w, q.w, xq[u].z, xq[u].w);
    }
#pragma unroll
    for (int j = 0; j < 4; j++) red[i][warp][lane][j] = acc[j];
  }
  __syncthreads();
  // one thread per output value: the warps' sums in their order, epilogue, store
  constexpr int PER = SWIGLU ? 64 : 128;
  if ((int)threadIdx.x < (two ? 2 : 1) * PER) {
    const int i = (int)threadIdx.x / PER, idx = (int)threadIdx.x % PER, n0 = i ? tiles[1] : tiles[0];
    if (SWIGLU) {
      const int ln = idx >> 1, j = idx & 1;
      float vg = 0.f, vu = 0.f;
#pragma unroll
      for (int ww = 0; ww < SK_WARPS; ww++) { vg += red[i][ww][ln][j]; vu += red[i][ww][ln][j + 2]; }
      const int ng = n0 + (ln >> 2), nu = ng + 8, m = 2 * (ln & 3) + j;
      if (nu < N && m < M) {
        vg = skinny_scaled(vg, ng, colscale, colbias);
        vu = skinny_scaled(vu, nu, colscale, colbias);
        out[(size_t)m * ldo + (n0 >> 1) + (ln >> 2)] = from_f32<TO>(glu_epilogue<false>(accumulate, vg, vu));   // (the activation's code)
      }
    } else {
      const int ln = idx >> 2, j = idx & 3;
      float v = 0.f;
#pragma unroll
      for (int ww = 0; ww < SK_WARPS; ww++) v += red[i][ww][ln][j];
      const int n = n0 + (ln >> 2) + (j >= 2 ? 8 : 0), m = 2 * (ln & 3) + (j & 1);
      if (n < N && m < M) {
        skinny_store(v, n, out + (size_t)m * ldo + n, colscale, colbias, accumulate);
      }
    }
  }
}
// 17 to 32 rows: the same sums on another division of the work.  The kernel above holds a round of weights and activations in
// registers, which leaves one block of 17 and more rows an SM and 64 KB on their way (32 rows, 12288 -> 3072: 75 MB in 33 us).
// Here a block is four of the 16 warps' shares of K of two tiles of 16 columns, and the blocks of a cluster of four are the 16: a
// warp's weights and activations come by cp.async into a ring of its own, every thread its own pieces, so that nothing but
// the copies' arrival holds a warp up, and an activation serves two tiles.  The 16 shares are added in their order by
// the block whose values they are, read from the others' shared memory: the bits of the kernel above.
struct RingSmem {
  static constexpr int MG = 4, U = 4;                                // groups of 8 rows; steps of a share in a round, as above
  static constexpr int TILES = 2, WARPS = 4;
  static constexpr int D = 4;                                        // steps of a warp on their way
  static constexpr int STAGE = (2 * TILES + MG) * 32;                // 16-byte pieces of a step: two rows a tile, MG groups of activation rows
  static constexpr int SUMS = TILES * MG * 128;                      // a warp's sums (floats), in its ring when it is through
  static constexpr int BYTES = WARPS * D * STAGE * 16;
  static_assert(SUMS * 4 <= D * STAGE * 16, "the sums reuse the ring");
};
template <typename TO>
__global__ void __launch_bounds__(128, 3)
gemm_skinny_ring_kernel(const __nv_bfloat16* __restrict__ a, int lda, const __nv_bfloat16* __restrict__ w, int ldw,
                        TO* __restrict__ out, int ldo, const float* __restrict__ colscale, const float* __restrict__ colbias,
                        TlcEpi accumulate, int M, int N, int K) {
  asm volatile("griddepcontrol.launch_dependents;");
  using S = RingSmem;
  constexpr int D = S::D, MG = S::MG, U = S::U;
  extern __shared__ __align__(16) uint4 ring_sm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int rank = (int)(blockIdx.x & 3), n0 = (int)(blockIdx.x >> 2) * 32;    // clusters are runs of four blocks
  const int share = rank * 4 + warp;                                 // which of the 16 shares of K
  const int K8 = K >> 3, n_steps = (K8 + 3) >> 2;
  uint4* ring = ring_sm + warp * D * S::STAGE + lane;
  const uint4* wr[2 * S::TILES];
#pragma unroll
  for (int i = 0; i < 2 * S::TILES; i++) wr[i] = reinterpret_cast<const uint4*>(w + (size_t)min(n0 + 8 * i + g, N - 1) * ldw);   // clamped rows are never stored
  // step i of this share; past its end the copies bring zeros to nobody
  auto chunk_of = [&](int i) { return ((i / U) * SK_WARPS * U + share * U + i % U) * 4 + t; };
  auto copy = [&](uint4* dst, const uint4* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
  };
  auto fetch_w = [&](int i) {
    const int c = chunk_of(i);
    const bool in = c < K8;
#pragma unroll
    for (int q = 0; q < 2 * S::TILES; q++) copy(ring + (i % D) * S::STAGE + q * 32, wr[q] + (in ? c : 0), in);
  };
  auto fetch_x = [&](int i) {
    const int c = chunk_of(i);
#pragma unroll
    for (int mg = 0; mg < MG; mg++) {
      const int row = mg * 8 + g;
      const bool in = c < K8 && row < M;
      copy(ring + (i % D) * S::STAGE + (2 * S::TILES + mg) * 32, reinterpret_cast<const uint4*>(a + (size_t)(in ? row : 0) * lda) + (in ? c : 0), in);
    }
  };
  const int rounds = (n_steps + SK_WARPS * U - 1) / (SK_WARPS * U), last = n_steps - (rounds - 1) * SK_WARPS * U - share * U;
  const int mine = (rounds - 1) * U + min(max(last, 0), U);          // this share's steps
#pragma unroll
  for (int i = 0; i < D; i++) if (i < mine) fetch_w(i);
  tlc_wait(a, out);
#pragma unroll
  for (int i = 0; i < D; i++) {
    if (i < mine) fetch_x(i);
    asm volatile("cp.async.commit_group;" ::: "memory");             // (the weights of all of them go with the first)
  }
  float acc[S::TILES][MG][4];
#pragma unroll
  for (int i = 0; i < S::TILES; i++)
#pragma unroll
    for (int mg = 0; mg < MG; mg++)
#pragma unroll
      for (int j = 0; j < 4; j++) acc[i][mg][j] = 0.f;
#pragma unroll 1
  for (int i = 0; i < mine; i++) {
    asm volatile("cp.async.wait_group %0;" ::"n"(D - 1) : "memory"); // (a thread reads its own pieces alone)
    const uint4* st = ring + (i % D) * S::STAGE;
    uint4 wv[2 * S::TILES];
#pragma unroll
    for (int q = 0; q < 2 * S::TILES; q++) wv[q] = st[q * 32];
#pragma unroll
    for (int mg = 0; mg < MG; mg++) {
      const uint4 x = st[(2 * S::TILES + mg) * 32];
#pragma unroll
      for (int q = 0; q < S::TILES; q++) {
        mma_bf16_16816(acc[q][mg], wv[2 * q].x, wv[2 * q + 1].x, wv[2 * q].y, wv[2 * q + 1].y, x.x, x.y);
        mma_bf16_16816(acc[q][mg], wv[2 * q].z, wv[2 * q + 1].z, wv[2 * q].w, wv[2 * q + 1].w, x.z, x.w);
      }
    }
    if (i + D < mine) { fetch_w(i + D); fetch_x(i + D); }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
  float* sums = reinterpret_cast<float*>(ring_sm + warp * D * S::STAGE);   // [tile][mg][lane][4]
#pragma unroll
  for (int q = 0; q < S::TILES; q++)
#pragma unroll
    for (int mg = 0; mg < MG; mg++)
      *reinterpret_cast<float4*>(sums + ((q * MG + mg) * 32 + lane) * 4) = make_float4(acc[q][mg][0], acc[q][mg][1], acc[q][mg][2], acc[q][mg][3]);
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  const float* from[4];
#pragma unroll
  for (int r = 0; r < 4; r++) {
    unsigned long long at;                                           // the same word in the block of rank r, for ordinary loads
    asm("mapa.u64 %0, %1, %2;" : "=l"(at) : "l"((unsigned long long)(uintptr_t)ring_sm), "r"(r));
    from[r] = reinterpret_cast<const float*>((uintptr_t)at);
  }
  // this block's quarter of the values
  for (int idx = rank * (S::SUMS / 4) + threadIdx.x; idx < (rank + 1) * (S::SUMS / 4); idx += 128) {
    const int j = idx & 3, ln = (idx >> 2) & 31, qm = idx >> 7;
    float part[SK_WARPS];
#pragma unroll
    for (int ww = 0; ww < SK_WARPS; ww++) part[ww] = from[ww >> 2][(ww & 3) * D * S::STAGE * 4 + idx];
    float v = 0.f;
#pragma unroll
    for (int ww = 0; ww < SK_WARPS; ww++) v += part[ww];
    const int n = n0 + 16 * (qm / MG) + (ln >> 2) + (j >= 2 ? 8 : 0), m = qm % MG * 8 + 2 * (ln & 3) + (j & 1);
    if (n < N && m < M) {
      skinny_store(v, n, out + (size_t)m * ldo + n, colscale, colbias, accumulate);
    }
  }
  // no block leaves while another may still read its sums
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
static int g_skinny_ring = 1;         // 0: never that division of the work (for comparisons)

// The launch of gemm_skinny_ring_kernel for `tiles` tiles of 16 columns; how many of its clusters the GPU runs at once.
static cudaLaunchConfig_t ring_config(unsigned tiles, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((tiles + 1) / 2 * 4);
  cfg.blockDim = dim3(128);
  cfg.dynamicSmemBytes = RingSmem::BYTES;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 4;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = g_tlc_pdl ? 2 : 1;
  return cfg;
}
template <typename TO> static int ring_clusters() {
  static int n = -1;
  if (n < 0) {
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = ring_config(2, attr);
    cfg.numAttrs = 1;
    int got = 0;
    n = cudaOccupancyMaxActiveClusters(&got, gemm_skinny_ring_kernel<TO>, &cfg) == cudaSuccess ? got : 0;
    if (n == 0) cudaGetLastError();
  }
  return n;
}
// Whether an output of N columns is among those that the ring serves (where the rule's sides are measured: launch_skinny_mg).
extern "C" int tlc_linear_skinny_ring_takes(int N, int K, int sms, int clusters) {
  const int tiles = (N + 15) / 16, n_steps = ((K >> 3) + 3) >> 2;
  return tiles > sms && n_steps >= 128 && ((tiles + 1) / 2 <= clusters || (n_steps >= 256 && tiles <= sms * 3 / 2));
}

constexpr int SK_TWO_SMEM = 4 * 2 * SK_WARPS * 32 * (int)sizeof(uint4);
static int g_skinny_two = 1;          // 0: never two tiles a block (for comparisons)
// Whether two tiles a block serve an output of N columns: more tiles than the SMs hold blocks of one (two an SM), K of one round.
// With the activation the second tile's share has to be a little larger, the more the longer K is (a tile a block, two; 1 / 8 rows):
// 1280 -> 4752 4.07 / 4.17 and 4.14 / 4.53, -> 5600 4.71 / 4.71 and 4.41 / 4.70; 1800 -> 4752 5.01 / 5.65 and 5.55 / 6.29, -> 5600
// 5.64 / 6.24 and 5.91 / 6.60, -> 6400 6.29 / 6.80 and 6.14 / 6.66; 2048 -> 5600 5.61 / 6.11 and 5.72 / 6.17, -> 6400 6.51 / 6.45 and 5.97 /
// 6.35, -> 8192 7.47 / 7.65 and 6.55 / 6.91; without it 2048 -> 4752 5.49 / 5.91 and 5.25 / 5.71, 1032 -> 9472 5.48 / 5.94 and 4.71 / 5.19.
extern "C" int tlc_linear_skinny_two_takes(int N, int K, int activation, int sms) {
  const int tiles = (N + 15) / 16, n_steps = ((K >> 3) + 3) >> 2;
  const int from = 2 * sms + (activation ? (n_steps - 33) * sms / 64 : 0);
  return n_steps > SK_WARPS * 2 && n_steps <= SK_WARPS * 4 && tiles > from && tiles <= 4 * sms;
}

// Kernels that ask for more than 48 KB of shared memory: once a device, ahead of any stream capture where the library is set up
// first (tlc_linear_init), else with the first product that takes one of them.
template <typename TO> static bool simt_reserve() {
  const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
  return cudaFuncSetAttribute(gemm_tiled_f32x4_kernel<TO, 4, 4>, attr, ft_smem(4, 4)) == cudaSuccess &&
         cudaFuncSetAttribute(gemm_split_f32x4_kernel<TO, 8, 4, 8>, attr, fs_smem<8, 4, 8>(2)) == cudaSuccess &&
         cudaFuncSetAttribute(gemm_skinny_ring_kernel<TO>, attr, RingSmem::BYTES) == cudaSuccess &&
         cudaFuncSetAttribute(gemm_skinny_two_kernel<TO, false>, attr, SK_TWO_SMEM) == cudaSuccess &&
         cudaFuncSetAttribute(gemm_skinny_two_kernel<TO, true>, attr, SK_TWO_SMEM) == cudaSuccess;
}
int tlc_linear_simt_init() {
  static bool ready[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && ready[dev]) return 0;
  if (!simt_reserve<float>() || !simt_reserve<__nv_bfloat16>()) return tlc_fail(-2, "linear: cannot reserve %d bytes of shared memory", ft_smem(4, 4));
  if (dev >= 0 && dev < 64) ready[dev] = true;
  return 0;
}

template <typename TO, int MG, bool SWIGLU>
static void launch_skinny_mg(const __nv_bfloat16* a, int lda, const __nv_bfloat16* w, int ldw, TO* out, int ldo,
                             const float* colscale, const float* colbias, TlcEpi accumulate, int M, int N, int K,
                             cudaStream_t stream) {
  const unsigned blocks = (unsigned)((N + 15) / 16);
  const int n_steps = ((K >> 3) + 3) >> 2;
  if constexpr (!SWIGLU) {
    // few tiles and more than one round of K: two blocks a tile, each with half of K
    static int sms = 0;
    if (sms == 0) { int dev = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev); }
    const int per_round = SK_WARPS * (MG == 2 ? 2 : 4);
    if (g_skinny_pairs && MG <= 2 && (int)blocks <= sms && n_steps > per_round) {     // MG <= 2: two blocks fit on an SM
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(2 * blocks);
      cfg.blockDim = dim3(SK_WARPS * 32);
      cfg.stream = stream;
      cudaLaunchAttribute attr[2];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = 2;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[1].val.programmaticStreamSerializationAllowed = 1;
      cfg.attrs = attr;
      cfg.numAttrs = g_tlc_pdl ? 2 : 1;
      const int half = (n_steps + 1) / 2;
      if (half <= SK_WARPS * 2 || MG == 2)
        cudaLaunchKernelEx(&cfg, gemm_skinny_mma_kernel<TO, MG, 2, false, true>, a, lda, w, ldw, out, ldo, colscale, colbias, accumulate, M, N, K);
      else
        cudaLaunchKernelEx(&cfg, gemm_skinny_mma_kernel<TO, MG, 4, false, true>, a, lda, w, ldw, out, ldo, colscale, colbias, accumulate, M, N, K);
      return;
    }
  }
  if constexpr (MG == 1) {
    static int sms = 0;
    if (sms == 0) { int dev = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev); }
    if (g_skinny_two && tlc_linear_skinny_two_takes(N, K, SWIGLU, sms) && tlc_linear_simt_init() == 0) {
      tlc_launch(gemm_skinny_two_kernel<TO, SWIGLU>, dim3((blocks + 1) / 2), dim3(SK_WARPS * 32), SK_TWO_SMEM, stream, a, lda, w, ldw, out, ldo, colscale,
                 colbias, accumulate, M, N, K);
      return;
    }
  }
  if constexpr (MG == 4 && !SWIGLU) {
    // Narrow outputs of a long K.  Microseconds, the kernel below and the ring: 17 / 32 rows of 5376 -> 2560 16.2 / 17.8 and 11.5 /
    // 12.0, 8192 -> 2560 21.1 / 23.2 and 14.0 / 14.6, 4608 -> 3072 15.8 / 17.4 and 11.6 / 12.0, 12288 -> 3072 30.2 / 32.7 and 19.6 /
    // 21.1, but 4096 -> 2048 (128 tiles) 7.3 / 7.9 and 9.0 / 9.2.  A captured step of the 3B sizes at batch 24 4057 and 3610, of the 7B
    // sizes at batch 32 7041 and 5970.  (9 to 16 rows gained up to a tenth alone and lost in a step, beside kernels that want
    // another split of the SM's memory: 3B at batch 16 3253 and 3728.)  It pays while all clusters are resident at once, 104
    // here (208 tiles): 4096 -> 3328 13.7 / 15.1 and 10.2 / 10.7, 4096 -> 3360 13.7 / 15.1 and 14.8 / 15.4, 4096 -> 4064 14.1 /
    // 15.4 and 16.3 / 17.8, 5384 -> 3552 19.2 / 22.1 and 21.6 / 24.4; from K = 8192 on up to 222 tiles: 8192 -> 3360 22.7 / 24.7 and 21.8 /
    // 23.0, 12288 -> 3552 31.6 / 34.3 and 30.4 / 32.7, but 8192 -> 4064 23.5 / 25.5 and 24.7 / 25.2.  (Outputs of 4,096 and more
    // are another kernel's.)
    static int sms = 0;
    if (sms == 0) { int dev = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev); }
    if (g_skinny_ring && (int)blocks > sms && n_steps >= 128 && tlc_linear_simt_init() == 0 && tlc_linear_skinny_ring_takes(N, K, sms, ring_clusters<TO>())) {
      cudaLaunchAttribute attr[2];
      cudaLaunchConfig_t cfg = ring_config(blocks, attr);
      cfg.stream = stream;
      cudaLaunchKernelEx(&cfg, gemm_skinny_ring_kernel<TO>, a, lda, w, ldw, out, ldo, colscale, colbias, accumulate, M, N, K);
      return;
    }
  }
  // U steps per warp and round: with one row group and U <= 4, or two and U = 2, two blocks fit on an SM
  // (a warp holds the weights and the activations of a round in registers)
  if (MG == 4 && blocks > 296)      // 17..32 rows, many row tiles: one step a round keeps two blocks on an SM
    tlc_launch(gemm_skinny_mma_kernel<TO, MG, 1, SWIGLU, false>, dim3(blocks), dim3(SK_WARPS * 32), 0, stream, a, lda, w, ldw, out, ldo, colscale, colbias, accumulate, M, N, K);
  else if (n_steps <= SK_WARPS * 2 || MG == 2)
    tlc_launch(gemm_skinny_mma_kernel<TO, MG, 2, SWIGLU, false>, dim3(blocks), dim3(SK_WARPS * 32), 0, stream, a, lda, w, ldw, out, ldo, colscale, colbias, accumulate, M, N, K);
  else
    tlc_launch(gemm_skinny_mma_kernel<TO, MG, 4, SWIGLU, false>, dim3(blocks), dim3(SK_WARPS * 32), 0, stream, a, lda, w, ldw, out, ldo, colscale, colbias, accumulate, M, N, K);
}

template <typename TO, bool SWIGLU>
static int launch_skinny_mma(const void* a, int lda, const void* w, int ldw, void* out, int ldo, const float* colscale,
                             const float* colbias, TlcEpi accumulate, int M, int N, int K, cudaStream_t stream) {
  const __nv_bfloat16* ap = (const __nv_bfloat16*)a;
  const __nv_bfloat16* wp = (const __nv_bfloat16*)w;
  if (M <= 8) launch_skinny_mg<TO, 1, SWIGLU>(ap, lda, wp, ldw, (TO*)out, ldo, colscale, colbias, accumulate, M, N, K, stream);
  else if (M <= 16) launch_skinny_mg<TO, 2, SWIGLU>(ap, lda, wp, ldw, (TO*)out, ldo, colscale, colbias, accumulate, M, N, K, stream);
  else if (M <= 32) launch_skinny_mg<TO, 4, SWIGLU>(ap, lda, wp, ldw, (TO*)out, ldo, colscale, colbias, accumulate, M, N, K, stream);
  else launch_skinny_mg<TO, 8, SWIGLU>(ap, lda, wp, ldw, (TO*)out, ldo, colscale, colbias, accumulate, M, N, K, stream);
  TLC_CHECK_LAUNCH("linear(skinny mma)");
  return 0;
}

// bfloat16 operands with 16-byte aligned rows and at most 64 rows: the weight-streaming kernel.
extern "C" int tlc_linear_skinny_ok(int a_dtype, int lda, const void* a, int w_dtype, int ldw, const void* w, int M, int K) {
  return a_dtype == TLC_BF16 && w_dtype == TLC_BF16 && M <= 64 && K % 8 == 0 && lda % 8 == 0 && ldw % 8 == 0 &&
         ((uintptr_t)a % 16 == 0) && ((uintptr_t)w % 16 == 0);
}

extern "C" int tlc_linear_skinny(const void* a, int lda, const void* w, int ldw, void* out, int out_dtype, int ldo,
                                 const float* colscale, const float* colbias, int accumulate, int M, int N, int K,
                                 cudaStream_t stream) {
  if (out_dtype == TLC_F32)
    return launch_skinny_mma<float, false>(a, lda, w, ldw, out, ldo, colscale, colbias, accumulate, M, N, K, stream);
  if (out_dtype == TLC_BF16)
    return launch_skinny_mma<__nv_bfloat16, false>(a, lda, w, ldw, out, ldo, colscale, colbias, accumulate, M, N, K, stream);
  return tlc_fail(-1, "linear: unknown output dtype %d", out_dtype);
}

extern "C" void tlc_linear_skinny_pairs(int on) { g_skinny_pairs = on; }
extern "C" void tlc_linear_skinny_two(int on) { g_skinny_two = on; }
extern "C" void tlc_linear_skinny_ring(int on) { g_skinny_ring = on; }

extern "C" int tlc_linear_skinny_swiglu(const void* a, int lda, const void* w, int ldw, void* out, int out_dtype, int ldo,
                                        const float* colscale, const float* colbias, int M, int N, int K, int act_code,
                                        float limit, float alpha, cudaStream_t stream) {
  const TlcEpi act(act_code, limit, alpha);
  if (out_dtype == TLC_F32)
    return launch_skinny_mma<float, true>(a, lda, w, ldw, out, ldo, colscale, colbias, act, M, N, K, stream);
  if (out_dtype == TLC_BF16)
    return launch_skinny_mma<__nv_bfloat16, true>(a, lda, w, ldw, out, ldo, colscale, colbias, act, M, N, K, stream);
  return tlc_fail(-1, "linear: unknown output dtype %d", out_dtype);
}
