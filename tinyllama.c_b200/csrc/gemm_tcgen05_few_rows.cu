// bfloat16 linear layer for up to 128 rows (decode steps of that many sequences, short prompts) on the 5th-generation tensor cores,
// with the WEIGHTS on the M side of tcgen05.mma:  out[M, N] (+)= (A[M, K] @ W[N, K]^T) * colscale + colbias.
//
// With so few rows the time is the time to stream the weights once.  The product for prompts puts the activations
// on the 128-row side and pads them, and has too few tiles for the GPU where N is small; the weight-streaming
// mma.sync kernel of the smallest batches re-reads the activations for every 16 output columns.  Here a tile is
// 128 weight rows x 16, 32, 64 or 128 activation rows: D[n, m] = sum_k W[n, k] A[m, k], an accumulator of 128 lanes x NB
// columns of tensor memory.  Weight tiles [128, 64] and activation tiles [NB, 64] arrive by TMA (128-byte
// swizzle, rows past the matrices read as zero) in a ring of shared-memory stages; one thread issues the
// products; four warps take the result out of tensor memory, a thread per weight row.
//
// N / 128 tiles do not fill 148 SMs (65 for N = 8240, 16 for N = 2048), so the K-steps of a tile are shared
// among the up to 8 blocks of a thread-block CLUSTER: every block leaves its partial sums [NB, 128] in its own
// shared memory, the cluster meets at a barrier, and block r adds up its share of the rows of all blocks' sums,
// read through distributed shared memory in the order of the ranks (so the result does not depend on
// timing), applies the epilogue and stores: a warp a row, a lane four weight rows in 16-byte pieces (a thread a weight
// row instead, with 4-byte reads: 64 rows of 2048 -> 8240 11.5 us, so 10.8).  What the sums are added to is asked for while the
// products run.  A second barrier keeps every block's shared memory alive until all have read it.  A block that has the
// whole of K writes from tensor memory.  With SWIGLU the weight rows come in groups of 16 = 8 gate rows and their
// 8 up rows, and the block writes silu(gate) * up ([M, N / 2]).
//
// What bounds it: the stream of the weights; a copy loop of the same boxes without products takes 26.7 us for 24576 x 3072
// (151 MB), the product of 64 rows 28.7 (34.2 before the 16-byte reads and the unshared tiles' own way out).  Where a block has
// few K-steps, the chain from the wait on the kernel before to the last store (activations, products, the meeting of the
// sums: 3 to 4 us) counts as much as the stream: 64 rows of 4096 -> 2048 added to what is there 8.4 us (10.0), of which the
// 17 MB are 2.6.
//
// Every mbarrier wait is bounded (codes 31-33 of the error word); a block whose wait ran out still goes to both
// cluster barriers, so that no block of its cluster waits for it.
#include "common.cuh"
#include "mbarrier.cuh"
#include "tcgen05.cuh"
#include <algorithm>

namespace {

constexpr int WM = 128;                 // weight rows of a tile
constexpr int FBK = 64;                 // K of a stage
constexpr int FR_THREADS = 192;         // loader warp, issuer warp, four epilogue warps

template <int NB, int STAGES>
struct FrSmem {
  static constexpr int W_BYTES = WM * FBK * 2;
  static constexpr int X_BYTES = NB * FBK * 2;
  static constexpr int TILES = STAGES * (W_BYTES + X_BYTES);
  static constexpr int PART = NB * WM * 4;                  // the block's sums [NB][128], in the stages' memory once the products are done
  static constexpr int N_BARS = 2 * STAGES + 1;             // full, empty per stage; accumulator complete
  static constexpr int TOTAL = TILES + N_BARS * 8 + 16 + 1024;
  static_assert(PART <= TILES, "the partial sums reuse the stages");
};

// The same shared-memory word in the block of another rank of the cluster, as a generic address: loads through
// it are ordinary loads, which the compiler may have many of in flight (a volatile asm load a value made the sum
// a chain of round trips: 10 us for 32 rows of two blocks).
__device__ __forceinline__ const float* in_rank(const float* p, int rank) {
  unsigned long long q;
  asm("mapa.u64 %0, %1, %2;" : "=l"(q) : "l"((unsigned long long)(uintptr_t)p), "r"(rank));
  return reinterpret_cast<const float*>((uintptr_t)q);
}

__device__ __forceinline__ float4 read4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 read4(const __nv_bfloat16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
}
__device__ __forceinline__ void write4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void write4(__nv_bfloat16* p, float4 v) {
  const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
  *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const unsigned*>(&lo), *reinterpret_cast<const unsigned*>(&hi));
}

template <typename TO, int NB, int STAGES, bool SWIGLU>
__global__ void __launch_bounds__(FR_THREADS, 2)
gemm_few_rows_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                     TO* __restrict__ out, int ldo, const float* __restrict__ colscale,
                     const float* __restrict__ colbias, TlcEpi accumulate, int M, int N, int K, int split, ErrWords* err) {
  asm volatile("griddepcontrol.launch_dependents;");
  using S = FrSmem<NB, STAGES>;
  constexpr int CW = NB < 32 ? 16 : 32;                     // columns of tensor memory an epilogue warp reads at a time
  constexpr int TCOLS = NB < 32 ? 32 : NB;                  // (tensor memory comes in 32 columns or more)
  extern __shared__ uint8_t fr_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)fr_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* w_tiles = smem;
  uint8_t* x_tiles = smem + STAGES * S::W_BYTES;
  float* part = reinterpret_cast<float*>(smem);
  uint64_t* bars = (uint64_t*)(smem + S::TILES);
  uint32_t* tmem_slot = (uint32_t*)(bars + S::N_BARS);
  const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + STAGES), acc_full = smem_u32(bars + 2 * STAGES);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long wait_limit = mbar_wait_limit(err);
  const int rank = split > 1 ? (int)cluster_rank() : 0;     // clusters are runs of `split` consecutive blocks
  const int n0 = ((int)blockIdx.x / split) * WM;
  const int num_k = (K + FBK - 1) / FBK, k_per = (num_k + split - 1) / split;
  const int k_begin = min(num_k, rank * k_per), k_end = min(num_k, k_begin + k_per);
  const int n_k = k_end - k_begin;                          // this block's K-steps (the last ranks may have none)

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 1); }
    mbar_init(acc_full, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TCOLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {                                        // ---- TMA loader ----
      // the weights do not depend on the previous kernel of the stream: the first stages' weight tiles are on
      // their way before the wait on it, the activation tiles follow after it
      bool ok = true, waited = false;
      int issued = 0;
      for (int i = 0; i < n_k && ok; i++) {
        const int s = i % STAGES, k = k_begin + i;
        if (i >= STAGES) ok = mbar_wait(empty0 + 8 * s, (uint32_t)(((i - STAGES) / STAGES) & 1), err, 31, wait_limit);
        if (!ok) break;
        if (!waited && i == min(n_k, STAGES) - 1) {
          // last of the first fills: wait, then hand in the activation tiles of all of them
          mbar_expect_tx(full0 + 8 * s, S::W_BYTES + S::X_BYTES);
          tma_load_2d(smem_u32(w_tiles + s * S::W_BYTES), &map_w, full0 + 8 * s, k * FBK, n0);
          asm volatile("griddepcontrol.wait;" ::: "memory");
          waited = true;
          for (int j = 0; j <= i; j++)
            tma_load_2d(smem_u32(x_tiles + (j % STAGES) * S::X_BYTES), &map_x, full0 + 8 * (j % STAGES), (k_begin + j) * FBK, 0);
        } else if (!waited) {
          mbar_expect_tx(full0 + 8 * s, S::W_BYTES + S::X_BYTES);
          tma_load_2d(smem_u32(w_tiles + s * S::W_BYTES), &map_w, full0 + 8 * s, k * FBK, n0);
        } else {
          mbar_expect_tx(full0 + 8 * s, S::W_BYTES + S::X_BYTES);
          tma_load_2d(smem_u32(w_tiles + s * S::W_BYTES), &map_w, full0 + 8 * s, k * FBK, n0);
          tma_load_2d(smem_u32(x_tiles + s * S::X_BYTES), &map_x, full0 + 8 * s, k * FBK, 0);
        }
        issued = i + 1;
      }
      if (!waited) asm volatile("griddepcontrol.wait;" ::: "memory");
      if (!ok || *(volatile int*)&err->flag != 0) {
        // something went wrong: let the copies still in flight land before the block goes on to its end
        for (int i = max(0, issued - STAGES); i < issued; i++)
          mbar_wait(full0 + 8 * (i % STAGES), (uint32_t)((i / STAGES) & 1), err, 34, wait_limit);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {                                        // ---- MMA issuer ----
      constexpr uint32_t idesc = instr_desc(WM, NB);
      bool ok = true;
      for (int i = 0; i < n_k; i++) {
        const int s = i % STAGES;
        ok = mbar_wait(full0 + 8 * s, (uint32_t)((i / STAGES) & 1), err, 32, wait_limit);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t w_addr = smem_u32(w_tiles + s * S::W_BYTES), x_addr = smem_u32(x_tiles + s * S::X_BYTES);
#pragma unroll
        for (int kk = 0; kk < FBK / UMMA_K; kk++)
          umma(tmem, smem_desc(w_addr + kk * UMMA_K * 2), smem_desc(x_addr + kk * UMMA_K * 2), idesc, (i > 0 || kk > 0) ? 1u : 0u);
        umma_commit(empty0 + 8 * s);
      }
      if (ok && n_k > 0) umma_commit(acc_full);
      else if (n_k == 0) mbar_arrive(acc_full);             // nothing to wait for: the epilogue takes zeros
    }
  } else {                                                  // ---- epilogue warps 2..5 ----
    const int quarter = warp & 3;                           // a warp may touch lanes 32 * (warp % 4) .. + 31 only
    const int row = quarter * 32 + lane;                    // weight row of the tile
    asm volatile("griddepcontrol.wait;" ::: "memory");      // `out` may still be read or written by the previous kernel
    auto read_columns = [&](int c, uint32_t (&r)[CW]) {
      __syncwarp();                                         // (the reads want a whole warp; waits, loads and stores by lane lie before them)
      const uint32_t at = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(c * CW);
      if constexpr (CW == 32) tmem_ld32(at, r);
      else tmem_ld16(at, r);
    };
    if (split == 1) {
      // the block has the whole sum: out of tensor memory and straight to the output, a lane a weight row
      const int n = n0 + row;
      const bool n_in = n < N, add = !SWIGLU && accumulate;
      const float cs = (colscale && n_in) ? colscale[n] : 1.0f, cb = (colbias && n_in) ? colbias[n] : 0.0f;
      mbar_wait(acc_full, 0, err, 33, wait_limit);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int c = 0; c < NB / CW; c++) {
        float old[CW];
#pragma unroll
        for (int j = 0; j < CW; j++) old[j] = (add && n_in && c * CW + j < M) ? to_f32(out[(size_t)(c * CW + j) * ldo + n]) : 0.f;
        uint32_t r[CW];
        read_columns(c, r);
#pragma unroll
        for (int j = 0; j < CW; j++) {
          const int m = c * CW + j;
          if (m >= M) break;
          const float v = __uint_as_float(r[j]) * cs + cb;
          if (SWIGLU) {                                     // the up rows sit eight lanes above their gate rows
            const float u = __shfl_down_sync(0xffffffffu, v, 8);
            if (!(row & 8) && n + 8 < N) out[(size_t)m * ldo + (n0 >> 1) + ((row >> 4) << 3) + (row & 7)] = from_f32<TO>(glu_epilogue<false>(accumulate, v, u));      // (with SWIGLU the argument carries the activation's code)
          } else if (n_in) {
            out[(size_t)m * ldo + n] = from_f32<TO>(add ? v + old[j] : v);
          }
        }
      }
    } else {
      // Rows m_begin .. m_end are this block's to finish: a warp takes every fourth of them, a lane four weight rows of it
      // (16-byte reads of every rank's sums, all of a group of RB rows in flight together).  What the sums are added to
      // is asked for while the products run.
      const int rows_per = (NB + split - 1) / split, m_begin = rank * rows_per, m_end = min(min(M, NB), m_begin + rows_per);
      const int n = n0 + 4 * lane;
      const bool add = !SWIGLU && accumulate;
      const bool vec = n + 4 <= N && ((size_t)ldo * sizeof(TO)) % (4 * sizeof(TO)) == 0 && ((uintptr_t)out) % (4 * sizeof(TO)) == 0;
      auto column = [&](const float* p, float none) {
        return make_float4(p && n < N ? p[n] : none, p && n + 1 < N ? p[n + 1] : none, p && n + 2 < N ? p[n + 2] : none, p && n + 3 < N ? p[n + 3] : none);
      };
      const float4 cs = column(colscale, 1.0f), cb = column(colbias, 0.0f);
      constexpr int RB = 2;                                 // rows of a group
      auto before = [&](int m) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (add && m < m_end) {
          const TO* o = out + (size_t)m * ldo + n;
          if (vec) v = read4(o);
          else v = make_float4(n < N ? to_f32(o[0]) : 0.f, n + 1 < N ? to_f32(o[1]) : 0.f, n + 2 < N ? to_f32(o[2]) : 0.f, n + 3 < N ? to_f32(o[3]) : 0.f);
        }
        return v;
      };
      float4 old[RB];
#pragma unroll
      for (int i = 0; i < RB; i++) old[i] = before(m_begin + quarter + 4 * i);
      mbar_wait(acc_full, 0, err, 33, wait_limit);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int c = 0; c < NB / CW; c++) {
        uint32_t r[CW];
        read_columns(c, r);
#pragma unroll
        for (int j = 0; j < CW; j++) part[(c * CW + j) * WM + row] = n_k > 0 ? __uint_as_float(r[j]) : 0.f;
      }
      // every block's sums are in its shared memory (the stages are free: every product that read them is complete)
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      asm volatile("barrier.cluster.arrive.release;" ::: "memory");
      asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
      const float* src[8];                                  // the sums of every rank, this lane's weight rows
#pragma unroll
      for (int q = 0; q < 8; q++) src[q] = in_rank(part, min(q, split - 1)) + 4 * lane;
#pragma unroll 1
      for (int m0 = m_begin + quarter; m0 < m_end; m0 += 4 * RB) {
        float4 x[RB][8];
#pragma unroll
        for (int i = 0; i < RB; i++)
#pragma unroll
          for (int q = 0; q < 8; q++)
            x[i][q] = (q < split && m0 + 4 * i < m_end) ? *reinterpret_cast<const float4*>(src[q] + (m0 + 4 * i) * WM) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < RB; i++) {
          const int m = m0 + 4 * i;
          if (m >= m_end) break;                            // (the same for the whole warp)
          float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int q = 0; q < 8; q++) { v.x += x[i][q].x; v.y += x[i][q].y; v.z += x[i][q].z; v.w += x[i][q].w; }   // in the order of the ranks; absent ranks add zero
          v = make_float4(v.x * cs.x + cb.x, v.y * cs.y + cb.y, v.z * cs.z + cb.z, v.w * cs.w + cb.w);
          if (SWIGLU) {                                     // the up rows sit two lanes above their gate rows
            const float4 u = make_float4(__shfl_down_sync(0xffffffffu, v.x, 2), __shfl_down_sync(0xffffffffu, v.y, 2),
                                         __shfl_down_sync(0xffffffffu, v.z, 2), __shfl_down_sync(0xffffffffu, v.w, 2));
            if (!(lane & 2) && n + 8 < N) {                 // (N is a multiple of 16: the four features are there or none is)
              TO* o = out + (size_t)m * ldo + (n0 >> 1) + ((lane >> 2) << 3) + (lane & 1) * 4;
              const float4 y = make_float4(glu_epilogue<false>(accumulate, v.x, u.x), glu_epilogue<false>(accumulate, v.y, u.y),
                                           glu_epilogue<false>(accumulate, v.z, u.z), glu_epilogue<false>(accumulate, v.w, u.w));
              if (((uintptr_t)o) % (4 * sizeof(TO)) == 0) write4(o, y);
              else { o[0] = from_f32<TO>(y.x); o[1] = from_f32<TO>(y.y); o[2] = from_f32<TO>(y.z); o[3] = from_f32<TO>(y.w); }
            }
          } else {
            if (add) { v.x += old[i].x; v.y += old[i].y; v.z += old[i].z; v.w += old[i].w; }
            TO* o = out + (size_t)m * ldo + n;
            if (vec) write4(o, v);
            else {
              if (n < N) o[0] = from_f32<TO>(v.x);
              if (n + 1 < N) o[1] = from_f32<TO>(v.y);
              if (n + 2 < N) o[2] = from_f32<TO>(v.z);
              if (n + 3 < N) o[3] = from_f32<TO>(v.w);
            }
          }
        }
#pragma unroll
        for (int i = 0; i < RB; i++) old[i] = before(m0 + 4 * (RB + i));
      }
    }
  }
  __syncwarp();                                             // the loader's and the issuer's warps are whole again
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  if (split > 1 && warp < 2) {                              // the epilogue warps met above
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  }
  // no block leaves while another may still read its sums
  if (split > 1) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  } else {
    __syncthreads();
  }
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TCOLS) : "memory");
}

int g_few_rows = 1;                     // test hook: 0 = never this kernel
int g_force_split = 0;                  // test hook: blocks per tile (0: chosen)
int g_max_rows = 128;                   // test hook: products of more rows go to the tiles of the prompt product
int g_min_tiles = 0;                    // test hook: outputs of fewer tiles of 128 weight rows stay with the other kernels (0: by the rows)
bool g_configured = false;
int g_max_split[4] = {0, 0, 0, 0};      // [log2 split]: how many clusters of that size run at once (0: that size is not available)

template <typename TO, int NB, int STAGES, bool SWIGLU>
int launch_few(const CUtensorMap& mw, const CUtensorMap& mx, void* out, int ldo, const float* colscale, const float* colbias,
               TlcEpi accumulate, int M, int N, int K, int split, cudaStream_t stream) {
  using S = FrSmem<NB, STAGES>;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(gemm_few_rows_kernel<TO, NB, STAGES, SWIGLU>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::TOTAL) != cudaSuccess)
      return tlc_fail(-2, "linear(few rows): cannot reserve %d bytes of shared memory", S::TOTAL);
    attr_set = true;
  }
  const int tiles = (N + WM - 1) / WM;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles * split);
  cfg.blockDim = dim3(FR_THREADS);
  cfg.dynamicSmemBytes = S::TOTAL;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (split > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = split;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = 1;
    na++;
  }
  if (g_tlc_pdl) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    na++;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  cudaLaunchKernelEx(&cfg, gemm_few_rows_kernel<TO, NB, STAGES, SWIGLU>, mw, mx, (TO*)out, ldo, colscale, colbias, accumulate, M, N,
                     K, split, tlc_error_words());
  TLC_CHECK_LAUNCH("linear(few rows)");
  return 0;
}

// Stages of a block's ring.  Two blocks fit on an SM up to 113 KB each, which five stages of 32 rows (102 KB) would still do; but
// what runs beside a layer's products (attention, the scan of the other mixer) then finds no room there: a step of the 7B sizes
// at batch 32 7.29 ms with four, 7.85 with five.  So 32, 64 and 128 rows stay below 98 KB (82, 98 and 98).  16 rows come from
// vocabularies alone, beside which nothing runs: six (110 KB).
constexpr int fr_stages(int NB) { return NB == 16 ? 6 : NB <= 64 ? 4 : 3; }

// How many blocks share a tile's K-steps: as many (2, 4, 8) as bring the grid closest to two blocks an SM (what
// fits beside one another) without passing it, each with at least 4 K-steps.  (64 rows of 2048 -> 8240, 65 tiles, four blocks
// each: 10.8 us.)
int pick_split(int N, int K, int NB, int sms) {
  const int tiles = (N + WM - 1) / WM, num_k = (K + FBK - 1) / FBK;
  int split = 1;
  while (split < 8 && tiles * split * 2 <= 2 * sms && num_k / (split * 2) >= 4 && NB % (split * 2) == 0) split *= 2;
  return split;
}

template <bool SWIGLU>
int run_few(const void* a, int lda, const void* w, int ldw, void* out, int out_dtype, int ldo, const float* colscale,
            const float* colbias, TlcEpi accumulate, int M, int N, int K, int force_split, cudaStream_t stream) {
  static int sms = 0;
  if (sms == 0) { int dev = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev); }
  const int NB = M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128;
  const int split = force_split > 0 ? force_split : pick_split(N, K, NB, sms);
  CUtensorMap mw, mx;
  if (int rc = tlc_tensor_map_bf16(w, N, K, ldw, FBK, WM, &mw)) return rc;
  if (int rc = tlc_tensor_map_bf16(a, M, K, lda, FBK, NB, &mx)) return rc;
#define TLC_FEW(TO_, NB_) launch_few<TO_, NB_, fr_stages(NB_), SWIGLU>(mw, mx, out, ldo, colscale, colbias, accumulate, M, N, K, split, stream)
#define TLC_FEW_NB(TO_) (NB == 16 ? TLC_FEW(TO_, 16) : NB == 32 ? TLC_FEW(TO_, 32) : NB == 64 ? TLC_FEW(TO_, 64) : TLC_FEW(TO_, 128))
  if (out_dtype == TLC_F32) return TLC_FEW_NB(float);
  if (out_dtype == TLC_BF16) return TLC_FEW_NB(__nv_bfloat16);
#undef TLC_FEW_NB
#undef TLC_FEW
  return tlc_fail(-1, "linear: unknown output dtype %d", out_dtype);
}

// bfloat16 operands with 16-byte aligned rows, up to 128 rows, where this kernel is the quickest (microseconds in a captured
// loop over operand sets larger than the L2):
//   * from 17 rows on, an output that is wide enough, 32 tiles of 128 weight rows, 16 with more than 32 rows, and not more
//     tiles than two an SM (96 rows, 3072 -> 130048: 141 with the tiles of the product for prompts, 149 here).  At 64 rows
//     2048 -> 8240 10.8, 4096 -> 2048 8.4, 2560 -> 16384 18.7 (with SwiGLU 20.7), 3072 -> 24576 28.7 (34.9);
//   * up to 32 rows, a plain 32-bit output of 128 tiles or more, a vocabulary: there the weight-streaming mma.sync kernel
//     re-reads the activations for every 16 columns, and its rounds of K (2,048; from 9 rows on 1,024) may end in a part
//     of one (32 rows, 3072 -> 130048: 240 with that kernel, 129 here; 16 rows, 2560 -> 65536: 67 and 53; 8 rows, 3072 ->
//     130048 143 and 120; 1 row 125 and 117).  Up to 4 rows with full rounds it is as quick (2048 -> 65536: 40.9 and 42.1)
//     and keeps them.
// Narrower outputs of up to 32 rows would gain as well (32 rows, 12288 -> 3072: 31.6 and 15.9), but their sums would be made
// in another order, and what a layer rounds to 16 bits after them would move the tokens that a model picks; a logit is
// not rounded again.
// With a forced split (tests) any output of at least one tile qualifies, from 9 rows on.
int few_rows_ok(int a_dtype, int lda, const void* a, int w_dtype, int ldw, const void* w, int M, int N, int K, bool plain32) {
  static int sms = 0;
  if (sms == 0) { int dev = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev); }
  if (!g_few_rows || a_dtype != TLC_BF16 || w_dtype != TLC_BF16 || M > g_max_rows || K % 8 != 0 || lda % 8 != 0 || ldw % 8 != 0 ||
      (uintptr_t)a % 16 != 0 || (uintptr_t)w % 16 != 0 || tlc_error_words_here() == nullptr)
    return 0;
  const int tiles = (N + WM - 1) / WM;
  if (g_force_split > 0) return M > 8 && N >= WM;
  if (M <= 32 && plain32 && tiles >= 128) return M > 4 || K % 2048 != 0;
  return M > 16 && N >= (g_min_tiles > 0 ? g_min_tiles : M > 32 ? 16 : 32) * WM && tiles <= 2 * sms;
}

}  // namespace

// Test hooks: whether products of up to 128 rows may take this kernel; a fixed number of blocks per tile (0: chosen).
extern "C" void tlc_linear_few_rows(int on) { g_few_rows = on; }
extern "C" void tlc_linear_few_rows_split(int split) { g_force_split = split; }
extern "C" void tlc_linear_few_rows_min_tiles(int tiles) { g_min_tiles = tiles; }
extern "C" void tlc_linear_few_rows_max_rows(int rows) { g_max_rows = rows; }

// plain32: the output is 32-bit and overwritten, not added to.
int tlc_linear_few_rows_takes(int a_dtype, int lda, const void* a, int w_dtype, int ldw, const void* w, int M, int N, int K, bool plain32) {
  return few_rows_ok(a_dtype, lda, a, w_dtype, ldw, w, M, N, K, plain32);
}
extern "C" int tlc_linear_few_rows_ok(int a_dtype, int lda, const void* a, int w_dtype, int ldw, const void* w, int M, int N, int K) {
  return few_rows_ok(a_dtype, lda, a, w_dtype, ldw, w, M, N, K, false);
}

int tlc_linear_few_rows_run(const void* a, int lda, const void* w, int ldw, void* out, int out_dtype, int ldo,
                            const float* colscale, const float* colbias, TlcEpi accumulate, int M, int N, int K,
                            cudaStream_t stream) {
  return run_few<false>(a, lda, w, ldw, out, out_dtype, ldo, colscale, colbias, accumulate, M, N, K, g_force_split, stream);
}

int tlc_linear_few_rows_swiglu(const void* a, int lda, const void* w, int ldw, void* out, int out_dtype, int ldo,
                               const float* colscale, const float* colbias, int M, int N, int K, TlcEpi act, cudaStream_t stream) {
  return run_few<true>(a, lda, w, ldw, out, out_dtype, ldo, colscale, colbias, act, M, N, K, g_force_split, stream);
}
