// Products of few activation rows (batched decode: 2..128) on the 5th-generation tensor cores:
// C[M,N] = A[M,K] * W[N,K]^T, bounded by streaming W once.
//
// The weights are the M operand of tcgen05.mma (128 rows of W a tile) and the activation rows its N operand (MT = 16, 32, 64
// or 128 columns), so nothing is multiplied or staged for rows that do not exist beyond MT.
//   warp 0   : TMA producer - [128 x 128 B] tiles of W and [MT x 128 B] tiles of A into a ring.  The first ring of W tiles is
//              requested BEFORE the dependency wait, A's after it.  The launch may overlap the ones before it only where the caller
//              says that W is resident, written long before; otherwise it is an ordinary launch, which starts after them.  The ring
//              is small enough for two CTAs an SM, so that under programmatic dependent launch this projection's stream starts
//              while the kernels ahead of it drain;
//   warp 1   : MMA issuer;
//   warps 2-5: epilogue - accumulator out of TMEM through shared memory, so that a warp stores 128 consecutive columns of a row.
// K is split over the S CTAs of a cluster (S <= 8), and the partial tiles are added over distributed shared memory, in slice
// order, each CTA finishing 1 / S of the tile.  No workspace, no tickets, and the sum does not depend on timing.
// Measured back to back in a graph (weights of every launch cold): 64 rows, 2560 x 9216 35.6 -> 15.0 us, 2560 x 4096 19.3 -> 12.1 us
// against the 128-row tiles with partial tiles in global memory (with slices that fill the machine 14.6 and 10.4 us); 8 rows 25.0 ->
// 11.8 us and 10.0 -> 6.9 us against the mma.sync GEMV; gate|up 18432 x 2560 of 64 rows with the product 24.9 -> 21.5 us.  What is left
// is the chain of latencies of one launch (dependency, first A tile, accumulator, cluster exchange, store), about 4 us.
#include <algorithm>

#include "act_type.cuh"
#include "sm100.cuh"

namespace {

using namespace sm100;

constexpr int kRowsTile = 128, kRowsKB = 128;        // weight rows a tile; bytes of a row a k-block
constexpr int kRowsThreads = 192;

struct RowsArgs {
  void* C; int64_t ldc;
  const bf16* residual; int64_t ldr;
  const float* row_scale; const float* col_scale;    // int8: scales of the activation rows / of the weight rows
  float* C2; int64_t ldc2; int n_main;               // columns from n_main on leave as fp32 in C2 (null: none)
  int c_f32;
  int act; float act_a, act_b;
  int M, N, up_off;                                  // N: output columns; SWIGLU: gate row n is paired with row up_off + n
  int n_tiles, k_blocks;
  int wt;                                            // rows of W a tile: 128 or 64 (SWIGLU: half of them gate, half up)
  int kper;                                          // k-blocks of a slice, the last one shorter (0: even slices)
  int round_halves;                                  // SWIGLU of gate and up as bf16 holds them
  int scale_rows_first;                              // int8: (sum * row scale) * column scale instead of sum * (row scale * column scale)
  int* status;
};

__device__ __forceinline__ uint64_t rows_now() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
// bounded by the clock (2 s)
__device__ __forceinline__ bool rows_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  if (mbar_try(bar, parity)) return true;
  const uint64_t t0 = rows_now();
  for (;;) {
    for (int i = 0; i < 256; ++i)
      if (mbar_try(bar, parity)) return true;
    if (*abort_flag) return false;
    if (rows_now() - t0 > 2000000000ull) return false;
  }
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

// sum of the slices' partial values at byte offset `off` of their staging areas, in slice order (int8: exact, in integers)
template <bool I8>
__device__ __forceinline__ float4 rows_gather(uint32_t base, uint32_t off, int S, const float* own) {
  if (S == 1) {
    float4 v = *reinterpret_cast<const float4*>(reinterpret_cast<const char*>(own) + off);
    if (I8)
      v = make_float4((float)__float_as_int(v.x), (float)__float_as_int(v.y), (float)__float_as_int(v.z), (float)__float_as_int(v.w));
    return v;
  }
  float4 p[8];
#pragma unroll
  for (int s = 0; s < 8; ++s)
    if (s < S) p[s] = ld_cluster_f4(map_to_cta(base + off, (uint32_t)s));
  if (I8) {
    int4 t = make_int4(0, 0, 0, 0);
#pragma unroll
    for (int s = 0; s < 8; ++s)
      if (s < S) { t.x += __float_as_int(p[s].x); t.y += __float_as_int(p[s].y); t.z += __float_as_int(p[s].z); t.w += __float_as_int(p[s].w); }
    return make_float4((float)t.x, (float)t.y, (float)t.z, (float)t.w);
  }
  float4 t = p[0];
#pragma unroll
  for (int s = 1; s < 8; ++s)
    if (s < S) { t.x += p[s].x; t.y += p[s].y; t.z += p[s].z; t.w += p[s].w; }
  return t;
}

template <int MT, int STAGES, bool I8, bool SWIGLU>
__global__ void __launch_bounds__(kRowsThreads, 2)
gemm_rows_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmA, const RowsArgs a) {
  constexpr int W_BYTES = kRowsTile * kRowsKB, A_BYTES = MT * kRowsKB, STAGE_BYTES = W_BYTES + A_BYTES;
  constexpr int BK = I8 ? 128 : 64;                  // elements of a k-block
  constexpr uint32_t TMEM_COLS = 2 * MT;             // two accumulators (a power of two >= 32)
  constexpr uint32_t IDESC = umma_idesc(kRowsTile, MT, 1, I8 ? 2 : 1);
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* ring = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  float* chunk = reinterpret_cast<float*>(ring + (size_t)STAGES * STAGE_BYTES);   // [16][128], one slice only
  __shared__ uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;
  volatile int* abort_flag = &abort_s;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = gridDim.x, ks = blockIdx.x;          // the cluster is the whole x extent of the grid
  const int kb0 = a.kper ? ks * a.kper : (int)((int64_t)a.k_blocks * ks / S);
  const int kb1 = a.kper ? min(a.k_blocks, kb0 + a.kper) : (int)((int64_t)a.k_blocks * (ks + 1) / S);
  const int wt = a.wt, tn = SWIGLU ? wt / 2 : wt;    // output columns of a tile
  const int cbits = __ffs(tn) - 3;                   // log2 of its groups of four columns
  const int first = min(kb1 - kb0, STAGES);
  auto load_w = [&](int tile, int kb, int s) {
    unsigned char* st = ring + (size_t)s * STAGE_BYTES;
    mbar_expect_tx(&full_bar[s], wt * kRowsKB + A_BYTES);
    tma_load_2d(st, &tmW, &full_bar[s], kb * BK, tile * tn);
    if (SWIGLU) tma_load_2d(st + tn * kRowsKB, &tmW, &full_bar[s], kb * BK, a.up_off + tile * tn);
  };
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 4); }
    abort_s = 0;
    mbar_fence_init();
    for (int i = 0; i < first; ++i) load_w(blockIdx.y, kb0 + i, i);
  }
  // tensor memory is taken before dependents may start: one that took it first would hold it while it waits for this kernel
  if (warp == 1) {
    tmem_alloc(&tmem_base_s, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  griddep_launch();

  if (warp == 0) {
    // ------------------------------- TMA producer -----------------------------------------
    if (lane == 0) {
      auto load_a = [&](int kb, int s) { tma_load_2d(ring + (size_t)s * STAGE_BYTES + W_BYTES, &tmA, &full_bar[s], kb * BK, 0); };
      griddep_wait();
      for (int i = 0; i < first; ++i) load_a(kb0 + i, i);
      uint32_t it = 0;
      for (int tile = blockIdx.y; tile < a.n_tiles && !*abort_flag; tile += gridDim.y) {
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          if ((int)it < first) continue;
          const int s = it % STAGES;
          if (!rows_wait(&empty_bar[s], ((it / STAGES) & 1) ^ 1, abort_flag)) { atomicExch(a.status, 91); abort_s = 1; break; }
          load_w(tile, kb, s);
          load_a(kb, s);
        }
      }
    }
  } else {
    const uint32_t tmem_base = tmem_base_s;
    if (warp == 1) {
      // ------------------------------- MMA issuer -----------------------------------------
      if (lane == 0) {
        uint32_t it = 0, tcount = 0;
        for (int tile = blockIdx.y; tile < a.n_tiles && !*abort_flag; tile += gridDim.y, ++tcount) {
          const uint32_t acc = tcount & 1;
          if (!rows_wait(&acc_empty[acc], ((tcount >> 1) & 1) ^ 1, abort_flag)) { atomicExch(a.status, 92); abort_s = 1; break; }
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + acc * MT;
          bool ok = true;
          for (int kb = kb0; kb < kb1; ++kb, ++it) {
            const int s = it % STAGES;
            if (!rows_wait(&full_bar[s], (it / STAGES) & 1, abort_flag)) { atomicExch(a.status, 93); abort_s = 1; ok = false; break; }
            tc_fence_after();
            const unsigned char* st = ring + (size_t)s * STAGE_BYTES;
            const uint64_t wd = umma_desc_sw128(st), xd = umma_desc_sw128(st + W_BYTES);
#pragma unroll
            for (int k = 0; k < 4; ++k) {            // 32 bytes along K inside the swizzle atom: +2 in 16-byte units
              if (I8) umma_i8(d_tmem, wd + 2 * k, xd + 2 * k, IDESC, ((kb - kb0) | k) != 0);
              else umma_f16(d_tmem, wd + 2 * k, xd + 2 * k, IDESC, ((kb - kb0) | k) != 0);
            }
            umma_commit(&empty_bar[s]);
          }
          if (!ok) break;
          umma_commit(&acc_full[acc]);
        }
      }
    }
  }
  const int et = (int)threadIdx.x - 64;              // epilogue thread, 0..127
  // four columns n.. of output row m from their sums
  auto finish = [&](int m, int n, float4 v, float4 u) {
    if (m >= a.M || n >= a.N) return;                // N is a multiple of 8
    if (I8) {
      const float rs = a.row_scale[m];
      // scales may start anywhere (111 rows, 20176 x 544: 14.9 us with vector loads, 16.6 without)
      const bool vec = ((uintptr_t)a.col_scale & 15) == 0;
      auto scales = [&](const float* p) { return vec ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]); };
      const float4 cs = scales(a.col_scale + n);
      if (a.scale_rows_first) { v.x = v.x * rs * cs.x; v.y = v.y * rs * cs.y; v.z = v.z * rs * cs.z; v.w = v.w * rs * cs.w; }
      else { v.x *= rs * cs.x; v.y *= rs * cs.y; v.z *= rs * cs.z; v.w *= rs * cs.w; }
      if (SWIGLU) {
        const float4 cu = scales(a.col_scale + a.up_off + n);
        u.x *= rs * cu.x; u.y *= rs * cu.y; u.z *= rs * cu.z; u.w *= rs * cu.w;
      }
    }
    if (SWIGLU && a.round_halves) {
      v.x = act_round<bf16>(v.x); v.y = act_round<bf16>(v.y); v.z = act_round<bf16>(v.z); v.w = act_round<bf16>(v.w);
      u.x = act_round<bf16>(u.x); u.y = act_round<bf16>(u.y); u.z = act_round<bf16>(u.z); u.w = act_round<bf16>(u.w);
    }
    if (SWIGLU) { v.x = silu_f(v.x) * u.x; v.y = silu_f(v.y) * u.y; v.z = silu_f(v.z) * u.z; v.w = silu_f(v.w) * u.w; }
    if (a.act) {
      v.x = epi_act(a.act, v.x, a.act_a, a.act_b); v.y = epi_act(a.act, v.y, a.act_a, a.act_b);
      v.z = epi_act(a.act, v.z, a.act_a, a.act_b); v.w = epi_act(a.act, v.w, a.act_a, a.act_b);
    }
    if (a.residual) {
      const float4 r = act_load4(a.residual + (int64_t)m * a.ldr + n);
      v.x += r.x; v.y += r.y; v.z += r.z; v.w += r.w;
    }
    if (a.c_f32) act_store4(reinterpret_cast<float*>(a.C) + (int64_t)m * a.ldc + n, v);
    else if (a.C2 && n >= a.n_main) act_store4(a.C2 + (int64_t)m * a.ldc2 + n - a.n_main, v);
    else act_store4(reinterpret_cast<bf16*>(a.C) + (int64_t)m * a.ldc + n, v);
  };
  bool staged = true;
  if (warp >= 2) {
    // ------------------------------- epilogue ---------------------------------------------
    griddep_wait();                                  // the residual and C belong to earlier kernels until here
    const int q = warp & 3;
    const uint32_t lane_base = tmem_base_s + ((uint32_t)(q * 32) << 16);
    uint32_t tcount = 0;
    for (int tile = blockIdx.y; tile < a.n_tiles && !*abort_flag; tile += gridDim.y, ++tcount) {
      const uint32_t acc = tcount & 1;
      if (!rows_wait(&acc_full[acc], (tcount >> 1) & 1, abort_flag)) {
        if (lane == 0) { atomicExch(a.status, 94); abort_s = 1; }
        staged = false;
        break;
      }
      tc_fence_after();
      if (S > 1) {
        // one tile a cluster: the ring is idle now, the whole partial tile goes there as [m][128]
        float* part = reinterpret_cast<float*>(ring);
#pragma unroll 1
        for (int c0 = 0; c0 < MT && c0 < a.M && q * 32 < wt; c0 += 16) {
          uint32_t r[16];
          tmem_ld16(lane_base + acc * MT + c0, r);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) part[(c0 + i) * 128 + q * 32 + lane] = __uint_as_float(r[i]);
        }
        break;
      }
#pragma unroll 1
      for (int c0 = 0; c0 < MT && c0 < a.M; c0 += 16) {
        uint32_t r[16];
        if (q * 32 < wt) {
          tmem_ld16(lane_base + acc * MT + c0, r);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) chunk[i * 128 + q * 32 + lane] = __uint_as_float(r[i]);
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        for (int e = et; e < 16 << cbits; e += 128) {
          const int m = e >> cbits, n = (e & ((1 << cbits) - 1)) * 4;
          const float4 v = rows_gather<I8>(0, (uint32_t)(m * 128 + n) * 4, 1, chunk);
          const float4 u = SWIGLU ? rows_gather<I8>(0, (uint32_t)(m * 128 + tn + n) * 4, 1, chunk) : v;
          finish(c0 + m, tile * tn + n, v, u);
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[acc]);
    }
  }
  __syncwarp();
  if (S > 1) {
    cluster_sync_all();                              // every slice's partial tile is in place
    if (warp >= 2 && staged) {
      const uint32_t base = smem_u32(ring);
      const int tile = blockIdx.y, total = a.M << cbits;
      for (int e = ks * 128 + et; e < total; e += S * 128) {
        const int m = e >> cbits, n = (e & ((1 << cbits) - 1)) * 4;
        const float4 v = rows_gather<I8>(base, (uint32_t)(m * 128 + n) * 4, S, nullptr);
        const float4 u = SWIGLU ? rows_gather<I8>(base, (uint32_t)(m * 128 + tn + n) * 4, S, nullptr) : v;
        finish(m, tile * tn + n, v, u);
      }
    }
    cluster_sync_all();                              // nobody leaves while its shared memory is being read
  }
  // ------------------------------- teardown ---------------------------------------------------
  tc_fence_before();
  __syncthreads();
  if (abort_s) {  // give copies still in flight time to land before the shared memory is released
    const uint64_t t0 = rows_now();
    while (rows_now() - t0 < 2000000ull) __nanosleep(1000);
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base_s, TMEM_COLS);
  }
}

int rows_sms() {
  static int sms = 0;
  if (!sms) {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    sms = n > 0 ? n : 148;
  }
  return sms;
}

// Decode projections of two to eight rows: as many slices of K per output tile as one wave of CTAs takes.  Pairs fill both CTAs of
// every SM (up to 296 CTAs); wider clusters have to fit into the SMs of one GPC and leave some idle, so beyond about 1.4 CTAs an SM a
// second wave starts.  Measured at 16 rows: 2560 x 4096 (20 tiles) 21.8 / 12.7 / 8.6 / 6.9 us with 1 / 2 / 4 / 8 slices; 12352 x 2560
// (97 tiles) 15.6 / 13.8 / 16.6 with 1 / 2 / 4; 6176 x 2560 (49 tiles) 12.0 us with 6 slices (294 CTAs).  Odd slice counts lose to the
// even ones beside them (TPCs are pairs of SMs).
int fill_slices(int64_t tiles, int64_t kb) {
  const int64_t sms = rows_sms();
  int s = 8;
  while (s > 1 && (tiles * s > (s == 2 ? 2 * sms : sms * 7 / 5) || kb < 4 * s)) s = s > 2 ? s - 2 : 1;   // a slice has at least four k-blocks
  return s;
}

// Batched products: slices of ceil(k_blocks / s) k-blocks, s by the estimate below: the bytes a CTA moves into shared memory with
// tiles of 256, 128 or 64 rows of W and one CTA an SM, against what adding s partial tiles costs.  The slices are part of a product's
// value: bf16 residuals and recurrent states carry a changed order of sums through all layers that follow (64 rows of the 32-layer
// shape: half an rms at single elements of the states), so they stay as they are when kernels change.
int planned_slices(int64_t M, int64_t N, int64_t Kbytes, int narrowest, int* width = nullptr) {
  const int64_t sms = rows_sms(), kb = (Kbytes + 127) / 128, K = Kbytes / 2;
  double best = 1e300;
  int64_t slices = 1;
  for (int bn = 256; bn >= narrowest; bn /= 2) {
    const int64_t tiles = (N + bn - 1) / bn;
    int64_t s = std::max<int64_t>(1, std::min<int64_t>(32, std::min(sms / tiles, kb / 4)));
    for (;;) {                           // no slice may be empty: s = ceil(kb / ceil(kb / s))
      const int64_t kper = (kb + s - 1) / s, s2 = (kb + kper - 1) / kper;
      if (s2 == s) break;
      s = s2;
    }
    const int64_t waves = (tiles * s + sms - 1) / sms;
    const double stream = (double)waves * (bn + M) * ((double)K / s) * 2.0 / 130e3;        // us at ~130 GB/s per SM
    const double cost = stream + (s > 1 ? (double)s * M * bn * 4.0 / 100e3 + 2.0 : 0.0);
    if (cost < best) {
      best = cost;
      slices = s;
      if (width) *width = bn;
    }
  }
  return (int)slices;
}

template <int MT, int STAGES, bool I8, bool SWIGLU>
int launch_rows(const CUtensorMap& tmW, const CUtensorMap& tmA, const RowsArgs& a, int S, int resident, cudaStream_t st) {
  const size_t smem = (size_t)STAGES * (kRowsTile + MT) * kRowsKB + 16 * 128 * 4 + 1024;
  auto kern = gemm_rows_kernel<MT, STAGES, I8, SWIGLU>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  const int most = 2 * rows_sms() / S;
  const int y = a.n_tiles < most || S > 1 ? a.n_tiles : most;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)S, (unsigned)y);
  cfg.blockDim = dim3(kRowsThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)S;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = g_cb_use_pdl && resident ? 2 : 1;
  if (g_cb_trace_names) cb_trace_name((const void*)kern);
  return (int)cudaLaunchKernelEx(&cfg, kern, tmW, tmA, a);
}

template <bool I8, bool SWIGLU>
int rows_run(const void* A, int64_t lda, const void* W, int64_t ldw, int64_t w_rows, int64_t K, int fill, int resident, RowsArgs a,
             cudaStream_t st) {
  constexpr int BK = I8 ? 128 : 64;
  const CUtensorMapDataType dt = I8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  const int mt = a.M <= 16 ? 16 : (a.M <= 32 ? 32 : (a.M <= 64 ? 64 : 128));
  a.k_blocks = (int)((K + BK - 1) / BK);
  a.wt = kRowsTile;
  const int64_t tiles = (w_rows + kRowsTile - 1) / kRowsTile;
  const int planned = fill ? 0 : planned_slices(a.M, w_rows, K * (I8 ? 1 : 2), I8 ? 128 : 64);
  int S = fill_slices(tiles, a.k_blocks);
  if (I8) {
    a.scale_rows_first = planned == 1;               // integer sums do not depend on the slices
  } else if (planned >= 1 && planned <= 8) {
    S = planned;
    a.kper = (a.k_blocks + S - 1) / S;
    // as many CTAs as fit in a wave.  64 rows of A: 12352 x 2560 (97 tiles, one slice) 20.5 us with 128-row tiles, 19.4 with 64-row ones;
    // 2560 x 9216 (20 tiles, 7 slices) 15.1 and 22.6 us (280 CTAs in clusters of 7 take two waves)
    if (S > 1 ? 2 * tiles * S <= rows_sms() * 7 / 5 : tiles <= rows_sms()) a.wt = kRowsTile / 2;
  }
  const int tn = SWIGLU ? a.wt / 2 : a.wt;
  CUtensorMap tmW, tmA;
  int rc = cb_make_tmap_2d(&tmW, dt, I8 ? 1 : 2, W, (uint64_t)w_rows, (uint64_t)K, (uint64_t)ldw, tn, BK);
  if (rc) return rc;
  rc = cb_make_tmap_2d(&tmA, dt, I8 ? 1 : 2, A, (uint64_t)a.M, (uint64_t)K, (uint64_t)lda, mt, BK);
  if (rc) return rc;
  a.n_tiles = (a.N + tn - 1) / tn;
  if (mt == 16) return launch_rows<16, 5, I8, SWIGLU>(tmW, tmA, a, S, resident, st);
  if (mt == 32) return launch_rows<32, 5, I8, SWIGLU>(tmW, tmA, a, S, resident, st);
  if (mt == 64) return launch_rows<64, 4, I8, SWIGLU>(tmW, tmA, a, S, resident, st);
  return launch_rows<128, 3, I8, SWIGLU>(tmW, tmA, a, S, resident, st);
}

int rows_args(void* C, int64_t ldc, const void* residual, int64_t ldr, int64_t M, int64_t N, int64_t K, int64_t form, void* status,
              RowsArgs* out) {
  if (M < 1 || M > kRowsTile || N < 1 || K < 1 || N % 8 || form < 0 || form > 3 || !C || !status) return CB_ERR_SHAPE;
  if (ldc % (form == 1 ? 4 : 8) || (residual && (ldr % 8 || form == 1))) return CB_ERR_SHAPE;
  if (((uintptr_t)C & (form == 1 ? 15 : 7)) || ((uintptr_t)residual & 7)) return CB_ERR_SHAPE;      // results travel by fours
  RowsArgs a = {};
  a.C = C; a.ldc = ldc; a.residual = (const bf16*)residual; a.ldr = ldr; a.c_f32 = form == 1;
  a.round_halves = form == 3;
  a.M = (int)M; a.N = (int)N; a.up_off = (int)N; a.status = (int*)status;
  *out = a;
  return CB_OK;
}

}  // namespace

// Width of the 128-row tiles that take a bf16 product instead of this kernel (0: this kernel takes it).  Above 64 rows the rows fill
// such a tile, and an unsplit product has no partial tiles to save: 128 rows, 12352 x 2560 25.1 us here, 20.3 us there; 20000 x 1024 18.9
// and 15.4 us; 72 rows, 40000 x 2560 51.7 and 50.6 us.  In slices it stays (128 rows, 4096 x 1024: 9.8 and 22.2 us).  The same sums.
int cb_gemm_rows_tile(int64_t M, int64_t N, int64_t K) {
  int bn = 256;
  return M > 64 && M <= kRowsTile && planned_slices(M, N, K * 2, 64, &bn) == 1 ? bn : 0;
}
CB_EXPORT int cb_gemm_bf16(const void* A, int64_t lda, const void* W, int64_t ldw, void* C, int64_t ldc, const void* residual, int64_t ldr,
                           int64_t M, int64_t N, int64_t K, int64_t bn, const void* pf, int64_t pf_seq, void* status, void* stream);
CB_EXPORT int cb_gemm_bf16_f32out(const void* A, int64_t lda, const void* W, int64_t ldw, void* C, int64_t ldc, int64_t M, int64_t N,
                                  int64_t K, int64_t resident, void* status, void* stream);

// C[M,N] = A[M,K] x W[N,K]^T, M <= 128; form 0: bf16 (+ residual), 1: fp32, 2: SwiGLU of the rows [0, N) and [N, 2N) of W, 3: the
// same of gate and up rounded to bf16, as a product and cb_swiglu after it give it.  fill: K split to fill the machine, else by the plan of the batched
// products.  resident: no launch that may still run has written W.
CB_EXPORT int cb_gemm_rows_bf16(const void* A, int64_t lda, const void* W, int64_t ldw, void* C, int64_t ldc, const void* residual,
                                int64_t ldr, int64_t M, int64_t N, int64_t K, int64_t form, int64_t fill, int64_t resident, void* status, void* stream) {
  RowsArgs a;
  if (rows_args(C, ldc, residual, ldr, M, N, K, form, status, &a) || K % 8) return CB_ERR_SHAPE;
  const int bn = form < 2 && !fill && !(((uintptr_t)C | (uintptr_t)residual) & 15) ? cb_gemm_rows_tile(M, N, K) : 0;
  if (bn && form == 0) return cb_gemm_bf16(A, lda, W, ldw, C, ldc, residual, ldr, M, N, K, bn, nullptr, 0, status, stream);
  if (bn) return cb_gemm_bf16_f32out(A, lda, W, ldw, C, ldc, M, N, K, resident, status, stream);
  if (form >= 2) return rows_run<false, true>(A, lda, W, ldw, 2 * N, K, fill != 0, resident != 0, a, (cudaStream_t)stream);
  return rows_run<false, false>(A, lda, W, ldw, N, K, fill != 0, resident != 0, a, (cudaStream_t)stream);
}

// The same from int8 rows and weights: (A_q x W_q^T) * row_scale[m] * col_scale[n], summed exactly.
CB_EXPORT int cb_gemm_rows_i8(const void* A, int64_t lda, const void* W, int64_t ldw, void* C, int64_t ldc, const void* residual,
                              int64_t ldr, const void* row_scale, const void* col_scale, int64_t M, int64_t N, int64_t K, int64_t form,
                              int64_t fill, int64_t resident, void* status, void* stream) {
  RowsArgs a;
  if (rows_args(C, ldc, residual, ldr, M, N, K, form, status, &a)) return CB_ERR_SHAPE;
  if (K % 16 || lda % 16 || ldw % 16 || !row_scale || !col_scale) return CB_ERR_SHAPE;
  a.row_scale = (const float*)row_scale; a.col_scale = (const float*)col_scale;
  if (form >= 2) return rows_run<true, true>(A, lda, W, ldw, 2 * N, K, fill != 0, resident != 0, a, (cudaStream_t)stream);
  return rows_run<true, false>(A, lda, W, ldw, N, K, fill != 0, resident != 0, a, (cudaStream_t)stream);
}

// Forms of gemm_tc.cu's entry points for few rows (arguments checked there): xIELU in the epilogue; the columns from n_main on as
// fp32 in C2.
int cb_gemm_rows_xielu(const void* A, int64_t lda, const void* W, int64_t ldw, void* C, int64_t ldc, int64_t M, int64_t N, int64_t K,
                       float act_a, float act_b, int64_t resident, void* status, void* stream) {
  RowsArgs a;
  if (rows_args(C, ldc, nullptr, 0, M, N, K, 0, status, &a)) return CB_ERR_SHAPE;
  a.act = 1; a.act_a = act_a; a.act_b = act_b;
  return rows_run<false, false>(A, lda, W, ldw, N, K, 0, resident != 0, a, (cudaStream_t)stream);
}
int cb_gemm_rows_mixed(const void* A, int64_t lda, const void* W, int64_t ldw, void* C, int64_t ldc, void* C2, int64_t ldc2, int64_t n_main,
                       int64_t M, int64_t N, int64_t K, int64_t resident, void* status, void* stream) {
  RowsArgs a;
  if (rows_args(C, ldc, nullptr, 0, M, N, K, 0, status, &a)) return CB_ERR_SHAPE;
  if ((uintptr_t)C2 & 15) return CB_ERR_SHAPE;
  a.C2 = (float*)C2; a.ldc2 = ldc2; a.n_main = (int)n_main;
  return rows_run<false, false>(A, lda, W, ldw, N, K, 0, resident != 0, a, (cudaStream_t)stream);
}
