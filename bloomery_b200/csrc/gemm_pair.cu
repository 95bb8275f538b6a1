// bf16 grouped GEMM of long prompts on pairs of CTAs (tcgen05 cta_group::2, sm_100a only):
//   C[t, n] = sum_k X[t, k] * W[g][n, k]        fp32 accumulate in tensor memory
//
// A CTA that multiplies 128 x 256 on its own fetches 48 KB for a 64-deep step of 512 tensor-core clocks, and 148 of them ask L2
// for 13 TB/s, which is what bounds them (QKV of 4,096 ids, 2,048 x 5,120: 77 us, 1.11 PFLOP/s).  A pair shares one 256 x 256
// product: each CTA fetches half of either operand, 32 KB a step, and the tensor cores of both read the other's half (70.5 us,
// 1.22 PFLOP/s; 671 MB from L2, 9.2 TB/s, tensor pipe 73 % busy).  What is left is the last wave: 320 tiles on at most 74 pairs are
// 4.3 waves of five.
//
// The weights are the M side (256 rows of a pair, 128 of each CTA) and the tokens the N side, 64 to 256 of a tile, so a group of a
// hundred rows pays for 128, not for 256, and a group's weights are read once.  The gated form (gate and up) gives each CTA 64 rows
// of either matrix: its accumulator holds both products of the same 64 outputs, in different lanes, and the epilogue's warps hand
// each other half of them through shared memory.
//
// Each CTA: warp 0 fetches its halves (the bytes of both CTAs complete on the leader's barrier), warp 1 of the leader issues the
// MMAs, whose commits release the stage and publish the accumulator in both CTAs, warps 2 to 9 store the CTA's 128 lanes while
// the next tile's products run (two accumulators of 256 columns).  (Four of them took 110 clocks a token, more than its products.)
//
// Every wait is bounded by the global timer; on expiry a CTA raises status word 1, leaves its loops, meets its peer at the cluster
// barrier (which always completes), frees its tensor memory and returns.
//
// Role in the reference: see gemm_tcgen05.cu.
#include "tc_common.cuh"

#include <atomic>

namespace bl {

constexpr int PK = 64;                            // depth of a stage: one swizzle atom row of 128 bytes
constexpr int PM = 256, PN = 256;                 // weight rows and tokens of a tile, most of them
constexpr int PSTAGES = 6;
constexpr int PTHREADS = 64 + 256;                // TMA, MMA, eight epilogue warps
constexpr int P_A_BYTES = 128 * PK * 2;           // a CTA's weight rows of a stage
constexpr int P_B_BYTES = PN / 2 * PK * 2;        // a CTA's tokens of a stage, at most
constexpr int P_STAGE = P_A_BYTES + P_B_BYTES;
constexpr int P_SWAP = 16 * 64;                   // floats of one direction of the gated exchange, for 32 tokens
constexpr size_t kPairSmem = (size_t)PSTAGES * P_STAGE + 8 * P_SWAP * 4 + 1024;

struct PTile { int group, row0, row_end, pad; };  // token tile: rows row0 .. of X use weight matrix `group`

struct PairArgs {
  int N, K;
  int tiles_w;                // weight tiles of a matrix: 256 rows, or 128 of either in the gated form
  const PTile* tiles;
  const int* n_tiles;
  int max_tiles;
  const int* dst_row;         // optional scatter of token rows (< 0 = drop)
  TokenOut out;
  unsigned* status;
};

__device__ __forceinline__ uint32_t cta_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cta_addr(const void* p, int cta) {  // the same variable in the shared memory of a CTA of the pair
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(cta));
  return a;
}
__device__ __forceinline__ void pair_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// A box of rows into this CTA's shared memory; the bytes complete on the leader's barrier
__device__ __forceinline__ void pair_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar) : "memory");
}
__device__ __forceinline__ void pair_load_2d(void* dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(c0), "r"(c1), "r"(bar) : "memory");
}
__device__ __forceinline__ void pair_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, e;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "elect.sync _|e, 0xFFFFFFFF;\n\t"
      "@e tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// arrives on the barriers `own` and `peer` (the same one in the other CTA) once the MMAs issued so far are done
__device__ __forceinline__ void pair_commit(uint32_t own, uint32_t peer) {
  asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xFFFFFFFF;\n\t"
               "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t"
               "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%1];\n\t}" ::"r"(own), "r"(peer) : "memory");
}
__device__ __forceinline__ void remote_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool all_of_256(bool mine) {                // of the eight epilogue warps
  uint32_t all;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbarrier.cta.red.and.pred q, 3, 256, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
               : "=r"(all) : "r"((uint32_t)mine) : "memory");
  return all != 0;
}
__device__ __forceinline__ int tile_cols(int n_rows) { return (n_rows + 63) & ~63; }       // N of the tile's MMAs

template <bool GATED>
__global__ void __launch_bounds__(PTHREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tma_x, const __grid_constant__ CUtensorMap tma_x64,
                 const __grid_constant__ CUtensorMap tma_x32, const __grid_constant__ CUtensorMap tma_w, const __grid_constant__ CUtensorMap tma_w2, const PairArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[PSTAGES], empty_bar[PSTAGES], acc_full[2], acc_empty[2];
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_abort;
  uint8_t* smem = smem_raw + (1024 - (smem_u32(smem_raw) & 1023)) % 1024;
  float* const swap = reinterpret_cast<float*>(smem + PSTAGES * P_STAGE);        // [2 groups of four warps][2 chunks][up, gate][16 tokens][64 outputs]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cta_rank();
  if (threadIdx.x == 0) {
    for (int s = 0; s < PSTAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 16); }
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  pair_sync();                                     // the peer's barriers are set up, and its tensor memory is there
  tc_fence_after();
  pdl_wait();
  pdl_launch();
  const uint32_t tmem_base = s_tmem_base;
  volatile int* abort_flag = &s_abort;

  const int n_tt = min(*a.n_tiles, a.max_tiles);
  const int total = n_tt * a.tiles_w, kblocks = a.K / PK;
  const int first = blockIdx.x / 2, step = gridDim.x / 2;

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0, issued = 0;
      uint32_t phase = 0;
      for (int t = first; t < total && !*abort_flag; t += step) {
        const PTile mt = a.tiles[t / a.tiles_w];
        const int half = tile_cols(min(PN, mt.row_end - mt.row0)) / 2;           // tokens of this CTA
        const int x0 = mt.row0 + (int)rank * half;
        const int n0 = (t % a.tiles_w) * (GATED ? 128 : PM) + (int)rank * (GATED ? 64 : 128);
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag)) break;
          uint8_t* sa = smem + (size_t)stage * P_STAGE;
          uint8_t* sb = sa + P_A_BYTES;
          if (rank == 0) mbar_expect_tx(&full_bar[stage], 2 * (P_A_BYTES + half * PK * 2));
          const uint32_t bar = cta_addr(&full_bar[stage], 0);
          pair_load_3d(sa, &tma_w, kb * PK, n0, mt.group, bar);
          if (GATED) pair_load_3d(sa + P_A_BYTES / 2, &tma_w2, kb * PK, n0, mt.group, bar);
          if (half == 128) {
            pair_load_2d(sb, &tma_x, kb * PK, x0, bar);
          } else {
            int r = 0;
            if (half >= 64) { pair_load_2d(sb, &tma_x64, kb * PK, x0, bar); r = 64; }
            if (r < half) pair_load_2d(sb + r * PK * 2, &tma_x32, kb * PK, x0 + r, bar);
          }
          ++issued;
          if (++stage == PSTAGES) { stage = 0; phase ^= 1; }
        }
      }
      if (*abort_flag) {
        // copies of this thread may still be landing in shared memory: the CTA must not exit under them
        unsigned long long t0 = globaltimer();
        while (issued > 0 && globaltimer() - t0 < 2000000ull) {}
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {
      const uint32_t empty0 = cta_addr(&empty_bar[0], 0), empty1 = cta_addr(&empty_bar[0], 1);
      const uint32_t full0 = cta_addr(&acc_full[0], 0), full1 = cta_addr(&acc_full[0], 1);
      int stage = 0, it = 0;
      uint32_t phase = 0;
      for (int t = first; t < total; t += step) {
        const PTile mt = a.tiles[t / a.tiles_w];
        const uint32_t idesc = umma_idesc(PM, tile_cols(min(PN, mt.row_end - mt.row0)));
        const int ab = it & 1;
        const uint32_t acc_phase = (it >> 1) & 1;
        ++it;
        if (!mbar_wait_warp(&acc_empty[ab], acc_phase ^ 1, abort_flag)) break;
        tc_fence_after();
        const uint32_t d0 = tmem_base + ab * PN;
        bool ok = true;
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait_warp(&full_bar[stage], phase, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + (size_t)stage * P_STAGE);
          const uint64_t da = umma_desc(sa), db = umma_desc(sa + P_A_BYTES);
#pragma unroll
          for (int k = 0; k < PK / UMMA_K; ++k)
            pair_mma(d0, da + (uint64_t)(k * UMMA_K * 2 / 16), db + (uint64_t)(k * UMMA_K * 2 / 16), idesc, (kb > 0 || k > 0) ? 1u : 0u);
          pair_commit(empty0 + stage * 8, empty1 + stage * 8);       // free in both CTAs once these MMAs have read it
          if (++stage == PSTAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        pair_commit(full0 + ab * 8, full1 + ab * 8);
      }
    }
  } else {
    const int q = warp & 3, grp = (warp - 2) >> 2;   // TMEM lane quarter of this warp; which chunks of 32 tokens it stores
    const uint32_t release = cta_addr(&acc_empty[0], 0);
    int it = 0, chunk = 0;
    for (int t = first; t < total; t += step) {
      const PTile mt = a.tiles[t / a.tiles_w];
      const int n_rows = min(PN, mt.row_end - mt.row0);
      const int n = (t % a.tiles_w) * (GATED ? 128 : PM) + (int)rank * (GATED ? 64 : 128) + (GATED ? (q & 1) * 32 : q * 32) + lane;
      const int ab = it & 1;
      const uint32_t acc_phase = (it >> 1) & 1;
      ++it;
      // lane l fetches the routing of token rows l, l + 32, ... while the products run
      int out_row[PN / 32];
      float out_scale[PN / 32];
#pragma unroll
      for (int b = 0; b < PN / 32; ++b) {
        const int r = mt.row0 + 32 * b + lane;
        out_row[b] = -1;
        out_scale[b] = 1.0f;
        if (32 * b + lane < n_rows) {
          out_row[b] = a.dst_row ? a.dst_row[r] : r;
          if (a.out.row_scale) out_scale[b] = a.out.row_scale[r];
        }
      }
      // the warps go on, or give up, together: they meet at barriers below
      if (!all_of_256(mbar_wait_warp(&acc_full[ab], acc_phase, abort_flag))) break;
      tc_fence_after();
      const uint32_t tbase = tmem_base + ((uint32_t)(q * 32) << 16) + ab * PN;
#pragma unroll
      for (int b = 0; b < PN / 32; ++b) {
        if (32 * b >= n_rows) break;
        if ((b & 1) != grp) continue;
        uint32_t v[32];
        tmem_ld32(tbase + 32 * b, v);
        tmem_ld_wait();
        if constexpr (GATED) {
          // warps 0 and 1 of the quarters hold the gate's products, 2 and 3 the up products of the same outputs: the former
          // finish tokens 0 .. 15 of the chunk and hand over their 16 .. 31, the latter the other way round
          float* const up = swap + (grp * 2 + (chunk & 1)) * 2 * P_SWAP;
          float* const gate = up + P_SWAP;
          ++chunk;
          const int col = (q & 1) * 32 + lane;
          float* const give = q < 2 ? gate : up;
          const float* const take = q < 2 ? up : gate;
#pragma unroll
          for (int i = 0; i < 16; ++i) give[i * 64 + col] = __uint_as_float(q < 2 ? v[16 + i] : v[i]);
          asm volatile("bar.sync %0, 128;" ::"r"(1 + grp) : "memory");
          float f[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float other = take[i * 64 + col];
            const float g = q < 2 ? __uint_as_float(v[i]) : other, u = q < 2 ? other : __uint_as_float(v[16 + i]);
            f[i] = (g / (1.0f + __expf(-g))) * u;
          }
          store_tokens<16>(a.out, f, out_row[b], out_scale[b], q < 2 ? 0 : 16, n);
        } else {
          float f[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) f[i] = __uint_as_float(v[i]);
          store_tokens<32>(a.out, f, out_row[b], out_scale[b], 0, n);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) remote_arrive(release + ab * 8);
    }
  }

  tc_fence_before();
  __syncthreads();
  __syncwarp();
  pair_sync();                                       // nobody leaves while the peer still arrives here or reads this memory
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
  }
  __syncwarp();
  pair_sync();
  if (threadIdx.x == 0 && s_abort && a.status) atomicMax(a.status, 1u);
}

// Pairs that this device holds at once: a pair lies within one GPC, whose processors may be odd in number.
static int gemm_pairs() {
  static std::atomic<int> known[64];
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64) return 0;
  if ((n = known[dev].load(std::memory_order_relaxed)) > 0) return n;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = 2;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.gridDim = dim3(2);
  cfg.blockDim = dim3(PTHREADS);
  cfg.dynamicSmemBytes = kPairSmem;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (cudaFuncSetAttribute(gemm_pair_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPairSmem) != cudaSuccess ||
      cudaFuncSetAttribute(gemm_pair_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPairSmem) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, gemm_pair_kernel<false>, &cfg) != cudaSuccess) return 0;
  known[dev].store(n, std::memory_order_relaxed);
  return n;
}

}  // namespace bl

using namespace bl;

extern "C" {

// C[dst_row[t] or t, n] = row_scale[t] * sum_k X[t, k] W[g][n, k] (+ resid), per token tile of the table.
//   X [rows_x, K] bf16 (ldx elements); W, W2 [n_groups, N, K] bf16; tiles: {group, row0, row_end, -} of at most 256 token rows;
//   exactly one of c_f32 / c_bf16; W2 != null: output = silu(X W^T) * (X W2^T), no resid.
//   status: device word, set to 1 if a wait ran out.
int bl_gemm_pair(const void* X, long ldx, long rows_x, const void* W, const void* W2, int n_groups, int N, int K,
                 const void* tiles, const int* n_tiles, int max_tiles, float* c_f32, void* c_bf16, long ldc,
                 const int* dst_row, const float* row_scale, const float* resid, long ldr, unsigned* status, cudaStream_t st) {
  BL_REQUIRE(K >= PK && K % PK == 0 && N >= 1 && rows_x >= 1 && n_groups >= 1 && max_tiles >= 1 && ldx % 8 == 0, BL_ERR_SHAPE);
  BL_REQUIRE((c_f32 != nullptr) != (c_bf16 != nullptr) && !(W2 && resid) && ldc >= 0 && ldr >= 0 && ldc < 1L << 30 && ldr < 1L << 30, BL_ERR_SHAPE);
  BL_REQUIRE(X && W && (((uintptr_t)X | (uintptr_t)W | (uintptr_t)W2) & 15) == 0, BL_ERR_ALIGN);
  CUtensorMap mx, mx64, mx32, mw, mw2;
  {
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows_x};
    cuuint64_t str[1] = {(cuuint64_t)ldx * 2};
    cuuint32_t box[2] = {PK, 128}, box64[2] = {PK, 64}, box32[2] = {PK, 32};
    int rc = make_map(&mx, X, 2, dims, str, box);
    if (rc) return rc;
    rc = make_map(&mx64, X, 2, dims, str, box64);
    if (rc) return rc;
    rc = make_map(&mx32, X, 2, dims, str, box32);
    if (rc) return rc;
  }
  {
    cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)N, (cuuint64_t)n_groups};
    cuuint64_t str[2] = {(cuuint64_t)K * 2, (cuuint64_t)K * 2 * (cuuint64_t)N};
    cuuint32_t box[3] = {PK, (cuuint32_t)(W2 ? 64 : 128), 1};
    int rc = make_map(&mw, W, 3, dims, str, box);
    if (rc) return rc;
    rc = make_map(&mw2, W2 ? W2 : W, 3, dims, str, box);
    if (rc) return rc;
  }
  PairArgs a{};
  a.N = N; a.K = K;
  a.tiles_w = W2 ? (N + 127) / 128 : (N + PM - 1) / PM;
  a.tiles = (const PTile*)tiles; a.n_tiles = n_tiles; a.max_tiles = max_tiles;
  a.dst_row = dst_row; a.status = status;
  a.out = TokenOut{c_f32, (__nv_bfloat16*)c_bf16, (unsigned)ldc, row_scale, resid, (unsigned)ldr, N};
  const int pairs = gemm_pairs();
  BL_REQUIRE(pairs >= 1, BL_ERR_LIMIT);
  const long most = (long)max_tiles * a.tiles_w;
  const int grid = 2 * (int)(most < pairs ? most : pairs);
  return (int)launch_cluster(W2 ? gemm_pair_kernel<true> : gemm_pair_kernel<false>, dim3(grid), dim3(PTHREADS), kPairSmem, 2, st, mx, mx64, mx32, mw, mw2, a);
}

}  // extern "C"
