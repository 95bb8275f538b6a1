// Prompt (prefill) flash attention on the 5th-generation tensor cores: scores and the output accumulator live in
// tensor memory, the probabilities go from registers back into the columns of their scores and from there into the second
// product, and nothing of the score matrix ever reaches HBM.
//
// One CTA = two tiles of 128 query positions (the 128 lanes of tensor memory) that read the same keys: two query heads of
// one KV head, as a rule.  Their softmaxes and products take turns, so that one tile's exponentials (16,384 at 16 a clock a
// processor, as long as its MMAs) run under the other's products, and a key / value tile is fetched once for both.
// Per tile and 128 keys:
//   S = Q K^T          tcgen05.mma kind::f16, M = N = 128, depth 128 (two 64-wide swizzle atoms), into TMEM
//   softmax            one thread per query row: the row's scores stay in registers between the maximum and the
//                      exponentials (running max / sum in base 2, causal mask on the diagonal tiles); the probabilities go
//                      back as bf16 into the score columns they came from
//   O = O * corr       the running output is rescaled in TMEM (tcgen05.ld / tcgen05.st) and only when the row maximum moved
//                      by more than 2^8: until then the old maximum keeps scaling the exponentials (they stay below 2^8, far
//                      inside fp32 and bf16), so most tiles skip the round trip
//   O += P V           tcgen05.mma with P as the A operand in tensor memory and the (dims x keys) value tile as B
// Tensor memory is full: scores and output of both tiles, 128 columns each.  The issuer runs P V of key tile t and then Q K^T
// of t + 1 for one tile, then for the other.  MMAs of one thread execute in order: the new scores replace the probabilities
// behind the product that reads them, and a commit behind Q K^T says that the P V in front of it is complete too.
// One tile a CTA with two threads a row took 234 us a layer for 4,096 tokens of the 30 B shape (32 heads over 4) and 258 us for 700
// behind 9,000; this takes 140 and 174.
// A few hundred queries behind a long prefix are fewer CTAs than processors, each with a long walk over the keys: there
// `splits` CTAs share the key tiles of a pair.  Each leaves its unnormalised output, maximum and sum of every row in a buffer,
// and the warp that arrives last at its 32 rows (a ticket) adds the parts up in ascending order, its own out of tensor memory.
// 700 queries behind 9,000 keys: 96 CTAs of 76 key tiles, 174 us; 288 of 25, 130 us.
// Roles: warps 0..3 softmax of the first tile, 4..7 of the second (warp id modulo 4 = TMEM lane quarter), warp 8 the TMA
// producer (two-stage rings for keys and values), warp 9 the MMA issuer and TMEM owner.  Every TMA load is a plain tile load
// of this GPU's own memory.
//
// Inputs are what the prompt path already builds: queries bf16 [n_q][T][128] (normalised, rotated, pre-scaled),
// keys bf16 [n_kv][t_pad][128], values transposed bf16 [n_kv][128][t_pad]; output bf16 [T][n_q * 128].
// Every wait is bounded (1 s); on expiry the CTA raises the status word, frees its TMEM and returns.
//
// Reference counterpart: crates/gpu/src/flash_gqa_prefill.rs:1-80 (mma.sync m16n8k16 tiles, cp.async staging).
#include "tc_common.cuh"

namespace bl {

constexpr int FQ = 128, FKEYS = 128, FD = 128;
constexpr int FATOM = 64;                               // bf16 values per 128-byte swizzle row
constexpr int FHALF = 128 * FATOM * 2;                  // 16 KiB: 128 rows x 64 values
constexpr int FTILE = 2 * FHALF;                        // 32 KiB: a 128 x 128 bf16 tile as two swizzle atoms
constexpr int FSMEM = 2 * FTILE /*Q*/ + 2 * FTILE /*K*/ + 2 * FTILE /*V*/ + 1024 /*alignment*/;
constexpr float kLog2e = 1.4426950408889634f;

struct FlashPrefillArgs {
  int T, n_q, n_kv, group;    // query rows per head; heads; KV heads; query heads per KV head
  int pos0;                   // position of query row 0 (keys 0 .. pos0 + T - 1 exist)
  int t_pad;                  // key rows per KV head in K = key columns per row in Vt
  __nv_bfloat16* out; long ldo;
  unsigned* status;
  int splits;                 // CTAs that share a pair's keys
  float4* part;               // splits > 1: [pair][split][tile][column / 4][row] unnormalised outputs
  float2* part_ml;            // [pair][split][tile][row]: maximum, sum
  int* tickets;               // [pair][tile][4 warps], zero between launches
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 p = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&p);
}

constexpr int FTHREADS = 320;
constexpr int kMaxSplits = 4;
constexpr float kLazy = 8.0f;                           // the maximum may lag by 2^8 before the output is rescaled

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
               "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}

__global__ void __launch_bounds__(FTHREADS, 1)
flash_prefill_kernel(const __grid_constant__ CUtensorMap tma_q, const __grid_constant__ CUtensorMap tma_k,
                     const __grid_constant__ CUtensorMap tma_v, const FlashPrefillArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t q_full, k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], p_full[2], o_done[2];
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_abort;
  uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sQ = smem;                // [2 tiles][2 halves]
  uint8_t* sK = sQ + 2 * FTILE;      // [2 stages][2 halves]
  uint8_t* sV = sK + 2 * FTILE;      // [2 stages][2 halves]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Query tiles of a KV head in descending order of position, its heads side by side: tile i = heads i % group at
  // position tile n_qt - 1 - i / group.  A CTA takes two that follow each other; the ones with the most keys start first.
  const int n_qt = (a.T + FQ - 1) / FQ;
  const int pair = (int)blockIdx.x / a.splits, split = (int)blockIdx.x % a.splits;
  const int kvh = pair % a.n_kv, item0 = 2 * (pair / a.n_kv);
  const int n_x = item0 + 1 < n_qt * a.group ? 2 : 1;           // tiles of this CTA
  auto tile_q0 = [&](int x) { return (n_qt - 1 - (item0 + x) / a.group) * FQ; };
  auto tile_head = [&](int x) { return kvh * a.group + (item0 + x) % a.group; };
  const int last_q = a.pos0 + min(tile_q0(0) + FQ, a.T) - 1;    // position of the first tile's last query: no other is later
  const int all_t = last_q / FKEYS + 1;                         // key tiles of the pair
  const int t_lo = all_t * split / a.splits, n_t = all_t * (split + 1) / a.splits - t_lo;   // this CTA's: t_lo .. t_lo + n_t - 1
  // A second tile one position earlier (an odd number of heads) ends a key tile earlier: it must not meet the values behind it,
  // where a probability of zero times infinity is NaN.  A share holds two key tiles when it is the last, so never none of its.
  auto tiles_of = [&](int x) { return min(n_t, (a.pos0 + min(tile_q0(x) + FQ, a.T) - 1) / FKEYS + 1 - t_lo); };

  if (threadIdx.x == 0) {
    mbar_init(&q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1); mbar_init(&p_full[i], 4); mbar_init(&o_done[i], 1);
    }
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  pdl_launch();
  const uint32_t tmem_base = s_tmem_base;
  volatile int* abort_flag = &s_abort;
  const uint32_t tS0 = tmem_base, tO0 = tmem_base + 256;        // scores of tile x at column 128 x, its output at 256 + 128 x

  if (warp == 8) {
    if (lane == 0) {
      mbar_expect_tx(&q_full, n_x * FTILE);
      for (int x = 0; x < n_x; ++x) {
        tma_load_2d(sQ + x * FTILE, &tma_q, 0, tile_head(x) * a.T + tile_q0(x), &q_full);
        tma_load_2d(sQ + x * FTILE + FHALF, &tma_q, FATOM, tile_head(x) * a.T + tile_q0(x), &q_full);
      }
      for (int t = 0; t < n_t && !*abort_flag; ++t) {
        const int st = t & 1;
        const uint32_t par = (uint32_t)((t >> 1) & 1);
        if (!mbar_wait(&k_empty[st], par ^ 1, abort_flag)) break;
        mbar_expect_tx(&k_full[st], FTILE);
        tma_load_2d(sK + st * FTILE, &tma_k, 0, kvh * a.t_pad + (t_lo + t) * FKEYS, &k_full[st]);
        tma_load_2d(sK + st * FTILE + FHALF, &tma_k, FATOM, kvh * a.t_pad + (t_lo + t) * FKEYS, &k_full[st]);
        if (!mbar_wait(&v_empty[st], par ^ 1, abort_flag)) break;
        mbar_expect_tx(&v_full[st], FTILE);
        tma_load_2d(sV + st * FTILE, &tma_v, (t_lo + t) * FKEYS, kvh * FD, &v_full[st]);
        tma_load_2d(sV + st * FTILE + FHALF, &tma_v, (t_lo + t) * FKEYS + FATOM, kvh * FD, &v_full[st]);
      }
      if (*abort_flag) {
        // copies of ours may still be landing: give them a bounded moment before the block's memory goes away
        const unsigned long long t0 = globaltimer();
        while (globaltimer() - t0 < 2000000ull) { }
      }
    }
  } else if (warp == 9) {
    constexpr uint32_t idesc = umma_idesc(FQ, FKEYS);
    auto qk = [&](int x, int st) {
      const uint64_t dQ0 = umma_desc(smem_u32(sQ + x * FTILE)), dQ1 = umma_desc(smem_u32(sQ + x * FTILE + FHALF));
      const uint64_t dK0 = umma_desc(smem_u32(sK + st * FTILE)), dK1 = umma_desc(smem_u32(sK + st * FTILE + FHALF));
      const uint32_t tS = tS0 + x * FKEYS;
#pragma unroll
      for (int k = 0; k < FATOM / UMMA_K; ++k) umma_bf16(tS, dQ0 + (uint64_t)(k * 2), dK0 + (uint64_t)(k * 2), idesc, k > 0 ? 1u : 0u);
#pragma unroll
      for (int k = 0; k < FATOM / UMMA_K; ++k) umma_bf16(tS, dQ1 + (uint64_t)(k * 2), dK1 + (uint64_t)(k * 2), idesc, 1u);
      umma_commit(&s_full[x]);
    };
    bool ok = mbar_wait_warp(&q_full, 0, abort_flag) && mbar_wait_warp(&k_full[0], 0, abort_flag);
    const int n_tx[2] = {n_t, n_x > 1 ? tiles_of(1) : 0};
    if (ok) {
      tc_fence_after();
      for (int x = 0; x < n_x; ++x) qk(x, 0);
      umma_commit(&k_empty[0]);
    }
    for (int t = 0; ok && t < n_t; ++t) {
      const int st = t & 1, nx = (t + 1) & 1;
      const uint32_t par = (uint32_t)((t >> 1) & 1), nx_par = (uint32_t)(((t + 1) >> 1) & 1);
      const uint64_t dV0 = umma_desc(smem_u32(sV + st * FTILE)), dV1 = umma_desc(smem_u32(sV + st * FTILE + FHALF));
      for (int x = 0; x < n_x; ++x) {
        if (x == 0 && !mbar_wait_warp(&v_full[st], par, abort_flag)) { ok = false; break; }
        if (t < n_tx[x]) {
          if (!mbar_wait_warp(&p_full[x], (uint32_t)(t & 1), abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint32_t tP = tS0 + x * FKEYS, tO = tO0 + x * FD;
#pragma unroll
          for (int k = 0; k < FATOM / UMMA_K; ++k) umma_bf16_ta(tO, tP + k * 8, dV0 + (uint64_t)(k * 2), idesc, (t > 0 || k > 0) ? 1u : 0u);
#pragma unroll
          for (int k = 0; k < FATOM / UMMA_K; ++k) umma_bf16_ta(tO, tP + 32 + k * 8, dV1 + (uint64_t)(k * 2), idesc, 1u);
        }
        if (x == n_x - 1) umma_commit(&v_empty[st]);
        if (t + 1 < n_t && x == 0 && !mbar_wait_warp(&k_full[nx], nx_par, abort_flag)) { ok = false; break; }
        if (t + 1 < n_tx[x]) {
          tc_fence_after();
          qk(x, nx);
        } else if (t + 1 == n_tx[x]) {
          umma_commit(&o_done[x]);
        }
        if (t + 1 < n_t && x == n_x - 1) umma_commit(&k_empty[nx]);
      }
    }
  } else if ((warp >> 2) < n_x) {
    // ---- softmax: a thread per query row ------------------------------------------------------------------
    const int x = warp >> 2;
    const int q0 = tile_q0(x), h = tile_head(x), n_tx = tiles_of(x);
    const int r = (warp & 3) * 32 + lane;
    const int qrow = q0 + r;
    const int qpos = a.pos0 + qrow;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tS = tS0 + x * FKEYS + lane_base, tO = tO0 + x * FD + lane_base;
    float m = -INFINITY, l = 0.f;
    bool ok = true;
    for (int t = 0; t < n_tx; ++t) {
      ok = __all_sync(0xffffffffu, mbar_wait(&s_full[x], (uint32_t)(t & 1), abort_flag));
      if (!ok) break;
      tc_fence_after();
      uint32_t v[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld32(tS + 32 * c, v[c]);
      tmem_ld_wait();
      const int key0 = (t_lo + t) * FKEYS;
      if (key0 + FKEYS - 1 > a.pos0 + q0) {                     // some key of this tile lies past some query of it
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (key0 + 32 * c + i > qpos) v[c][i] = 0xff800000u;          // -inf
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};        // four chains instead of one
#pragma unroll
      for (int i = 0; i < 32; i += 2)
#pragma unroll
        for (int c = 0; c < 4; ++c) mx4[c] = fmaxf(fmaxf(mx4[c], __uint_as_float(v[c][i])), __uint_as_float(v[c][i + 1]));
      float m_new = fmaxf(m, fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])));
      if (m != -INFINITY && (m_new - m) * kLog2e <= kLazy) m_new = m;
      const float mb = (m_new == -INFINITY) ? 0.f : m_new * kLog2e;       // a row with no key yet keeps zeros
      const float corr = (m == -INFINITY) ? 0.f : ex2(m * kLog2e - mb);
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          // (s0, s1) * log2(e) - mb as one packed FMA; masked scores are -inf and 2^-inf = 0 (a row without any key
          // has mb = 0 and only -inf scores, so it needs no special case)
          uint32_t e0, e1;
          asm("{\n\t.reg .b64 rs, rk, rm, rr;\n\t"
              "mov.b64 rs, {%2, %3};\n\tmov.b64 rk, {%4, %4};\n\tmov.b64 rm, {%5, %5};\n\t"
              "fma.rn.f32x2 rr, rs, rk, rm;\n\tmov.b64 {%0, %1}, rr;\n\t}"
              : "=r"(e0), "=r"(e1) : "r"(v[c][i]), "r"(v[c][i + 1]), "f"(kLog2e), "f"(-mb));
          const float p0 = ex2(__uint_as_float(e0)), p1 = ex2(__uint_as_float(e1));
          sum[i & 2] += p0; sum[(i & 2) + 1] += p1;
          pk[i >> 1] = pack_bf16(p0, p1);
        }
        tmem_st16(tS + 16 * c, pk);
      }
      if (t > 0 && __any_sync(0xffffffffu, corr != 1.0f)) {     // the product of the last tile is complete: see above
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          uint32_t o[32];
          tmem_ld32(tO + c * 32, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
          tmem_st32(tO + c * 32, o);
        }
      }
      l = l * corr + ((sum[0] + sum[2]) + (sum[1] + sum[3]));
      m = m_new;
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[x]);
    }
    if (ok && __all_sync(0xffffffffu, mbar_wait(&o_done[x], 0, abort_flag))) {
      tc_fence_after();
      constexpr int PART = FD / 4 * FQ;                         // float4 of a tile's output
      const long base = ((long)pair * a.splits * 2 + x) * FQ;   // + 2 FQ a split
      bool mine = true;
      if (a.splits > 1) {
        float4* own = a.part + (((long)pair * a.splits + split) * 2 + x) * PART + r;
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          uint32_t o[32];
          tmem_ld32(tO + c * 32, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; i += 4)
            __stcg(own + (c * 8 + i / 4) * FQ, make_float4(__uint_as_float(o[i]), __uint_as_float(o[i + 1]), __uint_as_float(o[i + 2]),
                                                           __uint_as_float(o[i + 3])));
        }
        __stcg(a.part_ml + base + (long)split * 2 * FQ + r, make_float2(m, l));
        __threadfence();
        __syncwarp();
        int last = 0;
        if (lane == 0) {
          int* ticket = a.tickets + ((long)pair * 2 + x) * 4 + (warp & 3);
          last = atomicAdd(ticket, 1) == a.splits - 1;
          if (last) *ticket = 0;                                // ready for the next launch
        }
        mine = __shfl_sync(0xffffffffu, last, 0) != 0;
        if (mine) __threadfence();
      }
      if (mine) {
        float w[kMaxSplits];                                    // what each part counts, the normalisation included
        if (a.splits > 1) {
          float top = -INFINITY, all = 0.f;
#pragma unroll
          for (int sp = 0; sp < kMaxSplits; ++sp) {
            w[sp] = 0.f;
            if (sp < a.splits) {
              w[sp] = __ldcg(a.part_ml + base + (long)sp * 2 * FQ + r).x;
              top = fmaxf(top, w[sp]);
            }
          }
#pragma unroll
          for (int sp = 0; sp < kMaxSplits; ++sp)
            if (sp < a.splits) {
              w[sp] = w[sp] == -INFINITY ? 0.f : ex2((w[sp] - top) * kLog2e);
              all += w[sp] * __ldcg(a.part_ml + base + (long)sp * 2 * FQ + r).y;
            }
          const float inv = all > 0.f ? 1.0f / all : 0.f;
#pragma unroll
          for (int sp = 0; sp < kMaxSplits; ++sp) w[sp] *= inv;
        } else {
          w[0] = l > 0.f ? 1.0f / l : 0.f;
        }
        __nv_bfloat16* orow = a.out + (long)qrow * a.ldo + (long)h * FD;
        const float4* parts = a.part + ((long)pair * a.splits * 2 + x) * PART + r;
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          uint32_t v[32];
          tmem_ld32(tO + c * 32, v);
          tmem_ld_wait();
          float o[32];
          if (a.splits > 1) {
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = 0.f;
#pragma unroll 1
            for (int sp = 0; sp < a.splits; ++sp) {
              float ws = w[0];
#pragma unroll
              for (int k = 1; k < kMaxSplits; ++k) ws = sp == k ? w[k] : ws;
              if (sp == split) {
#pragma unroll
                for (int i = 0; i < 32; ++i) o[i] = fmaf(__uint_as_float(v[i]), ws, o[i]);
              } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                  const float4 q = __ldcg(parts + (long)sp * 2 * PART + (c * 8 + i) * FQ);
                  o[4 * i] = fmaf(q.x, ws, o[4 * i]); o[4 * i + 1] = fmaf(q.y, ws, o[4 * i + 1]);
                  o[4 * i + 2] = fmaf(q.z, ws, o[4 * i + 2]); o[4 * i + 3] = fmaf(q.w, ws, o[4 * i + 3]);
                }
              }
            }
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __uint_as_float(v[i]) * w[0];
          }
          if (qrow < a.T) {
#pragma unroll
            for (int i = 0; i < 32; i += 8)
              *reinterpret_cast<uint4*>(orow + c * 32 + i) = make_uint4(pack_bf16(o[i], o[i + 1]), pack_bf16(o[i + 2], o[i + 3]),
                                                                        pack_bf16(o[i + 4], o[i + 5]), pack_bf16(o[i + 6], o[i + 7]));
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
  }
  if (threadIdx.x == 0 && s_abort && a.status) atomicMax(a.status, 1u);
}

}  // namespace bl

using namespace bl;

extern "C" {

// Causal attention of T query rows per head (positions pos0 .. pos0 + T - 1) over keys 0 .. pos0 + T - 1.
//   q  bf16 [n_q][T][128]   k  bf16 [n_kv][t_pad][128]   vt  bf16 [n_kv][128][t_pad]   out  bf16 [T][ldo >= n_q * 128]
// t_pad is a multiple of 128 that covers the keys; value columns past the last key must be finite (zero).
// splits > 1 (up to 4; pos0 + 1 > 128 * splits, so that no share is empty): part holds 2 * pairs * splits * 16,384 floats,
// part_ml 2 * pairs * splits * 256, tickets 8 * pairs zeroed words, with pairs = n_kv * ceil(ceil(T / 128) * (n_q / n_kv) / 2); all
// of one stream at a time.
int bl_flash_prefill_split(const void* q, const void* k, const void* vt, void* out, long ldo, int T, int n_q, int n_kv, int pos0,
                           int t_pad, unsigned* status, int splits, float* part, float* part_ml, int* tickets, cudaStream_t st) {
  BL_REQUIRE(splits >= 1 && splits <= kMaxSplits && (splits == 1 || (pos0 >= 128 * splits && part && part_ml && tickets)), BL_ERR_SHAPE);
  BL_REQUIRE(((uintptr_t)part & 15) == 0 && ((uintptr_t)part_ml & 7) == 0, BL_ERR_ALIGN);
  BL_REQUIRE(T >= 1 && n_q >= 1 && n_kv >= 1 && n_q % n_kv == 0 && pos0 >= 0, BL_ERR_SHAPE);
  BL_REQUIRE(t_pad % 128 == 0 && t_pad >= pos0 + T && ldo >= (long)n_q * FD && ldo % 8 == 0, BL_ERR_SHAPE);
  BL_REQUIRE((((uintptr_t)q | (uintptr_t)k | (uintptr_t)vt | (uintptr_t)out) & 15) == 0, BL_ERR_ALIGN);
  CUtensorMap mq, mk, mv;
  {
    const cuuint64_t dims[2] = {(cuuint64_t)FD, (cuuint64_t)n_q * T};
    const cuuint64_t strides[1] = {(cuuint64_t)FD * 2};
    const cuuint32_t box[2] = {FATOM, FQ};
    int rc = make_map(&mq, q, 2, dims, strides, box);
    if (rc) return rc;
  }
  {
    const cuuint64_t dims[2] = {(cuuint64_t)FD, (cuuint64_t)n_kv * t_pad};
    const cuuint64_t strides[1] = {(cuuint64_t)FD * 2};
    const cuuint32_t box[2] = {FATOM, FKEYS};
    int rc = make_map(&mk, k, 2, dims, strides, box);
    if (rc) return rc;
  }
  {
    const cuuint64_t dims[2] = {(cuuint64_t)t_pad, (cuuint64_t)n_kv * FD};
    const cuuint64_t strides[1] = {(cuuint64_t)t_pad * 2};
    const cuuint32_t box[2] = {FATOM, FD};
    int rc = make_map(&mv, vt, 2, dims, strides, box);
    if (rc) return rc;
  }
  FlashPrefillArgs a{T, n_q, n_kv, n_q / n_kv, pos0, t_pad, (__nv_bfloat16*)out, ldo, status,
                     splits, (float4*)part, (float2*)part_ml, tickets};
  static PerDevice limit;
  if (limit.due()) {
    cudaFuncSetAttribute(flash_prefill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FSMEM);
    limit.mark();
  }
  const int items = (T + FQ - 1) / FQ * (n_q / n_kv);           // query tiles of a KV head
  dim3 grid((unsigned)((items + 1) / 2 * n_kv * splits));
  return (int)launch(flash_prefill_kernel, grid, dim3(FTHREADS), (size_t)FSMEM, st, mq, mk, mv, a);
}

}  // extern "C"
