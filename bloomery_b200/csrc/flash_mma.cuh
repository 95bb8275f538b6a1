// One warp's share of split-K decode attention over f16 keys and values, on warp-level tensor-core tiles.
//
// A decode row has at most eight query heads per KV head, half of an m16n8k16 tile.  The other half holds what f16
// leaves of the fp32 operands: rows 0..7 of the A operand are the high halves, rows 8..15 the remainders, so one MMA
// yields both partial products and every thread adds its pair (accumulator registers c0 + c2, c1 + c3 belong to one
// head).  Queries are first scaled by a power of two per head to a largest element in [512, 1024), probabilities by
// 2^10: high half and remainder then keep 22 bits of every element that matters, and keys and values enter as they are
// stored.  No probability ever exists in 16 bits alone; against 64 bits the output's error is 3.8e-7 where the fp32 loop
// this takes the place of had 9.2e-7 (64 rows of about 2,000 positions, 32 query heads, 4 KV heads).
//
// A warp works alone: 16 keys a step through its own cp.async ring, no barrier inside the loop.  The fp32 loop was bound
// by its multiply-adds and shuffles (one key a lane for the scores, 32 shuffles a tile for the values).
#pragma once
#include "common.cuh"

namespace bl {

__device__ __forceinline__ void wf_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void wf_ldsm4(uint32_t (&r)[4], const void* p) {
  const unsigned addr = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void wf_ldsm4_t(uint32_t (&r)[4], const void* p) {
  const unsigned addr = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// f16x2 of (x, y) and of what it leaves
__device__ __forceinline__ void wf_split(float x, float y, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(x, y);
  const float2 f = __half22float2(h);
  const __half2 r = __floats2half2_rn(x - f.x, y - f.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&r);
}

// The two partial products of one element.  An infinite key or value makes the remainder's product 0 * inf; the high one
// is then the answer, as in a plain fp32 sum (a key of score -inf weighs nothing, an infinite value stays infinite).
__device__ __forceinline__ float wf_join(float hi, float lo) { return fabsf(hi) < INFINITY ? hi + lo : hi; }
// The maximum that a NaN gets through: the vote on a new maximum then finds such a step, which costs the others nothing
// (joining every score took 6 % of a row of 16,000 keys).
__device__ __forceinline__ float wf_max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

template <int HEAD>
struct WarpFlash {
  static constexpr int kKeys = 16;                       // keys a step
  static constexpr int kStr = HEAD + 8;                  // f16 row stride: ldmatrix rows fall into different banks
  static constexpr int kTile = kKeys * kStr;             // f16 values of a key (or value) tile
  static constexpr int kStageBytes = 2 * kTile * 2;      // a key tile and a value tile
  static constexpr int KS = HEAD / 16, ND = HEAD / 8;
  static constexpr int kOut = HEAD + 8;                  // floats of a result row: eight rows start in different banks
  static_assert(kStageBytes >= 8 * kOut * 4, "a stage also holds the warp's result");
  uint32_t qa[KS][4];
  float q_inv;                                           // undoes the head's power of two
  float o[ND][4], m, l;                                  // m: of head lane / 4; l: this thread's share of the sum

  static constexpr int kQ = HEAD + 8;                    // floats from one query row to the next: as for kOut (rows of HEAD:
                                                         // 0.6 us more for a row of 12,000 keys)

  // queries of the KV head's group: G <= 8 rows of HEAD floats in shared memory, kQ apart
  __device__ __forceinline__ void init(const float* sq, int G, int lane) {
    const int g = lane >> 2, t = lane & 3;
    const float* q = sq + g * kQ + 2 * t;
    float2 x[HEAD / 8];
    float mx = 0.f;
#pragma unroll
    for (int i = 0; i < HEAD / 8; ++i) {
      x[i] = g < G ? *reinterpret_cast<const float2*>(q + 8 * i) : make_float2(0.f, 0.f);
      mx = fmaxf(mx, fmaxf(fabsf(x[i].x), fabsf(x[i].y)));
    }
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const int e = (int)(__float_as_uint(mx) >> 23);      // 127 + floor(log2)
    const int f = min(253, max(1, 263 - e));
    const float sc = __uint_as_float((uint32_t)f << 23);
    q_inv = __uint_as_float((uint32_t)(254 - f) << 23);
#pragma unroll
    for (int k = 0; k < KS; ++k) {
      wf_split(x[2 * k].x * sc, x[2 * k].y * sc, qa[k][0], qa[k][1]);
      wf_split(x[2 * k + 1].x * sc, x[2 * k + 1].y * sc, qa[k][2], qa[k][3]);
    }
    reset();
  }

  // no keys yet, the same queries
  __device__ __forceinline__ void reset() {
#pragma unroll
    for (int j = 0; j < ND; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
    m = -INFINITY; l = 0.f;
  }

  // 16 rows of keys or values into a tile; rows from n_valid on become zeros (they are not read)
  static __device__ __forceinline__ void issue_tile(__half* tile, const __half* src, int n_valid, int lane) {
    constexpr int CH = HEAD / 8;
#pragma unroll
    for (int c = lane; c < kKeys * CH; c += 32) {
      const int r = c / CH, cc = c % CH;
      const unsigned d = (unsigned)__cvta_generic_to_shared(tile + r * kStr + cc * 8);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src + (long)r * HEAD + cc * 8), "r"(r < n_valid ? 16u : 0u) : "memory");
    }
  }
  // 16 key rows and value rows into a stage
  static __device__ __forceinline__ void issue(__half* stage, const __half* k, const __half* v, int n_valid, int lane) {
    issue_tile(stage, k, n_valid, lane);
    issue_tile(stage + kTile, v, n_valid, lane);
  }

  // partial products of a tile of keys
  __device__ __forceinline__ void products(const __half* keys, int lane, float (&c)[2][2][4]) const {
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int h = 0; h < 2; ++h) c[nt][h][0] = c[nt][h][1] = c[nt][h][2] = c[nt][h][3] = 0.f;
#pragma unroll
    for (int kp = 0; kp < KS / 2; ++kp)
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        uint32_t b[4];
        wf_ldsm4(b, keys + (nt * 8 + (lane & 7)) * kStr + (kp * 4 + (lane >> 3)) * 8);
        wf_mma(c[nt][0], qa[2 * kp][0], qa[2 * kp][1], qa[2 * kp][2], qa[2 * kp][3], b[0], b[1]);
        wf_mma(c[nt][1], qa[2 * kp + 1][0], qa[2 * kp + 1][1], qa[2 * kp + 1][2], qa[2 * kp + 1][3], b[2], b[3]);
      }
  }
  // scores of the first n_valid keys (-inf for the others); their maximum a NaN gets through
  __device__ __forceinline__ float scores(const float (&c)[2][2][4], int n_valid, int lane, float (&s)[2][2]) const {
    const int t = lane & 3;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float x = ((c[nt][0][i] + c[nt][1][i]) + (c[nt][0][2 + i] + c[nt][1][2 + i])) * q_inv;
        s[nt][i] = nt * 8 + 2 * t + i < n_valid ? x : -INFINITY;
      }
    float nm = wf_max_nan(wf_max_nan(s[0][0], s[0][1]), wf_max_nan(s[1][0], s[1][1]));
    nm = wf_max_nan(nm, __shfl_xor_sync(0xffffffffu, nm, 1));
    return wf_max_nan(nm, __shfl_xor_sync(0xffffffffu, nm, 2));
  }
  // the same joined: an infinite key (or a NaN, which stays one)
  __device__ __forceinline__ float scores_joined(const float (&c)[2][2][4], int n_valid, int lane, float (&s)[2][2]) const {
    const int t = lane & 3;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float x = wf_join(c[nt][0][i] + c[nt][1][i], c[nt][0][2 + i] + c[nt][1][2 + i]) * q_inv;
        s[nt][i] = nt * 8 + 2 * t + i < n_valid ? x : -INFINITY;
      }
    float nm = fmaxf(fmaxf(s[0][0], s[0][1]), fmaxf(s[1][0], s[1][1]));
    nm = fmaxf(nm, __shfl_xor_sync(0xffffffffu, nm, 1));
    return fmaxf(nm, __shfl_xor_sync(0xffffffffu, nm, 2));
  }
  // a new maximum
  __device__ __forceinline__ void rescale(float nm) {
    const float corr = (m == -INFINITY) ? 0.f : __expf(m - nm);
    l *= corr;
#pragma unroll
    for (int j = 0; j < ND; ++j) { o[j][0] *= corr; o[j][1] *= corr; o[j][2] *= corr; o[j][3] *= corr; }
    m = nm;
  }
  // scores, with the maximum they bring
  __device__ __forceinline__ void softmax(const float (&c)[2][2][4], int n_valid, int lane, float (&s)[2][2]) {
    float nm = wf_max_nan(m, scores(c, n_valid, lane, s));
    if (__any_sync(0xffffffffu, nm != m)) {
      if (__any_sync(0xffffffffu, nm != nm)) nm = fmaxf(m, scores_joined(c, n_valid, lane, s));
      rescale(nm);
    }
  }
  // probabilities of a tile's scores under the maximum, times its values
  __device__ __forceinline__ void values(const float (&s)[2][2], const __half* v, int lane) {
    uint32_t a[4];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      const float p0 = (s[nt][0] == -INFINITY) ? 0.f : __expf(s[nt][0] - m);
      const float p1 = (s[nt][1] == -INFINITY) ? 0.f : __expf(s[nt][1] - m);
      l += p0 + p1;
      wf_split(p0 * 1024.f, p1 * 1024.f, a[2 * nt], a[2 * nt + 1]);
    }
#pragma unroll
    for (int dp = 0; dp < ND / 2; ++dp) {
      uint32_t b[4];
      wf_ldsm4_t(b, v + (lane & 15) * kStr + (2 * dp + (lane >> 4)) * 8);
      wf_mma(o[2 * dp], a[0], a[1], a[2], a[3], b[0], b[1]);
      wf_mma(o[2 * dp + 1], a[0], a[1], a[2], a[3], b[2], b[3]);
    }
  }

  // one step over a landed stage; the first n_valid (>= 1) keys count
  __device__ __forceinline__ void step(const __half* stage, int n_valid, int lane) {
    float c[2][2][4], s[2][2];
    products(stage, lane, c);
    softmax(c, n_valid, lane, s);
    values(s, stage + kTile, lane);
  }

  // this warp's sum and output under the maximum `top` of several warps, added to theirs (what store and wf_merge do for dims
  // 8 j + 2 (lane % 4) and the one behind of head lane / 4)
  __device__ __forceinline__ void add_to(float (&part)[ND][2], float& sum, float top) {
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    const float k = (m == -INFINITY) ? 0.f : __expf(m - top);
    sum = fmaf(l, k, sum);
#pragma unroll
    for (int j = 0; j < ND; ++j) {
      part[j][0] = fmaf(wf_join(o[j][0], o[j][2]) * (1.f / 1024.f), k, part[j][0]);
      part[j][1] = fmaf(wf_join(o[j][1], o[j][3]) * (1.f / 1024.f), k, part[j][1]);
    }
  }

  // the warp's maxima and sums [8] and unnormalised outputs [8][kOut] for the block's merge
  __device__ __forceinline__ void store(float* ml, float* out, int lane) {
    const int g = lane >> 2, t = lane & 3;
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    if (t == 0) { ml[2 * g] = m; ml[2 * g + 1] = l; }
#pragma unroll
    for (int j = 0; j < ND; ++j)
      *reinterpret_cast<float2*>(out + g * kOut + 8 * j + 2 * t) =
          make_float2(wf_join(o[j][0], o[j][2]) * (1.f / 1024.f), wf_join(o[j][1], o[j][3]) * (1.f / 1024.f));
  }
};

// Head hg of the results that n_w (up to eight) warps left, the w-th at slot s = (first + w) & mask, ml + 16 s and
// out + s * stride: lane's HEAD / 32 dims, the maximum and the sum, warps in ascending order.
template <int HEAD>
__device__ __forceinline__ void wf_merge(const float* ml, const float* out, size_t stride, int n_w, int hg, int lane,
                                         float (&acc)[HEAD / 32], float& m, float& l, int first = 0, int mask = 15) {
  constexpr int DPL = HEAD / 32;
  float mw = -INFINITY, lw = 0.f, o[8][DPL];             // lane w: maximum and sum of warp w
  if ((lane & 7) < n_w) {
    const float2 v = *reinterpret_cast<const float2*>(ml + 16 * ((first + (lane & 7)) & mask) + 2 * hg);
    mw = fmaxf(mw, v.x); lw = v.y;
  }
#pragma unroll
  for (int w = 0; w < 8; ++w)
    if (w < n_w) {
      const float* src = out + ((first + w) & mask) * stride + hg * WarpFlash<HEAD>::kOut + lane * DPL;
      if constexpr (DPL == 4) {
        const float4 v = *reinterpret_cast<const float4*>(src);
        o[w][0] = v.x; o[w][1] = v.y; o[w][2] = v.z; o[w][3] = v.w;
      } else {
        const float2 v = *reinterpret_cast<const float2*>(src);
        o[w][0] = v.x; o[w][1] = v.y;
      }
    }
  m = mw;
#pragma unroll
  for (int off = 1; off < 8; off <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
  const float k = (mw == -INFINITY) ? 0.f : __expf(mw - m);
  l = 0.f;
#pragma unroll
  for (int d = 0; d < DPL; ++d) acc[d] = 0.f;
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    const float kw = __shfl_sync(0xffffffffu, k, w), ls = __shfl_sync(0xffffffffu, lw, w);
    if (w < n_w) {
      l = fmaf(ls, kw, l);
#pragma unroll
      for (int d = 0; d < DPL; ++d) acc[d] = fmaf(o[w][d], kw, acc[d]);
    }
  }
}

}  // namespace bl
