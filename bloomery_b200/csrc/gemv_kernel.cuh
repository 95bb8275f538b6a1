// The kernel of the quantised GEMV (decode_gemv.cu), one translation unit a family of weight types.
#pragma once
#include "gemv_common.cuh"

namespace bl {

// ---- the rows of one warp ---------------------------------------------------------------
// A warp owns rows [r_lo, r_hi) of its segment and walks them R at a time; every load of a
// chunk is issued before anything is computed.  C = units per lane per inner step.
// `between` runs once per block, after the very first loads are in flight.
template <class T, int MB, int R, int C, class Between>
__device__ __forceinline__ void rows_q(const GemvArgs& a, const GemvSeg& s, int r_lo, int r_hi, int out_col0,
                                       const int8_t* sq, const float2* sds, const float* s_scale, Between&& between) {
  using U = Unit<T>;
  const int K = a.K, lane = threadIdx.x & 31;
  const int nunits = K / 64;
  constexpr bool PLANE_ROW = MB == 1 && (T::kType == WT_NVFP4 || T::kType == WT_FP8_B128);
  const unsigned push_epoch = a.push.n_ranks > 0 ? site_epoch(a.push.step, a.push.sites_per_step, a.push.site_index) : 0u;
  for (int r0 = r_lo; r0 < r_hi || r0 == r_lo; r0 += R) {
    float acc[R][MB];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int m = 0; m < MB; ++m) acc[r][m] = 0.f;
    for (int base = 0; base < nunits; base += 32 * C) {
      typename U::Regs regs[R][C];
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const int u = base + c * 32 + lane;
          // a weight row past the end is the segment's last one again; its result is dropped
          if (u < nunits && (!PLANE_ROW || r0 + r < r_hi)) U::loadu(s.w + (long)min(r0 + r, s.rows - 1) * s.row_bytes, u, K, regs[r][c]);
        }
      between();
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const int u = base + c * 32 + lane;
        if (u < nunits) {
          // No branch on the weight row: behind one, its codes and scales are taken apart again for every row m (eight rows of a 2,048
          // deep head: 351 us, 252 without).  One row of float planes has one, since their dots cost more than it saves.
#pragma unroll
          for (int m = 0; m < MB; ++m) {
            // the block's activation rows sit in the conflict-free chunk layout of its weight type
            ActRegs act;
            StagedAct<T>::load(sq + (long)m * K, sds + (long)m * (K / 32), u, nunits, act);
#pragma unroll
            for (int r = 0; r < R; ++r)
              if (!PLANE_ROW || r0 + r < r_hi) acc[r][m] = ActOf<T>::dot(regs[r][c], u, act, acc[r][m]);
          }
        }
      }
    }
    if constexpr (MB == 1 && R > 1) {
      // lane 8 r stores row r
      const float sum = warp_sum4(acc[0][0], acc[1][0], R > 2 ? acc[R - 1][0] : 0.f, 0.f);
      const int r = lane >> 3;
      if ((lane & 7) == 0 && r < R && r0 + r < r_hi) {
        const int col = out_col0 + r0 + r;
        float v = sum * s_scale[0];
        if (a.push.n_ranks > 0) push_store(a.push, push_epoch, col, v);
        else {
          if (a.resid) v += a.resid[col];
          a.out[col] = v;
        }
      }
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int m = 0; m < MB; ++m) acc[r][m] = warp_sum(acc[r][m]);
      if (lane == 0) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          if (r0 + r < r_hi) {
            const int col = out_col0 + r0 + r;
#pragma unroll
            for (int m = 0; m < MB; ++m)
              if (m < a.M) {
                float v = acc[r][m] * s_scale[m];
                if (a.push.n_ranks > 0) { push_store(a.push, push_epoch, (long)m * a.out_stride + col, v); continue; }
                if (a.resid) v += a.resid[(long)m * a.resid_stride + col];
                a.out[(long)m * a.out_stride + col] = v;
              }
          }
        }
      }
    }
    if (r0 + R >= r_hi) break;
  }
}

// The same for passes of several rows whose weight rows are at most 32 C units long: the weights of R rows stay in registers
// and the pass's rows walk past them one by one, so nothing is kept per (weight row, row of the pass) and the loop runs
// over live rows only.  Sums are those of rows_q.  Lane 8 r + m keeps the result of weight row r and row m and stores it at the end.
// (Accumulators of 2 x 8 instead spilled 1 KB a thread; five rows in a bucket of eight computed eight.)  The dots have no branch
// on the weight row, behind which its codes and scales would be taken apart once a row of the pass (head of 151,936 x 2,048, eight
// rows 230 us, 204 so); two units a lane are too many to be kept taken apart, so there two rows of the pass share that work
// (8,192 x 4,096 Q6_K, eight rows 33 us, 29 so).
template <class T, int R, int C, class Between>
__device__ __forceinline__ void rows_multi(const GemvArgs& a, const GemvSeg& s, int r_lo, int r_hi, int out_col0, unsigned live,
                                           const int8_t* sq, const float2* sds, const float* s_scale, Between&& between) {
  using U = Unit<T>;
  const int K = a.K, lane = threadIdx.x & 31;
  const int nunits = K / 64;
  const int my_m = lane & 7, my_r = lane >> 3;
  static_assert(R <= 4 && kMaxRows == 8, "a result a lane");
  constexpr int P = C == 2 && T::kType != WT_NVFP4 && T::kType != WT_FP8_B128 ? 2 : 1;
  const unsigned push_epoch = a.push.n_ranks > 0 ? site_epoch(a.push.step, a.push.sites_per_step, a.push.site_index) : 0u;
  for (int r0 = r_lo; r0 < r_hi || r0 == r_lo; r0 += R) {
    typename U::Regs regs[R][C];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int c = 0; c < C; ++c)
        if (c * 32 + lane < nunits) U::loadu(s.w + (long)min(r0 + r, s.rows - 1) * s.row_bytes, c * 32 + lane, K, regs[r][c]);
    between();
    const bool mine = my_r < R && r0 + my_r < r_hi && (live >> my_m & 1);
    const int col = out_col0 + r0 + my_r;
    float res = 0.f, old = 0.f;
    if (a.resid && a.push.n_ranks == 0 && mine) old = a.resid[(long)my_m * a.resid_stride + col];
#pragma unroll 1
    for (unsigned left = live; left;) {
      int ms[P];                     // the next rows; -1: there is none
#pragma unroll
      for (int i = 0; i < P; ++i) {
        ms[i] = __ffs(left) - 1;
        left &= left - 1;
      }
      float acc[P][R];
#pragma unroll
      for (int i = 0; i < P; ++i)
#pragma unroll
        for (int r = 0; r < R; ++r) acc[i][r] = 0.f;
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const int u = c * 32 + lane;
        if (u < nunits) {
#pragma unroll
          for (int i = 0; i < P; ++i) {
            if (i > 0 && ms[i] < 0) continue;
            ActRegs act;
            StagedAct<T>::load(sq + (long)ms[i] * K, sds + (long)ms[i] * (K / 32), u, nunits, act);
#pragma unroll
            for (int r = 0; r < R; ++r) acc[i][r] = ActOf<T>::dot(regs[r][c], u, act, acc[i][r]);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < P; ++i) {
        float sum;
        if constexpr (R == 1) sum = warp_sum(acc[i][0]);
        else sum = warp_sum4(acc[i][0], acc[i][1], R > 2 ? acc[i][R - 1] : 0.f, 0.f);
        if (my_m == ms[i]) res = sum;
      }
    }
    if (mine) {
      float v = res * s_scale[my_m];
      if (a.push.n_ranks > 0) {
        push_store(a.push, push_epoch, (long)my_m * a.out_stride + col, v);
      } else {
        if (a.resid) v += old;
        a.out[(long)my_m * a.out_stride + col] = v;
      }
    }
    if (r0 + R >= r_hi) break;
  }
}

// float weights (F32 / F16 / BF16) against fp32 x*gain rows
template <int MB, int R, class Between>
__device__ __forceinline__ void rows_f(const GemvArgs& a, const GemvSeg& s, int r_lo, int r_hi, int out_col0, unsigned live,
                                       const float* sx, const float* s_scale, Between&& between) {
  const int K = a.K, lane = threadIdx.x & 31;
  const unsigned push_epoch = a.push.n_ranks > 0 ? site_epoch(a.push.step, a.push.sites_per_step, a.push.site_index) : 0u;
  for (int r0 = r_lo; r0 < r_hi || r0 == r_lo; r0 += R) {
    float acc[R][MB];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int m = 0; m < MB; ++m) acc[r][m] = 0.f;
    for (int i = lane * 8; i < K; i += 256) {
      float wv[R][8];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const uint8_t* row = s.w + (long)min(r0 + r, s.rows - 1) * s.row_bytes;
        if (s.wtype == WT_F32) {
          float4 p = __ldg(reinterpret_cast<const float4*>(row) + i / 4), q = __ldg(reinterpret_cast<const float4*>(row) + i / 4 + 1);
          wv[r][0] = p.x; wv[r][1] = p.y; wv[r][2] = p.z; wv[r][3] = p.w; wv[r][4] = q.x; wv[r][5] = q.y; wv[r][6] = q.z; wv[r][7] = q.w;
        } else {
          uint4 p = __ldg(reinterpret_cast<const uint4*>(row) + i / 8);
          const uint32_t ws[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float2 f = (s.wtype == WT_F16) ? __half22float2(*reinterpret_cast<const __half2*>(&ws[j]))
                                           : __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&ws[j]));
            wv[r][2 * j] = f.x; wv[r][2 * j + 1] = f.y;
          }
        }
      }
      between();
#pragma unroll
      for (int m = 0; m < MB; ++m) {
        if (!(live >> m & 1)) continue;
        const float4 x0 = *reinterpret_cast<const float4*>(sx + (long)m * K + i);
        const float4 x1 = *reinterpret_cast<const float4*>(sx + (long)m * K + i + 4);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          float t = acc[r][m];
          t = fmaf(wv[r][0], x0.x, t); t = fmaf(wv[r][1], x0.y, t); t = fmaf(wv[r][2], x0.z, t); t = fmaf(wv[r][3], x0.w, t);
          t = fmaf(wv[r][4], x1.x, t); t = fmaf(wv[r][5], x1.y, t); t = fmaf(wv[r][6], x1.z, t); t = fmaf(wv[r][7], x1.w, t);
          acc[r][m] = t;
        }
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int m = 0; m < MB; ++m) acc[r][m] = warp_sum(acc[r][m]);
    if (lane == 0) {
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (r0 + r < r_hi) {
          const int col = out_col0 + r0 + r;
#pragma unroll
          for (int m = 0; m < MB; ++m)
            if (m < a.M && (live >> m & 1)) {
              float v = acc[r][m] * s_scale[m];
              if (a.push.n_ranks > 0) { push_store(a.push, push_epoch, (long)m * a.out_stride + col, v); continue; }
              if (a.resid) v += a.resid[(long)m * a.resid_stride + col];
              a.out[(long)m * a.out_stride + col] = v;
            }
        }
    }
    if (r0 + R >= r_hi) break;
  }
}

// FAM: 0 = ggml integer-dot types, 1 = those plus float rows, 2 = block-scaled float planes (NVFP4, FP8).
// One kernel per family keeps the register budget of the K-quant bodies free of the plane decoders.
// MULTI: rows_multi and the prologues that fetch all rows at once (two rows and more, weight rows of at most 32 C units);
// otherwise MB rows as a whole.
template <int MB, int R, int C, bool NORM, int FAM, bool MULTI>
__global__ void __launch_bounds__(256, 2) gemv_kernel(const GemvArgs a) {
  static_assert(!MULTI || MB == kMaxRows, "any number of rows");
  extern __shared__ __align__(16) uint8_t smem[];
  const int K = a.K;
  int8_t* sq = reinterpret_cast<int8_t*>(smem);
  const int rows_in = MULTI ? a.M : MB;
  float2* sds = reinterpret_cast<float2*>(smem + (size_t)rows_in * K);
  double* red = reinterpret_cast<double*>(sds + (size_t)rows_in * (K / 32));
  float* s_scale = reinterpret_cast<float*>(red + rows_in * 8);
  float* sx = s_scale + 8;  // float weights, or several rows to normalise
  unsigned live = (1u << MB) - 1;      // MULTI: the pass's rows that do not just fill its bucket
  if constexpr (MULTI) {
    live = 0;
#pragma unroll
    for (int m = 0; m < kMaxRows; ++m) live |= (m < a.M && (!a.row_seq || a.row_seq[m] >= 0) ? 1u : 0u) << m;
  }

  if (a.n_pf > 0 && threadIdx.x == 0) prefetch_spans_l2(a.pf_ptr, a.pf_bytes, a.n_pf);
  int si = 0, col0 = 0;
#pragma unroll
  for (int q = 1; q < 4; ++q)
    if (q < a.nseg && (int)blockIdx.x >= a.seg[q].blk0) { si = q; }
  for (int q = 0; q < si; ++q) col0 += a.seg[q].rows;
  // a block serves one weight type: its q8 activation rows take the chunk layout that type's units read without
  // bank conflicts (act_chunk_pos); float rows read the fp32 copy instead
  const int act_layout = staged_layout(a.seg[si].wtype);
  bool ready = false;
  auto between = [&]() {
    if (!ready) {
      pdl_wait();
      if constexpr (MULTI && NORM) {
        prologue_norm_rows<FAM == 1>(a, live, sq, sds, sx, s_scale, red, act_layout);
      } else if constexpr (MULTI) {
        prologue_q8_rows(a, live, sq, sds, s_scale, act_layout);
      } else if constexpr (NORM) {
        prologue_norm<MB, FAM == 1>(a, sq, sds, sx, s_scale, red, act_layout);
      } else {
        prologue_q8in<MB>(a, sq, sds, s_scale, act_layout);
      }
      pdl_launch();
      ready = true;
    }
  };
  {
    const GemvSeg& s = a.seg[si];
    // even split of the segment's rows over its warps
    const int W = s.nblk * 8, wg = ((int)blockIdx.x - s.blk0) * 8 + (threadIdx.x >> 5);
    const int rpw = (s.rows + W - 1) / W;
    const int r_lo = min(s.rows, wg * rpw), r_hi = min(s.rows, r_lo + rpw);
    auto rows = [&](auto t) {
      if constexpr (MULTI) rows_multi<decltype(t), R, C>(a, s, r_lo, r_hi, col0, live, sq, sds, s_scale, between);
      else rows_q<decltype(t), MB, R, C>(a, s, r_lo, r_hi, col0, sq, sds, s_scale, between);
    };
    if constexpr (FAM == 2) {
      switch (s.wtype) {
        case WT_NVFP4: rows(NvFp4{}); break;
        case WT_FP8_B128: rows(Fp8B128{}); break;
        case WT_Q2_K: rows(Q2K{}); break;
        case WT_Q3_K: rows(Q3K{}); break;
        case WT_Q4_0: rows(Q40{}); break;
        case WT_Q4_1: rows(Q41{}); break;
        case WT_Q5_0: rows(Q50{}); break;
        case WT_Q5_1: rows(Q51{}); break;
        default: break;
      }
    } else {
      switch (s.wtype) {
        case WT_Q4_K: rows(Q4K{}); break;
        case WT_Q6_K: rows(Q6K{}); break;
        case WT_Q5_K: rows(Q5K{}); break;
        case WT_Q8_0: rows(Q80{}); break;
        case WT_Q8_F32: rows(Q8F{}); break;
        default:
          if (FAM == 1) rows_f<MB, R>(a, s, r_lo, r_hi, col0, live, sx, s_scale, between);
      }
    }
  }
  between();
}

// M rows of activations, with their fp32 values or without
static inline size_t gemv_smem(int M, int K, bool values) {
  size_t b = (size_t)M * K + (size_t)M * (K / 32) * 8 + M * 8 * 8 + 8 * 4;
  if (values) b += (size_t)M * K * 4;
  return b;
}

constexpr size_t kSmemOfProcessor = 227 * 1024;      // shared memory of its blocks, each of which takes 1 KB more than it asks for

// How a call of several segments is launched.
struct GemvPlan {
  int grid, R, C;       // blocks; weight rows a warp takes at a time; units of a row a lane takes at a time
  // rows_multi: two rows and more whose weight rows a warp's registers hold, that are not sums over ranks and whose blocks fit a
  // processor two at a time, as they are counted.  The fp32 rows of its norm, 16 KB each at a width of 4,096, do not from six on:
  // QKV (8,192 + 512 + 512) of eight rows as a whole 45 us, 53 in two waves of rows_multi, of four 31 / 27; a head of 151,936 412 / 479
  // and 242 / 225.  Float planes with two units a lane cost more to take apart: behind the norm rows_multi never gains (QKV of NVFP4
  // for four rows 29 / 33, eight 43 / 64), without it from three rows on (passes of the 30 B shape, ms: NVFP4 two rows 3.19 /
  // 3.31, four 4.75 / 4.81, five 5.88 / 5.72, eight 6.88 / 6.84; FP8 two 4.55 / 4.64, three 6.07 / 5.75, five 8.61 / 7.76, eight
  // 10.19 / 9.71).
  bool multi;
  int MB;               // otherwise: the rows of the kernel
  size_t smem;
};

template <int MB, int R, int C, bool NORM, int FAM, bool MULTI>
static cudaError_t gemv_launch(const GemvArgs& a, const GemvPlan& p, cudaStream_t st) {
  static PerDevice limit;
  if (limit.due()) {
    cudaFuncSetAttribute(gemv_kernel<MB, R, C, NORM, FAM, MULTI>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    limit.mark();
  }
  return launch(gemv_kernel<MB, R, C, NORM, FAM, MULTI>, dim3(p.grid), dim3(256), p.smem, st, a);
}

template <bool NORM, int FAM, int MB, bool MULTI>
static cudaError_t gemv_dispatch_shape(const GemvArgs& a, const GemvPlan& p, cudaStream_t st) {
  if constexpr (!(MULTI && NORM && FAM == 2)) {
    if (p.C == 2) return gemv_launch<MB, 1, 2, NORM, FAM, MULTI>(a, p, st);
  }
  // several rows keep the decoded weights of float planes in registers from one row to the next, which leaves room for one;
  // a kernel that takes eight rows as a whole has no room for a third weight row's sums
  if constexpr (MULTI ? FAM == 0 : MB < kMaxRows) {
    if (p.R >= 3) return gemv_launch<MB, 3, 1, NORM, FAM, MULTI>(a, p, st);
  }
  if constexpr (!MULTI || FAM != 2) {
    if (p.R >= 2) return gemv_launch<MB, 2, 1, NORM, FAM, MULTI>(a, p, st);
  }
  return gemv_launch<MB, 1, 1, NORM, FAM, MULTI>(a, p, st);
}

template <bool NORM, int FAM, int MB>
static cudaError_t gemv_dispatch_whole(const GemvArgs& a, const GemvPlan& p, cudaStream_t st) {
  // Only a reduction in front brings rows here whose units one column a lane holds, and there up to three weight rows are in
  // flight (two of the half empty columns instead, two ranks: QKV of 2,048 for two rows 19.5 us, 18.5 so; a head 124, 105; four rows
  // of the head 193, 158).
  if constexpr (NORM) return gemv_dispatch_shape<NORM, FAM, MB, false>(a, p, st);
  else return gemv_launch<MB, 1, 2, NORM, FAM, false>(a, p, st);
}

// Several rows one by one; one row, and rows as a whole.
template <bool NORM, int FAM>
cudaError_t gemv_family(const GemvArgs& a, const GemvPlan& p, cudaStream_t st) {
  if (p.multi) return gemv_dispatch_shape<NORM, FAM, kMaxRows, true>(a, p, st);
  switch (p.MB) {
    case 1: return gemv_dispatch_shape<NORM, FAM, 1, false>(a, p, st);
    case 2: return gemv_dispatch_whole<NORM, FAM, 2>(a, p, st);
    case 4: return gemv_dispatch_whole<NORM, FAM, 4>(a, p, st);
    default: return gemv_dispatch_whole<NORM, FAM, kMaxRows>(a, p, st);
  }
}

}  // namespace bl
