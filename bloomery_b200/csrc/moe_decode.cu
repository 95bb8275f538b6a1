// Decode-time mixture-of-experts chain (m <= 8 rows), expert ids read on the device:
//   1. router           RMSNorm prologue + fp32 router GEMV + top-k by the last-arriving
//                       block (softmax / renormalised, or sigmoid + selection bias with
//                       optional group-limited choice); publishes the q8 normed rows
//   2. gate_up_sel      gate·x and up·x of the chosen experts, SwiGLU, q8 of the result
//   3. down_combine     y = resid + sum_j w_j * down_j(act_j), slots in ascending order
//
// Contracts followed from the reference: softmax router math and tie rule
// (crates/gpu/src/route_softmax.rs:28-58: max, exp f32, f64 sum, top-k desc prob with
// ties to the smaller id, chosen probs renormalised; non-finite logit -> router fault,
// NaN weights); sigmoid "noaux" rule where the bias steers the choice only
// (crates/model/src/arch/noaux.rs:23-94); combine order (crates/gpu/src/arch/qwen3moe/
// experts.rs:36-45); the elsewhere-sentinel for slots another tier serves
// (crates/gpu/src/kquant/sel.rs doc).  The completion counter instead of a grid barrier
// is the reference's measured choice (docs/gpu-design.md:52-64).
#include "gemv_common.cuh"
#include "route.cuh"

namespace bl {

// block-scaled planes and the re-laid 32-value block types share one kernel family
static inline bool is_plane_family(int t) {
  return t == WT_NVFP4 || t == WT_FP8_B128 || t == WT_Q4_0 || t == WT_Q4_1 || t == WT_Q5_0 || t == WT_Q5_1 || t == WT_Q2_K || t == WT_Q3_K;
}


// grid = E blocks (one expert each), 256 threads.  A thread owns 8 consecutive values per
// 2048-value chunk; the router row, gain and x are loaded together, the dot product of
// w with x*gain and the sum of squares run in the same sweep, and the RMS scale multiplies
// the finished logit (so nothing waits for a normalisation pass).
template <int MB>
__global__ void __launch_bounds__(256) router_kernel(const RouterArgs a0) {
  __shared__ float s_dot[8][MB];
  __shared__ double s_ss[8][MB];
  __shared__ float s_scale[MB];
  const int K = a0.K;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int e = blockIdx.x;
  RouterArgs a = a0;                      // row group blockIdx.y: rows [8 y, 8 y + M)
  if (blockIdx.y > 0) {
    const long r0 = (long)blockIdx.y * MB;
    a.x += r0 * a.x_stride; a.logits += r0 * a.E;
    if (a.xq_out) { a.xq_out += r0 * K; a.xds_out += r0 * (K / 32); }
    if (a.xn_out) a.xn_out += r0 * K;
  }
  a.M = min(MB, a0.M - (int)blockIdx.y * MB);
  const long rb = resident_row_bytes(a.wtype, K);
  const uint8_t* row = a.w + (long)e * rb;

  float dot[MB], ss[MB];
#pragma unroll
  for (int m = 0; m < MB; ++m) { dot[m] = 0.f; ss[m] = 0.f; }
  bool waited = false;
  __shared__ int s_gave_up;
  ReduceWait rw{0u, 0ull, &s_gave_up};
  for (int i0 = tid * 8; i0 < K; i0 += 2048) {
    float wv[8];
    if (a.wtype == WT_F32) {
      float4 p = __ldg(reinterpret_cast<const float4*>(row) + i0 / 4), q = __ldg(reinterpret_cast<const float4*>(row) + i0 / 4 + 1);
      wv[0] = p.x; wv[1] = p.y; wv[2] = p.z; wv[3] = p.w; wv[4] = q.x; wv[5] = q.y; wv[6] = q.z; wv[7] = q.w;
    } else {
      uint4 p = __ldg(reinterpret_cast<const uint4*>(row) + i0 / 8);
      const uint32_t ws[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float2 f = (a.wtype == WT_F16) ? __half22float2(*reinterpret_cast<const __half2*>(&ws[j]))
                                       : __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&ws[j]));
        wv[2 * j] = f.x; wv[2 * j + 1] = f.y;
      }
    }
    float4 g0 = __ldg(reinterpret_cast<const float4*>(a.gain + i0)), g1 = __ldg(reinterpret_cast<const float4*>(a.gain + i0 + 4));
    if (!waited) {
      pdl_wait(); waited = true;
      if (a.red.n_ranks > 0) {
        if (tid == 0) s_gave_up = (a.red.fault && *a.red.fault != 0xFFFFFFFFu) ? 1 : 0;   // a poisoned engine no longer waits
        __syncthreads();
        rw.epoch = site_epoch(a.red.step, a.red.sites_per_step, a.red.site_index);
      }
    }
#pragma unroll
    for (int m = 0; m < MB; ++m) {
      const int ms = m < a.M ? m : a.M - 1;
      const float* xr = a.x + (long)ms * a.x_stride;
      float4 x0, x1;
      if (a.red.n_ranks > 0) {
        x0 = *reinterpret_cast<const float4*>(xr + i0); x1 = *reinterpret_cast<const float4*>(xr + i0 + 4);
        float acc8[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
        reduce_sum8(a.red, rw, ms, i0, acc8);
        x0 = make_float4(acc8[0], acc8[1], acc8[2], acc8[3]); x1 = make_float4(acc8[4], acc8[5], acc8[6], acc8[7]);
        if (e == 0 && m < a.M) {
          *reinterpret_cast<float4*>(a.red.x_out + (long)m * a.red.x_out_stride + i0) = x0;
          *reinterpret_cast<float4*>(a.red.x_out + (long)m * a.red.x_out_stride + i0 + 4) = x1;
        }
      } else {
        x0 = *reinterpret_cast<const float4*>(xr + i0); x1 = *reinterpret_cast<const float4*>(xr + i0 + 4);
      }
      ss[m] += x0.x * x0.x + x0.y * x0.y + x0.z * x0.z + x0.w * x0.w + x1.x * x1.x + x1.y * x1.y + x1.z * x1.z + x1.w * x1.w;
      float t = dot[m];
      t = fmaf(wv[0], x0.x * g0.x, t); t = fmaf(wv[1], x0.y * g0.y, t); t = fmaf(wv[2], x0.z * g0.z, t); t = fmaf(wv[3], x0.w * g0.w, t);
      t = fmaf(wv[4], x1.x * g1.x, t); t = fmaf(wv[5], x1.y * g1.y, t); t = fmaf(wv[6], x1.z * g1.z, t); t = fmaf(wv[7], x1.w * g1.w, t);
      dot[m] = t;
    }
  }
  if (!waited) {
    pdl_wait();
    if (a.red.n_ranks > 0) {
      if (tid == 0) s_gave_up = (a.red.fault && *a.red.fault != 0xFFFFFFFFu) ? 1 : 0;   // a poisoned engine no longer waits
      __syncthreads();
      rw.epoch = site_epoch(a.red.step, a.red.sites_per_step, a.red.site_index);
    }
  }
  pdl_launch();
#pragma unroll
  for (int m = 0; m < MB; ++m) {
    float d = warp_sum(dot[m]);
    double q = warp_sum_d((double)ss[m]);
    if (lane == 0) { s_dot[warp][m] = d; s_ss[warp][m] = q; }
  }
  __syncthreads();
  if (tid < MB) {
    float d = 0.f; double q = 0.0;
#pragma unroll
    for (int w = 0; w < 8; ++w) { d += s_dot[w][tid]; q += s_ss[w][tid]; }
    const float scale = (float)(1.0 / sqrt(q / (double)K + (double)a.eps));
    s_scale[tid] = scale;
    if (tid < a.M) { a.logits[(long)tid * a.E + e] = d * scale; __threadfence(); }
  }
  __syncthreads();
  __shared__ int s_last;
  if (a.ticket) {
    // every logit of this block is stored: take a ticket; the block that draws the last one routes the rows
    if (tid == 0) {
      __threadfence();
      const unsigned t = atomicAdd(a.ticket + blockIdx.y, 1u);
      s_last = (t == gridDim.x - 1) ? 1 : 0;
      if (s_last) a.ticket[blockIdx.y] = 0u;         // zero again for the next launch (graph replay)
    }
    __syncthreads();
  }
  // every block knows the scale; block b publishes 32-value blocks b, b + E, ... of the q8 rows
  if (a.xq_out) {
    const int nb32 = K / 32;
    for (int b = e * 8 + warp; b < nb32 * a.M; b += gridDim.x * 8) {
      const int m = b / nb32, bb = b - m * nb32;
      const int i = bb * 32 + lane;
      const float xv = a.red.n_ranks > 0 ? reduce_value(a.red, rw, a.x + (long)m * a.x_stride, m, i) : a.x[(long)m * a.x_stride + i];
      const float v = xv * a.gain[i] * s_scale[m];
      float d, sm;
      int8_t qv = q8_lane(v, d, sm);
      a.xq_out[(long)m * K + i] = qv;
      if (a.xn_out) a.xn_out[(long)m * K + i] = v;
      if (lane == 0) a.xds_out[(long)m * nb32 + bb] = make_float2(d, sm);
    }
  }
  if (a.ticket && s_last) {
    __shared__ RouteShared rs;
    __threadfence();
    RouteParams p = a.route;
    p.logits = a.logits;
    for (int m = 0; m < a.M; ++m) {
      int id; float w;
      const bool ok = route_block(p, m, rs, id, w);
      if (a.pf_gate) {
        // prediction: publish the predicted slots for the prefetch launch that follows (one SM alone cannot issue
        // tens of megabytes of prefetches fast enough; the follower spreads them over the whole card)
        if (warp == 0 && lane < p.top_k) {
          int e = ok ? rs.ids[lane] : -1;
          if (e >= 0 && a.pf_slot_map) e = a.pf_slot_map[e];
          a.ids[(long)m * p.top_k + lane] = e;
        }
        __syncthreads();
        continue;
      }
      if (warp == 0) {
        if (!ok && lane == 0) raise_fault(a.fault, a.layer, FS_ROUTER);
        if (lane < p.top_k) {
          a.ids[(long)m * p.top_k + lane] = ok ? id : -3;
          a.wts[(long)m * p.top_k + lane] = w;
          if (ok && a.heat) atomicAdd(a.heat + id, 1u);
        }
      }
      __syncthreads();
    }
  }
}

// The router of many rows (a decode round past the chain, a short prompt): logits alone, and the normed rows as bf16 for
// the expert products.  A block takes eight rows and four experts: with one expert a block every row was read from L2 once
// an expert, 64 MB a layer at 64 rows.  The sums are router_kernel's, in its order.
constexpr int kRouteE = 4;
__global__ void __launch_bounds__(256) router_rows_kernel(const float* x, long x_stride, const float* gain, float eps, const uint8_t* w,
                                                          int wtype, int K, int E, int M, float* logits, __nv_bfloat16* xn, long xn_stride) {
  __shared__ float s_dot[8][8][kRouteE];
  __shared__ double s_ss[8][8];
  __shared__ float s_scale[8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int e0 = blockIdx.x * kRouteE, m0 = blockIdx.y * 8;
  const int rows = min(8, M - m0);
  const long rb = resident_row_bytes(wtype, K);
  float dot[8][kRouteE], ss[8];
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    ss[m] = 0.f;
#pragma unroll
    for (int j = 0; j < kRouteE; ++j) dot[m][j] = 0.f;
  }
  bool waited = false;
  for (int i0 = tid * 8; i0 < K; i0 += 2048) {
    float wv[kRouteE][8];
#pragma unroll
    for (int j = 0; j < kRouteE; ++j) {
      const uint8_t* row = w + (long)min(e0 + j, E - 1) * rb;
      if (wtype == WT_F32) {
        const float4 p = __ldg(reinterpret_cast<const float4*>(row) + i0 / 4), q = __ldg(reinterpret_cast<const float4*>(row) + i0 / 4 + 1);
        wv[j][0] = p.x; wv[j][1] = p.y; wv[j][2] = p.z; wv[j][3] = p.w; wv[j][4] = q.x; wv[j][5] = q.y; wv[j][6] = q.z; wv[j][7] = q.w;
      } else {
        const uint4 p = __ldg(reinterpret_cast<const uint4*>(row) + i0 / 8);
        const uint32_t ws[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float2 f = (wtype == WT_F16) ? __half22float2(*reinterpret_cast<const __half2*>(&ws[c]))
                                             : __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&ws[c]));
          wv[j][2 * c] = f.x; wv[j][2 * c + 1] = f.y;
        }
      }
    }
    const float4 g0 = __ldg(reinterpret_cast<const float4*>(gain + i0)), g1 = __ldg(reinterpret_cast<const float4*>(gain + i0 + 4));
    if (!waited) { pdl_wait(); waited = true; }
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      const float* xr = x + (long)(m0 + min(m, rows - 1)) * x_stride;
      const float4 x0 = *reinterpret_cast<const float4*>(xr + i0), x1 = *reinterpret_cast<const float4*>(xr + i0 + 4);
      ss[m] += x0.x * x0.x + x0.y * x0.y + x0.z * x0.z + x0.w * x0.w + x1.x * x1.x + x1.y * x1.y + x1.z * x1.z + x1.w * x1.w;
      const float xg[8] = {x0.x * g0.x, x0.y * g0.y, x0.z * g0.z, x0.w * g0.w, x1.x * g1.x, x1.y * g1.y, x1.z * g1.z, x1.w * g1.w};
#pragma unroll
      for (int j = 0; j < kRouteE; ++j)
#pragma unroll
        for (int c = 0; c < 8; ++c) dot[m][j] = fmaf(wv[j][c], xg[c], dot[m][j]);
    }
  }
  if (!waited) pdl_wait();
  pdl_launch();
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    const double q = warp_sum_d((double)ss[m]);
    if (lane == 0) s_ss[warp][m] = q;
#pragma unroll
    for (int j = 0; j < kRouteE; ++j) {
      const float d = warp_sum(dot[m][j]);
      if (lane == 0) s_dot[warp][m][j] = d;
    }
  }
  __syncthreads();
  if (tid < 8) {
    double q = 0.0;
#pragma unroll
    for (int i = 0; i < 8; ++i) q += s_ss[i][tid];
    s_scale[tid] = (float)(1.0 / sqrt(q / (double)K + (double)eps));
  }
  __syncthreads();
  if (tid < 8 * kRouteE) {
    const int m = tid / kRouteE, j = tid % kRouteE;
    float d = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) d += s_dot[i][m][j];
    if (m < rows && e0 + j < E) logits[(long)(m0 + m) * E + e0 + j] = d * s_scale[m];
  }
  // every block of a row group knows the scales: they share its normed rows
  if (xn)
    for (int i = (blockIdx.x * 256 + tid) * 4; i < rows * K; i += gridDim.x * 1024) {
      const int m = i / K, c = i - m * K;
      const float4 v = *reinterpret_cast<const float4*>(x + (long)(m0 + m) * x_stride + c);
      const float4 g = __ldg(reinterpret_cast<const float4*>(gain + c));
      const float sc = s_scale[m];
      __nv_bfloat162 o[2] = {__floats2bfloat162_rn(v.x * sc * g.x, v.y * sc * g.y), __floats2bfloat162_rn(v.z * sc * g.z, v.w * sc * g.w)};
      *reinterpret_cast<uint2*>(xn + (long)(m0 + m) * xn_stride + c) = *reinterpret_cast<const uint2*>(o);
    }
}

// ------------------------------------------------------------------------------------
// gate·up·SwiGLU over device-side expert ids
// grid (I/32, n_used, M), 256 threads: warp w computes activation rows 4w..4w+3 of the chunk
// ------------------------------------------------------------------------------------
constexpr int kMaxInput = 200 * 1024;       // bytes of a staged activation row

struct GateUpArgs {
  const int8_t* xq; const float2* xds;   // [M, K] q8
  RouteParams route;                     // route.logits == null: ids are given
  int* ids;                              // [M, n_used] read (given) or written (routed here)
  float* wts;                            // [M, n_used] written when routed here
  unsigned* heat;                        // optional [E] routed-count histogram
  const int* slot_map;                   // optional [E]: expert id -> resident slot (or kExpertElsewhere)
  const uint8_t* gate; const uint8_t* up; int gtype, utype;   // stacks [E_slots, I, K]
  int K, I, E, n_used, M;
  int8_t* actq; float2* actds;           // [M, n_used, I] q8
  float* act_f32;                        // optional fp32 copy
  unsigned* fault; int layer;
  const uint8_t* down; long down_expert_bytes;   // optional: the down stack, whose chosen matrices L2 is asked to prefetch
  // optional [M] (with route.logits): rows with a negative entry only fill the bucket.  They route nowhere, so neither this
  // launch nor the one behind it reads a weight for them (five rows in the bucket of eight were charged for eight).
  const int* row_seq;
};

// R activation outputs (R gate rows + R up rows) of one warp, the activations in shared memory (in the chunk layout of T): lane
// 8 r gets the gate's and the up product's sum of row r.
template <class T, int R>
__device__ __forceinline__ void gate_up_rows(const uint8_t* g0, const uint8_t* u0, long rb, int K, int lane,
                                             const int8_t* sq, const float2* sds, float& g, float& u_sum) {
  using U = Unit<T>;
  const int nunits = K / 64;
  float gacc[R], uacc[R];
#pragma unroll
  for (int r = 0; r < R; ++r) gacc[r] = uacc[r] = 0.f;
  for (int u = lane; u < nunits; u += 32) {
    typename U::Regs rg[R], ru[R];
#pragma unroll
    for (int r = 0; r < R; ++r) { U::loadu(g0 + r * rb, u, K, rg[r]); U::loadu(u0 + r * rb, u, K, ru[r]); }
    ActRegs act;
    StagedAct<T>::load(sq, sds, u, nunits, act);
#pragma unroll
    for (int r = 0; r < R; ++r) { gacc[r] = ActOf<T>::dot(rg[r], u, act, gacc[r]); uacc[r] = ActOf<T>::dot(ru[r], u, act, uacc[r]); }
  }
  g = warp_sum4(gacc[0], gacc[R - 1], uacc[0], uacc[R - 1]);
  u_sum = __shfl_down_sync(0xffffffffu, g, 16);
}

// grid (I/32, n_used, M), 256 threads: in turns of 8 R rows of the chunk, warp w computes activation rows R w .. R w + R - 1.
// When route.logits is set the grid is one wider in x: every block routes row m itself (redundantly, from the router
// launch's logits) so no block waits on a completion counter, and the block behind the chunks publishes ids / weights /
// heat for the launches that follow, which takes the weights' arithmetic off the path of those that multiply.
// One row is a chain of latencies (logits, picks, weights, sums), so what can overlap does: the activations come in under the
// picks, which one warp takes where route_pick serves, and the rows of later turns are asked into L2 while the first turn's
// are in flight.  30 B shape, one row, us behind the launch in front: 9.3 (10.3 with activations from L2 and picks by the block), of
// which 2 go to the picks, 3 to 5 to the first turn (1 of them to HBM), 1.5 to the second; its schedulers issue in 14 % of the
// cycles, and a warp waits for loads and for the picks.  Several rows are bound by their blocks'
// latencies in turns of the processors: five 30 us (36 before, 34 with R = 2).
// FAM 0 = ggml integer-dot types, FAM 2 = block-scaled float planes (one kernel per family keeps
// the plane decoders out of the K-quant bodies' register budget)
// R = 2, two blocks a processor, for one row; R = 1, three blocks, for several, which queue for the processors
template <int FAM, int R>
__global__ void __launch_bounds__(256, R == 2 ? 2 : 3) gate_up_sel_kernel(const GateUpArgs a) {
  extern __shared__ __align__(16) uint8_t s_in[];
  const int K = a.K;
  int8_t* sq = reinterpret_cast<int8_t*>(s_in);
  float2* sds = reinterpret_cast<float2*>(s_in + K);
  __shared__ float s_act[32];
  __shared__ RouteShared rs;
  const int chunk = blockIdx.x, j = blockIdx.y, m = blockIdx.z;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool publisher = chunk == a.I / 32;
  if (publisher && j != 0) return;
  pdl_wait();
  pdl_launch();
  if (a.row_seq && a.row_seq[m] < 0) {
    if (publisher && tid < a.n_used) {
      a.ids[(long)m * a.n_used + tid] = kExpertElsewhere;
      a.wts[(long)m * a.n_used + tid] = 0.f;
    }
    return;
  }
  const bool pick = a.route.logits && route_pick_ok(a.route);
  if (publisher) {
    if (pick && warp != 0) return;
    int id; float w;
    bool ok;
    if (pick) {
      float l;
      ok = route_pick(a.route, m, lane, a.n_used, id, l);
      w = ok ? route_pick_weight(a.route, lane, l) : __int_as_float(0x7fc00000);
    } else {
      ok = route_block(a.route, m, rs, id, w);
    }
    if (warp != 0) return;
    if (!ok && lane == 0) raise_fault(a.fault, a.layer, FS_ROUTER);
    if (lane < a.n_used) {
      a.ids[(long)m * a.n_used + lane] = ok ? id : 0;
      a.wts[(long)m * a.n_used + lane] = w;
      if (ok && a.heat) atomicAdd(a.heat + id, 1u);
    }
    return;
  }
  copy_q8_row(a.xq + (long)m * K, a.xds + (long)m * (K / 32), K, staged_layout(a.gtype), sq, sds);
  __shared__ int s_e;
  int e;
  if (pick) {
    if (warp == 0) {
      int id;
      float l;
      const bool ok = route_pick(a.route, m, lane, j + 1, id, l);
      if (lane == j) s_e = ok ? id : -3;
    }
    cp_async_wait<0>();
    __syncthreads();
    e = s_e;
  } else if (a.route.logits) {
    float w;
    e = route_block(a.route, m, rs, e, w) ? rs.ids[j] : -3;
  } else {
    e = a.ids[(long)m * a.n_used + j];
  }
  const long ob = ((long)m * a.n_used + j) * a.I + chunk * 32;
  bool skip = false, bad = false;
  if (e == kExpertElsewhere) skip = true;
  else if (e == -3) { skip = true; bad = true; }                 // router fault: NaN downstream
  else if (e < 0 || e >= a.E) { skip = true; bad = true; if (tid == 0 && chunk == 0) raise_fault(a.fault, a.layer, FS_EXPERT_ID); }
  else if (a.slot_map) { e = a.slot_map[e]; if (e < 0) skip = true; }
  if (skip) {
    cp_async_wait<0>();
    if (tid < 32) {
      a.actq[ob + tid] = 0;
      if (a.act_f32) a.act_f32[ob + tid] = bad ? __int_as_float(0x7fc00000) : 0.f;
    }
    if (tid == 0) a.actds[ob / 32] = bad ? make_float2(__int_as_float(0x7fc00000), 0.f) : make_float2(0.f, 0.f);
    return;
  }
  const long rb = resident_row_bytes(a.gtype, K), first = (long)e * a.I + chunk * 32;
  if (tid == 0 || tid == 128) {
    // the rows of the chunk behind the first turn's
    const uint8_t* p = (tid == 0 ? a.gate : a.up) + (first + 8 * R) * rb;
    const long bytes = (32 - 8 * R) * rb;
    for (long o = 0; o < bytes; o += 32768) {
      const unsigned nb = (unsigned)((bytes - o) < 32768 ? (bytes - o) : 32768);
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p + o), "r"(nb) : "memory");
    }
  }
  if (a.down && tid == 32) {
    // the down launch that follows streams expert e's matrix: this block asks L2 for its share of it
    const long share = (a.down_expert_bytes / (a.I / 32)) & ~15L;
    for (long o = 0; o < share; o += 32768) {
      const unsigned nb = (unsigned)((share - o) < 32768 ? (share - o) : 32768);
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a.down + (long)e * a.down_expert_bytes + (long)chunk * share + o), "r"(nb) : "memory");
    }
  }
  if (!pick) {
    cp_async_wait<0>();
    __syncthreads();
  }
#pragma unroll 1
  for (int turn = 0; turn < 4 / R; ++turn) {
    const long row0 = first + turn * 8 * R + warp * R;
    const uint8_t* g0 = a.gate + row0 * rb;
    const uint8_t* u0 = a.up + row0 * rb;
    float g = 0.f, u = 0.f;
    auto rows = [&](auto t) { gate_up_rows<decltype(t), R>(g0, u0, rb, K, lane, sq, sds, g, u); };
    if constexpr (FAM == 2) {
      switch (a.gtype) {
        case WT_NVFP4: rows(NvFp4{}); break;
        case WT_FP8_B128: rows(Fp8B128{}); break;
        case WT_Q2_K: rows(Q2K{}); break;
        case WT_Q3_K: rows(Q3K{}); break;
        case WT_Q4_0: rows(Q40{}); break;
        case WT_Q4_1: rows(Q41{}); break;
        case WT_Q5_0: rows(Q50{}); break;
        case WT_Q5_1: rows(Q51{}); break;
        default: g = __int_as_float(0x7fc00000);
      }
    } else {
      switch (a.gtype) {
        case WT_Q4_K: rows(Q4K{}); break;
        case WT_Q5_K: rows(Q5K{}); break;
        case WT_Q6_K: rows(Q6K{}); break;
        case WT_Q8_0: rows(Q80{}); break;
        case WT_Q8_F32: rows(Q8F{}); break;
        default: g = __int_as_float(0x7fc00000);
      }
    }
    if (lane == 0 || (R == 2 && lane == 8)) s_act[turn * 8 * R + warp * R + (lane >> 3)] = (g / (1.0f + expf(-g))) * u;
  }
  __syncthreads();
  if (warp == 0) {
    float v = s_act[lane];
    float d, s;
    int8_t q = q8_lane(v, d, s);
    a.actq[ob + lane] = q;
    if (a.act_f32) a.act_f32[ob + lane] = v;
    if (lane == 0) a.actds[ob / 32] = make_float2(d, s);
  }
}

// ------------------------------------------------------------------------------------
// down projection of every chosen expert + router-weighted sum + residual, one launch
// grid (H/8, M), 256 threads: warp w owns output row 8*blockIdx.x + w
// ------------------------------------------------------------------------------------
struct DownArgs {
  const int8_t* actq; const float2* actds;  // [M, n_used, I]
  const int* ids; const float* wts;         // [M, n_used]
  const int* slot_map;
  const uint8_t* down; int dtype;           // stack [E_slots, H, I]
  int I, H, E, n_used, M;
  const float* resid; long resid_stride;    // [M, H] or null
  const float* extra; long extra_stride;    // optional addend (shared expert / host leg sum)
  float* out; long out_stride;
  unsigned* fault; int layer;
  PushOut push;                             // n_ranks > 0: the result is this rank's partial update
};

// One row d of the sum over the chosen experts.  The activations of a row of the pass, slot by slot, are one row of
// n_used * I values, whose units go to the lanes in turn (t = lane + 32 c).  UPL = units per lane (all loaded before any is
// used: one DRAM round trip per row); lane j < n_used holds the expert and the weight of slot j.
template <class T, int UPL, class Landed>
__device__ __forceinline__ float down_row(const DownArgs& a, int d, int lane, const int (&slot)[UPL], const int (&unit)[UPL], int my_e, float my_w,
                                          const int8_t* sq, const float2* sds, Landed&& landed) {
  using U = Unit<T>;
  const int total = a.n_used * (a.I / 64);
  const long rb = resident_row_bytes(T::kType, a.I);
  typename U::Regs regs[UPL];
  bool use[UPL];
#pragma unroll
  for (int c = 0; c < UPL; ++c) {
    const int e = __shfl_sync(0xffffffffu, my_e, slot[c]);
    use[c] = lane + 32 * c < total && e >= 0;
    if (use[c]) U::loadu(a.down + ((long)e * a.H + d) * rb, unit[c], a.I, regs[c]);
  }
  landed();
  // the lane's units of a slot are added up, the router-weighted sum runs over its slots in ascending order, then one butterfly
  float y = 0.f, part = 0.f;
#pragma unroll
  for (int c = 0; c < UPL; ++c) {
    const float w = __shfl_sync(0xffffffffu, my_w, slot[c]);
    if (use[c]) {
      ActRegs act;
      StagedAct<T>::load(sq, sds, lane + 32 * c, total, act);
      part += ActOf<T>::dot(regs[c], unit[c], act, 0.f);
      if (c + 1 == UPL || lane + 32 * (c + 1) >= total || slot[c + 1 < UPL ? c + 1 : c] != slot[c]) { y = fmaf(w, part, y); part = 0.f; }
    }
  }
  return warp_sum(y);
}

// OCC = blocks a processor.  One row has 256 blocks for 148 processors and wants its registers; several rows queue for the
// processors (five rows: 34 us with two, 29 with three, before the activations were staged; FP8 rows 36 us either way).
// The launch in front asked L2 for the weights, so a row is bound by latencies (its schedulers issue in 38 % of the cycles), of which
// activations read from L2, sixteen bytes in every 64, were a large part.  With them in shared memory, one request for a super-block's
// head and the residual asked for in front, one row takes 6.5 us a layer of the 30 B shape (9.0 before), five 23 (28).
template <int UPL, int FAM, int OCC>
__global__ void __launch_bounds__(256, OCC) down_combine_kernel(const DownArgs a) {
  extern __shared__ __align__(16) uint8_t s_in[];
  const int width = a.n_used * a.I;
  int8_t* sq = reinterpret_cast<int8_t*>(s_in);
  float2* sds = reinterpret_cast<float2*>(s_in + width);
  const int m = blockIdx.y;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int upe = a.I / 64;              // units per expert row
  int slot[UPL], unit[UPL];
#pragma unroll
  for (int c = 0; c < UPL; ++c) {
    slot[c] = min((lane + 32 * c) / upe, a.n_used - 1);
    unit[c] = lane + 32 * c - slot[c] * upe;
  }
  const int d = blockIdx.x * 8 + warp, dr = min(d, a.H - 1);
  pdl_wait();
  pdl_launch();
  int my_e = -1;
  float my_w = 0.f;
  if (lane < a.n_used) {
    my_e = a.ids[(long)m * a.n_used + lane];
    my_w = a.wts[(long)m * a.n_used + lane];
  }
  copy_q8_row(a.actq + (long)m * width, a.actds + (long)m * (width / 32), width, staged_layout(a.dtype), sq, sds);
  float add = 0.f, old = 0.f;
  if (lane == 0) {
    if (a.extra) add = a.extra[(long)m * a.extra_stride + dr];
    if (a.resid && a.push.n_ranks == 0) old = a.resid[(long)m * a.resid_stride + dr];
  }
  if (my_e == kExpertElsewhere) my_e = -1;
  else if (my_e < 0 || my_e >= a.E) my_e = -2;
  else if (a.slot_map) { my_e = a.slot_map[my_e]; if (my_e < 0) my_e = -1; }
  const bool bad = __any_sync(0xffffffffu, my_e == -2);
  auto landed = [&]() {
    cp_async_wait<0>();
    __syncthreads();
  };
  float y;
  auto row = [&](auto t) { y = down_row<decltype(t), UPL>(a, dr, lane, slot, unit, my_e, my_w, sq, sds, landed); };
  if constexpr (FAM == 2) {
    switch (a.dtype) {
      case WT_NVFP4: row(NvFp4{}); break;
      case WT_FP8_B128: row(Fp8B128{}); break;
      case WT_Q2_K: row(Q2K{}); break;
      case WT_Q3_K: row(Q3K{}); break;
      case WT_Q4_0: row(Q40{}); break;
      case WT_Q4_1: row(Q41{}); break;
      case WT_Q5_0: row(Q50{}); break;
      case WT_Q5_1: row(Q51{}); break;
      default: y = __int_as_float(0x7fc00000);
    }
  } else {
    switch (a.dtype) {
      case WT_Q4_K: row(Q4K{}); break;
      case WT_Q6_K: row(Q6K{}); break;
      case WT_Q5_K: row(Q5K{}); break;
      case WT_Q8_0: row(Q80{}); break;
      case WT_Q8_F32: row(Q8F{}); break;
      default: y = __int_as_float(0x7fc00000);
    }
  }
  if (lane == 0 && d < a.H) {
    if (bad) { y = __int_as_float(0x7fc00000); if (d == 0) raise_fault(a.fault, a.layer, FS_EXPERT_ID); }
    if (a.extra) y += add;
    if (a.push.n_ranks > 0) {
      push_store(a.push, site_epoch(a.push.step, a.push.sites_per_step, a.push.site_index), (long)m * a.out_stride + d, y);
    } else {
      if (a.resid) y += old;
      a.out[(long)m * a.out_stride + d] = y;
    }
  }
}

}  // namespace bl

using namespace bl;

extern "C" {

// Router logits (RMS scale applied) for M rows + the q8 form of the normed rows.
// ticket != null (one zeroed word per group of 8 rows): the launch also routes, i.e. writes ids / wts (and heat).
int bl_router(const float* x, long x_stride, const float* gain, float eps, const void* w, int wtype,
              int K, int E, int M, float* logits, int8_t* xq_out, float* xds_out, float* xn_out,
              const void* red_desc, unsigned* fault, int layer,
              unsigned* ticket, const float* bias, int top_k, int mode, int renorm, float scale, int n_group, int topk_group,
              int* ids, float* wts, unsigned* heat,
              const void* pf_gate, const void* pf_up, const void* pf_down, long pf_gate_bytes, long pf_down_bytes,
              const int* pf_slot_map, cudaStream_t st) {
  BL_REQUIRE(E >= 1 && E <= kMaxExperts, BL_ERR_LIMIT);
  BL_REQUIRE(K % 256 == 0 && M >= 1 && M <= 8 * 65535, BL_ERR_SHAPE);
  BL_REQUIRE(wtype == WT_F32 || wtype == WT_F16 || wtype == WT_BF16, BL_ERR_TYPE);
  RouterArgs a{};
  a.x = x; a.x_stride = x_stride; a.gain = gain; a.eps = eps; a.w = (const uint8_t*)w; a.wtype = wtype;
  a.K = K; a.E = E; a.M = M; a.logits = logits; a.xq_out = xq_out; a.xds_out = (float2*)xds_out; a.xn_out = xn_out;
  a.fault = fault; a.layer = layer;
  if (red_desc) { a.red = *(const ReduceIn*)red_desc; BL_REQUIRE(M <= kMaxRows && a.red.n_ranks <= kMaxRanks && a.red.H == K, BL_ERR_SHAPE); }
  if (ticket) {
    BL_REQUIRE(E % 4 == 0 && top_k >= 1 && top_k <= kMaxTopK && top_k <= E && n_group >= 1 && n_group <= 16 && E % n_group == 0 &&
               topk_group >= 1 && topk_group <= n_group && ((ids && wts) || pf_gate), BL_ERR_SHAPE);
    a.ticket = ticket; a.ids = ids; a.wts = wts; a.heat = heat;
    if (pf_gate) {
      BL_REQUIRE(pf_up && pf_down && pf_gate_bytes > 0 && pf_down_bytes > 0 && (((uintptr_t)pf_gate | (uintptr_t)pf_up | (uintptr_t)pf_down) & 15) == 0 &&
                 pf_gate_bytes % 16 == 0 && pf_down_bytes % 16 == 0, BL_ERR_ALIGN);
      a.pf_gate = (const uint8_t*)pf_gate; a.pf_up = (const uint8_t*)pf_up; a.pf_down = (const uint8_t*)pf_down;
      a.pf_gate_bytes = pf_gate_bytes; a.pf_down_bytes = pf_down_bytes; a.pf_slot_map = pf_slot_map;
    }
    a.route = RouteParams{nullptr, bias, E, top_k, mode, renorm, scale, n_group, topk_group};
  }
  int mb = M <= 1 ? 1 : M <= 2 ? 2 : M <= 4 ? 4 : 8;
  dim3 grid(E, (M + mb - 1) / mb);
  switch (mb) {
    case 1: return (int)launch(router_kernel<1>, grid, dim3(256), 0, st, a);
    case 2: return (int)launch(router_kernel<2>, grid, dim3(256), 0, st, a);
    case 4: return (int)launch(router_kernel<4>, grid, dim3(256), 0, st, a);
    default: return (int)launch(router_kernel<8>, grid, dim3(256), 0, st, a);
  }
}

// Router logits of M rows and, with xn, the normed rows as bf16 (row stride xn_stride).  x and gain 16-byte aligned rows.
int bl_router_rows(const float* x, long x_stride, const float* gain, float eps, const void* w, int wtype, int K, int E, int M,
                   float* logits, void* xn, long xn_stride, cudaStream_t st) {
  BL_REQUIRE(E >= 1 && E <= kMaxExperts, BL_ERR_LIMIT);
  BL_REQUIRE(K % 256 == 0 && K >= 256 && M >= 1 && M <= 8 * 65535, BL_ERR_SHAPE);
  BL_REQUIRE(wtype == WT_F32 || wtype == WT_F16 || wtype == WT_BF16, BL_ERR_TYPE);
  BL_REQUIRE((((uintptr_t)x | (uintptr_t)gain | (uintptr_t)w) & 15) == 0 && x_stride % 4 == 0 && ((uintptr_t)xn & 7) == 0 &&
             xn_stride % 4 == 0, BL_ERR_ALIGN);
  return (int)launch(router_rows_kernel, dim3((E + kRouteE - 1) / kRouteE, (M + 7) / 8), dim3(256), 0, st, x, x_stride, gain, eps,
                     (const uint8_t*)w, wtype, K, E, M, logits, (__nv_bfloat16*)xn, xn_stride);
}

// Asks L2 to prefetch the gate / up (and optionally down) matrices of the experts named in ids[n] (negative = skip),
// 32 KB pieces dealt round-robin over the blocks; lane 0 of every warp issues.
__global__ void __launch_bounds__(256) prefetch_experts_kernel(const int* ids, int n, const uint8_t* gate, const uint8_t* up,
                                                               const uint8_t* down, long gate_bytes, long down_bytes) {
  pdl_wait();
  pdl_launch();
  const long gn = gate_bytes / 32768, dn = down ? down_bytes / 32768 : 0, per = 2 * gn + dn;
  const long total = per * n;
  const int wid = blockIdx.x * 8 + (threadIdx.x >> 5), nw = gridDim.x * 8;
  if ((threadIdx.x & 31) != 0) return;
  for (long c = wid; c < total; c += nw) {
    const int q = (int)(c / per);
    const long r = c - (long)q * per;
    const int e = ids[q];
    if (e < 0) continue;
    const uint8_t* src = r < gn ? gate + e * gate_bytes + r * 32768
                       : r < 2 * gn ? up + e * gate_bytes + (r - gn) * 32768
                       : down + e * down_bytes + (r - 2 * gn) * 32768;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(32768u) : "memory");
  }
}

// Standalone routing of M rows from logits (tests, prefill, host paths): one warp per row.
// row_seq (optional): rows with a negative entry fill a bucket and nothing else; they route nowhere and count nowhere.
__global__ void __launch_bounds__(256) route_rows_kernel(RouteParams p, int M, int* ids, float* wts, unsigned* heat,
                                                         unsigned* fault, int layer, const int* row_seq) {
  __shared__ RouteShared rs;
  pdl_wait();
  pdl_launch();
  const int lane = threadIdx.x & 31;
  if (route_pick_ok(p)) {
    // a warp a row (the grid has a block for eight): 4,096 rows of 128 experts took 28 us with a block a row, now 11
    const int m = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (m >= M) return;
    int id = kExpertElsewhere;
    float w = 0.f;
    if (!(row_seq && row_seq[m] < 0)) {
      float l;
      const bool ok = route_pick(p, m, lane, p.top_k, id, l);
      w = ok ? route_pick_weight(p, lane, l) : __int_as_float(0x7fc00000);
      if (!ok && lane == 0) raise_fault(fault, layer, FS_ROUTER);
      if (ok && heat && lane < p.top_k) atomicAdd(heat + id, 1u);
    }
    if (lane < p.top_k) {
      ids[(long)m * p.top_k + lane] = id;
      wts[(long)m * p.top_k + lane] = w;
    }
    return;
  }
  const int m = blockIdx.x;
  if (row_seq && row_seq[m] < 0) {
    if (threadIdx.x < p.top_k) {
      ids[(long)m * p.top_k + threadIdx.x] = kExpertElsewhere;
      wts[(long)m * p.top_k + threadIdx.x] = 0.f;
    }
    return;
  }
  int id; float w;
  const bool ok = route_block(p, m, rs, id, w);
  if (threadIdx.x >= 32) return;
  if (!ok && lane == 0) raise_fault(fault, layer, FS_ROUTER);
  if (lane < p.top_k) {
    ids[(long)m * p.top_k + lane] = ok ? id : 0;
    wts[(long)m * p.top_k + lane] = w;
    if (ok && heat) atomicAdd(heat + id, 1u);
  }
}

int bl_prefetch_experts(const int* ids, int n, const void* gate, const void* up, const void* down, long gate_bytes,
                        long down_bytes, int blocks, cudaStream_t st) {
  BL_REQUIRE(n >= 1 && gate && up && gate_bytes > 0 && blocks >= 1, BL_ERR_SHAPE);
  BL_REQUIRE((((uintptr_t)gate | (uintptr_t)up | (uintptr_t)down) & 15) == 0 && gate_bytes % 16 == 0 && down_bytes % 16 == 0, BL_ERR_ALIGN);
  return (int)launch(prefetch_experts_kernel, dim3(blocks), dim3(256), 0, st, ids, n, (const uint8_t*)gate, (const uint8_t*)up,
                     (const uint8_t*)down, gate_bytes, down_bytes);
}

int bl_route_rows(const float* logits, const float* bias, int E, int M, int top_k, int mode, int renorm, float scale,
                  int n_group, int topk_group, int* ids, float* wts, unsigned* heat, unsigned* fault, int layer,
                  const int* row_seq, cudaStream_t st) {
  BL_REQUIRE(E >= 4 && E % 4 == 0 && E <= kMaxExperts && top_k >= 1 && top_k <= kMaxTopK && top_k <= E, BL_ERR_LIMIT);
  BL_REQUIRE(n_group >= 1 && n_group <= 16 && E % n_group == 0 && topk_group >= 1 && topk_group <= n_group, BL_ERR_SHAPE);
  RouteParams p{logits, bias, E, top_k, mode, renorm, scale, n_group, topk_group};
  return (int)launch(route_rows_kernel, dim3(route_pick_ok(p) ? (M + 7) / 8 : M), dim3(256), 0, st, p, M, ids, wts, heat, fault, layer, row_seq);
}

// route_logits != null: every block routes its row from the logits (and block 0 writes
// ids / wts / heat); otherwise ids are read as given.
int bl_gate_up_sel(const int8_t* xq, const float* xds, const float* route_logits, const float* bias, int top_k_mode,
                   int renorm, float scale, int n_group, int topk_group, int* ids, float* wts, unsigned* heat,
                   const int* slot_map, const void* gate, const void* up, int gtype, int utype, int K, int I, int E,
                   int n_used, int M, int8_t* actq, float* actds, float* act_f32, unsigned* fault, int layer,
                   const void* down, long down_expert_bytes, const int* row_seq, cudaStream_t st) {
  BL_REQUIRE(!row_seq || route_logits, BL_ERR_SHAPE);
  BL_REQUIRE(K % 256 == 0 && I % 32 == 0 && M >= 1 && n_used >= 1 && n_used <= kMaxTopK, BL_ERR_SHAPE);
  BL_REQUIRE(gtype == utype, BL_ERR_TYPE);
  BL_REQUIRE(gtype == WT_Q4_K || gtype == WT_Q5_K || gtype == WT_Q6_K || gtype == WT_Q8_0 || gtype == WT_Q8_F32 || is_plane_family(gtype), BL_ERR_TYPE);
  BL_REQUIRE(E % 4 == 0 && E <= kMaxExperts && n_group >= 1 && n_group <= 16 && E % n_group == 0, BL_ERR_LIMIT);
  GateUpArgs a{};
  a.xq = xq; a.xds = (const float2*)xds;
  a.route = RouteParams{route_logits, bias, E, n_used, top_k_mode, renorm, scale, n_group, topk_group};
  a.ids = ids; a.wts = wts; a.heat = heat; a.slot_map = slot_map;
  a.gate = (const uint8_t*)gate; a.up = (const uint8_t*)up; a.gtype = gtype; a.utype = utype;
  a.K = K; a.I = I; a.E = E; a.n_used = n_used; a.M = M;
  a.actq = actq; a.actds = (float2*)actds; a.act_f32 = act_f32; a.fault = fault; a.layer = layer;
  BL_REQUIRE(((uintptr_t)down & 15) == 0 && down_expert_bytes % 16 == 0, BL_ERR_ALIGN);
  a.down = (const uint8_t*)down; a.down_expert_bytes = down_expert_bytes;
  a.row_seq = row_seq;
  const size_t smem = (size_t)K + K / 4;
  BL_REQUIRE(smem <= kMaxInput, BL_ERR_LIMIT);
  static PerDevice limit;
  if (limit.due()) {
    cudaFuncSetAttribute(gate_up_sel_kernel<0, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxInput);
    cudaFuncSetAttribute(gate_up_sel_kernel<2, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxInput);
    cudaFuncSetAttribute(gate_up_sel_kernel<0, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxInput);
    cudaFuncSetAttribute(gate_up_sel_kernel<2, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxInput);
    limit.mark();
  }
  const dim3 grid(I / 32 + (route_logits ? 1 : 0), n_used, M);
  if (M == 1) return (int)launch(is_plane_family(gtype) ? gate_up_sel_kernel<2, 2> : gate_up_sel_kernel<0, 2>, grid, dim3(256), smem, st, a);
  return (int)launch(is_plane_family(gtype) ? gate_up_sel_kernel<2, 1> : gate_up_sel_kernel<0, 1>, grid, dim3(256), smem, st, a);
}

int bl_down_combine(const int8_t* actq, const float* actds, const int* ids, const float* wts, const int* slot_map,
                    const void* down, int dtype, int I, int H, int E, int n_used, int M, const float* resid,
                    long resid_stride, const float* extra, long extra_stride, float* out, long out_stride,
                    const void* push_desc, unsigned* fault, int layer, cudaStream_t st) {
  BL_REQUIRE(I % 256 == 0 || ((dtype == WT_Q8_0 || dtype == WT_Q8_F32 || (is_plane_family(dtype) && dtype != WT_FP8_B128 && dtype != WT_Q2_K && dtype != WT_Q3_K)) && I % 64 == 0) ||
             (dtype == WT_FP8_B128 && I % 128 == 0), BL_ERR_SHAPE);
  BL_REQUIRE(M >= 1 && n_used >= 1 && n_used <= kMaxTopK, BL_ERR_SHAPE);
  BL_REQUIRE(dtype == WT_Q4_K || dtype == WT_Q5_K || dtype == WT_Q6_K || dtype == WT_Q8_0 || dtype == WT_Q8_F32 || is_plane_family(dtype), BL_ERR_TYPE);
  DownArgs a{actq, (const float2*)actds, ids, wts, slot_map, (const uint8_t*)down, dtype, I, H, E, n_used, M, resid,
             resid_stride, extra, extra_stride, out, out_stride, fault, layer, PushOut{}};
  if (push_desc) { a.push = *(const PushOut*)push_desc; BL_REQUIRE(a.push.n_ranks <= kMaxRanks && M <= kMaxRows, BL_ERR_SHAPE); }
  const long total = (long)n_used * (I / 64);
  BL_REQUIRE(total <= 512, BL_ERR_LIMIT);
  const dim3 grid((H + 7) / 8, M);
  const size_t smem = (size_t)total * 80;          // at most 40 KB
  const bool planes = is_plane_family(dtype);
  if (total <= 96) {
    if (M == 1) return (int)launch(planes ? down_combine_kernel<3, 2, 2> : down_combine_kernel<3, 0, 2>, grid, dim3(256), smem, st, a);
    return (int)launch(planes ? down_combine_kernel<3, 2, 3> : down_combine_kernel<3, 0, 3>, grid, dim3(256), smem, st, a);
  }
  if (total <= 192) return (int)launch(planes ? down_combine_kernel<6, 2, 1> : down_combine_kernel<6, 0, 1>, grid, dim3(256), smem, st, a);
  return (int)launch(planes ? down_combine_kernel<16, 2, 1> : down_combine_kernel<16, 0, 1>, grid, dim3(256), smem, st, a);
}

}  // extern "C"
