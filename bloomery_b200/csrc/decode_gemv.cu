// Quantised GEMV for the decode chain (m <= 8 activation rows), weights dequantised
// in registers and dotted with dp4a against q8 activations.
//
// Decode at one row is latency-bound, not bandwidth-bound, so the kernel is shaped to
// keep one DRAM round trip on the critical path:
//   * a warp owns R weight rows at a time and issues every load of its first tile into
//     registers BEFORE griddepcontrol.wait and before the activation prologue, so under
//     programmatic dependent launch the weight stream of kernel N+1 overlaps the tail
//     of kernel N and its own RMSNorm prologue;
//   * the prologue needs no second pass: q8 codes of x*gain do not depend on the RMS
//     scale (it is a per-row scalar), so sum-of-squares and quantisation run in one
//     sweep and the scale multiplies the finished dot products;
//   * blocks are type-uniform (a tile of 8*R rows never straddles two weight segments),
//     which keeps block-wide barriers out of divergent code.
// One launch covers up to four weight segments that share an input (q, k, v).
//
// Behavioural counterpart of q4k_gemv/q6k_gemv(_mcol) in crates/gpu/src/lib.rs:1604-1632
// and qwen3moe_qkv_q4k / qwen3moe_o_resid_q4k in crates/gpu/src/arch/qwen3moe/proj.rs:
// fixed lane split and a fixed xor-butterfly, so reruns are bit-identical and each row of
// an m-row call equals its own 1-row call.
#include "gemv_kernel.cuh"

namespace bl {

int g_use_pdl = 1;

template cudaError_t gemv_family<true, 0>(const GemvArgs&, const GemvPlan&, cudaStream_t);
template cudaError_t gemv_family<false, 0>(const GemvArgs&, const GemvPlan&, cudaStream_t);
extern template cudaError_t gemv_family<true, 1>(const GemvArgs&, const GemvPlan&, cudaStream_t);     // decode_gemv_float.cu
extern template cudaError_t gemv_family<true, 2>(const GemvArgs&, const GemvPlan&, cudaStream_t);     // decode_gemv_planes.cu
extern template cudaError_t gemv_family<false, 2>(const GemvArgs&, const GemvPlan&, cudaStream_t);

// Segments (but for their pointers) and shape of a call; fam: the kernel family of its weight types.  A contract code, or 0.
static int gemv_plan(int nseg, const int* rows, const int* wtypes, int K, int M, bool norm, bool reduce, int sm_count, GemvSeg* seg,
                     GemvPlan& p, int& fam) {
  bool floatw = false, planes = false, ggml = false;
  double total = 0, cost[4];
  long rbs[4];
  for (int s = 0; s < nseg; ++s) {
    rbs[s] = resident_row_bytes(wtypes[s], K);
    BL_REQUIRE(rbs[s] > 0, BL_ERR_TYPE);
    BL_REQUIRE(rows[s] >= 1, BL_ERR_SHAPE);
    cost[s] = (double)rows[s] * rbs[s] * (wtypes[s] == WT_Q6_K ? 1.5 : 1.0);
    total += cost[s];
    if (wtypes[s] == WT_F32 || wtypes[s] == WT_F16 || wtypes[s] == WT_BF16) floatw = true;
    else if (wtypes[s] == WT_NVFP4 || wtypes[s] == WT_FP8_B128 || wtypes[s] == WT_Q4_0 || wtypes[s] == WT_Q4_1 ||
             wtypes[s] == WT_Q5_0 || wtypes[s] == WT_Q5_1 || wtypes[s] == WT_Q2_K || wtypes[s] == WT_Q3_K) planes = true;
    else ggml = true;
  }
  BL_REQUIRE(!(floatw && !norm), BL_ERR_TYPE);
  BL_REQUIRE(!(planes && (floatw || ggml)), BL_ERR_TYPE);   // one family per call
  fam = planes ? 2 : floatw ? 1 : 0;
  // One wave: at most two resident blocks per SM; each segment gets a share of the blocks
  // in proportion to its bytes (and half as many again for Q6_K, whose dots are twice those of Q4_K for 1.56 times
  // its bytes), never more blocks than it has 8-row groups.
  const int budget = 2 * sm_count;
  p.C = (K / 64 > 32) ? 2 : 1;
  p.grid = 0;
  int rpw_max = 1;
  for (int s = 0; s < nseg; ++s) {
    int nb = (int)((double)budget * (cost[s] / total));
    const int cap = (rows[s] + 7) / 8;
    nb = nb < 1 ? 1 : nb > cap ? cap : nb;
    seg[s] = GemvSeg{nullptr, rows[s], wtypes[s], p.grid, nb, rbs[s]};
    p.grid += nb;
    const int rpw = (rows[s] + nb * 8 - 1) / (nb * 8);
    rpw_max = rpw > rpw_max ? rpw : rpw_max;
  }
  p.MB = M <= 1 ? 1 : M <= 2 ? 2 : M <= 4 ? 4 : kMaxRows;
  const size_t one_by_one = gemv_smem(M, K, floatw || norm);
  p.multi = M > 1 && !reduce && (p.C == 1 || (K / 64 <= 64 && (fam != 2 || (!norm && M > 2)) && 2 * (one_by_one + 1024) <= kSmemOfProcessor));
  const int most = p.multi ? (fam == 0 ? 3 : fam == 1 ? 2 : 1) : p.MB == kMaxRows ? 2 : 3;
  p.R = p.C == 2 ? 1 : rpw_max < most ? rpw_max : most;
  p.smem = p.multi ? one_by_one : gemv_smem(p.MB, K, floatw);
  return 0;
}

}  // namespace bl

using namespace bl;

extern "C" {

void bl_set_pdl(int on) { g_use_pdl = on ? 1 : 0; }

// out[m, :] = (resid[m, :] +) W_seg * act(m), for up to four weight segments.
//   norm != 0: act = q8(RMSNorm(x[m]) * gain); else act = (xq, xds) given.
// row_seq (optional, M > 1): rows with a negative entry fill a bucket and nothing else; they need not be computed.  Not with push_desc:
// the ranks that add the pushed rows up wait for every one of them.
// Returns 0, a negative contract code, or a positive cudaError_t.
int bl_gemv(int nseg, const void* const* w, const int* rows, const int* wtypes, int K, int M,
            int norm, const float* x, long x_stride, const float* gain, float eps,
            const int8_t* xq, const float* xds,
            float* out, long out_stride, const float* resid, long resid_stride,
            const void* red_desc, const void* push_desc, unsigned* fault, int layer, int sm_count,
            int n_pf, const void* const* pf_ptr, const long* pf_bytes, const int* row_seq, cudaStream_t st) {
  BL_REQUIRE(nseg >= 1 && nseg <= 4, BL_ERR_SHAPE);
  BL_REQUIRE(M >= 1 && M <= 8, BL_ERR_SHAPE);
  BL_REQUIRE(K > 0 && K % 256 == 0, BL_ERR_SHAPE);
  BL_REQUIRE(!norm || (K % 2048 == 0 || K % 64 == 0), BL_ERR_SHAPE);
  BL_REQUIRE(n_pf >= 0 && n_pf <= 6, BL_ERR_SHAPE);
  GemvArgs a = {};
  a.n_pf = n_pf;
  for (int i = 0; i < n_pf; ++i) {
    BL_REQUIRE(((uintptr_t)pf_ptr[i] & 15) == 0 && pf_bytes[i] >= 0, BL_ERR_ALIGN);
    a.pf_ptr[i] = (const uint8_t*)pf_ptr[i]; a.pf_bytes[i] = pf_bytes[i];
  }
  a.nseg = nseg;
  GemvPlan plan;
  int fam = 0;
  if (red_desc) a.red = *(const ReduceIn*)red_desc;
  const int bad = gemv_plan(nseg, rows, wtypes, K, M, norm, a.red.n_ranks > 0, sm_count, a.seg, plan, fam);
  if (bad) return bad;
  for (int s = 0; s < nseg; ++s) {
    BL_REQUIRE(((uintptr_t)w[s] & 15) == 0, BL_ERR_ALIGN);
    a.seg[s].w = (const uint8_t*)w[s];
  }
  a.K = K; a.M = M;
  a.row_seq = row_seq;
  a.x = x; a.x_stride = x_stride; a.gain = gain; a.eps = eps;
  a.xq = xq; a.xds = (const float2*)xds;
  a.out = out; a.out_stride = out_stride; a.resid = resid; a.resid_stride = resid_stride;
  a.fault = fault; a.layer = layer;
  if (red_desc) { BL_REQUIRE(norm && a.red.n_ranks <= kMaxRanks && a.red.H == K, BL_ERR_SHAPE); }
  BL_REQUIRE(!(push_desc && row_seq), BL_ERR_SHAPE);
  if (push_desc) { a.push = *(const PushOut*)push_desc; BL_REQUIRE(a.push.n_ranks <= kMaxRanks, BL_ERR_SHAPE); }
  BL_REQUIRE(plan.smem <= 200 * 1024, BL_ERR_LIMIT);
  cudaError_t e;
  if (fam == 2) e = norm ? gemv_family<true, 2>(a, plan, st) : gemv_family<false, 2>(a, plan, st);
  else if (norm) e = fam == 1 ? gemv_family<true, 1>(a, plan, st) : gemv_family<true, 0>(a, plan, st);
  else e = gemv_family<false, 0>(a, plan, st);
  return (int)e;
}

// The launch that bl_gemv makes of such a call: {blocks, R, C, rows as a whole (0: one by one), bytes of shared memory}.
int bl_gemv_plan(int nseg, const int* rows, const int* wtypes, int K, int M, int norm, int reduce, int sm_count, long* out) {
  BL_REQUIRE(nseg >= 1 && nseg <= 4 && M >= 1 && M <= 8 && K > 0 && K % 256 == 0, BL_ERR_SHAPE);
  GemvSeg seg[4];
  GemvPlan p;
  int fam = 0;
  const int bad = gemv_plan(nseg, rows, wtypes, K, M, norm, reduce != 0, sm_count, seg, p, fam);
  if (bad) return bad;
  out[0] = p.grid; out[1] = p.R; out[2] = p.C; out[3] = p.multi ? 0 : p.MB; out[4] = (long)p.smem;
  return 0;
}

}  // extern "C"
