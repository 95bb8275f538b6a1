// Grouped GEMM on tcgen05 whose weight operand stays block-quantised in HBM (sm_100a only):
//   C[t, n] = sum_k X[t, k] * W[g][n, k]          W resident Q4_K / Q5_K / Q6_K / Q8_0, X bf16, fp32 accumulate
//
// The product is issued transposed: the 128 weight rows of a tile are the M side of the MMA and the tokens the N side
// (32, 64 or 128 per tile), so a decode batch of a few rows per expert pays for the tokens it has instead of a 128-row
// tile, and a prompt tile expands each weight once for 128 tokens.
//
//   * weights: sixteen producer warps decode 64-value units in registers and store bf16 into the MMA's A operand in
//     tensor memory (tcgen05.st, lane = weight row) -- the bf16 form of a weight never exists in HBM or shared memory
//     (in shared memory its writes and the MMA's reads bound the launch).  The quantised super-blocks of the tile's 128
//     rows reach the producers through a ring of raw TMA boxes ([128 rows x one super-block] of bytes, several in
//     flight per SM, which is what a pass bound by weight streaming needs), or, for types without super-blocks, by
//     register loads one item ahead;
//   * tokens: one TMA thread loads [tokens x 64] bf16 boxes into the B stage of the same index;
//   * one elected thread issues tcgen05.mma (M = 128, N = tokens, K = 16) into TMEM, two accumulators (one for gate+up
//     at 128 tokens), so four epilogue warps read tile i back with tcgen05.ld while tile i + 1 accumulates;
//   * "dual" mode runs gate and up in one main loop and the epilogue writes silu(gate) * up;
//   * the epilogue scatters and scales like the bf16 GEMM (dst_row / row_scale / resid): lane = weight row, so one
//     token's 32 outputs of a warp are one contiguous 128-byte (fp32) or 64-byte (bf16) store.
//
// Every mbarrier wait is bounded by the global timer; on expiry the CTA raises status word 1, leaves its loops,
// frees its TMEM and returns.
//
// Role in the reference: the int8 mma.sync grouped GEMMs that read quantised experts directly
// (crates/gpu/src/gemm/q4k_sel.rs, q6k_sel.rs, kernels.rs); there the activations are quantised to q8 and the
// product runs on mma.sync -- here the weights are expanded in flight and the product runs on tcgen05.
#define BL_UNITS_GENERIC_LD 1      // weight units are also read out of shared memory here: plain loads
#include "tc_common.cuh"

#include <type_traits>

namespace bl {

constexpr int QBM = 128;                  // weight rows per tile (MMA M)
constexpr int QBK = 128;                  // depth per stage: two swizzle atoms of 64 values
constexpr int QPRODUCERS = 512;           // threads that expand weights: four per weight row
constexpr int QTHREADS = 256 + QPRODUCERS;

struct QTile { int group, row0, row_end, pad; };   // token tile: rows row0 .. of X use weight matrix `group`

struct QGemmArgs {
  const uint8_t* w;           // [n_groups][N rows][row_bytes]
  const uint8_t* w2;          // dual: the second matrix (same type and shape)
  long group_bytes, row_bytes;
  int N, K;
  int tiles_w;                // ceil(N / 128)
  const QTile* tiles;
  const int* n_tiles;
  int max_tiles;
  float* c_f32;
  __nv_bfloat16* c_bf16;
  long ldc;
  const int* dst_row;         // optional scatter of token rows (< 0 = drop)
  const float* row_scale;     // optional per-token factor
  const float* resid;         // optional addend, indexed like the output
  long ldr;
  unsigned* status;
  int fixed_tiles;            // the table holds max_tiles tiles and was written before the launches in flight
  int splits;                 // CTAs that share a tile's depth (1 with w2)
  float* partial;             // splits > 1: [tiles][splits][tile rows][128] sums
  int* tickets;               // splits > 1: one per tile, zero between launches
};

__device__ __forceinline__ uint4 q_pack8(const float* v) {
  uint4 o;
  __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
  __nv_bfloat162 c = __floats2bfloat162_rn(v[4], v[5]), d = __floats2bfloat162_rn(v[6], v[7]);
  o.x = *reinterpret_cast<uint32_t*>(&a); o.y = *reinterpret_cast<uint32_t*>(&b);
  o.z = *reinterpret_cast<uint32_t*>(&c); o.w = *reinterpret_cast<uint32_t*>(&d);
  return o;
}

// eight values as bf16 and as bf16 of what that leaves (exact in fp32)
__device__ __forceinline__ void q_split8(const float* v, uint4& hi, uint4& lo) {
  hi = q_pack8(v);
  const uint32_t h[4] = {hi.x, hi.y, hi.z, hi.w};
  float r[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    r[2 * i] = v[2 * i] - __uint_as_float(h[i] << 16);
    r[2 * i + 1] = v[2 * i + 1] - __uint_as_float(h[i] & 0xFFFF0000u);
  }
  lo = q_pack8(r);
}

// How a weight reaches the tensor cores; see the expanders below.
enum QForm { Q_SHORT = 0, Q_EXACT = 1, Q_SPLIT = 2 };

// ---- fast expanders ---------------------------------------------------------------------
// Integer-to-float conversions run at a quarter of the FMA rate, so the K-quant expanders avoid them.
//   exact form (prompts): a code byte q (< 128) dropped into mantissa bits 16..22 of 1.0f reads as X = 1 + q / 128, and the
//   block's affine map v = s * q + o becomes one FMA v = (128 s) * X + (o - 128 s) on a packed pair (fma.rn.f32x2), rounded
//   to bf16 once.  The result equals the fp32 decode to within an fp32 rounding of the offset (a scale is an f16 times a
//   small integer, so the offset is exact unless s and o are far apart).
//   split form (prompts that would otherwise run on the chain, whose integer dots round no weight): the same fp32 value as a
//   bf16 and a bf16 remainder, 16 bits together.  The halves fill two consecutive stages over the same tokens, so the tensor
//   cores do twice the products, of which there is room, and the expanders write twice.
//   short form (decode rounds, which the expanders' integer pipe bounds): two code bytes become the bf16 pair
//   (128 + q0, 128 + q1) with one byte permute, a packed bf16 subtract gives (q0, q1) exactly and a packed bf16 FMA gives
//   s * q + o with s and o rounded to bf16: half the integer instructions.  Its error is at most 2^-9 (|s q| + |o|) and one bf16
//   rounding of the sum, which is no bound in ulps of the weight: near zero s q and o nearly cancel (Q4_K, Q5_K).  Gate+up
//   of 24 rows, 95 of 128 experts (Q4_K, 768 x 2048): 56 us short (33 us of blocks at the copy rate).
// FastUnit<T>::codes yields the unit's 64 code bytes in value order (16 words; word w belongs to group w / 4) and the
// (scale, offset) pair of each of the four groups of 16 values.
template <class T> struct FastUnit { static constexpr bool kHas = false; };

template <> struct FastUnit<Q4K> {
  static constexpr bool kHas = true;
  static __device__ __forceinline__ void codes(const Q4K::Regs& r, int u, uint32_t* cw, float* s, float* o) {
    const int j = u & 3;
    const uint32_t w[8] = {r.q0.x, r.q0.y, r.q0.z, r.q0.w, r.q1.x, r.q1.y, r.q1.z, r.q1.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) { cw[i] = w[i] & 0x0F0F0F0Fu; cw[8 + i] = (w[i] >> 4) & 0x0F0F0F0Fu; }
    int sc0, mn0, sc1, mn1;
    Q4K::scale_min(r, 2 * j, sc0, mn0);
    Q4K::scale_min(r, 2 * j + 1, sc1, mn1);
    const float d = half_bits_to_float((uint16_t)(r.dm & 0xFFFF)), dmin = half_bits_to_float((uint16_t)(r.dm >> 16));
    s[0] = s[1] = d * sc0; o[0] = o[1] = -(dmin * mn0);
    s[2] = s[3] = d * sc1; o[2] = o[3] = -(dmin * mn1);
  }
};
template <> struct FastUnit<Q5K> {
  static constexpr bool kHas = true;
  static __device__ __forceinline__ void codes(const Q5K::Regs& r, int u, uint32_t* cw, float* s, float* o) {
    const int j = u & 3;
    Q5K::codes(r, u, cw, cw + 8);
    Q4K::Regs t; t.s0 = r.s0; t.s1 = r.s1; t.s2 = r.s2;
    int sc0, mn0, sc1, mn1;
    Q4K::scale_min(t, 2 * j, sc0, mn0);
    Q4K::scale_min(t, 2 * j + 1, sc1, mn1);
    const float d = half_bits_to_float((uint16_t)(r.dm & 0xFFFF)), dmin = half_bits_to_float((uint16_t)(r.dm >> 16));
    s[0] = s[1] = d * sc0; o[0] = o[1] = -(dmin * mn0);
    s[2] = s[3] = d * sc1; o[2] = o[3] = -(dmin * mn1);
  }
};
template <> struct FastUnit<Q6K> {
  static constexpr bool kHas = true;
  static __device__ __forceinline__ void codes(const Q6K::Regs& r, int u, uint32_t* cw, float* s, float* o) {
    const int n = (u >> 1) & 1, h = u & 1;
    uint32_t c[4][4];
    Q6K::codes(r, c);
    const float d = half_bits_to_float((uint16_t)r.d);
#pragma unroll
    for (int g = 0; g < 4; ++g) {
#pragma unroll
      for (int i = 0; i < 4; ++i) cw[4 * g + i] = c[g][i];
      s[g] = d * (float)Q6K::scale(r, 8 * n + 2 * g + h);
      o[g] = -32.0f * s[g];
    }
  }
};

// (a * x0 + c, a * x1 + c) with one packed FMA
__device__ __forceinline__ void fma2_f32(uint32_t x0, uint32_t x1, float a, float c, float* v) {
  asm("{\n\t.reg .b64 ra, rx, rc, rr;\n\t"
      "mov.b64 ra, {%2, %2};\n\tmov.b64 rx, {%3, %4};\n\tmov.b64 rc, {%5, %5};\n\t"
      "fma.rn.f32x2 rr, ra, rx, rc;\n\tmov.b64 {%0, %1}, rr;\n\t}"
      : "=f"(v[0]), "=f"(v[1]) : "f"(a), "r"(x0), "r"(x1), "f"(c));
}
__device__ __forceinline__ void fast8(uint32_t w0, uint32_t w1, float a, float c, float* v) {
  w0 |= 0x80808080u; w1 |= 0x80808080u;
  fma2_f32(__byte_perm(w0, 0x3F000000u, 0x7044), __byte_perm(w0, 0x3F000000u, 0x7144), a, c, v);
  fma2_f32(__byte_perm(w0, 0x3F000000u, 0x7244), __byte_perm(w0, 0x3F000000u, 0x7344), a, c, v + 2);
  fma2_f32(__byte_perm(w1, 0x3F000000u, 0x7044), __byte_perm(w1, 0x3F000000u, 0x7144), a, c, v + 4);
  fma2_f32(__byte_perm(w1, 0x3F000000u, 0x7244), __byte_perm(w1, 0x3F000000u, 0x7344), a, c, v + 6);
}

// bf16x2 FMA on raw register pairs
__device__ __forceinline__ uint32_t bf2_fma(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ uint32_t bf2_sub(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t bf2_dup(float v) {
  __nv_bfloat162 p = __float2bfloat162_rn(v);
  return *reinterpret_cast<uint32_t*>(&p);
}
__device__ __forceinline__ uint4 short8(uint32_t w0, uint32_t w1, uint32_t s2, uint32_t o2) {
  constexpr uint32_t k128 = 0x43004300u;                       // (128, 128) in bf16
  uint4 out;
  out.x = bf2_fma(bf2_sub(__byte_perm(w0, k128, 0x5150), k128), s2, o2);   // bytes (low to high): q0, 0x43, q1, 0x43
  out.y = bf2_fma(bf2_sub(__byte_perm(w0, k128, 0x5352), k128), s2, o2);
  out.z = bf2_fma(bf2_sub(__byte_perm(w1, k128, 0x5150), k128), s2, o2);
  out.w = bf2_fma(bf2_sub(__byte_perm(w1, k128, 0x5352), k128), s2, o2);
  return out;
}

// ---- slabs: the super-block types, whole stages at a time ------------------------------------
// A slab is 64 consecutive values.  Slab<T>::Regs holds a row's 128 values of a stage (slabs i and i + 1 of its super-block
// `sb`, i even) with their scales; codes() yields the x-th one's 64 code bytes in value order (16 words) and the (scale,
// offset) pair of each of its four groups of 16.  The packed scales are taken apart four at a time, and a byte becomes a float
// as the low mantissa byte of 2^23: half of an expander's integer instructions were those of its scales.
template <class T> struct Slab;

// byte `SEL` of w as a float, less `bias`
template <int SEL>
__device__ __forceinline__ float byte_float(uint32_t w, float bias = 8388608.0f) {
  return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440 + SEL)) - bias;
}
// scales and offsets of slab i: sub-blocks 2i and 2i + 1 of the eight 6-bit (scale, min) pairs of Q4_K and Q5_K
__device__ __forceinline__ void k_scales(const u32x4& hdr, int i, float* s, float* o) {
  uint32_t sw, mw;
  if (i < 2) {
    sw = hdr.y & 0x3F3F3F3Fu;
    mw = hdr.z & 0x3F3F3F3Fu;
  } else {
    sw = (hdr.w & 0x0F0F0F0Fu) | ((hdr.y >> 2) & 0x30303030u);
    mw = ((hdr.w >> 4) & 0x0F0F0F0Fu) | ((hdr.z >> 2) & 0x30303030u);
  }
  sw >>= 16 * (i & 1);
  mw >>= 16 * (i & 1);
  const float d = half_bits_to_float((uint16_t)(hdr.x & 0xFFFF)), dmin = half_bits_to_float((uint16_t)(hdr.x >> 16));
  s[0] = s[1] = d * byte_float<0>(sw); o[0] = o[1] = -(dmin * byte_float<0>(mw));
  s[2] = s[3] = d * byte_float<1>(sw); o[2] = o[3] = -(dmin * byte_float<1>(mw));
}

template <> struct Slab<Q4K> {
  static constexpr bool kHas = true;
  struct Regs { u32x4 hdr, q[4]; };
  static __device__ __forceinline__ void load(const uint8_t* sb, int i, Regs& r) {
    r.hdr = ld128(sb);
#pragma unroll
    for (int x = 0; x < 4; ++x) r.q[x] = ld128(sb + 16 + 32 * i + 16 * x);
  }
  static __device__ __forceinline__ void codes(const Regs& r, int x, int i, uint32_t* cw, float* s, float* o) {
    const u32x4 &a = r.q[2 * x], &b = r.q[2 * x + 1];
    const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int k = 0; k < 8; ++k) { cw[k] = w[k] & 0x0F0F0F0Fu; cw[8 + k] = (w[k] >> 4) & 0x0F0F0F0Fu; }
    k_scales(r.hdr, i, s, o);
  }
};
template <> struct Slab<Q5K> {
  static constexpr bool kHas = true;
  struct Regs { u32x4 hdr, h[2], q[4]; };
  static __device__ __forceinline__ void load(const uint8_t* sb, int i, Regs& r) {
    r.hdr = ld128(sb);
    r.h[0] = ld128(sb + 16);
    r.h[1] = ld128(sb + 32);
#pragma unroll
    for (int x = 0; x < 4; ++x) r.q[x] = ld128(sb + 48 + 32 * i + 16 * x);
  }
  static __device__ __forceinline__ void codes(const Regs& r, int x, int i, uint32_t* cw, float* s, float* o) {
    const u32x4 &a = r.q[2 * x], &b = r.q[2 * x + 1];
    const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    const uint32_t h[8] = {r.h[0].x, r.h[0].y, r.h[0].z, r.h[0].w, r.h[1].x, r.h[1].y, r.h[1].z, r.h[1].w};
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint32_t hb = h[k] >> (2 * i);
      cw[k] = (w[k] & 0x0F0F0F0Fu) | ((hb & 0x01010101u) << 4);
      cw[8 + k] = ((w[k] >> 4) & 0x0F0F0F0Fu) | ((hb & 0x02020202u) << 3);
    }
    k_scales(r.hdr, i, s, o);
  }
};
// Both slabs of a half super-block read the same bytes: the even one their low nibbles, the odd one the high ones.
template <> struct Slab<Q6K> {
  static constexpr bool kHas = true;
  struct Regs { u32x4 l[4], h[2]; uint32_t sc[2], d; };
  static __device__ __forceinline__ void load(const uint8_t* sb, int i, Regs& r) {
    const uint8_t* p = sb + 64 * (i >> 1);
#pragma unroll
    for (int x = 0; x < 4; ++x) r.l[x] = ld128(p + 16 * x);
#pragma unroll
    for (int x = 0; x < 2; ++x) r.h[x] = ld128(sb + 128 + 32 * (i >> 1) + 16 * x);
#pragma unroll
    for (int x = 0; x < 2; ++x) r.sc[x] = ld32(sb + 192 + 4 * (i + x));
    r.d = ld32(sb + 208);
  }
  static __device__ __forceinline__ void codes(const Regs& r, int x, int i, uint32_t* cw, float* s, float* o) {
    const int sh = 4 * x;
    const uint32_t h[8] = {r.h[0].x, r.h[0].y, r.h[0].z, r.h[0].w, r.h[1].x, r.h[1].y, r.h[1].z, r.h[1].w};
    const uint32_t w[16] = {r.l[0].x, r.l[0].y, r.l[0].z, r.l[0].w, r.l[1].x, r.l[1].y, r.l[1].z, r.l[1].w,
                            r.l[2].x, r.l[2].y, r.l[2].z, r.l[2].w, r.l[3].x, r.l[3].y, r.l[3].z, r.l[3].w};
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint32_t hb = h[k] >> sh;
      cw[k] = ((w[k] >> sh) & 0x0F0F0F0Fu) | ((hb & 0x03030303u) << 4);
      cw[8 + k] = ((w[8 + k] >> sh) & 0x0F0F0F0Fu) | ((hb & 0x0C0C0C0Cu) << 2);
    }
    const float d = half_bits_to_float((uint16_t)(r.d & 0xFFFF));
    const uint32_t sc = r.sc[x] ^ 0x80808080u;                      // signed bytes, 128 up
    s[0] = d * byte_float<0>(sc, 8388736.0f); s[1] = d * byte_float<1>(sc, 8388736.0f);
    s[2] = d * byte_float<2>(sc, 8388736.0f); s[3] = d * byte_float<3>(sc, 8388736.0f);
#pragma unroll
    for (int g = 0; g < 4; ++g) o[g] = -32.0f * s[g];
  }
};

// Slab x of `regs` into columns ta .. ta + 31.  `ready` waits for the stage behind the arithmetic, in front of the store.  (The split
// form goes unit by unit: in slabs the down products of 36 rows took the same time, and gate+up, whose three stages hold a
// block and a half, 168 us instead of 148.)
template <class T, int FORM, class Ready>
__device__ __forceinline__ bool expand_slab(const typename Slab<T>::Regs& regs, int x, int i, uint32_t ta, Ready ready) {
  uint32_t cw[16];
  float s[4], o[4];
  Slab<T>::codes(regs, x, i + x, cw, s, o);
  uint32_t v[32];
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    const uint32_t s2 = bf2_dup(s[g]), o2 = bf2_dup(o[g]);
    const float a = 128.0f * s[g], c = o[g] - a;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint4 q;
      if constexpr (FORM == Q_SHORT) {
        q = short8(cw[4 * g + 2 * h], cw[4 * g + 2 * h + 1], s2, o2);
      } else {
        float f[8];
        fast8(cw[4 * g + 2 * h], cw[4 * g + 2 * h + 1], a, c, f);
        q = q_pack8(f);
      }
      v[8 * g + 4 * h] = q.x; v[8 * g + 4 * h + 1] = q.y; v[8 * g + 4 * h + 2] = q.z; v[8 * g + 4 * h + 3] = q.w;
    }
  }
  if (!ready()) return false;
  tmem_st32(ta, v);
  return true;
}

// ---- float-coded types ---------------------------------------------------------------------
// ChunkUnit<T>::values(regs, pre, j) yields values 8j .. 8j+7 of the unit, never holding the unit's 64 floats.
//   FP8 (E4M3 codes, one f32 scale per 128 values): the hardware converter takes two codes to an f16 pair; the pair
//   widens to f32, takes the block scale and is rounded to bf16 once.
//   NVFP4 (E2M1 codes, E4M3 scale per 16 values, f32 tensor scale): a code's magnitude is one of eight values, so two
//   byte permutes with the code nibbles as selectors look up the low and the high byte of bf16(2 * magnitude) for four
//   codes at once; the sign bits are gathered with two more permutes.  Exact form: the pair widens to f32, takes the f32
//   scale and is rounded to bf16 once, as the expander of the bf16 copies does.  Short form: one packed bf16 multiply by
//   the scale rounded to bf16, so a weight is rounded twice (relative weight error over random codes and scales 2.1e-3
//   against 1.5e-3 once).
template <class T> struct ChunkUnit { static constexpr bool kHas = false, kOneForm = true; };

template <> struct ChunkUnit<Fp8B128> {
  static constexpr bool kHas = true;
  static constexpr bool kOneForm = true;
  struct Pre { float sc; };
  static __device__ __forceinline__ Pre pre(const Fp8B128::Regs& r) { return Pre{r.sc}; }
  static __device__ __forceinline__ void values(const Fp8B128::Regs& r, const Pre& pr, int j, float* f) {
    const u32x4& q = r.q[j >> 1];
    const uint32_t w0 = (j & 1) ? q.z : q.x, w1 = (j & 1) ? q.w : q.y;
    e4m3x4_to_float(w0, f);
    e4m3x4_to_float(w1, f + 4);
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] *= pr.sc;
  }
};

template <> struct ChunkUnit<NvFp4> {
  static constexpr bool kHas = true;
  static constexpr bool kOneForm = false;
  struct Pre { float sc[4]; };
  static __device__ __forceinline__ Pre pre(const NvFp4::Regs& r) {
    Pre pr;
    e4m3x4_to_float(r.sc, pr.sc);
#pragma unroll
    for (int g = 0; g < 4; ++g) pr.sc[g] = pr.sc[g] * r.g * 0.5f;                  // the table below holds 2 * magnitude
    return pr;
  }
  // bf16 pairs of 2 * magnitude with their signs
  static __device__ __forceinline__ void codes(const NvFp4::Regs& r, int j, uint32_t* m) {
    const uint32_t w = j == 0 ? r.q0.x : j == 1 ? r.q0.y : j == 2 ? r.q0.z : j == 3 ? r.q0.w
                     : j == 4 ? r.q1.x : j == 5 ? r.q1.y : j == 6 ? r.q1.z : r.q1.w;
    const uint32_t sel = w & 0x77777777u;
    const uint32_t sodd = w & 0x80808080u, seven = (w << 4) & 0x80808080u;   // signs of the odd / the even codes
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t c = h ? sel >> 16 : sel;
      const uint32_t lo4 = __byte_perm(0x40008000u, 0x4000C080u, c);
      const uint32_t hi4 = __byte_perm(0x40403F00u, 0x41414040u, c) | __byte_perm(seven, sodd, h ? 0x7362 : 0x5140);
      m[2 * h] = __byte_perm(lo4, hi4, 0x5140);
      m[2 * h + 1] = __byte_perm(lo4, hi4, 0x7362);
    }
  }
  static __device__ __forceinline__ void values(const NvFp4::Regs& r, const Pre& pr, int j, float* f) {
    uint32_t m[4];
    codes(r, j, m);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      f[2 * i] = __uint_as_float(m[i] << 16) * pr.sc[j >> 1];
      f[2 * i + 1] = __uint_as_float(m[i] & 0xFFFF0000u) * pr.sc[j >> 1];
    }
  }
  static __device__ __forceinline__ uint4 short8(const NvFp4::Regs& r, const Pre& pr, int j) {
    uint32_t m[4];
    codes(r, j, m);
    const uint32_t s2 = bf2_dup(pr.sc[j >> 1]);
    return make_uint4(bf2_fma(m[0], s2, 0u), bf2_fma(m[1], s2, 0u), bf2_fma(m[2], s2, 0u), bf2_fma(m[3], s2, 0u));
  }
};

// Unit u (64 values of this thread's weight row) of stage kb into the A operand in tensor memory: lane = weight row,
// 32-bit column c of the stage holds values 2c and 2c + 1.  A unit's groups of 16 values are contiguous in the row, so
// each is one 8-column store (split form: a second one at the next stage, `ta_lo`).  Warp-collective.
template <class T, int FORM>
__device__ __forceinline__ void expand_unit(const typename Unit<T>::Regs& regs, int u, int kb, uint32_t ta, uint32_t ta_lo) {
  auto col = [&](int g) { return (uint32_t)((Unit<T>::pos(u, 16 * g) - QBK * kb) >> 1); };
  auto put = [&](int g, const float* v) {
    if constexpr (FORM == Q_SPLIT) {
      uint4 h0, h1, l0, l1;
      q_split8(v, h0, l0);
      q_split8(v + 8, h1, l1);
      tmem_st8(ta + col(g), h0, h1);
      tmem_st8(ta_lo + col(g), l0, l1);
    } else {
      tmem_st8(ta + col(g), q_pack8(v), q_pack8(v + 8));
    }
  };
  if constexpr (FastUnit<T>::kHas) {
    uint32_t cw[16];
    float s[4], o[4];
    FastUnit<T>::codes(regs, u, cw, s, o);
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const float a = 128.0f * s[g], c = o[g] - a;
      float v[16];
      fast8(cw[4 * g], cw[4 * g + 1], a, c, v);
      fast8(cw[4 * g + 2], cw[4 * g + 3], a, c, v + 8);
      put(g, v);
    }
  } else if constexpr (ChunkUnit<T>::kHas) {
    using C = ChunkUnit<T>;
    const typename C::Pre pr = C::pre(regs);
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      if constexpr (FORM == Q_SHORT && !C::kOneForm) {
        tmem_st8(ta + col(g), C::short8(regs, pr, 2 * g), C::short8(regs, pr, 2 * g + 1));
      } else {
        float v[16];
        C::values(regs, pr, 2 * g, v);
        C::values(regs, pr, 2 * g + 1, v + 8);
        put(g, v);
      }
    }
  } else {
    float v[64];
    Unit<T>::decodeu(regs, u, v);
#pragma unroll
    for (int g = 0; g < 4; ++g) put(g, v + 16 * g);
  }
}

// Raw ring: slots of [matrices][128 rows][super-block bytes]; 0 slots = the register-load path.
template <class T> struct SbBytes { static constexpr int v = 0; };
template <> struct SbBytes<Q4K> { static constexpr int v = Q4K::kSbBytes; };
template <> struct SbBytes<Q5K> { static constexpr int v = Q5K::kSbBytes; };
template <> struct SbBytes<Q6K> { static constexpr int v = Q6K::kSbBytes; };
// Tensor memory (512 columns): accumulators of all tokens first (two sets; one for gate+up at 128 tokens, where two
// would leave nothing), the A stages behind them.
__host__ __device__ constexpr int q_accs(bool dual, int bn) { return (dual ? 2 : 1) * bn > 128 ? 1 : 2; }
__host__ __device__ constexpr int q_stages(bool dual, int bn) {
  const int n = (512 - q_accs(dual, bn) * (dual ? 2 : 1) * bn) / ((dual ? 2 : 1) * (QBK / 2));
  return n > 6 ? 6 : n;
}
// Whole stages by groups of four warps
__host__ __device__ constexpr bool q_slabs(int sb_bytes, int form) { return sb_bytes > 0 && form != Q_SPLIT; }
// One matrix in slabs: a warp waits for every second raw slot only.  With an odd ring it skips every other phase of a slot, and a
// wait by parity would pass where the copy of super-block s - slots has not landed yet.  It has where s - slots is among those
// that are known to have been read: the warp's own stage of s - 2 waited for the MMAs of one turn of the ring before, so all
// super-blocks up to s - 2 - ceil(stages / 2) have been.
__host__ __device__ constexpr int q_raw_slots(int sb_bytes, bool dual, int bn, int form) {
  if (sb_bytes == 0) return 0;
  int n = (220 * 1024 - q_stages(dual, bn) * 2 * bn * 128) / ((dual ? 2 : 1) * QBM * sb_bytes);
  if (n > 6) n = 6;
  if (!dual && q_slabs(sb_bytes, form) && n % 2 == 1 && n < 2 + (q_stages(dual, bn) + 1) / 2) --n;
  return n;
}

// 768 threads: warp 0 = TMA of the token tiles, warp 1 = MMA issuer and TMEM owner, warps 2..5 = epilogue, warp 6 = TMA
// of the raw weight super-blocks, warp 7 idle, warps 8..23 = weight expanders (warp id modulo 4 = TMEM lane quarter).
template <class T, bool DUAL, int BN, int FORM>
__global__ void __launch_bounds__(QTHREADS, 1)
qgemm_kernel(const __grid_constant__ CUtensorMap tma_x, const __grid_constant__ CUtensorMap tma_w,
             const __grid_constant__ CUtensorMap tma_w2, const QGemmArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  constexpr int SB = SbBytes<T>::v;
  constexpr int STAGES = q_stages(DUAL, BN);
  constexpr int RS = q_raw_slots(SB, DUAL, BN, FORM);                // raw ring slots (0: register loads)
  constexpr int RAW_MAT = QBM * SB;                                  // one matrix's 128 super-blocks
  constexpr int RAW_SLOT = (DUAL ? 2 : 1) * RAW_MAT;
  constexpr int B_ATOM = BN * 128;
  constexpr int B_STAGE = 2 * B_ATOM;
  constexpr int NACC = q_accs(DUAL, BN);
  constexpr int ACC_COLS = (DUAL ? 2 : 1) * BN;
  constexpr int A_MAT = QBK / 2;                                     // columns of one matrix's stage
  constexpr int A_COLS = (DUAL ? 2 : 1) * A_MAT;
  constexpr int HALVES = FORM == Q_SPLIT ? 2 : 1;                    // stages that hold one 128-deep block of weights
  constexpr bool SLABS = q_slabs(SB, FORM);                          // a group of four warps fills a matrix's stage alone
  constexpr int FILLERS = (DUAL ? 2 : 1) * (SLABS ? 4 : 8);          // warps that write one stage
  constexpr int READERS = SLABS && !DUAL ? 8 : 16;                   // warps that read a raw slot
  __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full[2], acc_empty[2];
  __shared__ __align__(8) uint64_t raw_full[RS > 0 ? RS : 1], raw_empty[RS > 0 ? RS : 1];
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_abort, s_last;
  uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* const raw_ring = smem + (size_t)STAGES * B_STAGE;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1 + FILLERS); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 4); }
    for (int r = 0; r < RS; ++r) { mbar_init(&raw_full[r], 1); mbar_init(&raw_empty[r], READERS); }
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // Weights never change, and neither does the tile table of a dense product: its weight stream starts while the launch
  // that writes the activations still runs.  Every other role waits for that launch.
  if (!(a.fixed_tiles && warp >= 6)) {
    pdl_wait();
    pdl_launch();
  }
  const uint32_t tmem_base = s_tmem_base;
  const uint32_t tmem_a = tmem_base + NACC * ACC_COLS;
  volatile int* abort_flag = &s_abort;

  const int n_tt = a.fixed_tiles ? a.max_tiles : min(*a.n_tiles, a.max_tiles);
  const int total_tiles = n_tt * a.tiles_w * a.splits;
  const int kblocks = a.K / QBK / a.splits;                          // stages of one tile: an even number

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0; uint32_t phase = 0;
      int issued = 0;
      for (int t = blockIdx.x; t < total_tiles && !*abort_flag; t += gridDim.x) {
        const QTile mt = a.tiles[t / a.splits / a.tiles_w];
        const int kb0 = (t % a.splits) * kblocks;
        for (int s = kb0 * HALVES; s < (kb0 + kblocks) * HALVES; ++s) {
          const int kb = s / HALVES;
          if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag)) break;
          uint8_t* sb = smem + (size_t)stage * B_STAGE;
          mbar_expect_tx(&full_bar[stage], B_STAGE);
          tma_load_2d(sb, &tma_x, kb * QBK, mt.row0, &full_bar[stage]);
          tma_load_2d(sb + B_ATOM, &tma_x, kb * QBK + 64, mt.row0, &full_bar[stage]);
          ++issued;
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
      if (*abort_flag) {
        // copies of this thread may still be landing in shared memory: the CTA must not exit under them
        unsigned long long t0 = globaltimer();
        while (issued > 0 && globaltimer() - t0 < 2000000ull) {}
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = umma_idesc(QBM, BN);
    int stage = 0; uint32_t phase = 0;
    int it = 0;
    for (int t = blockIdx.x; t < total_tiles; t += gridDim.x) {
      const int ab = it % NACC;
      const uint32_t acc_phase = (it / NACC) & 1;
      ++it;
      if (!mbar_wait_warp(&acc_empty[ab], acc_phase ^ 1, abort_flag)) break;
      tc_fence_after();
      const uint32_t d0 = tmem_base + ab * ACC_COLS;
      bool ok = true;
      for (int s = 0; s < kblocks * HALVES; ++s) {
        if (!mbar_wait_warp(&full_bar[stage], phase, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t sb = smem_u32(smem + (size_t)stage * B_STAGE);
        const uint32_t ta = tmem_a + stage * A_COLS;
#pragma unroll
        for (int k = 0; k < QBK / UMMA_K; ++k) {
          const uint64_t db = umma_desc(sb + (k >> 2) * B_ATOM) + (uint64_t)((k & 3) * UMMA_K * 2 / 16);
          const uint32_t acc = (s > 0 || k > 0) ? 1u : 0u;
          umma_bf16_ta(d0, ta + k * (UMMA_K / 2), db, idesc, acc);
          if (DUAL) umma_bf16_ta(d0 + BN, ta + A_MAT + k * (UMMA_K / 2), db, idesc, acc);
        }
        umma_commit(&empty_bar[stage]);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      if (!ok) break;
      umma_commit(&acc_full[ab]);
    }
  } else if (warp < 6) {
    const int q = warp & 3;
    const TokenOut out{a.c_f32, a.c_bf16, (unsigned)a.ldc, a.row_scale, a.resid, (unsigned)a.ldr, a.N};
    int it = 0;
    for (int t = blockIdx.x; t < total_tiles; t += gridDim.x) {
      const int tile = t / a.splits;
      const QTile mt = a.tiles[tile / a.tiles_w];
      const int n = (tile % a.tiles_w) * QBM + q * 32 + lane;      // weight row = output column of this thread
      const int ab = it % NACC;
      const uint32_t acc_phase = (it / NACC) & 1;
      ++it;
      const int n_rows = min(BN, mt.row_end - mt.row0);            // token rows of this tile
      // lane l fetches the routing of token rows l, l + 32, ... while the products run; the store loop broadcasts it
      int out_row[BN / 32];
      float out_scale[BN / 32];
      if (DUAL || a.splits == 1) {
#pragma unroll
        for (int b = 0; b < BN / 32; ++b) {
          const int r_l = mt.row0 + 32 * b + lane;
          out_row[b] = -1;
          out_scale[b] = 1.0f;
          if (32 * b + lane < n_rows) {
            out_row[b] = a.dst_row ? a.dst_row[r_l] : r_l;
            if (a.row_scale) out_scale[b] = a.row_scale[r_l];
          }
        }
      }
      if (!__all_sync(0xFFFFFFFFu, mbar_wait(&acc_full[ab], acc_phase, abort_flag))) break;
      tc_fence_after();
      const uint32_t tbase = tmem_base + ((uint32_t)(q * 32) << 16) + ab * ACC_COLS;
      if (!DUAL && a.splits > 1) {
        // a share's sums: [tile][split][token][128 weight rows]; the CTA that arrives last adds them up, see the end
        float* const own = a.partial + (long)t * (BN * QBM) + q * 32 + lane;
#pragma unroll 1
        for (int c = 0; c < n_rows; c += 16) {
          uint32_t v[16];
          tmem_ld16(tbase + c, v);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) __stcg(own + (c + i) * QBM, __uint_as_float(v[i]));
        }
        __threadfence();
      } else {
#pragma unroll
        for (int b = 0; b < BN / 32; ++b) {
          if (32 * b >= n_rows) break;
#pragma unroll 1
          for (int h = 0; h < 32 && 32 * b + h < n_rows; h += 16) {
            uint32_t v[16], u[DUAL ? 16 : 1];
            tmem_ld16(tbase + 32 * b + h, v);
            if constexpr (DUAL) tmem_ld16(tbase + BN + 32 * b + h, u);
            tmem_ld_wait();
            auto tokens = [&](auto count, int from) {
              constexpr int NT = decltype(count)::value;
              float f[NT];
#pragma unroll
              for (int i = 0; i < NT; ++i) {
                f[i] = __uint_as_float(v[from + i]);
                if constexpr (DUAL) f[i] = (f[i] / (1.0f + __expf(-f[i]))) * __uint_as_float(u[from + i]);
              }
              store_tokens<NT>(out, f, out_row[b], out_scale[b], h + from, n);
            };
            // a tile of a decode round has a few tokens: gate+up of 24 rows 57.5 us when all sixteen are worked out, 54.8 so
            const int left = n_rows - 32 * b - h;
            if (left > 8) {
              tokens(std::integral_constant<int, 16>{}, 0);
            } else {
              tokens(std::integral_constant<int, 4>{}, 0);
              if (left > 4) tokens(std::integral_constant<int, 4>{}, 4);
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[ab]);
    }
  } else if (warp == 6) {
    if (RS > 0 && lane == 0) {
      int rslot = 0; uint32_t rphase = 0;
      int issued = 0;
      for (int t = blockIdx.x; t < total_tiles && !*abort_flag; t += gridDim.x) {
        const int tile = t / a.splits;
        const int group = a.tiles[tile / a.tiles_w].group;
        const int n0 = (tile % a.tiles_w) * QBM;
        const int sb0 = (t % a.splits) * (kblocks / 2);
        for (int sbi = sb0; sbi < sb0 + kblocks / 2; ++sbi) {
          // rows n0 .. n0 + 127 of the group's matrix (rows past the matrix arrive as zeros and are never stored)
          if (!mbar_wait(&raw_empty[rslot], rphase ^ 1, abort_flag)) break;
          uint8_t* dst = raw_ring + (size_t)rslot * RAW_SLOT;
          mbar_expect_tx(&raw_full[rslot], RAW_SLOT);
          tma_load_3d(dst, &tma_w, sbi * SB, n0, group, &raw_full[rslot]);
          if (DUAL) tma_load_3d(dst + RAW_MAT, &tma_w2, sbi * SB, n0, group, &raw_full[rslot]);
          ++issued;
          if (++rslot == RS) { rslot = 0; rphase ^= 1; }
        }
      }
      if (*abort_flag) {
        unsigned long long t0 = globaltimer();
        while (issued > 0 && globaltimer() - t0 < 2000000ull) {}
      }
    }
  } else if (warp >= 8) {
    // Four groups of four warps, one per TMEM lane quarter: thread = weight row.  Gate+up: every group expands one unit
    // (matrix grp / 2, unit grp % 2) of every stage; one matrix: groups 0 and 1 the even stages, 2 and 3 the odd ones.
    // Slabs: a group fills whole stages, gate+up: groups 2m and 2m + 1 the even and odd stages of matrix m; one matrix: stage n by
    // group n % 4.
    using U = Unit<T>;
    constexpr int STEP = DUAL ? 1 : 2;                               // stages from one item of a group to its next
    const int grp = (warp - 8) >> 2, q = warp & 3;
    const int row = q * 32 + lane, mat = DUAL ? grp >> 1 : 0, half = grp & 1;
    const int kb_first = DUAL ? 0 : grp >> 1;
    const uint32_t ta0 = tmem_a + ((uint32_t)(q * 32) << 16) + mat * A_MAT;
    unsigned lin = (unsigned)kb_first * HALVES;                      // stages of this CTA so far, over all its tiles
    bool ok = true;
    auto emit = [&](int kb, const typename U::Regs& r) {
      const unsigned stage = lin % STAGES, phase = (lin / STAGES) & 1;
      const unsigned next = (lin + 1) % STAGES, next_phase = ((lin + 1) / STAGES) & 1;    // split form: the remainders' stage
      lin += STEP * HALVES;
      ok = __all_sync(0xFFFFFFFFu, mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag));
      if (ok && HALVES == 2) ok = __all_sync(0xFFFFFFFFu, mbar_wait(&empty_bar[next], next_phase ^ 1, abort_flag));
      if (!ok) return;
      tc_fence_after();
      expand_unit<T, FORM>(r, 2 * kb + half, kb, ta0 + stage * A_COLS, ta0 + next * A_COLS);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&full_bar[stage]);
        if (HALVES == 2) mbar_arrive(&full_bar[next]);
      }
    };
    if constexpr (SLABS) {
      // The hand-over of a stage (its stores must have landed) waits until the next values are read, which covers the stores'
      // latency.  It cannot lock the rings: a raw slot that this warp waits for is held up by a warp whose own stage is older
      // than the one kept back here, and stages are used in order.
      constexpr int NG = DUAL ? 2 : 4;                               // groups that share a matrix's stages, two a super-block
      static_assert(NG <= STAGES, "a group's next stage lies at most one turn of the ring ahead");
      const int mine = DUAL ? half : grp;
      int rslot = 0, stage = mine, turn = 0, pending = -1;           // stage: this group's next one
      uint32_t rphase = 0, phase = 0;
      auto hand_over = [&]() {
        if (pending < 0) return;
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&full_bar[pending]);
        pending = -1;
      };
      for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
        for (int sbi = 0; sbi < kblocks / 2 && ok; ++sbi) {
          const bool take = DUAL || turn == (mine >> 1);             // one matrix: the pairs of groups take super-blocks in turns
          turn ^= 1;
          if (take) {
            ok = mbar_wait_warp(&raw_full[rslot], rphase, abort_flag);
            if (!ok) break;
            typename Slab<T>::Regs r;
            Slab<T>::load(raw_ring + (size_t)rslot * RAW_SLOT + mat * RAW_MAT + row * SB, 2 * (mine & 1), r);
            __syncwarp();
            if (lane == 0) mbar_arrive(&raw_empty[rslot]);
            hand_over();
            auto ready = [&]() {
              ok = mbar_wait_warp(&empty_bar[stage], phase ^ 1, abort_flag);
              if (ok) tc_fence_after();
              return ok;
            };
            const uint32_t ta = ta0 + stage * A_COLS;
            if (!expand_slab<T, FORM>(r, 0, 2 * (mine & 1), ta, ready)) break;
            expand_slab<T, FORM>(r, 1, 2 * (mine & 1), ta + 32, [] { return true; });
            pending = stage;
            stage += NG;
            if (stage >= STAGES) { stage -= STAGES; phase ^= 1; }
          }
          if (++rslot == RS) { rslot = 0; rphase ^= 1; }
        }
      }
      if (ok) hand_over();
    } else if constexpr (RS > 0) {
      // raw ring: the tile's super-blocks arrive by TMA; a thread reads its row's units out of shared memory
      int rslot = 0; uint32_t rphase = 0;
      for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
        const int sb0 = (t % a.splits) * (kblocks / 2);
        for (int sbi = sb0; sbi < sb0 + kblocks / 2 && ok; ++sbi) {
          ok = __all_sync(0xFFFFFFFFu, mbar_wait(&raw_full[rslot], rphase, abort_flag));
          if (!ok) break;
          const uint8_t* rawrow = raw_ring + (size_t)rslot * RAW_SLOT + mat * RAW_MAT + row * SB - (long)sbi * SB;
          typename U::Regs r[DUAL ? 2 : 1];
#pragma unroll
          for (int h = 0; h < (DUAL ? 2 : 1); ++h) U::loadu(rawrow, 2 * (2 * sbi + h + kb_first) + half, a.K, r[h]);
          __syncwarp();
          if (lane == 0) mbar_arrive(&raw_empty[rslot]);
          if (++rslot == RS) { rslot = 0; rphase ^= 1; }
#pragma unroll
          for (int h = 0; h < (DUAL ? 2 : 1); ++h)
            if (ok) emit(2 * sbi + h + kb_first, r[h]);
        }
      }
    } else {
      // the blocks of a group's next item are fetched before the present one is decoded
      for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
        const int tile = t / a.splits;
        const int group = a.tiles[tile / a.tiles_w].group;
        int n = (tile % a.tiles_w) * QBM + row;
        n = n < a.N ? n : a.N - 1;                                   // rows past the matrix repeat the last one (never stored)
        const uint8_t* wrow = (mat ? a.w2 : a.w) + (long)group * a.group_bytes + (long)n * a.row_bytes;
        const int kb0 = (t % a.splits) * kblocks, kend = kb0 + kblocks;
        typename U::Regs ra, rb;
        int kb = kb0 + kb_first;
        U::loadu(wrow, 2 * kb + half, a.K, ra);
        for (; kb < kend && ok; kb += 2 * STEP) {
          if (kb + STEP < kend) U::loadu(wrow, 2 * (kb + STEP) + half, a.K, rb);
          emit(kb, ra);
          if (!ok) break;
          if (kb + 2 * STEP < kend) U::loadu(wrow, 2 * (kb + 2 * STEP) + half, a.K, ra);
          if (kb + STEP < kend) emit(kb + STEP, rb);
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if constexpr (!DUAL) {
    if (a.splits > 1) {
      // One share a CTA.  The CTA that finishes a tile's last share adds all of them up with all of its threads, eight in flight
      // each, in ascending order: same bits on every run.  (Four epilogue warps, one share after the other, took about 6 us of
      // the 21 of an output projection of 24 rows.)
      const int tile = (int)blockIdx.x / a.splits;
      if (threadIdx.x == 0) {
        __threadfence();
        s_last = tile < n_tt * a.tiles_w && atomicAdd(&a.tickets[tile], 1) == a.splits - 1;
        if (s_last) a.tickets[tile] = 0;                           // ready for the next launch
        __threadfence();
      }
      __syncthreads();
      if (s_last) {
        const QTile mt = a.tiles[tile / a.tiles_w];
        const int n = (tile % a.tiles_w) * QBM + (threadIdx.x & (QBM - 1)), n_rows = min(BN, mt.row_end - mt.row0);
        const float* part = a.partial + (long)tile * a.splits * (BN * QBM) + (threadIdx.x & (QBM - 1));
        if (n < a.N) {
#pragma unroll 2
          for (int i = threadIdx.x / QBM; i < n_rows; i += QTHREADS / QBM) {
            const int r = mt.row0 + i, orow = a.dst_row ? a.dst_row[r] : r;
            float f = 0.f;
            for (int sp0 = 0; sp0 < a.splits; sp0 += 8) {
              float v[8];
#pragma unroll
              for (int k = 0; k < 8; ++k)
                if (sp0 + k < a.splits) v[k] = __ldcg(part + ((long)(sp0 + k) * BN + i) * QBM);
#pragma unroll
              for (int k = 0; k < 8; ++k)
                if (sp0 + k < a.splits) f += v[k];
            }
            if (orow < 0) continue;
            if (a.row_scale) f *= a.row_scale[r];
            if (a.resid) f += a.resid[(long)orow * a.ldr + n];
            if (a.c_f32) a.c_f32[(long)orow * a.ldc + n] = f;
            else a.c_bf16[(long)orow * a.ldc + n] = __float2bfloat16_rn(f);
          }
        }
      }
    }
  }
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
  }
  if (threadIdx.x == 0 && s_abort && a.status) atomicMax(a.status, 1u);
}

template <class T, bool DUAL, int BN, int FORM>
static int qgemm_go(const CUtensorMap& mx, const QGemmArgs& a, int n_groups, int grid, cudaStream_t st) {
  constexpr int SB = SbBytes<T>::v;
  constexpr int RS = q_raw_slots(SB, DUAL, BN, FORM);
  constexpr size_t smem = (size_t)q_stages(DUAL, BN) * 2 * BN * 128 + (size_t)RS * (DUAL ? 2 : 1) * QBM * SB + 1024;
  static_assert(q_stages(DUAL, BN) >= 2 && (SB == 0 || RS >= 2), "operand rings");
  CUtensorMap mw = mx, mw2 = mx;
  if (RS > 0) {
    cuuint64_t dims[3] = {(cuuint64_t)a.row_bytes, (cuuint64_t)a.N, (cuuint64_t)n_groups};
    cuuint64_t str[2] = {(cuuint64_t)a.row_bytes, (cuuint64_t)a.group_bytes};
    cuuint32_t box[3] = {(cuuint32_t)SB, QBM, 1};
    int rc = make_map_u8(&mw, a.w, 3, dims, str, box);
    if (rc) return rc;
    if (DUAL) { rc = make_map_u8(&mw2, a.w2, 3, dims, str, box); if (rc) return rc; }
  }
  static PerDevice limit;
  if (limit.due()) {
    cudaFuncSetAttribute(qgemm_kernel<T, DUAL, BN, FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    limit.mark();
  }
  return (int)launch(qgemm_kernel<T, DUAL, BN, FORM>, dim3(grid), dim3(QTHREADS), smem, st, mx, mw, mw2, a);
}

template <class T, bool DUAL>
static int qgemm_pick(int form, int bn, const CUtensorMap& mx, const QGemmArgs& a, int n_groups, int grid, cudaStream_t st) {
  constexpr int kShort = !FastUnit<T>::kHas && ChunkUnit<T>::kOneForm ? Q_EXACT : Q_SHORT;   // types without a short form
  if (form == Q_SPLIT) {
    if (bn == 32) return qgemm_go<T, DUAL, 32, Q_SPLIT>(mx, a, n_groups, grid, st);
    if constexpr (!DUAL) { if (bn == 64) return qgemm_go<T, false, 64, Q_SPLIT>(mx, a, n_groups, grid, st); }
    return BL_ERR_SHAPE;
  }
  const bool exact = form == Q_EXACT;
  if (bn == 128) return qgemm_go<T, DUAL, 128, Q_EXACT>(mx, a, n_groups, grid, st);
  if (bn == 64) return exact ? qgemm_go<T, DUAL, 64, Q_EXACT>(mx, a, n_groups, grid, st) : qgemm_go<T, DUAL, 64, kShort>(mx, a, n_groups, grid, st);
  if (bn == 32) return exact ? qgemm_go<T, DUAL, 32, Q_EXACT>(mx, a, n_groups, grid, st) : qgemm_go<T, DUAL, 32, kShort>(mx, a, n_groups, grid, st);
  return BL_ERR_SHAPE;
}
template <class T>
static int qgemm_pick(bool dual, int form, int bn, const CUtensorMap& mx, const QGemmArgs& a, int n_groups, int grid, cudaStream_t st) {
  return dual ? qgemm_pick<T, true>(form, bn, mx, a, n_groups, grid, st) : qgemm_pick<T, false>(form, bn, mx, a, n_groups, grid, st);
}

}  // namespace bl

using namespace bl;

extern "C" {

// 1 when bl_qgemm has a kernel for this weight type
int bl_qgemm_supports(int wtype) {
  return wtype == WT_Q4_K || wtype == WT_Q5_K || wtype == WT_Q6_K || wtype == WT_Q8_0 || wtype == WT_FP8_B128 || wtype == WT_NVFP4 ||
         wtype == WT_Q8_F32;
}

// C[dst_row[t] or t, n] = row_scale[t] * sum_k X[t, k] W[g][n, k] (+ resid), per token tile of the table.
//   X [rows_x, K] bf16 (ldx elements); W, W2 [n_groups, N, row_bytes] resident blocks of type wtype;
//   tiles: {group, row0, row_end, -} token tiles of at most tile_rows (32, 64 or 128) rows; exactly one of c_f32 / c_bf16;
//   W2 != null: output = silu(X W^T) * (X W2^T).  status: device word, set to 1 when a wait ran out.
//   form: 0 short (exact at 128-row tiles), 1 exact, 2 split (tiles of 32 rows, and of 64 with one matrix); see the
//   expanders above.
//   fixed_tiles: the table has exactly max_tiles tiles, and no launch in flight writes the table, W or W2: the warps that
//   stream and expand weights read all three without waiting for the launch in front of this one.  splits > 1 (fixed tiles, one
//   matrix, K / 256 divisible): that many CTAs share a tile's depth; partial: max_tiles * ceil(N / 128) * splits *
//   tile_rows * 128 floats, tickets: max_tiles * ceil(N / 128) zeroed words, both of one stream at a time.
int bl_qgemm_split(const void* X, long ldx, long rows_x, const void* W, const void* W2, int wtype, int n_groups, int N, int K,
             const void* tiles, const int* n_tiles, int max_tiles, int tile_rows, float* c_f32, void* c_bf16, long ldc,
             const int* dst_row, const float* row_scale, const float* resid, long ldr, unsigned* status, int sm_count,
             int fixed_tiles, int form, int splits, float* partial, int* tickets, cudaStream_t st) {
  BL_REQUIRE(K >= 256 && K % 256 == 0 && N >= 1 && rows_x >= 1 && n_groups >= 1 && max_tiles >= 1, BL_ERR_SHAPE);
  BL_REQUIRE(tile_rows == 32 || tile_rows == 64 || tile_rows == 128, BL_ERR_SHAPE);
  BL_REQUIRE(ldx % 8 == 0 && ((uintptr_t)X & 15) == 0 && ((uintptr_t)W & 15) == 0 && ((uintptr_t)W2 & 15) == 0, BL_ERR_ALIGN);
  BL_REQUIRE((c_f32 != nullptr) != (c_bf16 != nullptr) && ldc < 1L << 30 && ldr < 1L << 30, BL_ERR_SHAPE);
  BL_REQUIRE(form >= Q_SHORT && form <= Q_SPLIT && (form != Q_SPLIT || tile_rows <= (W2 ? 32 : 64)), BL_ERR_SHAPE);
  BL_REQUIRE(splits == 1 || (splits > 1 && fixed_tiles && !W2 && partial && tickets && (K / 256) % splits == 0), BL_ERR_SHAPE);
  const long rb = resident_row_bytes(wtype, K);
  BL_REQUIRE(rb > 0 && bl_qgemm_supports(wtype), BL_ERR_TYPE);
  CUtensorMap mx;
  {
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows_x};
    cuuint64_t str[1] = {(cuuint64_t)ldx * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)tile_rows};
    int rc = make_map(&mx, X, 2, dims, str, box);
    if (rc) return rc;
  }
  QGemmArgs a{};
  a.w = (const uint8_t*)W; a.w2 = (const uint8_t*)W2;
  a.row_bytes = rb; a.group_bytes = rb * N;
  a.N = N; a.K = K; a.tiles_w = (N + QBM - 1) / QBM;
  a.tiles = (const QTile*)tiles; a.n_tiles = n_tiles; a.max_tiles = max_tiles;
  a.c_f32 = c_f32; a.c_bf16 = (__nv_bfloat16*)c_bf16; a.ldc = ldc;
  a.dst_row = dst_row; a.row_scale = row_scale; a.resid = resid; a.ldr = ldr; a.status = status;
  a.fixed_tiles = fixed_tiles; a.splits = splits; a.partial = partial; a.tickets = tickets;
  const long tiles_total = (long)max_tiles * a.tiles_w * splits;
  const int grid = (int)(splits > 1 || tiles_total < sm_count ? tiles_total : sm_count);   // a share has a CTA of its own
  const bool dual = W2 != nullptr;
  switch (wtype) {
    case WT_Q4_K: return qgemm_pick<Q4K>(dual, form, tile_rows, mx, a, n_groups, grid, st);
    case WT_Q5_K: return qgemm_pick<Q5K>(dual, form, tile_rows, mx, a, n_groups, grid, st);
    case WT_Q6_K: return qgemm_pick<Q6K>(dual, form, tile_rows, mx, a, n_groups, grid, st);
    case WT_Q8_0: return qgemm_pick<Q80>(dual, form, tile_rows, mx, a, n_groups, grid, st);
    case WT_FP8_B128: return qgemm_pick<Fp8B128>(dual, form, tile_rows, mx, a, n_groups, grid, st);
    case WT_NVFP4: return qgemm_pick<NvFp4>(dual, form, tile_rows, mx, a, n_groups, grid, st);
    case WT_Q8_F32: return qgemm_pick<Q8F>(dual, form, tile_rows, mx, a, n_groups, grid, st);
  }
  return BL_ERR_TYPE;
}

int bl_qgemm(const void* X, long ldx, long rows_x, const void* W, const void* W2, int wtype, int n_groups, int N, int K,
             const void* tiles, const int* n_tiles, int max_tiles, int tile_rows, float* c_f32, void* c_bf16, long ldc,
             const int* dst_row, const float* row_scale, const float* resid, long ldr, unsigned* status, int sm_count,
             cudaStream_t st) {
  return bl_qgemm_split(X, ldx, rows_x, W, W2, wtype, n_groups, N, K, tiles, n_tiles, max_tiles, tile_rows, c_f32, c_bf16, ldc,
                        dst_row, row_scale, resid, ldr, status, sm_count, 0, 0, 1, nullptr, nullptr, st);
}

}  // extern "C"
