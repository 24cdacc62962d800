// Decode GEMV for block-scaled activations: D[m x n] = A[m x k] (NVFP4) * B[n x k]^T with 1 <= n <= 8 and B either INT8 with one
// FP32 scale per 16 values (W4A8), NVFP4 (W4A4), or dense values that the kernel itself makes INT8 (nvfp4a_b200_gemv_w4a8: the bytes of quantizing first).  Per output
// and 16-block the kernel forms the EXACT sum of a * b, then acc = fma(p * sa, sb, acc) in FP32 -- the arithmetic of the reference's blocked GEMV
// (src/gemv_nvfp4effma.cuh:26-234 there); the order of the FP32 additions over k is this kernel's own, so results agree
// with the exact definition within the FP32 accumulation bound.
//
// Weights come as in gemv_stream.cu: sixteen warps, units of 16 rows x 128 values into registers, two ahead, nibbles to FP16 by hardware conversions.  The
// activations (integers up to 128, or E2M1 values, times 2^8) are FP16 values too, and a block's sum of 16 products is a multiple of 2^6 below 2^22, which
// mma.sync.m16n8k16 accumulates in FP32 without rounding.  So that every block keeps a sum of its own, the MMA's columns are (quad lane, vector) pairs: column 2 l + j
// holds vector j's values in the k positions of lane l's block and zeros elsewhere; four MMAs give lane l the sums of ITS block for two vectors.
// The order of a row's additions depends on k alone: its bits depend neither on the matrix around it nor on the other vectors.
//
// What bounds it: instruction issue and the chains between instructions (14336 x 4096, four vectors made INT8 here: 322 instructions per unit with all set-up, 57 % of the issue slots; per
// instruction warps wait 2.5 cycles for their own arithmetic, 0.8 for shared memory, 0.4 for weights).  CUDA graph, INT8 vectors given, int8 MMAs on weights decoded by byte permutes (11 instructions per 8 weights, 7
// here) with one unit ahead and then: 14336 x 4096 with 1 / 4 / 8 vectors 15.8 / 19.8 / 27.6 and 13.6 / 16.5 / 25.8 us, 4096 x 4096 7.5 / 8.6 / 11.2 and 6.1 / 7.4 / 10.3,
// 4096 x 14336 15.2 / 18.7 / 26.8 and 14.0 / 16.6 / 24.5, 1024 x 1024 2.9 / 3.1 / 3.6 and 3.1 / 3.3 / 4.0.  Dense BF16 vectors, quantized by a launch of their own and
// then here: 14336 x 4096 18.0 / 21.7 / 29.1 and 14.2 / 17.5 / 27.4, 1024 x 1024 4.4 / 4.5 / 5.7 and 3.6 / 3.8 / 4.8.
//
// A long k (more than kXLimit bytes for eight vectors): a cluster of 2, 4 or 8 CTAs takes a section of k each; the sections' sums go to the first CTA (DSMEM), which adds
// them in order.
#include <atomic>
#include "gemv_stream.cuh"

namespace nvb {

namespace {

constexpr int kMaxN = 8, kWarps = 16, kThreads = 32 * kWarps;
constexpr int kAhead = 2;                        // units of a warp in flight
constexpr int kSmemMax = 226 * 1024;
constexpr int kChunkBytes = 512 + 64;            // a vector's chunk of 256 values: FP16, and 16 block scales
constexpr int kXLimit = 150 * 1024;              // eight vectors' share of a section

struct GemvQArgs {
  int m, n, k;
  Fp4Operand A;
  BOperand B;                      // INT8 / NVFP4, or dense: quantized here
  Epilogue e;
  EpilogueEx ex;
  int sections, sec_chunks;        // CTAs per cluster, chunks of a section
  int kgroups;                     // warps that share a slice's k (the others take other slices)
  int per;                         // slices per cluster
  int round;                       // slices whose sums fit shared memory
};

// Activations are 2^8 times themselves in their operand (at most 2^15: exact), because the weights' scales come as 2^-8 of themselves (scale_pair): a block's sum times its scale
// is then the true one.  Sums kept 2^-8 as large were FP32 subnormals eight powers of two early; the factor on the scales instead costs a unit two multiplies (a call of
// 14336 x 4096 with four vectors 17.79 us, 17.66 so).
constexpr uint32_t kXScale = 0x5C005C00u;   // (2^8, 2^8)
__device__ __forceinline__ float ue5m3_low(uint32_t c) { return __fmul_rn(__uint_as_float(c << 20), 0x1p104f); }   // ue5m3_to_f32 times 2^-8

__device__ __forceinline__ uint32_t pack_h2(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}
// four int8 values -> two pairs of FP16, times 2^8: 0x64xx is 1024 + xx, and xx = value + 128
__device__ __forceinline__ void int8_to_f16(uint32_t w, uint32_t &o0, uint32_t &o1) {
  const uint32_t t = w ^ 0x80808080u;
  asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(o0) : "r"(byte_perm(t, 0x64646464u, 0x4140u)), "r"(0x64806480u));
  asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(o1) : "r"(byte_perm(t, 0x64646464u, 0x4342u)), "r"(0x64806480u));
  o0 = h2mul(o0, kXScale); o1 = h2mul(o1, kXScale);
}
// A block's 16 values -> 2^8 times its INT8 values (as floats) in the arithmetic of quant_int8_kernel (quant.cu), which says why; returns the scale.
__device__ __forceinline__ float int8_block(float (&v)[16]) {
  uint32_t top = 0;
#pragma unroll
  for (int i = 0; i < 16; ++i) top = max(top, __float_as_uint(v[i]) & 0x7FFFFFFFu);
  float bmax = __uint_as_float(top);
  if (top > 0x7F800000u) {
    bmax = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) bmax = fmaxf(bmax, fabsf(v[i]));
  }
  const float sb = __fdiv_rn(bmax, 127.f);
  if (top >= 0x20000000u && top < 0x60000000u) {
    const float inv = __frcp_rn(sb);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float x = v[i], y = __fmul_rn(x, inv);
      v[i] = __fmaf_rn(__fadd_rn(__fmaf_rn(__fmaf_rn(-y, sb, x), inv, y), 12582912.f), 256.f, -256.f * 12582912.f);   // (exact)
    }
  } else {
#pragma unroll 1
    for (int i = 0; i < 16; ++i) {
      const float q = sb > 0.f ? fminf(fmaxf(rintf(__fdiv_rn(v[0], sb)), -127.f), 127.f) : 0.f;
#pragma unroll
      for (int e = 0; e < 15; ++e) v[e] = v[e + 1];
      v[15] = 256.f * q;
    }
  }
  return sb;
}

// a load that lanes without `on` skip: their registers stay as they are
__device__ __forceinline__ void lds16_if(bool on, uint32_t a, uint32_t *r) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %5, 0;\n\t@p ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]) : "r"(a), "r"((uint32_t)on));
}
// pairs of FP32 values in one instruction; each is rounded by itself
__device__ __forceinline__ uint64_t pair_of(float lo, float hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// P: pairs of vectors.  IMG: A is an image.
template <int P, bool IMG>
__global__ void __launch_bounds__(kThreads, 1) gemv_q8_kernel(const GemvQArgs g) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ float colscale[2 * P];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, q = lane & 3;
  const int gm = g.m, gk = g.k, n = g.n;
  sm100::pdl_launch_dependents();
  const int S = g.sections, rank = S > 1 ? (int)sm100::cluster_ctarank() : 0, cluster = blockIdx.x / S;
  const int KG = g.kgroups, SG = kWarps / KG, kg = warp & (KG - 1), sg = warp / KG;
  const int sec = g.sec_chunks, c_first = rank * sec, kloc = max(min(gk - c_first * 256, sec * 256), 0);   // values of this CTA's range of k
  const int nloc = (kloc + 255) >> 8, units = (kloc + kStreamUnitK - 1) / kStreamUnitK;
  const int s_first = cluster * g.per, s_count = min(g.per, ((gm + 15) >> 4) - s_first);
  uint8_t *const xs = smem;                                      // FP16 activations [chunk][8][n][4 lanes][8 values]
  const int chunk_x = 512 * n, nb = sec * 16;
  uint8_t *const zeros = xs + (size_t)sec * chunk_x;             // half a chunk of zeros (one pair)
  float *const sx = (float *)(zeros + 256 * n);                  // [16 sec][2 P] block scales
  float *const part = sx + 2 * P * nb;                               // [slice of a round][KG warps][n][16 rows]
  float *const res = part + g.round * KG * n * 16;               // [section][slice of a round][n][16 rows] (first CTA of a cluster)

  UnitStream<IMG> f(g.A, gm, s_first, s_count, c_first, kloc, KG, warp, kWarps, lane);
  f.prefetch(kAhead);
  if (S > 1) sm100::cluster_arrive_release();
  sm100::pdl_wait();
  f.start_behind_wait();
  WeightUnit ahead[kAhead];
#pragma unroll
  for (int i = 0; i < kAhead; ++i) ahead[i] = f.fetch();

  // ---- the activations: a thread per block of 16 values ----
  const int dtype = g.B.dtype, blocks = kloc >> 4;
  const uint8_t *const xb = (const uint8_t *)behind_wait(g.B.data);
  const float *const s8 = behind_wait(g.B.s8);
  Fp4Operand xq = g.B.q;
  xq.data = behind_wait(xq.data); xq.sc = behind_wait(xq.sc);
  if (P == 1)
    for (int i = tid; i < 16 * n; i += kThreads) ((uint4 *)zeros)[i] = make_uint4(0, 0, 0, 0);
  // block b of vector j: two operands of eight values for the MMAs, and the scale
  auto put_block = [&](int j, int b, const uint32_t (&o)[8], float scale) {
    // value k = 128 h + 32 q + 8 i of a chunk: lane q's operand of the MMAs of word i, half h
    const int r = (2 * b) & 31;
    uint8_t *const d = xs + (size_t)(b >> 4) * chunk_x + ((((r >> 4) * 4 + (r & 3)) * n + j) * 4 + ((r >> 2) & 3)) * 16;
    *(uint4 *)d = make_uint4(o[0], o[1], o[2], o[3]);
    *(uint4 *)(d + 64 * n) = make_uint4(o[4], o[5], o[6], o[7]);
    sx[b * (2 * P) + j] = scale;
  };
  const int padded = nloc * 16, total = n * padded;              // (blocks past the end of k are zeros)
  if (dtype == NVFP4A_INT8) {
#pragma unroll 4
    for (int t = tid; t < total; t += kThreads) {
      const int j = t / padded, b = t - j * padded;
      uint4 w = make_uint4(0, 0, 0, 0);
      float scale = 0.f;
      if (b < blocks) {
        w = ld16((const uint4 *)(xb + (size_t)j * g.B.ld + 16 * (size_t)(c_first * 16 + b)));
        scale = s8[(size_t)j * g.B.lds8 + c_first * 16 + b];
      }
      uint32_t o[8];
      int8_to_f16(w.x, o[0], o[1]); int8_to_f16(w.y, o[2], o[3]); int8_to_f16(w.z, o[4], o[5]); int8_to_f16(w.w, o[6], o[7]);
      put_block(j, b, o, scale);
    }
  } else if (dtype == NVFP4A_NVFP4) {
#pragma unroll 1
    for (int t = tid; t < total; t += kThreads) {
      const int j = t / padded, b = t - j * padded;
      const uint2 w = b < blocks ? xq.block(j, c_first * 16 + b) : make_uint2(0, 0);
      uint32_t lo[4], hi[4];
      e2m1_to_f16(w.x, lo);
      e2m1_to_f16(w.y, hi);
      uint32_t o[8] = {lo[0], lo[1], lo[2], lo[3], hi[0], hi[1], hi[2], hi[3]};
#pragma unroll
      for (int i = 0; i < 8; ++i) o[i] = h2mul(o[i], kXScale);
      put_block(j, b, o, b < blocks ? xq.scale(j, c_first * 16 + b) : 0.f);
    }
  } else {
    const int esz = dtype == NVFP4A_FP32 ? 4 : 2;
    constexpr int kBatch = 2;
#pragma unroll 1
    for (int t0 = tid; t0 < total; t0 += kBatch * kThreads) {
      uint4 raw[kBatch][4];
#pragma unroll
      for (int h = 0; h < kBatch; ++h) {
        const int t = t0 + h * kThreads, j = t / padded, b = t - j * padded;
        const bool live = t < total && b < blocks;
        const uint4 *src = (const uint4 *)(xb + ((size_t)j * g.B.ld + 16 * (size_t)(c_first * 16 + b)) * esz);
#pragma unroll
        for (int i = 0; i < 4; ++i) raw[h][i] = live && (i < 2 || esz == 4) ? ld16(src + i) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int h = 0; h < kBatch; ++h) {
        const int t = t0 + h * kThreads, j = t / padded, b = t - j * padded;
        if (t >= total) break;
        const uint32_t ws[16] = {raw[h][0].x, raw[h][0].y, raw[h][0].z, raw[h][0].w, raw[h][1].x, raw[h][1].y, raw[h][1].z, raw[h][1].w,
                                 raw[h][2].x, raw[h][2].y, raw[h][2].z, raw[h][2].w, raw[h][3].x, raw[h][3].y, raw[h][3].z, raw[h][3].w};
        float v[16];
        if (dtype == NVFP4A_BF16) {
#pragma unroll
          for (int i = 0; i < 8; ++i) { v[2 * i] = __uint_as_float(ws[i] << 16); v[2 * i + 1] = __uint_as_float(ws[i] & 0xFFFF0000u); }
        } else if (dtype == NVFP4A_FP16) {
#pragma unroll
          for (int i = 0; i < 8; ++i) { const float2 f2 = __half22float2(*(const __half2 *)&ws[i]); v[2 * i] = f2.x; v[2 * i + 1] = f2.y; }
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(ws[i]);
        }
        const float scale = int8_block(v);
        uint32_t o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = pack_h2(v[2 * i], v[2 * i + 1]);
        put_block(j, b, o, scale);
      }
    }
  }
  if (2 * P > n)                 // scales of the vectors that fill up the last pairs
    for (int t = tid; t < padded; t += kThreads)
#pragma unroll
      for (int j = 0; j < 2 * P; ++j)
        if (j >= n) sx[t * (2 * P) + j] = 0.f;
  if (g.ex.mask & kExNorm)
    for (int j = warp; j < n; j += kWarps) {
      const float s = warp_norm_scale(g.ex, j, lane);
      if (lane == 0) colscale[j] = s;
    }
  const float ga0 = g.e.ga && !g.e.ga_stride ? g.e.ga[0] : 1.f;
  __syncthreads();

  const Epilogue &e = g.e;
  float amax = 0.f;
  int slice = sg, u = kg;        // the unit at hand
  uint64_t acc[2][P];            // [row][two vectors] of the lane's blocks, FP32 pairs
#pragma unroll
  for (int p = 0; p < P; ++p) acc[0][p] = acc[1][p] = 0;
  // A lane whose column is not its own block's has zeros for an operand.  One pair of vectors: it loads them from shared memory; several: its registers hold zeros
  // that no load ever touches, because the loads would cost four wavefronts each (14336 x 4096 with 8 / 4 / 2 vectors 25.9 / 16.6 / 13.6 us so, 30.3 / 18.3 / 13.0
  // with loaded zeros).  A last vector without a partner: its lanes read what follows it, for a column nobody looks at.
  const bool diag = (gq >> 1) == q, ue = g.A.ue != 0;
  const int nx = 64 * n;
  constexpr bool kLoadZeros = P == 1;
  const uint32_t xa0 = kLoadZeros && !diag ? sm100::smem_u32(zeros) : sm100::smem_u32(xs) + ((gq & 1) * 4 + q) * 16, xa_step = kLoadZeros && !diag ? 0 : 4 * nx;
  uint32_t xr[2][8];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) xr[i][j] = 0;
  const float *const sx0 = sx + 2 * q * (2 * P);
  auto compute = [&](const WeightUnit &w) {
    const uint32_t xa = xa0 + u * xa_step;
    const float *const su = sx0 + 8 * u * (2 * P);
    float fa[2], fb[2];          // the scales of the lane's blocks, rows gq and gq + 8, times 2^-8
    if (!ue) {
      const uint32_t sa = scale_pair(w.ca), sb = scale_pair(w.cb);
      const float2 a = __half22float2(*(const __half2 *)&sa), b = __half22float2(*(const __half2 *)&sb);
      fa[0] = a.x; fa[1] = a.y; fb[0] = b.x; fb[1] = b.y;
    } else {
      fa[0] = ue5m3_low(w.ca & 0xFFu); fa[1] = ue5m3_low(w.ca >> 8); fb[0] = ue5m3_low(w.cb & 0xFFu); fb[1] = ue5m3_low(w.cb >> 8);
    }
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      uint32_t p[2][4], r[2][4];
      const uint64_t sa2 = pair_of(fa[b], fa[b]), sb2 = pair_of(fb[b], fb[b]);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        e2m1_to_f16(word(w.wa, 2 * b + i), p[i]);
        e2m1_to_f16(word(w.wb, 2 * b + i), r[i]);
      }
#pragma unroll
      for (int pr = 0; pr < P; ++pr) {
        if (P > 1 && 2 * pr >= n) break;
        float d[4];
        uint32_t (&x)[8] = xr[pr & 1];
        if constexpr (kLoadZeros) {
          const uint4 lo = lds16(xa + (2 * b) * nx), hi = lds16(xa + (2 * b + 1) * nx);
          x[0] = lo.x; x[1] = lo.y; x[2] = lo.z; x[3] = lo.w; x[4] = hi.x; x[5] = hi.y; x[6] = hi.z; x[7] = hi.w;
        } else {
          lds16_if(diag, xa + (2 * b) * nx + pr * 128, x);
          lds16_if(diag, xa + (2 * b + 1) * nx + pr * 128, x + 4);
        }
        mma16_first(d, p[0][0], r[0][0], p[0][1], r[0][1], x[0], x[1]);
        mma16(d, p[0][2], r[0][2], p[0][3], r[0][3], x[2], x[3]);
        mma16(d, p[1][0], r[1][0], p[1][1], r[1][1], x[4], x[5]);
        mma16(d, p[1][2], r[1][2], p[1][3], r[1][3], x[6], x[7]);
        const float2 xv = *(const float2 *)(su + b * (2 * P) + 2 * pr);
        acc[0][pr] = fma_f32x2(mul_f32x2(pair_of(d[0], d[1]), sa2), pair_of(xv.x, xv.y), acc[0][pr]);
        acc[1][pr] = fma_f32x2(mul_f32x2(pair_of(d[2], d[3]), sb2), pair_of(xv.x, xv.y), acc[1][pr]);
      }
    }
  };
  // the warp's sums of a slice -> part
  auto put = [&](int at) {
    float *const p = part + (size_t)(at * KG + kg) * n * 16;
    // The four lanes of a quad add their 4 P values; a lane ends up with P of them: those of row gq + 8 (q & 1) and of the first or second of each pair of vectors.
#pragma unroll
    for (int pr = 0; pr < P; ++pr) {
      if (P > 1 && 2 * pr >= n) break;
      const uint64_t keep = q & 1 ? acc[1][pr] : acc[0][pr], give = q & 1 ? acc[0][pr] : acc[1][pr];
      const float k0 = __uint_as_float((uint32_t)keep), k1 = __uint_as_float((uint32_t)(keep >> 32));
      const float t0 = __fadd_rn(k0, __shfl_xor_sync(0xFFFFFFFFu, __uint_as_float((uint32_t)give), 1));
      const float t1 = __fadd_rn(k1, __shfl_xor_sync(0xFFFFFFFFu, __uint_as_float((uint32_t)(give >> 32)), 1));
      const float t = __fadd_rn(q & 2 ? t1 : t0, __shfl_xor_sync(0xFFFFFFFFu, q & 2 ? t0 : t1, 2));
      const int j = 2 * pr + (q >> 1);
      if (j < n) p[j * 16 + gq + 8 * (q & 1)] = t;
    }
#pragma unroll
    for (int p2 = 0; p2 < P; ++p2) acc[0][p2] = acc[1][p2] = 0;
  };
  // a CTA's sum over its range of k: the warps', pairwise
  auto own_sum = [&](int o) {
    const int sl = (o >> 4) / n, in = o - sl * n * 16;
    const float *const t0 = part + (size_t)sl * KG * n * 16 + in;
    float t[kWarps];
#pragma unroll
    for (int w = 0; w < kWarps; ++w) t[w] = w < KG ? t0[w * n * 16] : 0.f;
#pragma unroll
    for (int step = kWarps / 2; step; step >>= 1)
#pragma unroll
      for (int w = 0; w < step; ++w) t[w] = __fadd_rn(t[2 * w], t[2 * w + 1]);
    return t[0];
  };

#pragma unroll 1
  for (int base = 0; base < s_count; base += g.round) {     // (one round unless a CTA has so many slices that their sums do not fit shared memory)
    const int end = min(base + g.round, s_count);
    if (kg < units) {
      if (base > 0 && slice < s_count) {
        f.restart(slice);
#pragma unroll
        for (int i = 0; i < kAhead; ++i) ahead[i] = f.fetch();
      }
#pragma unroll 1
      while (slice < end) {
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
          if (slice >= end) break;
          const WeightUnit w = ahead[i];
          ahead[i] = f.fetch();
          compute(w);
          u += KG;
          if (u >= units) { put(slice - base); u = kg; slice += SG; }
        }
      }
    } else {
      for (int s = sg; s < end - base; s += SG) put(s);     // zeros
    }
    __syncthreads();
    const int outs = (end - base) * n * 16;
    auto epilogue = [&](auto sum_of) { slices_epilogue(e, g.ex, n, s_first + base, outs, gm, ga0, colscale, amax, sum_of); };
    if (S == 1) {
      epilogue(own_sum);
      if (end < s_count) __syncthreads();
    } else {
      sm100::cluster_wait_acquire();                        // every CTA runs, and the first has read the round before
      for (int o = tid; o < outs; o += kThreads) sm100::st_peer_f32(res + (size_t)rank * g.round * n * 16 + o, 0, own_sum(o));
      __syncwarp();
      sm100::cluster_arrive_release();
      sm100::cluster_wait_acquire();
      if (rank == 0)
        epilogue([&](int o) {
          float s = res[o];
          for (int r = 1; r < S; ++r) s = __fadd_rn(s, res[(size_t)r * g.round * n * 16 + o]);
          return s;
        });
      if (end < s_count) sm100::cluster_arrive_release();
    }
  }
  if (rank == 0 && e.amax) warp_amax_commit(e.amax, amax);
}

// sections of k: by k alone
int sections_for(int k) {
  const int chunks = (k + 255) >> 8;
  for (int s = 1; s <= 8; s *= 2)
    if (s == 8 || kMaxN * ((chunks + s - 1) / s) * kChunkBytes <= kXLimit) return s;
  return 8;
}
int pairs_of(int n) { return n <= 2 ? 1 : n <= 4 ? 2 : 4; }
int fixed_bytes(int n, int sec_chunks) { return n * (sec_chunks * 512 + 256) + 2 * pairs_of(n) * sec_chunks * 64; }

}  // namespace

bool gemv_q8_supports(const GemmArgs &g) {
  if (!(g.n >= 1 && g.n <= kMaxN && g.k >= 64)) return false;
  const int chunks = (g.k + 255) >> 8, sec = (chunks + sections_for(g.k) - 1) / sections_for(g.k);
  if (sec > kSmemMax / kChunkBytes || fixed_bytes(g.n, sec) > kSmemMax - 16 * 1024) return false;   // (16 KiB: the sums of a slice, at most)
  if (g.B.dtype == NVFP4A_NVFP4 && g.B.q.image) return false;
  if (g.B.dtype != NVFP4A_NVFP4 && (((uintptr_t)g.B.data & 15) || g.B.ld % 16)) return false;
  return g.A.image || (((uintptr_t)g.A.data & 15) == 0 && g.A.ld % 32 == 0 && ((uintptr_t)g.A.sc & 3) == 0 && g.A.sld % 4 == 0);
}

template <int P, bool IMG> static cudaError_t launch(const GemvQArgs &a, int clusters, int smem, cudaStream_t s) {
  static std::atomic<bool> attr_set[64];   // zero-initialised; set once per device (a repeated cudaFuncSetAttribute is harmless)
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set[dev & 63]) {
    if (cudaError_t e = cudaFuncSetAttribute(gemv_q8_kernel<P, IMG>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax)) return e;
    attr_set[dev & 63] = true;
  }
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof cfg);
  cfg.gridDim = dim3(clusters * a.sections, 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (a.sections > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = a.sections; attr[na].val.clusterDim.y = 1; attr[na].val.clusterDim.z = 1;
    ++na;
  }
  if (pdl_enabled()) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = attr; cfg.numAttrs = na;
  return cudaLaunchKernelEx(&cfg, gemv_q8_kernel<P, IMG>, a);
}
template <int P> static cudaError_t launch_pairs(const GemvQArgs &a, int clusters, int smem, cudaStream_t s) {
  return a.A.image ? launch<P, true>(a, clusters, smem, s) : launch<P, false>(a, clusters, smem, s);
}

cudaError_t launch_gemv_q8(const GemmArgs &g, cudaStream_t s) {
  GemvQArgs a;
  a.m = g.m; a.n = g.n; a.k = g.k;
  a.A = g.A; a.B = g.B; a.e = g.e; a.ex = g.x;
  const int chunks = (g.k + 255) >> 8;
  a.sections = sections_for(g.k);
  a.sec_chunks = (chunks + a.sections - 1) / a.sections;
  const int units = min(2 * a.sec_chunks, (g.k + kStreamUnitK - 1) / kStreamUnitK);
  a.kgroups = 1;
  while (a.kgroups < kWarps && a.kgroups * 2 <= units) a.kgroups *= 2;
  if (a.kgroups > 2 && (units + a.kgroups - 1) / a.kgroups * a.kgroups * 8 > units * 9) a.kgroups /= 2;   // (as in gemv_stream.cu)
  const int slices = (g.m + 15) / 16, most = device_sms() / a.sections;
  a.per = (slices + most - 1) / most;
  const int clusters = (slices + a.per - 1) / a.per;
  const int slice_bytes = (a.kgroups + (a.sections > 1 ? a.sections : 0)) * g.n * 64;
  const int fixed = fixed_bytes(g.n, a.sec_chunks);
  a.round = min(a.per, (kSmemMax - fixed) / slice_bytes);
  const int smem = fixed + a.round * slice_bytes;
  return g.n <= 2 ? launch_pairs<1>(a, clusters, smem, s) : g.n <= 4 ? launch_pairs<2>(a, clusters, smem, s) : launch_pairs<4>(a, clusters, smem, s);
}

}  // namespace nvb
