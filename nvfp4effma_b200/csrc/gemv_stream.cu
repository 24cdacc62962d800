// Decode GEMV for one and two BF16 activation vectors (W4A16), E4M3 block scales: D[m x n] = A[m x k] (NVFP4) * B[n x k]^T.  The FP4 tensor-core GEMV
// (gemv_fp4.cu) keeps the large matrices; gemv.cu has three to eight vectors and UE5M3 scales.
//
// Weights.  A CTA of sixteen warps per SM owns a run of 16-row slices; the warps deal a slice's k out in units of 16 rows x 128 values and
// load them straight into registers, the next two units in flight while one is computed, slice after slice without a barrier; the warps' sums meet in
// shared memory once, at the end.  Before the programmatic wait each warp asks for its first units' lines in L2.  (A prefetch into L2 reads
// nothing: a predecessor may still be writing the weights.)
//
// Arithmetic.  cvt.rn.f16x2.e2m1x2 turns a byte into two exact FP16 values (7 instructions per 8 weights; shifts and masks into BF16, as in gemv.cu, take 20
// with the scale) and mma.sync.m16n8k16 accumulates in FP32.  The MMA's columns are (quad lane, vector) pairs: column 2 l + j holds vector j's values in the
// k positions of lane l's block and zeros elsewhere, so that four MMAs give lane l the sum of ITS block and the block's scale applies to that sum.
// The activations become FP16 exactly: the largest magnitude of a vector's chunk of 256 values is brought into [2^14, 2^15) by a power of two,
// and a BF16 value no more than 2^31 below it has an FP16 value.  Values further down are left out there (plane 0) and added in planes of their own,
// each scaled up by another 2^32; a chunk without such values -- nearly every one -- pays nothing for them, a chunk with some one more MMA pass per plane.
// Inf and NaN stay what they are.  Relative error against 64 bits (2-norm, FP32 D, 4096 x 4096): 7.0e-8, 1.2e-7 where activations are products that spread
// far (gemv_kernel: 1.2e-7 and 5.5e-7).  The order of a row's additions depends on k and n alone: a row's bits do not depend on
// the matrix (or tensor-parallel shard) around it.
//
// What bounds it: launch and one memory round trip for the activations, then load latency and instruction issue
// (4096 x 14336: 187 instructions per unit with all set-up, 45 % of the issue slots; per instruction warps wait 3.2 cycles for memory and 1.6 for their own arithmetic).  CUDA graph, one vector, before (gemv_kernel) and now: 1024 x 1024 3.1 and 2.8 us, 512 x 4096 4.65 and 3.75, 4096 x 4096 6.9 and 5.6, 6144 x
// 4096 8.6 and 7.1, 4096 x 14336 17.4 and 13.2; two vectors 3.1 and 3.1, 4.7 and 4.4, 6.95 and 6.1, 9.0 and 7.6, 17.4 and 14.5.  Starting under the
// previous kernel's tail is 1.1 us of each.  Slower: units of 16 x 256 (registers spill), three units ahead (5.7 / 7.1 / 13.0), CTAs of eight warps two
// of which fit an SM (7.4 / 9.2 / 18.1), bulk copies into a ring of shared memory with a cluster of four per k (6.9 / 8.0 / 16.0).
// Three and more vectors as the MMA's columns, with the scales on the weights, gain nothing over gemv_kernel (eight: 8.7 against 7.6 at 4096 x
// 4096): converting the activations takes every CTA a microsecond there.
//
// A long k (more than 128 KiB of FP16 activations): a cluster of 2, 4 or 8 CTAs takes a section of k each; the sections' sums go to the first CTA (DSMEM),
// which adds them in order.
#include <atomic>
#include "gemv_stream.cuh"

namespace nvb {

namespace {

constexpr int kWarps = 16, kThreads = 32 * kWarps;
constexpr int kAhead = 2;                                         // units of a warp in flight
constexpr int kSmemMax = 226 * 1024;
constexpr int kXLimit = 128 * 1024;                                // activations of a CTA at most
constexpr unsigned kMinExp = 14;                                  // smallest biased exponent a vector is scaled by: 2^(141 - 14) is a float

struct StreamArgs {
  int m, n, k;
  Fp4Operand A;
  const uint16_t *x; int ldx;      // BF16 activations [n][ldx]
  Epilogue e;
  EpilogueEx ex;
  TpPush tp;
  int sections, sec_chunks;        // CTAs per cluster, chunks of a section
  int kgroups;                     // warps that share a slice's k (the others take other slices)
  int per;                         // slices per cluster
  int round;                       // slices whose sums fit shared memory
};

__device__ __forceinline__ float pow2i(int e) { return __int_as_float((e + 127) << 23); }   // -126 <= e <= 127
// v * 2^e for any e that a vector's scale can be, by two exact factors
__device__ __forceinline__ float scale2(float v, int e) {
  const int a = max(min(e, 100), -100);
  return __fmul_rn(__fmul_rn(v, pow2i(a)), pow2i(max(min(e - a, 127), -126)));
}
// eight BF16 values of plane p > 0 of a vector whose largest biased exponent is eb, as FP16 values scaled by 2^(141 - eb + 32 p); values of other planes are 0
__device__ __forceinline__ uint4 plane_values(const uint4 &v, int eb, int p) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  uint32_t o[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float f[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t b = h ? w[i] >> 16 : w[i] & 0xFFFFu;
      const int d = eb - max((int)((b >> 7) & 0xFFu), 1);
      int ex = 141 - eb + 32 * p;
      float t = (d >> 5) == p ? __uint_as_float(b << 16) : 0.f;
#pragma unroll
      for (int q = 0; q < 4; ++q) { const int s = max(min(ex, 120), -120); t = __fmul_rn(t, pow2i(s)); ex -= s; }
      f[h] = t;
    }
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(o[i]) : "f"(f[1]), "f"(f[0]));
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}

// N: vectors.  IMG: A is an image.
template <int N, bool IMG>
__global__ void __launch_bounds__(kThreads, 1) gemv_stream_kernel(const StreamArgs g) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ float colscale[N];
  __shared__ int any_more_s;          // some chunk has planes beyond the first
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, q = lane & 3;
  const int gm = g.m, gk = g.k, n = N;
  sm100::pdl_launch_dependents();
  const int S = g.sections, rank = S > 1 ? (int)sm100::cluster_ctarank() : 0, cluster = blockIdx.x / S;
  const int KG = g.kgroups, SG = kWarps / KG, kg = warp & (KG - 1), sg = warp / KG;
  const int sec = g.sec_chunks, c_first = rank * sec, kloc = max(min(gk - c_first * 256, sec * 256), 0);   // values of this CTA's range of k
  const int nloc = (kloc + 255) >> 8, units = (kloc + kStreamUnitK - 1) / kStreamUnitK;
  const int s_first = cluster * g.per, s_count = min(g.per, ((gm + 15) >> 4) - s_first);
  uint8_t *const xs = smem;                                                            // FP16 activations [chunk][8][n][4 lanes][8 values]
  const int chunk_x = 512 * n;
  uint8_t *const zeros = xs + (size_t)sec * chunk_x;                                   // a chunk of zeros
  float *const factor = (float *)(zeros + chunk_x);                                    // [chunk][n] what a unit of the sums is worth
  int *const more = (int *)(factor + sec * n);                                         // [chunk] planes beyond the first
  float *const part = (float *)(more + sec);                                           // [slice of a round][KG warps][n][16 rows]
  float *const res = part + g.round * KG * n * 16;                                     // [section][slice of a round][n][16 rows] (first CTA of a cluster)

  UnitStream<IMG> f(g.A, gm, s_first, s_count, c_first, kloc, KG, warp, kWarps, lane);
  f.prefetch(kAhead);
  if (S > 1) sm100::cluster_arrive_release();
  sm100::pdl_wait();
  f.start_behind_wait();
  WeightUnit ahead[kAhead];
#pragma unroll
  for (int i = 0; i < kAhead; ++i) ahead[i] = f.fetch();
  // tensor-parallel layers in the deferred form: the activations are complete once every peer has posted the previous gather (the weights are on their way)
  if (g.tp.world > 1 && (g.tp.deferred & 1)) tp_wait_posts(g.tp.flags, g.tp.world, g.tp.rank, g.tp.status, g.tp.tag, g.tp.wait_cycles);
  if (tid == 0) any_more_s = 0;
  for (int i = tid; i < sec; i += kThreads) more[i] = 0;
  for (int i = tid; i < chunk_x / 16; i += kThreads) ((uint4 *)zeros)[i] = make_uint4(0, 0, 0, 0);

  // ---- the activations: FP16 values, a chunk of a vector per warp and turn ----
  __syncthreads();
  const uint16_t *const x = behind_wait(g.x);
  const int kvec = (gk - c_first * 256) >> 3;            // vectors of eight values up to the end of k
  constexpr int kBatch = 4;
#pragma unroll 1
  for (int t0 = warp; t0 < n * nloc; t0 += kWarps * kBatch) {   // task t: vector t % n, chunk t / n
    uint4 b[kBatch];
    int cs[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int t = t0 + u * kWarps, c = t / N, v = c * 32 + lane;
      cs[u] = c;
      b[u] = t < n * nloc && v < kvec ? ld16((const uint4 *)(x + (size_t)(t - c * n) * g.ldx) + (size_t)c_first * 32 + v) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int t = t0 + u * kWarps, c = cs[u], j = t - c * n;
      if (t >= n * nloc) break;
      uint32_t w[4] = {b[u].x, b[u].y, b[u].z, b[u].w};
      uint32_t a = __vmaxu2(__vmaxu2(w[0] & 0x7FFF7FFFu, w[1] & 0x7FFF7FFFu), __vmaxu2(w[2] & 0x7FFF7FFFu, w[3] & 0x7FFF7FFFu));
      a = __reduce_max_sync(0xFFFFFFFFu, max(a & 0xFFFFu, a >> 16));
      const int eb = (int)max(min(a >> 7, 254u), kMinExp);               // the biased exponent this chunk of the vector is scaled by
      const float up = pow2i(141 - eb);
      const uint32_t least = eb <= 32 ? 1u : (uint32_t)(eb - 31) << 7;    // smallest magnitude of plane 0
      // (zeros count as the largest value here: 0 - 1 wraps)
      const uint32_t lo = __vminu2(__vminu2(__vsub2(w[0] & 0x7FFF7FFFu, 0x00010001u), __vsub2(w[1] & 0x7FFF7FFFu, 0x00010001u)),
                                   __vminu2(__vsub2(w[2] & 0x7FFF7FFFu, 0x00010001u), __vsub2(w[3] & 0x7FFF7FFFu, 0x00010001u)));
      int planes = 0;
      if (min(lo & 0xFFFFu, lo >> 16) < least - 1 && a < 0x7F80u) {       // some values belong to further planes
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint32_t mag = (w[i] >> (16 * h)) & 0x7FFFu;
            if (mag && mag < least) {
              planes = max(planes, (eb - max((int)(mag >> 7), 1)) >> 5);
              w[i] &= h ? 0x0000FFFFu : 0xFFFF0000u;
            }
          }
      }
      planes = __reduce_max_sync(0xFFFFFFFFu, planes);
      if (lane == 0) {
        factor[c * n + j] = pow2i(eb - 133);
        if (planes) { atomicMax(&more[c], planes); any_more_s = 1; }
      }
      uint32_t o[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(o[i]) : "f"(__fmul_rn(__uint_as_float(w[i] & 0xFFFF0000u), up)), "f"(__fmul_rn(__uint_as_float(w[i] << 16), up)));
      // value k = 128 h + 32 q + 8 i of a chunk: lane q's operand of the MMAs of word i, half h
      const int at = ((lane >> 4) * 4 + (lane & 3)) * n * 4 + j * 4 + ((lane >> 2) & 3);
      *(uint4 *)(xs + (size_t)c * chunk_x + at * 16) = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
  if (g.ex.mask & kExNorm)
    for (int j = warp; j < n; j += kWarps) {
      const float s = warp_norm_scale(g.ex, j, lane);
      if (lane == 0) colscale[j] = s;
    }
  const float ga0 = g.e.ga && !g.e.ga_stride ? g.e.ga[0] : 1.f;
  __syncthreads();

  const Epilogue &e = g.e;
  float amax = 0.f;
  const bool any_more = any_more_s != 0;
  int slice = sg, u = kg;        // the unit at hand
  float acc[4] = {0, 0, 0, 0};   // [2 row + vector] of the lane's blocks, true scale
  const bool diag = (gq >> 1) == q && (gq & 1) < N;
  const uint32_t xa0 = diag ? sm100::smem_u32(xs) + ((gq & 1) * 4 + q) * 16 : sm100::smem_u32(zeros), xa_step = diag ? 256 * N : 0;   // per 128 values of k
  auto compute = [&](const WeightUnit &w) {
    float sum[4] = {0, 0, 0, 0};   // of this unit
    const uint32_t xa = xa0 + u * xa_step;
    const uint32_t sa = scale_pair(w.ca), sb = scale_pair(w.cb);
#pragma unroll
    for (int b = 0; b < 2; ++b) {   // the lane's two blocks
      float d[4];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        uint32_t p[4], r[4];
        e2m1_to_f16(word(w.wa, 2 * b + i), p);
        e2m1_to_f16(word(w.wb, 2 * b + i), r);
        const uint4 xv = lds16(xa + (2 * b + i) * (64 * N));
        if (i == 0) mma16_first(d, p[0], r[0], p[1], r[1], xv.x, xv.y);
        else mma16(d, p[0], r[0], p[1], r[1], xv.x, xv.y);
        mma16(d, p[2], r[2], p[3], r[3], xv.z, xv.w);
      }
      const __half2 ha = *(const __half2 *)&sa, hb = *(const __half2 *)&sb;
      const float f0 = b ? __high2float(ha) : __low2float(ha), f1 = b ? __high2float(hb) : __low2float(hb);
#pragma unroll
      for (int j = 0; j < N; ++j) {
        sum[j] = __fmaf_rn(d[j], f0, sum[j]);
        sum[2 + j] = __fmaf_rn(d[2 + j], f1, sum[2 + j]);
      }
    }
    const int c = u >> 1;
    const float *const fc = factor + c * N;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      acc[j] = __fmaf_rn(sum[j], fc[j], acc[j]);
      acc[2 + j] = __fmaf_rn(sum[2 + j], fc[j], acc[2 + j]);
    }
    if (any_more && more[c]) {   // (the same for every lane) values that plane 0 could not hold
      const int planes = more[c], col = gq < N ? gq : 0, eb = (__float_as_int(fc[col]) >> 23) + 6;   // (the exponent of 2^(eb - 133), biased, is eb - 6)
      const uint4 *row = (const uint4 *)(x + (size_t)col * g.ldx) + (size_t)(c_first + c) * 32;
      const int vec_left = kvec - c * 32;
#pragma unroll 1
      for (int p = 1; p <= planes; ++p) {
        float d[4] = {0, 0, 0, 0};
#pragma unroll 1
        for (int i = 0; i < 4; ++i) {
          uint32_t pa[4], pb[4];
          const uint32_t sel = i & 2 ? 0x3232u : 0x1010u, s0 = byte_perm(sa, 0u, sel), s1 = byte_perm(sb, 0u, sel);
          e2m1_to_f16(word(w.wa, i), pa);
          e2m1_to_f16(word(w.wb, i), pb);
          const int v = (u & 1) * 16 + q * 4 + i;
          const uint4 xv = gq < N && v < vec_left ? plane_values(ld16(row + v), eb, p) : make_uint4(0, 0, 0, 0);
          mma16(d, h2mul(pa[0], s0), h2mul(pb[0], s1), h2mul(pa[1], s0), h2mul(pb[1], s1), xv.x, xv.y);
          mma16(d, h2mul(pa[2], s0), h2mul(pb[2], s1), h2mul(pa[3], s0), h2mul(pb[3], s1), xv.z, xv.w);
        }
        if (q == 0)       // columns 0 and 1 are the vectors here; lane 0 of a quad has them, and its sums join the others'
#pragma unroll
          for (int j = 0; j < N; ++j) {
            const int ex = (__float_as_int(fc[j]) >> 23) - 127 - 32 * p;
            acc[j] = __fadd_rn(acc[j], scale2(d[j], ex));
            acc[2 + j] = __fadd_rn(acc[2 + j], scale2(d[2 + j], ex));
          }
      }
      __syncwarp();
    }
  };
  // the warp's sums of a slice -> part
  auto put = [&](int at) {
    float *const p = part + (size_t)(at * KG + kg) * n * 16;
#pragma unroll
    for (int j = 0; j < N; ++j)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        float t = acc[2 * r + j];
        t = __fadd_rn(t, __shfl_xor_sync(0xFFFFFFFFu, t, 1));
        t = __fadd_rn(t, __shfl_xor_sync(0xFFFFFFFFu, t, 2));
        if (q == 0) p[j * 16 + gq + 8 * r] = t;
      }
    acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
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
  if (rank != 0) return;
  if (e.amax) warp_amax_commit(e.amax, amax);
  if (g.tp.world > 1 && (g.tp.deferred == 0 || (g.tp.deferred & 2))) {
    // All-gather fused into this kernel: the CTA that finishes last copies the rank's outputs (n rows of the activation
    // buffer, just written and still in L2) into every peer's buffer with 16-byte stores and joins the ranks' barrier.
    __shared__ int last_cta;
    __threadfence();
    __syncthreads();
    if (tid == 0) {
      unsigned *ctas = (unsigned *)(g.tp.flags[g.tp.rank] + kFlagCtas);
      const unsigned ticket = atomicAdd(ctas, 1u);
      last_cta = ticket == gridDim.x / S - 1;   // one ticket per cluster
      if (last_cta) *ctas = 0;
    }
    __syncthreads();
    if (last_cta) {
      __threadfence();
      const int esz = dense_bytes(e.d_dtype);
      const int drows = (g.ex.mask & kExSwiglu) ? gm / 2 : gm;
      const int vec_per_row = drows * esz / 16;
      for (int v = tid; v < vec_per_row * n; v += blockDim.x) {
        const int j = v / vec_per_row, c = v - j * vec_per_row;
        uint8_t *src = (uint8_t *)e.d + ((size_t)j * e.ldd * esz + (size_t)c * 16);
        const uint4 y = __ldcg((const uint4 *)src);
        for (int p = 0; p < g.tp.world; ++p)
          if (p != g.tp.rank) *(uint4 *)(src + g.tp.delta[p]) = y;
      }
      __syncthreads();   // the flags' release stores order every thread's copies (see tp_barrier_cta)
      // deferred form: tell the peers and leave; the next kernel of every rank waits for the posts at its start
      if (g.tp.deferred & 2) tp_post_epoch(g.tp.flags, g.tp.world, g.tp.rank);
      else tp_barrier_cta(g.tp.flags, g.tp.world, g.tp.rank, g.tp.status, g.tp.tag, g.tp.wait_cycles);
    }
  }
}

// sections of k: by k and n alone
int sections_for(int k, int n) {
  const int chunks = (k + 255) >> 8;
  for (int s = 1; s <= 8; s *= 2)
    if (s <= chunks && n * ((chunks + s - 1) / s) * 512 <= kXLimit) return s;
  return 0;
}

}  // namespace

bool gemv_stream_supports(const GemmArgs &g) {
  return g.n >= 1 && g.n <= 2 && g.B.dtype == NVFP4A_BF16 && g.k > 0 && !g.A.ue && ((uintptr_t)g.B.data & 15) == 0 && g.B.ld % 8 == 0 &&
         (g.A.image || (((uintptr_t)g.A.data & 15) == 0 && g.A.ld % 32 == 0 && ((uintptr_t)g.A.sc & 3) == 0 && g.A.sld % 4 == 0)) && sections_for(g.k, g.n) > 0;
}

template <int N, bool IMG> static cudaError_t launch(const StreamArgs &a, int clusters, int smem, cudaStream_t s) {
  static std::atomic<bool> attr_set[64];   // zero-initialised; set once per device (a repeated cudaFuncSetAttribute is harmless)
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set[dev & 63]) {
    if (cudaError_t e = cudaFuncSetAttribute(gemv_stream_kernel<N, IMG>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax)) return e;
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
  return cudaLaunchKernelEx(&cfg, gemv_stream_kernel<N, IMG>, a);
}

cudaError_t launch_gemv_stream(const GemmArgs &g, cudaStream_t s) {
  StreamArgs a;
  a.m = g.m; a.n = g.n; a.k = g.k;
  a.A = g.A;
  a.x = (const uint16_t *)g.B.data; a.ldx = g.B.ld;
  a.e = g.e; a.ex = g.x; a.tp = g.tp;
  a.tp.status = kernel_status_device_ptr();
  a.tp.tag = next_launch_tag();
  a.tp.wait_cycles = tp_wait_limit();
  const int chunks = (g.k + 255) >> 8;
  a.sections = sections_for(g.k, g.n);
  a.sec_chunks = (chunks + a.sections - 1) / a.sections;
  const int units = min(2 * a.sec_chunks, (g.k + kStreamUnitK - 1) / kStreamUnitK);
  a.kgroups = 1;
  while (a.kgroups < kWarps && a.kgroups * 2 <= units) a.kgroups *= 2;
  // (half as many where more than an eighth of the turns would be idle; an even number, so that a warp stays in the same half of an image's tiles)
  if (a.kgroups > 2 && (units + a.kgroups - 1) / a.kgroups * a.kgroups * 8 > units * 9) a.kgroups /= 2;
  const int slices = (g.m + 15) / 16, most = device_sms() / a.sections;
  a.per = (slices + most - 1) / most;
  const int clusters = (slices + a.per - 1) / a.per;
  const int slice_bytes = (a.kgroups + (a.sections > 1 ? a.sections : 0)) * g.n * 64;
  const int fixed = a.sec_chunks * (512 * g.n + 4 * g.n + 4) + 512 * g.n;
  a.round = min(a.per, (kSmemMax - fixed) / slice_bytes);
  const int smem = fixed + a.round * slice_bytes;
  if (g.A.image) return g.n == 1 ? launch<1, true>(a, clusters, smem, s) : launch<2, true>(a, clusters, smem, s);
  return g.n == 1 ? launch<1, false>(a, clusters, smem, s) : launch<2, false>(a, clusters, smem, s);
}

}  // namespace nvb
