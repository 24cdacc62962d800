// What the decode GEMVs on FP16 pairs share (gemv_stream.cu: BF16 activations, gemv_q8.cu: INT8 / NVFP4 activations): the weights' way into registers, their
// conversion, and the epilogue of a run of 16-row slices.
#pragma once
#include "operands.cuh"
#include "sm100.cuh"

namespace nvb {

constexpr int kStreamUnitK = 128;      // a warp's unit: 16 rows x 128 values

__device__ __forceinline__ void prefetch_line(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

__device__ __forceinline__ void mma16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// the first of a chain: nothing to add to
__device__ __forceinline__ void mma16_first(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ uint4 lds16(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ uint32_t ld2(const uint8_t *p) {
  uint16_t v;
  asm("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(p));
  return v;
}
// products of FP16 pairs
__device__ __forceinline__ uint32_t h2mul(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t word(const uint4 &v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }
// slices of 16 rows in the order a matrix is dealt out: the four slices of a 128-row tile whose scale codes share 16-byte lines follow one another
__device__ __forceinline__ int slice_row(int s, int m) {
  return s < ((m >> 7) << 3) ? (s >> 3) * 128 + (s & 3) * 32 + ((s >> 2) & 1) * 16 : s * 16;
}

// A warp's unit as a lane holds it: rows gq and gq + 8, 32 values of k and two scale codes each.
struct WeightUnit { uint4 wa, wb; uint32_t ca, cb; };

// The units of one warp: of every SG-th slice of a CTA's run, every KG-th unit of the CTA's range of k [256 c_first, 256 c_first + kloc).  KG is even, or a slice
// has one unit: a warp then stays in the same half of an image's tiles.
// Every address comes from `data` and `sc`: start_behind_wait() makes them values that the compiler cannot have known before the programmatic wait, so that no load
// of any slice moves up across it (see behind_wait).
template <bool IMG> struct UnitStream {
  const Fp4Operand &A;
  const uint8_t *data, *sc;   // A's
  int gm, s_first, s_count, c_first, kloc, units, KG, SG, kg, sg, gq, q;
  bool lin;
  int slice, unit;            // the next unit to be requested
  const uint8_t *w, *s;       // where it is for row gq
  uint32_t w8, s8;            // from there to row gq + 8
  uint32_t step_w, step_s;
  __device__ __forceinline__ UnitStream(const Fp4Operand &a, int gm_, int s_first_, int s_count_, int c_first_, int kloc_, int KG_, int warp, int warps, int lane)
      : A(a), data(a.data), sc(a.sc), gm(gm_), s_first(s_first_), s_count(s_count_), c_first(c_first_), kloc(kloc_), units((kloc_ + kStreamUnitK - 1) / kStreamUnitK), KG(KG_),
        SG(warps / KG_), kg(warp & (KG_ - 1)), sg(warp / KG_), gq(lane >> 2), q(lane & 3), lin(!IMG && a.sld > 0), w(a.data), s(a.data), w8(0), s8(0) {
    step_w = IMG ? (uint32_t)(KG >> 1) * kImgTileBytes : (uint32_t)KG * 64;
    step_s = IMG ? (uint32_t)(KG >> 1) * kImgTileBytes : (uint32_t)KG * (lin ? 8 : 1024);
    restart(sg);
  }
  __device__ __forceinline__ void start_slice() {
    const int row0 = slice_row(s_first + slice, gm);
    if (IMG) {
      const int rr = (row0 & 127) + gq;
      const uint8_t *t = data + ((size_t)(row0 >> 7) * A.ktiles + c_first + (kg >> 1)) * kImgTileBytes;
      w = t + rr * 128 + (kg & 1) * 64 + q * 16;
      s = t + kImgDataBytes + (kg & 1) * 1024 + (q >> 1) * 512 + (rr & 31) * 16 + (rr >> 5) * 4 + (q & 1) * 2;
      w8 = 1024; s8 = 128;
    } else {
      const int r0 = min(row0 + gq, gm - 1), r1 = min(row0 + gq + 8, gm - 1);
      const ScalePos sp{A.sld};
      w = data + (size_t)r0 * (A.ld >> 1) + (size_t)c_first * 128 + kg * 64 + q * 16;
      w8 = (uint32_t)(r1 - r0) * (uint32_t)(A.ld >> 1);
      s = sc + sp.row(r0) + (lin ? (size_t)c_first * 16 + kg * 8 + q * 2 : (size_t)c_first * 2048 + kg * 1024 + (q >> 1) * 512 + (q & 1) * 2);
      s8 = (uint32_t)(sp.row(r1) - sp.row(r0));
    }
  }
  __device__ __forceinline__ void restart(int at) {
    slice = kg < units ? at : s_count;
    unit = kg;
    if (slice < s_count) start_slice();
  }
  // after the programmatic wait: the first unit again
  __device__ __forceinline__ void start_behind_wait() {
    data = behind_wait(data);
    if (!IMG) sc = behind_wait(sc);
    restart(sg);
  }
  __device__ __forceinline__ bool in_k() const { return IMG || unit * kStreamUnitK + q * 32 < kloc; }   // (the last unit of a plain operand may be short)
  __device__ __forceinline__ void advance() {
    unit += KG; w += step_w; s += step_s;
    if (unit >= units) {
      unit = kg; slice += SG;
      if (slice < s_count) start_slice();
    }
  }
  // the first units' lines into L2 (a prefetch reads nothing: a predecessor may still be writing the weights); start_behind_wait() follows
  __device__ __forceinline__ void prefetch(int count) {
    for (int i = 0; i < count && slice < s_count; ++i) {
      if (in_k()) { prefetch_line(w); prefetch_line(w + w8); prefetch_line(s); }
      advance();
    }
  }
  __device__ __forceinline__ WeightUnit fetch() {
    WeightUnit v;
    v.wa = v.wb = make_uint4(0, 0, 0, 0);
    v.ca = v.cb = 0;
    if (slice < s_count) {
      if (in_k()) {
        v.wa = ld16((const uint4 *)w);
        v.wb = ld16((const uint4 *)(w + w8));
        v.ca = ld2(s);
        v.cb = ld2(s + s8);
      }
      advance();
    }
    return v;
  }
};

// The plain or extended epilogue of `outs` outputs, o = (slice, vector, row), of the slices from s0 on; sum_of(o) is an output's sum over k.
template <class Sum>
__device__ __forceinline__ void slices_epilogue(const Epilogue &e, const EpilogueEx &ex, int n, int s0, int outs, int gm, float ga0, const float *colscale, float &amax, Sum sum_of) {
  const int tid = threadIdx.x, lane = tid & 31;
  for (int o0 = 0; o0 < outs; o0 += blockDim.x) {
    const int o = o0 + tid;
    if ((o & ~31) >= outs) break;                       // (whole warps)
    const int ri = o & 15, cj = (o >> 4) % n, row0 = slice_row(s0 + (o >> 4) / n, gm), i = row0 + ri;
    const bool live = o < outs && i < gm;
    float v = 0.f;
    if (live) {
      float colp = epi_col_part(e, cj);
      if (ex.mask & kExNorm) colp = __fmul_rn(colp, colscale[cj]);
      v = epi_value(e, i, cj, sum_of(o), epi_scale(e, __fmul_rn(e.alpha, e.ga_stride ? e.ga[i] : ga0), colp));
    }
    if (ex.mask & kExSwiglu) {
      const float up = __shfl_down_sync(0xFFFFFFFFu, v, 8);
      if (live && ri < 8) {
        const float h = silu_mul(v, up);
        store_dense(e.d_dtype, e.d, (size_t)cj * e.ldd + (row0 >> 1) + ri, h);
        amax = fmaxf(amax, fabsf(h));
      }
    } else if (live) {
      store_dense(e.d_dtype, e.d, (size_t)cj * e.ldd + i, v);
      amax = fmaxf(amax, fabsf(v));
    }
    if (ex.mask & kExOut2) {
      float sq = 0.f;
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const float y = __shfl_sync(0xFFFFFFFFu, v, (lane & 16) + r);
        sq = __fadd_rn(sq, __fmul_rn(y, y));
      }
      if (live) store_dense(ex.d2_dtype, ex.d2, (size_t)cj * ex.ldd2 + i, __fmul_rn(v, load_dense(ex.w2_dtype, ex.w2, i)));
      if (live && ri == 0) ex.sq[(size_t)cj * ex.ld_sq + (i >> 4)] = sq;
    }
  }
  __syncwarp();
}

}  // namespace nvb
