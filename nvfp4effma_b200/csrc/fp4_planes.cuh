// What the GEMVs on the FP4 tensor cores (gemv_fp4.cu, gemv_fp4_n8.cu) share: BF16 activations as FP4 digit planes, and block scales that the
// tensor cores do not take as this library does.
//
// An activation is the 32-bit integer X = |x| * 2^(158 - eb), eb the largest biased exponent of its token in the CTA's range of k; plane d holds
// sign(x) * digit d of X to the base 4, the digits 0 .. 3 as the E2M1 codes of 0, 0.5, 1, 1.5.
//
// Building the planes is a serial part of every launch (the weights stream meanwhile, but only a ring's worth), 32 instructions per value when
// every digit was shifted and masked by itself and 37 through two transpositions of nibbles; here it is 16
// (4096 x 4096, eight vectors in clusters of four: 11.7 -> 10.8 us; a decode step of four 4096 / 14336 layers with eight vectors 251 -> 246 us).  X comes from one multiplication and one conversion to
// an integer; the bytes of the even and of the odd values of a group of eight are transposed by byte permutes (8 each), after which the
// digits of four values are a mask away from their places in the plane's word: nibble 2 j is even value j, nibble 2 j + 1 odd value j.
#pragma once
#include "operands.cuh"

namespace nvb {

constexpr int kPlaneMinExp = 31;   // eb is taken no smaller: 2^(158 - eb) has to be a float

__device__ __forceinline__ uint32_t u16x2_max(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("max.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t u16x2_min(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("min.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t u16x2_add(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("add.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
// the largest magnitude of eight BF16 values, as a 15-bit pattern
__device__ __forceinline__ uint32_t bf16x8_max(const uint4 &x) {
  const uint32_t m = u16x2_max(u16x2_max(x.x & 0x7FFF7FFFu, x.y & 0x7FFF7FFFu), u16x2_max(x.z & 0x7FFF7FFFu, x.w & 0x7FFF7FFFu));
  return max(m & 0xFFFFu, m >> 16);
}

// Non-zero if some of the eight values has bits below the last plane.  A value less than 2^24 below the token's
// largest has none, so the exact look at each is rare.
__device__ __forceinline__ uint32_t planes_lost_bits(const uint4 &x, int eb) {
  const uint32_t w[4] = {x.x, x.y, x.z, x.w};
  uint32_t m = 0xFFFFFFFFu;
#pragma unroll
  for (int j = 0; j < 4; ++j) m = u16x2_min(m, u16x2_add(w[j] & 0x7FFF7FFFu, 0xFFFFFFFFu));   // (zeros wrap round)
  if (min(m & 0xFFFFu, m >> 16) + 1u >= (uint32_t)max(eb - 24, 0) << 7) return 0;
  uint32_t lost = 0;
#pragma unroll 1
  for (int i = 0; i < 8; ++i) {
    const uint32_t h = (i < 2 ? w[0] : i < 4 ? w[1] : i < 6 ? w[2] : w[3]) >> (16 * (i & 1)) & 0x7FFFu, e = h >> 7, mant = (h & 0x7Fu) | (e ? 0x80u : 0u);
    const int sh = (int)max(e, 1u) - eb + 24;
    if (sh < 0) lost |= mant & ((1u << min(-sh, 8)) - 1u);
  }
  return lost;
}

// what the planes drop of value i of the eight (0 if nothing): x less its bits from the last plane up
__device__ __forceinline__ float planes_rest(const uint4 &x, int i, int eb) {
  const uint32_t h = ((i < 2 ? x.x : i < 4 ? x.y : i < 6 ? x.z : x.w) >> (16 * (i & 1))) & 0xFFFFu;
  const float v = __uint_as_float(h << 16), a = fabsf(v);
  const uint32_t X = __float2uint_rz(__fmul_rn(a, __int_as_float((158 - eb + 127) << 23)));
  const float rest = __fsub_rn(a, __fmul_rn(__fmul_rn((float)X, 0x1p-31f), __int_as_float(eb << 23)));   // (X below 2^8 or without lost bits: exact)
  return v < 0.f ? -rest : rest;
}

// word d of the sixteen planes of eight consecutive values; scale = 2^(158 - eb)
__device__ __forceinline__ void planes_of_8(const uint4 &x, float scale, uint32_t (&word)[16]) {
  const uint32_t w[4] = {x.x, x.y, x.z, x.w};
  uint32_t E[4], O[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    E[j] = __float2uint_rz(__fmul_rn(__uint_as_float((w[j] << 16) & 0x7FFF0000u), scale));   // exact unless bits are lost
    O[j] = __float2uint_rz(__fmul_rn(__uint_as_float(w[j] & 0x7FFF0000u), scale));
  }
  // signs: byte j of `s` has value 2 j's in bit 3 and value 2 j + 1's in bit 7
  const uint32_t lo = byte_perm(byte_perm(w[0], w[1], 0x0051u), byte_perm(w[2], w[3], 0x0051u), 0x5410u);
  const uint32_t hi = byte_perm(byte_perm(w[0], w[1], 0x0073u), byte_perm(w[2], w[3], 0x0073u), 0x5410u);
  const uint32_t s = ((lo >> 4) & 0x08080808u) | (hi & 0x80808080u);
  auto transpose = [](uint32_t (&v)[4]) {   // byte b of v[j] -> byte j of v[b]
    const uint32_t a = byte_perm(v[0], v[1], 0x5140u), b = byte_perm(v[2], v[3], 0x5140u);
    const uint32_t c = byte_perm(v[0], v[1], 0x7362u), d = byte_perm(v[2], v[3], 0x7362u);
    v[0] = byte_perm(a, b, 0x5410u);
    v[1] = byte_perm(a, b, 0x7632u);
    v[2] = byte_perm(c, d, 0x5410u);
    v[3] = byte_perm(c, d, 0x7632u);
  };
  transpose(E);
  transpose(O);
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    word[4 * b] = (E[b] & 0x03030303u) | ((O[b] << 4) & 0x30303030u) | s;
    word[4 * b + 1] = ((E[b] >> 2) & 0x03030303u) | ((O[b] << 2) & 0x30303030u) | s;
    word[4 * b + 2] = ((E[b] >> 4) & 0x03030303u) | (O[b] & 0x30303030u) | s;
    word[4 * b + 3] = ((E[b] >> 6) & 0x03030303u) | ((O[b] >> 2) & 0x30303030u) | s;
  }
}

// The planes' words -> rows 0 .. 15 (128 bytes each, 128-byte swizzle) of a token's 2 KiB of a chunk of 256 values; b = byte of the word in a row.
__device__ __forceinline__ void store_planes(uint8_t *base, int b, const uint32_t (&word)[16]) {
#pragma unroll
  for (int d = 0; d < 16; ++d) *(uint32_t *)(base + (d >> 3) * 1024 + (d & 7) * 128 + (b ^ ((d & 7) << 4))) = word[d];
}

// The tensor cores take block scales as unsigned: a negative code's sign moves into the block's sixteen weights.  `st`: a stage's nibbles, 256
// rows of 128 bytes with the 128-byte swizzle; `sf`: this lane's 16 bytes of the stage's first scale tile (word q of tile (h, j): blocks 4 j ..
// 4 j + 3 of row 128 h + 32 q + lane).
__device__ __forceinline__ void move_signs(uint8_t *st, uint8_t *sf, int lane) {
#pragma unroll 1
  for (int i = 0; i < 32; ++i) {
    uint32_t *const wp = (uint32_t *)(sf + (i >> 4) * 2048 + ((i >> 2) & 3) * 512) + (i & 3);
    const uint32_t w = *wp;
    const int row = (i >> 4) * 128 + (i & 3) * 32 + lane;
    for (int b = 0; b < 4; ++b)
      if (w >> (8 * b + 7) & 1u) {
        const int jj = (i & 12) + b;   // block of 16 weights within the chunk
        uint2 *const nib = (uint2 *)(st + (row >> 3) * 1024 + (row & 7) * 128 + (((jj >> 1) ^ (row & 7)) << 4) + (jj & 1) * 8);
        *nib = make_uint2(nib->x ^ 0x88888888u, nib->y ^ 0x88888888u);
      }
    *wp = w & 0x7F7F7F7Fu;
  }
}

// Block scale code 0x7F (with either sign) is 480 everywhere in this library, as in the reference's decode; the tensor cores take it for a NaN, which
// reaches the partial sums of that weight row and of no other (activations and weights are finite here).  Such a row's sum over the CTA's
// blocks [b0, b1) on the CUDA cores, from memory, in the order of the CUDA-core consumer below; never met in a matrix that a quantizer made from finite
// values.  (Inlined: as a function it costs every launch 4 us.)
__device__ __forceinline__ float code_7f_sum(const Fp4Operand &A, const uint16_t *x, int row, int b0, int b1) {
  float acc = 0.f;
  for (int b = b0; b < b1; ++b) {
    const uint2 w = A.block(row, b);
    float part = 0.f;
    for (int i = 0; i < 16; ++i) part = __fmaf_rn((float)e2m1_x2(((i < 8 ? w.x : w.y) >> (4 * (i & 7))) & 15u), __uint_as_float((uint32_t)x[16 * b + i] << 16), part);
    acc = __fmaf_rn(__fmul_rn(A.scale(row, b), 0.5f), part, acc);
  }
  return acc;
}

}  // namespace nvb
