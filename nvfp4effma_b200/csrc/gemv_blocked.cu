// Decode GEMV for block-scaled activations: D[m x n] = A[m x k] (NVFP4) * B[n x k]^T with 1 <= n <= 8 and B either INT8 with one
// FP32 scale per 16 values (W4A8) or NVFP4 (W4A4).  Per output and 16-block the kernel forms the EXACT integer sum of
// (2 a) * b (weights expanded to 2 * e2m1, activations as int8 / 2 * e2m1), then acc = fma(p * sa, sb, acc) in FP32
// and a final * 1/2 (INT8) or * 1/4 (NVFP4) -- the arithmetic of the reference's blocked GEMV
// (src/gemv_nvfp4effma.cuh:26-234 there); the order of the FP32 additions over k is this kernel's own, so results agree
// with the exact definition within the FP32 accumulation bound.
//
// The integer sums come from mma.sync.m16n8k32 (s8): sixteen weight rows against eight columns.  So that every 16-block keeps a sum of its own
// while the weights are read as they lie (lane l of a quad holds 16-byte chunk l -- two blocks -- of rows g and g + 8), the columns are
// (quad lane, vector) pairs: column 2 l + j holds vector j's values in the k positions of lane l's chunk and zeros in the other lanes'.
// Two MMAs (a block is two words of eight nibbles) then give lane l the sums of ITS block for two vectors, and its own block scales apply.
// (DP4A instead: eight times as many instructions at a fraction of the rate: 14336 x 4096, four vectors, same loads: 26.5 us.)
//
// A tile is G groups of 16 rows; S warps (at most 8) share a group and take its 256-value units in turn.  CTAs are persistent: the activations (int8,
// n x k bytes) and their block scales (FP32) are staged once per CTA, and a warp's next unit (2 KiB) -- of the next tile, at a tile's end -- is in
// flight while it computes one.  The lanes' and warps' sums are added in a fixed order, then the tile runs the plain or extended epilogue.
//
// What bounds it: instruction issue (decoding: 11 instructions per 8 weights) and the loads in flight (registers: 16 warps per SM).
// 14336 x 4096 with 1 / 4 / 8 vectors: 27.5 / 32.1 / 39.0 us with a warp per four rows, DP4A and no prefetch; 16.1 / 19.7 / 27.9 us here
// (HBM time 5.1 us).  Small matrices are bound by fetching the code: 1024 x 1024 with 1 / 4 / 8 vectors 3.0 / 3.55 / 4.1 us then, 3.1 / 3.6 / 4.4
// unrolled, 2.7 / 3.1 / 3.7 in the form for one unit per warp (CUDA graph); 256 x 64 with eight 3.6, 4.5, 3.1.
#include <atomic>
#include "operands.cuh"

namespace nvb {

namespace {

constexpr int kMaxN = 8, kMaxWarps = 16;   // warps of a CTA
constexpr int kSmemLimit = 200 * 1024;

struct GemvQArgs {
  int m, n, k;
  int ksplit;          // warps that share a group of 16 rows
  Fp4Operand A;
  BOperand B;
  Epilogue e;
  EpilogueEx ex;
};

// eight E2M1 nibbles -> eight int8 values 2 * e2m1 (lo: nibbles 0-3, hi: 4-7).  A set bit 3 of a PRMT selector nibble returns the looked-up
// byte's sign (0 here) instead of the byte: w picks the magnitudes of the positive nibbles, w ^ 0x88888888 those of the negative ones.
__device__ __forceinline__ void dec8(uint32_t w, uint32_t &lo, uint32_t &hi) {
  const uint32_t n = w ^ 0x88888888u;                                 // magnitudes 0 1 2 3 | 4 6 8 12
  lo = (byte_perm(0x03020100u, 0x0C080604u, w) - byte_perm(0x03020100u, 0x0C080604u, n) + 0x80808080u) ^ 0x80808080u;   // no borrow between bytes
  hi = (byte_perm(0x03020100u, 0x0C080604u, w >> 16) - byte_perm(0x03020100u, 0x0C080604u, n >> 16) + 0x80808080u) ^ 0x80808080u;
}

__device__ __forceinline__ void mma_s8(int (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// P: pairs of activation vectors.  HALVES: 128-value halves per unit of a warp, 2 or 1.  ONE: a warp has one unit of a tile at most (any n up to 8),
// whose pairs go through one short loop and leave for the epilogue at once -- the unrolled form of eight vectors is bound by fetching its
// code there.
template <int P, int HALVES, bool ONE>
__global__ void __launch_bounds__(32 * kMaxWarps, 1) gemv_blocked_kernel(const GemvQArgs g) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ float colscale[2 * P];
  const int gm = g.m, gn = g.n, gk = g.k, nb = gk >> 4;
  int8_t *xq = (int8_t *)smem;                       // [n][k]
  float *xs = (float *)(smem + (size_t)gn * gk);     // [n][k / 16]
  float *part = xs + gn * nb;                        // [2][warp][n][16 rows]: the warps' sums of a tile
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool fp4b = g.B.dtype == NVFP4A_NVFP4;
  const bool ue_a = g.A.ue != 0;

  // ---- rows ----
  const int T = blockDim.x, W = T >> 5, S = g.ksplit, G = W / S, kRows = 16 * G;   // S warps share a group of 16 rows, G groups are a tile
  const int tiles = (gm + kRows - 1) / kRows;
  const int nchunks = gk >> 5, units = (nchunks + 4 * HALVES - 1) / (4 * HALVES);   // a chunk: 32 values = 16 bytes = two blocks; a unit: 8 chunks (or 4)
  const int grp = warp / S, ws = warp - grp * S, gq = lane >> 2, tq = lane & 3;
  // A unit of a row: 128 bytes of nibbles, `du` bytes from the row's previous unit, and sixteen scale codes, `ds` from the previous ones
  // (linear: in sequence; swizzled and image: four to each 512-byte tile).
  const bool img = g.A.image, swz = img || g.A.sld <= 0;
  const int du = img ? kImgTileBytes : 128, ds = img ? kImgTileBytes : swz ? 2048 : 16;
  const int sc_half = swz ? 1024 : 8;
  const uint8_t *pw[2], *ps[2];
  int c_next = 0;
  auto start_row = [&](int tile, int v) {   // the lane's pointers to unit v of its two rows of a tile
    const int u = HALVES == 2 ? v : v >> 1, odd = HALVES == 2 ? 0 : v & 1;   // 256-value unit, its second half
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int row = min(tile * kRows + 16 * grp + gq + 8 * r, gm - 1), rr = row & 127;
      const size_t in_tile = (size_t)odd * 1024 + (tq >> 1) * 512 + (rr & 31) * 16 + (rr >> 5) * 4 + (tq & 1) * 2;
      if (img) {
        const uint8_t *t = g.A.data + ((size_t)(row >> 7) * g.A.ktiles + u) * kImgTileBytes;
        pw[r] = t + rr * 128 + odd * 64 + tq * 16;
        ps[r] = t + kImgDataBytes + in_tile;
      } else {
        pw[r] = g.A.data + (size_t)row * (g.A.ld >> 1) + (size_t)u * 128 + odd * 64 + tq * 16;
        ps[r] = swz ? g.A.sc + (size_t)(row >> 7) * ((size_t)((-g.A.sld) >> 2) * 512) + (size_t)u * 2048 + in_tile
                    : g.A.sc + (size_t)row * g.A.sld + (size_t)u * 16 + odd * 8 + tq * 2;
      }
    }
    c_next = 8 * u + 4 * odd + tq;
  };
  uint4 w_next[2][2];        // [chunk of the lane][row gq, gq + 8]
  uint32_t sc_next[2][2];
  auto prefetch = [&]() {
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (h < HALVES && c_next + 4 * h < nchunks)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          w_next[h][r] = __ldg((const uint4 *)(pw[r] + 64 * h));
          sc_next[h][r] = __ldg((const uint16_t *)(ps[r] + (h ? sc_half : 0)));
        }
  };
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int r = 0; r < 2; ++r) { w_next[h][r] = make_uint4(0, 0, 0, 0); sc_next[h][r] = 0; }
  start_row(blockIdx.x, ws);   // (the grid has no more CTAs than tiles)
  prefetch();

  // ---- stage the activations: int8 values and FP32 block scales (the first weights are on their way) ----
  if (fp4b) {
    for (int idx = tid; idx < gn * nb; idx += blockDim.x) {
      const int j = idx / nb, kb = idx - j * nb;
      const uint2 w = g.B.q.block(j, kb);
      uint4 d;
      dec8(w.x, d.x, d.y); dec8(w.y, d.z, d.w);
      *(uint4 *)(xq + (size_t)j * gk + 16 * kb) = d;
      xs[idx] = g.B.q.scale(j, kb);
    }
  } else {
    for (int idx = tid; idx < gn * nb; idx += blockDim.x) {
      const int j = idx / nb, kb = idx - j * nb;
      *(uint4 *)(xq + (size_t)j * gk + 16 * kb) = __ldg((const uint4 *)((const int8_t *)g.B.data + (size_t)j * g.B.ld + 16 * kb));
      xs[idx] = g.B.s8[(size_t)j * g.B.lds8 + kb];
    }
  }
  if (g.ex.mask & kExNorm) {   // a warp per vector in turn: a CTA may have fewer warps (four) than there are vectors
    for (int j = warp; j < gn; j += W) {
      const float s = warp_norm_scale(g.ex, j, lane);
      if (lane == 0) colscale[j] = s;
    }
  }
  __syncthreads();

  const bool diag = (gq >> 1) == tq;   // this lane's column of B is its own chunk's (see the head of the file)
  // two vectors j0, j0 + 1 against the lane's chunk c: use(row r, vector jj, the two blocks' sums times the weight scales, their activation scales)
  auto block_sums = [&](const uint32_t (&a)[4][4], const float (&sa)[2][2], int j0, int c, bool in, auto use) {
    const int jb = j0 + (gq & 1);
    uint4 x0 = make_uint4(0, 0, 0, 0), x1 = x0;
    if (diag && in && jb < gn) {
      x0 = *(const uint4 *)(xq + (size_t)jb * gk + 32 * c);
      x1 = *(const uint4 *)(xq + (size_t)jb * gk + 32 * c + 16);
    }
    // (an integer sum of at most 16 x 12 x 128 added to the bits of 1.5 * 2^23 is that float's value plus the sum)
    int c0[4] = {0x4B400000, 0x4B400000, 0x4B400000, 0x4B400000}, c1[4] = {0x4B400000, 0x4B400000, 0x4B400000, 0x4B400000};
    mma_s8(c0, a[0], x0.x, x0.y);
    mma_s8(c1, a[2], x1.x, x1.y);
    mma_s8(c0, a[1], x0.z, x0.w);
    mma_s8(c1, a[3], x1.z, x1.w);
#pragma unroll
    for (int jj = 0; jj < 2; ++jj) {
      float2 xsv = make_float2(0.f, 0.f);
      if (in) xsv = *(const float2 *)(xs + min(j0 + jj, gn - 1) * nb + 2 * c);
#pragma unroll
      for (int r = 0; r < 2; ++r)
        use(r, jj, __fmul_rn(__fadd_rn(__int_as_float(c0[2 * r + jj]), -12582912.f), sa[r][0]),
            __fmul_rn(__fadd_rn(__int_as_float(c1[2 * r + jj]), -12582912.f), sa[r][1]), xsv.x, xsv.y);
    }
  };
  const Epilogue &e = g.e;
  float amax = 0.f;
  int buf = 0;
#pragma unroll 1
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, buf ^= 1) {
  const int i0 = tile * kRows;
  if constexpr (ONE) {
    float *const mine = part + ((size_t)buf * W + warp) * gn * 16;
    const int c = c_next;
    const bool in = c < nchunks;   // (a lane past the end multiplies zeros)
    uint32_t a[4][4];              // [word][MMA operand register]
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      dec8(((const uint32_t *)&w_next[0][0])[i], a[i][0], a[i][2]);
      dec8(((const uint32_t *)&w_next[0][1])[i], a[i][1], a[i][3]);
    }
    float sa[2][2];
#pragma unroll
    for (int r = 0; r < 2; ++r) { sa[r][0] = scale_to_f32(sc_next[0][r] & 0xFFu, ue_a); sa[r][1] = scale_to_f32(sc_next[0][r] >> 8, ue_a); }
    if (tile + (int)gridDim.x < tiles) {
      start_row(tile + gridDim.x, ws);
      prefetch();
    }
#pragma unroll 1
    for (int j0 = 0; j0 < gn; j0 += 2) {
      float v[2][2];
      block_sums(a, sa, j0, c, in, [&](int r, int jj, float s0, float s1, float x0, float x1) { v[r][jj] = __fmaf_rn(s1, x1, __fmul_rn(s0, x0)); });
#pragma unroll
      for (int jj = 0; jj < 2; ++jj)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          float t = v[r][jj];
          t = __fadd_rn(t, __shfl_xor_sync(0xFFFFFFFFu, t, 1));
          t = __fadd_rn(t, __shfl_xor_sync(0xFFFFFFFFu, t, 2));
          if (tq == 0 && j0 + jj < gn) mine[(j0 + jj) * 16 + gq + 8 * r] = t;
        }
    }
  } else {
  float acc[2][2 * P];
#pragma unroll
  for (int j = 0; j < 2 * P; ++j) acc[0][j] = acc[1][j] = 0.f;
#pragma unroll 1
  for (int u = ws; u < units; u += S) {
    uint4 w[2][2];
    uint32_t sc[2][2];
    const int c_unit = c_next;
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int r = 0; r < 2; ++r) { w[h][r] = w_next[h][r]; sc[h][r] = sc_next[h][r]; }
    if (u + S < units) {
#pragma unroll
      for (int r = 0; r < 2; ++r) { pw[r] += (size_t)(S * HALVES / 2) * du; ps[r] += (size_t)(S * HALVES / 2) * ds; }   // (several 128-value units: S is 8)
      c_next += 4 * HALVES * S;
      prefetch();
    } else if (tile + (int)gridDim.x < tiles) {
      start_row(tile + gridDim.x, ws);
      prefetch();
    }
#pragma unroll
    for (int h = 0; h < HALVES; ++h) {
      if (P == 4 && h) __syncwarp();   // (keeps the compiler from interleaving the halves, for which the registers do not suffice)
      const int c = c_unit + 4 * h;
      const bool in = c < nchunks;       // (a lane past the end multiplies zeros and leaves its sums alone)
      uint32_t a[4][4];                  // [word][MMA operand register]
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        dec8(((const uint32_t *)&w[h][0])[i], a[i][0], a[i][2]);
        dec8(((const uint32_t *)&w[h][1])[i], a[i][1], a[i][3]);
      }
      float sa[2][2];
#pragma unroll
      for (int r = 0; r < 2; ++r) { sa[r][0] = scale_to_f32(sc[h][r] & 0xFFu, ue_a); sa[r][1] = scale_to_f32(sc[h][r] >> 8, ue_a); }
#pragma unroll
      for (int p = 0; p < P; ++p) {
        if (2 * p >= gn) break;
        block_sums(a, sa, 2 * p, c, in, [&](int r, int jj, float s0, float s1, float x0, float x1) {
          acc[r][2 * p + jj] = __fmaf_rn(s0, x0, acc[r][2 * p + jj]);
          acc[r][2 * p + jj] = __fmaf_rn(s1, x1, acc[r][2 * p + jj]);
        });
      }
    }
  }
  float *const mine = part + ((size_t)buf * W + warp) * gn * 16;
#pragma unroll
  for (int j = 0; j < 2 * P; ++j) {
    if (j >= gn) break;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      float v = acc[r][j];
      v = __fadd_rn(v, __shfl_xor_sync(0xFFFFFFFFu, v, 1));
      v = __fadd_rn(v, __shfl_xor_sync(0xFFFFFFFFu, v, 2));
      if (tq == 0) mine[j * 16 + gq + 8 * r] = v;
    }
  }
  }
  __syncthreads();

  // ---- epilogue: a thread per (row, column) of the tile; the S warps' sums are added pairwise (one after another, a sum is 6 % less exact) ----
  const bool neighbours = (g.ex.mask & (kExSwiglu | kExOut2)) != 0;
  const int outs = kRows * gn;
  for (int o = tid; o < outs; o += T) {
    const int ri = o % kRows, cj = o / kRows, i = i0 + ri;
    float *const p0 = part + ((size_t)buf * W + (ri >> 4) * S) * gn * 16 + cj * 16 + (ri & 15);
    float t[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) t[q] = q < S ? p0[q * gn * 16] : 0.f;
    const float sum = __fadd_rn(__fadd_rn(__fadd_rn(t[0], t[1]), __fadd_rn(t[2], t[3])), __fadd_rn(__fadd_rn(t[4], t[5]), __fadd_rn(t[6], t[7])));
    float v = 0.f;
    if (i < gm) {
      float colp = epi_col_part(e, cj);
      if (g.ex.mask & kExNorm) colp = __fmul_rn(colp, colscale[cj]);
      v = epi_value(e, i, cj, __fmul_rn(sum, fp4b ? 0.25f : 0.5f), epi_scale(e, epi_row_part(e, i), colp));
      if (!neighbours) { store_dense(e.d_dtype, e.d, (size_t)cj * e.ldd + i, v); amax = fmaxf(amax, fabsf(v)); }
    }
    if (neighbours) *p0 = v;   // (in the place of the first sum, which only this thread reads)
  }
  if (neighbours) {
    __syncthreads();
    for (int o = tid; o < outs; o += T) {
      const int ri = o % kRows, cj = o / kRows, i = i0 + ri;
      const float *const p0 = part + ((size_t)buf * W + (ri >> 4) * S) * gn * 16 + cj * 16 + (ri & 15);
      const float v = *p0;
      const bool live = i < gm;
      if (g.ex.mask & kExSwiglu) {
        if (live && !(ri & 8)) {
          const float h = silu_mul(v, p0[8]);
          store_dense(e.d_dtype, e.d, (size_t)cj * e.ldd + (i >> 4) * 8 + (i & 7), h);
          amax = fmaxf(amax, fabsf(h));
        }
      } else if (live) {
        store_dense(e.d_dtype, e.d, (size_t)cj * e.ldd + i, v);
        amax = fmaxf(amax, fabsf(v));
      }
      if (g.ex.mask & kExOut2) {
        if (live) store_dense(g.ex.d2_dtype, g.ex.d2, (size_t)cj * g.ex.ldd2 + i, __fmul_rn(v, load_dense(g.ex.w2_dtype, g.ex.w2, i)));
        if (live && !(ri & 15)) {
          float sq = 0.f;
#pragma unroll
          for (int r = 0; r < 16; ++r) sq = __fadd_rn(sq, __fmul_rn(p0[r], p0[r]));
          g.ex.sq[(size_t)cj * g.ex.ld_sq + (i >> 4)] = sq;
        }
      }
    }
  }
  }
  if (e.amax) warp_amax_commit(e.amax, amax);
}

size_t smem_bytes(int n, int k) { return (size_t)n * k + (size_t)n * (k / 16) * sizeof(float); }   // the activations
int part_bytes(int warps, int n) { return 2 * warps * n * 16 * (int)sizeof(float); }

}  // namespace

bool gemv_blocked_supports(const GemmArgs &g) {
  if (!(g.n >= 1 && g.n <= kMaxN && g.k >= 64 && (g.B.dtype == NVFP4A_INT8 || g.B.dtype == NVFP4A_NVFP4))) return false;
  if (g.B.dtype == NVFP4A_NVFP4 && g.B.q.image) return false;
  if (g.B.dtype == NVFP4A_INT8 && (((uintptr_t)g.B.data & 15) || g.B.ld % 16)) return false;
  return smem_bytes(g.n, g.k) <= (size_t)kSmemLimit;
}

template <int P, int HALVES, bool ONE = false>
static cudaError_t launch_pairs(GemvQArgs &a, int warps, cudaStream_t s) {
  static std::atomic<bool> attr_set[64];   // zero-initialised; set once per device (a repeated cudaFuncSetAttribute is harmless)
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set[dev & 63]) {
    if (cudaError_t e = cudaFuncSetAttribute(gemv_blocked_kernel<P, HALVES, ONE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit + part_bytes(kMaxWarps, kMaxN))) return e;
    attr_set[dev & 63] = true;
  }
  const int rows = 16 * (warps / a.ksplit), tiles = (a.m + rows - 1) / rows, smem = (int)smem_bytes(a.n, a.k) + part_bytes(warps, a.n);
  int per_sm = kMaxWarps / warps;   // (by its registers)
  while (per_sm > 1 && per_sm * (smem + 2048) > 227 * 1024) --per_sm;
  const int grid = tiles < per_sm * device_sms() ? tiles : per_sm * device_sms();
  gemv_blocked_kernel<P, HALVES, ONE><<<grid, warps * 32, smem, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_gemv_blocked(const GemmArgs &g, cudaStream_t s) {
  GemvQArgs a;
  a.m = g.m; a.n = g.n; a.k = g.k;
  a.A = g.A; a.B = g.B; a.e = g.e; a.ex = g.x;
  // How a row's k is dealt to warps depends on k alone, so that a row's bits do not depend on the matrix around it (or on n): eight warps in
  // 256-value units, or below 2048 values in 128-value half units (every warp has one: as many roundings on the way to a sum as a lane per
  // chunk and a butterfly; in 256-value units 1088 values are up to 3 % less exact).
  // CTAs of eight warps, two per SM; of sixteen (two groups) where a CTA gets one tile at most or the activations leave room for one CTA:
  // 4096 x 14336, 4 / 8 vectors 21.0 / 34.7 -> 18.8 / 26.0 us, 4096 x 4096, 8 vectors 11.8 -> 11.0 us.  Fewer than eight only if that gives more CTAs.
  const int groups = (g.m + 15) / 16, sms = device_sms();
  a.ksplit = 8;
  while (a.ksplit > 1 && a.ksplit * 64 >= g.k) a.ksplit >>= 1;
  int warps = 8;
  if (a.ksplit < 8 && groups <= 2 * sms) a.ksplit = warps = 4;   // (a warp without a unit adds zeros)
  if (g.k > 1024 && ((groups > sms && groups <= 2 * sms) || 2 * (smem_bytes(g.n, g.k) + part_bytes(8, g.n) + 2048) > 227 * 1024)) warps = 16;
  if (g.k <= 1024) return launch_pairs<4, 1, true>(a, warps, s);
  if (g.k < 2048) return g.n <= 2 ? launch_pairs<1, 1>(a, warps, s) : g.n <= 4 ? launch_pairs<2, 1>(a, warps, s) : launch_pairs<4, 1>(a, warps, s);
  return g.n <= 2 ? launch_pairs<1, 2>(a, warps, s) : g.n <= 4 ? launch_pairs<2, 2>(a, warps, s) : launch_pairs<4, 2>(a, warps, s);
}

}  // namespace nvb
