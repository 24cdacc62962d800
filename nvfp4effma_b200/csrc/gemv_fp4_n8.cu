// Decode GEMV on the FP4 tensor cores for 3 to 8 BF16 activation vectors (W4A16): D[m x n] = A[m x k] (NVFP4) * B[n x k]^T.
// (One and two vectors have a kernel of their own, gemv_fp4.cu: with a handful of pieces its single-tile clusters and one epilogue CTA
// finish sooner -- a decode step of four 4096 / 14336 layers took 212 us with this kernel for one vector against 198 us.)
//
// The weights are consumed as they are stored: TMA streams 256-row x 256-k tiles of nibbles and their block scales from
// HBM into a shared-memory ring and tcgen05.mma kind::mxf4nvf4 reads them with the E4M3 block scales in tensor memory.  No
// CUDA-core instruction touches a weight, so the kernel runs at the speed the memory system delivers A (0.5625 bytes per
// weight).
//
// The BF16 activations become FP4 operands by an exact digit expansion.  For one token and the k range of one CTA let eb be
// the largest biased exponent; every |x_i| is written as X_i * 2^(eb - 158) with the 32-bit integer X_i (for BF16, whose
// significand has 8 bits, this is exact unless |x_i| < 2^-24 max|x|: such elements lose their bits below 2^-31 max|x|).
// X_i = sum over d of t_d(i) * 4^d with the base-4 digits t_d in {0, 1, 2, 3}; the E2M1 codes 0..3 are the values t / 2, so
// "piece" d of the token is the FP4 vector sign(x_i) * t_d(i) / 2 and
//     sum_i a_i x_i = 2^(eb - 157) * sum_d 4^d * (sum_i a_i * piece_d(i)).
// The 16 pieces of a token are 16 rows of the MMA's M dimension (block scales 1.0) -- eight tokens fill its 128 rows, so the MMA work
// does not depend on n -- 256 weight rows are its N dimension, and the inner sums are what the tensor cores compute: accumulator lane
// 16 t + d, column r holds piece d of token t against weight row r.  With fewer tokens the rows past the pieces read whatever follows
// them in shared memory and produce accumulator lanes nobody looks at (every FP4 bit pattern is a finite number).
//
// Work split: a thread-block cluster of `splits` CTAs owns the 256-row tiles blockIdx.y, + gridDim.y, ...; each CTA takes a contiguous
// range of k, the same for all tiles, so that its pieces (built once, 8 warps, while the first weights are in flight) serve every tile and
// the weight stream never stops between tiles.  Per tile two warps per 32 accumulator lanes weight the pieces with their powers of four
// and add them by a halving butterfly, and store each weight row's partial sums into the shared memory of the CTA that owns the row
// (256 / splits rows each, DSMEM); it adds the partials in rank order -- deterministic, no atomics, no global scratch -- and
// runs the plain or extended epilogue, a thread per (row, token).
//
// Timeline of a launch: the set-up (barriers, tensor memory) touches no global memory and runs under programmatic dependent launch
// while the previous kernel drains; the ring's first fill is requested by several warps at once right after the cluster-wide barrier,
// because a copy instruction costs its warp 150-300 ns to issue whatever it moves (an image stage is two rank-4 tensor copies: 32
// KiB of nibbles, 4 KiB of scales).
//
// Semantics: FP32 accumulation in the tensor cores' order, within the FP32 accumulation bound of the exact definition
// (reference include/nvfp4effma.h:82-92 there), as the reference's own tensor-core GEMV (src/tensors/gemv_tc.cuh there).
// Against 64-bit sums the results are about twice as close as the mma.sync GEMV's (28672 x 4096, eight vectors, FP32 D: 6.7e-8 relative
// against 1.3e-7; activations spread over 2^-17 .. 1: 1.6e-7 against 6.2e-7).
// What bounds it: 28672 x 4096 takes 20.1 us for four vectors and 22.8 us for eight (66 MB, 10.6 us of HBM time; mma.sync: 30.6 and 33.6 us,
// which decodes every weight on the CUDA cores); past the stream it is the pieces (0.11 us per chunk and vector; 0.14 with digits taken one by one and the activations read twice) and the tiles' ends.
// Negative block scales keep their sign, as in the mma.sync GEMV (gemv.cu) that takes the calls this kernel leaves.
#include <math.h>
#include <atomic>
#include "operands.cuh"
#include "sm100.cuh"
#include "tp_barrier.cuh"
#include "fp4_planes.cuh"

namespace nvb {

using namespace sm100;

namespace {

struct GemvN8Args {
  int m, n, k;
  int a_image;
  Fp4Operand A;        // (for code_7f_sum)
  const uint8_t *sa;   // plain: block scale base; image: image base
  int sa_ld, ktiles;
  int linear;          // plain operand with linear block scales: a TMA box brings [256 rows][16 bytes], four warps re-tile it
  const uint16_t *x; int ldx;
  Epilogue e;
  EpilogueEx ex;
  unsigned *status;
  unsigned tag;        // this launch's tag in the status word
  int tp_world, tp_rank;                       // > 1: wait for the peers' posts before the activations are read (TpPush::deferred bit 0)
  unsigned long long *tp_flags[kMaxRanks];
  long long tp_wait_cycles;
  int stages;          // ring depth (2..6), chosen by the host from the shared memory left beside the pieces
  int piece_bytes;     // shared memory of the activation pieces: chunks per CTA x piece rows x 128
  int tiles;           // 256-row tiles
  int buffers;         // copies of the results' exchange buffer: 1 if a cluster has one tile, else 2
};

constexpr int kThreads = 448, kDecompThreads = 256;         // warps 0, 1: copies, MMAs; 2-9: pieces and epilogue; 10-13: block scales
constexpr int kRows = 256;                                  // weight rows per tile (the MMA's N)
constexpr int kDataBytes = kRows * 128, kSfBytes = kRows * 16, kStageBytes = kDataBytes + kSfBytes;  // 36 KiB per 256-k chunk
constexpr int kTmemCols = 512;                              // accumulator [0, 256), A scales (1.0) [256, 260), B scales [272, 272 + 32 * stages), stages <= 6
constexpr int kMaxStages = 6;
constexpr int kSmemLimit = 232448 - 1024;                   // dynamic shared memory of one CTA on sm_100, less the alignment slack
constexpr unsigned kStWaitFull = 0x201, kStWaitEmpty = 0x202, kStWaitAcc = 0x203, kStWaitPieces = 0x204, kStWaitRetile = 0x205, kStWaitAccFree = 0x206,
                   kStWaitResults = 0x207;
constexpr int kRawSfBytes = kRows * 16;                      // linear scales of one chunk as they lie in memory: [256 rows][16 bytes]

// 256-k chunks a CTA may own: its pieces (2 KiB per token and chunk) lie in shared memory beside at least two stages
__host__ __device__ constexpr int max_chunks(int ntok) { return ntok == 4 ? 14 : 7; }
// Shared memory of a CTA: [pieces | stages x 36 KiB | unit scales 512 | results buffers x NTOK x 256 floats | barriers and flags 512].
// The MMA reads 16 KiB from the start of a pieces chunk (its M is 128 rows), which stays inside the stages.
__host__ __device__ constexpr int fixed_bytes(int ntok, int buffers) { return 512 + buffers * ntok * 1024 + 512; }

__device__ __forceinline__ float pow2f(int e) { return __int_as_float((e + 127) << 23); }  // -126 <= e <= 127

template <int NTOK>
__global__ void __launch_bounds__(kThreads, 1)
gemv_fp4_n8_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_s, const GemvN8Args g) {
  constexpr int PR = 16 * NTOK, NI = (NTOK * max_chunks(NTOK) * 32 + kDecompThreads - 1) / kDecompThreads;   // NI: vectors of 8 activations per thread
  constexpr int kQuads = (PR + 31) / 32, kReaders = 2 * kQuads;   // accumulator quadrants with pieces; warps that read them (two each)
  const int kStages = g.stages;
  const uint32_t rank = cluster_ctarank(), splits = gridDim.x;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t *pieces = smem;
  uint8_t *stages = smem + g.piece_bytes;
  const bool linear = g.linear;
  const int stage_bytes = kStageBytes + (linear ? kRawSfBytes : 0);
  uint8_t *unit_sf = stages + kStages * stage_bytes;
  float *res = (float *)(unit_sf + 512);                   // [buffer][source rank][token][row of the 256 / splits this CTA owns]
  uint64_t *bars = (uint64_t *)(unit_sf + 512 + g.buffers * NTOK * 1024);
  uint64_t *full = bars, *empty = bars + kMaxStages, *sf_ready = bars + 2 * kMaxStages, *acc_full = bars + 3 * kMaxStages, *acc_empty = acc_full + 1,
           *pieces_ready = acc_empty + 1, *res_full = pieces_ready + 1;
  uint32_t *tmem_slot = (uint32_t *)(res_full + 2);
  volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
  uint32_t *wmax = tmem_slot + 2;                          // [NTOK] largest |x| bit pattern
  volatile int *inexact = (volatile int *)(wmax + NTOK);   // some activation of this CTA does not fit the digit planes
  int *consumed = (int *)(wmax + NTOK + 1);                // [stage] warps done with the stage (the CUDA-core consumer)

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gm = g.m, gn = g.n;
  const int tiles128 = (gm + 127) >> 7, tiles = g.tiles, tile_first = blockIdx.y, tile_step = gridDim.y;
  const int my_tiles = tile_first < tiles ? (tiles - tile_first + tile_step - 1) / tile_step : 0;
  const bool a_image = g.a_image;
  const uint8_t *const sa_base = g.sa;
  const int sa_ld = g.sa_ld;
  const int nk = g.k >> 8;
  const int c0 = (int)((long long)rank * nk / splits), c1 = (int)((long long)(rank + 1) * nk / splits), nloc = c1 - c0;   // (splits <= nk: at least one)
  const int total = my_tiles * nloc;                       // chunks through the ring
  unsigned *const status_word = g.status;

  // One stage of the weight ring: chunk it % nloc of this CTA's tile it / nloc.  A copy instruction costs the issuing warp 150-200 cycles
  // per active lane whatever it moves, so a stage is as few copies as its layout allows, issued by as many lanes of ONE instruction: an
  // image's nibbles (32 KiB, both 128-row halves) and block scales (4 KiB) are two rank-4 tensor copies in lanes 0 and 1.
  auto request_stage = [&](int it) {
    const int s = it % kStages, ti = it / nloc, c = c0 + it - ti * nloc, tm = tile_first + ti * tile_step;
    const bool second = tm * 2 + 1 < tiles128;             // the tile's second 128 rows exist
    uint8_t *sW = stages + (size_t)s * stage_bytes, *sSf = sW + kDataBytes;
    if (lane == 0) mbar_arrive_expect_tx(&full[s], kDataBytes + (linear ? (uint32_t)kRawSfBytes : ((second || a_image) ? 4096u : 2048u)));
    __syncwarp();
    if (a_image) {
      if (lane < 2) tma_load_4d(lane ? sSf : sW, lane ? &tmap_s : &tmap_a, 0, 0, c, 2 * tm, &full[s]);
    } else if (lane < 2) {
      if (lane == 0) {
        tma_load_2d(sW, &tmap_a, c * 128, tm * 256, &full[s]);
      } else if (linear) {
        tma_load_2d(sW + kStageBytes, &tmap_s, c * 4, tm * 256, &full[s]);   // 16 bytes (4 words) of 256 rows; rows past m read zeros
      }
    } else if (lane < 4 && !linear) {
      const int h = lane - 2;
      if (h == 0 || second) bulk_load(sSf + h * 2048, sa_base + (size_t)(2 * tm + h) * ((size_t)((-sa_ld) >> 2) * 512) + (size_t)c * 2048, 2048, &full[s]);
    }
    __syncwarp();
  };

  const int early = total < kStages ? total : kStages;   // the ring's first fill needs no wait

  // The set-up touches no global memory, so it may run while the stream's previous kernel finishes (programmatic dependent
  // launch); nothing before the cluster-wide barrier waits for memory either: the first weights are requested right after it.
  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    prefetch_tensormap(&tmap_a);
    if (a_image || linear) prefetch_tensormap(&tmap_s);
    for (int s = 0; s < kStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); mbar_init(&sf_ready[s], 1); }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, kReaders);
    mbar_init(pieces_ready, kDecompThreads / 32);
    for (int b = 0; b < 2; ++b) mbar_init(&res_full[b], splits * kReaders);
    *abort_flag = 0;
    *inexact = 0;
    for (int t = 0; t < NTOK; ++t) wmax[t] = 0;
    for (int s = 0; s < kStages; ++s) consumed[s] = 0;
    fence_barrier_init();
  }
  if (threadIdx.x < 128) ((uint32_t *)unit_sf)[threadIdx.x] = 0x38383838u;  // E4M3 1.0
  fence_proxy_async_smem();
  if (warp == 1) tmem_alloc(tmem_slot, kTmemCols);
  tc_fence_before();
  if (splits > 1) cluster_sync_all();   // the peers' barriers are initialised before anything arrives on them
  else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();
  // tensor-parallel layers in the deferred form: the activations are complete once every peer has posted the previous gather
  if (g.tp_world > 1) {
    tp_wait_posts(g.tp_flags, g.tp_world, g.tp_rank, g.status, g.tag, g.tp_wait_cycles);
    __syncthreads();
  }
  const uint16_t *const x = behind_wait(g.x);
  // The decomposition warps ask for their activations first.  The CTA's activations are gn x nvec vectors of 8 consecutive k, dealt to the 256 threads in one run (a warp's vectors belong to one token).
  const int t2 = threadIdx.x - 64, nvec = nloc * 32, items = gn * nvec;
  uint4 xq[NI];
  auto load_x = [&](int idx) {
    const int t = idx / nvec, v = idx - t * nvec;
    return ld16((const uint4 *)(x + (size_t)t * g.ldx + (size_t)c0 * 256) + v);
  };
  if (warp >= 2 && warp < 10) {
#pragma unroll
    for (int u = 0; u < NI; ++u) {
      const int idx = t2 + u * kDecompThreads;
      xq[u] = idx < items ? load_x(idx) : make_uint4(0, 0, 0, 0);
    }
  }

  const unsigned tag = g.tag;
  auto wait = [abort_flag, status_word, tag](uint64_t *bar, uint32_t parity, unsigned code) -> bool {
    if (mbar_try(bar, parity)) return true;   // the common case: no flag read, no clock read
    if (*abort_flag) return false;
    if (mbar_wait(bar, parity)) return true;
    *abort_flag = 1;
    atomicCAS(status_word, 0u, code | tag);
    return false;
  };

  // The ring's first fill, one stage per warp: a copy instruction is slow to issue (see request_stage).
  if (warp >= 8 && warp - 8 < early) request_stage(warp - 8);

  if (warp == 0) {
    // ---------------- producer: after the first fill, each stage as its slot comes free ----------------
    int requested = early;
    for (int it = early; it < total; ++it) {
      const int s = it % kStages;
      const bool okw = wait(&empty[s], ((it / kStages) & 1) ^ 1, kStWaitEmpty);
      if (!__all_sync(0xFFFFFFFFu, okw)) break;
      request_stage(it);
      requested = it + 1;
    }
    // No copy may be in flight when the CTA leaves.  On the normal path every fill has long been consumed and these waits return
    // at once; after a wait somewhere gave up they hold the CTA (bounded) until the last requested fill of every stage has landed.
    for (int it = requested - 1; it >= 0 && it >= requested - kStages; --it) mbar_wait(&full[it % kStages], (it / kStages) & 1);
  } else if (warp == 1) {
    // ---------------- MMA issuer: D[piece][weight row] += pieces (A, M = 128) x weights (B, N = 256) ----------------
    // The whole warp runs the loop and one elected lane issues: from inside a one-lane branch every tcgen05 instruction costs the
    // warp about 150 cycles, and a chunk needs twelve of them (eight scale-tile copies, four MMAs).
    constexpr uint32_t idesc = idesc_mxf4nvf4(128, kRows);
    const uint32_t sfa_tmem = tmem_base + 256;
    tmem_cp_32x128b_warpx4_elect(sfa_tmem, smem_desc_sf(smem_u32(unit_sf)));
    if (__all_sync(0xFFFFFFFFu, wait(pieces_ready, 0, kStWaitPieces)) && !*inexact) {   // (the CUDA cores consume the ring otherwise)
      tc_fence_after();
      bool ok = true;
      const uint64_t da0 = smem_desc_sw128(smem_u32(pieces));
      int it = 0;
      for (int ti = 0; ti < my_tiles && ok; ++ti) {
        ok = __all_sync(0xFFFFFFFFu, wait(acc_empty, (ti & 1) ^ 1, kStWaitAccFree));
        if (!ok) break;
        tc_fence_after();
        for (int cl = 0; cl < nloc; ++cl, ++it) {
          const int s = it % kStages;
          ok = __all_sync(0xFFFFFFFFu, wait(&sf_ready[s], (it / kStages) & 1, kStWaitRetile) && wait(&full[s], (it / kStages) & 1, kStWaitFull));
          if (!ok) break;
          tc_fence_after();
          const uint32_t sW = smem_u32(stages + (size_t)s * stage_bytes), sSf = sW + kDataBytes;
          const uint32_t sfb_tmem = tmem_base + 272 + 32 * s;
          const uint64_t da = da0 + (uint32_t)(cl * (PR * 128 >> 4)), db = smem_desc_sw128(sW);
          const uint64_t sf0 = smem_desc_sf(sSf), sf1 = smem_desc_sf(sSf + 2048);
#pragma unroll
          for (int j = 0; j < 4; ++j)   // descriptors advance in 16-byte units: 32 bytes along the operand rows, 512 bytes per scale tile
            cp2_mma_mxf4nvf4_elect(sfb_tmem + 8 * j, sf0 + 32 * j, sf1 + 32 * j, tmem_base, da + 2 * j, db + 2 * j, idesc, sfa_tmem, (uint32_t)((cl | j) != 0));
          tc_commit_elect(&empty[s]);
        }
        if (ok) tc_commit_elect(acc_full);
      }
    }
  } else if (warp >= 10) {
    // ---------------- block scales: signs, and linear ones [256 rows][16 bytes] -> the stage's eight 512-byte tiles ----------------
    // The tensor cores take block scales as unsigned: a negative code's sign is moved into the block's sixteen weights.
    // A stage belongs to one warp for the whole launch: a wait on the parity of fill f is only meaningful to a thread that
    // has seen fill f - 1 complete (on a barrier still in its first phase, a wait for the second fill's parity returns at once).
    // (Only once the verdict on the activations is in: the CUDA-core consumer reads the stages as they came, and nobody waits for these warps then.)
    if (__all_sync(0xFFFFFFFFu, wait(pieces_ready, 0, kStWaitPieces)) && !*inexact) {
      for (int it = 0; it < total; ++it) {
        const int s = it % kStages;
        if ((s & 3) != warp - 10) continue;
        if (!__all_sync(0xFFFFFFFFu, wait(&full[s], (it / kStages) & 1, kStWaitRetile))) break;
        uint8_t *st = stages + (size_t)s * stage_bytes;
        const uint8_t *raw = st + kStageBytes;
        uint8_t *sf = st + kDataBytes + lane * 16;   // word q of tile (h, j): blocks 4 j .. 4 j + 3 of row 128 h + 32 q + lane
        uint32_t any = 0;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint4 w;
            if (linear) {
              uint32_t wd[4];
#pragma unroll
              for (int q = 0; q < 4; ++q) wd[q] = *(const uint32_t *)(raw + (h * 128 + 32 * q + lane) * 16 + 4 * j);
              w = make_uint4(wd[0], wd[1], wd[2], wd[3]);
              *(uint4 *)(sf + h * 2048 + j * 512) = w;
            } else {
              w = *(const uint4 *)(sf + h * 2048 + j * 512);
            }
            any |= w.x | w.y | w.z | w.w;
          }
        const bool negative = __any_sync(0xFFFFFFFFu, any & 0x80808080u);
        if (negative) move_signs(st, sf, lane);
        if (linear || negative) fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sf_ready[s]);
      }
    }
  } else {
    // ---------------- 8 warps: activations -> FP4 pieces in shared memory, then the epilogue of every tile ----------------
    // Loops that run once per token or vector are NOT unrolled from here on: the code is cold in every launch, and fetching it cost eight
    // tokens five microseconds more than one (1024 x 1024, four CTAs per cluster: 10.1 against 4.9 us).
#pragma unroll
    for (int u = 0; u < NI; ++u) {
      const int idx = t2 + u * kDecompThreads;
      if (idx >= items) break;
      uint32_t a = bf16x8_max(xq[u]);
      a = __reduce_max_sync(0xFFFFFFFFu, a);
      if (lane == 0) atomicMax(&wmax[idx / nvec], a);
    }
    named_barrier(2, kDecompThreads);
    auto eb_of = [&](int t) { return max((int)(wmax[t] >> 7), kPlaneMinExp); };   // biased exponent the token's pieces refer to
    uint32_t lost = 0;
#pragma unroll 1
    for (int u = 0; u < NI; ++u) {
      const int idx = t2 + u * kDecompThreads;
      if (idx >= items) break;
      uint4 x = xq[0];   // (selects, not a reload: from L2 it cost each turn its latency)
#pragma unroll
      for (int q = 1; q < NI; ++q)
        if (u == q) x = xq[q];
      const int t = idx / nvec, v = idx - t * nvec;
      const int eb = eb_of(t);
      if (eb == 255) lost = 1;   // Inf or NaN: IEEE arithmetic on the CUDA cores gives each output its own Inf or NaN
      uint32_t word[16];
      planes_of_8(x, pow2f(158 - eb), word);
      lost |= planes_lost_bits(x, eb);
      store_planes(pieces + (size_t)(v >> 5) * (PR * 128) + t * 2048, (v & 31) * 4, word);
    }
    if (lost) *inexact = 1;
    fence_proxy_async_smem();
    named_barrier(3, kDecompThreads);   // every warp's verdict is in
    if (lane == 0) mbar_arrive(pieces_ready);
    const bool exact = *inexact == 0;
    if (!exact) {
      // Some element lies more than 2^24 below its token's largest, so its low bits (or all of it) would be dropped -- far below
      // the FP32 accumulation bound unless the large elements meet zero weights.  Then the tensor cores sit this CTA out: the
      // eight warps consume the ring themselves, one thread per weight row, decoding nibbles and block scales from the stages
      // and accumulating in FP32 against the activations (kept as FP32 in the pieces' memory).  Several times slower; rare.
      float *xs = (float *)pieces;   // [token][k of this CTA]
#pragma unroll 1
      for (int idx = t2; idx < items; idx += kDecompThreads) {
        const uint4 x = load_x(idx);
        const uint32_t w[4] = {x.x, x.y, x.z, x.w};
        float *dst = xs + (size_t)idx * 8;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          dst[2 * i] = __uint_as_float(w[i] << 16);
          dst[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
        }
      }
    }

    const int rows_per = kRows / (int)splits, quad = warp & 3, half = warp >= 6 ? 1 : 0;
    const bool reader = quad < kQuads;
    const int dlo = lane >> 2;
    const float flo = pow2f(2 * dlo), fhi = pow2f(2 * dlo + 16);
    const int fr = t2 % rows_per, ft = t2 / rows_per;   // the epilogue's row of this thread, its first token
    // (A wait that gave up leaves no warp out of the loop: the barriers among the eight below need them all.  The CTA's waits return at
    // once from then on, and what it computes does not matter any more.)
    for (int ti = 0; ti < my_tiles; ++ti) {
      bool ok = true;
      const int tm = tile_first + ti * tile_step, buf = g.buffers == 2 ? ti & 1 : 0;
      float *const slot = res + (size_t)buf * NTOK * 256 + (size_t)rank * NTOK * rows_per;   // (at the owner) this rank's partial sums
      // every warp is done with the previous tile's results: its arrivals below let the peers overwrite the buffer before that one
      named_barrier(3, kDecompThreads);
      const int ei = tm * 256 + (int)rank * rows_per + fr;
      const bool row_ok = ei < gm;
      const float e_rowp = row_ok ? epi_row_part(g.e, ei) : 0.f;   // in flight while the tile streams
      const float e_bias = (row_ok && g.e.bias) ? load_dense(g.e.bias_dtype, g.e.bias, ei) : 0.f;
      if (exact) {
        if (reader) {
          // A thread of the 16 x 256-bit load holds pieces d and d + 8 (d = lane / 4) of sixteen weight rows; it joins the two, and a
          // butterfly that halves the rows a thread keeps (8 + 4 + 2 exchanges) leaves rows 2 lane and 2 lane + 1 of 64 in each thread.
          ok = __all_sync(0xFFFFFFFFu, wait(acc_full, ti & 1, kStWaitAcc));
          tc_fence_after();
          const int ntq = min(gn - 2 * quad, 2);   // tokens in this quadrant's lanes
          uint32_t nans = 0;   // this lane's sums that are not numbers, two per turn
#pragma unroll 1
          for (int tq = 0; tq < 2 * ntq; ++tq) {     // 64 columns of one token per turn
            const int tok = 2 * quad + (tq >> 1), q = tq & 1;
            uint32_t r[32];
            tmem_ld_16x256b_x8(tmem_base + ((uint32_t)(16 * tok) << 16) + half * 128 + q * 64, r);
            const int ex = eb_of(tok) - 157, e1 = max(ex, -100);
            const float s1 = pow2f(e1), s2 = pow2f(ex - e1);
            tmem_ld_wait32(r);
            float v[16];
#pragma unroll
            for (int i = 0; i < 16; ++i)
              v[i] = __fmaf_rn(__uint_as_float(r[4 * (i >> 1) + 2 + (i & 1)]), fhi, __fmul_rn(__uint_as_float(r[4 * (i >> 1) + (i & 1)]), flo));
#pragma unroll
            for (int st = 0; st < 3; ++st) {
              const int o = 16 >> st, keep = 8 >> st;   // exchange with lane ^ o, keep that many values
              const bool up = (lane & o) != 0;
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                if (i < keep) {
                  const float got = __shfl_xor_sync(0xFFFFFFFFu, up ? v[i] : v[i + keep], o);
                  v[i] = __fadd_rn(up ? v[i + keep] : v[i], got);
                }
              }
            }
            const int row = half * 128 + q * 64 + 2 * lane, owner = row / rows_per;
            float *d = slot + tok * rows_per + row % rows_per;
            st_peer_f32(d, owner, __fmul_rn(__fmul_rn(v[0], s1), s2));
            st_peer_f32(d + 1, owner, __fmul_rn(__fmul_rn(v[1], s1), s2));
            nans |= (uint32_t)(v[0] != v[0]) << (2 * tq) | (uint32_t)(v[1] != v[1]) << (2 * tq + 1);
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(acc_empty);   // the MMA warp may start the next tile
          if (nans) {
            for (int b = 0; b < 8; ++b) {
              const int tok = 2 * quad + (b >> 2), row = half * 128 + ((b >> 1) & 1) * 64 + 2 * lane + (b & 1), i = tm * 256 + row;
              if ((nans >> b & 1u) && i < gm)
                st_peer_f32(slot + tok * rows_per + row % rows_per, row / rows_per, code_7f_sum(g.A, x + (size_t)tok * g.ldx, i, 16 * c0, 16 * c1));
            }
          }
        }
      } else {
        float acc[NTOK];
#pragma unroll
        for (int t = 0; t < NTOK; ++t) acc[t] = 0.f;
        const int r = t2;
        const float *const xs = (const float *)pieces;
        for (int cl = 0; cl < nloc; ++cl) {
          const int it = ti * nloc + cl, s = it % kStages;
          ok = __all_sync(0xFFFFFFFFu, wait(&full[s], (it / kStages) & 1, kStWaitFull));
          if (!ok) break;
          const uint8_t *st = stages + (size_t)s * stage_bytes;
          const uint8_t *rowp = st + (r >> 3) * 1024 + (r & 7) * 128;
          const uint8_t *sfp = linear ? st + kStageBytes + r * 16 : st + kDataBytes + (r >> 7) * 2048 + (r & 31) * 16 + ((r & 127) >> 5) * 4;
#pragma unroll 2
          for (int u16 = 0; u16 < 8; ++u16) {
            const uint4 q = *(const uint4 *)(rowp + ((u16 ^ (r & 7)) << 4));
            const uint32_t wd[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int b = 0; b < 2; ++b) {
              const int jj = 2 * u16 + b;   // block of 16 values within the chunk
              const float sc = __fmul_rn(e4m3_to_f32(linear ? sfp[jj] : sfp[(jj >> 2) * 512 + (jj & 3)]), 0.5f);
#pragma unroll
              for (int t = 0; t < NTOK; ++t) {
                if (t >= gn) break;
                const float *xv = xs + (size_t)t * nloc * 256 + (size_t)cl * 256 + jj * 16;
                float part = 0.f;
#pragma unroll
                for (int i = 0; i < 16; ++i)
                  part = __fmaf_rn((float)e2m1_x2((wd[2 * b + (i >> 3)] >> (4 * (i & 7))) & 0xFu), xv[i], part);
                acc[t] = __fmaf_rn(sc, part, acc[t]);
              }
            }
          }
          __threadfence_block();
          __syncwarp();
          // the eighth warp hands the stage back; the count is per stage because a warp may run several stages ahead of another,
          // but never a whole fill ahead on the same stage
          if (lane == 0 && (atomicAdd(&consumed[s], 1) & 7) == 7) mbar_arrive(&empty[s]);
        }
#pragma unroll
        for (int t = 0; t < NTOK; ++t) st_peer_f32(slot + t * rows_per + r % rows_per, r / rows_per, acc[t]);
        named_barrier(2, kDecompThreads);   // the readers' arrivals below stand for all eight warps' stores
      }
      if (reader) {   // tell every owner that this warp's partial sums are there
        __syncwarp();
        if (ok && lane < (int)splits) mbar_arrive_rank_release(&res_full[buf], lane);
      }

      // ---- this CTA's rows: the ranks' partial sums in rank order, then the epilogue, a thread per (row, token) ----
      {
        const uint32_t par = (g.buffers == 2 ? ti >> 1 : ti) & 1;
        ok = __all_sync(0xFFFFFFFFu, mbar_try_cluster(&res_full[buf], par) || (wait(&res_full[buf], par, kStWaitResults) && mbar_try_cluster(&res_full[buf], par)));
      }
      const Epilogue &e = g.e;
      const int mask = g.ex.mask;
      float *const mine = res + (size_t)buf * NTOK * 256;
      float amax = 0.f;
      const bool nb_needed = (mask & (kExSwiglu | kExOut2)) != 0;
      auto finish = [&](int tok, float val, const float *nb) {   // stores of one (row, token); nb: the values of the rows beside it
        if (mask & kExSwiglu) {
          if (row_ok && !(fr & 8)) {
            const float hh = silu_mul(val, nb[8]);
            store_dense(e.d_dtype, e.d, (size_t)tok * e.ldd + (ei >> 4) * 8 + (ei & 7), hh);
            amax = fmaxf(amax, fabsf(hh));
          }
        } else if (row_ok) {
          store_dense(e.d_dtype, e.d, (size_t)tok * e.ldd + ei, val);
          amax = fmaxf(amax, fabsf(val));
        }
        if ((mask & kExOut2) && row_ok) {
          store_dense(g.ex.d2_dtype, g.ex.d2, (size_t)tok * g.ex.ldd2 + ei, __fmul_rn(val, load_dense(g.ex.w2_dtype, g.ex.w2, ei)));
          if (!(fr & 15)) {
            float sq = 0.f;
#pragma unroll
            for (int r = 0; r < 16; ++r) sq = __fadd_rn(sq, __fmul_rn(nb[r], nb[r]));
            g.ex.sq[(size_t)tok * g.ex.ld_sq + (ei >> 4)] = sq;
          }
        }
      };
      const int last = ok ? gn : 0;   // (a wait that gave up: nothing is stored)
#pragma unroll 1
      for (int tok = ft; tok < last; tok += (int)splits) {   // (the same tokens for the whole warp)
        float acc = mine[(size_t)tok * rows_per + fr];
        for (uint32_t p = 1; p < splits; ++p) acc = __fadd_rn(acc, mine[((size_t)p * NTOK + tok) * rows_per + fr]);
        float colp = epi_col_part(e, tok);
        if (mask & kExNorm) colp = __fmul_rn(colp, warp_norm_scale(g.ex, tok, lane));
        float val = __fmul_rn(acc, epi_scale(e, e_rowp, colp));
        if (e.bias) val = __fadd_rn(val, e_bias);
        if (e.beta != 0.f && row_ok) val = __fmaf_rn(e.beta, load_dense(e.c_dtype, e.c, (size_t)tok * e.ldc + ei), val);
        if (nb_needed) mine[(size_t)tok * rows_per + fr] = row_ok ? val : 0.f;   // (in the place of the first rank's sum, which only this thread reads)
        else finish(tok, val, nullptr);
      }
      if (nb_needed) {
        named_barrier(2, kDecompThreads);
#pragma unroll 1
        for (int tok = ft; tok < last; tok += (int)splits) {
          const float *nb = mine + (size_t)tok * rows_per + fr;
          finish(tok, nb[0], nb);
        }
      }
      if (e.amax) warp_amax_commit(e.amax, amax);
    }
  }

  __syncwarp();
  tc_fence_before();
  __syncthreads();
  // A CTA whose waits all succeeded has received every peer's stores and arrivals of its last tile: nothing more comes to its shared
  // memory and it may leave.  After a wait that gave up, the CTAs that are still there (all that miss something) leave together.
  if (splits > 1 && *abort_flag) cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

}  // namespace

int gemv_fp4_pinned_splits();   // (gemv_fp4.cu) nvfp4a_b200_set_gemv_splits: 0 = automatic

// How a problem is cut: `splits` CTAs per cluster (a power of two, at most 8 and nk; every CTA's k range at most max_chunks), `clusters`
// clusters, each with `rounds` or one tile fewer.  Of a cluster size only so many clusters run at once (a cluster lies inside one GPC, a CTA
// takes an SM; 148, 74, 33 and 15 clusters of 1, 2, 4 and 8 by cudaOccupancyMaxActiveClusters): more are not launched, a cluster takes
// several tiles instead.  Automatic: the cut with the shortest estimate, fitted to CUDA-graph timings of 12 shapes from 1024 x 1024 to 28672 x
// 4096 and up to 8 vectors (within about 10 %): 4.4 us of set-up and tail (4.8 in a cluster), the stream (36 KiB per chunk at 61 GB/s
// per CTA or 5.4 TB/s in all), the pieces (0.14 us per chunk and vector past the first) and the tiles' ends, which clusters of eight pay most for.
// The pieces now take 0.11 us.  The estimate keeps 0.14: with 0.11 8192 x 8192 with six to eight vectors would come here (eight: 18.0 us, mma.sync 23.7),
// a middling gain for calls whose time would then depend on their data -- one activation outside the planes' range, and a CTA leaves the weights to
// its CUDA cores: 150 us there, 23.7 on the mma.sync GEMV.
struct GemvCut { int splits, clusters, rounds; double us; };
static int ntok_of(int n) { return n <= 4 ? 4 : 8; }   // tokens of the kernel instance
static GemvCut cut_for(int m, int k, int n, int splits) {
  const int nk = k >> 8, tiles = (m + kRows - 1) / kRows, sms = device_sms();
  const int nloc = (nk + splits - 1) / splits;
  if (splits > nk || nloc > max_chunks(ntok_of(n))) return {0, 0, 0, 0};
  const int cap = splits == 1 ? sms : splits == 2 ? sms / 2 : splits == 4 ? sms * 33 / 148 : sms * 15 / 148;
  const int rounds = (tiles + cap - 1) / cap, clusters = (tiles + rounds - 1) / rounds, ctas = clusters * splits;
  const double chunk = fmax(0.6, ctas * 36.9e3 / 5.4e6);
  const int more = ntok_of(n) - 1;
  return {splits, clusters, rounds, (splits > 1 ? 4.8 : 4.4) + (0.1 + 0.14 * nloc) * more + (0.06 * more + (splits == 8 ? 1.2 : 0.05)) * (rounds - 1) + rounds * nloc * chunk};
}
static GemvCut choose_cut(int m, int k, int n) {
  if (const int f = gemv_fp4_pinned_splits()) return cut_for(m, k, n, f);   // pinned (nvfp4a_b200_set_gemv_splits): that value if the problem can use it
  GemvCut best = {0, 0, 0, 0};
  for (int s = 1; s <= 8; s *= 2) {
    const GemvCut c = cut_for(m, k, n, s);
    if (c.splits && (!best.splits || c.us < best.us)) best = c;
  }
  // The mma.sync GEMV has less to set up and takes 3 us and 0.4 us per megabyte (same timings): it keeps small matrices, and middling ones
  // as the number of vectors grows (28672 x 4096: 30.6 against 20.1 us for four vectors, 33.6 against 22.8 us for eight; 8192 x 8192: 19.8
  // against 14.6 for four, which come here, 23.7 against 18.0 for eight, which do not; 4096 x 14336: 17.7 against 16.9 and 18.5 against 23.7; 4096 x 4096, eight: 7.6 against 10.8).
  if (best.us > 3.0 + 0.405 * (m * (k * 0.5625e-6)) * (1.0 + 0.012 * (n - 1))) best.splits = 0;
  return best;
}

bool gemv_fp4_n8_supports(const GemmArgs &g) {
  if (!(g.n >= 3 && g.n <= 8 && g.B.dtype == NVFP4A_BF16 && !g.A.ue && g.k >= 256 && g.k % 256 == 0)) return false;
  if (((uintptr_t)g.B.data & 15) || g.B.ld % 8) return false;
  // plain operands: scales in aligned 512-byte tiles (the swizzled layout), or linear with a 16-byte aligned base and pitch (TMA)
  if (!g.A.image && (((uintptr_t)g.A.data & 15) || g.A.ld % 32 || ((uintptr_t)g.A.sc & 15) || (g.A.sld > 0 && g.A.sld % 16))) return false;
  return choose_cut(g.m, g.k, g.n).splits > 0;
}

cudaError_t launch_gemv_fp4_n8(const GemmArgs &g, cudaStream_t s) {
  GemvN8Args a;
  memset(&a, 0, sizeof a);
  a.m = g.m; a.n = g.n; a.k = g.k;
  a.x = (const uint16_t *)g.B.data; a.ldx = g.B.ld;
  a.e = g.e; a.ex = g.x;
  a.status = kernel_status_device_ptr();
  a.tag = next_launch_tag();
  if (g.tp.world > 1 && (g.tp.deferred & 1)) {
    a.tp_world = g.tp.world; a.tp_rank = g.tp.rank; a.tp_wait_cycles = tp_wait_limit();
    for (int p = 0; p < g.tp.world; ++p) a.tp_flags[p] = g.tp.flags[p];
  }
  a.ktiles = (g.k + kImgK - 1) / kImgK;
  a.a_image = g.A.image;
  a.A = g.A;
  CUtensorMap ta, ts;
  memset(&ts, 0, sizeof ts);
  if (g.A.image) {
    if (!make_tmap_image_pair(&ta, g.A.data, 128, (uint64_t)a.ktiles, (uint64_t)((g.m + 127) / 128))) return cudaErrorInvalidValue;
    if (!make_tmap_image_pair(&ts, (const uint8_t *)g.A.data + kImgDataBytes, 16, (uint64_t)a.ktiles, (uint64_t)((g.m + 127) / 128))) return cudaErrorInvalidValue;
    a.sa = g.A.data;
  } else {
    if (!make_tmap_bytes(&ta, g.A.data, (uint64_t)g.k / 2, (uint64_t)g.m, (uint64_t)g.A.ld / 2, kRows)) return cudaErrorInvalidValue;
    a.sa = g.A.sc; a.sa_ld = g.A.sld;
    a.linear = g.A.sld > 0;
    if (a.linear && !make_tmap_dense(&ts, g.A.sc, 4, (uint64_t)g.k / 64, (uint64_t)g.m, (uint64_t)g.A.sld, 4, kRows)) return cudaErrorInvalidValue;
  }
  const GemvCut cut = choose_cut(g.m, g.k, g.n);
  const int splits = cut.splits, ntok = ntok_of(g.n);
  if (splits <= 0) return cudaErrorInvalidValue;
  void (*kern)(CUtensorMap, CUtensorMap, GemvN8Args) = ntok == 4 ? gemv_fp4_n8_kernel<4> : gemv_fp4_n8_kernel<8>;
  static std::atomic<bool> attr_set[64][2];   // zero-initialised; set once per device and kernel
  const int which = ntok == 8;
  int dev = 0;
  cudaGetDevice(&dev);
  const int nk = g.k >> 8, nloc_max = (nk + splits - 1) / splits;
  a.tiles = (g.m + kRows - 1) / kRows;
  a.buffers = cut.rounds > 1 ? 2 : 1;
  a.piece_bytes = nloc_max * 16 * ntok * 128;
  const int stage_bytes = kStageBytes + (a.linear ? kRawSfBytes : 0);
  a.stages = (kSmemLimit - a.piece_bytes - fixed_bytes(ntok, a.buffers)) / stage_bytes;
  if (a.stages > kMaxStages) a.stages = kMaxStages;
  if (a.stages < 2) return cudaErrorInvalidValue;
  const int smem_bytes = 1024 + a.piece_bytes + a.stages * stage_bytes + fixed_bytes(ntok, a.buffers);
  if (!attr_set[dev & 63][which]) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit + 1024);
    if (e != cudaSuccess) return e;
    attr_set[dev & 63][which] = true;
  }
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof cfg);
  cfg.gridDim = dim3(splits, cut.clusters, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = smem_bytes;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = splits; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // the kernel's set-up overlaps the previous kernel's tail
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = pdl_enabled() ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, ta, ts, a);
}

}  // namespace nvb

