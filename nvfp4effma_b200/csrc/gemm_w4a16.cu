// NVFP4 weights x BF16 activations (W4A16) GEMM on the 5th-generation tensor cores: tcgen05.mma kind::f16 (BF16 in, FP32
// accumulators in tensor memory) on weights expanded to exact BF16 in tensor memory.
//
// An NVFP4 value times its block scale has at most 2 + 4 significant bits, so e2m1 * scale is exact in BF16; the tensor
// cores then form exact products with the BF16 activations and accumulate in FP32 -- the reference's "exact" W4A16
// definition (include/nvfp4effma.h:82-92 there) up to the order of the FP32 additions, like its own tensor-core path.
//
// CTA pairs (tcgen05.mma.cta_group::2): a tile is 256 weight rows (MMA M, 128 per CTA) x up to 256 tokens (MMA N, half of them in
// each CTA's shared memory), a stage covers 64 values of k.  The expanded weights are the MMA's A operand IN TENSOR MEMORY: an
// expansion thread owns a weight row = a tensor memory lane and writes its 64 values with two tcgen05.st, so that the expansion costs
// no shared-memory traffic, no swizzled addressing and no proxy fence, and shared memory is left to the activations (read once per
// pair and stage).  Tensor memory: columns [0, 256) one accumulator of 256 columns or two of 128, [256, 512) eight weight stages (grouped: a
// third accumulator of 128 columns, then four stages).
// Roles, 20 warps per CTA:
//   warp 0      TMA producer of the activations: this CTA's half of the tile's tokens (no multicast); the bytes of both CTAs are
//               counted on the even CTA's barrier
//   warp 1      MMA issuer (even CTA; 8 or 12 x K16 per unit of work, one elected lane), owner of the tensor memory
//   warp 2      TMA producer of the weight nibbles: [128 rows][128 bytes] = 256 values of k per slot, so that the expansion
//               reads shared memory and never waits for a trip to L2
//   warps 4-11  epilogue (144 registers each, taken from the others by setmaxnreg), one 32-lane quadrant and one half of the columns
//               each: the accumulator block goes into registers at once and back to the MMA warp before any arithmetic; then
//               plain or extended epilogue (RMSNorm column scale, SwiGLU, second output + sums of squares), D through
//               shared-memory staging tiles and TMA stores when its layout allows
//   warps 12-19 weight expansion, two groups of four warps on alternate pairs of stages.  The eight magnitudes of E2M1 times a block scale
//               are eight 16-bit floats (exact: 2 x 4 significant bits); for BF16 a 4 KiB table holds their high and low bytes for each of
//               the 256 scale codes, so a block costs one 16-byte table read and four values cost three byte permutes (the packed
//               nibbles ARE the permute's selectors: high bytes, low bytes, signs), two of them again to interleave, and two
//               logical operations -- 2 instructions per value where shifts, masks, the multiply and reordering took 3.  (FP16: see below.)
// Instruction issue, not the tensor pipe, bounded the former kernel (a thread-per-row expansion through shared memory with a proxy
// fence per stage: 1240 cycles per stage of 512 cycles of MMAs, 41 % of the tensor pipe).
// The last round of tiles over the SM pairs is cut along the tokens, or into parts of k (see choose_tail), when it would leave pairs idle, and a tile at the end of the
// tokens is only as wide (in steps of 64) as the tokens left.
// Every wait is bounded; a wait that gives up raises the CTA's abort flag and the kernel status word.
//
// FP16 activations (F16): e2m1 x E4M3 is a multiple of 2^-10 up to 2880 with at most 6 significant bits, exact in FP16, so the same
// kernel runs on FP16 operands.  FP16 weights come from the hardware's conversions of E2M1 pairs and one packed multiply by the block's scale, both exact: 1.4
// instructions per value and no table, whose sixteen-byte reads at 32 unrelated addresses also met in the banks (in a graph, FP16 4096 x 4096 on 700 tokens 45.8 -> 41.6 us,
// 3584 x 3584 on 1500 61 -> 56, 4864 x 6208 on 600 70 -> 57; INT8, whose first pass runs on them too and which the MMAs bound, 6144 x 4096 on 1000 80.6 -> 79.5).
//
// Segments.  The tensor cores truncate the running sum at every instruction, so that one chain over all of k drifts towards zero: at k = 4096 its
// error against 64 bits is 1.3e-6 (BF16 / FP16 activations) and 9.9e-6 (INT8, three chains in one) where the ordered FP32 sums of the
// CUDA-core kernels have 2.2e-7 and 2.9e-7.  The calls that those kernels would take otherwise -- FP16 activations, INT8 groups -- are therefore
// summed in segments: 4 stages (256 values of k) go into one of two accumulators, the epilogue warps add each to running FP32 sums in
// their registers (64 per thread: tiles of at most 128 tokens) while the next one fills, and INT8's two small planes, whose drift does
// not matter, have an accumulator of their own for all of k.  Error: 1.05e-7 and 9.8e-8 at k = 4096 (normal data; 2.9e-7 and 1.4e-7 against
// 6.9e-7 and 2.9e-7 with activations spread over ten binades).  Below k = 1024 segments are 2 stages, below 512 one (INT8 at k = 512:
// 6.2e-8 against 1.08e-7; FP16 at k = 512, 128 and 64: 6.3e-8, 4.2e-8 and 4.0e-8 against 6.9e-8, 4.1e-8 and 3.7e-8).
// 8 experts of 2048 x 4096 on 1100 tokens take 94 us, FP16 4096 x 4096 on 333 tokens 31; the CUDA-core kernels 602 and 1932 us.
//
// Grouped (mixture of experts): A stacks the weights of all groups, a group owns the tokens [seg[q], seg[q + 1]); the CTAs read seg
// (device memory) into a table of tile counts and find a tile's group there.  (INT8 activations only, plain epilogue, 16-bit D.)
//
// INT8 activations (W4A8, FP32 scale s_b per 16 values) run on the same kernel as planes [token][5 or 3][k] that small kernels make first.
// PLANES = 2 (one weight): x = q * s_b is t1 + t2, two FP16 terms of 11 bits each, on a grid that puts the token's largest below 2^15 (the epilogue
// takes that power of two back).  t2 is the exact remainder's rounding: together they are x to within 2^-23 of it, or 2^-25 on the grid, which the
// (k + 2) 2^-24 of the accumulation bound covers for every value while a token's scales lie within 2^12 of each other.  A token whose scales do not, or
// are not near enough to one for the grid's power of two to be a float, is three BF16 planes instead, t1 + t2 + t3 = fl(q * s_b) exactly (8 + 8 + 8 bits),
// and so are all tokens where the weights' scales are UE5M3 (products leave FP16's range).  In the planes of the other kind a token is zero: a tile with
// tokens of both kinds goes over k twice, on the same accumulator, and no token's result depends on its neighbours.  One chain in the
// tensor cores, 2-norm error at k = 512 / 1024 / 4096 / 8192: 0.97e-6, 1.9e-6, 8.2e-6, 1.69e-5 (three planes: 1.4e-6, 2.6e-6, 9.9e-6, 1.91e-5).
// Scales 2^0 / 2^6 / 2^12 apart, k = 1024: 1.82e-6, 2.25e-6, 2.47e-6 (three planes: 2.60e-6, 2.74e-6, 2.85e-6).
// 6144 x 4096 on 1000 tokens 125 us with three planes and an MMA issue per plane, 93 with two, 76 with what followed; 124 with one token of BF16 planes.
// PLANES = 3 (grouped): always three BF16 planes, the last two in an accumulator of their own (see Segments).  Two FP16 planes would be 94 us instead of 96
// (8 experts of 2048 x 4096 on 1100 tokens), but 11-bit terms lose more to the truncation in the tensor cores than 8-bit ones, whose sums stay
// on a coarse grid: 1.6e-7 instead of 0.74e-7 at k = 4096.
#include <atomic>
#include <cuda_bf16.h>
#include "operands.cuh"
#include "sm100.cuh"

namespace nvb {

using namespace sm100;

namespace {

struct W4A16Args {
  int m, n, k;
  Fp4Operand A;
  Epilogue e;
  EpilogueEx x;
  unsigned *status;
  unsigned tag;  // this launch's tag in the status word
  int d_tma;     // the output goes through the staging tiles and TMA stores (SwiGLU: 64 output rows per tile)
  int width;     // tokens per tile: 64, 128, 192 or 256
  int nfull, cut;   // tiles 0 .. nfull - 1 are `width` tokens wide; the rest (to `tiles`) are parts of width / cut tokens
  int tiles;
  int seg_stages;   // F16, GROUPED: stages per segment of k
  int unit;         // stages per unit: 1 or 2 (see the MMA issuer)
  const int *seg; int groups;   // GROUPED: m is the rows of ONE group's weight, n the bound on seg[groups]
  // kEpiPart, kEpiTail: the tiles from nfull on take k in `parts` runs of part_stages stages, each one's sums in partial [tile - nfull][part][width tokens][256 rows]
  int parts, part_stages; float *partial;
  const float *tscale;          // PLANES = 2: what each token's sums are multiplied by; word n: 0 all tokens are two FP16 planes, 1 some, 2 none; behind it
                                // a byte per token, non-zero for three BF16 planes
};

// tensor maps of D in the peers' buffers (tensor-parallel all-gather fused into the epilogue's TMA stores); n = 0: none
struct alignas(64) PeerMaps {
  CUtensorMap map[kMaxRanks - 1];
  int n;
};

template <int PLANES, bool GROUPED>
struct Cfg {
  // PLANES = 1: the weight and the activation ring advance together and share their `empty` barriers (one commit per stage)
  static constexpr int kA = PLANES == 3 ? 4 : 8, kB = 8, kRaw = 3;
  static constexpr int kACols = 512 - 32 * kA;   // first tensor memory column of the weight stages (32 columns each)
  static constexpr int kBBytes = 128 * 128, kRawBytes = 128 * 128, kStagingBytes = 8192;
  static constexpr int kSmemBytes = 1024 + kB * kBBytes + kRaw * kRawBytes + 4 * kStagingBytes + 4096 /* expansion table */ + 256 * 4 /* column scales */ +
                                    512 /* barriers */ + 2 * 257 * 4 + 8 /* groups */;
};
static_assert(Cfg<1, false>::kSmemBytes <= 232448 && Cfg<2, false>::kSmemBytes <= 232448, "shared memory budget");
constexpr int kSegmentWidth = 128;   // tokens per tile where k is summed in segments: the running sums have to fit the epilogue's registers

constexpr int kThreads = 640, kRegsRest = 48, kRegsEpi = 144, kRegsConv = 72;
static_assert(128 * kRegsRest + 256 * kRegsEpi + 256 * kRegsConv <= kThreads * 96, "the split draws on the registers of the launch: 96 per thread");
constexpr unsigned kStWaitFullA = 0x301, kStWaitFullB = 0x302, kStWaitEmpty = 0x303, kStWaitTmemFull = 0x304, kStWaitTmemEmpty = 0x305,
                   kStWaitConv = 0x306, kStWaitRaw = 0x307;

__device__ __forceinline__ uint32_t h2mul(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t bf16x2_rn(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}
// four 8 x 8 blocks of 16-bit values in MMA fragment layout, each stored transposed: lane 8 q + j gives the address of row j (16 bytes,
// the fragment's column j) of block q
__device__ __forceinline__ void stmatrix_x4_trans(void *row, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(smem_u32(row)), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// Four MMAs (K = 16 each: 8 tensor memory columns of A, 32 bytes along B's 128-byte rows) over a CTA pair, twice, and the commit that hands the
// slots back in both CTAs, in one statement issued by one elected lane of a converged warp.
__device__ __forceinline__ void mma8_f16_commit_pair_elect(uint32_t d0, uint32_t a0, uint64_t b0, uint32_t acc0, uint32_t d1, uint32_t a1, uint64_t b1, uint32_t acc1,
                                                           uint32_t idesc, uint64_t *bar) {
  asm volatile("{\n\t.reg .pred p, u, q, t;\n\tsetp.ne.b32 p, %3, 0;\n\tsetp.ne.b32 u, %7, 0;\n\tsetp.eq.u32 t, %8, %8;\n\telect.sync _|q, 0xFFFFFFFF;\n\t"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %8, p;\n\t"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%9], %10, %8, t;\n\t"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%11], %12, %8, t;\n\t"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%13], %14, %8, t;\n\t"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%4], [%5], %6, %8, u;\n\t"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%4], [%15], %16, %8, t;\n\t"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%4], [%17], %18, %8, t;\n\t"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%4], [%19], %20, %8, t;\n\t"
               "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%21], %22;\n\t}"
               ::"r"(d0), "r"(a0), "l"(b0), "r"(acc0), "r"(d1), "r"(a1), "l"(b1), "r"(acc1), "r"(idesc), "r"(a0 + 8), "l"(b0 + 2), "r"(a0 + 16), "l"(b0 + 4),
                 "r"(a0 + 24), "l"(b0 + 6), "r"(a1 + 8), "l"(b1 + 2), "r"(a1 + 16), "l"(b1 + 4), "r"(a1 + 24), "l"(b1 + 6), "r"(smem_u32(bar)), "h"((uint16_t)3)
               : "memory");
}
__device__ __forceinline__ void mma4_f16_commit_pair_elect(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate,
                                                           uint64_t *bar) {
  asm volatile("{\n\t.reg .pred p, q, t;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.eq.u32 t, %3, %3;\n\telect.sync _|q, 0xFFFFFFFF;\n\t"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%5], %6, %3, t;\n\t"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%7], %8, %3, t;\n\t"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%9], %10, %3, t;\n\t"
               "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%11], %12;\n\t}"
               ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(a_tmem + 8), "l"(b_desc + 2), "r"(a_tmem + 16), "l"(b_desc + 4),
                 "r"(a_tmem + 24), "l"(b_desc + 6), "r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}

// one weight stage against three planes: the first into d0, the others into d1
__device__ __forceinline__ void mma12_f16_commit_pair_elect(uint32_t d0, uint32_t a, uint64_t b0, uint32_t acc0, uint32_t d1, uint64_t b1, uint32_t acc1, uint64_t b2,
                                                            uint32_t idesc, uint64_t *bar) {
  asm volatile("{\n\t.reg .pred p, u, q, t;\n\tsetp.ne.b32 p, %3, 0;\n\tsetp.ne.b32 u, %6, 0;\n\tsetp.eq.u32 t, %8, %8;\n\telect.sync _|q, 0xFFFFFFFF;\n\t"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %8, p;\n\t"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%9], %12, %8, t;\n\t"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%10], %13, %8, t;\n\t"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%11], %14, %8, t;\n\t"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%4], [%1], %5, %8, u;\n\t"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%4], [%9], %15, %8, t;\n\t"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%4], [%10], %16, %8, t;\n\t"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%4], [%11], %17, %8, t;\n\t"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%4], [%1], %7, %8, t;\n\t"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%4], [%9], %18, %8, t;\n\t"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%4], [%10], %19, %8, t;\n\t"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%4], [%11], %20, %8, t;\n\t"
               "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%21], %22;\n\t}"
               ::"r"(d0), "r"(a), "l"(b0), "r"(acc0), "r"(d1), "l"(b1), "r"(acc1), "l"(b2), "r"(idesc), "r"(a + 8), "r"(a + 16), "r"(a + 24), "l"(b0 + 2), "l"(b0 + 4),
                 "l"(b0 + 6), "l"(b1 + 2), "l"(b1 + 4), "l"(b1 + 6), "l"(b2 + 2), "l"(b2 + 4), "l"(b2 + 6), "r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}

// A tile of the schedule: 128-row tiles 2 * tm and 2 * tm + 1 (one per CTA of the pair) against the tokens [j0, j0 + width), of which
// those below jend exist (width: a multiple of 64; 0: nothing to do).  Grouped: ro = the group's first row in the stacked weights.
// A part of k: the stages [k0, k0 + nk), `unit` its place in the partial sums; -1: a whole tile.
struct Tile { int tm, j0, jend, width, ro, unit, k0, nk; };
constexpr int kMaxGroups = 256;

// EPI: what the epilogue is compiled for.  0: everything; 1: a 16-bit D, alpha, globals and bias; 2: the same and SwiGLU.  The whole of it is 150 KiB of code in
// which a plain call's instructions lie far apart: fetching them made a chunk of 32 columns take 5000 cycles, in which the tensor cores wait for the
// accumulator or, at the end, the caller for the result.  28672 x 4096 with SwiGLU on 2048 tokens: 412 -> 344 us; FP16 4096 x 4096 on 333
// tokens 37.5 -> 35.2; 5504 x 3584 with SwiGLU on 121 tokens 32.1 -> 27.0.
// 3: no epilogue, the sums of a part of k as they are (see w4a16_join_kernel); 8: as 1 for whole tiles, as 3 for the parts of the last ones; 9: the same with everything
// for the whole ones (a row's sums are cut the same way whatever is asked for beside them).
// 4 .. 7: a 16-bit D, at run time an amax, and one of: RMSNorm scale and SwiGLU (28672 x 4096 on 2048 tokens 400 -> 330 us, INT8 activations 679 -> 628); second
// output and sums of squares (4096 x 14336 214 -> 186); RMSNorm scale (6144 x 4096 103 -> 82; 4096 x 4096 on 100 tokens 30.3 -> 25.3); beta * C (131
// -> 126, 32.9 -> 30.5: its two-byte loads of C remain).
enum { kEpiAny = 0, kEpiPlain = 1, kEpiSwiglu = 2, kEpiPart = 3, kEpiNormGlu = 4, kEpiOut2 = 5, kEpiNorm = 6, kEpiAdd = 7, kEpiTail = 8, kEpiTailAny = 9 };
template <int PLANES, bool F16, bool GROUPED, int EPI>
__global__ void __launch_bounds__(kThreads, 1)
gemm_w4a16_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_b, const __grid_constant__ CUtensorMap tmap_d,
                  const __grid_constant__ PeerMaps peers, const W4A16Args g) {
  using C = Cfg<PLANES, GROUPED>;
  constexpr bool SEG = F16 || PLANES == 3;   // k is summed in segments: see the head of the file
  constexpr int kA = C::kA, kB = C::kB, kRaw = C::kRaw, kACols = C::kACols, kSmallCols = 256;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t *const sB = smem, *const sRaw = sB + kB * C::kBBytes, *const staging = sRaw + kRaw * C::kRawBytes;
  uint4 *lut = (uint4 *)(staging + 4 * C::kStagingBytes);           // scale code -> bytes of the eight products (see e2m1_expand4)
  float *colscale = (float *)(lut + 256);                           // RMSNorm column scales of the current token tile
  uint64_t *bars = (uint64_t *)(colscale + 256);
  uint64_t *a_full = bars, *b_full = a_full + kA, *b_empty = b_full + kB, *a_empty = PLANES == 1 ? b_empty : b_empty + kB,
           *raw_full = b_empty + kB + kA, *raw_empty = raw_full + kRaw, *tmem_full = raw_empty + kRaw, *tmem_empty = tmem_full + 2;
  uint32_t *tmem_slot = (uint32_t *)(tmem_empty + 2);
  volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
  int *gseg = (int *)((uint8_t *)bars + 512), *gcum = gseg + kMaxGroups + 1;   // GROUPED: seg, and the token tiles of the groups before each

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank();
  const int gm = g.m, gn = g.n, gk = g.k, seg_stages = SEG ? g.seg_stages : 0;
  const int unit = PLANES != 1 ? 1 : F16 ? g.unit : 2;   // stages per unit
  const int lgA = PLANES != 1 ? (kA == 8 ? 3 : 2) : unit == 2 ? 2 : 3, lgB = unit == 2 || PLANES != 1 ? 2 : 3;   // the rings' slots, as powers of two
  const int nA = 1 << lgA, nB = 1 << lgB, subA = kA >> lgA;
  constexpr int kSub = PLANES == 3 ? C::kBBytes / 2 : C::kBBytes;   // bytes of a stage of one plane (three planes: tiles of at most 128 tokens)
  const int slot_bytes = (kB * C::kBBytes) >> lgB;
  constexpr bool PART = EPI == kEpiPart, TAIL = EPI == kEpiTail || EPI == kEpiTailAny, CUT_K = PART || TAIL, ANY = EPI == kEpiAny || EPI == kEpiTailAny;
  constexpr bool AMAX = ANY || (EPI >= kEpiNormGlu && !TAIL), ADD = ANY || EPI == kEpiAdd;
  const int tile_first = blockIdx.x >> 1, tile_step = gridDim.x >> 1;
  const int tiles_m = (gm + 255) / 256, nk_all = gk / 64, nslots_all = (nk_all + 3) / 4;   // 256-row tiles
  const bool ue = g.A.ue != 0;
  unsigned *const status_word = g.status;

  // The set-up touches no global memory: under programmatic dependent launch it runs while the stream's previous kernel drains.
  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int s = 0; s < kA; ++s) mbar_init(&a_full[s], 8);   // the unit's four expansion warps of both CTAs
    if (PLANES != 1) for (int s = 0; s < kA; ++s) mbar_init(&a_empty[s], 1);
    for (int s = 0; s < kB; ++s) { mbar_init(&b_full[s], 1); mbar_init(&b_empty[s], 1); }
    for (int s = 0; s < kRaw; ++s) { mbar_init(&raw_full[s], 1); mbar_init(&raw_empty[s], 8); }
    for (int a = 0; a < 2; ++a) { mbar_init(&tmem_full[a], 1); mbar_init(&tmem_empty[a], 16); }
    *abort_flag = 0;
    fence_barrier_init();
    prefetch_tensormap(&tmap_w);
    prefetch_tensormap(&tmap_b);
  }
  for (int i = threadIdx.x; i < (F16 ? 0 : 256); i += kThreads) {   // (FP16 weights come from conversions)
    const float sc = scale_to_f32((uint32_t)i, ue);
    uint32_t hi[2] = {0, 0}, lo[2] = {0, 0};
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const uint32_t h = __float_as_uint(__fmul_rn(e2m1_to_f32(c), sc)) >> 16;   // exact in 16 bits
      hi[c >> 2] |= (h >> 8) << (8 * (c & 3));
      lo[c >> 2] |= (h & 0xFFu) << (8 * (c & 3));
    }
    lut[i] = make_uint4(hi[0], hi[1], lo[0], lo[1]);
  }
  if (warp == 1) tmem_alloc_pair(tmem_slot, 512);
  tc_fence_before();
  cluster_sync_all();   // the peer's barriers are initialised before anything arrives on them
  tc_fence_after();
  // (all of the tensor memory is this CTA's, so that it begins at address 0; as a constant it leaves the MMA issuer's operands in uniform registers)
  const uint32_t tmem_base = 0;
  pdl_wait();   // from here on the previous kernel has completed and its writes are visible
  const float *tscale = nullptr;
  int all_kinds = 1;   // kinds of tokens (see the head of the file): bit 0 two FP16 planes (or whatever PLANES says), bit 1 three BF16 planes
  if constexpr (PLANES == 2) {
    tscale = behind_wait(g.tscale);
    const float w = tscale[gn];
    all_kinds = w == 0.f ? 1 : w == 1.f ? 3 : 2;
  }
  auto kinds_of = [&](const Tile &p) -> int {   // those in a tile, each a pass over k (warp-wide)
    if (PLANES != 2 || all_kinds != 3) return all_kinds;
    const uint8_t *const three = (const uint8_t *)(tscale + gn + 1);
    uint32_t f = 0;
    for (int j = p.j0 + lane; j < min(p.j0 + p.width, gn); j += 32) f |= three[j] ? 2u : 1u;
    return (int)__reduce_or_sync(0xFFFFFFFFu, f);
  };
  constexpr int kKinds = PLANES == 2 ? 2 : 1, per_slot = PLANES == 3 ? 3 : 2;   // (per_slot: planes in a ring slot)

  const unsigned tag = g.tag;
  auto wait = [abort_flag, status_word, tag](uint64_t *bar, uint32_t parity, unsigned code) -> bool {
    if (__builtin_expect(mbar_try(bar, parity), 1)) return true;   // the common case: no flag read, no clock read
    if (*abort_flag) return false;
    if (mbar_wait(bar, parity)) return true;
    *abort_flag = 1;
    atomicCAS(status_word, 0u, code | tag);
    return false;
  };
  const int W = g.width, nfull = g.nfull, cut = g.cut;
  int ntiles = g.tiles;
  if (GROUPED) {   // token tiles per group, then their running sum; a group whose rows are not inside [0, n) has none
    const int groups = g.groups;
    for (int q = threadIdx.x; q <= groups; q += kThreads) gseg[q] = g.seg[q];
    __syncthreads();
    if (warp == 0) {
      int base = 0;
      for (int q0 = 0; q0 < groups; q0 += 32) {
        const int q = q0 + lane;
        const int lo = q < groups ? gseg[q] : 0, hi = q < groups ? gseg[q + 1] : 0;
        int v = (lo >= 0 && hi > lo && hi <= gn) ? (hi - lo + W - 1) / W : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xFFFFFFFFu, v, o); if (lane >= o) v += u; }
        if (q < groups) gcum[q + 1] = base + v;
        base += __shfl_sync(0xFFFFFFFFu, v, 31);
      }
      if (lane == 0) gcum[0] = 0;
    }
    __syncthreads();
    ntiles = gcum[groups] * tiles_m;
  }
  auto tile_of = [=](int t) -> Tile {
    if (GROUPED) {
      const int tt = t / tiles_m;
      int q = 0, hi = g.groups;   // the last q with gcum[q] <= tt (the group holding token tile tt has gcum[q + 1] > tt)
      while (hi - q > 1) { const int mid = (q + hi) >> 1; if (gcum[mid] <= tt) q = mid; else hi = mid; }
      const int j0 = gseg[q] + (tt - gcum[q]) * W, left = gseg[q + 1] - j0;
      return Tile{t % tiles_m, j0, gseg[q + 1], left < W ? (left + 63) & ~63 : W, q * gm, -1, 0, nk_all};
    }
    int w = W, part = 0, u = -1, k0 = 0, nk = nk_all;
    if (CUT_K && t >= nfull) {
      u = t - nfull;
      k0 = u % g.parts * g.part_stages;
      nk = min(g.part_stages, nk_all - k0);
      t = nfull + u / g.parts;
    } else if (!TAIL && t >= nfull) { w = W / cut; part = (t - nfull) % cut; t = nfull + (t - nfull) / cut; }
    const int j0 = t / tiles_m * W + part * w, left = gn - j0;
    return Tile{t % tiles_m, j0, gn, left <= 0 ? 0 : left < w ? (left + 63) & ~63 : w, 0, u, k0, nk};
  };
  // accumulators: two of 128 columns while tiles are that narrow, else one of 256
  const int nacc = W > 128 ? 1 : 2;

  if (warp < 4) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsRest));
  if (warp == 0) {
    // ---------------- producer: this CTA's half of the tile's tokens, one plane of one stage per slot ----------------
    // (the whole warp runs the loop, one elected lane issues: see tma_load_3d_pair_elect)
    const uint32_t sub_bytes = 2u * (uint32_t)(W / 2) * 128u;   // a box is always W / 2 rows per CTA, however many of them the tile uses
    uint32_t it = 0;
    for (int t = tile_first; t < ntiles; t += tile_step) {
      const Tile p = tile_of(t);
      if (p.width == 0) continue;
      const int row0 = p.j0 + rank * (p.width >> 1), kinds = kinds_of(p), nk = CUT_K ? p.nk : nk_all, k0 = CUT_K ? p.k0 : 0;
#pragma unroll 1
      for (int kind = 0; kind < kKinds; ++kind) {
      if (kKinds == 2 && !(kinds >> kind & 1)) continue;
      const int pl_end = PLANES == 2 ? (kind ? 5 : 2) : PLANES;   // (PLANES = 2: planes 0 and 1, then 2 to 4)
#pragma unroll 1
      for (int ks = 0; ks < nk; ks += unit) {
#pragma unroll 1
        for (int pl = 2 * kind; pl < pl_end; pl += per_slot, ++it) {   // a slot: two stages, or two or three planes of one (plane pl of a token's row starts 2 k bytes after plane pl - 1)
          const int s = it & (nB - 1), nsub = PLANES == 1 ? min(unit, nk - ks) : min(per_slot, pl_end - pl);
          if (!__all_sync(0xFFFFFFFFu, wait(&b_empty[s], (it >> lgB & 1) ^ 1, kStWaitEmpty))) goto done;
          if (rank == 0) mbar_arrive_expect_tx_elect(&b_full[s], nsub * sub_bytes);
          const uint32_t dst = smem_u32(sB) + (uint32_t)(s * slot_bytes), bar = mbar_addr_rank(&b_full[s], 0);
          for (int i = 0; i < nsub; ++i)
            tma_load_3d_pair_elect(dst + i * kSub, &tmap_b, PLANES == 1 ? (k0 + ks + i) * 128 : (pl + i) * 2 * gk + (k0 + ks) * 128, row0, 0, bar);
        }
      }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (even CTA) ----------------
    // The whole warp runs the loop and one elected lane issues; from inside a one-lane branch every tcgen05.mma costs ~150 cycles.  Alone, a pair
    // takes 64 cycles for 256 x 128 x 16 and 128 for twice the tokens, but this warp shares its scheduler and its instruction cache with 18 others: with two
    // waits, four MMAs and a commit per plane of a stage an MMA took about 180 cycles whatever the tile's width.  A unit of work is therefore two stages,
    // or all planes of one, behind one wait for the weights and one for the activations, with one commit, in one statement, its operands in uniform
    // registers: now 94 - 165 cycles for 128 tokens and 127 for 256.  With the planes above, 8 experts of 2048 x 4096 on 1100 tokens: 123 -> 96 us.
    if (rank == 0) {
      const uint64_t db0 = smem_desc_sw128(smem_u32(sB));
      uint32_t ia = 0, ib = 0, acc_i = 0;
      for (int t = tile_first; t < ntiles; t += tile_step) {
        const Tile p = tile_of(t);
        if (p.width == 0) continue;
        const int kinds = kinds_of(p), nk = CUT_K ? p.nk : nk_all;
        for (int ks0 = 0; ks0 < nk; ks0 += SEG ? seg_stages : nk, ++acc_i) {
          const int acc = nacc == 2 ? acc_i & 1 : 0, ks1 = SEG ? min(ks0 + seg_stages, nk) : nk;
          const uint32_t acc_par = (nacc == 2 ? acc_i >> 1 : acc_i) & 1;
          if (!__all_sync(0xFFFFFFFFu, wait(&tmem_empty[acc], acc_par ^ 1, kStWaitTmemEmpty))) goto done;
          // (the small terms' accumulator was read together with the previous tile's last segment, whose accumulator is the next one's)
          if (SEG && PLANES != 1 && ks0 == 0 && !__all_sync(0xFFFFFFFFu, wait(&tmem_empty[acc ^ 1], (((acc_i + 1) >> 1) & 1) ^ 1, kStWaitTmemEmpty))) goto done;
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + acc * 128;
#pragma unroll 1
          for (int kind = 0; kind < kKinds; ++kind) {
          if (kKinds == 2 && !(kinds >> kind & 1)) continue;
          const uint32_t idesc = idesc_f16(256, p.width, PLANES == 2 ? kind : F16 ? 0 : 1);
          const bool second = kind && (kinds & 1);   // on the sums of the first pass
#pragma unroll 1
          for (int ks = ks0; ks < ks1; ks += unit, ++ia, ++ib) {
            const int sa = ia & (nA - 1);
            int sb = ib & (nB - 1);
            if (!__all_sync(0xFFFFFFFFu, wait(&a_full[sa], ia >> lgA & 1, kStWaitFullA) && wait(&b_full[sb], ib >> lgB & 1, kStWaitFullB))) goto done;
            tc_fence_after();
            const uint32_t a_tmem = tmem_base + kACols + sa * subA * 32;
            uint64_t db = db0 + (uint32_t)(sb * (slot_bytes >> 4));
            if (PLANES == 1) {
              if (ks + 1 < ks1 && unit == 2)
                mma8_f16_commit_pair_elect(d_tmem, a_tmem, db, ks != ks0, d_tmem, a_tmem + 32, db + (kSub >> 4), 1, idesc, &b_empty[sb]);
              else
                mma4_f16_commit_pair_elect(d_tmem, a_tmem, db, idesc, ks != ks0, &b_empty[sb]);
            } else if (PLANES == 3) {   // (the small planes are summed over all of k, apart from the segments)
              mma12_f16_commit_pair_elect(d_tmem, a_tmem, db, ks != ks0, tmem_base + kSmallCols, db + (kSub >> 4), ks != 0, db + 2 * (kSub >> 4), idesc, &b_empty[sb]);
              tc_commit_pair_elect(&a_empty[sa]);
            } else {
              mma8_f16_commit_pair_elect(d_tmem, a_tmem, db, second || ks != ks0, d_tmem, a_tmem, db + (kSub >> 4), 1, idesc, &b_empty[sb]);
              if (kind) {
                ++ib;
                sb = ib & (nB - 1);
                if (!__all_sync(0xFFFFFFFFu, wait(&b_full[sb], ib >> lgB & 1, kStWaitFullB))) goto done;
                tc_fence_after();
                db = db0 + (uint32_t)(sb * (slot_bytes >> 4));
                mma4_f16_commit_pair_elect(d_tmem, a_tmem, db, idesc, 1, &b_empty[sb]);
              }
              tc_commit_pair_elect(&a_empty[sa]);
            }
          }
          }
          tc_commit_pair_elect(&tmem_full[acc]);
        }
      }
    }
  } else if (warp == 2) {
    // ---------------- producer: this CTA's 128 weight rows, 256 values of k per slot ----------------
    const bool img = g.A.image;
    const int ktiles = g.A.ktiles;
    uint32_t it = 0;
    for (int t = tile_first; t < ntiles; t += tile_step) {
      const Tile p = tile_of(t);
      if (p.width == 0) continue;
      const int row_tile = 2 * p.tm + rank, k0 = CUT_K ? p.k0 : 0, nslots = CUT_K ? (p.nk + 3) / 4 : nslots_all;
      for (int pass = kKinds == 2 ? __popc(kinds_of(p)) : 1; pass > 0; --pass) {
#pragma unroll 1
      for (int sl = 0; sl < nslots; ++sl, ++it) {
        const int s = it % kRaw;
        if (!__all_sync(0xFFFFFFFFu, wait(&raw_empty[s], ((it / kRaw) & 1) ^ 1, kStWaitRaw))) goto done;
        mbar_arrive_expect_tx_elect(&raw_full[s], C::kRawBytes);
        const uint32_t dst = smem_u32(sRaw + (size_t)s * C::kRawBytes), bar = smem_u32(&raw_full[s]);
        // (rows past the matrix read zeros; their scales are those of its last row, and no row past it is stored)
        if (img) tma_load_3d_elect(dst, &tmap_w, 0, 0, row_tile * ktiles + (k0 >> 2) + sl, bar);
        else tma_load_3d_elect(dst, &tmap_w, ((k0 >> 2) + sl) * 128, p.ro + row_tile * 128, 0, bar);
      }
      }
    }
  }
  } else if (warp < 12) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsEpi));
    // ---------------- epilogue ----------------
    const int quad = warp & 3, half = (warp - 4) >> 2, bar_id = 2 + half;   // barrier 1: all eight warps; 2 and 3: the four of a half
    // (rarely used parameters are read from the constant bank where they are needed: the registers belong to the accumulator block)
    const float gb0 = !PART && g.e.gb ? *g.e.gb : 1.f;   // B's global: dense B has none, INT8 B one for the tensor (a multiply by 1 is exact)
    uint8_t *const dptr = (uint8_t *)g.e.d;
    const int d_dtype = g.e.d_dtype, mask = EPI == kEpiSwiglu ? kExSwiglu : EPI == kEpiNormGlu ? kExNorm | kExSwiglu : EPI == kEpiOut2 ? kExOut2 : EPI == kEpiNorm ? kExNorm : SEG || EPI == kEpiPlain || EPI == kEpiAdd || PART || TAIL ? 0 : g.x.mask;   // (segments: a 16-bit D and the plain epilogue)
    const bool d_tma = g.d_tma;
    // The accumulator is read as MMA fragments (16 lanes x 8 columns per register quad): a thread holds rows rb + 16 hh + 8 u (hh, u in
    // {0, 1}) of columns 8 gq + cp + e (e in {0, 1}) of a chunk of 32, register 16 hh + 4 gq + 2 u + e.  Gate and up rows of SwiGLU (8
    // apart) then meet in one thread, neighbouring columns pack into one conversion, and stmatrix transposes 8 x 8 blocks on their
    // way into the staging box: 4 instructions per chunk where a lane per row took 32 two-byte stores (and a shuffle per SwiGLU pair).
    // With SwiGLU the epilogue, which shares issue slots with the expansion, took 140 of 490 us at 28672 x 2048 x 4096.
    const int cp = 2 * (lane & 3), l7 = lane & 7, mi = lane >> 3;
    const bool leader = quad == 0 && lane == 0;
    uint8_t *const boxes = staging + half * 2 * C::kStagingBytes;
    float amax = 0.f;
    uint32_t acc_i = 0, box = 0;
    // A staging tile is free when the store before the last one has been read (the two tiles alternate).  Every turn commits a group, an empty
    // one where nothing was stored by TMA (a group's last tokens, a CTA without rows): "all but the last group" is then the tile's own.
    auto next_box = [&]() -> uint8_t * {
      if (leader) bulk_wait_read_one();
      named_barrier(bar_id, 128);
      return boxes + (box++ & 1) * C::kStagingBytes;
    };
    for (int t = tile_first; t < ntiles; t += tile_step) {
      const Tile p = tile_of(t);
      if (p.width == 0) continue;
      const int tm = 2 * p.tm + rank, jt = p.j0, jend = min(p.j0 + p.width, p.jend), nk = CUT_K ? p.nk : nk_all;
      // this warp's block: width / 2 columns, one to four chunks of 32
      const int hw = p.width >> 1, nchunks = min(hw, jend - jt - half * hw + 31) >> 5;   // (chunks past the last token are left alone)
      uint32_t r[32], rn[32];
      auto load_chunk = [&](uint32_t col, int c, uint32_t (&v)[32]) {
        const uint32_t a = tmem_base + ((uint32_t)(quad * 32) << 16) + col + half * hw + 32 * c;
        tmem_ld_16x256b_x4(a, v);
        tmem_ld_16x256b_x4(a + (16u << 16), v + 16);
      };
      auto release = [&](int acc) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_rank(&tmem_empty[acc], 0);
      };
      if constexpr (SEG) {   // the running sums of chunk 0 are kept in r, those of chunk 1 in rn
#pragma unroll
        for (int q = 0; q < 32; ++q) r[q] = rn[q] = 0;
        auto join = [&](uint32_t col, int c, uint32_t (&sum)[32]) {
          uint32_t v[32];
          load_chunk(col, c, v);
          tmem_ld_wait32(v);
#pragma unroll
          for (int q = 0; q < 32; ++q) sum[q] = __float_as_uint(__fadd_rn(__uint_as_float(sum[q]), __uint_as_float(v[q])));
        };
        for (int ks = 0; ks < nk; ks += seg_stages, ++acc_i) {
          const int acc = acc_i & 1;
          if (!__all_sync(0xFFFFFFFFu, wait(&tmem_full[acc], (acc_i >> 1) & 1, kStWaitTmemFull))) { *abort_flag = 1; break; }
          tc_fence_after();
          if (nchunks > 0) join(acc * 128, 0, r);
          if (nchunks > 1) join(acc * 128, 1, rn);
          if (PLANES != 1 && ks + seg_stages >= nk) {
            if (nchunks > 0) join(kSmallCols, 0, r);
            if (nchunks > 1) join(kSmallCols, 1, rn);
          }
          release(acc);
        }
      }
      const int rb = tm * 128 + quad * 32 + (lane >> 2);
      const bool tile_ok = tm * 128 < gm;   // (an odd number of 128-row tiles leaves the last pair's second CTA without rows)
      float rowp[4], bias[4];               // row 8 q of this thread's four: alpha gA, bias
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int i = rb + 8 * q;
        rowp[q] = !PART && i < gm ? __fmul_rn(g.e.alpha, g.e.ga ? g.e.ga[(size_t)(p.ro + i) * g.e.ga_stride] : 1.f) : 0.f;
        bias[q] = (!PART && i < gm && g.e.bias) ? load_dense(g.e.bias_dtype, g.e.bias, p.ro + i) : -0.f;   // (adding -0 changes nothing)
        if (!(mask & kExNorm)) rowp[q] = __fmul_rn(__fmul_rn(rowp[q], gb0), g.e.gf);   // ((alpha gA) * gB) * gf
      }
      if (mask & kExNorm) {  // column scales of this token tile (the previous tile's are no longer in use: see the barrier below)
        named_barrier(1, 256);
        if (g.x.colscales) {  // computed before the launch, one float per token
          for (int jj = (warp - 4) * 32 + lane; jj < p.width; jj += 256) colscale[jj] = __ldcg(g.x.colscales + min(jt + jj, gn - 1));
        }
        // The defining order (reference include/nvfp4effma.h:224-226 there): lane l adds parts l, l + 32, ... in ascending
        // order, then an xor butterfly 16..1.  A warp takes 8 tokens at a time so that their loads fly together.
        for (int j8 = (warp - 4) * 8; j8 < p.width && !g.x.colscales; j8 += 64) {
          float sum[8];
          if (g.x.norm_nparts <= 256) {
            float v[8][8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              const int j = min(jt + j8 + u, gn - 1);
              const float *p = g.x.norm_parts + (size_t)j * g.x.norm_ld + lane;
#pragma unroll
              for (int q = 0; q < 8; ++q) v[u][q] = (32 * q + lane < g.x.norm_nparts) ? __ldcg(p + 32 * q) : 0.f;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              float a = 0.f;
#pragma unroll
              for (int q = 0; q < 8; ++q)
                if (32 * q + lane < g.x.norm_nparts) a = __fadd_rn(a, v[u][q]);
              sum[u] = a;
            }
          } else {
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              const int j = min(jt + j8 + u, gn - 1);
              const float *p = g.x.norm_parts + (size_t)j * g.x.norm_ld;
              float a = 0.f;
              for (int q = lane; q < g.x.norm_nparts; q += 32) a = __fadd_rn(a, __ldcg(p + q));
              sum[u] = a;
            }
          }
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            float a = sum[u];
#pragma unroll
            for (int o = 16; o; o >>= 1) a = __fadd_rn(a, __shfl_xor_sync(0xFFFFFFFFu, a, o));
            if (lane == 0) colscale[j8 + u] = __frsqrt_rn(__fadd_rn(__fmul_rn(a, g.x.norm_inv_n), g.x.norm_eps));
          }
        }
      }
      const int acc = nacc == 2 ? acc_i & 1 : 0;
      if constexpr (!SEG) {
        if (!wait(&tmem_full[acc], (nacc == 2 ? acc_i >> 1 : acc_i) & 1, kStWaitTmemFull)) *abort_flag = 1;
        ++acc_i;
      }
      // the eight epilogue warps go on together or not at all (another role may raise the flag between two warps' looks at it, and a warp that
      // leaves alone would keep the others at their next barrier)
      if (named_barrier_or(1, 256, *abort_flag != 0)) goto done;
      tc_fence_after();
      // One sum over k: the chunk after the next is requested while one is processed; the accumulator goes back to the MMA warp with the last
      // chunk's load.  (A 256-column accumulator is alone in tensor memory: until then the weight stages fill up behind it, eight deep, and
      // the MMAs catch up from there.)
      if constexpr (!SEG) {
        if (nchunks > 0) load_chunk(acc * 128, 0, rn);
        else release(acc);
      }
      for (int c = 0; c < nchunks; ++c) {
        __syncwarp();   // (the tensor memory loads and waits are warp-wide)
        if constexpr (!SEG) tmem_ld_wait32(rn);
        if (!SEG || c != 0) {
#pragma unroll
          for (int q = 0; q < 32; ++q) r[q] = rn[q];
        }
        if constexpr (!SEG) {
          if (c + 1 < nchunks) load_chunk(acc * 128, c + 1, rn);
          if (c == (nchunks > 1 ? nchunks - 2 : 0)) {   // every column of this warp's block is in registers
            if (nchunks > 1) tmem_ld_wait32(rn);
            release(acc);
          }
        }
        const int cc = half * hw + c * 32;   // first column of the chunk in the tile
        const int j0 = jt + cc;
        const int nvalid = min(32, jend - j0);
        if (PART || (TAIL && p.unit >= 0)) {   // eight lanes write 32 contiguous bytes of a token's sums
          float *const p32 = g.partial + ((size_t)p.unit * W + cc) * 256 + rank * 128 + quad * 32 + (lane >> 2);
#pragma unroll
          for (int ce = 0; ce < 8; ++ce) {
            const int jj = 8 * (ce >> 1) + cp + (ce & 1);
            if (jj >= nvalid) continue;
            const float ts = PLANES == 2 ? tscale[j0 + jj] : 1.f;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const float v = __uint_as_float(r[16 * (q >> 1) + 4 * (ce >> 1) + 2 * (q & 1) + (ce & 1)]);
              if (rb + 8 * q < gm) p32[jj * 256 + 8 * q] = PLANES == 2 ? __fmul_rn(v, ts) : v;
            }
          }
          continue;
        }
        const bool tma = d_tma && (!GROUPED || nvalid == 32);   // (a group's last box would reach into the next group's tokens)
        // values before the output rounding, kept in r[] as FP32 bits
#pragma unroll
        for (int gq = 0; gq < 4; ++gq) {
          float2 cs = make_float2(0.f, 0.f);
          if (mask & kExNorm) cs = *(const float2 *)&colscale[cc + 8 * gq + cp];
          float ts[2] = {1.f, 1.f};
          if constexpr (PLANES == 2) {   // (powers of two)
#pragma unroll
            for (int e = 0; e < 2; ++e) ts[e] = tscale[min(j0 + 8 * gq + cp + e, gn - 1)];
          }
#pragma unroll
          for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              uint32_t &x = r[16 * (q >> 1) + 4 * gq + 2 * (q & 1) + e];
              const float sc = (mask & kExNorm) ? __fmul_rn(__fmul_rn(rowp[q], __fmul_rn(gb0, e ? cs.y : cs.x)), g.e.gf) : rowp[q];
              float v = __fmul_rn(PLANES == 2 ? __fmul_rn(__uint_as_float(x), ts[e]) : __uint_as_float(x), sc);
              v = __fadd_rn(v, bias[q]);
              const int jj = 8 * gq + cp + e;
              if (ADD && g.e.beta != 0.f && rb + 8 * q < gm && jj < nvalid)
                v = __fmaf_rn(g.e.beta, load_dense(g.e.c_dtype, g.e.c, (size_t)(j0 + jj) * g.e.ldc + rb + 8 * q), v);
              x = __float_as_uint(v);
            }
        }
        if (mask & kExOut2) {  // second output v * w2[i] and the slice's sum of squares (rows 16 q .. 16 q + 15 in ascending order)
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            const int i = rb + 16 * hh;   // (m is a multiple of 16: rows i and i + 8 exist together)
            const float w20 = i < gm ? load_dense(g.x.w2_dtype, g.x.w2, i) : 0.f, w21 = i < gm ? load_dense(g.x.w2_dtype, g.x.w2, i + 8) : 0.f;
#pragma unroll
            for (int ce = 0; ce < 8; ++ce) {
              const int jj = 8 * (ce >> 1) + cp + (ce & 1);
              const float v0 = __uint_as_float(r[16 * hh + 4 * (ce >> 1) + (ce & 1)]), v1 = __uint_as_float(r[16 * hh + 4 * (ce >> 1) + 2 + (ce & 1)]);
              if (i < gm && jj < nvalid) {
                store_dense(g.x.d2_dtype, g.x.d2, (size_t)(j0 + jj) * g.x.ldd2 + i, __fmul_rn(v0, w20));
                store_dense(g.x.d2_dtype, g.x.d2, (size_t)(j0 + jj) * g.x.ldd2 + i + 8, __fmul_rn(v1, w21));
              }
              const float vv0 = __fmul_rn(v0, v0), vv1 = __fmul_rn(v1, v1);
              float sq = 0.f;
#pragma unroll
              for (int q = 0; q < 8; ++q) sq = __fadd_rn(sq, __shfl_sync(0xFFFFFFFFu, vv0, 4 * q + (lane & 3)));
#pragma unroll
              for (int q = 0; q < 8; ++q) sq = __fadd_rn(sq, __shfl_sync(0xFFFFFFFFu, vv1, 4 * q + (lane & 3)));
              if (i < gm && lane < 4 && jj < nvalid) g.x.sq[(size_t)(j0 + jj) * g.x.ld_sq + (i >> 4)] = sq;
            }
          }
        }
        const bool glu = (mask & kExSwiglu) != 0;
        if (glu) {  // rows 16 q + r (gate) and 16 q + 8 + r (up) -> output row 8 q + r: 64 output rows per 128-row tile
          // (the results take the gate's registers: 16 hh + 4 gq + e)
#pragma unroll
          for (int hh = 0; hh < 2; ++hh)
#pragma unroll
            for (int ce = 0; ce < 8; ++ce) {
              const int at = 16 * hh + 4 * (ce >> 1) + (ce & 1);
              r[at] = __float_as_uint(silu_mul(__uint_as_float(r[at]), __uint_as_float(r[at + 2])));
            }
        }
        if (AMAX && g.e.amax) {
#pragma unroll
          for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int ce = 0; ce < 8; ++ce)
              if (rb + 8 * q < gm && 8 * (ce >> 1) + cp + (ce & 1) < nvalid && !(glu && (q & 1)))
                amax = fmaxf(amax, fabsf(__uint_as_float(r[16 * (q >> 1) + 4 * (ce >> 1) + 2 * (q & 1) + (ce & 1)])));
        }
        const int orow = glu ? tm * 64 : tm * 128, orows = glu ? gm >> 1 : gm;   // the tile's first output row, rows of D
        if (!SEG && ANY && d_dtype == NVFP4A_FP32) {   // eight lanes write 32 contiguous bytes of a column
          float *const d32 = (float *)dptr + (size_t)j0 * g.e.ldd + orow + (lane >> 2);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            if (glu && (q & 1)) continue;
            const int o = glu ? quad * 16 + 4 * q : quad * 32 + 8 * q;   // output row inside the tile, less lane / 4
            if (rb + 8 * q < gm) {
#pragma unroll
              for (int ce = 0; ce < 8; ++ce) {
                const int jj = 8 * (ce >> 1) + cp + (ce & 1);
                if (jj < nvalid) d32[(size_t)jj * g.e.ldd + o] = __uint_as_float(r[16 * (q >> 1) + 4 * (ce >> 1) + 2 * (q & 1) + (ce & 1)]);
              }
            }
          }
          continue;
        }
        // 16-bit D: neighbouring columns into one register (in place of column 0), then 8 x 8 blocks transposed into a box of
        // [32 tokens][64 rows] with the 128-byte swizzle (two boxes without SwiGLU)
        if (d_dtype == NVFP4A_BF16) {
          uint32_t nan = 0;
#pragma unroll
          for (int q = 0; q < 32; q += 2) {
            r[q] = bf16x2_rn(__uint_as_float(r[q]), __uint_as_float(r[q + 1]));
            nan |= (r[q] & 0x7FFF7FFFu) + 0x00010001u;   // (the hardware rounds every NaN to 0x7FFF, which nothing else gives)
          }
          if (nan & 0x80008000u) {
#pragma unroll
            for (int q = 0; q < 32; q += 2) {
              if ((r[q] & 0x7FFFu) == 0x7FFFu) r[q] = (r[q] & 0xFFFF0000u) | 0x7FC0u;
              if ((r[q] & 0x7FFF0000u) == 0x7FFF0000u) r[q] = (r[q] & 0xFFFFu) | 0x7FC00000u;
            }
          }
        } else {
#pragma unroll
          for (int q = 0; q < 32; q += 2) {
            const __half2 h = __floats2half2_rn(__uint_as_float(r[q]), __uint_as_float(r[q + 1]));
            r[q] = *reinterpret_cast<const uint32_t *>(&h);
          }
        }
        uint8_t *const st = next_box();
        __syncwarp();
        if (glu) {
#pragma unroll
          for (int gp = 0; gp < 2; ++gp)   // matrices: column groups 2 gp and 2 gp + 1, each 16-row half
            stmatrix_x4_trans(st + (8 * (2 * gp + (mi >> 1)) + l7) * 128 + (((2 * quad + (mi & 1)) ^ l7) << 4), r[8 * gp], r[16 + 8 * gp], r[4 + 8 * gp],
                              r[20 + 8 * gp]);
        } else {
#pragma unroll
          for (int gq = 0; gq < 4; ++gq)   // matrices: the four 8-row groups of the warp's 32 rows
            stmatrix_x4_trans(st + (quad >> 1) * 4096 + (8 * gq + l7) * 128 + (((4 * (quad & 1) + mi) ^ l7) << 4), r[4 * gq], r[4 * gq + 2], r[16 + 4 * gq],
                              r[18 + 4 * gq]);
        }
        if (tma) {
          fence_proxy_async_smem();
          named_barrier(bar_id, 128);
          if (leader && tile_ok) {
            for (int b = 0; b < (glu ? 1 : 2); ++b) {
              const int o = orow + 64 * b;
              if (o >= orows) break;
              tma_store_2d(&tmap_d, st + b * 4096, o, j0);
              for (int q = 0; q < peers.n; ++q) tma_store_2d(&peers.map[q], st + b * 4096, o, j0);   // the same box into every peer's buffer
            }
          }
        } else {   // D that TMA cannot store, or a group's last tokens: a thread per row
          named_barrier(bar_id, 128);
          const int th = quad * 32 + lane, row = glu ? th & 63 : th, step = glu ? 2 : 1;
          if (orow + row < orows) {
            const uint8_t *src = st + (row >> 6) * 4096 + (row & 7) * 2;
            for (int jj = glu ? th >> 6 : 0; jj < nvalid; jj += step)
              ((uint16_t *)dptr)[(size_t)(j0 + jj) * g.e.ldd + orow + row] = *(const uint16_t *)(src + jj * 128 + ((((row >> 3) & 7) ^ (jj & 7)) << 4));
          }
        }
        if (leader) bulk_commit();
      }
    }
    if (leader) bulk_wait_all();
    if (AMAX && g.e.amax) warp_amax_commit(g.e.amax, amax);
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsConv));
    // ---------------- weight expansion: NVFP4 -> 16-bit floats in tensor memory ----------------
    // Two groups of four warps take the even and the odd pairs of stages of a tile (a slot's halves; on alternate stages every wait and hand-over came
    // twice as often: 28672 x 4096 with SwiGLU on 2048 tokens 340 us instead of 318, FP16 4096 x 4096 on 333 tokens 34.3 instead of 31.2); inside a group thread r owns row r of the CTA's 128 (and
    // tensor memory lane r: warp % 4 is its quadrant): a stage's 64 nibbles are two 16-byte words of the slot's swizzled row, its 4 scale bytes one word fetched a slot (four stages)
    // ahead.
    const int cwarp = warp - 12, group = cwarp >> 2;
    const int row = (cwarp & 3) * 32 + lane, r7 = row & 7;
    const Fp4Operand A = g.A;
    const ScalePos sp{A.sld};
    const bool img = A.image, swz = A.sld < 0;
    // scale words of this group's two stages of slot sl (stages past the end of k: zeros)
    auto fetch_scales = [&](const uint8_t *scp, int k0, int nk, int sl, uint32_t (&v)[2]) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int ks = 4 * sl + 2 * group + h;
        const size_t off = img ? (size_t)((k0 >> 2) + sl) * kImgTileBytes + (ks & 3) * 512 : swz ? (size_t)(k0 + ks) * 512 : (size_t)(k0 + ks) * 4;
        v[h] = ks < nk ? *(const uint32_t *)(scp + off) : 0u;
      }
    };
    const int tile_units_all = (nk_all + unit - 1) / unit;
    uint32_t isl = 0, it0 = 0;   // slots so far; units of the finished passes over k
    for (int t = tile_first; t < ntiles; t += tile_step) {
      const Tile p = tile_of(t);
      if (p.width == 0) continue;
      const int kinds = kinds_of(p), k0 = CUT_K ? p.k0 : 0, nk = CUT_K ? p.nk : nk_all, nslots = CUT_K ? (nk + 3) / 4 : nslots_all,
                tile_units = CUT_K ? (nk + unit - 1) / unit : tile_units_all;
      const int r = min((2 * p.tm + rank) * 128 + row, gm - 1);
      const uint8_t *scp = img ? A.data + (size_t)(r >> 7) * A.ktiles * kImgTileBytes + kImgDataBytes + (r & 31) * 16 + ((r & 127) >> 5) * 4
                               : A.sc + sp.row(p.ro + r);
#pragma unroll 1
      for (int kind = 0; kind < kKinds; ++kind) {
      if (kKinds == 2 && !(kinds >> kind & 1)) continue;
      uint32_t sc[2], sc_next[2] = {0, 0};
      fetch_scales(scp, k0, nk, 0, sc);
#pragma unroll 1
      for (int sl = 0; sl < nslots; ++sl, ++isl) {
        if (sl + 1 < nslots) fetch_scales(scp, k0, nk, sl + 1, sc_next);
        const int rs = isl % kRaw;
        if (!__all_sync(0xFFFFFFFFu, wait(&raw_full[rs], (isl / kRaw) & 1, kStWaitRaw))) goto done;
        const uint8_t *src = sRaw + (size_t)rs * C::kRawBytes + row * 128;
        uint4 w[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) w[q] = *(const uint4 *)(src + (((4 * group + q) ^ r7) << 4));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int ks = 4 * sl + 2 * group + h;
          if (ks >= nk) break;
          const uint32_t it = it0 + (unit == 2 ? ks >> 1 : ks);
          const int s = it & (nA - 1);
          // (the vote also brings the warp together again: lanes whose first poll failed come later, and the stores below are warp-wide)
          if ((h == 0 || unit == 1) && !__all_sync(0xFFFFFFFFu, wait(&a_empty[s], (it >> lgA & 1) ^ 1, kStWaitConv))) goto done;
          tc_fence_after();   // the MMAs of the stage's previous round have read it
          const uint32_t dst = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + kACols + (unit == 2 ? 2 * s + h : s) * 32;
#pragma unroll
          for (int u = 0; u < 2; ++u) {   // 32 values: two blocks, 16 columns
            const uint32_t wv[4] = {w[2 * h + u].x, w[2 * h + u].y, w[2 * h + u].z, w[2 * h + u].w};
            uint32_t o[16];
            if (F16 || (PLANES == 2 && kind == 0)) {   // (E4M3 scales) conversions to FP16 and one multiply per pair of values, exact
              const uint32_t s2 = h2mul(scale_pair(sc[h] >> (16 * u)), 0x5C005C00u);   // (2^8: scale_pair's are that much smaller)
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                uint32_t v[4];
                e2m1_to_f16(wv[q], v);
                const uint32_t sb = byte_perm(s2, s2, q >> 1 ? 0x3232u : 0x1010u);
#pragma unroll
                for (int e = 0; e < 4; ++e) o[4 * q + e] = h2mul(v[e], sb);
              }
              tmem_st16(dst + 16 * u, o);
              continue;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {  // 8 values per word
              const uint4 t4 = lut[(sc[h] >> (16 * u + 8 * (q >> 1))) & 0xFF];
              e2m1_expand4(wv[q], t4, o[4 * q], o[4 * q + 1]);
              e2m1_expand4(wv[q] >> 16, t4, o[4 * q + 2], o[4 * q + 3]);
            }
            tmem_st16(dst + 16 * u, o);
          }
          if (unit == 2 && h == 0 && ks + 1 < nk) continue;   // the unit's second stage follows
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_rank(&a_full[s], 0);
        }
        // The slot goes back only now that its words have been USED: a load that is merely issued may still be queued behind the epilogue's
        // stores when the producer's next copy lands (seen as words of the following slot in a handful of rows).
        __syncwarp();
        if (lane == 0) mbar_arrive(&raw_empty[rs]);
        sc[0] = sc_next[0]; sc[1] = sc_next[1];
      }
      it0 += tile_units;
      }
    }
  }
done:
  __syncwarp();
  if (*abort_flag) { bulk_wait_all(); settle_after_abort(); }
  __syncwarp();
  tc_fence_before();
  cluster_sync_all();   // neither CTA leaves (or frees tensor memory) while the other may still arrive on its barriers
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

// What a stage of a tile costs, in nanoseconds (64 tiles of one round, k = 8192 less k = 2048).  One plane: the expansion, almost whatever the
// tokens (32 to 128: 280 - 300; 192: 320; 256: 323).  Two planes: the MMAs (64 and 128: 440 - 450; 192: 497; 256: 623).  Three: 470 - 500.
constexpr int kNarrow = 128;   // a tile narrower than this saves nothing
long long stage_cost(int width, int planes) {
  if (planes == 1) return width > 128 ? 322 : 295;
  return planes == 3 ? 480 : width > 192 ? 623 : width > 128 ? 497 : 445;
}
// Tile width and cut for a problem of `rows256` 256-row tiles and n tokens: the width whose rounds over the SM pairs cost least; the tiles of
// the last round are cut in two while the pairs can take the halves all at once.
struct Plan { int width, nfull, cut, tiles; };
Plan make_plan(int rows256, int n, int planes, int pairs, int widest) {
  Plan best = {0, 0, 1, 0};
  long long best_cost = 0;
  for (int w = widest; w >= 64; w -= w > 128 ? 64 : w / 2) {   // 256, 192, 128, 64
    if (w > 64 && (w > 128 ? w - 64 : w / 2) >= n) continue;   // the next width covers every token
    const int tiles = rows256 * ((n + w - 1) / w), rest = tiles % pairs;
    int cut = 1;
    while (tiles > pairs && rest && w / (2 * cut) >= kNarrow && rest * 2 * cut <= pairs) cut *= 2;
    const long long c = tiles / pairs * stage_cost(w, planes) + (rest ? stage_cost(w / cut, planes) : 0);
    if (!best.width || c < best_cost) {
      best_cost = c;
      best = Plan{w, cut > 1 ? tiles - rest : tiles, cut, cut > 1 ? tiles - rest + rest * cut : tiles};
    }
  }
  return best;
}

// Parts of k.  A problem with few tiles leaves most SM pairs idle while each tile is a serial chain over k (0.3 to 0.6 us per 64 values).  Up to eight pairs
// take a run of at least 512 values each (the last one what is left); their FP32 sums meet in memory, which is L2, and a small kernel adds them in order.  That kernel, its launch and
// the memory cost 8 us of a caller's time and the traffic (0.5 ns per KB), so that k has to be long enough to gain more.  A call in eager mode: INT8
// 4928 x 4608 on 35 tokens 47.8 -> 30.2 us, 832 x 4480 on 12 45.6 -> 28.2, BF16 2688 x 4736 on 46 25.3 -> 17.0; with less to gain, INT8 2594 x 1792 on
// 12 tokens 26.3 -> 28.5 and BF16 872 x 5376 on 1030 29.6 -> 31.2, which this rule leaves whole.
// (The number of tiles decides: a plain weight's rows and a shard of them may be cut differently and then differ in the last bits.)  Not for nvfp4a_gemm_ex (see
// GemmArgs::whole_k), nor for images of BF16 problems: the outputs of a tensor-parallel shard are those of the whole matrix bit for bit, however many tiles either has.
bool parts_allowed(const GemmArgs &g) {
  const bool tp_twin = g.A.image && g.B.dtype == NVFP4A_BF16;
  return !(tp_twin || g.no_alloc || g.whole_k || g.tp.world > 1 || g.x.mask);
}
// parts of k, and the slots of 256 values in each but the last, for `tiles` tiles that have the pairs to themselves
int most_parts(int k, int tiles, int pairs, int *run) {
  const int slots = (k + 255) / 256;
  int parts = pairs / tiles;
  if (parts > 8) parts = 8;
  if (parts > slots / 2) parts = slots / 2;
  if (parts < 2) return 1;
  *run = (slots + parts - 1) / parts;
  return (slots + *run - 1) / *run;   // (equal runs: no empty part)
}
int choose_parts(const GemmArgs &g, int planes, const Plan &p, int pairs) {
  int run = 0;
  if (!parts_allowed(g) || p.cut > 1 || p.tiles > pairs) return 1;
  const int parts = most_parts(g.k, p.tiles, pairs, &run);
  if (parts < 2) return 1;
  const int saved = ((g.k + 255) / 256 - run) * 4;   // stages
  return saved * stage_cost(p.width, planes) > 8000 + 8ll * parts * g.n * g.m / 2000 ? parts : 1;
}
// The same for the last round of a problem of several: at a width whose last round has at most half as many tiles as there are pairs, those run in parts beside the whole ones.
// The sums' way through memory and the join took 7 to 9 us up to 9000 tokens x parts of tiles (17000 of them 12 and more: there the last round is better left half as
// wide), which the model's 5 us and 0.4 ns each stand for; the four per cent that a tail has to gain are what it does not know.  In a graph, INT8 2500 x 4288 on 1793 tokens 92.1 -> 78.1 us,
// BF16 18997 x 7168 on 250 81.5 -> 61.6, FP16 4864 x 6208 on 600 85 - 95 -> 70 - 78, 4096 x 4096 on 700 51.0 -> 45.6, 3584 x 3584 on 1500 64.6 -> 61.3; forced, INT8 6144 x 4096
// on 1000 80.8 -> 92.8 and BF16 49.0 -> 53.2, which the rule leaves whole.
int choose_tail(const GemmArgs &g, int planes, int rows256, int pairs, int widest, Plan *p) {
  if (!parts_allowed(g) || p->tiles <= pairs) return 1;
  const int stages = (g.k + 63) / 64;
  const long long last = p->cut > 1 || p->tiles % pairs ? stage_cost(p->width / p->cut, planes) : 0;
  const long long whole = (p->nfull / pairs * stage_cost(p->width, planes) + last) * stages;
  long long best = whole - whole / 25;
  int parts = 1;
  for (int w = widest; w >= 64; w -= w > 128 ? 64 : w / 2) {
    const int tiles = rows256 * ((g.n + w - 1) / w), tail = tiles % pairs;
    int run = 0;
    const int q = tiles > pairs && tail ? most_parts(g.k, tail, pairs, &run) : 1;
    const long long c = (tiles / pairs * stages + run * 4) * stage_cost(w, planes) + 5000 + (long long)q * tail * w * 2 / 5;
    if (q < 2 || c >= best) continue;
    best = c;
    parts = q;
    *p = Plan{w, tiles - tail, 1, tiles};
  }
  return parts;
}
size_t partial_bytes(int tiles, int parts, int width) { return (size_t)tiles * parts * width * 256 * sizeof(float); }

// Grouped: only the average number of tokens per group is known here, and each group ends in a tile as wide as its last tokens (in steps
// of 64).  `tiles` bounds the grid, the kernel counts the tiles itself.
Plan make_grouped_plan(int rows256, int n, int groups, int planes, int pairs, int widest) {
  Plan best = {0, 0, 1, 0};
  long long best_cost = 0;
  const int avg = (n + groups - 1) / groups;
  for (int w = widest; w >= 64; w /= 2) {
    const int whole = (avg - 1) / w, last = avg - whole * w;
    const long long tiles = (long long)rows256 * groups * (whole + 1);
    const long long cost = whole * stage_cost(w, planes) + stage_cost((last + 63) & ~63, planes);   // of a group's tiles in one row of tiles
    const long long c = tiles <= pairs ? stage_cost(whole ? w : (last + 63) & ~63, planes) : (long long)rows256 * groups * cost / pairs;
    if (!best.width || c < best_cost) {
      const long long bound = (long long)rows256 * ((n + w - 1) / w + groups);
      best_cost = c;
      best = Plan{w, 0, 1, (int)(bound < (1 << 30) ? bound : 1 << 30)};
    }
  }
  return best;
}

template <int PLANES, bool F16, bool GROUPED, int EPI>
cudaError_t launch_epi(const CUtensorMap &tw, const CUtensorMap &tb, const CUtensorMap &td, const PeerMaps &pm, const W4A16Args &a, cudaStream_t s) {
  using C = Cfg<PLANES, GROUPED>;
  static std::atomic<bool> attr_set[64];   // zero-initialised; set once per device (a repeated cudaFuncSetAttribute is harmless)
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set[dev & 63]) {
    const cudaError_t e = cudaFuncSetAttribute(gemm_w4a16_kernel<PLANES, F16, GROUPED, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
    if (e != cudaSuccess) return e;
    attr_set[dev & 63] = true;
  }
  const int pairs = device_sms() / 2;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof cfg);
  cfg.gridDim = dim3(2 * (a.tiles < pairs ? a.tiles : pairs), 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = C::kSmemBytes;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = pdl_enabled() ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, gemm_w4a16_kernel<PLANES, F16, GROUPED, EPI>, tw, tb, td, pm, a);
}

template <int PLANES, bool F16, bool GROUPED = false>
cudaError_t launch_cfg(const CUtensorMap &tw, const CUtensorMap &tb, const CUtensorMap &td, const PeerMaps &pm, const W4A16Args &a, cudaStream_t s) {
  const bool scaled = a.e.beta == 0.f && a.e.d_dtype != NVFP4A_FP32, plain = scaled && !a.e.amax;
  if constexpr (!GROUPED) {
    if (a.parts > 1 && a.nfull) return plain ? launch_epi<PLANES, F16, GROUPED, kEpiTail>(tw, tb, td, pm, a, s) : launch_epi<PLANES, F16, GROUPED, kEpiTailAny>(tw, tb, td, pm, a, s);
    if (a.parts > 1) return launch_epi<PLANES, F16, GROUPED, kEpiPart>(tw, tb, td, pm, a, s);
  }
  if constexpr (!F16 && !GROUPED && PLANES < 3) {
    if (scaled && a.x.mask == (kExNorm | kExSwiglu)) return launch_epi<PLANES, F16, GROUPED, kEpiNormGlu>(tw, tb, td, pm, a, s);
    if (scaled && a.x.mask == kExNorm) return launch_epi<PLANES, F16, GROUPED, kEpiNorm>(tw, tb, td, pm, a, s);
    if (a.e.beta != 0.f && a.e.d_dtype != NVFP4A_FP32 && a.x.mask == 0) return launch_epi<PLANES, F16, GROUPED, kEpiAdd>(tw, tb, td, pm, a, s);
    if (scaled && a.x.mask == kExOut2) return launch_epi<PLANES, F16, GROUPED, kEpiOut2>(tw, tb, td, pm, a, s);
  }
  if constexpr (!F16 && !GROUPED)
    if (plain && a.x.mask == kExSwiglu) return launch_epi<PLANES, F16, GROUPED, kEpiSwiglu>(tw, tb, td, pm, a, s);
  if (plain && a.x.mask == 0) return launch_epi<PLANES, F16, GROUPED, kEpiPlain>(tw, tb, td, pm, a, s);
  return launch_epi<PLANES, F16, GROUPED, kEpiAny>(tw, tb, td, pm, a, s);
}

// the tile plan of one weight; *parts: the parts of k, of all its tiles (nfull = 0) or of those from nfull on
Plan plan_parts(const GemmArgs &g, int planes, bool f16, int *parts) {
  const int rows256 = (g.m + 255) / 256, pairs = device_sms() / 2;
  const int widest = f16 || planes == 3 ? kSegmentWidth : 256;
  Plan p = make_plan(rows256, g.n, planes, pairs, widest);
  *parts = choose_parts(g, planes, p, pairs);
  if (*parts > 1) p.nfull = 0;
  else *parts = choose_tail(g, planes, rows256, pairs, widest, &p);
  return p;
}

// what every launch of the kernel shares: arguments, the schedule, the maps of the weights, of the activations (`row_bytes` bytes per
// token, `pitch` between tokens) and of D
bool set_up(const GemmArgs &g, int planes, bool f16, int groups, const void *act, uint64_t row_bytes, uint64_t pitch, W4A16Args *a, CUtensorMap *tw, CUtensorMap *tb,
            CUtensorMap *td) {
  memset(a, 0, sizeof *a);
  a->m = g.m; a->n = g.n; a->k = g.k;
  a->A = g.A;
  a->e = g.e; a->x = g.x;
  a->status = kernel_status_device_ptr();
  a->tag = next_launch_tag();
  a->parts = 1;
  const Plan p = groups ? make_grouped_plan((g.m + 255) / 256, g.n, groups, planes, device_sms() / 2, kSegmentWidth) : plan_parts(g, planes, f16, &a->parts);
  const uint64_t wrows = (uint64_t)g.m * (groups ? groups : 1);
  a->unit = planes == 1 && !(f16 && g.k < 512) ? 2 : 1;
  a->seg_stages = g.k >= 1024 ? 4 : g.k >= 512 ? 2 : 1;   // (the longest that keep the sums no less exact than the CUDA-core kernels': see the head of the file)
  a->width = p.width; a->nfull = p.nfull; a->cut = p.cut; a->tiles = p.tiles;
  if (a->parts > 1) {
    const int slots = (g.k + 255) / 256;
    a->part_stages = (slots + a->parts - 1) / a->parts * 4;
    a->tiles = p.nfull + (p.tiles - p.nfull) * a->parts;
  }
  const uint64_t wtiles = (uint64_t)((g.m + 127) / 128) * g.A.ktiles;
  if (g.A.image ? !make_tmap_bytes(tw, g.A.data, 128, 128, 128, 128, wtiles, kImgTileBytes)
                : !make_tmap_bytes(tw, g.A.data, (uint64_t)g.k / 2, wrows, (uint64_t)g.A.ld / 2, 128, 1, (uint64_t)g.A.ld / 2 * wrows))
    return false;
  if (!make_tmap_bytes(tb, act, row_bytes, (uint64_t)g.n, pitch, p.width / 2, 1, pitch * g.n)) return false;
  memset(td, 0, sizeof *td);
  const int esz = dense_bytes(g.e.d_dtype);
  const bool glu = (g.x.mask & kExSwiglu) != 0;
  const int drows = glu ? g.m / 2 : g.m;   // SwiGLU: the output has m / 2 rows, 64 per 128-row tile
  a->d_tma = (a->parts == 1 || a->nfull) && esz == 2 && ((uintptr_t)g.e.d & 15) == 0 && ((size_t)g.e.ldd * esz) % 16 == 0 && ((size_t)drows * esz) % 16 == 0 &&
             make_tmap_dense(td, g.e.d, esz, (uint64_t)drows, (uint64_t)g.n, (uint64_t)g.e.ldd * esz, 64, 32, 128);
  return true;
}

// INT8 activations q [n][ld] with one FP32 scale s per 16 values -> planes 0 and 1 of [n][5][k], FP16: t1 + t2 is q * s * 2^(7 - E) to within 2^-23 of
// itself or 2^-25, E the exponent of the token's largest scale; tscale[token] = 2^(E - 7).  A token whose scales two planes do not
// take (see the head of the file) is zeros there, and marked in wide[token].  One CTA per token, a thread per 8 values: 8 bytes in, two 16-byte stores out.
constexpr int kPlanesThreads = 256, kPlanesSpread = 12;
__global__ void __launch_bounds__(kPlanesThreads) w4a8_planes_kernel(const int8_t *q_in, int ld, const float *sc_in, int lds, int k, uint16_t *planes, float *tscale,
                                                                     uint8_t *wide) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ uint32_t red[2][kPlanesThreads / 32];
  const int j = blockIdx.x;
  const float *const srow = behind_wait(sc_in) + (size_t)j * lds;
  const int8_t *const qrow = behind_wait(q_in) + (size_t)j * ld;
  uint2 raw_next = make_uint2(0, 0);   // this thread's first values: on their way while the scales are looked through
  if ((int)threadIdx.x < (k >> 3)) raw_next = *(const uint2 *)(qrow + 8 * threadIdx.x);
  uint32_t hi = 0, lo = 0xFFFFFFFFu;   // largest and smallest non-zero |s| (less one), as bits
  for (int b = threadIdx.x; b < (k >> 4); b += kPlanesThreads) {
    const uint32_t u = __float_as_uint(srow[b]) & 0x7FFFFFFFu;
    hi = max(hi, u);
    lo = min(lo, u - 1u);
  }
  hi = __reduce_max_sync(0xFFFFFFFFu, hi);
  lo = __reduce_min_sync(0xFFFFFFFFu, lo);
  if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = hi; red[1][threadIdx.x >> 5] = lo; }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kPlanesThreads / 32; ++w) { hi = max(hi, red[0][w]); lo = min(lo, red[1][w]); }
  const int eh = hi ? (int)(hi >> 23) : 127, el = hi ? (int)((lo + 1u) >> 23) : 127;   // biased exponents (Inf, NaN: 255)
  const bool narrow = eh >= 27 && eh <= 227 && eh - el <= kPlanesSpread;
  if (threadIdx.x == 0) {
    tscale[j] = __uint_as_float((uint32_t)(narrow ? eh - 7 : 127) << 23);
    wide[j] = !narrow;
  }
  uint16_t *const row0 = planes + (size_t)j * 5 * k;
  if (!narrow) {
    for (int c = threadIdx.x; c < (k >> 3); c += kPlanesThreads)
#pragma unroll
      for (int p = 0; p < 2; ++p) *(uint4 *)(row0 + (size_t)p * k + 8 * c) = make_uint4(0, 0, 0, 0);
    return;
  }
  const float up = __uint_as_float((uint32_t)(261 - eh) << 23);   // 2^(7 - E), a normal number
  for (int c = threadIdx.x; c < (k >> 3); c += kPlanesThreads) {
    const uint2 raw = raw_next;
    if (c + kPlanesThreads < (k >> 3)) raw_next = *(const uint2 *)(qrow + 8 * (c + kPlanesThreads));
    const float s = __fmul_rn(srow[c >> 1], up);   // exact
    uint32_t t[2][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float v[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) v[e] = (float)(int)(int8_t)(((i < 2 ? raw.x : raw.y) >> (16 * (i & 1) + 8 * e)) & 0xFFu);
      const __half2 t1 = __floats2half2_rn(__fmul_rn(v[0], s), __fmul_rn(v[1], s));
      const float2 f1 = __half22float2(t1);
      const __half2 t2 = __floats2half2_rn(__fmaf_rn(v[0], s, -f1.x), __fmaf_rn(v[1], s, -f1.y));   // (the remainders are exact)
      t[0][i] = *reinterpret_cast<const uint32_t *>(&t1);
      t[1][i] = *reinterpret_cast<const uint32_t *>(&t2);
    }
    uint16_t *const row = row0 + 8 * c;
#pragma unroll
    for (int p = 0; p < 2; ++p) *(uint4 *)(row + (size_t)p * k) = make_uint4(t[p][0], t[p][1], t[p][2], t[p][3]);
  }
}

// Runs behind it: tells the GEMM which planes there are (tscale[n], see W4A16Args), and if some token is wide, or all are (`force`), writes the last three of
// each token's `per_token` planes, BF16: t1 + t2 + t3 = fl(q * s) exactly, tscale 1, of the wide ones, zeros of the others.
__global__ void __launch_bounds__(256) w4a8_wide_planes_kernel(const int8_t *q_in, int ld, const float *sc_in, int lds, int n, int k, uint16_t *planes, int per_token,
                                                               float *tscale, const uint8_t *wide_in, int force) {
  pdl_launch_dependents();
  pdl_wait();
  const uint8_t *const wide = behind_wait(wide_in);
  const int8_t *const q = behind_wait(q_in);
  const float *const sc = behind_wait(sc_in);
  int any = force;
  for (int j = threadIdx.x; j < n && !force; j += blockDim.x) any |= wide[j];
  any = __syncthreads_or(any);
  if (blockIdx.x == 0 && threadIdx.x == 0) tscale[n] = force ? 2.f : any ? 1.f : 0.f;
  if (!any) return;
  const long long per_row = k >> 3;
  for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < per_row * n; v += (long long)gridDim.x * blockDim.x) {
    const int j = (int)(v / per_row), c = (int)(v - (long long)j * per_row);   // token, group of 8 values
    uint16_t *const row = planes + ((size_t)j * per_token + per_token - 3) * k + 8 * c;
    if (!force && !wide[j]) {
#pragma unroll
      for (int p = 0; p < 3; ++p) *(uint4 *)(row + (size_t)p * k) = make_uint4(0, 0, 0, 0);
      continue;
    }
    if (c == 0) tscale[j] = 1.f;
    const uint2 raw = *(const uint2 *)(q + (size_t)j * ld + 8 * c);
    const float s = sc[(size_t)j * lds + (c >> 1)];
    uint32_t t[3][4];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int qi = (int)(int8_t)(((i < 4 ? raw.x : raw.y) >> (8 * (i & 3))) & 0xFFu);
      float r = __fmul_rn((float)qi, s);
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        const float tp = __bfloat162float(__float2bfloat16_rn(r));   // 8 significant bits, round to nearest even
        const uint32_t h = __float_as_uint(tp) >> 16;
        if (i & 1) t[p][i >> 1] |= h << 16;
        else t[p][i >> 1] = h;
        r = __fsub_rn(r, tp);   // exact: the remainder has at most 16, then 8 significant bits
      }
    }
#pragma unroll
    for (int p = 0; p < 3; ++p) *(uint4 *)(row + (size_t)p * k) = make_uint4(t[p][0], t[p][1], t[p][2], t[p][3]);
  }
}

// The parts' sums of the tiles from nfull on (one per blockIdx.x) added in order, then the plain epilogue: a thread per row, a token per blockIdx.y.
__global__ void __launch_bounds__(256) w4a16_join_kernel(const float *partial_in, int parts, int width, int nfull, int m, int n, const Epilogue e) {
  pdl_launch_dependents();
  pdl_wait();
  const int tiles_m = (m + 255) / 256, t = nfull + blockIdx.x;
  const int i = t % tiles_m * 256 + threadIdx.x, j = t / tiles_m * width + blockIdx.y;
  if (j >= n) return;
  const size_t step = (size_t)width * 256;
  const float *const p = behind_wait(partial_in) + (size_t)blockIdx.x * parts * step + blockIdx.y * 256 + threadIdx.x;
  float amax = 0.f;
  if (i < m) {
    float s = p[0];
    for (int q = 1; q < parts; ++q) s = __fadd_rn(s, p[q * step]);
    const float v = epi_value(e, i, j, s, epi_scale(e, epi_row_part(e, i), epi_col_part(e, j)));
    store_dense(e.d_dtype, e.d, (size_t)j * e.ldd + i, v);
    amax = fabsf(v);
  }
  if (e.amax) warp_amax_commit(e.amax, amax);
}

}  // namespace

// tensor parallel: true when this kernel stores D into the peers' buffers itself (its output path is the TMA store)
bool gemm_w4a16_pushes(const GemmArgs &g) {
  if (g.tp.world <= 1) return false;
  const int esz = dense_bytes(g.e.d_dtype);
  const int drows = (g.x.mask & kExSwiglu) ? g.m / 2 : g.m;
  return esz == 2 && ((uintptr_t)g.e.d & 15) == 0 && ((size_t)g.e.ldd * esz) % 16 == 0 && ((size_t)drows * esz) % 16 == 0;
}

bool gemm_w4a16_supports(const GemmArgs &g) {
  // FP16 activations: E4M3 scales (UE5M3 products leave FP16's range) and a 16-bit D (the kernel's FP32 stores are for one sum over k)
  const bool f16 = g.B.dtype == NVFP4A_FP16 && !g.A.ue && g.e.d_dtype != NVFP4A_FP32;
  if ((g.B.dtype != NVFP4A_BF16 && !f16) || g.k < 64 || ((uintptr_t)g.B.data & 15) || g.B.ld % 8) return false;
  if (!g.A.image && (((uintptr_t)g.A.data & 15) || g.A.ld % 32 || ((uintptr_t)g.A.sc & 1))) return false;
  return true;
}

// The planes' memory comes from a pool of this library's own, one per device, that keeps what it has been given (release threshold
// at the maximum): a stream-ordered allocation from it costs microseconds and synchronises nothing, whereas the device's default
// pool hands its memory back at every synchronisation, so that a caller who synchronises once per step would pay a fresh
// allocation per call.  The pool holds the largest planes buffer in use so far until nvfp4a_b200_trim_scratch or process exit.
static std::atomic<cudaMemPool_t> g_planes_pool[64];
static cudaError_t planes_pool(cudaMemPool_t *pool) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  cudaMemPool_t p = g_planes_pool[dev & 63].load();
  if (!p) {
    cudaMemPoolProps props;
    memset(&props, 0, sizeof props);
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    e = cudaMemPoolCreate(&p, &props);
    if (e != cudaSuccess) return e;
    unsigned long long keep = ~0ull;
    cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
    cudaMemPool_t expected = nullptr;
    if (!g_planes_pool[dev & 63].compare_exchange_strong(expected, p)) {   // another thread was first: use its pool
      cudaMemPoolDestroy(p);
      p = expected;
    }
  }
  *pool = p;
  return cudaSuccess;
}
// The scratch of one call comes from the thread's allocator where it has set one (nvfp4a_b200_set_scratch_alloc: torch's, for the torch operators), else
// from the pool.  In a capture memory of the pool would be a node of the caller's graph, which then cannot be a child of another graph nor be
// instantiated twice: only calls that have no other kernel with a like result take it there (`in_capture`).
static thread_local ScratchAlloc g_scratch_alloc = {nullptr, nullptr};
void set_scratch_alloc(const ScratchAlloc &a) { g_scratch_alloc = a; }
ScratchAlloc get_scratch_alloc() { return g_scratch_alloc; }
static thread_local int g_last_parts = 0;
int last_parts() { return g_last_parts; }
struct Scratch { void *p; bool pooled; };
static Scratch take_scratch(size_t bytes, cudaStream_t s, bool in_capture) {
  if (g_scratch_alloc.fn) {
    void *const p = g_scratch_alloc.fn(g_scratch_alloc.ctx, bytes);
    return {((uintptr_t)p & 255) ? nullptr : p, false};
  }
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  cudaMemPool_t pool;
  void *p = nullptr;
  if ((!in_capture && (cudaStreamIsCapturing(s, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone)) || planes_pool(&pool) != cudaSuccess ||
      cudaMallocFromPoolAsync(&p, bytes, pool, s) != cudaSuccess) {
    (void)cudaGetLastError();
    return {nullptr, false};
  }
  return {p, true};
}
static cudaError_t give_scratch(const Scratch &t, cudaStream_t s) { return t.pooled ? cudaFreeAsync(t.p, s) : cudaSuccess; }

// the join behind a GEMM in parts of k
static cudaError_t launch_join(const W4A16Args &a, cudaStream_t s) {
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof cfg);
  cfg.gridDim = dim3((unsigned)((a.tiles - a.nfull) / a.parts), (unsigned)(a.width < a.n ? a.width : a.n), 1);
  cfg.blockDim = dim3(256, 1, 1);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = pdl_enabled() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, w4a16_join_kernel, (const float *)a.partial, a.parts, a.width, a.nfull, a.m, a.n, a.e);
}
cudaError_t trim_planes_pool() {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  cudaMemPool_t p = g_planes_pool[dev & 63].load();
  return p ? cudaMemPoolTrimTo(p, 0) : cudaSuccess;
}

// W4A8 on the tensor cores (see the header): from 64 tokens and 128 weight rows up, where the planes' set-up pays whatever the rest.  The call
// takes the planes from the pool above (stream-ordered: capturable, no synchronisation) and gives them back after the GEMM.
// Fewer tokens came from the DP4A kernel, whose ordered sums are more exact than one chain: they are summed in segments (three planes, a 16-bit D, the
// plain epilogue; nvfp4a_gemm_ex stays on the DP4A kernel, see GemmArgs::whole_k), and only where the reduction is long enough for that and for the planes to pay: 835 x 2176 on 30 tokens 158 us there, 30 here,
// 640 x 3840 on 10 tokens 267 and 41, 1024 x 512 on 32 tokens 49 and 17.
bool gemm_w4a8_tc_supports(const GemmArgs &g) {
  if (g.B.dtype != NVFP4A_INT8 || g.k < 64 || g.m < 128 || g.no_alloc || g.tp.world > 1 || g.e.gb_stride) return false;
  if (g.n < kW4A8ChainMinN && (g.n <= 8 || g.k < 512 || g.whole_k || g.e.d_dtype == NVFP4A_FP32 || g.x.mask || g.A.ue)) return false;
  if (((uintptr_t)g.B.data & 7) || g.B.ld % 8 || !g.B.s8 || ((uintptr_t)g.B.s8 & 3)) return false;
  if (!g.A.image && (((uintptr_t)g.A.data & 15) || g.A.ld % 32 || ((uintptr_t)g.A.sc & 1))) return false;
  return true;
}

// The same for nvfp4a_gemm_grouped: problems whose D is 16-bit (an FP32 D keeps the exact block sums of the DP4A kernel) and whose reduction
// is long enough to pay for the planes and for segments no less exact than the DP4A kernel's ordered sums (see the head of the file).  8
// experts of 2048 x 4096 on 1100 tokens, INT8 quantization of the tokens included: 602 us on the DP4A kernel, 96 us here.
bool gemm_w4a8_grouped_supports(const GemmArgs &g, int groups) {
  return g.n >= kW4A8ChainMinN && gemm_w4a8_tc_supports(g) && !g.A.image && groups <= kMaxGroups && g.k >= 512 && g.e.d_dtype != NVFP4A_FP32;
}

// seg == NULL: one weight; else `groups` stacked weights of g.m rows.  Without scratch nothing is launched and cudaErrorMemoryAllocation returned; up to
// 63 tokens, which the DP4A kernel takes as well, there is none from the pool in a capture.
cudaError_t launch_gemm_w4a8_tc(const GemmArgs &g, const int *seg, int groups, cudaStream_t s) {
  const bool three = seg || g.n < kW4A8ChainMinN;   // in segments
  const bool in_capture = g.n >= kW4A8ChainMinN;
  cudaError_t e = cudaSuccess;
  // planes [n][3 or 5][k], n token scales and the word behind them, n marks; the sums of parts of k, if there are any
  const int per_token = three ? 3 : 5;
  const size_t plane_bytes = (size_t)g.n * per_token * g.k * sizeof(uint16_t), small_bytes = (plane_bytes + (size_t)(g.n + 1) * sizeof(float) + g.n + 255) / 256 * 256;
  GemmArgs w = g;
  int parts = 1;
  const Plan p = seg ? Plan{} : plan_parts(g, three ? 3 : 2, false, &parts);
  Scratch scratch = {nullptr, false};
  if (parts > 1) {
    scratch = take_scratch(small_bytes + partial_bytes(p.tiles - p.nfull, parts, p.width), s, in_capture);
    if (!scratch.p) w.no_alloc = 1;   // k stays whole
  }
  if (!scratch.p) scratch = take_scratch(small_bytes, s, in_capture);
  if (!scratch.p) return cudaErrorMemoryAllocation;
  uint16_t *const planes = (uint16_t *)scratch.p;
  float *const tscale = (float *)((uint8_t *)planes + plane_bytes);
  uint8_t *const wide = (uint8_t *)(tscale + g.n + 1);
  const bool force = three || g.A.ue;   // three BF16 planes whatever the scales (products with UE5M3 scales leave FP16's range)
  // Each kernel starts while the one before it ends (a quantizer, usually) and waits for its results; the planes may still be in use by the GEMM before the
  // quantizer, which that one has waited for.
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof cfg);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = pdl_enabled() ? 1 : 0;
  if (!force) {
    cfg.gridDim = dim3((unsigned)g.n, 1, 1);
    cfg.blockDim = dim3(kPlanesThreads, 1, 1);
    e = cudaLaunchKernelEx(&cfg, w4a8_planes_kernel, (const int8_t *)g.B.data, g.B.ld, g.B.s8, g.B.lds8, g.k, planes, tscale, wide);
  }
  if (e == cudaSuccess) {
    cfg.gridDim = dim3(force ? (unsigned)(((long long)g.n * (g.k >> 3) + 255) / 256) : (unsigned)device_sms(), 1, 1);
    cfg.blockDim = dim3(256, 1, 1);
    e = cudaLaunchKernelEx(&cfg, w4a8_wide_planes_kernel, (const int8_t *)g.B.data, g.B.ld, g.B.s8, g.B.lds8, g.n, g.k, planes, per_token, tscale, (const uint8_t *)wide, force ? 1 : 0);
  }
  if (e == cudaSuccess) {
    W4A16Args a;
    CUtensorMap tw, tb, td;
    PeerMaps pm;
    memset(&pm, 0, sizeof pm);
    const uint64_t row_bytes = (uint64_t)g.k * per_token * sizeof(uint16_t);
    if (!set_up(w, three ? 3 : 2, false, seg ? groups : 0, planes, row_bytes, row_bytes, &a, &tw, &tb, &td)) e = cudaErrorInvalidValue;
    else {
      a.tscale = tscale;
      a.seg = seg; a.groups = groups;
      a.partial = (float *)((uint8_t *)planes + small_bytes);
      g_last_parts = a.parts;
      e = seg ? launch_cfg<3, false, true>(tw, tb, td, pm, a, s) : three ? launch_cfg<3, false>(tw, tb, td, pm, a, s) : launch_cfg<2, false>(tw, tb, td, pm, a, s);
      if (e == cudaSuccess && a.parts > 1) e = launch_join(a, s);
    }
  }
  const cudaError_t ef = give_scratch(scratch, s);
  return e != cudaSuccess ? e : ef;
}

cudaError_t launch_gemm_w4a16(const GemmArgs &g, cudaStream_t s) {
  W4A16Args a;
  CUtensorMap tw, tb, td;
  if (!set_up(g, 1, g.B.dtype == NVFP4A_FP16, 0, g.B.data, (uint64_t)g.k * 2, (uint64_t)g.B.ld * 2, &a, &tw, &tb, &td)) return cudaErrorInvalidValue;
  PeerMaps pm;
  memset(&pm, 0, sizeof pm);
  if (gemm_w4a16_pushes(g)) {   // tensor parallel: the epilogue's TMA stores also go to every peer's copy of D
    const int esz = dense_bytes(g.e.d_dtype);
    const bool glu = (g.x.mask & kExSwiglu) != 0;
    const int drows = glu ? g.m / 2 : g.m;
    for (int p = 0; p < g.tp.world; ++p) {
      if (p == g.tp.rank) continue;
      if (!make_tmap_dense(&pm.map[pm.n], (uint8_t *)g.e.d + g.tp.delta[p], esz, (uint64_t)drows, (uint64_t)g.n, (uint64_t)g.e.ldd * esz, 64, 32, 128))
        return cudaErrorInvalidValue;
      ++pm.n;
    }
  }
  auto go = [&]() { return g.B.dtype == NVFP4A_FP16 ? launch_cfg<1, true>(tw, tb, td, pm, a, s) : launch_cfg<1, false>(tw, tb, td, pm, a, s); };
  Scratch scratch = {nullptr, false};
  if (a.parts > 1) {
    scratch = take_scratch(partial_bytes(a.tiles - a.nfull, 1, a.width), s, false);
    a.partial = (float *)scratch.p;
    if (!scratch.p) {   // k stays whole
      GemmArgs whole = g;
      whole.no_alloc = 1;
      if (!set_up(whole, 1, g.B.dtype == NVFP4A_FP16, 0, g.B.data, (uint64_t)g.k * 2, (uint64_t)g.B.ld * 2, &a, &tw, &tb, &td)) return cudaErrorInvalidValue;
    }
  }
  g_last_parts = a.parts;
  if (a.parts == 1) return go();
  cudaError_t e = go();
  if (e == cudaSuccess) e = launch_join(a, s);
  const cudaError_t ef = give_scratch(scratch, s);
  return e != cudaSuccess ? e : ef;
}

}  // namespace nvb
