// Tensor-core GEMM (nine tokens and more, five to eight where reserved) from the packed B3 / D2 arenas on tcgen05 INT8.
//
//   Y[m,n] = a[m] * sum over (tile column j, plane p, group g) of s[n,j,p,g] * I[m,n,j,p,g],
//   I = sum over the 128 trits of the group of t * q          (exact int32)
//
// One persistent CTA per SM owns output tiles of 128 weight rows x TT tokens (TT = 32, 64, 128 or
// 256) and walks the K dimension in slabs of one (tile column, plane, scale group) = 128 trits:
//   * expander warps (one weight row per thread; a group of four warps builds a slab) keep several
//     tile-planes of packed words in flight with cp.async, turn them into int8 trits (see
//     b3_trits) and write the slab as a K-major, 128-byte-swizzled tile in shared memory (A operand,
//     UMMA M = 128).  EXP groups work on consecutive tile-planes at once;
//   * a copy warp loads the int8 activations of the tile column (B operand) by TMA from the scratch
//     written by the quantisation pre-pass, already in the expanders' k-slot order;
//   * two MMA warps issue four tcgen05.mma (kind::i8, N = TT, K = 32 each) per slab into a ring of TMEM
//     accumulators, one slab each of a 256-token tile's tile-planes, alternate tile-planes of a smaller
//     tile; the first MMA of a slab overwrites, so nothing has to be stored to TMEM;
//   * eight epilogue warps (one TMEM lane = one weight row per thread, half of the tile's tokens
//     each) read a finished accumulator, hand it back, and add the slab's exact integer sums times
//     the row's f16 group scale to fp32 running sums in their REGISTERS.
//
// What bounds it.  A 256-token tile: every slab costs the tensor core 512 clocks, and the drain one
// conversion and one multiply-add for each of its 32,768 sums (measured alone: 645 clocks with scalar
// FFMA, 733 with packed FFMA2, whose register pairs cost moves).  Conversions, byte permutes and logic
// share the ALU pipe at 2 clocks per warp: 423 such instructions per scheduler and slab, 847 of the
// about 1,580 clocks a slab takes (ncu: 1,060 instructions per scheduler and slab, issue slots 67 %).
// A smaller tile: the expansion, three groups at once (5120 x 17408, 2 planes, 16 tokens, ncu with cold
// caches: 59,500 clocks per CTA for 45 tile-planes, start, combine and outputs among them; issue
// slots 70 %, DRAM 13 %).
// Measured against the previous form (running sums and pre-loaded start values in TMEM, the
// expanders' loads word by word), 3 planes, 6912 x 2560, 2048 tokens: 217 -> 147 us; 2 planes,
// 34816 x 5120, 4096 tokens: 2,767 -> 1,768 us; 5120 x 17408, 16 tokens: 61 -> 37 us.  About a third of
// that came from the outputs: a load in front of every store cost 270 clocks per output.
//
// TMEM: kAccBufs accumulators of kAccCols columns.  All waits on barriers are bounded; a timeout sets
// TBF_WAIT_TIMEOUT and every role leaves its loop, the allocating warp frees TMEM, and the kernel
// returns.  The one wait that cannot be bounded, setmaxnreg's for registers, is ruled out before the
// launch (Tile::pool_holds).  No TMA multicast is used.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>

#include "tb_internal.h"

namespace {

constexpr int kRows = 128;        // weight rows per tile (UMMA M)
// Warps: 0 copies activations, 1-2 issue the MMAs (1 owns TMEM), 3 idle, 4-11 epilogue (lane quadrant =
// warp % 4; 4-7 take the first half of the tile's tokens, 8-11 the second), then the expanders.
constexpr int kFirstEpilogueWarp = 4, kEpilogueWarps = 8, kFirstExpandWarp = kFirstEpilogueWarp + kEpilogueWarps, kGroupWarps = 4;
constexpr uint32_t kTileABytes = kRows * 128;
constexpr uint32_t kStageBytes = 32 * 64;      // one tile-plane of an expander warp's 32 rows

// Per token tile.  A 256-token tile keeps 128 running sums in every epilogue thread, which leaves
// registers for two expander groups; smaller tiles are bound by the expansion and take three.
// Each group owns one slot of the A ring (the two slabs of a tile-plane).  `kDepth` tile-planes
// per expander warp are staged: with few tokens they come from HBM and need the bytes in flight,
// with many they mostly meet L2 and the activations need the shared memory.
template <int TT> struct Tile {
  static constexpr int kExpGroups = TT == 256 ? 2 : 3;
  static constexpr int kThreads = 32 * (kFirstExpandWarp + kGroupWarps * kExpGroups);
  // an accumulator holds one slab of a 256-token tile, the two slabs of a tile-plane of a smaller one
  static constexpr bool kSingle = TT == 256;
  static constexpr bool kMaySplit = !kSingle;   // a 256-token tile's sums are too many to pass through memory
  static constexpr int kAccBufs = TT >= 128 ? 2 : 4;
  static constexpr uint32_t kAccCols = kSingle ? TT : TT * 2;
  // "Weights are in shared memory" barriers and their counterparts.  256 tokens: one per slab, so that
  // a slab is written while the MMAs of its group's other slab run (with one per tile-plane the
  // expansion and the MMAs of a group took turns).  Else one per tile-plane; as the MMA warps take
  // alternate tile-planes there and a group's consecutive ones go to different warps, each warp gets
  // a "full" barrier of its own per group: a waiter that skips a phase could not tell two phases
  // apart by parity.
  static constexpr int kFullBars = 2 * kExpGroups, kEmptyBars = kSingle ? 2 * kExpGroups : kExpGroups;
  static constexpr int kDepth = TT >= 128 ? 2 : 3;
  // tile columns of activations in flight (two slabs each): a small tile's columns pass faster than a copy arrives
  static constexpr int kStagesB = TT == 32 ? 6 : TT == 64 ? 3 : 2;
  static constexpr uint32_t kTileBBytes = TT * 128;   // one slab of activations
  static constexpr size_t kSmem = 1024 + size_t(2 * kExpGroups) * kTileABytes + size_t(kStagesB) * 2 * kTileBBytes +
                                  size_t(kGroupWarps * kExpGroups) * kDepth * kStageBytes + size_t(kEpilogueWarps) * 32 * 4;
  // Registers follow the work: each role sets its share per thread with setmaxnreg.  The pool is what the
  // CTA got at launch, threads x the registers the compiler allotted (launch bounds: 96 per thread with
  // 640 threads, 80 with 768), and a setmaxnreg.inc waits without limit for registers that the others
  // have not given back, so the shares must add up to no more than the pool:
  //   TT = 256:  128 x 32 (copy, MMA, idle) + 256 x 160 (epilogue) + 256 x 64 (expanders) = 61,440  = 640 x 96
  //   else:      128 x 40 + 256 x 112 + 384 x 72                                          = 61,440  = 768 x 80
  // Another compiler or other flags may allot other counts: the launch asks the built kernel and is
  // refused unless pool_holds (a share below the launch count is given back, one above it is drawn).
  static constexpr int kControlRegs = TT == 256 ? 32 : 40, kEpilogueRegs = TT == 256 ? 160 : 112, kExpandRegs = TT == 256 ? 64 : 72;
  static constexpr bool pool_holds(int launch_regs) {
    return launch_regs >= kControlRegs && launch_regs >= kExpandRegs && launch_regs <= kEpilogueRegs &&
           32 * (kFirstEpilogueWarp * kControlRegs + kEpilogueWarps * kEpilogueRegs + kGroupWarps * kExpGroups * kExpandRegs) <= kThreads * launch_regs;
  }
};

constexpr uint32_t kSpin = 1u << 22;
constexpr uint32_t kBarEpilogue = 1;           // named barrier of all epilogue warps (split-K combine)
constexpr uint32_t kWaitCycles = 2000000000u;
constexpr uint32_t kMaxSplitTiles = 256;       // arrival counters the backend keeps for split output tiles

struct PrefillParams {
  const uint8_t* payload; const uint16_t* scales;
  const float* ascale;                         // token scales from the pre-pass
  void* y; int32_t* acc_dump; const float* row_scale; const float* residual;
  uint32_t* status;
  uint32_t m, m_pad, n, k, tpr, y_dtype;
  uint32_t n_tiles, m_tiles;
  // Split K: `splits` CTAs share an output tile, each walks a range of tile columns and leaves its
  // fp32 running sums in `partial` [split][m_pad][n] (m_pad: whole token tiles); the last of them to finish (a counter per
  // tile) adds the parts in split order and finishes the outputs.  splits == 1: none of this.
  uint32_t splits;
  float* partial; uint32_t* tile_counters;
};

// ---------------------------------------------------------------- PTX helpers
__device__ __forceinline__ uint32_t saddr(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t c) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(b)), "r"(c)); }
__device__ __forceinline__ void mbar_arrive(uint64_t* b) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(saddr(b)) : "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(saddr(b)), "r"(bytes) : "memory");
}
// Barriers by shared-memory address (one register) or by pointer.
__device__ __forceinline__ bool mbar_try(uint32_t b, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
               : "=r"(ok) : "r"(b), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_try(uint64_t* b, uint32_t parity) { return mbar_try(saddr(b), parity); }
__device__ __forceinline__ void mbar_arrive(uint32_t b) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(b) : "memory"); }
// Bounded wait.  After kWaitCycles SM clocks (about a second) it records TBF_WAIT_TIMEOUT and raises
// the CTA's abort flag; from then on NO wait in this CTA blocks any more: every role runs its
// loops to the end on whatever data is there (the host discards the result), so that all
// barrier arrivals still happen and the kernel ends.  The hardware suspends the waiting thread for up to
// kWaitHintNs per try, which leaves the issue slots to the warps that have work.
struct WaitCtx { volatile uint32_t* abort_flag; uint32_t* status; };
constexpr uint32_t kWaitHintNs = 20000;
__device__ __forceinline__ void mbar_wait(uint32_t b, uint32_t parity, const WaitCtx& ctx, uint32_t where) {
  if (mbar_try(b, parity)) return;
  const uint32_t t0 = clock();   // 32 bits: the limit is below one wrap, and registers are short here
  for (;;) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok) : "r"(b), "r"(parity), "r"(kWaitHintNs) : "memory");
    if (ok || *ctx.abort_flag) return;
    if (uint32_t(clock()) - t0 > kWaitCycles) {
      *ctx.abort_flag = 1;
      if (atomicOr(&ctx.status[TBS_FLAGS], TBF_WAIT_TIMEOUT) == 0) { ctx.status[TBS_INFO0] = parity; ctx.status[TBS_INFO1] = where; }
      return;
    }
  }
}
__device__ __forceinline__ void mbar_wait(uint64_t* b, uint32_t parity, const WaitCtx& ctx, uint32_t where) { mbar_wait(saddr(b), parity, ctx, where); }
__device__ __forceinline__ void named_sync(uint32_t id, uint32_t count) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory"); }
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r; asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel)); return r;
}
__device__ __forceinline__ uint32_t hfma2(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t r; asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c)); return r;
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(saddr(dst)), "l"(map), "r"(x), "r"(y), "r"(saddr(bar)) : "memory");
}
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(pred));
  return pred != 0;
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(saddr(bar)) : "memory");
}
// D[tmem] (+)= A[smem] * B[smem], int8 operands, int32 accumulate; the first K step of a slab overwrites.
// The descriptors differ in their low words only.
constexpr uint32_t kDescHigh = (1024u >> 4) | (1u << 14) | (2u << 29);   // stride 1024 bytes, descriptor version 1, 128-byte swizzle
__device__ __forceinline__ void tc_mma_i8(uint32_t d_tmem, uint32_t adesc, uint32_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n .reg .b64 da, db;\n mov.b64 da, {%1, %6};\n mov.b64 db, {%2, %6};\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::i8 [%0], da, db, %3, {%5, %5, %5, %5}, p;\n}\n"
      ::"r"(d_tmem), "r"(adesc), "r"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u), "n"(kDescHigh) : "memory");
}
#define TB_R16(a, o) "=r"(a[o+0]), "=r"(a[o+1]), "=r"(a[o+2]), "=r"(a[o+3]), "=r"(a[o+4]), "=r"(a[o+5]), "=r"(a[o+6]), "=r"(a[o+7]), \
                     "=r"(a[o+8]), "=r"(a[o+9]), "=r"(a[o+10]), "=r"(a[o+11]), "=r"(a[o+12]), "=r"(a[o+13]), "=r"(a[o+14]), "=r"(a[o+15])
// 32 lanes x 16 columns of 32 bits: this thread's lane, 16 consecutive columns
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : TB_R16(r, 0) : "r"(taddr) : "memory");
}
#define TB_U8(a, o) "+r"(a[o+0]), "+r"(a[o+1]), "+r"(a[o+2]), "+r"(a[o+3]), "+r"(a[o+4]), "+r"(a[o+5]), "+r"(a[o+6]), "+r"(a[o+7])
// waits for every TMEM load of the thread; the registers of the one in question are operands, so that no use moves in front
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&r)[16]) { asm volatile("tcgen05.wait::ld.sync.aligned;" : TB_U8(r, 0), TB_U8(r, 8)::"memory"); }
__device__ __forceinline__ void lds128(uint32_t addr, uint32_t* v) {
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(addr));
}

// Low word of a shared-memory matrix descriptor: K-major tile of 128-byte rows, 128-byte swizzle, 8-row
// groups 1024 bytes apart (start address in 16-byte units; the leading byte offset is unused for
// swizzled K-major).  Adding 2 selects the next 32-byte K slice inside the swizzled row.
__device__ __forceinline__ uint32_t smem_desc(uint32_t addr) { return ((addr & 0x3ffffu) >> 4) | (1u << 16); }
// Instruction descriptor: s32 accumulate, A/B formats, K-major both, N, M.
__host__ __device__ constexpr uint32_t instr_desc_n(uint32_t n) {
  return (2u << 4)                    // s32 accumulator
         | (1u << 7) | (1u << 10)     // A and B are signed 8-bit
         | ((n >> 3) << 17) | ((uint32_t(kRows) >> 4) << 24);
}

// ---------------------------------------------------------------- k-slot order of a slab
// Trit (0..255 of its tile) in k-slot s (slab 0: slots 0..127, slab 1: 128..255); see the expander.
// Packed words are laid out digit-major (quad 5w + i = digit i of the word's four bytes); B3 words
// 6 (bytes 24..27, which straddles the scale groups) and 12 (bytes 48..51, four padding digits) in
// the order that takes the fewest byte permutes.
__host__ __device__ constexpr uint32_t b3_trit(uint32_t byte, uint32_t digit) { return 5 * byte + digit; }
__host__ __device__ constexpr uint32_t b3_trit_of_slot(uint32_t s) {
  const uint32_t quad = s >> 2, e = s & 3;
  if (quad < 30) return b3_trit(4 * (quad / 5) + e, quad % 5);                     // words 0..5
  if (quad == 30) return b3_trit(24 + (e & 1), e >> 1);                            // (24,25) x digits 0, 1
  if (quad == 31) return e < 2 ? b3_trit(24 + e, 2) : b3_trit(24, 1 + e);          // digit 2 of both, digits 3, 4 of byte 24
  if (quad < 34) return b3_trit(26 + (e & 1), 2 * (quad - 32) + (e >> 1));         // (26,27) x digits 0, 1 and 2, 3
  if (quad == 34) return e < 3 ? b3_trit(25 + e, 4) : b3_trit(25, 3);
  if (quad < 60) return b3_trit(4 * (7 + (quad - 35) / 5) + e, (quad - 35) % 5);   // words 7..11
  if (quad == 60) return b3_trit(48 + e, 0);
  return e < 3 ? b3_trit(48 + e, quad - 60) : b3_trit(48 + (quad - 61), 4);
}
__host__ __device__ constexpr uint32_t d2_trit_of_slot(uint32_t s) {
  const uint32_t quad = s >> 2, e = s & 3;   // quad 4w + i = slot i of the word's four bytes
  return 16 * (quad >> 2) + 4 * e + (quad & 3);
}
template <int CODEC> struct alignas(16) SlotTable {
  uint8_t trit[256];
  constexpr SlotTable() : trit{} {
    for (uint32_t s = 0; s < 256; ++s) trit[s] = uint8_t(CODEC == tbf::kB3 ? b3_trit_of_slot(s) : d2_trit_of_slot(s));
  }
};
template <int CODEC> constexpr bool slots_are_a_permutation() {
  const SlotTable<CODEC> t;
  bool seen[256] = {};
  for (uint32_t s = 0; s < 256; ++s) {
    if (seen[t.trit[s]] || (t.trit[s] >> 7) != (s >> 7)) return false;   // every trit once, in its own group's slab
    seen[t.trit[s]] = true;
  }
  return true;
}
static_assert(slots_are_a_permutation<tbf::kB3>() && slots_are_a_permutation<tbf::kD2>(), "k-slot order");
// In global memory: every lane wants another entry, which constant memory would hand out one at a time.
__device__ const SlotTable<tbf::kB3> d_b3_slots{};
__device__ const SlotTable<tbf::kD2> d_d2_slots{};

// ---------------------------------------------------------------- quantisation pre-pass
struct QuantParams {
  const void* x; const float* act_scale_in; const float* act_absmax_in;
  const float* relu2_up;   // squared-ReLU gate (x fp32): activation = (max(x, 0)^2) * relu2_up; null = none
  int8_t* qperm; float* ascale;
  uint32_t m, k, x_dtype, codec;
  uint32_t vec;            // x starts on a 16-byte boundary, and so does each row: eight values per load (the gate is read value by value)
  uint32_t* status;
};

// Eight consecutive activations starting at element `at`, as fp32 (int8 codes as their values).
__device__ __forceinline__ void load_act8(const QuantParams& p, size_t at, float (&v)[8]) {
  if (p.vec) {
    if (p.x_dtype == TB_F32) {
      const float4 a = __ldg(reinterpret_cast<const float4*>(p.x) + at / 4), b = __ldg(reinterpret_cast<const float4*>(p.x) + at / 4 + 1);
      v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else if (p.x_dtype == TB_BF16) {
      const uint4 u = __ldg(reinterpret_cast<const uint4*>(p.x) + at / 8);
      const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) { v[2 * i] = __uint_as_float(w[i] << 16); v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u); }
    } else {
      const uint2 u = __ldg(reinterpret_cast<const uint2*>(p.x) + at / 8);
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = float(int(int8_t((i < 4 ? u.x : u.y) >> (8 * (i & 3)))));
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      v[i] = p.x_dtype == TB_F32 ? static_cast<const float*>(p.x)[at + i]
             : p.x_dtype == TB_BF16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(p.x)[at + i])
                                    : float(static_cast<const int8_t*>(p.x)[at + i]);
  }
  if (p.relu2_up) {   // (max(g, 0)^2) * u with the reference's association and no contraction
#pragma unroll
    for (int i = 0; i < 8; ++i) { const float r = fmaxf(v[i], 0.0f); v[i] = __fmul_rn(__fmul_rn(r, r), p.relu2_up[at + i]); }
  }
}

// One CTA per token: per-token absmax, int8 codes, the codes in k-slot order.  Bound by latency: the
// second reading of the row meets L1 / L2.  Every thread takes eight consecutive activations per step
// (one 16-byte load of bf16), the codes change order through shared memory and leave as whole words;
// rows of few tokens take 1,024 threads so that a row is two or three steps.  (Byte by byte, with
// 256 threads: 13.3 us for 16 tokens of 17,408, 42.7 us for 4,096 of 5,120.)
template <int THREADS>
__global__ void __launch_bounds__(THREADS) prefill_quant_kernel(const QuantParams p) {
  constexpr uint32_t kChunk = THREADS * 8;
  __shared__ float red[THREADS / 32];
  __shared__ __align__(16) uint8_t codes[2][kChunk];
  __shared__ __align__(16) uint8_t slots[256];
  // The tensor-core kernel behind this one may start now: its expanders do not depend on the
  // activations, only its copy warp and its stores wait (griddepcontrol.wait) for this grid.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const uint32_t t = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t* qrow = reinterpret_cast<uint32_t*>(p.qperm + size_t(t) * p.k);
  if (t >= p.m) {   // padding tokens: zero codes
    for (uint32_t i = tid; i < p.k / 4; i += THREADS) qrow[i] = 0u;
    if (tid == 0) p.ascale[t] = 0.f;
    return;
  }
  if (tid < 64) reinterpret_cast<uint32_t*>(slots)[tid] = __ldg(reinterpret_cast<const uint32_t*>(p.codec == tbf::kB3 ? d_b3_slots.trit : d_d2_slots.trit) + tid);
  const size_t row = size_t(t) * p.k;
  float scale_q = 1.f;
  if (p.x_dtype != TB_I8) {
    float gamma;
    if (p.act_absmax_in) gamma = p.act_absmax_in[t];
    else {
      float mx = 0.f;
      for (uint32_t i = tid * 8; i < p.k; i += kChunk) {
        float v[8];
        load_act8(p, row + i, v);
#pragma unroll
        for (int e = 0; e < 8; ++e) mx = fmaxf(mx, fabsf(v[e]));
      }
      for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      if (lane == 0) red[warp] = mx;
      __syncthreads();
      gamma = 0.f;
#pragma unroll
      for (int w = 0; w < THREADS / 32; ++w) gamma = fmaxf(gamma, red[w]);
    }
    scale_q = gamma > 0.f ? __fdiv_rn(127.0f, gamma) : 0.f;
    if (tid == 0) p.ascale[t] = __fdiv_rn(gamma, 127.0f);
  } else if (tid == 0) {
    p.ascale[t] = p.act_scale_in[t];
  }
  uint32_t buf = 0;
  for (uint32_t base = 0; base < p.k; base += kChunk, buf ^= 1) {
    const uint32_t i = base + tid * 8;
    if (i < p.k) {
      float v[8];
      load_act8(p, row + i, v);
      uint32_t packed[2] = {0u, 0u};
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        int q;
        if (p.x_dtype == TB_I8) q = int(v[e]);
        else {
          // a NaN would clamp to a finite code: report non-finite activations instead
          if (!(fabsf(v[e]) <= 3.402823466e+38f) && atomicOr(&p.status[TBS_FLAGS], TBF_NONFINITE_ACT) == 0) {
            p.status[TBS_INFO0] = uint32_t(t * p.k + i + e); p.status[TBS_INFO1] = __float_as_uint(v[e]);
          }
          q = int(fminf(127.f, fmaxf(-128.f, rintf(__fmul_rn(v[e], scale_q)))));
        }
        packed[e >> 2] |= uint32_t(q & 0xff) << (8 * (e & 3));
      }
      *reinterpret_cast<uint2*>(codes[buf] + tid * 8) = make_uint2(packed[0], packed[1]);
    }
    __syncthreads();   // the other buffer is written next: one barrier per chunk
    const uint32_t words = min(kChunk, p.k - base) / 4;
    for (uint32_t o = tid; o < words; o += THREADS) {
      const uint32_t at = *reinterpret_cast<const uint32_t*>(slots + 4 * (o & 63));
      const uint8_t* tile = codes[buf] + 256 * (o >> 6);
      qrow[base / 4 + o] = uint32_t(tile[at & 255u]) | uint32_t(tile[(at >> 8) & 255u]) << 8 | uint32_t(tile[(at >> 16) & 255u]) << 16 |
                           uint32_t(tile[at >> 24]) << 24;
    }
  }
}

// ---------------------------------------------------------------- weight expansion
// B3 word (four bytes) -> five registers of int8 trits: digit i - 1 of bytes 0..3 in byte lanes 0..3.
//
// The quotients q_i = floor(b / 3^i) come from a half-precision FMA chain on 1024 + b: the rounding of
// the FMA does the floor, every result is an integer below 2048.  d_i = q_i - 3 q_(i+1) is then one
// 32-bit multiply-add for all four bytes.  The halves hold bytes (0,2) and (1,3), so that
// P_i = A_i + 256 B_i packs a quotient register, and every half carries an offset of its own such
// that P_i = q_i + C_i with 3 C_(i+1) = C_i - 0x7F7F7F7F (mod 2^32, C_0 = 0 as P_0 is the word
// itself): each multiply-add then leaves d_i + 127 in every lane, and one exclusive-or with 0x80
// turns {127, 128, 129} into the int8 values {-1, 0, 1}.  Two's-complement trits cost one
// instruction per four of them here, where correcting the sums of unsigned digits would cost one per
// sum in the drain.  The constants were found by exhaustive search over the multiplier and the addend
// for each offset and checked for every byte value.
__device__ __forceinline__ void b3_trits(uint32_t w, uint32_t (&r)[5]) {
  const uint32_t a0 = (w & 0x00ff00ffu) | 0x64006400u, b0 = prmt(w, 0x64646464u, 0x4341u);
  const uint32_t a1 = hfma2(a0, 0x35553555u, 0x623761abu), b1 = hfma2(b0, 0x35553555u, 0x62e1618du);
  const uint32_t a2 = hfma2(a0, 0x2f192f19u, 0x64466472u), b2 = hfma2(b0, 0x2f192f19u, 0x646263a8u);
  const uint32_t a3 = hfma2(a1, 0x2f192f1cu, 0x63f76400u), b3 = hfma2(b1, 0x2f1a2f18u, 0x64516435u);
  const uint32_t a4 = hfma2(a2, 0x2f1a2f22u, 0x6313641cu), b4 = hfma2(b2, 0x2f1f2f1cu, 0x64516451u);
  const uint32_t p1 = a1 + 256u * b1, p2 = a2 + 256u * b2, p3 = a3 + 256u * b3, p4 = a4 + 256u * b4;
  r[0] = (w - 3u * p1) ^ 0x80808080u;
  r[1] = (p1 - 3u * p2) ^ 0x80808080u;
  r[2] = (p2 - 3u * p3) ^ 0x80808080u;
  r[3] = (p3 - 3u * p4) ^ 0x80808080u;
  r[4] = (p4 + 0x400a4fd7u) ^ 0x80808080u;   // 0x7F7F7F7F - C_4
}
// 2-bit codes t + 1 in slot `s` of a D2 word's four bytes -> int8 trits (same last step)
__device__ __forceinline__ uint32_t d2_trits(uint32_t w, int s) { return (((w >> (2 * s)) & 0x03030303u) + 0x7f7f7f7fu) ^ 0x80808080u; }
// store 16 bytes = quads 4*chunk .. 4*chunk+3 of a row into a swizzled K-major tile (row_xor = (row % 8) * 16)
__device__ __forceinline__ void store_chunk(uint32_t row_base, uint32_t row_xor, uint32_t chunk, uint32_t q0, uint32_t q1, uint32_t q2, uint32_t q3) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(row_base + ((chunk << 4) ^ row_xor)), "r"(q0), "r"(q1), "r"(q2), "r"(q3) : "memory");
}

// work item = (row tile, token tile, K split); a split walks tile columns [j0, j1)
__device__ __forceinline__ void split_range(const PrefillParams& p, uint32_t tile, uint32_t& j0, uint32_t& j1) {
  const uint32_t sp = tile % p.splits;
  j0 = uint32_t(uint64_t(p.tpr) * sp / p.splits);
  j1 = uint32_t(uint64_t(p.tpr) * (sp + 1) / p.splits);
}

// ---------------------------------------------------------------- roles
// Copy warp: the int8 activations of a tile column (two slabs of TT x 128 bytes).
template <int TT>
__device__ __forceinline__ void copy_role(const PrefillParams& p, const CUtensorMap& map_q, uint32_t tiles, uint8_t* tile_b, uint64_t* b_full,
                                          uint64_t* b_empty, const WaitCtx& wctx, uint32_t lane) {
  constexpr uint32_t kTileBBytes = Tile<TT>::kTileBBytes;
  // launched with programmatic stream serialisation: everything this warp loads was written by
  // the quantisation pre-pass, the previous grid on the stream
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (lane != 0) return;
  uint32_t fill = 0;
  for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const uint32_t mt = (tile / p.splits) % p.m_tiles;
    uint32_t j0, j1;
    split_range(p, tile, j0, j1);
    for (uint32_t j = j0; j < j1; ++j, ++fill) {
      const uint32_t s = fill % Tile<TT>::kStagesB, round = fill / Tile<TT>::kStagesB;
      if (round > 0) mbar_wait(&b_empty[s], (round - 1) & 1, wctx, 300);
      mbar_expect_tx(&b_full[s], 2 * kTileBBytes);
      for (int gsel = 0; gsel < 2; ++gsel)
        tma_load_2d(tile_b + (s * 2 + gsel) * kTileBBytes, &map_q, int((2 * j + gsel) * 128), int(mt * TT), &b_full[s]);
    }
  }
  // copies in flight must land before the CTA's shared memory goes away
  for (uint32_t back = 0; back < uint32_t(Tile<TT>::kStagesB) && back < fill; ++back) {
    const uint32_t f = fill - 1 - back;
    for (uint32_t i = 0; i < kSpin && !mbar_try(&b_full[f % Tile<TT>::kStagesB], (f / Tile<TT>::kStagesB) & 1); ++i) {}
  }
}

// Two MMA warps.  A step of the chain wait - wait - issue - commit takes a warp several hundred clocks
// whatever the MMAs cost, so one warp could not keep the tensor core fed: with a 256-token tile each
// warp takes one slab of every tile-plane (and the accumulator of that slab), with smaller tiles the
// warps take alternate tile-planes (one wait for the weights, one for the accumulator and eight MMAs
// per tile-plane).  The whole warp walks the loop (so that addresses and descriptors stay in uniform
// registers); one elected lane issues.
template <int PLANES, int TT>
__device__ __forceinline__ void mma_role(const PrefillParams& p, uint32_t tiles, uint32_t tmem_base, uint32_t which, uint8_t* tile_a,
                                         uint8_t* tile_b, uint64_t* a_full, uint64_t* a_empty, uint64_t* b_full, uint64_t* b_empty,
                                         uint64_t* acc_full, uint64_t* acc_empty, const WaitCtx& wctx) {
  using T = Tile<TT>;
  constexpr uint32_t kIdesc = instr_desc_n(TT);
  constexpr uint32_t kSlabA = kTileABytes >> 4, kSlabB = T::kTileBBytes >> 4;   // descriptor start addresses are in 16-byte units
  const uint32_t first = T::kSingle ? which : 0u;
  const uint32_t a_desc0 = smem_desc(saddr(tile_a)) + first * kSlabA, b_desc0 = smem_desc(saddr(tile_b)) + first * kSlabB;
  uint32_t grp = 0, full = 0, pa = 0, buf = first, pacc = 1, sb = 0, pb = 0;   // ring positions, parities to wait for
  uint32_t turn = 0;
  for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    uint32_t j0, j1;
    split_range(p, tile, j0, j1);
    for (uint32_t j = j0; j < j1; ++j) {
      mbar_wait(&b_full[sb], pb, wctx, 301);
#pragma unroll 1
      for (uint32_t pl = 0; pl < PLANES; ++pl) {
        if (T::kSingle || turn == which) {
          const uint32_t a_desc = a_desc0 + 2 * grp * kSlabA, b_desc = b_desc0 + 2 * sb * kSlabB;
          mbar_wait(&a_full[T::kSingle ? 2 * grp + which : full], pa, wctx, 302);
          mbar_wait(&acc_empty[buf], pacc, wctx, 303);   // passes at once while the ring is first filled
          tc_fence_after();
          if (elect_one()) {
#pragma unroll
            for (uint32_t g = 0; g < (T::kSingle ? 1u : 2u); ++g)
#pragma unroll
              for (uint32_t kc = 0; kc < 4; ++kc)
                tc_mma_i8(tmem_base + buf * T::kAccCols + g * TT, a_desc + g * kSlabA + 2 * kc, b_desc + g * kSlabB + 2 * kc, kIdesc, kc > 0 ? 1u : 0u);
            tc_commit(&acc_full[buf]);
            tc_commit(&a_empty[T::kSingle ? 2 * grp + which : grp]);
          }
          __syncwarp();
        }
        turn ^= 1u;
        if (++grp == uint32_t(T::kExpGroups)) { grp = 0; if (T::kSingle) pa ^= 1; }
        if (!T::kSingle && ++full == uint32_t(T::kFullBars)) { full = 0; pa ^= 1; }
        if (T::kSingle) pacc ^= 1;   // a warp's own accumulator, once per tile-plane
        else if (++buf == uint32_t(T::kAccBufs)) { buf = 0; pacc ^= 1; }
      }
      if (elect_one()) tc_commit(&b_empty[sb]);
      __syncwarp();
      if (++sb == uint32_t(T::kStagesB)) { sb = 0; pb ^= 1; }
    }
  }
}

// Expander warps (groups of four: one lane per weight row of the 128-row slab).  Group g expands the
// tile-planes whose running number is g modulo EXP into its own slot of the A ring (two slabs).
//
// Rows are hundreds of bytes apart in the arena, so a lane that fetched its own row word by word
// would touch one sector per load.  Instead a warp copies its 32 rows' words of a tile-plane with
// cp.async, 16 bytes per lane and eight rows per instruction, into a staging area of its own, kDepth
// tile-planes deep, and every lane picks up its row with four 16-byte loads (chunks permuted by row:
// no bank conflicts).  A D2 tile-plane is 64 aligned bytes.  A B3 tile-plane is 52 bytes on a 4-byte
// boundary: the 64 bytes from the 16-byte boundary below it hold it, and two selects per word take
// it out.  (Word copies, two rows per instruction, kept a warp 560 clocks in the load / store queue
// where these take under 150, and every barrier access of the CTA queued behind them.)
template <int CODEC, int PLANES, int TT>
__device__ __forceinline__ void expander_role(const PrefillParams& p, uint32_t tiles, uint32_t wexp_all, uint32_t lane, uint8_t* tile_a_ptr,
                                              uint8_t* stage_ptr, uint64_t* a_full, uint64_t* a_empty, const WaitCtx& wctx) {
  using T = Tile<TT>;
  constexpr int EXP = T::kExpGroups, kDepth = T::kDepth;
  constexpr uint32_t kWords = CODEC == tbf::kB3 ? 13 : 16, kPlaneBytes = 4 * kWords;
  const uint32_t grp = wexp_all / kGroupWarps, wexp = wexp_all % kGroupWarps, r = wexp * 32 + lane;
  const uint32_t stage = saddr(stage_ptr) + wexp_all * (kDepth * kStageBytes);
  const size_t row_bytes = size_t(p.tpr) * PLANES * kPlaneBytes;
  constexpr uint32_t kRowsPerIt = 8, kIts = 4;
  const uint32_t lrow = lane >> 2, lpart = lane & 3;
  const uint32_t dst0 = stage + lrow * 64 + ((lpart ^ ((lrow >> 1) & 3u)) << 4);
  uint32_t total = 0;   // tile-planes this CTA expands over all its work items
  for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    uint32_t j0, j1;
    split_range(p, tile, j0, j1);
    total += (j1 - j0) * PLANES;
  }
  // ---- the feed: next tile-plane to copy, `feed_i` of `feed_count` of work item `feed_tile`
  uint32_t feed_tile = blockIdx.x, feed_i = grp, feed_count = 0;
  bool feed_whole = false;
  const uint8_t* feed_ptr = nullptr;   // first byte of this lane's first row in the item's tile-plane 0
  uint32_t feed_row = 0;
  uint32_t lane_mis = 0, mis = 0;      // B3: words between the 16-byte boundary and the lane's row in tile-plane 0; two bits per slot
  const uint32_t feed_last = p.n - 1;
  const size_t row_step = kRowsPerIt * row_bytes;
  const auto copy_part = [&](uint32_t dst, const uint8_t* src) {
    const uintptr_t from = (reinterpret_cast<uintptr_t>(src) & ~uintptr_t(15)) + lpart * 16;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(from) : "memory");
  };
  const auto open_item = [&]() {
    uint32_t j0, j1;
    split_range(p, feed_tile, j0, j1);
    feed_count = (j1 - j0) * PLANES;
    feed_row = feed_tile / (p.m_tiles * p.splits) * kRows + wexp * 32;
    feed_whole = feed_row + 31 < p.n;
    feed_ptr = p.payload + size_t(min(feed_row + lrow, feed_last)) * row_bytes + size_t(j0 * PLANES) * kPlaneBytes;
    lane_mis = min(feed_row + lane, feed_last) * (p.tpr * PLANES) + j0 * PLANES;   // 13 words per tile-plane: 13 = 1 (mod 4)
  };
  const auto feed = [&](uint32_t slot) {
    while (feed_tile < tiles && feed_i >= feed_count) {
      feed_i -= feed_count;
      feed_tile += gridDim.x;
      if (feed_tile < tiles) open_item();
    }
    if (feed_tile < tiles) {
      const uint32_t dst = dst0 + slot * kStageBytes;
      const uint8_t* src = feed_ptr + feed_i * kPlaneBytes;
      mis = (mis & ~(3u << (2 * slot))) | (((lane_mis + feed_i) & 3u) << (2 * slot));
      if (feed_whole) {
#pragma unroll
        for (uint32_t it = 0; it < kIts; ++it, src += row_step) copy_part(dst + it * (kRowsPerIt * 64), src);
      } else {   // rows past the end repeat the last row; never stored
#pragma unroll 1
        for (uint32_t it = 0; it < kIts; ++it)
          copy_part(dst + it * (kRowsPerIt * 64), src + size_t(min(it * kRowsPerIt, feed_last - min(feed_row + lrow, feed_last))) * row_bytes);
      }
    }
    feed_i += EXP;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  open_item();
#pragma unroll
  for (int d = 0; d < kDepth - 1; ++d) feed(d);
  const uint32_t t0 = saddr(tile_a_ptr) + 2 * grp * kTileABytes + r * 128, t1 = t0 + kTileABytes, rx = (r & 7u) << 4;
  uint32_t slot = 0, parity = 1;   // the wait before the first use of the ring slot passes at once
  for (uint32_t seq = grp; seq < total; seq += EXP, parity ^= 1) {
    feed(slot == 0 ? kDepth - 1 : slot - 1);
    asm volatile("cp.async.wait_group %0;" ::"n"(kDepth - 1) : "memory");
    __syncwarp();
    uint32_t w[kWords];
    {
      uint32_t v[16];
      const uint32_t from = stage + slot * kStageBytes + lane * 64;
#pragma unroll
      for (uint32_t i = 0; i < 4; ++i) lds128(from + ((i ^ ((lane >> 1) & 3u)) << 4), &v[4 * i]);
      if (CODEC == tbf::kB3) {
        const bool two = (mis >> (2 * slot)) & 2u, one = (mis >> (2 * slot)) & 1u;
#pragma unroll
        for (uint32_t i = 0; i < 14; ++i) v[i] = two ? v[i + 2] : v[i];
#pragma unroll
        for (uint32_t i = 0; i < 13; ++i) w[i] = one ? v[i + 1] : v[i];
      } else {
#pragma unroll
        for (uint32_t i = 0; i < kWords; ++i) w[i] = v[i];
      }
    }
    __syncwarp();   // the slot may be overwritten
    if (++slot == uint32_t(kDepth)) slot = 0;
    mbar_wait(a_empty + (T::kSingle ? 2 * grp : grp), parity, wctx, 304);
    if (CODEC == tbf::kB3) {
      uint32_t d[5], e[5], f[5], g[5];
      b3_trits(w[0], d); b3_trits(w[1], e); b3_trits(w[2], f); b3_trits(w[3], g);
      store_chunk(t0, rx, 0, d[0], d[1], d[2], d[3]);
      store_chunk(t0, rx, 1, d[4], e[0], e[1], e[2]);
      store_chunk(t0, rx, 2, e[3], e[4], f[0], f[1]);
      store_chunk(t0, rx, 3, f[2], f[3], f[4], g[0]);
      store_chunk(t0, rx, 4, g[1], g[2], g[3], g[4]);
      b3_trits(w[4], d); b3_trits(w[5], e); b3_trits(w[6], f);
      store_chunk(t0, rx, 5, d[0], d[1], d[2], d[3]);
      store_chunk(t0, rx, 6, d[4], e[0], e[1], e[2]);
      store_chunk(t0, rx, 7, e[3], e[4], prmt(f[0], f[1], 0x5410u), prmt(prmt(f[2], f[3], 0x0410u), f[4], 0x4210u));
      if (T::kSingle) {   // the first slab is complete; the second one's slot
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(a_full + 2 * grp);
        mbar_wait(a_empty + 2 * grp + 1, parity, wctx, 305);
      }
      b3_trits(w[7], d); b3_trits(w[8], e);
      store_chunk(t1, rx, 0, prmt(f[0], f[1], 0x7632u), prmt(f[2], f[3], 0x7632u), prmt(f[4], f[3], 0x5321u), d[0]);
      store_chunk(t1, rx, 1, d[1], d[2], d[3], d[4]);
      b3_trits(w[9], f); b3_trits(w[10], g);
      store_chunk(t1, rx, 2, e[0], e[1], e[2], e[3]);
      store_chunk(t1, rx, 3, e[4], f[0], f[1], f[2]);
      store_chunk(t1, rx, 4, f[3], f[4], g[0], g[1]);
      b3_trits(w[11], d); b3_trits(w[12], e);
      store_chunk(t1, rx, 5, g[2], g[3], g[4], d[0]);
      store_chunk(t1, rx, 6, d[1], d[2], d[3], d[4]);
      store_chunk(t1, rx, 7, e[0], prmt(e[1], e[4], 0x4210u), prmt(e[2], e[4], 0x5210u), prmt(e[3], e[4], 0x6210u));
    } else {
#pragma unroll
      for (uint32_t c = 0; c < 8; ++c) store_chunk(t0, rx, c, d2_trits(w[c], 0), d2_trits(w[c], 1), d2_trits(w[c], 2), d2_trits(w[c], 3));
      if (T::kSingle) {   // the first slab is complete; the second one's slot
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(a_full + 2 * grp);
        mbar_wait(a_empty + 2 * grp + 1, parity, wctx, 305);
      }
#pragma unroll
      for (uint32_t c = 0; c < 8; ++c)
        store_chunk(t1, rx, c, d2_trits(w[8 + c], 0), d2_trits(w[8 + c], 1), d2_trits(w[8 + c], 2), d2_trits(w[8 + c], 3));
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) mbar_arrive(a_full + (T::kSingle ? 2 * grp + 1 : seq % T::kFullBars));
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// Sixteen outputs of a row, tokens tok0 .. tok0 + 15: token scale, optional row scale and residual, store.
// Everything that is loaded is asked for before the first store, so that a chunk costs one latency
// (a load in front of every store cost 270 clocks per output).
__device__ __forceinline__ void finish_outputs(const PrefillParams& p, const float* sum, uint32_t tok0, uint32_t n, float rs) {
  const float4* a4 = reinterpret_cast<const float4*>(p.ascale + tok0);   // padded to whole token tiles
  float a[16];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 v = __ldg(a4 + i);
    a[4 * i] = v.x; a[4 * i + 1] = v.y; a[4 * i + 2] = v.z; a[4 * i + 3] = v.w;
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    a[i] = __fmul_rn(sum[i], a[i]);
    if (p.row_scale) a[i] = __fmul_rn(a[i], rs);
  }
  const size_t at = size_t(tok0) * p.n + n;
  if (p.residual) {
#pragma unroll
    for (int h = 0; h < 16; h += 8) {
      float res[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) res[i] = tok0 + h + i < p.m ? __ldg(p.residual + at + size_t(h + i) * p.n) : 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) a[h + i] = __fadd_rn(res[i], a[h + i]);
    }
  }
  if (p.y_dtype == TB_F32) {
    float* y = static_cast<float*>(p.y) + at;
#pragma unroll
    for (int i = 0; i < 16; ++i, y += p.n)
      if (tok0 + i < p.m) *y = a[i];
  } else {
    __nv_bfloat16* y = static_cast<__nv_bfloat16*>(p.y) + at;
#pragma unroll
    for (int i = 0; i < 16; ++i, y += p.n)
      if (tok0 + i < p.m) *y = __float2bfloat16_rn(a[i]);
  }
}

// Epilogue warps: TMEM lane = weight row, running sums of half the tile's tokens in registers.
template <int PLANES, int TT, bool DUMP>
__device__ __forceinline__ void epilogue_role(const PrefillParams& p, uint32_t tiles, uint32_t tmem_base, uint32_t warp, uint32_t lane,
                                              uint32_t scale_slot, uint32_t* combine_flag, uint64_t* acc_full, uint64_t* acc_empty, const WaitCtx& wctx) {
  using T = Tile<TT>;
  constexpr uint32_t kCW = TT / 2, kLd = 16, kChunks = kCW / kLd;   // columns (tokens) per thread, and per TMEM load
  const uint32_t quad = warp & 3, colhalf = (warp - kFirstEpilogueWarp) >> 2, r = quad * 32 + lane;
  const uint32_t lane_addr = tmem_base + ((quad * 32u) << 16) + colhalf * kCW;
  const uint32_t full0 = saddr(acc_full), empty0 = saddr(acc_empty);
  float y[kCW];
#pragma unroll
  for (uint32_t i = 0; i < kCW; ++i) y[i] = 0.f;
  uint32_t buf = 0, parity = 0;
  bool waited = false;
  for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const uint32_t sp = tile % p.splits, out_tile = tile / p.splits, nt = out_tile / p.m_tiles, mt = out_tile % p.m_tiles;
    uint32_t j0, j1;
    split_range(p, tile, j0, j1);
    const uint32_t n = nt * kRows + r;
    // A tile-plane's two group scales are one word.  It is fetched a tile-plane ahead, so that no slab's
    // drain waits for a load, into a word of shared memory of the thread's own: the sums leave no
    // register for it (kept in a register it was spilled as it arrived, and the spill waited 800 clocks).
    const auto fetch_scale = [&](uint32_t tp) {   // tile-plane index from the start of the arena: below 2^32 as there are that many scales at most
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(scale_slot), "l"(reinterpret_cast<const uint32_t*>(p.scales) + tp) : "memory");
    };
    const uint32_t tok0 = mt * TT + colhalf * kCW;
    const bool live = T::kSingle || tok0 < p.m;   // else the drain would only take issue slots from the expanders
    const uint32_t row_tp = min(n, p.n - 1) * (p.tpr * PLANES);
    uint32_t tp = row_tp + j0 * PLANES;
    const uint32_t tp_end = row_tp + j1 * PLANES;
    fetch_scale(tp);
#pragma unroll 1
    for (; tp < tp_end; ++tp) {
      asm volatile("cp.async.wait_all;" ::: "memory");
      uint32_t sc;
      asm volatile("ld.shared.b32 %0, [%1];" : "=r"(sc) : "r"(scale_slot) : "memory");
      if (tp + 1 < tp_end) fetch_scale(tp + 1);
      if (!live) {   // nothing but padding tokens in this half: hand the accumulator back
        mbar_wait(full0 + 8 * buf, parity, wctx, 306);
        __syncwarp();   // a lane that still polls would miss this phase once the accumulator is refilled
        if (lane == 0) mbar_arrive(empty0 + 8 * buf);
      } else
#pragma unroll
      for (uint32_t gsel = 0; gsel < 2; ++gsel) {
        const float sv = __half2float(__ushort_as_half(uint16_t(gsel ? sc >> 16 : sc & 0xffffu)));
        if (T::kSingle || gsel == 0) {
          mbar_wait(full0 + 8 * (T::kSingle ? gsel : buf), parity, wctx, 306);
          tc_fence_after();
        }
        const uint32_t d_addr = lane_addr + (T::kSingle ? gsel * T::kAccCols : buf * T::kAccCols + gsel * TT);
        // the next columns are on their way while these are added
        uint32_t dv[2][kLd];
        tmem_ld(d_addr, dv[0]);
#pragma unroll
        for (uint32_t c = 0; c < kChunks; ++c) {
          tmem_wait_ld(dv[c & 1]);
          if (c + 1 < kChunks) tmem_ld(d_addr + (c + 1) * kLd, dv[(c + 1) & 1]);
          else if (T::kSingle || gsel == 1) {   // everything is read: the accumulator may be overwritten
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(empty0 + 8 * (T::kSingle ? gsel : buf));
          }
#pragma unroll
          for (uint32_t i = 0; i < kLd; ++i) y[c * kLd + i] = __fmaf_rn(__int2float_rn(int(dv[c & 1][i])), sv, y[c * kLd + i]);
          if (DUMP) {
            if (n < p.n) {
              const uint32_t jp = tp - row_tp, j = jp / PLANES, pl = jp - j * PLANES;
#pragma unroll
              for (uint32_t i = 0; i < kLd; ++i) {
                const uint32_t mtok = tok0 + c * kLd + i;
                if (mtok < p.m) p.acc_dump[((size_t(mtok) * p.n + n) * (p.tpr * 2) + 2 * j + gsel) * PLANES + pl] = int(dv[c & 1][i]);
              }
            }
          }
        }
      }
      if (T::kSingle) parity ^= 1;
      else if (++buf == uint32_t(T::kAccBufs)) { buf = 0; parity ^= 1; }
    }
    // ---- the tile (or this split of it) is complete
    if (!waited) {   // the token scales were written by the pre-pass, the previous grid on the stream
      asm volatile("griddepcontrol.wait;" ::: "memory");
      waited = true;
    }
    const float rs = p.row_scale ? p.row_scale[min(n, p.n - 1)] : 1.0f;
    if (live && n < p.n) {
      if (T::kMaySplit && p.splits > 1) {
        float* part = p.partial + (size_t(sp) * p.m_pad + tok0) * p.n + n;   // padding tokens too: the scratch holds m_pad rows
#pragma unroll
        for (uint32_t i = 0; i < kCW; ++i, part += p.n) *part = y[i];
      } else {
#pragma unroll
        for (uint32_t c = 0; c < kCW; c += 16) finish_outputs(p, &y[c], tok0 + c, n, rs);
      }
    }
#pragma unroll
    for (uint32_t i = 0; i < kCW; ++i) y[i] = 0.f;
    if (T::kMaySplit && p.splits > 1) {
      // Split K: count this split in; whoever completes the count adds the splits' sums in split
      // order (every run gives the same bits) and finishes the tile's outputs.
      __threadfence();
      named_sync(kBarEpilogue, 32 * kEpilogueWarps);
      if (warp == kFirstEpilogueWarp && lane == 0) {
        const uint32_t arrived = atomicAdd(p.tile_counters + out_tile, 1u);
        *combine_flag = arrived == p.splits - 1 ? 1u : 0u;
        if (*combine_flag) p.tile_counters[out_tile] = 0u;   // ready for the next launch
      }
      named_sync(kBarEpilogue, 32 * kEpilogueWarps);
      if (*combine_flag && n < p.n) {
        __threadfence();
        // Each round of loads is one latency of L2, so as many as the registers hold (16 at a time: 2560 x 2560,
        // 1 plane, 16 tokens 13.4 us a call, 12.0 now)
        constexpr uint32_t kAtOnce = kCW < 32 ? kCW : 32;
#pragma unroll 1
        for (uint32_t c = 0; c < kCW && tok0 + c < p.m; c += kAtOnce) {
          const float* part = p.partial + size_t(tok0 + c) * p.n + n;
          float sum[kAtOnce];
#pragma unroll
          for (uint32_t i = 0; i < kAtOnce; ++i) sum[i] = __ldcg(part + size_t(i) * p.n);
#pragma unroll 1
          for (uint32_t s2 = 1; s2 < p.splits; ++s2) {
            part += size_t(p.m_pad) * p.n;
            float more[kAtOnce];
#pragma unroll
            for (uint32_t i = 0; i < kAtOnce; ++i) more[i] = __ldcg(part + size_t(i) * p.n);
#pragma unroll
            for (uint32_t i = 0; i < kAtOnce; ++i) sum[i] = __fadd_rn(sum[i], more[i]);
          }
#pragma unroll
          for (uint32_t i = 0; i < kAtOnce; i += 16) finish_outputs(p, &sum[i], tok0 + c + i, n, rs);
        }
      }
      named_sync(kBarEpilogue, 32 * kEpilogueWarps);   // the flag has been read
    }
  }
}

// ---------------------------------------------------------------- the kernel
template <int CODEC, int PLANES, int TT, bool DUMP>
__global__ void __launch_bounds__(Tile<TT>::kThreads, 1) gemm_kernel(const PrefillParams p, const __grid_constant__ CUtensorMap map_q) {
  using T = Tile<TT>;
  constexpr uint32_t kTmemCols = T::kAccBufs * T::kAccCols;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* tile_a = smem;
  uint8_t* tile_b = tile_a + 2 * T::kExpGroups * kTileABytes;
  uint8_t* stage = tile_b + T::kStagesB * 2 * T::kTileBBytes;
  uint8_t* scale_words = stage + size_t(kGroupWarps * T::kExpGroups) * T::kDepth * kStageBytes;   // one per epilogue thread
  __shared__ uint64_t a_full[T::kFullBars], a_empty[T::kEmptyBars], b_full[T::kStagesB], b_empty[T::kStagesB];
  __shared__ uint64_t acc_full[T::kAccBufs], acc_empty[T::kAccBufs];
  __shared__ uint32_t tmem_base_s, abort_flag, combine_flag;

  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    abort_flag = 0;
    for (int s = 0; s < T::kFullBars; ++s) mbar_init(&a_full[s], kGroupWarps);
    for (int s = 0; s < T::kEmptyBars; ++s) mbar_init(&a_empty[s], 1);
    for (int s = 0; s < T::kStagesB; ++s) { mbar_init(&b_full[s], 1); mbar_init(&b_empty[s], 2); }
    for (int s = 0; s < T::kAccBufs; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], kEpilogueWarps); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(&tmem_base_s)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_s;
  const uint32_t tiles = p.n_tiles * p.m_tiles * p.splits;   // work items
  const WaitCtx wctx{&abort_flag, p.status};

  if (warp < kFirstEpilogueWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(T::kControlRegs));
    if (warp == 0) copy_role<TT>(p, map_q, tiles, tile_b, b_full, b_empty, wctx, lane);
    else if (warp <= 2) mma_role<PLANES, TT>(p, tiles, tmem_base, warp - 1, tile_a, tile_b, a_full, a_empty, b_full, b_empty, acc_full, acc_empty, wctx);
  } else if (warp < kFirstExpandWarp) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(T::kEpilogueRegs));
    epilogue_role<PLANES, TT, DUMP>(p, tiles, tmem_base, warp, lane, saddr(scale_words) + (tid - 32 * kFirstEpilogueWarp) * 4, &combine_flag, acc_full, acc_empty, wctx);
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(T::kExpandRegs));
    expander_role<CODEC, PLANES, TT>(p, tiles, warp - kFirstExpandWarp, lane, tile_a, stage, a_full, a_empty, wctx);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
}

// ---------------------------------------------------------------- host side
using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                 const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled encode_tiled_fn() {
  static EncodeTiled fn = [] {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult res;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &res) != cudaSuccess ||
        res != cudaDriverEntryPointSuccess)
      sym = nullptr;
    return reinterpret_cast<EncodeTiled>(sym);
  }();
  return fn;
}

// Widest token tile that `m` tokens take, and the tokens padded to it (the rows of the scratch).
uint32_t widest_tile(uint32_t m) { return m <= 32 ? 32 : m <= 64 ? 64 : m <= 128 ? 128 : 256; }
uint32_t pad_tokens(uint32_t m) { const uint32_t t = widest_tile(m); return (m + t - 1) / t * t; }
// Token tile: one of 32, 64 or 128 tokens for that many tokens; beyond that 256, or 128 where
//   * the tiles of 128 still fit one wave, or take half as many waves again at most and a row has no more than
//     40 tile-planes: a CTA is done with a 128-token tile in 0.65 to 0.7 of a 256-token tile's time (half
//     the drain and outputs, three expander groups in place of two), longer rows at the upper end;
//   * a row has no more than four tile-planes: the outputs then outweigh the sums, and the 256-token
//     tile's unrolled output code is twice as long when it has to come from memory first.
// Measured, tiles of 256 -> 128, us (caches flushed in front of each call): 512 x 1024, 1 plane, 256 tokens
// 33.7 -> 19.5; 2560 x 2560, 3 planes, 256 tokens 62.6 -> 42.0; 6912 x 512, 1 plane, 2048 tokens 54.2 -> 48.0.
// Where 256 stays: 6912 x 2560, 3 planes, 2048 tokens 165 against 194.
uint32_t tile_tokens(const tb_weights* w, uint32_t m, uint32_t sm_count) {
  if (m <= 128) return widest_tile(m);
  const uint64_t n_tiles = (w->n + kRows - 1) / kRows, tile_planes = w->k / 256 * w->uniform_planes;
  const auto waves = [&](uint32_t tt) { return (n_tiles * ((m + tt - 1) / tt) + sm_count - 1) / sm_count; };
  const uint64_t half = waves(128), whole = waves(256);
  return half == whole || (2 * half <= 3 * whole && tile_planes <= 40) || tile_planes <= 4 ? 128 : 256;
}
// K splits of an output tile, for token tiles of up to 128: as many as keep every CTA of one wave busy, at most one
// per tile column.  A 128-token tile passes 64 KB of sums through memory per part and the last CTA adds them up, about
// 6 us with two or three parts: it is split where that saves a CTA ten tile-planes, with six parts twelve, with
// more 14.  Measured, whole / split, us: two and three parts, 4 and 5 saved 16.4 / 17.5, 15.8 / 17.8 (6912 x 1024, 2 planes,
// and 5120 x 2048, 1 plane, 100 tokens), 10 saved 23.3 / 21.1, 28.6 / 25.2 (5120 x 2048, 2 planes, 128; 2560 x 5120, 1 plane, 300),
// 18 saved 42.3 / 31.4 (8192 x 3072, 3 planes, 100); six parts, 10 saved 20.6 / 21.2, 13 saved 23.9 / 22.4 (1024 x 3072 and 4096,
// 1 plane, 300); seven, 13 saved 21.6 / 22.8, 16 saved 26.0 / 23.9 (2560 x 4096, 1 plane, and 2560, 2 planes, 128); eight, 7 saved
// 15.3 / 20.0, 14 saved 21.8 / 20.5 (1024 x 2048, 1 plane, 128, and 2 planes, 100).
uint32_t splits_of(const tb_weights* w, uint32_t m, uint32_t tt, uint32_t sm_count) {
  const uint32_t tpr = uint32_t(w->k / 256), out_tiles = uint32_t((w->n + kRows - 1) / kRows) * ((m + tt - 1) / tt);
  if (tt > 128 || out_tiles >= sm_count || out_tiles > kMaxSplitTiles) return 1;
  const uint32_t splits = std::max(1u, std::min(std::min(sm_count / out_tiles, tpr), 8u));
  const uint32_t worth = std::max(10u, std::min(2u * splits, 14u));
  if (tt == 128 && (tpr - (tpr + splits - 1) / splits) * w->uniform_planes < worth) return 1;
  return splits;
}

struct Scratch { int8_t* qperm; float* ascale; float* partial; size_t fixed; };
Scratch carve(void* base, uint32_t m_pad, uint32_t k) {
  uint8_t* b = static_cast<uint8_t*>(base);
  Scratch s;
  s.qperm = reinterpret_cast<int8_t*>(b);
  size_t off = (size_t(m_pad) * k + 255) & ~size_t(255);
  s.ascale = reinterpret_cast<float*>(b + off);
  off += (size_t(m_pad) * 4 + 255) & ~size_t(255);
  s.partial = reinterpret_cast<float*>(b + off);   // [splits][m_pad][n], only when K is split
  s.fixed = off;
  return s;
}

// One instantiation of the kernel and what its launch needs.
struct GemmKernel {
  void (*fn)(PrefillParams, CUtensorMap);
  std::atomic<int>* regs;   // registers per thread it was built with, 0 until asked for: a fact of this library, the same on every device
  int threads;
  size_t smem;
  bool (*pool_holds)(int);
};
template <int CODEC, int PLANES, int TT, bool DUMP> std::atomic<int> g_built_regs{0};
template <int CODEC, int PLANES, int TT, bool DUMP>
GemmKernel kernel_instance() {
  using T = Tile<TT>;
  return {gemm_kernel<CODEC, PLANES, TT, DUMP>, &g_built_regs<CODEC, PLANES, TT, DUMP>, T::kThreads, T::kSmem, T::pool_holds};
}
template <int CODEC, int TT, bool DUMP>
GemmKernel kernel_of_planes(uint32_t planes) {
  return planes == 1 ? kernel_instance<CODEC, 1, TT, DUMP>() : planes == 2 ? kernel_instance<CODEC, 2, TT, DUMP>() : kernel_instance<CODEC, 3, TT, DUMP>();
}
template <int CODEC, bool DUMP>
GemmKernel kernel_of_tile(uint32_t tt, uint32_t planes) {
  return tt == 32    ? kernel_of_planes<CODEC, 32, DUMP>(planes)
         : tt == 64  ? kernel_of_planes<CODEC, 64, DUMP>(planes)
         : tt == 128 ? kernel_of_planes<CODEC, 128, DUMP>(planes)
                     : kernel_of_planes<CODEC, 256, DUMP>(planes);
}
GemmKernel kernel_of(int codec, uint32_t tt, uint32_t planes, bool dump) {
  if (codec == tbf::kB3) return dump ? kernel_of_tile<tbf::kB3, true>(tt, planes) : kernel_of_tile<tbf::kB3, false>(tt, planes);
  return dump ? kernel_of_tile<tbf::kD2, true>(tt, planes) : kernel_of_tile<tbf::kD2, false>(tt, planes);
}

}  // namespace

bool tb_prefill_supported(const tb_weights* w, uint32_t m) {
  return w->fast && m >= 1 && w->k >= 256 && encode_tiled_fn() != nullptr;
}

bool tb_prefill_registers_hold(uint32_t m, int launch_regs) {
  return kernel_of(tbf::kB3, widest_tile(m), 1, false).pool_holds(launch_regs);   // the same for every codec and plane count
}

namespace {
uint32_t sm_count_of(const tb_weights* w) { return w->owner ? uint32_t(w->owner->prop.multiProcessorCount) : 148u; }
}  // namespace
size_t tb_prefill_scratch_bytes(const tb_weights* w, uint32_t m) {
  const uint32_t tt = tile_tokens(w, m, sm_count_of(w)), rows = (m + tt - 1) / tt * tt, splits = splits_of(w, m, tt, sm_count_of(w));
  return carve(nullptr, pad_tokens(m), uint32_t(w->k)).fixed + (splits > 1 ? size_t(splits) * rows * w->n * 4 : 0) + 256;
}
// Split tiles number no more than the SMs, so the parts of all of them hold no more than an output tile per SM.
size_t tb_prefill_reserve_bytes(const tb_weights* w, uint32_t max_m) {
  return carve(nullptr, pad_tokens(max_m), uint32_t(w->k)).fixed + size_t(sm_count_of(w)) * std::min(widest_tile(max_m), 128u) * kRows * 4 + 256;
}

cudaError_t tb_launch_prefill(const PrefillArgs& a, int sm_count, cudaStream_t stream) {
  const tb_weights* w = a.w;
  const uint32_t m_pad = pad_tokens(a.m), k = uint32_t(w->k);
  if (!a.scratch || a.scratch_bytes < tb_prefill_scratch_bytes(w, a.m)) return cudaErrorInvalidValue;
  const Scratch sc = carve(a.scratch, m_pad, k);
  const uint32_t tt = tile_tokens(w, a.m, uint32_t(sm_count)), m_tiles = (a.m + tt - 1) / tt, rows = m_tiles * tt;   // rows <= m_pad
  const GemmKernel kernel = kernel_of(w->codec, tt, w->uniform_planes, a.acc_dump != nullptr);
  cudaError_t err = cudaSuccess;
  int regs = kernel.regs->load(std::memory_order_relaxed);
  if (!regs) {
    cudaFuncAttributes built;
    if ((err = cudaFuncGetAttributes(&built, kernel.fn)) != cudaSuccess) return err;
    kernel.regs->store(regs = built.numRegs, std::memory_order_relaxed);
  }
  if (!kernel.pool_holds(regs)) return cudaErrorInvalidConfiguration;   // its setmaxnreg would wait for ever
  err = cudaFuncSetAttribute(kernel.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kernel.smem));
  if (err != cudaSuccess) return err;

  QuantParams qp{};
  qp.x = a.x; qp.act_scale_in = a.act_scale_in; qp.act_absmax_in = a.act_absmax_in;
  if (a.relu2_up) {
    if (a.x_dtype != TB_F32) return cudaErrorInvalidValue;
    qp.relu2_up = a.relu2_up;
  }
  qp.qperm = sc.qperm; qp.ascale = sc.ascale;
  qp.vec = (reinterpret_cast<uintptr_t>(a.x) & 15u) == 0;   // k is a multiple of 256: every row starts like the first
  qp.m = a.m; qp.k = k; qp.x_dtype = uint32_t(a.x_dtype); qp.codec = uint32_t(w->codec); qp.status = a.status;
  // Up to two rows per SM that take 256 threads more than one step: wide CTAs, for the latency of one row
  // (16 tokens: 2,560 columns 5.0 against 5.7 us, 17,408 columns 9.0 against 14.1; but 1,024 columns 4.8
  // against 4.4).  Else several rows share an SM (512 tokens of 2,560 columns: 6.6 against 8.4 us).
  if (rows <= 2u * uint32_t(sm_count) && k > 2048) prefill_quant_kernel<1024><<<rows, 1024, 0, stream>>>(qp);
  else prefill_quant_kernel<256><<<rows, 256, 0, stream>>>(qp);
  err = cudaGetLastError();
  if (err != cudaSuccess) return err;

  // activations as a 2-D int8 tensor [rows][k bytes]; a box is one slab of one token tile
  CUtensorMap map;
  const cuuint64_t dims[2] = {k, rows};
  const cuuint64_t strides[1] = {k};
  const cuuint32_t box[2] = {128, tt};
  const cuuint32_t elem[2] = {1, 1};
  if (encode_tiled_fn()(&map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, sc.qperm, dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return cudaErrorInvalidValue;

  PrefillParams pp{};
  pp.payload = w->d_payload; pp.scales = w->d_scales;
  pp.ascale = sc.ascale;
  pp.y = a.y; pp.acc_dump = a.acc_dump; pp.row_scale = a.row_scale; pp.status = a.status; pp.residual = a.residual;
  pp.m = a.m; pp.m_pad = rows; pp.n = uint32_t(w->n); pp.k = k; pp.tpr = k / 256; pp.y_dtype = uint32_t(a.y_dtype);
  pp.n_tiles = (pp.n + kRows - 1) / kRows; pp.m_tiles = m_tiles;
  pp.splits = splits_of(w, a.m, tt, uint32_t(sm_count));
  if (pp.splits > 1) {
    if (!a.tile_counters) return cudaErrorInvalidValue;
    pp.partial = sc.partial; pp.tile_counters = a.tile_counters;
  }
  // may start under the tail of the quantisation pre-pass (see copy_role)
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(std::min<uint32_t>(pp.n_tiles * pp.m_tiles * pp.splits, uint32_t(sm_count)));
  cfg.blockDim = dim3(unsigned(kernel.threads)); cfg.dynamicSmemBytes = kernel.smem; cfg.stream = stream;
  cfg.attrs = attr; cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel.fn, pp, map);
}
