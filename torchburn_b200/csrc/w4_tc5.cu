// Batched grouped-INT4 product on the 5th-generation tensor cores (tcgen05):
// out[m, j] = sum_g scale[j, g] * sum_{k in g} x[m, k] * code(w[j, k])  (+ bias, + residual, or the SwiGLU of
// a gate/up pair).  gemm_w4a32_grouped, src/quantization/gemv.rs:1690-1725; fused_swiglu_mlp_batched,
// src/quantization/fused_ops.rs:1267-1319.
//
// The 4-bit codes are exact in bf16, so the weights enter the tensor core as they are and the scale is applied
// OUTSIDE it, once per group: every group of K gets a fresh fp32 accumulator in tensor memory, which the
// epilogue warps read back, multiply by scale[row, group] and add to their registers while the next groups are
// being multiplied.  The fp32 activations are split once per call (pre-pass, with the fused RMSNorm) into three
// bf16 pieces that carry all 24 bits of every value, whatever its neighbours are.  (Two fp16 pieces behind a power of two
// per row are 12% faster at 301 x 4096 x 14330, 104 against 116 us, but lose the bits of a value below 2^-17 of the row's
// largest: an outlier in a row costs every other element of it.)  Products of a 4-bit code and a piece are exact and the tensor core adds them in
// fp32, the small pieces first.
//
// The weights are the M = 128 side of the MMA, the activation rows its N.  A CTA works on NW tiles of 128 weight
// rows (the gate and the up rows of a pair, or 256 consecutive rows) times MP activation rows; two weight tiles
// share every activation image, which halves the L2 traffic of the images (3 * MP * 128 bytes per 64 elements of
// K and SM: the bound at one tile per CTA and long prompts).  A weight row lives in one LANE of tensor memory:
// the thread that unpacks row r writes its codes with tcgen05.st straight from registers (A operand from tensor
// memory), so the weights pass through shared memory only as packed nibbles.
//
//   unpacking    4, 8 or 16 warps (thread = weight row) turn the nibbles in the ring into codes in tensor memory.  One warp
//                takes ~1080 cycles for 64 elements of K (reading and unpacking 415, its waits for the stage and the
//                unit ~440), a chain that no ring depth shortens; with few activation rows nothing else is as slow, so
//                more warps take turns at the units.  16 rather than 8 at up to 32 rows: 42.2 -> 37.7 us for the pair
//                of 16 x 4096 x 14336, 46.0 -> 43.9 for 32 rows.  From 96 columns on the epilogue needs the registers.
//   epilogue     8 warps: two teams of 128 threads (thread = weight row, all activation rows) that take every
//                other VISIT: the accumulators of up to four groups, 128 columns of tensor memory, handed over
//                at once.  The fixed cost of a hand-over (commit, barrier, tcgen05.ld latency: ~400 cycles) was what
//                bounded one hand-over per group and both teams at every one of them.
//   issue        3 warps, one lane each: issuer i owns accumulator slot i and takes visit i, i + 3, ..., so that one
//                waits for its operands or its slot while another issues
//   copies       1 warp, one lane: TMA boxes of 128 weight rows x 64 bytes (128 elements of K) and of their scales,
//                bulk copies of the activation images, each into a ring.  (Copied by the rows' own threads with
//                cp.async, every 16 bytes of a warp's 32 rows are 32 different lines: the shared-memory pipe was
//                busy with them half of the time and every read of the ring waited ~500 cycles behind them.)
//
// CTAs are persistent: every role walks the CTA's list of tiles, or its range of the units of K of all tiles, by itself, so a
// tile's prologue and epilogue lie under its neighbours' streaming.  Every wait is bounded.  No cluster features, no multicast.
#include <cuda_bf16.h>

#include "tb_common.cuh"
#include "tc5.cuh"
#include "tma_map.cuh"
#include "w4_math.cuh"

namespace tb {

namespace {

constexpr int kTileN = 128;     // weight rows per MMA (its M)
constexpr int kKC = 64;         // K elements per stage: one 128-byte row of bf16
constexpr int kUnit = 128;      // K elements per copy of a weight tile: 64 bytes of nibbles a row
constexpr int kUnitBytes = kTileN * 64;
constexpr int kUnitScaleBytes = kTileN * 16;   // 32-element groups: four scales a row
constexpr int kPieces = 3;      // bf16 pieces of an activation
constexpr int kTmemCols = 512;
constexpr int kSlots = 3;       // accumulator slots of 128 columns; the first 128 columns hold the codes
// Barriers of the stage rings, by chunk of K.  More of them than stages: a role that runs ahead (three issuers, two unpacking
// teams) may wait for a chunk while one up to ten chunks older is still open, and a wait on a barrier two phases ahead
// would pass at once.
constexpr uint32_t kRing = 16;
constexpr int kMaxSplit = 8;    // most CTAs that share a tile's K
constexpr int kMaxRows = 512;   // activation rows per launch (bounds the workspace)
constexpr int kMinRows = 9;     // below: the streaming kernel (w4_rows.cu)
constexpr int kSureRows = 17;   // from here on always this one, in between the one that costs less (w4_mma_cost)

__device__ int g_tc5_fault = 0;

struct Tc5Params {
  CUtensorMap w[2];          // [n, k / 2] bytes, boxes of 64 x 128 rows
  CUtensorMap s[2];          // 32-element groups: [n, ng] scales, boxes of 4 x 128 rows
  const float* scales[2];
  const float* bias[2];
  const float* resid;
  float* out;
  float* parts;              // ranges: sums [CTA][its first tile, its last one][column][128 weight rows]
  int* tickets;              // [tile]: parts that have arrived; zero, and left zero
  const unsigned char* xq;   // [activation tile][64-element chunk of K][piece][MP rows x 128 B], swizzled
  int m;                     // activation rows
  int n, k, ng;
  int mtiles, ntiles;        // tiles of activation rows and of weight rows
  int per, more;             // ranges: units of K (of all tiles, one after another) of a CTA, the first `more` CTAs take one more; per 0: whole tiles in turn
  int pair;                  // the second weight tile is the up matrix
};

using namespace tc5;
// Inlined: a call would need registers by the calling convention, which a kernel with split registers cannot give.
__device__ __forceinline__ bool mbar_wait_fast(uint64_t* bar, uint32_t parity, volatile int* s_abort) {
  return mbar_ready(bar, parity) ? true : tc5::mbar_wait(bar, parity, s_abort, &g_tc5_fault);
}
// The same for a whole converged warp: every lane asks, the warp votes, so that all lanes take the same way (also when
// the wait is given up) without a branch of one lane in front of every warp-wide instruction.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* s_abort) {
  long long t0 = 0;
  for (uint32_t i = 0;; ++i) {
    if (__all_sync(0xffffffffu, mbar_ready(bar, parity))) return true;
    if ((i & 127) == 127) {
      const long long now = __shfl_sync(0xffffffffu, clock64(), 0);
      if (t0 == 0) t0 = now;
      const bool late = now - t0 > kWaitCycles;
      if (late && (threadIdx.x & 31) == 0) {
        *s_abort = 1;
        atomicExch(&g_tc5_fault, 1);
      }
      if (late || __any_sync(0xffffffffu, *s_abort != 0)) return false;
    }
  }
}
// One arrival for the warp, by its lane 0 and without a branch; behind a __syncwarp, which orders the other lanes' accesses before it.
__device__ __forceinline__ void mbar_arrive_warp(uint64_t* bar, int lane) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.s32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(smem_u32(bar)), "r"(lane) : "memory");
}

// D (tensor memory, fp32) (+)= A (tensor memory, bf16) * B (shared memory, bf16)^T
// b_lo: the lower word of B's shared-memory descriptor; the upper word is the same for every tile.
template <int ACC>
__device__ __forceinline__ void mma_bf16_ts(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t idesc) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      ".reg .b64 bd;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "mov.b64 bd, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], bd, %4, p;\n\t"
      "}\n" ::"r"(d_tmem),
      "r"(a_tmem), "r"(b_lo), "r"(kDescHi), "r"(idesc), "n"(ACC)
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(r[0]),
      "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]),
      "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// Two fp32 fused multiply-adds in one issue slot: a += x * s.
__device__ __forceinline__ void fma2(float& a0, float& a1, uint32_t x0, uint32_t x1, float s) {
  asm("{\n\t.reg .b64 a, x, s;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 x, {%2, %3};\n\tmov.b64 s, {%4, %4};\n\t"
      "fma.rn.f32x2 a, x, s, a;\n\tmov.b64 {%0, %1}, a;\n\t}"
      : "+f"(a0), "+f"(a1)
      : "r"(x0), "r"(x1), "f"(s));
}

constexpr int floor_pow2(int v) { return v >= 4 ? 4 : (v >= 2 ? 2 : 1); }

// Everything that follows from the template parameters.
template <int MP, int NW, int G>
struct Shape {
  static constexpr int kCols = MP * NW;                    // accumulator columns of one group
  static constexpr int kFit = floor_pow2(128 / kCols);
  static constexpr int kGps = kFit < kUnit / G ? kFit : kUnit / G;   // groups per visit
  static constexpr int kVk = kGps * G;                     // K elements per visit: 32, 64 or 128
  static constexpr int kSteps = kVk / 16;                  // K16 steps per visit
  static constexpr int kVisitsPerStage = kVk >= kKC ? 1 : kKC / kVk;
  static constexpr int kDW = NW == 2 && kCols <= 64 ? 16 : (kCols <= 96 ? 8 : 4);   // unpacking warps
  // Teams of four of them: each for one weight tile (kTeamTile) or all of them, and for every kUnitStride-th unit.
  static constexpr bool kTeamTile = NW == 2 && kDW >= 8;
  static constexpr int kUnitStride = kDW / (kTeamTile ? 8 : 4);
  static constexpr int kThreads = (kDW + 12) * 32;
  // registers: (kDW + 4) warps give back to the 8 epilogue warps; the sum stays at what the block was launched with
  static constexpr int kRegsLaunch = kDW == 16 ? 72 : (kDW == 8 ? 96 : 128), kRegsFew = kDW == 16 ? 48 : (kDW == 8 ? 64 : 56), kRegsMany = kDW == 16 ? 128 : (kDW == 8 ? 144 : 200);
  static_assert((kDW + 4) * kRegsFew + 8 * kRegsMany <= (kDW + 12) * kRegsLaunch, "register split");
  static constexpr int kStagesA = 128 / (32 * NW);
  static constexpr int kStagesB = MP <= 16 ? 16 : (MP <= 32 ? 8 : (MP <= 48 ? 5 : 4));   // up to 96 KB
  static constexpr int kUnits = NW == 2 ? (MP <= 48 ? 4 : 3) : 8;   // ring of weight units: 64 KB, 48 KB in the largest shape
  static constexpr int kScales = G != 32 ? 8 : (kCols <= 64 ? 8 : 4);   // units (32-element groups) or visits of scales in flight
  static constexpr int kBBytes = kPieces * MP * 128;       // the activation images of a stage
  static constexpr int kScaleBytes = NW * kGps * 4;        // of one visit and row
  static constexpr size_t kOffNib = (size_t)kStagesB * kBBytes;
  static constexpr size_t kOffScale = kOffNib + (size_t)kUnits * NW * kUnitBytes;
  static constexpr size_t kOffEx = kOffScale + (size_t)kScales * (G == 32 ? NW * kUnitScaleBytes : 256 * kScaleBytes);
  static constexpr size_t kSmem = kOffEx + (size_t)kCols * 128 * 4 + 1024;
  static_assert(kSmem <= 226 * 1024, "shared memory");
};

__device__ __forceinline__ void epilogue_barrier() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

template <int MP, int NW, int G>
__global__ void __launch_bounds__(Shape<MP, NW, G>::kThreads, 1) w4_tc5_kernel(const __grid_constant__ Tc5Params p) {
  using S = Shape<MP, NW, G>;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full_a[kRing], full_b[kRing], done[kRing], full_w[8], empty_w[8], empty_s[8], acc_full[2 * kSlots], acc_empty[kSlots], drained[kSlots];
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort, s_ticket, s_first, s_parts[2], s_tile, s_unit, s_visits;

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  // The CTA's units of K, numbered from 0, are units g0 ... of its own list of tiles (t0, t0 + ts, ...): a range of all tiles' units,
  // which may begin and end inside a tile, or whole tiles in turn.
  const int nunits = p.k / kUnit;   // of one tile
  const int bx = (int)blockIdx.x, tiles = p.mtiles * p.ntiles;
  const int g0 = p.per ? bx * p.per + min(bx, p.more) : 0;
  const int my_units = p.per ? p.per + (bx < p.more ? 1 : 0) : (tiles - bx + (int)gridDim.x - 1) / (int)gridDim.x * nunits;
  const int t0 = p.per ? 0 : bx, ts = p.per ? 1 : (int)gridDim.x;
  constexpr uint32_t SA = S::kStagesA, SB = S::kStagesB;

  if (p.per && (tid == 32 || tid == 64)) {   // the CTAs that share the CTA's first and its last tile
    auto cta_of = [&](int unit) {
      const int wide = p.more * (p.per + 1);
      return unit < wide ? unit / (p.per + 1) : p.more + (unit - wide) / p.per;
    };
    const int t = (tid == 32 ? g0 : g0 + my_units - 1) / nunits, c0 = cta_of(t * nunits);
    s_parts[tid == 32 ? 0 : 1] = cta_of(t * nunits + nunits - 1) - c0 + 1;
    if (tid == 32) s_first = c0;
  }
  if (tid == 0) {
    s_abort = 0;
    s_tile = t0 + g0 / nunits * ts; s_unit = g0 % nunits; s_visits = my_units * (kUnit / S::kVk);   // where the epilogue begins and ends
    for (uint32_t s = 0; s < kRing; ++s) {
      mbar_init(&full_a[s], S::kTeamTile ? 8 : 4);   // one lane of each unpacking warp of the stage
      mbar_init(&full_b[s], 1);
      mbar_init(&done[s], S::kVisitsPerStage);   // the MMAs that read the stage have finished: one commit per visit
    }
    for (int s = 0; s < S::kUnits; ++s) {
      mbar_init(&full_w[s], 1);
      mbar_init(&empty_w[s], S::kTeamTile ? 8 : 4);   // one lane of each warp that reads the unit
    }
    for (int s = 0; s < S::kScales; ++s) mbar_init(&empty_s[s], S::kGps == 4 ? 4 : 8);   // one team reads a unit's scales, or both
    for (int s = 0; s < kSlots; ++s) {
      mbar_init(&acc_empty[s], 4);   // one lane of each warp of the team that read it
      mbar_init(&drained[s], 1);
    }
    // by visit modulo 6: the visits of one barrier belong to one team, which has waited for the one before
    for (int s = 0; s < 2 * kSlots; ++s) mbar_init(&acc_full[s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  constexpr int kIssue0 = S::kDW + 8;   // first issuing warp
  if (warp == kIssue0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;

  if (warp >= kIssue0) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(S::kRegsFew));
    const bool one = elect_one();
    if (one && warp - kIssue0 < kSlots) {
      // ---------------- MMA issue ----------------
      const uint32_t me = (uint32_t)(warp - kIssue0);
      // instruction descriptor: fp32 accumulator, bf16 x bf16, B K-major, N = MP, M = 128
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(MP >> 3) << 17) | ((uint32_t)(kTileN >> 4) << 24);
      const uint32_t b_lo0 = (smem_u32(smem) >> 4) | (1u << 16);
      const uint32_t d_base = tmem + 128u + me * 128u;
      const uint32_t nv = (uint32_t)(my_units * (kUnit / S::kVk));
      bool ok = true;
      uint32_t turn = 0;   // visits of this slot so far
      for (uint32_t v = me; v < nv; v += kSlots, ++turn) {
        if (turn > 0) {          // the epilogue must have read this slot's previous sums
          ok = mbar_wait_fast(&acc_empty[me], (turn - 1u) & 1u, &s_abort);
          if (!ok) break;
          tc_fence_after();
        }
        constexpr int kStagesPerVisit = S::kSteps > 4 ? 2 : 1;
        constexpr int kStepsHere = S::kSteps > 4 ? 4 : S::kSteps;   // of one stage
        constexpr int kStepsPerGroup = G / 16, kTogether = kStepsPerGroup < kStepsHere ? kStepsPerGroup : kStepsHere;
#pragma unroll
        for (int sv = 0; sv < kStagesPerVisit; ++sv) {
          const uint32_t c = kStagesPerVisit == 2 ? 2 * v + sv : v / S::kVisitsPerStage;
          const uint32_t ks0 = S::kVisitsPerStage == 2 ? (v & 1u) * 2u : 0u;
          ok = mbar_wait_fast(&full_a[c % kRing], (c / kRing) & 1u, &s_abort) && mbar_wait_fast(&full_b[c % kRing], (c / kRing) & 1u, &s_abort);
          if (!ok) break;
          tc_fence_after();
          const uint32_t b_lo = b_lo0 + (c % SB) * (uint32_t)(S::kBBytes >> 4) + ks0 * 2u;
          const uint32_t a_base = tmem + (c % SA) * (32u * NW) + ks0 * 8u;
#pragma unroll
          for (int k0 = 0; k0 < kStepsHere; k0 += kTogether)
#pragma unroll
            for (int pc = kPieces - 1; pc >= 0; --pc)   // a group's small pieces first: the tensor core truncates what it adds to a large sum
#pragma unroll
              for (int ks = k0; ks < k0 + kTogether; ++ks) {   // 16 bf16 = 32 bytes of an image row = 8 columns of codes
                const int t = sv * 4 + ks, gi = t / kStepsPerGroup;    // K16 step and group of this visit
#pragma unroll
                for (int q = 0; q < NW; ++q) {
                  const uint32_t d = d_base + (uint32_t)(gi * S::kCols + q * MP), a = a_base + (uint32_t)(q * 32 + ks * 8);
                  const uint32_t b = b_lo + (uint32_t)(ks * 2) + (uint32_t)(pc * (MP * 128 >> 4));
                  if (t % kStepsPerGroup == 0 && pc == kPieces - 1) mma_bf16_ts<0>(d, a, b, idesc);
                  else mma_bf16_ts<1>(d, a, b, idesc);
                }
              }
          if (sv == kStagesPerVisit - 1) mma_commit(&acc_full[me + (turn & 1u) * kSlots]);
          mma_commit(&done[c % kRing]);
        }
        if (!ok) break;
      }
      // nothing may still be running on the tensor core when the tensor memory is given back
      mma_commit(&drained[me]);
      mbar_wait_fast(&drained[me], 0u, &s_abort);
    } else if (one) {
      // ---------------- copies ----------------
      uint32_t c = 0, u = 0;
      bool ok = true;
      const uint32_t w_at = smem_u32(smem + S::kOffNib), s_at = smem_u32(smem + S::kOffScale);
      auto weights = [&](uint32_t wu, int n0, int i) {   // unit wu of the CTA: unit i of the tile at weight row n0
        const uint32_t ws = wu % S::kUnits, ss = wu % S::kScales;
        if (wu >= S::kUnits) ok = mbar_wait_fast(&empty_w[ws], (wu / S::kUnits - 1u) & 1u, &s_abort);
        if (G == 32 && ok && wu >= S::kScales) ok = mbar_wait_fast(&empty_s[ss], (wu / S::kScales - 1u) & 1u, &s_abort);
        if (!ok) return;
        // the scales arrive with the codes: who has seen sums of the unit has seen its scales
        mbar_expect_tx(&full_w[ws], NW * (kUnitBytes + (G == 32 ? kUnitScaleBytes : 0)));
#pragma unroll
        for (int q = 0; q < NW; ++q)
          tma_box(w_at + (ws * NW + q) * kUnitBytes, &p.w[p.pair ? q : 0], i * 64, n0 + (p.pair ? 0 : q * kTileN), smem_u32(&full_w[ws]));
        if constexpr (G == 32) {
#pragma unroll
          for (int q = 0; q < NW; ++q)
            tma_box(s_at + (ss * NW + q) * kUnitScaleBytes, &p.s[p.pair ? q : 0], i * 4, n0 + (p.pair ? 0 : q * kTileN), smem_u32(&full_w[ws]));
        }
      };
      // The first weights, a ring of them, do not depend on the pre-pass, which this kernel is launched beside (programmatic
      // serialization); the images do.
      static_assert(S::kScales >= S::kUnits, "scales of the first units");
      uint32_t ahead = 0;
      const int tf = t0 + g0 / nunits * ts, i0 = g0 % nunits;   // where the CTA begins
      // What a tile decides is computed at its start: two divisions per unit in this thread were what bounded one weight tile of up to 64 rows
      // (17 x 4096 x 14336 30.5 -> 26.4 us, 24 x 896 x 151936 57.4 -> 48.9, 301 x 4864 x 896 23.5 -> 20.6).
      const int row_step = p.pair ? kTileN : kTileN * NW;
      for (int t = tf, i = i0, n0 = tf / p.mtiles * row_step; ahead < (uint32_t)my_units && ahead < S::kUnits; ++ahead) {
        weights(ahead, n0, i);
        if (++i == nunits) { i = 0; t += ts; n0 = t / p.mtiles * row_step; }
      }
      asm volatile("griddepcontrol.wait;" ::: "memory");
      int n0 = tf / p.mtiles * row_step;
      const unsigned char* src = p.xq + ((size_t)(tf % p.mtiles) * nunits + i0) * (2 * S::kBBytes);
      for (int t = tf, i = i0; u < (uint32_t)my_units && ok; ++u) {
        if (u >= ahead) weights(u, n0, i);
        if (!ok) break;
        for (int h = 0; h < 2; ++h, ++c) {
          if (c >= SB) ok = mbar_wait_fast(&done[(c - SB) % kRing], ((c - SB) / kRing) & 1u, &s_abort);
          if (!ok) break;
          mbar_expect_tx(&full_b[c % kRing], S::kBBytes);
          bulk_g2s(smem + (size_t)(c % SB) * S::kBBytes, src, S::kBBytes, &full_b[c % kRing]);
          src += S::kBBytes;
        }
        if (++i == nunits) {
          i = 0;
          t += ts;
          n0 = t / p.mtiles * row_step;
          src = p.xq + (size_t)(t % p.mtiles) * nunits * (2 * S::kBBytes);
        }
      }
      // copies in flight must have landed before the CTA gives its shared memory back (all have, unless a wait was given up)
      if (!ok) {
        int no_abort = 0;
        for (uint32_t i = c > SB ? c - SB : 0; i < c; ++i) mbar_wait_fast(&full_b[i % kRing], (i / kRing) & 1u, &no_abort);
        if (u < ahead) u = ahead;
        for (uint32_t i = u > S::kUnits ? u - S::kUnits : 0; i < u; ++i) mbar_wait_fast(&full_w[i % S::kUnits], (i / S::kUnits) & 1u, &no_abort);
      }
    }
  } else if (warp < S::kDW) {
    // ---------------- unpacking: thread = weight row ----------------
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(S::kRegsFew));
    // eight or more warps: teams of four, each for one weight tile and, with 16 warps or one tile, every other unit of 128 elements
    constexpr bool kTeamTile = S::kTeamTile;
    constexpr int kTiles = S::kDW == 4 ? NW : 1;       // weight tiles of one thread
    const int team = warp >> 2, row = tid & 127;
    const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    // the ring: [slot][tile][row][64 bytes]; the copy's swizzle rotates a row's 16-byte pieces so that a quarter warp
    // touches every bank once
    const uint32_t ring = smem_u32(smem + S::kOffNib) + (uint32_t)row * 64u;
    const uint32_t swz = (uint32_t)((row >> 1) & 3);
    uint32_t u = (uint32_t)(kTeamTile ? team >> 1 : (S::kDW == 4 ? 0 : team));   // the CTA's units run through all its tiles
    const uint32_t nu = (uint32_t)my_units;
    bool ok = true;
    for (; u < nu && ok; u += (uint32_t)S::kUnitStride) {
      const uint32_t ws = u % S::kUnits;
      ok = mbar_wait_warp(&full_w[ws], (u / S::kUnits) & 1u, &s_abort);
      if (!ok) break;
#pragma unroll
      for (uint32_t h = 0; h < 2; ++h) {
        const uint32_t c = 2 * u + h;
        const uint32_t a_col = lane_base + (c % SA) * (32u * NW);
#pragma unroll
        for (int i = 0; i < kTiles; ++i) {
          const int q = kTeamTile ? team & 1 : i;
          const uint32_t src = ring + (ws * NW + (uint32_t)q) * kUnitBytes, col = a_col + (uint32_t)q * 32u;
          // the codes are ready in registers before the stage is free (16 warps, 48 registers each: half of them)
          constexpr int kHold = S::kDW == 16 ? 1 : 2;
#pragma unroll
          for (uint32_t e0 = 0; e0 < 2; e0 += kHold) {
            uint32_t v[kHold][16];
#pragma unroll
            for (uint32_t e = 0; e < kHold; ++e) {   // 32 elements = 16 columns per 16 bytes of nibbles
              uint32_t wd[4];
              asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(wd[0]), "=r"(wd[1]), "=r"(wd[2]), "=r"(wd[3]) : "r"(src + (((2 * h + e0 + e) ^ swz) * 16u)));
#pragma unroll
              for (int w = 0; w < 4; ++w) unpack8(wd[w], &v[e][4 * w]);
            }
            if (i == 0 && e0 == 0) {
              if (c >= SA) ok = mbar_wait_warp(&done[(c - SA) % kRing], ((c - SA) / kRing) & 1u, &s_abort);
              if (!ok) break;
              tc_fence_after();
            }
#pragma unroll
            for (uint32_t e = 0; e < kHold; ++e) tmem_st16(col + 16u * (e0 + e), v[e]);
          }
          if (!ok) break;
        }
        if (!ok) break;
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
        __syncwarp();   // lane 0 arrives for all: behind the other lanes' loads and stores
        if (h == 1) mbar_arrive_warp(&empty_w[ws], lane);
        mbar_arrive_warp(&full_a[c % kRing], lane);
      }
    }
  } else {
    // ---------------- per-group scaling and the epilogue: thread = weight row, team = every other visit ----------------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(S::kRegsMany));
    const int team = (warp - S::kDW) >> 2, row = tid & 127;
    const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const int et = tid - S::kDW * 32;
    const uint32_t sring = smem_u32(smem + S::kOffScale) + (G == 32 ? (uint32_t)row * 16u : (uint32_t)et * S::kScaleBytes);
    float* ex = reinterpret_cast<float*>(smem + S::kOffEx);
    // 32-element groups: the scales lie in their ring, four a row and unit.  Larger groups: the rows' scales need not start on
    // 16 bytes, so every thread copies its own with cp.async: tile, visit within it, ring slot
    int ft = t0 + g0 / nunits * ts, fv = g0 % nunits * (kUnit / S::kVk) + team;
    uint32_t fs = 0;
    const float* fp[NW];
    auto open_tile = [&](int t) {
      const int n0 = t / p.mtiles * (p.pair ? kTileN : kTileN * NW);
#pragma unroll
      for (int q = 0; q < NW; ++q) {
        const int j = n0 + (p.pair ? 0 : q * kTileN) + row;
        fp[q] = j < p.n ? (p.pair && q ? p.scales[1] : p.scales[0]) + (size_t)j * p.ng : nullptr;   // (past the last tile: none)
      }
    };
    open_tile(ft);
    auto fetch = [&]() {
      while (fv >= p.k / S::kVk) {   // (a few visits past the CTA's last one are fetched, too, and not used)
        fv -= p.k / S::kVk;
        ft += p.per ? 1 : (int)gridDim.x;
        open_tile(ft);
      }
#pragma unroll
      for (int q = 0; q < NW; ++q)
        if (fp[q] != nullptr)
          asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(sring + fs * (256u * S::kScaleBytes) + (uint32_t)(q * S::kGps * 4)),
                       "l"(fp[q] + (size_t)fv * S::kGps), "n"(S::kGps * 4)
                       : "memory");
      fv += 2;
      fs = fs + 1 == S::kScales ? 0 : fs + 1;
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if constexpr (G != 32)
#pragma unroll 1
      for (int i = 0; i < S::kScales - 1; ++i) fetch();
    uint32_t v = (uint32_t)team, rs = 0, at6 = (uint32_t)team, par6 = 0;   // at6: v modulo 6, par6: its round's parity
    int read_s = -1;
    bool ok = true;
    // What only a tile's ends need is read again there: registers are short between them.
    volatile int* const again = &s_unit;
    volatile int* const visits = &s_visits;
    int tile_end = -*again * (kUnit / S::kVk);
    for (int t = s_tile; tile_end < *visits; t += p.per ? 1 : (int)gridDim.x) {
      tile_end += p.k / S::kVk;
      const uint32_t stop = (uint32_t)min(tile_end, *visits);
      float acc[S::kCols];
#pragma unroll
      for (int i = 0; i < S::kCols; ++i) acc[i] = 0.f;
      if (p.per && et == 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.tickets + t));
      for (; v < stop && ok; v += 2) {
        if constexpr (G != 32) {
          asm volatile("cp.async.wait_group %0;" ::"n"(S::kScales - 2) : "memory");
          __syncwarp();
        }
        ok = mbar_wait_warp(&acc_full[at6], par6, &s_abort);
        if (!ok) break;
        tc_fence_after();
        if (G == 32 && read_s >= 0) {   // scales that the last visit has used: handed back only now, when every lane has them
          __syncwarp();
          mbar_arrive_warp(&empty_s[read_s], lane);
          read_s = -1;
        }
        float sc[NW][S::kGps];
        constexpr uint32_t kPerUnit = 128 / S::kVk;   // visits per unit
#pragma unroll
        for (int q = 0; q < NW; ++q) {
          const uint32_t a = G == 32 ? sring + ((v / kPerUnit % S::kScales) * NW + (uint32_t)q) * kUnitScaleBytes + (v % kPerUnit) * (uint32_t)(S::kGps * 4)
                                     : sring + rs * (256u * S::kScaleBytes) + (uint32_t)(q * S::kGps * 4);
          if constexpr (S::kGps == 4)
            asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(sc[q][0]), "=f"(sc[q][1]), "=f"(sc[q][S::kGps - 2]), "=f"(sc[q][S::kGps - 1]) : "r"(a));
          else if constexpr (S::kGps == 2) asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(sc[q][0]), "=f"(sc[q][S::kGps - 1]) : "r"(a));
          else asm volatile("ld.shared.f32 %0, [%1];" : "=f"(sc[q][0]) : "r"(a));
        }
        // Into the slot that the visit before has read.  Here, and not behind the arithmetic, it leaves the registers to the sums: the
        // pair of 200 rows 4096 -> 14336 with groups of 64 158 -> 153 us.
        if constexpr (G != 32) fetch();
        const uint32_t slot = at6 >= kSlots ? at6 - kSlots : at6;
        const uint32_t d = lane_base + 128u + slot * 128u;
        constexpr int kN16 = S::kGps * S::kCols / 16;          // 16-column loads of the visit
        constexpr int kBatch = S::kCols > 32 && kN16 % 2 == 0 ? 2 : (S::kCols > 64 ? 2 : (kN16 < 4 ? kN16 : (kN16 % 4 == 0 ? 4 : 3)));   // in flight at once
        static_assert(kN16 % kBatch == 0, "loads per visit");
#pragma unroll
        for (int b = 0; b < kN16 / kBatch; ++b) {
          uint32_t r[kBatch][16];
#pragma unroll
          for (int i = 0; i < kBatch; ++i) tmem_ld16(d + (uint32_t)((b * kBatch + i) * 16), r[i]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (b == kN16 / kBatch - 1) {   // the slot's sums are in registers: hand it back before the arithmetic
            tc_fence_before();
            __syncwarp();
            mbar_arrive_warp(&acc_empty[slot], lane);
          }
#pragma unroll
          for (int i = 0; i < kBatch; ++i) {
            const int col = (b * kBatch + i) * 16, g = col / S::kCols, at = col % S::kCols;
            const float s = sc[at / MP][g];
#pragma unroll
            for (int e = 0; e < 16; e += 2) fma2(acc[at + e], acc[at + e + 1], r[i][e], r[i][e + 1], s);
          }
        }
        if constexpr (G == 32) {
          if (S::kGps > 1 || (v & 2u)) read_s = (int)(v / kPerUnit % S::kScales);   // this team's last look at the unit's scales
        } else {
          rs = rs + 1 == S::kScales ? 0 : rs + 1;
          __syncwarp();
        }
        at6 += 2;
        if (at6 >= 2 * kSlots) { at6 -= 2 * kSlots; par6 ^= 1u; }
      }
      const int mt = t % p.mtiles, n0 = t / p.mtiles * (p.pair ? kTileN : kTileN * NW);
      // ---- the teams' sums: each finishes half of the activation rows ----
      constexpr int kHalf = MP / 2;
      epilogue_barrier();   // the last tile's exchange has been read
#pragma unroll
      for (int q = 0; q < NW; ++q)
#pragma unroll
        for (int i = 0; i < kHalf; ++i) ex[((team * NW + q) * kHalf + i) * 128 + row] = team ? acc[q * MP + i] : acc[q * MP + kHalf + i];
      epilogue_barrier();
      float* mine = ex + (team ^ 1) * NW * kHalf * 128 + row;   // what the other team left for this thread; the sums go back there
#pragma unroll
      for (int q = 0; q < NW; ++q)
#pragma unroll
        for (int i = 0; i < kHalf; ++i) mine[(q * kHalf + i) * 128] += team ? acc[q * MP + kHalf + i] : acc[q * MP + i];
      const int i0 = t == s_tile ? *again : 0;   // the CTA's first unit of the tile
      if (i0 || tile_end > *visits) {
        // Parts of K: every CTA writes its sums, the last one to arrive adds all of them in the order of the parts, the same
        // order whichever it is, so that equal calls give equal bits.  Sixteen bytes a thread, in short loops: the tail's code
        // comes from memory after every other kernel (a sum per thread and column, unrolled: 2 us more a launch).
        // The CTAs of the tile follow one another; it is the last tile of the first of them and the first tile of the others.
        constexpr int kPart = S::kCols * 128;   // floats
        const int c0 = i0 ? s_first : bx, nparts = s_parts[i0 ? 0 : 1];
        const float4* rest = reinterpret_cast<const float4*>(p.parts + (size_t)(2 * c0) * kPart) + et;   // part z at 2 z * kPart floats, the first one kPart further
        const bool wide = (p.n & 3) == 0 && ((reinterpret_cast<uintptr_t>(p.out) | reinterpret_cast<uintptr_t>(p.resid) | reinterpret_cast<uintptr_t>(p.bias[0])) & 15) == 0;
        epilogue_barrier();   // the teams' sums are complete
        {
          float4* part = reinterpret_cast<float4*>(p.parts + (size_t)(2 * bx + (i0 ? 0 : 1)) * kPart) + et;
#pragma unroll 4
          for (int i = 0; i < kPart / 4; i += 256) part[i] = reinterpret_cast<const float4*>(ex)[i + et];
        }
        epilogue_barrier();
        if (et == 0) {   // one fence on either side of the ticket, for all threads that the barriers order with it
          __threadfence();
          const int ticket = atomicAdd(p.tickets + t, 1);
          __threadfence();
          if (ticket == nparts - 1) p.tickets[t] = 0;   // for the next launch
          s_ticket = ticket;
        }
        epilogue_barrier();
        if (s_ticket != nparts - 1 || !ok) continue;
        auto sum_of = [&](int at) {   // at: in float4, behind this thread's first
          float4 v[kMaxSplit];
#pragma unroll
          for (int z = 0; z < kMaxSplit; ++z) v[z] = z < nparts ? __ldcg(rest + (2 * z + (z == 0 ? 1 : 0)) * (kPart / 4) + at) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int z = 1; z < kMaxSplit; ++z) { v[0].x += v[z].x; v[0].y += v[z].y; v[0].z += v[z].z; v[0].w += v[z].w; }
          return v[0];
        };
        if (NW == 2 && p.pair) {
#pragma unroll 1
          for (int i = 0; i < kPart / 8; i += 256) {   // four features of one activation row a thread
            const int c = (i + et) >> 5, half = c / kHalf;   // column of the gate sums; in either half as many of the up sums follow
            const int mrow = mt * MP + (half ? 0 : kHalf) + c % kHalf, j = n0 + (et & 31) * 4;
            if (mrow >= p.m || j >= p.n) continue;
            const float4 g4 = sum_of(i + half * kHalf * 32), u4 = sum_of(i + (half + 1) * kHalf * 32);
            const float ga[4] = {g4.x, g4.y, g4.z, g4.w}, up[4] = {u4.x, u4.y, u4.z, u4.w};
            float* dst = p.out + (size_t)mrow * p.n + j;
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (j + e < p.n) {
                const float a = ga[e] + (p.bias[0] ? p.bias[0][j + e] : 0.f), b = up[e] + (p.bias[1] ? p.bias[1][j + e] : 0.f);
                dst[e] = (a / (1.0f + expf(-a))) * b;   // src/llm/decoder.rs:1319-1322
              }
          }
          continue;
        }
#pragma unroll 1
        for (int i = 0; i < kPart / 4; i += 256) {   // four features of one activation row a thread
          const int c = (i + et) >> 5, q = c / kHalf % NW;
          const int mrow = mt * MP + (c < NW * kHalf ? kHalf : 0) + c % kHalf;   // a team's sums lie in the other one's half
          const int j = n0 + q * kTileN + (et & 31) * 4;
          if (mrow >= p.m || j >= p.n) continue;
          const size_t at = (size_t)mrow * p.n + j;
          float4 bias = make_float4(0.f, 0.f, 0.f, 0.f), add = bias;
          if (wide) {
            if (p.bias[0]) bias = *reinterpret_cast<const float4*>(p.bias[0] + j);
            if (p.resid) add = *reinterpret_cast<const float4*>(p.resid + at);
          }
          const float4 v = sum_of(i);
          if (wide) {
            *reinterpret_cast<float4*>(p.out + at) = make_float4(v.x + bias.x + add.x, v.y + bias.y + add.y, v.z + bias.z + add.z, v.w + bias.w + add.w);
          } else {
            const float o[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (j + e < p.n) p.out[at + e] = o[e] + (p.bias[0] ? p.bias[0][j + e] : 0.f) + (p.resid ? p.resid[at + e] : 0.f);
          }
        }
        continue;
      }
      if (!ok) continue;
      const int rows = min(kHalf, p.m - mt * MP - team * kHalf);   // of this thread's columns that are activation rows
      float b0 = 0.f, b1 = 0.f;
      if (p.bias[0] && n0 + row < p.n) b0 = __ldg(p.bias[0] + n0 + row);
      if (NW == 2 && p.pair) { if (p.bias[1] && n0 + row < p.n) b1 = __ldg(p.bias[1] + n0 + row); }
      else if (NW == 2 && p.bias[0] && n0 + kTileN + row < p.n) b1 = __ldg(p.bias[0] + n0 + kTileN + row);
      // The residual may be the output itself: added, eight rows at a time, before the first row is written, or every row would wait
      // for its own.
      if (p.resid) {
#pragma unroll
        for (int q = 0; q < NW; ++q) {
          const int j = n0 + q * kTileN + row;
          if (j >= p.n) continue;
          const float* src = p.resid + (size_t)(mt * MP + team * kHalf) * p.n + j;
#pragma unroll 1
          for (int i = 0; i < rows; i += 8) {
            float r[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) r[u] = i + u < rows ? src[(size_t)(i + u) * p.n] : 0.f;
#pragma unroll
            for (int u = 0; u < 8; ++u) mine[(q * kHalf + i + u) * 128] += r[u];
          }
        }
      }
#pragma unroll 4
      for (int i = 0; i < rows; ++i) {   // from shared memory: the code of this loop must not push the one above out of the instruction cache
        float* dst = p.out + (size_t)(mt * MP + team * kHalf + i) * p.n;
        float sum[NW];
#pragma unroll
        for (int q = 0; q < NW; ++q) sum[q] = mine[(q * kHalf + i) * 128] + (q ? b1 : b0);
        if (NW == 2 && p.pair) {
          const int j = n0 + row;
          if (j < p.n) dst[j] = (sum[0] / (1.0f + expf(-sum[0]))) * sum[NW - 1];   // src/llm/decoder.rs:1319-1322
        } else {
#pragma unroll
          for (int q = 0; q < NW; ++q) {
            const int j = n0 + q * kTileN + row;
            if (j < p.n) dst[j] = sum[q];
          }
        }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kIssue0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
}

// One activation row -> kPieces rows of bf16 images (with the fused RMSNorm).  Inside every 8 elements the order is 0 4 1 5
// 2 6 3 7, the order in which the codes leave a 32-bit word of nibbles.  One block per row of the padded tiles (rows past
// m are zero); a thread takes pieces of 8 elements and keeps up to NI of them in registers between the pass that
// finds the sum of squares and the pass that writes (NI 0: any length, read twice).
constexpr int kPrepThreads = 512;
template <int NI>
__global__ void __launch_bounds__(kPrepThreads) tc5_prep_kernel(const float* __restrict__ x, const float* __restrict__ norm_w, float eps,
                                                                unsigned char* __restrict__ xq, int m, int mp, int k) {
  __shared__ float s_ss[kPrepThreads / 32];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // the product may set up and fetch weights; its images wait for this grid's end
  const int row = blockIdx.x, tid = threadIdx.x, step = (int)blockDim.x * 8;
  const bool live = row < m;
  const float* xr = x + (size_t)(live ? row : 0) * k;
  float v[NI > 0 ? NI : 1][8];
  auto load = [&](const float* src, float (&o)[8]) {
    const float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + 4);
    o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w; o[4] = b.x; o[5] = b.y; o[6] = b.z; o[7] = b.w;
  };
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    const int e = i * step + tid * 8;
#pragma unroll
    for (int j = 0; j < 8; ++j) v[i][j] = 0.f;
    if (live && e < k) load(xr + e, v[i]);
  }
  float inv = 1.f;
  if (norm_w != nullptr) {   // fast_rms_norm, src/quantization/fused_ops.rs:1066-1117
    float ss = 0.f;
    if constexpr (NI > 0) {
#pragma unroll
      for (int i = 0; i < NI; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) ss = fmaf(v[i][j], v[i][j], ss);
    } else if (live) {
      for (int e = tid * 8; e < k; e += step) {
        load(xr + e, v[0]);
#pragma unroll
        for (int j = 0; j < 8; ++j) ss = fmaf(v[0][j], v[0][j], ss);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((tid & 31) == 0) s_ss[tid >> 5] = ss;
    __syncthreads();
    ss = 0.f;
    for (int i = 0; i < (int)blockDim.x / 32; ++i) ss += s_ss[i];
    inv = 1.0f / sqrtf(ss / (float)k + eps);
  }
  auto write = [&](int e, float (&o)[8]) {
    if (norm_w != nullptr) {
      float w[8];
      load(norm_w + e, w);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = (o[j] * inv) * w[j];
    }
    uint32_t img[kPieces][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {   // the pair (i, i + 4)
      float r0 = o[i], r1 = o[i + 4];
#pragma unroll
      for (int pc = 0; pc < kPieces; ++pc) {   // the upper 16 bits are a bf16 number; the remainder is exact, the last one fits
        const uint32_t h0 = __float_as_uint(r0) & 0xFFFF0000u, h1 = __float_as_uint(r1) & 0xFFFF0000u;
        r0 -= __uint_as_float(h0);
        r1 -= __uint_as_float(h1);
        img[pc][i] = (h0 >> 16) | h1;
      }
    }
    const int c = e >> 6, jp = (e >> 3) & 7, r = row % mp;
    unsigned char* dst = xq + ((size_t)(row / mp) * (k / kKC) + c) * (size_t)(kPieces * mp * 128) + r * 128 + ((jp ^ (r & 7)) * 16);
#pragma unroll
    for (int pc = 0; pc < kPieces; ++pc)
      *reinterpret_cast<uint4*>(dst + (size_t)pc * mp * 128) = make_uint4(img[pc][0], img[pc][1], img[pc][2], img[pc][3]);
  };
  if constexpr (NI > 0) {
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int e = i * step + tid * 8;
      if (e < k) write(e, v[i]);
    }
  } else {
    for (int e = tid * 8; e < k; e += step) {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[0][j] = 0.f;
      if (live) load(xr + e, v[0]);
      write(e, v[0]);
    }
  }
}

int g_tc5_enabled = 1;

using Kernel = void (*)(const Tc5Params);
struct Variant { int mp, nw; Kernel kern[3]; int threads[3]; size_t smem[3]; };
template <int MP, int NW>
constexpr Variant variant() {
  return Variant{MP, NW, {w4_tc5_kernel<MP, NW, 32>, w4_tc5_kernel<MP, NW, 64>, w4_tc5_kernel<MP, NW, 128>},
                 {Shape<MP, NW, 32>::kThreads, Shape<MP, NW, 64>::kThreads, Shape<MP, NW, 128>::kThreads},
                 {Shape<MP, NW, 32>::kSmem, Shape<MP, NW, 64>::kSmem, Shape<MP, NW, 128>::kSmem}};
}
const Variant kVariants[] = {variant<16, 1>(), variant<32, 1>(), variant<48, 1>(), variant<64, 1>(),
                             variant<16, 2>(), variant<32, 2>(), variant<48, 2>(), variant<64, 2>()};

// Whole tiles in turn leave SMs idle when they do not fill the last wave: 112 CTAs of 148 for a gate/up pair of 14336 features or for
// 4096 features and 333 rows.  A range of units of K for every CTA, which may begin and end inside a tile, leaves none, but
// the ends cost an exchange through memory: an end 1.6 + 0.017 per accumulator column, and what the last CTA of a tile reads.
// Measured, whole tiles (or equal parts) / ranges over all SMs, groups of 32: 333 x 14336 -> 4096 153 / 128 us, 200 x 4096 -> 14336 94 / 90, the pair of
// 200 rows 4096 -> 14336 186 / 166, of 100 rows 105 / 97, of 16 rows 35.9 / 33.8; but 333 x 4096 -> 6144 55 / 64, 200 x 4096 -> 4096 32 / 36.
// The cost of a launch in microseconds, pre-pass included, chosen so that the plan it picks is near the best one of 624 calls (4796 plans
// of every variant, 16 to 512 rows, 26 matrices of 1024 to 28672 rows, groups of 32 to 128): 0.4% from it on average, 9% at worst; the constants before the
// copying thread lost its divisions picked plans 1.7% from the best on average and 15% at worst on a part of them.  A stage of 64 elements takes what kStage
// says - the roles' instruction chains, not HBM or the tensor pipe -, a tile's end 0.051 per accumulator column.
constexpr int kPadRows = 64;   // padding of the last tile: less than the largest tile
constexpr int kTickets = 1024;
constexpr double kStage[2][4] = {{0.288, 0.281, 0.341, 0.393}, {0.451, 0.479, 0.709, 0.712}};   // one or two weight tiles, 16 to 64 rows
constexpr double kLarge[2][2][4] = {{{0.90, 0.90, 0.915, 0.911}, {1.104, 1.093, 0.898, 0.894}},   // of that with groups of 64
                                    {{0.90, 0.893, 0.883, 0.887}, {1.025, 1.059, 0.757, 0.852}}};   // and of 128
struct Plan { const Variant* v; int mtiles, ntiles, grid, per, more; double cost; };   // per, more: Tc5Params
double plan_cost(const Plan& p, int64_t k, int g) {
  const int nw = p.v->nw - 1, mp = p.v->mp / 16 - 1;
  const double stage = kStage[nw][mp] * (g > 32 ? kLarge[g / 128][nw][mp] : 1.0), cols = p.v->mp * p.v->nw;
  const int64_t tiles = (int64_t)p.mtiles * p.ntiles, ku = k / kUnit;
  const double prep = 3.3 + 0.12e-3 * (double)k;
  if (p.per == 0) return (double)((tiles + p.grid - 1) / p.grid) * ((double)(k / kKC) * stage + 0.051 * cols) + prep;
  const int units = p.per + (p.more ? 1 : 0);
  const double share = (double)units / (double)ku;                                                    // of a tile, or tiles, a CTA
  const double ends = share >= 1.0 ? share + 1.0 : (p.more == 0 && ku % units == 0 ? 1.0 : 1.0 + share);   // tiles that a CTA ends or leaves
  const double shared = ends < 2.0 ? ends : 2.0, parts = share >= 1.0 ? 2.0 : (double)p.grid / (double)tiles;
  return units * (kUnit / kKC) * stage + ends * 0.051 * cols + shared * (1.64 + 0.0171 * cols + 0.0067 * cols * parts) + prep;
}
// At 9 to 16 rows, the choice between this kernel and the integer one: what this kernel cost with whole tiles or equal parts of K, eight
// unpacking warps and its pre-pass in front, as the two were measured against each other (w4_mma_cost).  It costs less now, so that calls near the
// line are left where they were and not where they take least: the pair of 16 rows 4096 -> 1792 takes 23.8 us on the integer kernel, of 17 rows 16.3 here.
double few_rows_cost(int m, int64_t n, int64_t k, int g, bool pair) {
  double best = 1e30;
  for (int nw = pair ? 2 : 1; nw <= 2; ++nw)
    for (int mp = 16; mp <= 64; mp += 16)
      for (int ks = 1; ks <= kMaxSplit; ++ks) {
        if (ks > 1 && (pair || (k / kUnit) % ks != 0)) continue;
        const int rows = pair ? kTileN : kTileN * nw;
        const int64_t tiles = (int64_t)((m + mp - 1) / mp) * ((n + rows - 1) / rows) * ks;
        const double stage = (nw == 2 ? 0.43 + 0.0044 * mp : 0.24 + 0.0023 * mp) * (g > 32 ? 0.85 : 1.0), cols = mp * nw;
        const double c = (double)((tiles + sm_count() - 1) / sm_count()) * ((double)(k / ks / kKC) * stage + 0.05 * cols + (ks > 1 ? 3.0 + 0.024 * cols * ks : 0.0)) + 5.0;
        if (c < best) best = c;
      }
  return best;
}
// Parts of K: 32768 columns of partial sums per row (4096 x 14336 in 8 parts), 40 MB at most.
size_t part_bytes(int m) {
  const size_t rows = (size_t)(m < kMaxRows ? m : kMaxRows) + kPadRows;
  return (rows < 320 ? rows : 320) * 32768 * sizeof(float);
}
Plan choose_plan(int m, int64_t n, int64_t k, int g, bool pair) {
  const int sms = sm_count();
  Plan best{};
  best.cost = 1e30;
  for (const Variant& v : kVariants) {
    if (pair && v.nw != 2) continue;
    const int rows = pair ? kTileN : kTileN * v.nw;
    Plan p{&v, (m + v.mp - 1) / v.mp, (int)((n + rows - 1) / rows), 0, 0, 0, 0.0};
    const int64_t tiles = (int64_t)p.mtiles * p.ntiles, ku = k / kUnit;
    p.grid = (int)(tiles < sms ? tiles : sms);
    p.cost = plan_cost(p, k, g);
    if (p.cost < best.cost) best = p;
    if (tiles > kTickets) continue;
    // Ranges of units: one CTA per SM, or as many as leave every tile the same number of parts
    for (int parts = 0; parts <= kMaxSplit; ++parts) {
      const int64_t grid = parts ? tiles * parts : sms;
      if (parts == 1 || grid > sms || grid > tiles * ku) continue;
      if (2 * (size_t)grid * v.mp * v.nw * kTileN * sizeof(float) > part_bytes(m)) continue;
      p.grid = (int)grid; p.per = (int)(tiles * ku / grid); p.more = (int)(tiles * ku % grid);
      if (p.more == 0 && p.per % ku == 0) continue;   // whole tiles
      if ((p.more == 0 && ku % p.per == 0 ? ku / p.per : (ku - 2) / p.per + 2) > kMaxSplit) continue;
      p.cost = plan_cost(p, k, g);
      if (p.cost < best.cost) best = p;
    }
  }
  return best;
}

size_t image_bytes(int rows, int64_t k) { return (size_t)(k / kKC) * kPieces * (size_t)rows * 128; }
}  // namespace

void set_tc5_enabled(int on) { g_tc5_enabled = on; }

int tc5_fault_flag() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_tc5_fault, sizeof(int)) != cudaSuccess) return -1;
  return v;
}

// Images, then the parts of K.
size_t w4_tc5_scratch_bytes(int m, int64_t k) {
  const int rows = (m < kMaxRows ? m : kMaxRows) + kPadRows;
  return image_bytes(rows, (k + kKC - 1) / kKC * kKC) + part_bytes(m);
}

bool w4_tc5_supported(const GemvArgs& a) {
  if (!g_tc5_enabled || a.m < kMinRows || !tma_encoder()) return false;
  if (a.k % 128 != 0 || a.n < 1 || (a.g != 32 && a.g != 64 && a.g != 128)) return false;
  if (a.x_ss8 || a.out_scaled || a.out_ss8 || a.x_normed_out) return false;
  if ((reinterpret_cast<uintptr_t>(a.w) & 15) || (a.w2 && (reinterpret_cast<uintptr_t>(a.w2) & 15))) return false;
  if ((reinterpret_cast<uintptr_t>(a.scales) & 15) || (a.w2 && (reinterpret_cast<uintptr_t>(a.scales2) & 15))) return false;   // boxes and copies of up to 16 bytes
  return a.m >= kSureRows || few_rows_cost(a.m, a.n, a.k, a.g, a.w2 != nullptr) < w4_mma_cost(a.n, a.k, a.w2 != nullptr);
}

// Launches of one call: kMaxRows rows at a time, the pre-pass and the product.
int w4_tc5_launches(int m) { return 2 * ((m + kMaxRows - 1) / kMaxRows); }

tb_status launch_w4_tc5(const GemvArgs& a, void* scratch, int* tickets, cudaStream_t stream) {
  if (!w4_tc5_supported(a)) return fail(TB_ERR_UNSUPPORTED, "TB_UNSUPPORTED: tcgen05 product: m=%d n=%lld k=%lld", a.m, (long long)a.n, (long long)a.k);
  const bool pair = a.w2 != nullptr;
  const int gi = a.g == 32 ? 0 : (a.g == 64 ? 1 : 2);
  unsigned char* xq = static_cast<unsigned char*>(scratch);
  const int slabs = (a.m + kMaxRows - 1) / kMaxRows, per = (a.m + slabs - 1) / slabs;
  for (int m0 = 0; m0 < a.m; m0 += per) {
    const int mc = a.m - m0 < per ? a.m - m0 : per;
    const Plan plan = choose_plan(mc, a.n, a.k, a.g, pair);
    const Variant& v = *plan.v;
    Tc5Params p;
    p.scales[0] = a.scales; p.scales[1] = a.scales2; p.bias[0] = a.bias; p.bias[1] = a.bias2;
    p.resid = a.resid ? a.resid + (size_t)m0 * a.n : nullptr;
    p.out = a.out + (size_t)m0 * a.n;
    p.xq = xq;
    p.parts = reinterpret_cast<float*>(xq + image_bytes(plan.mtiles * v.mp, a.k));
    p.tickets = tickets;
    p.m = mc; p.n = (int)a.n; p.k = (int)a.k; p.ng = (int)(a.k / a.g);
    p.mtiles = plan.mtiles; p.ntiles = plan.ntiles; p.per = plan.per; p.more = plan.more;
    p.pair = pair ? 1 : 0;
    for (int q = 0; q < (pair ? 2 : 1); ++q) {
      if (!tma_matrix_map(&p.w[q], CU_TENSOR_MAP_DATA_TYPE_UINT8, q ? a.w2 : a.w, a.k / 2, a.n, a.k / 2, 64, kTileN, CU_TENSOR_MAP_SWIZZLE_64B) ||
          (a.g == 32 && !tma_matrix_map(&p.s[q], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, q ? a.scales2 : a.scales, p.ng, a.n, (int64_t)p.ng * 4, 4, kTileN, CU_TENSOR_MAP_SWIZZLE_NONE)))
        return fail(TB_ERR_CUDA, "tcgen05 product: no TMA description of a %lld x %lld matrix", (long long)a.n, (long long)a.k);
    }
    const int ni = (int)((a.k + kPrepThreads * 8 - 1) / (kPrepThreads * 8));
    int threads = (int)((a.k / 8 + 31) / 32 * 32);
    if (threads > kPrepThreads) threads = kPrepThreads;
    const auto prep = ni == 1 ? tc5_prep_kernel<1> : ni == 2 ? tc5_prep_kernel<2> : ni <= 4 ? tc5_prep_kernel<4> : tc5_prep_kernel<0>;
    prep<<<(unsigned)(plan.mtiles * v.mp), threads, 0, stream>>>(a.x + (size_t)m0 * a.k, a.norm_w, a.eps, xq, mc, v.mp, (int)a.k);
    TB_CUDA_TRY(cudaGetLastError());
    TB_CUDA_TRY(cudaFuncSetAttribute(v.kern[gi], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)v.smem[gi]));
    // Beside the pre-pass (which itself starts when all in front of it is complete): the tensor memory, the barriers and the first
    // ring of weights are ready when the images are.  The MLP of 16 rows at 4096 / 14336: 71.1 -> 66.2 us; 333 rows gain nothing.
    // (Weights that ran ahead of the images all the way, not only by the first ring, cost 27 -> 40 us at 16 x 14336 x 4096: the
    // copying thread's wait for a unit held back images that others waited for.)
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)plan.grid);
    cfg.blockDim = dim3((unsigned)v.threads[gi]);
    cfg.dynamicSmemBytes = v.smem[gi];
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    TB_CUDA_TRY(cudaLaunchKernelEx(&cfg, v.kern[gi], p));
  }
  return TB_OK;
}

}  // namespace tb
