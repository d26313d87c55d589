// Grouped INT4 W4A32 products for 2 to 8 activation rows on mma.sync, the weights read from HBM once
// (gemm_w4a32_grouped, src/quantization/gemv.rs:1690-1725; fused_swiglu_mlp_batched, src/quantization/fused_ops.rs:1267-1319).
//
// The 4-bit codes are exact in bf16 and the fp32 activations are split into three bf16 pieces that carry all 24 bits of
// every value (rows_prep_kernel, with the fused RMSNorm; splitting them in every CTA instead, without a pre-pass, made the
// consumers' chains longer: 37.7 against 35.1 us for the gate/up pair).  Per 32 elements of K a warp multiplies 16 weight rows with 8
// activation rows in six mma.sync.m16n8k16 into fresh fp32 accumulators, one per piece, and adds their sums, times their
// rows' scale, to its registers: about 45 instructions per 16 x 32 codes.  (The integer form that was here combined
// three int32 sums, converted and rescaled them per block and activation, and its 16-byte cp.async of every (row, block) cost as
// many instructions again.)
//
// What bounds it is the streaming, so the CTA is laid out for that: persistent, one per SM, 16 consumer warps, one warp whose lanes
// issue the copies and three that fetch the scales (a row's may begin on 4 bytes; one warp for all of them needed 3 us a stage, four
// times as long as HBM).  K is the outer loop: a CTA takes ALL of its weight rows through a ring of stages of 256 or 512
// elements of K, so that the images of the activations, 1.5 KB per 32 elements, as many bytes as 75 weight rows, pass once per CTA and
// not once per tile.  Within a stage a warp takes one 32-element block, for every tile of 16 rows (up to seven tiles, stages of 512:
// sixteen blocks for sixteen warps) or for every other one (up to fourteen, stages of 256): images are read from shared memory
// once for up to seven tiles, a lane's words of a tile are two 4-byte reads that the copy's 128-byte swizzle spreads over all
// banks.  A warp goes through the stages one after the other, so what it does in one is a chain that bounds narrow matrices;
// hence the long stages and an accumulator per piece (one for all six products: six times the latency of one).
// The warps' sums meet in shared memory at the end.  CTAs begin at different places of K (and go around): all of them read the same
// images, and the same lines at the same time queue up in L2.  K is never split over CTAs: a CTA with one or two
// tiles mostly reads images, and that costs less than an exchange of sums (clusters of 4 with distributed shared memory: 8 us
// more a launch).
//
// A gate/up pair puts eight gate rows and the same eight up rows into one tile: the finer tiles balance the SMs, and both sums of a
// neuron end in one lane's registers.
//
// Launched behind its pre-pass with programmatic serialization: the ring fills with weights while the pre-pass runs.  The
// pre-pass itself is launched in plain order, so everything in front of it is complete before either starts.  Every mbarrier wait is
// bounded.
#include <cuda_bf16.h>

#include <type_traits>

#include "tb_common.cuh"
#include "tc5.cuh"
#include "tma_map.cuh"
#include "w4_math.cuh"

namespace tb {

namespace {

using namespace tc5;

constexpr int kWarps = 16;               // consumers
constexpr int kScaleThreads = 96;
constexpr int kThreads = kWarps * 32 + 32 + kScaleThreads;
constexpr int kTileBytes = 16 * 128;     // 16 weight rows x 256 elements of K
constexpr int kPieces = 3;
constexpr int kImageBytes = kPieces * 512;   // of one block: [piece][lane][16 bytes]
constexpr int kMaxTiles = 14, kWarpTiles = kMaxTiles / 2;   // tiles of a CTA's pass and of a warp
constexpr int kMaxStages = 8;
constexpr size_t kSmemMax = 226 * 1024;
constexpr int kMaxRowsM = 8;

__device__ int g_rows_fault = 0;
int g_rows_enabled = 1;

struct RowsParams {
  CUtensorMap w[2];          // [n, k / 2] bytes, boxes of 128 x 16 rows (a pair: x 8 rows)
  const float* scales[2];
  const float* bias[2];
  const float* resid;
  float* out;
  const unsigned char* xq;   // [block of K][piece][lane][16 bytes]
  int m, n, nb32, ng, gshift;
  int tiles;                 // of the matrix
  int pass_tiles, stages;    // tiles per pass of a CTA, ring depth
  int copy;                  // bytes per copy of scales: 16, 8 or 4
};

__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void consumer_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kWarps * 32) : "memory"); }
// kBytes (16, 8 or 4) to shared memory, of which the first `live` from memory and zeros behind them.
template <int kBytes>
__device__ __forceinline__ void cp_async(uint32_t dst, const void* src, int live) {
  if (kBytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live) : "memory");
  else if (kBytes == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(live) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(live) : "memory");
}

// One stage of a warp: its block of 32 elements for its N tiles, kStep bytes apart.  images, words and scales: this lane's of the
// first tile.
template <int N, int kStep>
__device__ __forceinline__ void stage_tiles(float (&acc)[kWarpTiles][4], const unsigned char* images, const unsigned char* words, const unsigned char* scales, int scale_8) {
  uint32_t b[kPieces][4];
#pragma unroll
  for (int pc = 0; pc < kPieces; ++pc) {
    const uint4 v = *reinterpret_cast<const uint4*>(images + pc * 512);
    b[pc][0] = v.x; b[pc][1] = v.y; b[pc][2] = v.z; b[pc][3] = v.w;
  }
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const uint32_t w0 = *reinterpret_cast<const uint32_t*>(words + i * kStep), w1 = *reinterpret_cast<const uint32_t*>(words + i * kStep + 1024);
    const float s0 = *reinterpret_cast<const float*>(scales + i * (kStep / kTileBytes * 2) * scale_8);
    const float s1 = *reinterpret_cast<const float*>(scales + i * (kStep / kTileBytes * 2) * scale_8 + scale_8);
    uint32_t u0[4], u1[4];
    unpack8(w0, u0);
    unpack8(w1, u1);
    float d[kPieces][4];
#pragma unroll
    for (int pc = 0; pc < kPieces; ++pc) {
#pragma unroll
      for (int e = 0; e < 4; ++e) d[pc][e] = 0.f;
      mma_bf16(d[pc], u0[0], u1[0], u0[1], u1[1], b[pc][0], b[pc][1]);
      mma_bf16(d[pc], u0[2], u1[2], u0[3], u1[3], b[pc][2], b[pc][3]);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[i][e] = fmaf(d[0][e] + (d[1][e] + d[2][e]), e < 2 ? s0 : s1, acc[i][e]);
  }
}

template <bool PAIR, int kBlocks>
__global__ void __launch_bounds__(kThreads, 1) w4_rows_kernel(const __grid_constant__ RowsParams p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full[kMaxStages], empty[kMaxStages];
  __shared__ int s_abort;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  constexpr int kHalves = 16 / kBlocks;     // 1: a warp takes every tile, 2: every other one
  constexpr int kSlots = kBlocks / 2;       // of partial sums
  constexpr int kPanels = kBlocks / 8;      // boxes of 256 elements of K
  const int TS = p.pass_tiles, NS = p.stages;
  const int row_scales = kBlocks >> p.gshift;                       // scales of a row and stage
  const int w_bytes = TS * kTileBytes * kPanels, s_bytes = TS * 16 * row_scales * 4;
  const int stage_bytes = (w_bytes + s_bytes + kBlocks * kImageBytes + 1023) & ~1023;
  float* red = reinterpret_cast<float*>(smem + (size_t)NS * stage_bytes);   // [kSlots][TS][4][32]
  const int tile0 = (int)((int64_t)p.tiles * blockIdx.x / gridDim.x), tile1 = (int)((int64_t)p.tiles * (blockIdx.x + 1) / gridDim.x);
  const int nk = (p.nb32 + kBlocks - 1) / kBlocks;   // stages of K
  const int kfirst = (int)((int64_t)blockIdx.x * nk / gridDim.x);   // where this CTA begins
  const int passes = (tile1 - tile0 + TS - 1) / TS;

  if (tid == 0) {
    s_abort = 0;
    for (int s = 0; s < NS; ++s) {
      mbar_init(&full[s], 1 + kScaleThreads);   // the bytes announced by the producer, and every scale thread's copies
      mbar_init(&empty[s], kWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  const int total = passes * nk;   // stages of this CTA
  if (warp > kWarps) {
    // ---------------- scales: zeros past the matrix (a stale one could be anything, and 0 times it NaN) ----------------
    const int me = tid - (kWarps + 1) * 32, bytes = row_scales * 4;
    constexpr int kRows = (kMaxTiles * 16 + kScaleThreads - 1) / kScaleThreads;   // rows of a stage a thread takes
    const char* src[kRows];
    bool live[kRows];
    auto stream = [&](auto width) {
      constexpr int kCopy = decltype(width)::value;
      for (int it = 0, kc = kfirst, pass = 0; it < total; ++it) {
        const int slot = it % NS, t0 = tile0 + pass * TS, nt = min(TS, tile1 - t0);
        if (kc == kfirst) {
#pragma unroll
          for (int j = 0; j < kRows; ++j) {
            const int r = me + j * kScaleThreads, q = PAIR ? (r >> 3) & 1 : 0, row = PAIR ? (t0 + (r >> 4)) * 8 + (r & 7) : t0 * 16 + r;
            live[j] = r < nt * 16 && row < p.n;
            src[j] = reinterpret_cast<const char*>((q ? p.scales[1] : p.scales[0]) + (live[j] ? (int64_t)row * p.ng : 0));
          }
        }
        if (it >= NS && !mbar_wait(&empty[slot], (uint32_t)(it / NS - 1) & 1u, &s_abort, &g_rows_fault)) break;
        const int at = kc * bytes, want = p.ng * 4 - at;   // bytes into a row, and what the row still has
        const uint32_t dst = smem_u32(smem) + (uint32_t)(slot * stage_bytes + w_bytes);
#pragma unroll
        for (int j = 0; j < kRows; ++j) {
          const int r = me + j * kScaleThreads;
          if (r >= nt * 16) break;
          for (int b = 0; b < bytes; b += kCopy) {
            const bool have = live[j] && b < want;   // (whole copies: a row's end is a multiple of the copy's width)
            cp_async<kCopy>(dst + (uint32_t)(r * bytes + b), src[j] + (have ? at + b : 0), have ? kCopy : 0);
          }
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&full[slot])) : "memory");
        if (++kc == nk) kc = 0;
        if (kc == kfirst) ++pass;
      }
    };
    if (p.copy == 16) stream(std::integral_constant<int, 16>());
    else if (p.copy == 8) stream(std::integral_constant<int, 8>());
    else stream(std::integral_constant<int, 4>());
    asm volatile("cp.async.wait_all;" ::: "memory");
    return;
  }
  if (warp == kWarps) {
    // ---------------- copies ----------------
    auto weights = [&](int pass, int kc, int slot) {
      const int t0 = tile0 + pass * TS, nt = min(TS, tile1 - t0);
      const int panels = kPanels == 1 || (kc * kBlocks + 8 < p.nb32) ? kPanels : 1;   // (the last stage may hold one of two)
      if (lane == 0) mbar_expect_tx(&full[slot], (uint32_t)(nt * kTileBytes * panels + kBlocks * kImageBytes));
      __syncwarp();
      if (lane < nt * panels) {
        const int pn = lane / nt, tile = lane - pn * nt;
        const uint32_t dst = smem_u32(smem) + (uint32_t)(slot * stage_bytes + (pn * TS + tile) * kTileBytes), bar = smem_u32(&full[slot]);
        const int kx = (kc * kPanels + pn) * 128;
        if (PAIR) {
          tma_box(dst, &p.w[0], kx, (t0 + tile) * 8, bar);
          tma_box(dst + kTileBytes / 2, &p.w[1], kx, (t0 + tile) * 8, bar);
        } else {
          tma_box(dst, &p.w[0], kx, (t0 + tile) * 16, bar);
        }
      }
    };
    auto images = [&](int kc, int slot) {
      if (lane == 0)
        bulk_g2s(smem + (size_t)slot * stage_bytes + w_bytes + s_bytes, p.xq + (size_t)kc * (kBlocks * kImageBytes), kBlocks * kImageBytes, &full[slot]);
    };
    const int first = min(NS, total);
    int it = 0, kc = kfirst, pass = 0;
    auto next = [&] {
      if (++kc == nk) kc = 0;
      if (kc == kfirst) ++pass;
    };
    for (; it < first; ++it, next()) weights(pass, kc, it);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    // Behind the own wait, so that completion stays transitive along a chain.  The attention of a step is launched early behind its QKV
    // product: two sequences of width 1024 347 -> 335 us a step, four of width 2048 543 -> 526.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    for (int i = 0, c = kfirst; i < first; ++i) {
      images(c, i);
      if (++c == nk) c = 0;
    }
    for (; it < total; ++it, next()) {
      const int slot = it % NS;
      if (!__all_sync(0xffffffffu, mbar_wait(&empty[slot], (uint32_t)(it / NS - 1) & 1u, &s_abort, &g_rows_fault))) break;
      weights(pass, kc, slot);
      images(kc, slot);
    }
    if (it < total) {   // given up: the copies in flight land before the shared memory goes
      int no_abort = 0;
      for (int i = max(0, it - NS); i < it; ++i) mbar_wait(&full[i % NS], (uint32_t)(i / NS) & 1u, &no_abort, &g_rows_fault);
    }
    return;
  }

  // ---------------- consumers ----------------
  const int kw = warp % kBlocks, half = warp / kBlocks, g = lane >> 2, t = lane & 3;
  const int scale_8 = 8 * row_scales * 4;   // eight rows of scales
  const int word_at = ((kw >> 3) * TS + half) * kTileBytes + g * 128 + (((kw & 7) ^ g) << 4) + t * 4;   // this lane's word of the first tile's row g (g + 8: 1024 on)
  const int scale_at = w_bytes + half * 2 * scale_8 + (g * row_scales + (kw >> p.gshift)) * 4;
  const int image_at = w_bytes + s_bytes + kw * kImageBytes + lane * 16;
  int it = 0;
  for (int pass = 0; pass < passes; ++pass) {
    const int t0 = tile0 + pass * TS, nt = min(TS, tile1 - t0), mine = (nt - half + kHalves - 1) / kHalves;   // tiles half, half + kHalves, ...
    float acc[kWarpTiles][4];
#pragma unroll
    for (int i = 0; i < kWarpTiles; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][e] = 0.f;
    for (int c = 0, kc = kfirst; c < nk; ++c, ++it, kc = kc + 1 == nk ? 0 : kc + 1) {
      const int slot = it % NS;
      if (!__all_sync(0xffffffffu, mbar_wait(&full[slot], (uint32_t)(it / NS) & 1u, &s_abort, &g_rows_fault))) break;
      const unsigned char* st = smem + slot * stage_bytes;
      if (kc * kBlocks + kw < p.nb32) {   // (the last stage may hold fewer blocks)
        constexpr int kStep = kHalves * kTileBytes;
        switch (mine) {   // whole chains of tiles, so that their products overlap
          case 1: stage_tiles<1, kStep>(acc, st + image_at, st + word_at, st + scale_at, scale_8); break;
          case 2: stage_tiles<2, kStep>(acc, st + image_at, st + word_at, st + scale_at, scale_8); break;
          case 3: stage_tiles<3, kStep>(acc, st + image_at, st + word_at, st + scale_at, scale_8); break;
          case 4: stage_tiles<4, kStep>(acc, st + image_at, st + word_at, st + scale_at, scale_8); break;
          case 5: stage_tiles<5, kStep>(acc, st + image_at, st + word_at, st + scale_at, scale_8); break;
          case 6: stage_tiles<6, kStep>(acc, st + image_at, st + word_at, st + scale_at, scale_8); break;
          case 7: stage_tiles<7, kStep>(acc, st + image_at, st + word_at, st + scale_at, scale_8); break;
        }
      }
      __syncwarp();   // lane 0 arrives for all: behind the other lanes' reads
      if (lane == 0) mbar_arrive(&empty[slot]);
    }
    // ---- the warps that shared a tile's K: the upper half leaves its sums, the lower half adds its own ----
    consumer_barrier();   // the last pass's sums have been read
    if (kw >= kSlots)
#pragma unroll
      for (int i = 0; i < kWarpTiles; ++i)
        if (i < mine)
#pragma unroll
          for (int e = 0; e < 4; ++e) red[(((kw - kSlots) * TS + kHalves * i + half) * 4 + e) * 32 + lane] = acc[i][e];
    consumer_barrier();
    if (kw < kSlots)
#pragma unroll
      for (int i = 0; i < kWarpTiles; ++i)
        if (i < mine)
#pragma unroll
          for (int e = 0; e < 4; ++e) red[((kw * TS + kHalves * i + half) * 4 + e) * 32 + lane] += acc[i][e];
    consumer_barrier();
    // ---- outputs: neighbouring threads take neighbouring features ----
    constexpr int kFeatures = PAIR ? 8 : 16;   // of a tile
    const int feats = nt * kFeatures;
    auto sum = [&](int tile, int reg, int ln) {
      const float* at = red + (tile * 4 + reg) * 32 + ln;
      float v = 0.f;
#pragma unroll
      for (int z = 0; z < kSlots; ++z) v += at[z * TS * 128];
      return v;
    };
    for (int o = tid; o < feats * p.m; o += kWarps * 32) {
      const int m = o / feats, f = o - m * feats, tile = f / kFeatures, r = f - tile * kFeatures;
      const int row = (t0 + tile) * kFeatures + r, ln = (r & 7) * 4 + (m >> 1);
      if (row >= p.n) continue;
      float v;
      if (PAIR) {
        const float gg = sum(tile, m & 1, ln) + (p.bias[0] ? p.bias[0][row] : 0.f);
        const float uu = sum(tile, 2 + (m & 1), ln) + (p.bias[1] ? p.bias[1][row] : 0.f);
        v = (gg / (1.0f + expf(-gg))) * uu;   // src/quantization/fused_ops.rs:1305-1311
      } else {
        v = sum(tile, (r >> 3) * 2 + (m & 1), ln) + (p.bias[0] ? p.bias[0][row] : 0.f);
        if (p.resid) v = p.resid[(int64_t)m * p.n + row] + v;
      }
      p.out[(int64_t)m * p.n + row] = v;
    }
  }
}

// x (rows m, after the fused RMSNorm) -> images.  Four threads share a block of 32 elements, eight elements each; one block row
// of the grid per activation row, the padded ones and the blocks past K zeros.
constexpr int kPrepThreads = 512;
__global__ void __launch_bounds__(kPrepThreads) rows_prep_kernel(const float* __restrict__ x, const float* __restrict__ norm_w, float eps,
                                                                 unsigned char* __restrict__ xq, int m_rows, int k, int blocks,
                                                                 float* __restrict__ x_normed_out) {
  __shared__ float s_part[kPrepThreads / 32];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // the product may fill its ring meanwhile; it waits for this grid's end
  const int m = blockIdx.x;
  const bool live = m < m_rows;
  const float* xr = x + (int64_t)(live ? m : 0) * k;
  const int blk = blockIdx.y * (kPrepThreads / 4) + ((int)threadIdx.x >> 2), t = threadIdx.x & 3, at = blk * 32 + t * 8;
  float v[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = 0.f;
  if (live && at < k) {
    const float4 a = *reinterpret_cast<const float4*>(xr + at), b = *reinterpret_cast<const float4*>(xr + at + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  }
  if (norm_w != nullptr && live) {   // fast_rms_norm, src/quantization/fused_ops.rs:1066-1117
    float ss = 0.f;
    for (int i = threadIdx.x; i < (k >> 2); i += kPrepThreads) {
      const float4 f = reinterpret_cast<const float4*>(xr)[i];
      ss = fmaf(f.x, f.x, ss); ss = fmaf(f.y, f.y, ss); ss = fmaf(f.z, f.z, ss); ss = fmaf(f.w, f.w, ss);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < kPrepThreads / 32; ++i) tot += s_part[i];
    const float inv_rms = 1.0f / sqrtf(tot / (float)k + eps);
    if (at < k) {
      const float4 a = *reinterpret_cast<const float4*>(norm_w + at), b = *reinterpret_cast<const float4*>(norm_w + at + 4);
      const float w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        v[j] = (v[j] * inv_rms) * w[j];
        if (x_normed_out != nullptr) x_normed_out[(int64_t)m * k + at + j] = v[j];
      }
    }
  }
  if (blk >= blocks) return;
  unsigned char* dst = xq + (size_t)blk * kImageBytes + ((m & 7) * 4 + t) * 16;
  uint32_t img[kPieces][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {   // the pair (i, i + 4)
    float r0 = v[i], r1 = v[i + 4];
#pragma unroll
    for (int pc = 0; pc < kPieces; ++pc) {   // the upper 16 bits are a bf16 number; the remainder is exact, the last one fits
      const uint32_t h0 = __float_as_uint(r0) & 0xFFFF0000u, h1 = __float_as_uint(r1) & 0xFFFF0000u;
      r0 -= __uint_as_float(h0);
      r1 -= __uint_as_float(h1);
      img[pc][i] = (h0 >> 16) | h1;
    }
  }
#pragma unroll
  for (int pc = 0; pc < kPieces; ++pc) *reinterpret_cast<uint4*>(dst + pc * 512) = make_uint4(img[pc][0], img[pc][1], img[pc][2], img[pc][3]);
}

int padded_blocks(int64_t k) { return (int)((k / 32 + 15) / 16 * 16); }

struct Plan { int tiles, blocks, pass_tiles, stages; size_t smem; };
Plan choose_plan(int64_t n, int g, bool pair) {
  const int sms = sm_count(), rows = pair ? 8 : 16;
  Plan p;
  p.tiles = (int)((n + rows - 1) / rows);
  const int most = (p.tiles + sms - 1) / sms, passes = (most + kMaxTiles - 1) / kMaxTiles;
  p.pass_tiles = (most + passes - 1) / passes;
  p.blocks = p.pass_tiles <= kWarpTiles ? 16 : 8;
  const size_t stage = ((size_t)p.pass_tiles * (kTileBytes * p.blocks / 8 + 16 * (p.blocks / (g / 32)) * 4) + p.blocks * kImageBytes + 1023) / 1024 * 1024;
  const size_t red = (size_t)p.blocks / 2 * p.pass_tiles * 512;
  const size_t fit = (kSmemMax - 1024 - red) / stage;
  p.stages = fit < kMaxStages ? (int)fit : kMaxStages;
  p.smem = 1024 + p.stages * stage + red;
  return p;
}

// Where the integer kernel (w4_mma.cu) takes less.  Tiles: of the CTA with most of them, and per pass.  Measured with 32-element groups
// at 8 rows over 28 x 13 sizes (2 to 8 rows cost the same), us, integer / this kernel:
//   one tile a CTA and a long K, which it splits over four CTAs: 1024 x 8192 13.2 / 15.2, 2048 x 11008 17.7 / 19.0, 1024 x 14336 16.3 / 22.6;
//   next to no K, this kernel's start alone: 256 x 512 4.0 / 4.8, 2560 x 512 4.8 / 5.1, but 8960 x 512 6.7 / 6.4;
//   eight tiles a pass, the first count with stages of 256: pairs 8960 x 1536 13.1 / 15.1, 18944 x 4096 39.5 / 48.3, 9472 x 8960 48.8 / 51.1, single
//   18944 x 1536 13.8 / 14.4 (from K = 2048 on even); seven tiles, 14336 x 4096: 28.3 / 21.6;
//   many tiles of short rows, in pairs: 13824 x 1024 13.9 / 14.5, 24576 x 2048 31.6 / 32.9 (x 3072 44.1 / 44.4).
// Its reads want rows of 128 bytes: at K = 896 it is 1.2 to 1.5 times as slow as this kernel, but for 18944 pairs (16.1 / 18.2).
bool integer_takes_less(const GemvArgs& a) {
  const bool pair = a.w2 != nullptr, whole = a.k % 256 == 0;
  const Plan p = choose_plan(a.n, a.g, pair);
  const int most = (p.tiles + sm_count() - 1) / sm_count();
  const bool eight = p.pass_tiles == kWarpTiles + 1, one_pass = most <= kMaxTiles;
  if (pair) return eight ? whole || !one_pass : whole && a.k <= (one_pass ? (most >= 12 ? 1024 : 0) : 2048);
  if (most == 1 && a.k >= 8192) return true;
  return whole && (a.k <= 512 ? most <= 2 || most >= 6 : eight && a.k >= 1024 && a.k < 2048);
}

}  // namespace

void set_rows_enabled(int enabled) { g_rows_enabled = enabled; }

int rows_fault_flag() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_rows_fault, sizeof(int)) != cudaSuccess) return -1;
  return v;
}

size_t w4_rows_scratch_bytes(int64_t k) { return (size_t)padded_blocks(k) * kImageBytes; }

bool w4_rows_supported(const GemvArgs& a) {
  return g_rows_enabled && a.m >= 2 && a.m <= kMaxRowsM && a.k % 32 == 0 && tma_encoder() &&
         !((reinterpret_cast<uintptr_t>(a.w) | reinterpret_cast<uintptr_t>(a.w2) | reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.norm_w)) & 15) &&
         !integer_takes_less(a);
}

tb_status launch_w4_rows(const GemvArgs& a, void* scratch, cudaStream_t stream) {
  if (!w4_rows_supported(a)) return fail(TB_ERR_UNSUPPORTED, "TB_UNSUPPORTED: product of few rows: m=%d n=%lld k=%lld", a.m, (long long)a.n, (long long)a.k);
  const bool pair = a.w2 != nullptr;
  const Plan plan = choose_plan(a.n, a.g, pair);
  RowsParams p;
  p.scales[0] = a.scales; p.scales[1] = a.scales2; p.bias[0] = a.bias; p.bias[1] = a.bias2;
  p.resid = a.resid; p.out = a.out; p.xq = static_cast<const unsigned char*>(scratch);
  p.m = a.m; p.n = (int)a.n; p.nb32 = (int)(a.k / 32); p.ng = (int)(a.k / a.g); p.gshift = a.g == 32 ? 0 : (a.g == 64 ? 1 : 2);
  p.tiles = plan.tiles; p.pass_tiles = plan.pass_tiles; p.stages = plan.stages;
  const uintptr_t align = reinterpret_cast<uintptr_t>(a.scales) | (pair ? reinterpret_cast<uintptr_t>(a.scales2) : 0) | (uintptr_t)(p.ng * 4);
  const int row_bytes = (plan.blocks >> p.gshift) * 4;
  p.copy = align % 16 == 0 && row_bytes % 16 == 0 ? 16 : (align % 8 == 0 ? 8 : 4);
  for (int q = 0; q < (pair ? 2 : 1); ++q)
    if (!tma_matrix_map(&p.w[q], CU_TENSOR_MAP_DATA_TYPE_UINT8, q ? a.w2 : a.w, a.k / 2, a.n, a.k / 2, 128, pair ? 8 : 16, CU_TENSOR_MAP_SWIZZLE_128B))
      return fail(TB_ERR_CUDA, "product of few rows: no TMA description of a %lld x %lld matrix", (long long)a.n, (long long)a.k);
  const int blocks = padded_blocks(a.k);
  rows_prep_kernel<<<dim3(kMaxRowsM, (unsigned)((blocks + kPrepThreads / 4 - 1) / (kPrepThreads / 4))), kPrepThreads, 0, stream>>>(
      a.x, a.norm_w, a.eps, static_cast<unsigned char*>(scratch), a.m, (int)a.k, blocks, a.x_normed_out);
  TB_CUDA_TRY(cudaGetLastError());
  auto kern = plan.blocks == 16 ? (pair ? w4_rows_kernel<true, 16> : w4_rows_kernel<false, 16>) : (pair ? w4_rows_kernel<true, 8> : w4_rows_kernel<false, 8>);
  TB_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(plan.tiles < sm_count() ? plan.tiles : sm_count()));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = plan.smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  TB_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, p));
  return TB_OK;
}

}  // namespace tb
