// Windowed attention with mixed heads for a portion of one sequence in bf16: the two steps of
// window_attention.cu on the tensor cores.
//
//   scores   64 queries x one head per CTA: S = scale * Q K^T (mma.sync bf16, fp32 sums), masked.  To scratch goes
//            exp(S - m) with the row's running maximum m after the tile of 64 keys, and m beside it, so that an exponential
//            is taken once per score; with each row's maximum and sum at the end.  (A weight is then two exponentials' product instead of
//            one: against 64 bits 0.7e-7 to 1.7e-7 over 64 to 4096 keys either way, before the 16 bits of its two pieces, 2.4e-6.)
//   mix      16 queries x a group of up to 16 heads per CTA, 32 keys at a time.  weights = exp(S - max) / sum of
//            ALL heads at a (query, key), the scratch times one factor exp(m - max) / sum per (query, head, tile), are
//            contracted with T over the heads: one mma.sync per 16 x 16 heads
//            and 8 keys (T is exact in bf16; a weight goes in as two bf16 pieces, the second one the rounding
//            error of the first: 16 mantissa bits).  The mixed weights, again two pieces, meet the values in
//            two mma.sync each.  Scores and values of the next 32 keys stream in meanwhile.  With few query
//            blocks several CTAs share the keys of one; their parts are plain sums (the weights are normalised
//            already) and a last kernel adds them in order.
//
// Keys are numbered by the visible positions of the 64-query block: the kept positions, then one run from the
// first query's window to the last query.
#include "dense.cuh"
#include "window_attention.cuh"

namespace tb {

namespace {

constexpr int kQB = 64;      // queries per scores CTA; they share a key numbering
constexpr int kKeys = 64;    // keys per tile of the scores kernel
constexpr int kQM = 16;      // queries per mix CTA
constexpr int kKT = 32;      // keys per tile of the mix kernel
constexpr int kMixThreads = 512, kMixWarps = 16;
constexpr int kUnits = 8;      // most 16-column output units per warp of the mix kernels
constexpr int kWStride = kKT + 8;
constexpr int kWHead = 2 * kQM * kWStride + 32;   // elements of one head's two pieces
constexpr int kSStride = kKT + 4;                 // floats per (query, head) row of staged scores
constexpr int kMaxKeySplits = 4;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp16z(void* dst, const void* src, bool live) {   // zeros when not live
  const int n = live ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void ldm4(uint32_t (&r)[4], uint32_t at) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void ldm4(uint32_t (&r)[4], const void* p) { ldm4(r, smem_addr(p)); }
__device__ __forceinline__ void ldm4t(uint32_t (&r)[4], uint32_t at) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

struct MmaShape {
  int64_t stride;   // floats per (row, head) of the score scratch
  int refs;         // where a row's references, one per 64 keys, begin in it
  int row0, rows;   // rows of this pass
  int hg, kvs;      // mix: heads per group, most kv heads a group touches
  int score_splits; // scores: CTAs that share a query block's keys
  int key_splits;   // mix: CTAs that share a query block's keys
};

// grid (heads, blocks of 64 queries, score splits), 128 threads.  Bound by the shared-memory and store pipes (half of their slots)
// and by chains: matrix instructions take a fifth of the time.  KS: heads of KS * 16 elements, whose query fragments stay in
// registers; 0: any size, fragments read again for every tile.  With these, and with keys laid out so that a thread stores four
// at once, 512 queries behind 1000 to 2000 keys of 32 heads of 128 take 47 us instead of 53.
template <int KS>
__global__ void __launch_bounds__(128, 4) window_scores_mma_kernel(const WindowAttnArgs a, const MmaShape sh) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  const int ld = a.dpad + 8;   // row stride in elements: 16 bytes past a multiple of 32 bytes
  __nv_bfloat16* s_q = reinterpret_cast<__nv_bfloat16*>(s_raw);
  __nv_bfloat16* s_k = s_q + kQB * ld;             // two tiles
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h = (int)blockIdx.x, kv = h / (a.heads / a.kv_heads);
  const int b0 = (int)blockIdx.y * kQB;            // first row of the block within the pass
  const int nrows = min(kQB, sh.rows - b0);
  grid_dep_launch();
  grid_dep_wait();
  const int r0 = sh.row0 + b0;
  const int pos0 = a.r.pos[r0];
  const BlockKeys keys(pos0, pos0 + nrows - 1, a.window, a.keep_first);
  const __nv_bfloat16* kc = static_cast<const __nv_bfloat16*>(a.k_cache) + (size_t)a.r.slots[r0] * a.geom.rows * (size_t)(a.kv_heads * a.dpad) + (size_t)kv * a.dpad;
  const int pieces = a.dpad >> 3;
  int lsh = 1;                                     // 2^lsh threads per row
  while ((1 << lsh) < pieces) ++lsh;
  const int c0 = tid & ((1 << lsh) - 1), rr0 = tid >> lsh, rstep = 128 >> lsh;
  if (c0 < pieces)
    for (int r = rr0; r < kQB; r += rstep) {
      const bool live = r < nrows;
      cp16z(s_q + r * ld + c0 * 8, a.q16 + ((size_t)(r0 + (live ? r : 0)) * a.heads + h) * a.dpad + c0 * 8, live);
    }
  const int krow = a.kv_heads * a.dpad;
  auto fetch = [&](int t) {
    __nv_bfloat16* dst = s_k + (t & 1) * kKeys * ld;
    const RunRows rows(keys, a.geom, t * kKeys);
    if (c0 < pieces)
      for (int r = rr0; r < kKeys; r += rstep) {
        const int v = t * kKeys + r;
        const bool live = v < keys.count;
        // in shared memory at row 8 b + 2 q + i of its sixteen, for key 4 q + 2 b + i: a thread's sums are then four keys in a row
        cp16z(dst + ((r & ~15) + ((r & 2) << 2) + ((r >> 1) & 6) + (r & 1)) * ld + c0 * 8, kc + (size_t)(live ? rows.row(v) : 0) * krow + c0 * 8, live);
      }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int tiles = (keys.count + kKeys - 1) / kKeys;
  const int t0 = (int)((int64_t)tiles * blockIdx.z / sh.score_splits), t1 = (int)((int64_t)tiles * (blockIdx.z + 1) / sh.score_splits);
  if (t0 < t1) fetch(t0);
  // the warp's 16 queries: this thread holds rows lane / 4 and lane / 4 + 8, keys 4 (lane & 3) and the next three of every sixteen
  const int qr[2] = {warp * 16 + (lane >> 2), warp * 16 + (lane >> 2) + 8};
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
  uint32_t qf[KS ? KS : 1][4];
  for (int t = t0; t < t1; ++t) {
    if (t + 1 < t1) {
      fetch(t + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const __nv_bfloat16* k = s_k + (t & 1) * kKeys * ld;
    float acc[8][4];
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[j][i] = 0.f;
    if constexpr (KS > 0) {
      if (t == t0)
#pragma unroll
        for (int c = 0; c < KS; ++c) ldm4(qf[c], s_q + (warp * 16 + (lane & 15)) * ld + c * 16 + (lane >> 4) * 8);
      const uint32_t kat = smem_addr(k + ((lane & 7) + ((lane >> 4) << 3)) * ld + ((lane >> 3) & 1) * 8);
#pragma unroll
      for (int c = 0; c < KS; ++c)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint32_t kb[4];
          ldm4(kb, kat + (uint32_t)((j * 16 * (KS * 16 + 8) + c * 16) * 2));
          mma16816(acc[2 * j], qf[c], kb[0], kb[1]);
          mma16816(acc[2 * j + 1], qf[c], kb[2], kb[3]);
        }
    } else {
      for (int c = 0; c < a.dpad; c += 16) {
        uint32_t qa[4];
        ldm4(qa, s_q + (warp * 16 + (lane & 15)) * ld + c + (lane >> 4) * 8);
#pragma unroll
        for (int j = 0; j < 4; ++j) {   // 16 keys: matrices (keys 0-7, k 0-7) (keys 0-7, k 8-15) (keys 8-15, ...) ...
          uint32_t kb[4];
          ldm4(kb, k + (j * 16 + (lane & 7) + ((lane >> 4) << 3)) * ld + c + ((lane >> 3) & 1) * 8);
          mma16816(acc[2 * j], qa, kb[0], kb[1]);
          mma16816(acc[2 * j + 1], qa, kb[2], kb[3]);
        }
      }
    }
    // every key of the tile seen by every query of the block?
    const int vf = t * kKeys;
    const bool all_seen = nrows == kQB && vf >= keys.nk && vf + kKeys <= keys.count && keys.position(vf + kKeys - 1) <= pos0 &&
                          pos0 + kQB - 1 - keys.position(vf) < a.window;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int pos = pos0 + qr[e];
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i) acc[j][2 * e + i] *= a.scale;
      if (!all_seen) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int v = t * kKeys + (j >> 1) * 16 + (lane & 3) * 4 + (j & 1) * 2 + i;
            const int p = keys.position(v);
            if (!(v < keys.count && qr[e] < nrows && p <= pos && (pos - p < a.window || p < a.keep_first))) acc[j][2 * e + i] = -INFINITY;
          }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) mx = fmaxf(mx, fmaxf(acc[j][2 * e], acc[j][2 * e + 1]));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      const float m1 = fmaxf(m[e], mx);
      const float ref = m1 == -INFINITY ? 0.f : m1;   // nothing seen yet: exp(-inf) = 0
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        acc[j][2 * e] = expf(acc[j][2 * e] - ref);
        acc[j][2 * e + 1] = expf(acc[j][2 * e + 1] - ref);
        sum += acc[j][2 * e] + acc[j][2 * e + 1];
      }
      if (m1 != -INFINITY) {
        l[e] = l[e] * expf(m[e] - m1) + sum;
        m[e] = m1;
      }
      if (qr[e] < nrows) {   // all of the tile: zeros past the last key
        float* row = a.scores + ((size_t)(b0 + qr[e]) * a.heads + h) * sh.stride;
        float* dst = row + t * kKeys + (lane & 3) * 4;
#pragma unroll
        for (int j = 0; j < 8; j += 2) *reinterpret_cast<float4*>(dst + j * 8) = make_float4(acc[j][2 * e], acc[j][2 * e + 1], acc[j + 1][2 * e], acc[j + 1][2 * e + 1]);
        if ((lane & 3) == 0) row[sh.refs + t] = m1;   // nothing seen: -inf, a factor of 0
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    l[e] += __shfl_xor_sync(0xffffffffu, l[e], 1);
    l[e] += __shfl_xor_sync(0xffffffffu, l[e], 2);
    if ((lane & 3) == 0 && qr[e] < nrows) {
      float* p = a.part + (((size_t)(b0 + qr[e]) * a.heads + h) * sh.score_splits + blockIdx.z) * 2;
      p[0] = m[e];
      p[1] = l[e];
    }
  }
}

// grid (head groups, blocks of 16 queries, key splits)
template <bool STAGED>
__global__ void __launch_bounds__(kMixThreads, 1) window_mix_mma_kernel(const WindowAttnArgs a, const MmaShape sh) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  __shared__ int2 s_unit[kUnits * kMixWarps];   // per 16-column output unit: where its head's weights and its values begin (bytes)
  const int gq = a.heads / a.kv_heads, hp = (a.heads + 15) & ~15;
  const int h0 = (int)blockIdx.x * sh.hg, nh = min(sh.hg, a.heads - h0);
  const int kv0 = h0 / gq, nkv = (h0 + nh - 1) / gq - kv0 + 1;
  const int vld = sh.kvs * a.vpad + 8, tld = hp + 8;
  float2* s_ml = reinterpret_cast<float2*>(s_raw);                                // [hp][kQM] (max, 1 / sum)
  float* s_f = reinterpret_cast<float*>(s_ml + hp * kQM);                         // [2][hp][kQM] a tile's references, then factors
  __nv_bfloat16* s_t = reinterpret_cast<__nv_bfloat16*>(s_f + 2 * hp * kQM);      // [16][tld] rows of T
  __nv_bfloat16* s_w = s_t + 16 * tld;                                            // [hg][kWHead]
  __nv_bfloat16* s_v = s_w + sh.hg * kWHead;                                      // [2][kKT][vld]
  float* s_s = reinterpret_cast<float*>(s_v + 2 * kKT * vld);                     // [kQM][heads][kSStride] when STAGED
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int q0 = (int)blockIdx.y * kQM;              // first row within the pass
  const int nrows = min(kQM, sh.rows - q0);
  const int b0 = q0 / kQB * kQB;
  grid_dep_launch();
  for (int i = tid; i < 16 * hp; i += kMixThreads) {
    const int h = i / hp, g = i - h * hp;
    s_t[h * tld + g] = __float2bfloat16_rn(h < nh && g < a.heads ? a.talk[(size_t)(h0 + h) * a.heads + g] : 0.f);
  }
  grid_dep_wait();
  const int pos_b = a.r.pos[sh.row0 + b0];
  const BlockKeys keys(pos_b, pos_b + min(kQB, sh.rows - b0) - 1, a.window, a.keep_first);
  const int pos0 = pos_b + q0 - b0, pos1 = pos0 + nrows - 1;
  const int vrow = a.kv_heads * a.vpad;
  const __nv_bfloat16* vc = static_cast<const __nv_bfloat16*>(a.v_cache) + (size_t)a.r.slots[sh.row0] * a.geom.rows * (size_t)vrow + (size_t)kv0 * a.vpad;
  for (int i = tid; i < hp * kQM; i += kMixThreads) {
    const int g = i / kQM, q = i - g * kQM;
    float2 v = make_float2(INFINITY, 0.f);           // a dead row's factors are exp(-inf) = 0
    if (q < nrows && g < a.heads) {
      const float* p = a.part + ((size_t)(q0 + q) * a.heads + g) * sh.score_splits * 2;
      float m = p[0], l = p[1];
      for (int z = 1; z < sh.score_splits; ++z) {      // in order
        const float m2 = p[2 * z], l2 = p[2 * z + 1], m1 = fmaxf(m, m2);
        l = (m == -INFINITY ? 0.f : l * expf(m - m1)) + (m2 == -INFINITY ? 0.f : l2 * expf(m2 - m1));
        m = m1;
      }
      v = make_float2(m, 1.0f / l);
    }
    s_ml[i] = v;
    s_f[i] = s_f[hp * kQM + i] = 0.f;
  }
  // tiles that hold a key one of these queries sees: the kept positions (their numbers are the positions), the run
  const VisibleRange first(pos0, a.window, a.keep_first);
  const int win1 = (keys.nk + pos1 - keys.lo) / kKT;
  const int kept = min((min(a.keep_first, keys.count) + kKT - 1) / kKT, win1 + 1);
  const int win0 = max(kept, (keys.nk + first.lo - keys.lo) / kKT);
  const int total = kept + win1 + 1 - win0;
  const int n0 = (int)((int64_t)total * blockIdx.z / sh.key_splits), n1 = (int)((int64_t)total * (blockIdx.z + 1) / sh.key_splits);
  const int pieces = nkv * a.vpad >> 3;
  auto fetch = [&](int n) {
    const int t = n < kept ? n : win0 + n - kept;
    __nv_bfloat16* dst = s_v + (n & 1) * kKT * vld;
    const RunRows rows(keys, a.geom, t * kKT);
    for (int r = warp; r < kKT; r += kMixWarps) {
      const int v = t * kKT + r;
      const bool live = v < keys.count;
      const __nv_bfloat16* src = vc + (size_t)(live ? rows.row(v) : 0) * vrow;
      for (int c = lane; c < pieces; c += 32) cp16z(dst + r * vld + c * 8, src + c * 8, live);
    }
    for (int i = tid; i < hp * kQM; i += kMixThreads) {
      const int g = i / kQM, q = i - g * kQM;
      if (q < nrows && g < a.heads)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(s_f + (n & 1) * hp * kQM + i)),
                     "l"(a.scores + ((size_t)(q0 + q) * a.heads + g) * sh.stride + sh.refs + t * kKT / kKeys)
                     : "memory");
    }
    if (STAGED) {
      // warp = query, 4 heads x 8 pieces of 4 keys at a time
      const int q = warp < nrows ? warp : 0;
      const float* src = a.scores + (size_t)(q0 + q) * a.heads * sh.stride + t * kKT + (lane & 7) * 4;
      float* d = s_s + (size_t)warp * a.heads * kSStride + (lane & 7) * 4;
      for (int g = lane >> 3; g < a.heads; g += 4) cp16z(d + g * kSStride, src + (size_t)g * sh.stride, true);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int upv = a.vpad >> 4, units = nh * upv;     // 16-column output units
  const int per = (units + kMixWarps - 1) / kMixWarps, unit0 = warp * per, mine = min(per, units - unit0);   // this warp's
  if (tid < units) {   // (the divisions of every unit and tile were a quarter of the instructions)
    const int h = tid / upv, c = (tid - h * upv) * 16;
    s_unit[tid] = make_int2(h * kWHead * 2, (((h0 + h) / gq - kv0) * a.vpad + c) * 2);
  }
  float acc[kUnits][2][4];
#pragma unroll
  for (int u = 0; u < kUnits; ++u)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[u][j][i] = 0.f;
  if (n0 < n1) fetch(n0);
  for (int n = n0; n < n1; ++n) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    float* fac = s_f + (n & 1) * hp * kQM;
    for (int i = tid; i < hp * kQM; i += kMixThreads) fac[i] = expf(fac[i] - s_ml[i].x) * s_ml[i].y;   // of what this thread has fetched
    __syncthreads();
    // ---- mixed weights of query `warp` at the tile's keys: lane / 4 = column n of the MMA = keys 4 n .. 4 n + 3 ----
    const int t = n < kept ? n : win0 + n - kept;
    const int kn = (lane >> 2) * 4;
    float d[4][4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int i = 0; i < 4; ++i) d[k][i] = 0.f;
    const float* sp = STAGED ? s_s + (size_t)warp * a.heads * kSStride + kn
                             : a.scores + (size_t)(q0 + (warp < nrows ? warp : 0)) * a.heads * sh.stride + t * kKT + kn;
    const int64_t gstride = STAGED ? kSStride : sh.stride;
    for (int kg = 0; kg < hp; kg += 16) {
      uint32_t ta[4];
      ldm4(ta, s_t + (lane & 15) * tld + kg + (lane >> 4) * 8);
      float p[4][4];                                   // [head of the fragment][key]
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int g = kg + (lane & 3) * 2 + (j & 1) + (j >> 1) * 8;
        float4 s4 = make_float4(0.f, 0.f, 0.f, 0.f);
        if (g < a.heads) s4 = *reinterpret_cast<const float4*>(sp + (size_t)g * gstride);
        const float f = fac[g * kQM + warp];
        p[j][0] = s4.x * f;
        p[j][1] = s4.y * f;
        p[j][2] = s4.z * f;
        p[j][3] = s4.w * f;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        uint32_t hi[2], lo[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const __nv_bfloat162 hv = __floats2bfloat162_rn(p[2 * j][k], p[2 * j + 1][k]);
          const float2 hf = __bfloat1622float2(hv);
          const __nv_bfloat162 lv = __floats2bfloat162_rn(p[2 * j][k] - hf.x, p[2 * j + 1][k] - hf.y);
          hi[j] = *reinterpret_cast<const uint32_t*>(&hv);
          lo[j] = *reinterpret_cast<const uint32_t*>(&lv);
        }
        mma16816(d[k], ta, hi[0], hi[1]);
        mma16816(d[k], ta, lo[0], lo[1]);
      }
    }
    // d[k][2 a + b]: head lane / 4 + 8 a, column 2 (lane & 3) + b, key k of the column
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int h = (lane >> 2) + (i >> 1) * 8, key = ((lane & 3) * 2 + (i & 1)) * 4;
      if (h < nh) {
        const __nv_bfloat162 h01 = __floats2bfloat162_rn(d[0][i], d[1][i]), h23 = __floats2bfloat162_rn(d[2][i], d[3][i]);
        const float2 f01 = __bfloat1622float2(h01), f23 = __bfloat1622float2(h23);
        const __nv_bfloat162 l01 = __floats2bfloat162_rn(d[0][i] - f01.x, d[1][i] - f01.y), l23 = __floats2bfloat162_rn(d[2][i] - f23.x, d[3][i] - f23.y);
        __nv_bfloat16* wp = s_w + (size_t)h * kWHead + warp * kWStride + key;
        *reinterpret_cast<uint2*>(wp) = make_uint2(*reinterpret_cast<const uint32_t*>(&h01), *reinterpret_cast<const uint32_t*>(&h23));
        *reinterpret_cast<uint2*>(wp + kQM * kWStride) = make_uint2(*reinterpret_cast<const uint32_t*>(&l01), *reinterpret_cast<const uint32_t*>(&l23));
      }
    }
    __syncthreads();
    if (n + 1 < n1) fetch(n + 1);
    const uint32_t w_at = smem_addr(s_w + (lane & 15) * kWStride + (lane >> 4) * 8);
    const uint32_t v_at = smem_addr(s_v + (n & 1) * kKT * vld + (lane & 15) * vld + (lane >> 4) * 8);
#pragma unroll
    for (int kk = 0; kk < kKT; kk += 16) {
      uint32_t hi[4], lo[4], vb[4];
      int of = -1;   // whose weights the fragments are: a warp's units follow one another, most of them of one head
#pragma unroll
      for (int u = 0; u < kUnits; ++u) {
        if (u >= mine) break;
        const int2 at = s_unit[unit0 + u];
        if (at.x != of) {
          of = at.x;
          ldm4(hi, w_at + (uint32_t)(at.x + kk * 2));
          ldm4(lo, w_at + (uint32_t)(at.x + (kQM * kWStride + kk) * 2));
        }
        // V is [key][column]: transposed loads give (keys 0-7, cols 0-7) (keys 8-15, cols 0-7) (keys 0-7, cols 8-15) ...
        ldm4t(vb, v_at + (uint32_t)(at.y + kk * vld * 2));
        mma16816(acc[u][0], hi, vb[0], vb[1]);
        mma16816(acc[u][1], hi, vb[2], vb[3]);
        mma16816(acc[u][0], lo, vb[0], vb[1]);
        mma16816(acc[u][1], lo, vb[2], vb[3]);
      }
    }
  }
  const int cols = a.heads * a.vdim;
#pragma unroll
  for (int u = 0; u < kUnits; ++u) {
    const int unit = unit0 + u;
    if (u >= mine) break;
    const int h = unit / upv, c = (unit - h * upv) * 16;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int q = (lane >> 2) + (i >> 1) * 8, col = c + j * 8 + (lane & 3) * 2 + (i & 1);
        if (q >= nrows || col >= a.vdim) continue;
        const int k = (h0 + h) * a.vdim + col;
        if (sh.key_splits > 1) a.parts[((size_t)blockIdx.z * sh.rows + q0 + q) * cols + k] = acc[u][j][i];
        else act_store1<true>(a.out, sh.row0 + q0 + q, k, acc[u][j][i]);
      }
  }
  if (sh.key_splits == 1 && h0 + nh == a.heads)
    for (int q = 0; q < nrows; ++q)
      for (int k = cols + tid; k < a.out.kp; k += kMixThreads) act_store1<true>(a.out, sh.row0 + q0 + q, k, 0.f);
}

// 17 to 32 heads, an even number per key head: a CTA takes 8 queries and ALL heads, so that the weights of a (query, key)
// are split into pieces and contracted once and not once per group of 16 output heads, which was half of the kernel's
// instructions.  The MMA's 16 rows are two heads of one key head times 8 queries.  Traffic is the same (half the queries, so half the
// scores, against the values of all heads).  Values are fetched a phase before scores: their place is free earlier.  A prompt of
// 2501 tokens, eight layers of 32 heads of 128: 19.86 ms in groups of 16, 18.2 so.  Bound by shared memory and the latency of
// its phases: issue slots 36% busy, a third of the stalls on shared memory, 96 KB through L2 per tile of 32 keys.
// grid (1, blocks of 8 queries, key splits)
constexpr int kQA = 8;
__global__ void __launch_bounds__(kMixThreads, 1) window_mix_all_kernel(const WindowAttnArgs a, const MmaShape sh) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  __shared__ int2 s_unit[kUnits * kMixWarps];   // per 16-column output unit: where its pair's weights and its values begin (bytes)
  constexpr int kHP = 32, tld = kHP + 8;
  const int gq = a.heads / a.kv_heads, vld = a.kv_heads * a.vpad + 8, qh = kQA * a.heads;
  float2* s_ml = reinterpret_cast<float2*>(s_raw);                                // [query][head] (max, 1 / sum)
  float* s_f = reinterpret_cast<float*>(s_ml + kQA * kHP);                        // [2][query][head] a tile's references, then factors
  __nv_bfloat16* s_t = reinterpret_cast<__nv_bfloat16*>(s_f + 2 * kQA * kHP);     // [32][tld] rows of T
  __nv_bfloat16* s_w = s_t + kHP * tld;                                           // [pair][kWHead]
  __nv_bfloat16* s_v = s_w + kHP / 2 * kWHead;                                    // [2][kKT][vld]
  float* s_s = reinterpret_cast<float*>(s_v + 2 * kKT * vld);                     // [query][head][kSStride]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int q0 = (int)blockIdx.y * kQA;              // first row within the pass
  const int nrows = min(kQA, sh.rows - q0), live_qh = nrows * a.heads;
  const int b0 = q0 / kQB * kQB;
  grid_dep_launch();
  for (int i = tid; i < kHP * kHP; i += kMixThreads) {
    const int h = i / kHP, g = i % kHP;
    s_t[h * tld + g] = __float2bfloat16_rn(h < a.heads && g < a.heads ? a.talk[(size_t)h * a.heads + g] : 0.f);
  }
  const int upv = a.vpad >> 4, units = a.heads / 2 * upv;
  const int per = (units + kMixWarps - 1) / kMixWarps, unit0 = warp * per, mine = min(per, units - unit0);   // this warp's
  if (tid < units) {
    const int pair = tid / upv, c = (tid - pair * upv) * 16;
    s_unit[tid] = make_int2(pair * kWHead * 2, (pair * 2 / gq * a.vpad + c) * 2);
  }
  grid_dep_wait();
  const int pos_b = a.r.pos[sh.row0 + b0];
  const BlockKeys keys(pos_b, pos_b + min(kQB, sh.rows - b0) - 1, a.window, a.keep_first);
  const int pos0 = pos_b + q0 - b0, pos1 = pos0 + nrows - 1;
  const int vrow = a.kv_heads * a.vpad;
  const __nv_bfloat16* vc = static_cast<const __nv_bfloat16*>(a.v_cache) + (size_t)a.r.slots[sh.row0] * a.geom.rows * (size_t)vrow;
  const float* scores = a.scores + (size_t)q0 * a.heads * sh.stride;   // this CTA's rows of scratch follow one another
  if (tid < qh) {
    float2 v = make_float2(INFINITY, 0.f);           // a dead row's factors are exp(-inf) = 0
    if (tid < live_qh) {
      const float* p = a.part + ((size_t)q0 * a.heads + tid) * sh.score_splits * 2;
      float m = p[0], l = p[1];
      for (int z = 1; z < sh.score_splits; ++z) {      // in order
        const float m2 = p[2 * z], l2 = p[2 * z + 1], m1 = fmaxf(m, m2);
        l = (m == -INFINITY ? 0.f : l * expf(m - m1)) + (m2 == -INFINITY ? 0.f : l2 * expf(m2 - m1));
        m = m1;
      }
      v = make_float2(m, 1.0f / l);
    }
    s_ml[tid] = v;
    s_f[tid] = s_f[kQA * kHP + tid] = 0.f;
  }
  // tiles that hold a key one of these queries sees: the kept positions (their numbers are the positions), the run
  const VisibleRange first(pos0, a.window, a.keep_first);
  const int win1 = (keys.nk + pos1 - keys.lo) / kKT;
  const int kept = min((min(a.keep_first, keys.count) + kKT - 1) / kKT, win1 + 1);
  const int win0 = max(kept, (keys.nk + first.lo - keys.lo) / kKT);
  const int total = kept + win1 + 1 - win0;
  const int n0 = (int)((int64_t)total * blockIdx.z / sh.key_splits), n1 = (int)((int64_t)total * (blockIdx.z + 1) / sh.key_splits);
  const int pieces = vrow >> 3;
  auto fetch_values = [&](int n) {
    const int t = n < kept ? n : win0 + n - kept;
    const RunRows rows(keys, a.geom, t * kKT);
#pragma unroll
    for (int r = warp; r < kKT; r += kMixWarps) {
      const int v = t * kKT + r;
      const bool live = v < keys.count;
      const __nv_bfloat16* src = vc + (size_t)(live ? rows.row(v) : 0) * vrow + lane * 8;
      __nv_bfloat16* dst = s_v + ((n & 1) * kKT + r) * vld + lane * 8;
      for (int c = lane; c < pieces; c += 32, src += 256, dst += 256) cp16z(dst, src, live);
    }
  };
  auto fetch_scores = [&](int n) {
    const int t = n < kept ? n : win0 + n - kept;
    if (tid < live_qh)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(s_f + (n & 1) * kQA * kHP + tid)), "l"(scores + (size_t)tid * sh.stride + sh.refs + t * kKT / kKeys)
                   : "memory");
    for (int i = tid; i < qh * (kKT / 4); i += kMixThreads) {   // (a dead row's scores: those of the first one, with factors of 0)
      const int row = i >> 3, c = (i & 7) * 4;
      cp16z(s_s + row * kSStride + c, scores + (size_t)(row < live_qh ? row : 0) * sh.stride + t * kKT + c, true);
    }
  };
  float acc[kUnits][2][4];
#pragma unroll
  for (int u = 0; u < kUnits; ++u)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[u][j][i] = 0.f;
  const int q = warp >> 1, kh = (warp & 1) * 16;     // mixing: this warp's query and half of the tile's keys
  if (n0 < n1) {
    fetch_values(n0);
    fetch_scores(n0);
  }
  for (int n = n0; n < n1; ++n) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    float* fac = s_f + (n & 1) * kQA * kHP;
    if (tid < qh) fac[tid] = expf(fac[tid] - s_ml[tid].x) * s_ml[tid].y;   // of what this thread has fetched
    __syncthreads();
    if (n + 1 < n1) fetch_values(n + 1);   // in the place of the ones that were used before the barrier
    // ---- mixed weights: lane / 4 = column of the MMA = two keys ----
    float d[2][2][4];
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int i = 0; i < 4; ++i) d[mt][k][i] = 0.f;
    const float* sp = s_s + q * a.heads * kSStride + kh + (lane >> 2) * 2;
    const float* fp = fac + q * a.heads;
#pragma unroll
    for (int kg = 0; kg < kHP; kg += 16) {
      uint32_t ta[2][4];
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) ldm4(ta[mt], s_t + (mt * 16 + (lane & 15)) * tld + kg + (lane >> 4) * 8);
      float p[4][2];                                   // [head of the fragment][key]
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int g = kg + (lane & 3) * 2 + (j & 1) + (j >> 1) * 8;
        float2 s2 = make_float2(0.f, 0.f);
        float f = 0.f;
        if (g < a.heads) {
          s2 = *reinterpret_cast<const float2*>(sp + g * kSStride);
          f = fp[g];
        }
        p[j][0] = s2.x * f;
        p[j][1] = s2.y * f;
      }
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        uint32_t hi[2], lo[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const __nv_bfloat162 hv = __floats2bfloat162_rn(p[2 * j][k], p[2 * j + 1][k]);
          hi[j] = *reinterpret_cast<const uint32_t*>(&hv);
          const __nv_bfloat162 lv = __floats2bfloat162_rn(p[2 * j][k] - __uint_as_float(hi[j] << 16), p[2 * j + 1][k] - __uint_as_float(hi[j] & 0xFFFF0000u));
          lo[j] = *reinterpret_cast<const uint32_t*>(&lv);
        }
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
          mma16816(d[mt][k], ta[mt], hi[0], hi[1]);
          mma16816(d[mt][k], ta[mt], lo[0], lo[1]);
        }
      }
    }
    // d[mt][k][2 x + y]: head 16 mt + lane / 4 + 8 x, column 2 (lane & 3) + y, key k of the column: four keys in a row
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const int h = mt * 16 + (lane >> 2) + 8 * x;
        const __nv_bfloat162 h01 = __floats2bfloat162_rn(d[mt][0][2 * x], d[mt][1][2 * x]), h23 = __floats2bfloat162_rn(d[mt][0][2 * x + 1], d[mt][1][2 * x + 1]);
        const uint32_t u01 = *reinterpret_cast<const uint32_t*>(&h01), u23 = *reinterpret_cast<const uint32_t*>(&h23);
        const __nv_bfloat162 l01 = __floats2bfloat162_rn(d[mt][0][2 * x] - __uint_as_float(u01 << 16), d[mt][1][2 * x] - __uint_as_float(u01 & 0xFFFF0000u));
        const __nv_bfloat162 l23 = __floats2bfloat162_rn(d[mt][0][2 * x + 1] - __uint_as_float(u23 << 16), d[mt][1][2 * x + 1] - __uint_as_float(u23 & 0xFFFF0000u));
        __nv_bfloat16* wp = s_w + (h >> 1) * kWHead + ((h & 1) * kQA + q) * kWStride + kh + (lane & 3) * 4;
        *reinterpret_cast<uint2*>(wp) = make_uint2(u01, u23);
        *reinterpret_cast<uint2*>(wp + kQM * kWStride) = make_uint2(*reinterpret_cast<const uint32_t*>(&l01), *reinterpret_cast<const uint32_t*>(&l23));
      }
    __syncthreads();
    if (n + 1 < n1) fetch_scores(n + 1);
    const uint32_t w_at = smem_addr(s_w + (lane & 15) * kWStride + (lane >> 4) * 8);
    const uint32_t v_at = smem_addr(s_v + ((n & 1) * kKT + (lane & 15)) * vld + (lane >> 4) * 8);
#pragma unroll
    for (int kk = 0; kk < kKT; kk += 16) {
      uint32_t hi[4], lo[4], vb[4];
      int of = -1;   // whose weights the fragments are: a warp's units follow one another, most of them of one head
#pragma unroll
      for (int u = 0; u < kUnits; ++u) {
        if (u >= mine) break;
        const int2 at = s_unit[unit0 + u];
        if (at.x != of) {
          of = at.x;
          ldm4(hi, w_at + (uint32_t)(at.x + kk * 2));
          ldm4(lo, w_at + (uint32_t)(at.x + (kQM * kWStride + kk) * 2));
        }
        // V is [key][column]: transposed loads give (keys 0-7, cols 0-7) (keys 8-15, cols 0-7) (keys 0-7, cols 8-15) ...
        ldm4t(vb, v_at + (uint32_t)(at.y + kk * vld * 2));
        mma16816(acc[u][0], hi, vb[0], vb[1]);
        mma16816(acc[u][1], hi, vb[2], vb[3]);
        mma16816(acc[u][0], lo, vb[0], vb[1]);
        mma16816(acc[u][1], lo, vb[2], vb[3]);
      }
    }
  }
  const int cols = a.heads * a.vdim, row = lane >> 2;
#pragma unroll
  for (int u = 0; u < kUnits; ++u) {
    const int unit = unit0 + u;
    if (u >= mine || row >= nrows) break;
    const int pair = unit / upv, c = (unit - pair * upv) * 16;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int col = c + j * 8 + (lane & 3) * 2 + (i & 1);
        if (col >= a.vdim) continue;
        const int k = (pair * 2 + (i >> 1)) * a.vdim + col;
        if (sh.key_splits > 1) a.parts[((size_t)blockIdx.z * sh.rows + q0 + row) * cols + k] = acc[u][j][i];
        else act_store1<true>(a.out, sh.row0 + q0 + row, k, acc[u][j][i]);
      }
  }
  if (sh.key_splits == 1)
    for (int r = 0; r < nrows; ++r)
      for (int k = cols + tid; k < a.out.kp; k += kMixThreads) act_store1<true>(a.out, sh.row0 + q0 + r, k, 0.f);
}
size_t mix_all_bytes(const WindowAttnArgs& a) {
  return (size_t)kQA * 32 * 16 + (size_t)32 * 40 * 2 + (size_t)16 * kWHead * 2 + (size_t)2 * kKT * (a.kv_heads * a.vpad + 8) * 2 + (size_t)kQA * a.heads * kSStride * 4;
}

size_t mix_bytes(const WindowAttnArgs& a, int hg, int kvs, bool staged) {
  const int hp = (a.heads + 15) & ~15;
  return (size_t)hp * kQM * 16 + (size_t)16 * (hp + 8) * 2 + (size_t)hg * kWHead * 2 + (size_t)2 * kKT * (kvs * a.vpad + 8) * 2 +
         (staged ? (size_t)kQM * a.heads * kSStride * 4 : 0);
}
int group_kv_heads(const WindowAttnArgs& a, int hg) {   // most kv heads a group of hg query heads touches
  const int gq = a.heads / a.kv_heads;
  const int n = hg % gq == 0 ? hg / gq : (gq % hg == 0 ? 1 : (hg + gq - 2) / gq + 1);
  return n < a.kv_heads ? n : a.kv_heads;
}
constexpr size_t kSmemMax = 226 * 1024;   // (1 KB of static shared memory beside it)
bool mix_all_fits(const WindowAttnArgs& a) {
  return a.heads > 16 && a.heads <= 32 && a.heads / a.kv_heads % 2 == 0 && a.heads / 2 * (a.vpad / 16) <= kUnits * kMixWarps && mix_all_bytes(a) <= kSmemMax;
}

}  // namespace

bool window_mma_supported(const WindowAttnArgs& a) {
  return a.one_sequence && a.q16 != nullptr && a.r.rows >= kQM && a.dpad <= 256 && a.vpad <= 256 && a.heads <= 256 && (a.scratch_rows >= kQB || a.scratch_rows >= a.r.rows) &&
         mix_bytes(a, 1, 1, false) <= kSmemMax;
}

tb_status launch_window_attention_mma(const WindowAttnArgs& a, cudaStream_t st, int* launches) {
  // heads per group: as many as one MMA holds and accumulators and shared memory allow
  int hg = 16;
  while (hg > 1 && (hg / 2 >= a.heads || hg * a.vpad > kUnits * kMixWarps * 16 || mix_bytes(a, hg, group_kv_heads(a, hg), false) > kSmemMax)) hg /= 2;
  MmaShape sh;
  sh.hg = hg;
  sh.kvs = group_kv_heads(a, hg);
  sh.stride = (int64_t)window_attn_score_stride(a.max_visible);
  sh.refs = (int)pad_to(a.max_visible + kQB, kKeys);
  const bool staged = mix_bytes(a, hg, sh.kvs, true) <= kSmemMax;
  // passes of equal size, in whole query blocks, as many rows as the score scratch holds
  const int64_t blocks = (a.r.rows + kQB - 1) / kQB, fit = a.scratch_rows / kQB;
  const int64_t passes = a.scratch_rows >= a.r.rows ? 1 : (blocks + fit - 1) / fit;
  const int64_t pass = (blocks + passes - 1) / passes * kQB;
  const bool all = mix_all_fits(a);
  const int groups = all ? 1 : (a.heads + hg - 1) / hg, block = all ? kQA : kQM;
  const size_t ssm = (size_t)(kQB + 2 * kKeys) * (a.dpad + 8) * 2, msm = all ? mix_all_bytes(a) : mix_bytes(a, hg, sh.kvs, staged);
  for (int64_t r0 = 0; r0 < a.r.rows; r0 += pass) {
    sh.row0 = (int)r0;
    sh.rows = (int)(a.r.rows - r0 < pass ? a.r.rows - r0 : pass);
    const int64_t qb = (sh.rows + kQB - 1) / kQB;
    sh.score_splits = 1;
    while (sh.score_splits < 8 && a.heads * qb * sh.score_splits < 4 * sm_count() && a.max_visible >= (int64_t)kKeys * 4 * sh.score_splits) sh.score_splits *= 2;
    const auto scores = a.dpad == 128 ? window_scores_mma_kernel<8> : (a.dpad == 64 ? window_scores_mma_kernel<4> : window_scores_mma_kernel<0>);
    TB_TRY(launch_kernel(scores, dim3((unsigned)a.heads, (unsigned)qb, (unsigned)sh.score_splits), dim3(128), ssm, st, a.pdl, 1, a, sh));
    const int qblocks = (sh.rows + block - 1) / block;
    sh.key_splits = 1;
    while (sh.key_splits < kMaxKeySplits && a.parts_rows >= 2 * (int64_t)sh.rows * sh.key_splits && groups * qblocks * sh.key_splits * 3 / 2 < sm_count() &&
           a.max_visible >= (int64_t)kKT * 8 * sh.key_splits)
      sh.key_splits *= 2;
    auto* kern = all ? window_mix_all_kernel : staged ? window_mix_mma_kernel<true> : window_mix_mma_kernel<false>;
    TB_TRY(launch_kernel(kern, dim3((unsigned)groups, (unsigned)qblocks, (unsigned)sh.key_splits), dim3(kMixThreads), msm, st, a.pdl, 1, a, sh));
    *launches += 2;
    if (sh.key_splits > 1) {
      TB_TRY(launch_window_parts(Precision::kBf16, a, sh.key_splits, sh.row0, sh.rows, st));
      ++*launches;
    }
  }
  return TB_OK;
}

}  // namespace tb
