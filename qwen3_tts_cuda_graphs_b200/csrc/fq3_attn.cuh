// fq3_attn.cuh — softmax attention of many queries on tcgen05: heads of 128, keys and values bf16.
//
// Included by fq3_codec.cu behind fq3_gemm.cuh.  Serves the talker's prompt (FQ3C_ATTN with flags bit 0: queries, keys and values in the projected
// rows) and prompt portions of the sequence models (FQ3C_CACHE_ATTN over a bf16 cache).
#pragma once

struct AttnArgs {
  const void* q;            // PROMPT: bf16 rows, else f32 rows; head h at column h * 128
  const bf16 *k, *v;        // row j of key / value head g at j * ld + g * 128
  long ldq, ldk, ldv;
  int H, G, M;
  int groups;               // row groups per CTA: 1 or 2
  int ends;                 // 1: a CTA's two groups are one from the end of the rows and one from their beginning (the ENDS variant), else they are neighbours
  int two_from;             // > 0: launched with one, but behind more positions than these a CTA takes two and every other one leaves
  const int* p0;            // position of query 0 (device), or null: 0
  float scale, cap, mult;   // mult != 0 multiplies the output
  int window, keep, chunk;  // 0: none
  const float *r12, *sink, *gate;
  int gate_ld, entry, out_f32;
  void* out;
  long ldo;
  int tries;                // of a wait before it gives up
  int lost;                 // 1: the first key tile is never asked for (tests of the error path)
};
enum { AT_PROMPT, AT_PLAIN, AT_CAP, AT_DIST };   // AT_PROMPT: scores rounded to bf16 before and behind the scale; AT_DIST: cap and distance penalty, both optional
constexpr int AT_KEYS = 128, AT_THREADS = 640, AT_LOADERS = 96;
constexpr int AT_TILE = 128 * 128 * 2;           // a query, key or value tile: two halves of 64 columns, 128-byte lines, 128-byte swizzle
constexpr int AT_SMEM = 6 * AT_TILE + 1024 + 256 + 2 * 2 * 256 * 4;   // tiles, alignment, barriers, the half rows' maxima (two tiles in turn)
constexpr float AT_L2E = 1.4426950408889634f;
constexpr float AT_SLACK = 11.f;                 // a row's reference moves when its maximum is further above it than this (in powers of two)

__device__ __forceinline__ void tmem_ld32(const uint32_t a, float* f) {
  uint32_t v[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, "
      "%20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
        "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]),
        "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]),
        "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(a)
      : "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) f[i] = __uint_as_float(v[i]);
}
// the lowest n bits (none below 0, all from 32 on)
__device__ __forceinline__ uint32_t first_bits(const int n) { return n >= 32 ? 0xffffffffu : (1u << max(n, 0)) - 1u; }
// 2^n for a whole number n <= 0, exactly (0 below the normal range)
__device__ __forceinline__ float pow2_down(const float n) { return n < -126.f ? 0.f : __int_as_float(((int)n + 127) << 23); }
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st16(const uint32_t a, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(a), "r"(v[0]), "r"(v[1]), "r"(v[2]),
      "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// D[128 x 128] (+)= A (tensor memory, bf16 pairs) . B (shared memory)
__device__ __forceinline__ void umma_bf16_ta(const uint32_t d, const uint32_t a, const uint64_t db, const uint32_t idesc, const uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d), "r"(a), "l"(db), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ float ex2f(const float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// cap * tanh(x), cap * tanh(y) for |x|, |y| up to AT_NEAR: x (1 - t/3 + 2 t^2/15 - 17 t^3/315 + 62 t^4/2835), t = x^2, the first terms of the series, which leave 2.4e-7 of the result.  Seven
// packed multiply-adds for two scores, where the exponential and the reciprocal of fast_tanh (1e-6) are two more turns each on the special-function unit beside the weight's own.
constexpr float AT_NEAR = 0.35f;
__device__ __forceinline__ float max_nan(const float x, const float y) {      // a NaN stays one
  float m;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(m) : "f"(x), "f"(y));
  return m;
}
__device__ __forceinline__ void cap_near(float& x, float& y, const float cap) {
  const f32x2 v = pack2(x, y), t = mul2<true>(v, v);
  f32x2 p = fma2<true>(t, pack2(62.f / 2835.f, 62.f / 2835.f), pack2(-17.f / 315.f, -17.f / 315.f));
  p = fma2<true>(t, p, pack2(2.f / 15.f, 2.f / 15.f));
  p = fma2<true>(t, p, pack2(-1.f / 3.f, -1.f / 3.f));
  const f32x2 c = mul2<true>(v, pack2(cap, cap));
  p = fma2<true>(mul2<true>(t, p), c, c);
  x = lo2(p); y = hi2(p);
}
// 16 finished entries of an output row, f32 or rounded
__device__ __forceinline__ void at_store(const AttnArgs& a, const size_t at, const float (&v)[16]) {
  if (a.out_f32) {
    float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(a.out) + at);
#pragma unroll
    for (int j = 0; j < 4; ++j) dst[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
  } else {
    uint32_t w[8];
    pack16(v, w);
    uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(a.out) + at);
    dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
    dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
  }
}
// Sixteen columns of an output row over the keys that the row sees, and no others, times sc and, where there is one, the sigmoid of the entry's gate.  The products above
// multiply the weight 0 of an unseen key with its value, which is no 0 where the value is infinite or NaN: a row that came out so is formed again here, one thread per
// row.  (It stores by itself: entries handed over by address would leave the registers in the other path too.)
template <int MODE>
__device__ __noinline__ void at_row_again(const AttnArgs& a, const int m, const int head, const int col, const int pos, const int lo, const int keep, const float ref, const float sc,
                                          const float* gate) {
  const int HG = a.H / a.G, kvh = head / HG;
  float out[16];
  for (int j = 0; j < 16; ++j) out[j] = 0.f;
  const size_t qat = (size_t)m * a.ldq + (size_t)head * 128;
  for (int key = 0; key <= pos; ++key) {
    if (key < lo && key >= keep) { key = lo - 1; continue; }
    const bf16* k = a.k + (size_t)key * a.ldk + kvh * 128;
    float s = 0.f;
    for (int c = 0; c < 128; ++c) {
      const float q = MODE == AT_PROMPT ? __bfloat162float(reinterpret_cast<const bf16*>(a.q)[qat + c]) : bf16r(reinterpret_cast<const float*>(a.q)[qat + c]);
      s = fmaf(q, __bfloat162float(k[c]), s);
    }
    if (MODE == AT_PROMPT) {
      s = bf16r(bf16r(s) * a.scale);
    } else {
      s *= a.scale;
      if (a.cap > 0.f) s = a.cap * fast_tanh(s / a.cap);
      if (MODE == AT_DIST && a.r12) s -= a.r12[head] * __logf(fmaf(a.r12[a.H + head], (float)(pos - key), 1.f));
    }
    const float w = exp2f(fmaf(s, AT_L2E, -ref));
    const bf16* v = a.v + (size_t)key * a.ldv + kvh * 128 + col;
    for (int j = 0; j < 16; ++j) out[j] = fmaf(w, __bfloat162float(v[j]), out[j]);
  }
  for (int j = 0; j < 16; ++j) {
    out[j] *= sc;
    if (gate) out[j] *= sigmoid_f(gate[j]);
  }
  at_store(a, (size_t)m * a.ldo + (size_t)head * 128 + col, out);
}

// A CTA takes two groups of 128 rows (or one: launch_attn_tc) of one key / value head; a row is a (query, head of the group) pair, so that all heads sharing the keys score the same
// staged tile.  Warps 0-7 and 8-15: two threads per row of group 0 and 1, 64 keys of a tile each; warps 16-18 stage key and value tiles of 128 positions (two
// stages); warp 19 issues the MMAs.  Per group and tile: S = Q K^T into tensor memory; the row's threads scale, cap and mask its 128 scores, agree on the
// maximum, take 2^(score log2 e - reference) and write every weight as a bf16 pair hi + mid (16 mantissa bits) over S; O += hi V + mid V with the weights read from
// tensor memory.  AT_PROMPT's weights keep their 24 bits: what the pair lacks goes over the hi parts as soon as the products with those have ended, while the ones
// with the mid parts run, and makes a third product.  While one group's threads work, the tensor pipe has the other group's products.  The reference is a whole
// number next to the first tile's maximum, so that neither it nor a rescaling rounds anything, and moves only when a later maximum is more than 2^11 above it: then
// the row's output is rescaled in tensor memory.  Tiles outside every row's window, chunk and kept positions are not fetched.
// Bound by the chain scores -> maximum -> weights -> output of a group (24 MMAs of 64 cycles a tile are about half of it; the other group fills part of the
// rest) and, with a cap, by the special-function unit (three a score).
// Without a wave's worth of row groups a CTA has one, so that no group waits for the other's issue slots; one group's next scores are issued in front of its values.
// A tile takes one group some 3.7 us with a cap, two 6.0.  Norm and attention of 85 prompt rows of 16 heads over 8 10.9 us, 144 13.3, 262 17.0.
// ENDS: two groups may be from either end of the rows (a variant of its own: a second group that is not behind the first costs the tiles' loop registers, 0.8 us of 12.6 for 200 prompt rows
// of 16 heads over 8).
template <int MODE, bool ENDS>
__global__ void __launch_bounds__(AT_THREADS, 1) fq3c_attn_tc_kernel(const __grid_constant__ AttnArgs a) {
  extern __shared__ unsigned char at_raw[];
  const uint32_t raw = smem_u32(at_raw), base = (raw + 1023u) & ~1023u;
  unsigned char* gbase = at_raw + (base - raw);
  const uint32_t q_s = base, k_s = base + 2 * AT_TILE, v_s = base + 4 * AT_TILE, bars = base + 6 * AT_TILE;
  const uint32_t q_full = bars, k_full = bars + 16, k_empty = bars + 32, v_full = bars + 48, v_empty = bars + 64, s_full = bars + 80, p_full = bars + 96, o_done = bars + 112, drain = bars + 144, h_done = bars + 152, l_full = bars + 168;      // (behind the words)
  uint32_t* words = reinterpret_cast<uint32_t*>(gbase + 6 * AT_TILE + 128);
  volatile int* dead = reinterpret_cast<volatile int*>(words + 1);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  int groups = a.groups, gx = gridDim.x;
  if (a.two_from > 0) {
    grid_dep_wait();
    if (*a.p0 > a.two_from) {
      groups = 2;
      gx = (gx + 1) / 2;
      if ((int)blockIdx.x >= gx) return;
    }
  }
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(q_full + 8u * i, 8);
      mbar_init(k_full + 8u * i, AT_LOADERS); mbar_init(k_empty + 8u * i, 1);
      mbar_init(v_full + 8u * i, AT_LOADERS); mbar_init(v_empty + 8u * i, 1);
      mbar_init(s_full + 8u * i, 1); mbar_init(p_full + 8u * i, 8); mbar_init(o_done + 8u * i, 1);
      mbar_init(h_done + 8u * i, 1); mbar_init(l_full + 8u * i, 8);
    }
    mbar_init(drain, 1);
    words[1] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 19) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(words)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const bool leader = elect_one();
  const uint32_t tmem = __shfl_sync(0xffffffffu, words[0], 0);   // S0 | S1 | O0 | O1, 128 columns each
  grid_dep_launch();
  grid_dep_wait();

  const int HG = a.H / a.G, QB = 128 / HG, kvh = blockIdx.y;
  const bool one = groups == 1;      // its tiles take the score columns of both groups in turn
  // the last queries (most keys) start first
  int m0 = (gx - 1 - (int)blockIdx.x) * groups * QB, m1 = m0 + QB;      // each group's first query
  if (ENDS && !one) {
    const int late = (a.M + QB - 1) / QB - 1 - (int)blockIdx.x;
    m0 = late * QB;
    m1 = (int)blockIdx.x < late ? (int)blockIdx.x * QB : a.M;
  }
  auto row0 = [&](const int g) { return ENDS ? (g ? m1 : m0) : m0 + g * QB; };
  const int P = a.p0 ? *a.p0 : 0;
  int nq[2], first[2], last[2], tiles[2], tlo[2];                 // per group: live queries, their positions, tiles up to the last, first tile of window or chunk
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    nq[g] = g < groups ? max(0, min(QB, a.M - row0(g))) : 0;
    first[g] = P + row0(g);
    last[g] = first[g] + nq[g] - 1;
    tiles[g] = nq[g] > 0 ? last[g] / AT_KEYS + 1 : 0;
    int lo = a.window > 0 ? max(0, first[g] - a.window + 1) : 0;
    if (a.chunk > 0) lo = max(lo, first[g] - first[g] % a.chunk);
    tlo[g] = lo / AT_KEYS;
  }
  const int tkeep = a.window > 0 && a.chunk <= 0 ? (a.keep + AT_KEYS - 1) / AT_KEYS : 0;
  const int ntiles = max(tiles[0], tiles[1]), jend = ENDS ? (nq[1] > 0 ? max(last[0], last[1]) : last[0]) : P + min(a.M, m0 + groups * QB) - 1;
  auto need = [&](const int g, const int t) { return t < tiles[g] && (t >= tlo[g] || t < tkeep); };

  if (warp == 19) {
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 4) << 24);   // F32 += BF16 x BF16, both K-major; columns: bits 17..
    const uint32_t idesc_o = idesc | ((128u >> 3) << 17) | (1u << 16);                                                        // B (values: rows = keys) MN-major
    bool pend[2] = {false, false}, begun[2] = {false, false};
    int prev = 0;
    bool gone = false;      // a wait gave up: nothing more is issued
    if (!gp_wait_warp(q_full, 0, dead, a.tries)) gone = true;
    if (nq[1] > 0 && !gp_wait_warp(q_full + 8, 0, dead, a.tries)) gone = true;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    int nl[2] = {0, 0};
    // steps of 16 keys of tile t up to the group's last position: what lies behind is neither scored nor multiplied
    auto steps = [&](const int g, const int t) { return min(8, (last[g] - t * AT_KEYS) / 16 + 1); };
    // O[g] += P[g] V of the tile in stage st
    auto values = [&](const int g, const int st, const int tile) {
      const uint32_t pa = tmem + (one ? st : g) * 128, d = tmem + 256 + g * 128;
      const int ks = steps(g, tile);
      // MN-major, 128-byte swizzle: 64 columns further is a half tile further, eight keys further 1024 bytes
      const uint64_t vd = (uint64_t)(((v_s + st * AT_TILE) & 0x3ffffu) >> 4) | ((uint64_t)(AT_TILE / 2 >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
      auto part = [&](const uint32_t col, const bool later) {      // (a whole tile: no condition per step)
        if (ks == 8) {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) umma_bf16_ta(d, pa + (kk >> 1) * 32 + col + (kk & 1) * 8, vd + kk * (2048 >> 4), idesc_o, (later || kk) ? 1u : 0u);
        } else {
#pragma unroll 1
          for (int kk = 0; kk < ks; ++kk) umma_bf16_ta(d, pa + (kk >> 1) * 32 + col + (kk & 1) * 8, vd + kk * (2048 >> 4), idesc_o, (later || kk) ? 1u : 0u);
        }
      };
      if (leader && !gone) {
        part(0, begun[g]);
        if (MODE == AT_PROMPT) umma_commit(h_done + 8u * g);
        part(16, true);
      }
      if (MODE == AT_PROMPT) {
        if (!gp_wait_warp(l_full + 8u * g, (uint32_t)(nl[g]++ & 1), dead, a.tries)) gone = true;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (leader && !gone) part(0, true);
      }
      if (leader && !gone && tile == tiles[g] - 1) umma_commit(o_done + 8u * g);
      begun[g] = true;
    };
    auto scores = [&](const int g, const int st, const int t, const int buf) {
      if (leader && !gone) {
        const uint32_t idesc_s = idesc | ((uint32_t)steps(g, t) << 18);
        const uint64_t qd = umma_desc_sw128(q_s + g * AT_TILE), kd = umma_desc_sw128(k_s + st * AT_TILE);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint32_t off = (kk >> 2) * (AT_TILE / 2 >> 4) + (kk & 3) * 2;
          umma_bf16(tmem + buf * 128, qd + off, kd + off, idesc_s, kk ? 1u : 0u);
        }
        umma_commit(s_full + 8u * buf);
      }
    };
    int n = 0, np[2] = {0, 0};
    if (one) {
      // One group: the next tile's scores are issued in front of this one's values, into the other score columns, so that its threads go on without waiting for the products
      // (5 600 cycles a tile when they did).  Score columns, weights and stages of tile n have the parity of n; barriers of their own each, since two tiles may be ahead.
      auto finish = [&](const int k, const int tile) {
        const int st = k & 1;
        if (!gp_wait_warp(v_full + 8u * st, (uint32_t)((k >> 1) & 1), dead, a.tries)) gone = true;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (!gp_wait_warp(p_full + 8u * st, (uint32_t)((k >> 1) & 1), dead, a.tries)) gone = true;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        values(0, st, tile);
        if (leader && !gone) umma_commit(v_empty + 8u * st);
      };
      for (int t = 0; t < ntiles; ++t) {
        if (!need(0, t)) continue;
        const int st = n & 1;
        if (!gp_wait_warp(k_full + 8u * st, (uint32_t)((n >> 1) & 1), dead, a.tries)) gone = true;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        scores(0, st, t, st);
        if (leader && !gone) umma_commit(k_empty + 8u * st);
        if (n > 0) finish(n - 1, prev);
        prev = t;
        ++n;
      }
      finish(n - 1, prev);
    } else {
    for (int t = 0; t <= ntiles; ++t) {
      const bool more = t < ntiles;
      const bool n0 = more && need(0, t), n1 = more && need(1, t);
      if (more && !n0 && !n1) continue;
      const int st = n & 1;
      if (more) {
        if (!gp_wait_warp(k_full + 8u * st, (uint32_t)((n >> 1) & 1), dead, a.tries)) gone = true;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      }
      if (pend[0] || pend[1]) {
        if (!gp_wait_warp(v_full + 8u * (st ^ 1), (uint32_t)(((n - 1) >> 1) & 1), dead, a.tries)) gone = true;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      }
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        if (pend[g]) {
          if (!gp_wait_warp(p_full + 8u * g, (uint32_t)(np[g]++ & 1), dead, a.tries)) gone = true;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          values(g, st ^ 1, prev);
          pend[g] = false;
        }
        if (g ? n1 : n0) {
          scores(g, st, t, g);
          pend[g] = true;
        }
      }
      if (leader && !gone) {
        if (n > 0) umma_commit(v_empty + 8u * (st ^ 1));
        if (more) umma_commit(k_empty + 8u * st);
      }
      prev = t;
      ++n;
    }
    }
  } else if (warp >= 16) {
    // ---- key and value tiles ----
    const int lt = tid - 512;
    bool gone = false;
    const bf16 *kc = a.k + (size_t)kvh * 128, *vc = a.v + (size_t)kvh * 128;
    auto stage = [&](const bf16* src, const long ld, const uint32_t dst, const int j0, const uint32_t bar) {
      if (gone) return;
      const int n16 = min(8, (jend - j0) / 16 + 1) * 256;      // 16 lanes read a row; rows behind the last steps of 16 keys are not looked at
      for (int i = lt; i < n16; i += AT_LOADERS) {
        const int r = i >> 4, c = i & 15, j = j0 + r;
        const bool ok = j <= jend;
        const uint32_t at = dst + (uint32_t)((c >> 3) * (AT_TILE / 2) + r * 128 + (((c & 7) ^ (r & 7)) << 4));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at), "l"(src + (size_t)(ok ? j : 0) * ld + c * 8), "r"(ok ? 16 : 0) : "memory");
      }
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");   // when this thread's copies have landed
    };
    int n = 0;
    for (int t = 0; t < ntiles; ++t) {
      if (!need(0, t) && !need(1, t)) continue;
      const int st = n & 1;
      const uint32_t ph = (uint32_t)(((n >> 1) - 1) & 1);
      if (n >= 2 && !gp_wait_warp(k_empty + 8u * st, ph, dead, a.tries)) gone = true;
      if (n > 0 || !a.lost) stage(kc, a.ldk, k_s + st * AT_TILE, t * AT_KEYS, k_full + 8u * st);
      if (n >= 2 && !gp_wait_warp(v_empty + 8u * st, ph, dead, a.tries)) gone = true;
      stage(vc, a.ldv, v_s + st * AT_TILE, t * AT_KEYS, v_full + 8u * st);
      ++n;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else {
    // ---- two threads per row ----
    const int g = warp >> 3, half = (warp >> 2) & 1, wq = warp & 3;
    const int nqg = g ? nq[1] : nq[0], firstg = g ? first[1] : first[0], tilesg = g ? tiles[1] : tiles[0];
    if (nqg > 0) {
      {   // the group's queries: a warp per row, rounded to bf16 once
        unsigned char* qt = gbase + g * AT_TILE;
        typedef typename std::conditional<MODE == AT_PROMPT, uint2, float4>::type Quad;
        const int c = lane >> 1;
#pragma unroll
        for (int b = 0; b < 16; b += 8) {      // eight rows on their way together (one by one, behind a condition each: 4 600 cycles of bf16 rows, 8 400 of f32)
          Quad x[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int r = (half * 4 + wq) * 16 + b + i, qi = min(r / HG, nqg - 1), hh = min(r - qi * HG, HG - 1);
            x[i] = *reinterpret_cast<const Quad*>(reinterpret_cast<const typename std::conditional<MODE == AT_PROMPT, bf16, float>::type*>(a.q) +
                                                  (size_t)(row0(g) + qi) * a.ldq + (size_t)(kvh * HG + hh) * 128 + lane * 4);
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int r = (half * 4 + wq) * 16 + b + i;
            uint2 w;
            if constexpr (MODE == AT_PROMPT) w = x[i];
            else w = make_uint2(bf_pair(x[i].x, x[i].y), bf_pair(x[i].z, x[i].w));
            if (r / HG >= nqg) w = make_uint2(0u, 0u);
            *reinterpret_cast<uint2*>(qt + (c >> 3) * (AT_TILE / 2) + r * 128 + (((c & 7) ^ (r & 7)) << 4) + (lane & 1) * 8) = w;
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(q_full + 8u * g);
      }
      const int r = wq * 32 + lane, qi = r / HG, head = kvh * HG + (r - qi * HG), pos = firstg + qi;
      const bool live = qi < nqg;
      const int wfirst = firstg + (wq * 32) / HG, wlast = firstg + min(nqg - 1, (wq * 32 + 31) / HG);
      const bool wfull = (wq * 32 + 31) / HG < nqg;
      const int lo = max(a.window > 0 ? pos - a.window + 1 : 0, a.chunk > 0 ? pos - pos % a.chunk : 0);
      const int keep = a.window > 0 && a.chunk <= 0 ? a.keep : 0;
      const float icap = a.cap > 0.f ? 1.f / a.cap : 0.f;
      float r1 = 0.f, r2 = 0.f;
      if (MODE == AT_DIST && a.r12) { r1 = a.r12[head]; r2 = a.r12[a.H + head]; }
      const uint32_t lanes = (uint32_t)(wq * 32) << 16, s_0 = tmem + lanes + g * 128 + half * 64, o_t = tmem + lanes + 256 + g * 128 + half * 64;
      // where this thread and the row's other one leave a number for each other, two tiles in turn; the two warps meet at a barrier of their own
      float* mine = reinterpret_cast<float*>(gbase + 6 * AT_TILE + 256) + g * 256 + half * 128 + r;
      const float* other = reinterpret_cast<float*>(gbase + 6 * AT_TILE + 256) + g * 256 + (half ^ 1) * 128 + r;
      const int pair_bar = 1 + g * 4 + wq;
      auto meet = [&](const float v, const int turn) {
        mine[turn * 512] = v;
        asm volatile("bar.sync %0, 64;" ::"r"(pair_bar) : "memory");
        return other[turn * 512];
      };
      // the score of entry i of the tile in front of the mask, from the raw product
      auto score2 = [&](float& x, float& y, const int key, const bool near) {
        if (MODE == AT_PROMPT) {
          round2(x, y);
          x *= a.scale; y *= a.scale;
          round2(x, y);
        } else {
          x *= a.scale; y *= a.scale;
          if (MODE == AT_CAP || (MODE == AT_DIST && a.cap > 0.f)) {
            x *= icap; y *= icap;
            if (near) cap_near(x, y, a.cap);
            else { x = a.cap * fast_tanh(x); y = a.cap * fast_tanh(y); }
          }
          if (MODE == AT_DIST && a.r12) {
            x -= r1 * __logf(fmaf(r2, fmaxf((float)(pos - key), 0.f), 1.f));
            y -= r1 * __logf(fmaf(r2, fmaxf((float)(pos - key - 1), 0.f), 1.f));
          }
        }
      };
      float ref = -INFINITY, sum = 0.f;
      int c = 0;
      for (int t = 0; t < tilesg; ++t) {
        if (!need(g, t)) continue;
        const int buf = one ? c & 1 : g;
        const uint32_t s_t = one ? s_0 + buf * 128 : s_0;
        gp_wait_warp(s_full + 8u * buf, (uint32_t)((one ? c >> 1 : c) & 1), dead, a.tries);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int j0 = t * AT_KEYS, k0 = j0 + half * 64;
        // tiles that every row of the warp sees whole need no per-score test
        const bool whole = wfull && j0 + AT_KEYS - 1 <= wfirst && (a.window <= 0 || wlast - j0 < a.window) && (a.chunk <= 0 || j0 >= wlast - wlast % a.chunk);
        const int hi_k = live ? pos - k0 : -1, lo_k = lo - k0, kp_k = keep - k0;
        float mx = -INFINITY;
        float s[2][32];
        tmem_ld32(s_t, s[0]);
        tmem_ld_wait();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (h == 0) tmem_ld32(s_t + 32, s[1]);      // on its way while the first half is worked on
          if (k0 + h * 32 <= wlast) {      // (keys behind every row of the warp: masked below, whatever they are)
            bool near = false;
            if (MODE == AT_CAP || (MODE == AT_DIST && a.cap > 0.f)) {      // of a whole warp: no score of its rows is far up the cap.  A NaN counts as far, where it becomes -cap, whatever the others are
              float far = fabsf(s[h][0]);
#pragma unroll
              for (int i = 1; i < 32; ++i) far = max_nan(far, fabsf(s[h][i]));
              near = __all_sync(0xffffffffu, far * fabsf(a.scale) * icap <= AT_NEAR);
            }
            if (near) {
#pragma unroll
              for (int i = 0; i < 32; i += 2) score2(s[h][i], s[h][i + 1], k0 + h * 32 + i, true);
            } else {
#pragma unroll
              for (int i = 0; i < 32; i += 2) score2(s[h][i], s[h][i + 1], k0 + h * 32 + i, false);
            }
          }
          if (!whole) {
            // which of the 32 keys the row sees, as bits: conditions per score became divergent branches (8 400 cycles a tile)
            const uint32_t sees = first_bits(hi_k + 1 - h * 32) & (~first_bits(lo_k - h * 32) | first_bits(kp_k - h * 32));
#pragma unroll
            for (int i = 0; i < 32; ++i) s[h][i] = (sees >> i) & 1u ? s[h][i] : -INFINITY;
          }
#pragma unroll
          for (int i = 0; i < 32; ++i) mx = fmaxf(mx, s[h][i]);
          if (h == 0) tmem_ld_wait();
        }
        mx = fmaxf(mx, meet(mx, c & 1));
        const float mk = rintf(mx * AT_L2E);
        if (c == 0) ref = mk;
        else if (__any_sync(0xffffffffu, mk > ref + AT_SLACK)) {      // (from -inf too: nothing summed yet)
          const bool up = mk > ref + AT_SLACK;
          const float al = up ? (ref == -INFINITY ? 0.f : pow2_down(ref - mk)) : 1.f;
          if (up) ref = mk;
          sum *= al;
          if (one) {      // the product in front ends (of two groups it has: this tile's scores were issued behind it)
            gp_wait_warp(v_empty + 8u * (buf ^ 1), (uint32_t)(((c - 1) >> 1) & 1), dead, a.tries);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          }
#pragma unroll 1
          for (int i = 0; i < 4; ++i) {
            uint32_t x[16];
            tmem_ld16(o_t + i * 16, x);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) x[j] = __float_as_uint(__uint_as_float(x[j]) * al);
            tmem_st16(o_t + i * 16, x);
          }
        }
        const float u = ref == -INFINITY ? 0.f : -ref;
        uint32_t rest[2][16];      // AT_PROMPT
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t hi[16], lw[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float p = ex2f(fmaf(s[h][2 * j], AT_L2E, u)), q = ex2f(fmaf(s[h][2 * j + 1], AT_L2E, u));
            sum += p + q;
            hi[j] = bf_pair(p, q);
            const float p1 = p - __uint_as_float(hi[j] << 16), q1 = q - __uint_as_float(hi[j] & 0xffff0000u);
            lw[j] = bf_pair(p1, q1);
            if (MODE == AT_PROMPT) rest[h][j] = bf_pair(p1 - __uint_as_float(lw[j] << 16), q1 - __uint_as_float(lw[j] & 0xffff0000u));
          }
          tmem_st16(s_t + h * 32, hi);
          tmem_st16(s_t + h * 32 + 16, lw);
        }
        tmem_st_wait();
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full + 8u * buf);
        if (MODE == AT_PROMPT) {
          gp_wait_warp(h_done + 8u * g, (uint32_t)(c & 1), dead, a.tries);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          tmem_st16(s_t, rest[0]);
          tmem_st16(s_t + 32, rest[1]);
          tmem_st_wait();
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(l_full + 8u * g);
        }
        ++c;
      }
      // what the output is divided and multiplied by, while the last product runs
      float f = 1.f, den = sum + meet(sum, c & 1);
      if (MODE != AT_PROMPT && a.sink && live) {
        const float sk = a.sink[head], mm = fmaxf(ref, rintf(sk * AT_L2E));
        f = ref == -INFINITY ? 0.f : pow2_down(ref - mm);
        den = den * f + exp2f(fmaf(sk, AT_L2E, -mm));
      }
      const int m = pos - P;
      float sc = f / den;
      if (MODE != AT_PROMPT && live) {
        if (a.gate && !a.entry) sc *= sigmoid_f(a.gate[(size_t)m * a.gate_ld + head]);
        if (a.mult != 0.f) sc *= a.mult;
      }
      gp_wait_warp(o_done + 8u * g, 0, dead, a.tries);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const float* ge = MODE != AT_PROMPT && a.entry ? a.gate + (size_t)m * a.gate_ld + (size_t)head * 128 + half * 64 : nullptr;
      const size_t at = (size_t)m * a.ldo + (size_t)head * 128 + half * 64;
#pragma unroll 1
      for (int i = 0; i < 4; ++i) {
        uint32_t x[16];
        tmem_ld16(o_t + i * 16, x);
        tmem_ld_wait();
        if (live) {
          float v[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(x[j]);
          float far = 0.f;      // NaN as soon as one of them is not finite
#pragma unroll
          for (int j = 0; j < 16; ++j) far = fmaf(v[j], 0.f, far);
          if (far != 0.f && fabsf(sc) < INFINITY) {
            at_row_again<MODE>(a, m, head, half * 64 + i * 16, pos, lo, keep, ref == -INFINITY ? 0.f : ref, sc, ge ? ge + i * 16 : nullptr);
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] *= sc;
            if (ge) {
#pragma unroll
              for (int j = 0; j < 16; ++j) v[j] *= sigmoid_f(ge[i * 16 + j]);
            }
            at_store(a, at + i * 16, v);
          }
        }
        __syncwarp();
      }
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*dead) {      // products still on their way end before the memory they use is given back (every loading thread has waited for its own copies)
    if (warp == 19 && leader) {
      umma_commit(drain);
      mbar_wait_bounded(drain, 0u, 1 << 14);
    }
    const int n = (nq[0] + nq[1]) * HG * 128;
    for (int i = tid; i < n; i += AT_THREADS) {
      const int q = i / (HG * 128), m = ENDS && q >= nq[0] ? m1 + q - nq[0] : m0 + q;
      const size_t at = (size_t)m * a.ldo + (size_t)kvh * HG * 128 + i % (HG * 128);
      if (a.out_f32) reinterpret_cast<float*>(a.out)[at] = __int_as_float(0x7fffffff);
      else reinterpret_cast<uint16_t*>(a.out)[at] = 0x7fff;
    }
    __syncthreads();
  }
  if (warp == 19) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}
