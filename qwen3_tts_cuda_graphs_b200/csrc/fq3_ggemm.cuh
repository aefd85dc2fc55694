// fq3_ggemm.cuh — grouped products of routed experts on tcgen05 (FQ3C_GGEMM, bf16): sorted rows of each expert against that expert's weights.
//
// Included by fq3_codec.cu behind fq3_gemm.cuh, whose barriers, copies and products it uses.
#pragma once

// grid (ceil(N / GT_BN), ceil(rows / 128) + experts): a CTA takes 128 rows of one expert (found from the segment starts, which the launch in front wrote) and GT_BN of its columns.
// Warps 0-7 gather the rows by 16-byte copies into the swizzled stages (a row list for the first product, the rows themselves for the second), the last warp asks for the weights by TMA,
// one box a stage, the one before it issues the MMAs; warps 0-7 then take the accumulator through the epilogue, a row per lane, 16 columns at a time.  Two CTAs share an SM, so that one's
// epilogue runs beside the other's products; 96 KB of stages each.
// What bounds it: the latency of the three stages along a tile's 12 - 32 k-blocks (four stages of 64 columns: 21.0 and 12.2 us); rows behind an expert's last one are zeros.  1402 rows of 16 experts: 1536 x 1024 with gated units
// 34.8 us on mma.sync, 16.9 here; 1024 x 768 24.5 and 9.2.  (Activations by a flag per tile: with one per entry the second product fetched their code sixteen times over, 17.6 us.)
constexpr int GT_BN = 128, GT_ST = 3, GT_LOADERS = 256, GT_THREADS = GT_LOADERS + 64;
constexpr int GT_A_BYTES = TM * TK * 2, GT_STAGE_BYTES = GT_A_BYTES + GT_BN * TK * 2, GT_SMEM = GT_ST * GT_STAGE_BYTES + 1024 + 128;

template <bool GLU>
__device__ __forceinline__ void gt_epilogue(const SeqGemm& g, const int r, const int n0, const uint32_t (&acc)[16], const float w, const bool whole) {
  float v[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(acc[j]);
  if constexpr (GLU) {
    if (whole && n0 + 16 <= g.N && !(g.flags & FQ3C_OUT_F32)) {
      float y[8];
      if (g.flags & FQ3C_GELU_TANH) {
#pragma unroll
        for (int j = 0; j < 8; ++j) y[j] = gelu_tanh_f(w * v[2 * j]) * (w * v[2 * j + 1]);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) y[j] = silu_f(w * v[2 * j]) * (w * v[2 * j + 1]);
      }
      *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(g.C) + (size_t)r * g.ldc + (n0 >> 1)) = make_uint4(bf_pair(y[0], y[1]), bf_pair(y[2], y[3]), bf_pair(y[4], y[5]), bf_pair(y[6], y[7]));
      return;
    }
#pragma unroll
    for (int j = 0; j < 16; j += 2)
      if (n0 + j + 1 < g.N) sg_store_glu(g, r, 0, n0 + j, v[j], v[j + 1], w);
  } else {
    if (g.flags & FQ3C_GELU) {
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = gelu_f(v[j]);
    }
    if (g.flags & FQ3C_GELU_TANH) {
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = gelu_tanh_f(v[j]);
    }
    if (g.flags & FQ3C_SIGMOID) {
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = sigmoid_f(v[j]);
    }
    if (g.flags & FQ3C_RELU2) {
#pragma unroll
      for (int j = 0; j < 16; ++j) { v[j] = fmaxf(v[j], 0.f); v[j] *= v[j]; }
    }
    const size_t at = (size_t)r * g.ldc + n0;
    if (g.flags & FQ3C_OUT_F32) {
      float* c = reinterpret_cast<float*>(g.C) + at;
      if (whole && n0 + 16 <= g.N) {
#pragma unroll
        for (int h = 0; h < 16; h += 8) {
          uint32_t x[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) x[j] = __float_as_uint(v[h + j]);
          st32(c + h, x);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) if (n0 + j < g.N) c[j] = v[j];
      }
    } else {
      bf16* c = reinterpret_cast<bf16*>(g.C) + at;
      if (whole && n0 + 16 <= g.N) {
        uint32_t x[8];
        pack16(v, x);
        st32(c, x);
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) if (n0 + j < g.N) c[j] = __float2bfloat16_rn(v[j]);
      }
    }
  }
}

template <bool GLU>
__global__ void __launch_bounds__(GT_THREADS, 2) fq3s_ggemm_tc_kernel(const __grid_constant__ SeqGemm g, const __grid_constant__ CUtensorMap tmB, const int whole) {
  constexpr int MMA_WARP = GT_LOADERS / 32, TMA_WARP = MMA_WARP + 1;
  seq_dep_begin(g.M);
  int row0 = -1, row_end = 0, e = 0;
  for (int t = blockIdx.y; e < g.E; ++e) {
    const int s0 = g.seg[e], s1 = g.seg[e + 1], nt = (s1 - s0 + TM - 1) / TM;
    if (t < nt) { row0 = s0 + t * TM; row_end = min(s1, row0 + TM); break; }
    t -= nt;
  }
  if (row0 < 0) return;
  extern __shared__ unsigned char gt_raw[];
  const uint32_t raw = smem_u32(gt_raw), base = (raw + 1023u) & ~1023u;
  unsigned char* gbase = gt_raw + (base - raw);
  // rows of a stage are there, its weights are there (a barrier of their own: the copy engine alone completes it, also when the loaders gave up; the second wait a k-block costs up to 1 %), the stage is free, all products are done
  const uint32_t full = base + GT_ST * GT_STAGE_BYTES, boxes = full + 8u * GT_ST, empty = boxes + 8u * GT_ST, done = empty + 8u * GT_ST;
  uint32_t* words = reinterpret_cast<uint32_t*>(gbase + GT_ST * GT_STAGE_BYTES + 24 * GT_ST + 8);      // tensor-memory address | a wait ran out | weight boxes asked for
  volatile int* dead = reinterpret_cast<volatile int*>(words + 1);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31, n0 = blockIdx.x * GT_BN, KT = (g.K + TK - 1) / TK, tries = g.lost ? GP_TRIES_TEST : GP_TRIES;
  if (tid == 0) {
    for (int s = 0; s < GT_ST; ++s) { mbar_init(full + 8u * s, GT_LOADERS); mbar_init(boxes + 8u * s, 1); mbar_init(empty + 8u * s, 1); }
    mbar_init(done, 1);
    words[1] = 0;
    words[2] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(words)), "r"(GT_BN) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xffffffffu, words[0], 0);
  const bool leader = elect_one();
  bool there = true;
  if (warp == TMA_WARP) {
    int n = 0;
    for (int kt = 0, st = 0; kt < KT && there; ++kt) {
      if (kt >= GT_ST && !gp_wait_all(empty + 8u * st, (uint32_t)((kt / GT_ST - 1) & 1), dead, tries)) { there = false; break; }
      if (leader) {
        mbar_expect(boxes + 8u * st, GT_BN * TK * 2);
        if (kt > 0 || !g.lost) tma_2d(base + st * GT_STAGE_BYTES + GT_A_BYTES, &tmB, kt * TK, e * g.N + n0, boxes + 8u * st);
      }
      ++n;
      if (++st == GT_ST) st = 0;
    }
    if (leader) words[2] = (uint32_t)n;
  } else if (warp == MMA_WARP) {
    // instruction descriptor: D = F32, A = B = BF16, both K-major, N = GT_BN, M = 128
    constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(GT_BN >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);
    const uint64_t d0 = umma_desc_sw128(base);
    for (int kt = 0, st = 0; kt < KT; ++kt) {
      if (!gp_wait_all(boxes + 8u * st, (uint32_t)((kt / GT_ST) & 1), dead, tries) || !gp_wait_all(full + 8u * st, (uint32_t)((kt / GT_ST) & 1), dead, tries)) { there = false; break; }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // the rows came through the generic proxy
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint64_t da = d0 + st * (GT_STAGE_BYTES >> 4), db = da + (GT_A_BYTES >> 4);
      if (leader) {
#pragma unroll
        for (int kk = 0; kk < TK / 16; ++kk) umma_bf16(tmem, da + 2 * kk, db + 2 * kk, idesc, kt | kk ? 1u : 0u);
        umma_commit(empty + 8u * st);
      }
      __syncwarp();
      if (++st == GT_ST) st = 0;
    }
    if (leader && there) umma_commit(done);
    __syncwarp();
  } else {
    const int piece = tid & 7, lr = tid >> 3;
    const bf16* src[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = row0 + lr + 32 * i;
      src[i] = r < row_end ? reinterpret_cast<const bf16*>(g.A) + (size_t)(g.rows ? g.rows[r] : r) * g.lda + piece * 8 : nullptr;
    }
    unsigned char* dst = gbase + lr * 128 + ((piece ^ (lr & 7)) << 4);      // (rows 32 apart share the swizzle)
    for (int kt = 0, st = 0; kt < KT; ++kt) {
      if (kt >= GT_ST) {      // (all lanes: with one that polls for the others 17.8 and 9.8 us)
        there = gp_wait_all(empty + 8u * st, (uint32_t)((kt / GT_ST - 1) & 1), dead, tries);
        if (!there) break;
      }
      const bool in = kt * TK + piece * 8 < g.K;
#pragma unroll
      for (int i = 0; i < 4; ++i) cp_async16(dst + st * GT_STAGE_BYTES + i * 32 * 128, in && src[i] ? src[i] + kt * TK : reinterpret_cast<const bf16*>(g.A), in && src[i]);
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(full + 8u * st) : "memory");
      if (++st == GT_ST) st = 0;
    }
    // warp w reads tensor-memory lanes 32 (w & 3) .. +31; the first four warps take the lower columns
    if (there) there = gp_wait_warp(done, 0u, dead, tries);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int r = row0 + (warp & 3) * 32 + lane, c0 = (warp >> 2) * (GT_BN / 2);
    const uint32_t ta = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0;
    const float w = GLU && r < row_end ? sg_row_scale(g, r) : 1.f;
    if (row0 + (warp & 3) * 32 < row_end)
#pragma unroll 1
      for (int p = 0; p < GT_BN / 2 && n0 + c0 + p < g.N; p += 32) {
        uint32_t x[16], y[16];
        tmem_ld16(ta + p, x);
        tmem_ld16(ta + p + 16, y);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (r < row_end) {
          gt_epilogue<GLU>(g, r, n0 + c0 + p, x, w, whole);
          gt_epilogue<GLU>(g, r, n0 + c0 + p + 16, y, w, whole);
        }
      }
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  if (!there && lane == 0) wait_ran_out();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*dead) {      // copies and products on their way end before their memory is given back; the tile's outputs become NaN
    if (warp == MMA_WARP && leader) {
      umma_commit(done);
      mbar_wait_bounded(done, 0u, 1 << 14);
    }
    if (tid < GT_ST && tid < (int)words[2]) {
      const int i = (int)words[2] - 1 - tid;
      mbar_wait_bounded(boxes + 8u * (i % GT_ST), (uint32_t)((i / GT_ST) & 1), 1 << 14);
    }
    const int cols = GLU ? GT_BN / 2 : GT_BN, width = GLU ? g.N / 2 : g.N, c0 = GLU ? n0 / 2 : n0;
    for (int i = tid; i < (row_end - row0) * cols; i += GT_THREADS) {
      const int c = c0 + i % cols;
      const size_t at = (size_t)(row0 + i / cols) * g.ldc + c;
      if (c >= width) continue;
      if (g.flags & FQ3C_OUT_F32) reinterpret_cast<float*>(g.C)[at] = __int_as_float(0x7fffffff);
      else reinterpret_cast<uint16_t*>(g.C)[at] = 0x7fff;
    }
  }
  __syncthreads();
  if (warp == MMA_WARP) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(GT_BN) : "memory");
}
