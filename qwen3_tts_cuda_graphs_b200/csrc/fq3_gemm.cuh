// fq3_gemm.cuh — the tcgen05 GEMM of the op lists: persistent, warp-specialised, operand tiles by TMA.
//
// Included by fq3_codec.cu behind its epilogues.  C = epi(A . B^T), A [rows, K] activations (rows shifted per tap for the implicit
// convolutions), B [N, K] weights, both bf16, accumulators f32 in tensor memory.
#pragma once

// What the host decides about a launch.
struct GemmPlan {
  int bn;        // columns of a tile (multiple of 16)
  int stages;    // operand stages in shared memory
  int a_rows;    // rows of the A box: 128, or what a single row tile needs (multiple of 8; the accumulator rows behind it are never read)
  int mt, nt;    // row and column tiles
  int parts;     // runs of a tile's k-blocks that are summed by themselves, each in an accumulator of its own, and then added in order
  int splits;    // CTAs that share a tile's parts: a cluster, its partial tiles meet in shared memory
  int per;       // parts of a CTA: one or two (the last CTA may have one less)
  int kpt, kb;   // k-blocks per tap, in all
  int tail;      // MMAs (16 columns each) of a tap's last k-block
  int acc_cols;  // tensor-memory columns of one accumulator (power of two); two of them, of a staged tile as many as the CTA has parts
  int early_b;   // B is not written by the launches in front: its first stages are asked for before they have ended
  int vec16;     // the epilogue may move 16 columns of a row at a time
  int staged;    // the epilogue takes its tile from shared memory, spread over all threads: split sums, and few rows (a CTA has one tile then)
  int tries;     // of a wait before it gives up
  int lost;      // k-block whose rows are never asked for (tests of the error path), else -1
};
__host__ __device__ constexpr int gp_threads(int epi_warps) { return (epi_warps + 2) * 32; }
constexpr int GP_PAR = 256;         // columns of a tile at most: its bias, scale and SnakeBeta parameters lie in shared memory
constexpr int GP_BAR_BYTES = 512 + 4 * GP_PAR * 4;   // barriers, tensor-memory address, error word; parameters
__host__ __device__ constexpr int gp_a_bytes(int a_rows) { return (a_rows * TK * 2 + 1023) & ~1023; }
__host__ __device__ constexpr int gp_stage_bytes(int a_rows, int bn) { return gp_a_bytes(a_rows) + bn * TK * 2; }
__host__ __device__ constexpr int gp_part_pitch(int bn) { return bn + 4; }   // floats per row of a partial tile: 16-byte rows, 4 banks apart

// A bounded wait.  When its tries run out (about a second) it sets the block's word `dead`; the block's other waits give up
// when they see `dead`.  A lane whose wait gave up (false) issues no more copies, products or commits, so that no barrier gets an arrival that its phase does not
// expect; it sets the error words behind its loop (a call inside would keep the loop's operands out of the uniform registers), and at its end the kernel waits
// for what had been issued and fills its outputs with NaN.
constexpr int GP_TRIES = 1 << 20, GP_TRIES_TEST = 4096;
__device__ __forceinline__ bool gp_wait(const uint32_t bar, const uint32_t parity, volatile int* dead, const int tries) {
  if (mbar_try_wait(bar, parity)) return true;
  for (int i = 1; !mbar_try_wait(bar, parity); ++i)
    if (i > 256 || i > tries) {      // (a try suspends the thread for a while by itself)
      if (*dead || i > tries) {
        *dead = 1;
        return false;
      }
      __nanosleep(i > 8192 ? 1000 : 20);
    }
  return true;
}
// the same for a whole warp that goes on together: each lane tries for itself (with a vote per try the waiting warps took issue slots from the working ones)
__device__ __forceinline__ bool gp_wait_warp(const uint32_t bar, const uint32_t parity, volatile int* dead, const int tries) {
  const bool there = gp_wait(bar, parity, dead, tries);
  if (!there) wait_ran_out();
  __syncwarp();
  return there;
}
// and for the issuing warps: one answer for all lanes, so that they leave their loops together
__device__ __forceinline__ bool gp_wait_all(const uint32_t bar, const uint32_t parity, volatile int* dead, const int tries) {
  return __all_sync(0xffffffffu, gp_wait(bar, parity, dead, tries));
}
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void mbar_expect(const uint32_t bar, const uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(const uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void umma_bf16(const uint32_t d, const uint64_t da, const uint64_t db, const uint32_t idesc, const uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d), "l"(da), "l"(db), "r"(idesc), "r"(acc)
      : "memory");
}
// arrives on the barrier when the MMAs issued so far are done (implies tcgen05.fence::before_thread_sync)
__device__ __forceinline__ void umma_commit(const uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tma_2d(const uint32_t dst, const CUtensorMap* map, const int x, const int y, const uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(x), "r"(y),
               "r"(bar)
               : "memory");
}
__device__ __forceinline__ void tmem_ld16(const uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),
        "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}
// 32 bytes of a row in one instruction (a whole sector): the rows of a warp are apart, so every store or load of a lane is a sector of its own
__device__ __forceinline__ void st32(void* p, const uint32_t (&w)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
               : "memory");
}
__device__ __forceinline__ void ld32(const void* p, uint32_t (&w)[8]) {
  asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
               : "l"(p)
               : "memory");
}
__device__ __forceinline__ uint32_t bf_pair(const float a, const float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
// both rounded to bf16
__device__ __forceinline__ void round2(float& a, float& b) {
  const uint32_t w = bf_pair(a, b);
  a = __uint_as_float(w << 16);
  b = __uint_as_float(w & 0xffff0000u);
}
__device__ __forceinline__ void round16(float (&v)[16]) {
#pragma unroll
  for (int j = 0; j < 16; j += 2) round2(v[j], v[j + 1]);
}
__device__ __forceinline__ void pack16(const float (&v)[16], uint32_t (&w)[8]) {
#pragma unroll
  for (int j = 0; j < 8; ++j) w[j] = bf_pair(v[2 * j], v[2 * j + 1]);
}

// Epilogue of 16 consecutive columns of one row: the arithmetic and order of epilogue_pair, every access a whole 32-byte sector.  The host
// has checked sizes, pitches and addresses (gemm_vec16).  r: the residual's 16 entries, asked for before the accumulator was read.  par: the tile's
// parameters from this column on (bias, scale, SnakeBeta's two, GP_PAR floats apart): from global memory they missed the few KB of L1 that are left
// beside the stages, behind the streaming residual (72 % of the stalls of a 96-column layer).
__device__ __forceinline__ void epilogue_row16(const fq3c_op& o, const int row, const int col, const uint32_t (&acc)[16], const uint32_t (&r)[8], const float* par) {
  if (row >= o.M || col >= o.N) return;
  float v[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(acc[j]);
  if (o.flags & FQ3C_BIAS) {
    const float4* b = reinterpret_cast<const float4*>(par);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 q = b[j];
      v[4 * j] += q.x; v[4 * j + 1] += q.y; v[4 * j + 2] += q.z; v[4 * j + 3] += q.w;
    }
  }
  if (o.flags & FQ3C_RELU2) {
#pragma unroll
    for (int j = 0; j < 16; ++j) { v[j] = fmaxf(v[j], 0.f); v[j] *= v[j]; }
  }
  const bool round = !(o.flags & FQ3C_NOROUND);
  if (round) round16(v);
  if (o.flags & FQ3C_SWIGLU) {
    float y[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) y[j] = round ? bf16r(bf16r(silu_f(v[2 * j])) * v[2 * j + 1]) : glu_f(o.flags, v[2 * j], v[2 * j + 1]);
    const size_t at = (size_t)row * o.ldc + (col >> 1);
    if (!round && (o.flags & FQ3C_OUT_F32)) {
      uint32_t w[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) w[j] = __float_as_uint(y[j]);
      st32(reinterpret_cast<float*>(o.C) + at, w);
    } else {
      *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(o.C) + at) = make_uint4(bf_pair(y[0], y[1]), bf_pair(y[2], y[3]), bf_pair(y[4], y[5]), bf_pair(y[6], y[7]));
    }
    return;
  }
  if (o.flags & FQ3C_GELU) {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = gelu_f(v[j]);
    if (round) round16(v);
  }
  if (o.flags & FQ3C_SILU) {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = silu_f(v[j]);
    round16(v);
  }
  if (o.flags & FQ3C_SCALE) {
    const float4* s = reinterpret_cast<const float4*>(par + GP_PAR);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 q = s[j];
      v[4 * j] *= q.x; v[4 * j + 1] *= q.y; v[4 * j + 2] *= q.z; v[4 * j + 3] *= q.w;
    }
    round16(v);
  }
  if (o.flags & FQ3C_RESID) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v[2 * j] += __uint_as_float(r[j] << 16);
      v[2 * j + 1] += __uint_as_float(r[j] & 0xffff0000u);
    }
    round16(v);
  }
  if (o.flags & FQ3C_CLAMP) {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = fminf(fmaxf(v[j], -1.f), 1.f);
  }
  const size_t at = (size_t)row * o.ldc + col;
  uint32_t w[8];
  if (o.flags & FQ3C_OUT_F32) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (int j = 0; j < 8; ++j) w[j] = __float_as_uint(v[8 * h + j]);
      st32(reinterpret_cast<float*>(o.C) + at + 8 * h, w);
    }
  } else {
    pack16(v, w);
    st32(reinterpret_cast<bf16*>(o.C) + at, w);
  }
  if (o.flags & FQ3C_SNAKE2) {
    const float4* ea = reinterpret_cast<const float4*>(par + 2 * GP_PAR);
    const float4* ib = reinterpret_cast<const float4*>(par + 3 * GP_PAR);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 a = ea[j], b = ib[j];
      const float x0 = v[4 * j] * a.x, x1 = v[4 * j + 1] * a.y, x2 = v[4 * j + 2] * a.z, x3 = v[4 * j + 3] * a.w;
      if (fmaxf(fmaxf(fabsf(x0), fabsf(x1)), fmaxf(fabsf(x2), fabsf(x3))) < SIN_SQ_NEAR) {
        v[4 * j] = fmaf(b.x, sin_sq_near(x0), v[4 * j]); v[4 * j + 1] = fmaf(b.y, sin_sq_near(x1), v[4 * j + 1]);
        v[4 * j + 2] = fmaf(b.z, sin_sq_near(x2), v[4 * j + 2]); v[4 * j + 3] = fmaf(b.w, sin_sq_near(x3), v[4 * j + 3]);
      } else {
        v[4 * j] = fmaf(b.x, sin_sq_far(x0), v[4 * j]); v[4 * j + 1] = fmaf(b.y, sin_sq_far(x1), v[4 * j + 1]);
        v[4 * j + 2] = fmaf(b.z, sin_sq_far(x2), v[4 * j + 2]); v[4 * j + 3] = fmaf(b.w, sin_sq_far(x3), v[4 * j + 3]);
      }
    }
    pack16(v, w);
    st32(reinterpret_cast<bf16*>(o.C2) + at, w);
  }
}
// shapes and addresses without whole sectors: out of line, so that the other path's code stays together
__device__ __noinline__ void epilogue_odd16(const fq3c_op& o, const int row, const int col, const float* acc) {
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = acc[8 * h + j];
    epilogue_row8(o, row, col + 8 * h, v);
  }
}
__device__ __forceinline__ void gp_epilogue(const fq3c_op& o, const GemmPlan& g, const int row, const int col, const uint32_t (&acc)[16], const uint32_t (&r)[8],
                                            const float* par) {
  if (g.vec16) {
    epilogue_row16(o, row, col, acc, r, par);
  } else {
    float v[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(acc[j]);
    epilogue_odd16(o, row, col, v);
  }
}

// NaN in place of `n` (even) columns of an output row, both outputs: a wait ran out
__device__ __noinline__ void poison(const fq3c_op& o, const int row, const int col, const int n) {
  if (row >= o.M) return;
  const bool glu = o.flags & FQ3C_SWIGLU, f32 = (o.flags & FQ3C_OUT_F32) && (!glu || (o.flags & FQ3C_NOROUND));
  for (int c = col; c < min(col + n, o.N); c += glu ? 2 : 1) {
    const size_t at = (size_t)row * o.ldc + (glu ? c >> 1 : c);
    if (f32) reinterpret_cast<float*>(o.C)[at] = __int_as_float(0x7fffffff);
    else reinterpret_cast<uint16_t*>(o.C)[at] = 0x7fff;
    if (o.flags & FQ3C_SNAKE2) reinterpret_cast<uint16_t*>(o.C2)[at] = 0x7fff;
  }
}

// One CTA per SM (or two small ones) walks the tiles t = blockIdx.x, + gridDim.x, ..; a tile is 128 rows x bn columns.  The last warp asks for the operand
// boxes up to `stages` k-blocks ahead, across tiles; the one before it issues the MMAs of tile n + 1 into the second accumulator while the others take tile n
// through the epilogue.  What bounds that is latency (accumulator, residual, a chain of conversions per row), so an SM has sixteen such warps, of one CTA or of two:
// with eight, 1900 x 6144 x 1024 with gated units took 33 us, with sixteen 24.  A tile whose sums come in parts is a cluster's: each CTA takes one or two parts, leaves their f32 partial tiles in its
// shared memory, and each then adds the partial tiles of a share of the rows in the parts' order.
// The launch may begin before the ones in front of it have ended (programmatic dependent launch): nothing but B (early_b) is touched before
// grid_dep_wait.
template <int MINB, int EPI_WARPS>
__global__ void __launch_bounds__(gp_threads(EPI_WARPS), MINB) fq3c_gemm_persist_kernel(const __grid_constant__ fq3c_op o, const __grid_constant__ GemmPlan g,
                                                                              const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB) {
  constexpr int MMA_WARP = EPI_WARPS, TMA_WARP = EPI_WARPS + 1, THREADS = gp_threads(EPI_WARPS), GROUPS = EPI_WARPS / 4;
  extern __shared__ unsigned char gp_raw[];
  const uint32_t raw = smem_u32(gp_raw), base = (raw + 1023u) & ~1023u;
  unsigned char* gbase = gp_raw + (base - raw);
  const int sb = gp_stage_bytes(g.a_rows, g.bn), ab = gp_a_bytes(g.a_rows);
  const uint32_t bars = base + g.stages * sb;
  const uint32_t full = bars, empty = bars + 8u * g.stages, acc_full = bars + 16u * g.stages, acc_empty = acc_full + 16;
  uint32_t* words = reinterpret_cast<uint32_t*>(gbase + g.stages * sb + 16 * g.stages + 32);   // tensor-memory address | dead | k-blocks asked for
  volatile int* dead = reinterpret_cast<volatile int*>(words + 1);
  const uint32_t drain = acc_empty + 32;      // (behind the words)
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int tiles = g.mt * g.nt, z = g.splits > 1 ? (int)(blockIdx.x % g.splits) : 0;
  const int t0 = g.splits > 1 ? (int)(blockIdx.x / g.splits) : (int)blockIdx.x, dt = g.staged ? tiles : (int)gridDim.x;
  const int part0 = z * g.per, own = min(g.per, g.parts - part0);      // this CTA's parts: k-blocks kb0 .. kbm and, of two, kbm .. kb1
  auto part_at = [&](const int p) { return p * g.kb / g.parts; };
  const int kb0 = part_at(part0), kbm = part_at(part0 + 1), kb1 = part_at(part0 + own);
  const int bufs = g.staged ? g.per : 2;
  const uint32_t cols = (uint32_t)(g.acc_cols * bufs);

  if (tid == 0) {
    for (int s = 0; s < g.stages; ++s) { mbar_init(full + 8u * s, 1); mbar_init(empty + 8u * s, 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(acc_full + 8u * b, 1); mbar_init(acc_empty + 8u * b, EPI_WARPS); }
    mbar_init(drain, 1);
    words[1] = 0;
    words[2] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(words)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (warp == TMA_WARP && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmA) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmB) : "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xffffffffu, words[0], 0);

  // The two issuing warps run their loops whole, with one elected lane at the copies, products and commits: in code of a single lane every operand goes
  // through per-lane registers (700 - 800 cycles a k-block with `lane == 0`, 380 with the election around the loop).  What bounds a k-block of narrow tiles is
  // the chain of instructions from one issue to the next, so the inner loops hold no more than a pointer's step each: taps and their last, shorter k-blocks are
  // outside of them.  347 -> 300 cycles a k-block (40 x 1024 x 8192: 25.9 -> 22.9 us); the tensor pipe needs 160 - 256 up to 128 columns.
  const bool leader = elect_one();
  if (warp == TMA_WARP) {
    const uint32_t tx = (uint32_t)(g.a_rows * TK * 2 + g.bn * TK * 2), ring = 8u * g.stages;
    int it = 0, early = 0;
    if (g.early_b && t0 < tiles) {   // the first tile's weights
      early = min(g.stages, kb1 - kb0);
      const int n0 = (t0 / g.mt) * g.bn;
      int tap = kb0 / g.kpt, c = kb0 - tap * g.kpt;
      for (int i = 0; i < early; ++i) {
        if (leader) {
          mbar_expect(full + 8u * i, tx);
          tma_2d(base + i * sb + ab, &tmB, tap * o.cin + c * TK, n0, full + 8u * i);
        }
        if (++c == g.kpt) { c = 0; ++tap; }
      }
    }
    grid_dep_wait();
    grid_dep_launch();
    bool there = true, wrapped = false;
    uint32_t st8 = 0, dst = base, ph = 1;      // 8 x stage, its memory, the parity that the end of its last use has
    for (int t = t0; t < tiles && there; t += dt) {
      const int n0 = (t / g.mt) * g.bn, m0 = o.m_begin + (t % g.mt) * TM;
      int tap = kb0 / g.kpt, c = kb0 - tap * g.kpt;
      for (int m = kb1 - kb0; m > 0 && there; ++tap, c = 0) {
        const int run = min(g.kpt - c, m), row = m0 + o.tap_off[tap];
        int x = c * TK, xb = tap * o.cin + x;
#pragma unroll 1
        for (int i = run; i > 0; --i) {
          if (wrapped && !gp_wait_all(empty + st8, ph, dead, g.tries)) { there = false; break; }
          if (leader) {
            if (it >= early) {
              mbar_expect(full + st8, tx);
              tma_2d(dst + ab, &tmB, xb, n0, full + st8);
            }
            if (it != g.lost) tma_2d(dst, &tmA, x, row, full + st8);
          }
          ++it;
          x += TK; xb += TK; st8 += 8; dst += sb;
          if (st8 == ring) { st8 = 0; dst = base; ph ^= 1u; wrapped = true; }
        }
        m -= run;
      }
    }
    if (leader) words[2] = (uint32_t)max(it, early);
    if (!there) wait_ran_out();
  } else if (warp == MMA_WARP) {
    grid_dep_wait();
    // instruction descriptor: D = F32, A = B = BF16, both K-major, N = bn, M = 128
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(g.bn >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);
    const uint64_t d0 = umma_desc_sw128(base);
    const uint32_t ring = 8u * g.stages, sb16 = (uint32_t)sb >> 4, ab16 = (uint32_t)ab >> 4;
    uint32_t st8 = 0, off = 0, ph = 0;      // 8 x stage, its memory / 16, parity
    bool there = true;
    int n = 0;
    for (int t = t0, k0 = kb0, k1 = kbm; t < tiles && there; ++n) {
      const int buf = n & 1;
      const uint32_t d = tmem + (uint32_t)(buf * g.acc_cols);
      if (n >= 2 && !gp_wait_all(acc_empty + 8u * buf, (uint32_t)((n / 2 - 1) & 1), dead, g.tries)) { there = false; break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      uint32_t acc = 0;
      for (int m = k1 - k0, c = k0 % g.kpt; m > 0 && there; c = 0) {
        const int run = min(g.kpt - c, m);
        const bool tail = c + run == g.kpt && g.tail != TK / 16;      // the tap's last k-block has fewer columns
#pragma unroll 1
        for (int i = run - (tail ? 1 : 0); i > 0; --i) {
          if (!gp_wait_all(full + st8, ph, dead, g.tries)) { there = false; break; }      // (filled by the copy engine: no tensor-memory fence)
          const uint64_t da = d0 + off, db = da + ab16;
          if (leader) {
            umma_bf16(d, da, db, idesc, acc);
#pragma unroll
            for (int kk = 1; kk < TK / 16; ++kk) umma_bf16(d, da + 2 * kk, db + 2 * kk, idesc, 1u);      // 16 columns = 32 bytes further
            umma_commit(empty + st8);
          }
          __syncwarp();
          acc = 1; st8 += 8; off += sb16;
          if (st8 == ring) { st8 = 0; off = 0; ph ^= 1u; }
        }
        if (tail && there) {
          there = gp_wait_all(full + st8, ph, dead, g.tries);
          const uint64_t da = d0 + off, db = da + ab16;
          if (leader && there) {
            for (int kk = 0; kk < g.tail; ++kk) umma_bf16(d, da + 2 * kk, db + 2 * kk, idesc, kk ? 1u : acc);
            umma_commit(empty + st8);
          }
          __syncwarp();
          acc = 1; st8 += 8; off += sb16;
          if (st8 == ring) { st8 = 0; off = 0; ph ^= 1u; }
        }
        m -= run;
      }
      if (leader && there) umma_commit(acc_full + 8u * buf);
      __syncwarp();
      if (k1 < kb1) { k0 = k1; k1 = kb1; }      // the CTA's other part
      else t += dt;
    }
    if (!there) wait_ran_out();
  } else {
    grid_dep_wait();
    // warp w reads tensor-memory lanes 32 (w & 3) .. +31 (= rows of the tile); each four warps take a run of the 16-column pieces
    const int pieces = g.bn / 16, p0 = (warp >> 2) * pieces / GROUPS, p1 = ((warp >> 2) + 1) * pieces / GROUPS;
    const int r_in = (warp & 3) * 32 + lane;
    const bool resid = g.vec16 && (o.flags & FQ3C_RESID);
    float* par = reinterpret_cast<float*>(gbase + g.stages * sb + 512);
    const bool params = g.vec16 && (o.flags & (FQ3C_BIAS | FQ3C_SCALE | FQ3C_SNAKE2));
    int n = 0, par_n0 = -1;
    if (g.staged) {      // the CTA's tile, once every product of it has ended: the partial tiles lie where its operands did
      const bool rows = o.m_begin + (t0 % g.mt) * TM + (warp & 3) * 32 < o.M;
      for (int h = 0; h < own; ++h) gp_wait_warp(acc_full + 8u * h, 0u, dead, g.tries);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int h = 0; h < own && rows; ++h) {
        float* part = reinterpret_cast<float*>(gbase) + (size_t)(h * g.a_rows + r_in) * gp_part_pitch(g.bn);
        const uint32_t ta = tmem + (uint32_t)(h * g.acc_cols) + ((uint32_t)((warp & 3) * 32) << 16);
        for (int p = p0; p < p1; p += 2) {
          uint32_t x[16], y[16];
          const bool two = p + 1 < p1;
          tmem_ld16(ta + p * 16, x);
          if (two) tmem_ld16(ta + p * 16 + 16, y);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (r_in < g.a_rows) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              *reinterpret_cast<uint4*>(part + p * 16 + 4 * j) = make_uint4(x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]);
              if (two) *reinterpret_cast<uint4*>(part + p * 16 + 16 + 4 * j) = make_uint4(y[4 * j], y[4 * j + 1], y[4 * j + 2], y[4 * j + 3]);
            }
          }
        }
      }
    } else
    for (int t = t0; t < tiles; t += dt, ++n) {
      const int buf = n & 1, n0 = (t / g.mt) * g.bn, m0 = o.m_begin + (t % g.mt) * TM;
      if (params && n0 != par_n0) {      // another column tile (rows go first): its parameters, when the epilogue warps have left the last one's
        par_n0 = n0;
        asm volatile("bar.sync 1, %0;" ::"n"(EPI_WARPS * 32) : "memory");
        const int col = n0 + tid;
        if (tid < g.bn && col < o.N) {
          const int c = col % o.col_mod;
          if (o.flags & FQ3C_BIAS) par[tid] = reinterpret_cast<const float*>(o.bias)[c];
          if (o.flags & FQ3C_SCALE) par[GP_PAR + tid] = reinterpret_cast<const float*>(o.scale)[c];
          if (o.flags & FQ3C_SNAKE2) {
            par[2 * GP_PAR + tid] = reinterpret_cast<const float*>(o.p0)[c];
            par[3 * GP_PAR + tid] = reinterpret_cast<const float*>(o.p1)[c];
          }
        }
        asm volatile("bar.sync 1, %0;" ::"n"(EPI_WARPS * 32) : "memory");
      }
      const int row = m0 + r_in;
      const bool rows = m0 + (warp & 3) * 32 < o.M;      // (warp-uniform)
      uint32_t rx[8], ry[8];
      // a piece of the residual, on its way while the accumulator is waited for or another piece is worked on
      auto ask = [&](const int p, uint32_t (&x)[8]) {
        if (resid && p < p1 && row < o.M && n0 + p * 16 < o.N) ld32(reinterpret_cast<const bf16*>(o.res) + (size_t)row * o.ldr + n0 + p * 16, x);
      };
      if (rows) { ask(p0, rx); ask(p0 + 1, ry); }
      gp_wait_warp(acc_full + 8u * buf, (uint32_t)((n / 2) & 1), dead, g.tries);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t ta = tmem + (uint32_t)(buf * g.acc_cols) + ((uint32_t)((warp & 3) * 32) << 16);
      if (rows)
        for (int p = p0; p < p1; p += 2) {
          uint32_t x[16], y[16];
          const bool two = p + 1 < p1;
          tmem_ld16(ta + p * 16, x);
          if (two) tmem_ld16(ta + p * 16 + 16, y);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (p + 2 >= p1) {      // this warp's last read of the accumulator
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty + 8u * buf);
          }
          gp_epilogue(o, g, row, n0 + p * 16, x, rx, par + p * 16);
          ask(p + 2, rx);
          if (two) gp_epilogue(o, g, row, n0 + p * 16 + 16, y, ry, par + p * 16 + 16);
          ask(p + 3, ry);
        }
      if ((!rows || p0 >= p1) && lane == 0) mbar_arrive(acc_empty + 8u * buf);
    }
  }
  __syncwarp();
  if (g.staged) {
    const int n0 = (t0 / g.mt) * g.bn, m0 = o.m_begin + (t0 % g.mt) * TM;
    const int pieces = g.bn / 8, items = min(TM, o.M - m0) * pieces;
    const int i0 = items / 2 * z / g.splits * 2, i1 = items / 2 * (z + 1) / g.splits * 2;      // (a row has an even number of pieces)
    int lost = 0;
    if (g.splits > 1) {      // every CTA of the cluster comes here, also after a wait that ran out
      asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
      if (tid < g.splits) {      // whether that CTA's part can be used; looked at behind the sums
        uint32_t far;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(far) : "r"(smem_u32(words + 1)), "r"(tid));
        asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(lost) : "r"(far) : "memory");
      }
    } else {
      __syncthreads();
      lost = *dead;
    }
    // Two lanes share two pieces: each adds up the lower or the upper four columns of both, so that a warp reads whole rows, and they swap the finished sums
    // (39 x 1024 x 2048 in eight parts 6.9 -> 6.3 us).
    for (int b = i0 + warp * 32; b < i1; b += THREADS) {
      const int i = min(b + lane, i1 - 1), r = i / pieces, p = i - r * pieces;
      const uint32_t mine = base + (uint32_t)((r * gp_part_pitch(g.bn) + (p & ~1) * 8 + (lane & 1) * 4) * 4), slot = (uint32_t)(g.a_rows * gp_part_pitch(g.bn) * 4);
      float4 q[8][2];      // every part is on its way before the first is added
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (s < g.parts) {
          uint32_t far = g.per == 2 && (s & 1) ? mine + slot : mine;
          if (g.splits > 1) asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(far) : "r"(far), "r"(g.per == 2 ? s >> 1 : s));
#pragma unroll
          for (int j = 0; j < 2; ++j)
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(q[s][j].x), "=f"(q[s][j].y), "=f"(q[s][j].z), "=f"(q[s][j].w) : "r"(far + 32u * j) : "memory");
        }
      float a[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] = 0.f;
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (s < g.parts) {
#pragma unroll
          for (int j = 0; j < 2; ++j) { a[4 * j] += q[s][j].x; a[4 * j + 1] += q[s][j].y; a[4 * j + 2] += q[s][j].z; a[4 * j + 3] += q[s][j].w; }
        }
#pragma unroll
      for (int j = 0; j < 4; ++j) {      // the even lane keeps the first piece: its lower half, and the odd lane's upper one
        const float got = __shfl_xor_sync(0xffffffffu, lane & 1 ? a[j] : a[4 + j], 1);
        if (lane & 1) a[j] = got; else a[4 + j] = got;
      }
      if (b + lane < i1) epilogue_row8(o, m0 + r, n0 + p * 8, a);
    }
    if (__syncthreads_or(lost))
      for (int i = i0 + tid; i < i1; i += THREADS) poison(o, m0 + i / pieces, n0 + i % pieces * 8, 8);
    if (g.splits > 1) {      // the others have read this CTA's partial tile (reads only: nothing to publish)
      asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*dead) {      // copies and products still on their way end before the memory they use is given back
    if (warp == MMA_WARP && leader) {
      umma_commit(drain);
      mbar_wait_bounded(drain, 0u, 1 << 14);
    }
    if (tid < g.stages && tid < (int)words[2]) {
      const int i = (int)words[2] - 1 - tid;
      mbar_wait_bounded(full + 8u * (i % g.stages), (uint32_t)((i / g.stages) & 1), 1 << 14);
    }
    if (!g.staged)
      for (int t = t0; t < tiles; t += dt) {
        const int n0 = (t / g.mt) * g.bn, m0 = o.m_begin + (t % g.mt) * TM, pieces = g.bn / 8;
        for (int i = tid; i < TM * pieces; i += THREADS) poison(o, m0 + i / pieces, n0 + i % pieces * 8, 8);
      }
  }
  __syncthreads();
  if (warp == MMA_WARP) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
}
