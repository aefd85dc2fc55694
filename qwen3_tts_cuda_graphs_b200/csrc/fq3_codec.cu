// fq3_codec.cu — kernels of the 12 Hz speech-tokenizer decoder (include/fq3_codec.h).
//
// Activations are channels-last bf16 [time, channels]; every convolution is an implicit GEMM over (tap, c_in)
// whose A rows are time-shifted views of the same buffer (no im2col), so causal padding is a bounds check.
#include <cuda.h>  // CUtensorMap (types only: the encoder is fetched with cudaGetDriverEntryPoint, nothing links against libcuda)
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <type_traits>

#include "../../include/fq3_codec.h"

typedef __nv_bfloat16 bf16;

extern "C" {
static bool device_attrs_ready();      // shared-memory limits of the kernels, once per device
}

namespace {

thread_local std::string g_err;
// launches of the whole process (several scheduler threads may run op lists at once: one per GPU) and of the calling thread alone
std::atomic<int64_t> g_launches{0};
thread_local int64_t t_launches = 0;
inline void count_launches(int64_t n) { g_launches += n; t_launches += n; }

// Programmatic dependent launch: a kernel that the host launches with launch_after may begin before the ones in front of it have ended.  It waits for their end itself before it touches
// memory (but for weights that no op of the list writes, and its own arguments), and says when the next launch may come up.  Without the launch attribute both return at once.
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// One launch ahead: with the next one let in before this wait, launches pile up on the SMs (28 layers of a prompt of 39 rows 1128 us, this way 1118; a codec window 717 and 705).
// ahead: the next one at once.  For many rows, whose launches take longer than those behind them need to come up (four layers of 1000 rows 413 and 416), and for the norm of wide rows, in
// front of a product whose weights are worth asking for early (six layers of 17 rows, 2048 wide, 373 us at once, 391 behind the wait; 1024 wide 24 - 80 rows are 0.5 - 3 % faster behind it).
__device__ __forceinline__ void grid_dep_begin(const bool ahead = false) {
  if (ahead) grid_dep_launch();
  grid_dep_wait();
  if (!ahead) grid_dep_launch();
}

__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
  const int sz = valid ? 16 : 0;  // src-size 0 => zero fill
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(sz) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)));
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

constexpr int BM = 64, BN = 64, BK = 32, PAD = 8, LDS = BK + PAD;

__device__ __forceinline__ float gelu_f(float x) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float silu_f(float x) { return x / (1.f + expf(-x)); }
__device__ __forceinline__ float gelu_tanh_f(float z) {
  return 0.5f * z * (1.f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}
// sin(x)^2, the periodic half of SnakeBeta.  x is reduced by the nearest multiple of pi / 2 (Cody and Waite: two parts, the first product exact) to
// [-pi/4, pi/4], where sin^2 = u + u^2 Q(u), u = r^2, with a cubic Q (least-maximum fit of sin^2, error 2.4e-10); behind an odd multiple it is 1 - sin^2(r).
// Within 1.1e-7 of sin^2, 1.9e-8 root mean square (the square of a correctly rounded sine: 0.9e-7 and 2.7e-8).  Beyond SIN_SQ_NEAR, where the multiple's own
// rounding leaves the fitted range, through sinf.
constexpr float SIN_SQ_NEAR = 2.5e5f;
__device__ __forceinline__ float sin_sq_near(const float x) {
  const float m = fmaf(x, 0.6366197723675814f, 12582912.f), n = m - 12582912.f;      // the multiple in m's low bits
  float r = fmaf(n, -1.5707963705062866f, x);
  r = fmaf(n, 4.371138828673793e-08f, r);
  const float u = r * r;
  float q = fmaf(u, 0.0001339026930509135f, -0.0031702169217169285f);
  q = fmaf(u, q, 0.04444332420825958f);
  q = fmaf(u, q, -0.33333322405815125f);
  const float sg = __uint_as_float(__float_as_uint(m) * 0x80000000u + 0x3f800000u);      // -1 behind an odd multiple, else 1
  const float su = sg * u;
  return fmaf(su * u, q, su) + fmaf(sg, -0.5f, 0.5f);
}
__device__ __noinline__ float sin_sq_far(const float x) {
  const float s = sinf(x);
  return s * s;
}
__device__ __forceinline__ float sin_sq(const float x) { return fabsf(x) < SIN_SQ_NEAR ? sin_sq_near(x) : sin_sq_far(x); }
// a gated unit: silu(gate) * up, or with FQ3C_GELU_TANH gelu_tanh(gate) * up
__device__ __forceinline__ float glu_f(const int flags, const float gate, const float up) {
  return (flags & FQ3C_GELU_TANH) ? gelu_tanh_f(gate) * up : silu_f(gate) * up;
}

__device__ __forceinline__ void stf_any(const fq3c_op& o, const size_t at, const float v) {
  if (o.flags & FQ3C_OUT_F32) reinterpret_cast<float*>(o.C)[at] = v;
  else reinterpret_cast<bf16*>(o.C)[at] = __float2bfloat16_rn(v);
}
// Epilogue for one (row, even col) pair of accumulators; order documented in include/fq3_codec.h / DESIGN.md §5.
__device__ __forceinline__ void epilogue_pair(const fq3c_op& o, int row, int col, float v0, float v1) {
  if (row >= o.M || col >= o.N) return;
  const bool has1 = (col + 1 < o.N);
  const int cm0 = col % o.col_mod, cm1 = (col + 1) % o.col_mod;
  if (o.flags & FQ3C_BIAS) {
    const float* b = reinterpret_cast<const float*>(o.bias);
    v0 += b[cm0];
    if (has1) v1 += b[cm1];
  }
  if (o.flags & FQ3C_RELU2) { v0 = fmaxf(v0, 0.f); v0 *= v0; v1 = fmaxf(v1, 0.f); v1 *= v1; }   // on the f32 sum: one rounding, after the square
  if (!(o.flags & FQ3C_NOROUND)) {
    v0 = bf16r(v0);
    v1 = bf16r(v1);
  }
  if (o.flags & FQ3C_SWIGLU) {  // interleaved (gate, up) columns -> one output column
    if (o.flags & FQ3C_NOROUND) {
      if (has1) stf_any(o, (size_t)row * o.ldc + (col >> 1), glu_f(o.flags, v0, v1));
      return;
    }
    const float y = bf16r(bf16r(silu_f(v0)) * v1);
    reinterpret_cast<bf16*>(o.C)[(size_t)row * o.ldc + (col >> 1)] = __float2bfloat16_rn(y);
    return;
  }
  if (o.flags & FQ3C_GELU) {
    v0 = gelu_f(v0); v1 = gelu_f(v1);
    if (!(o.flags & FQ3C_NOROUND)) { v0 = bf16r(v0); v1 = bf16r(v1); }
  }
  if (o.flags & FQ3C_SILU) { v0 = bf16r(silu_f(v0)); v1 = bf16r(silu_f(v1)); }
  if (o.flags & FQ3C_SCALE) {
    const float* s = reinterpret_cast<const float*>(o.scale);
    v0 = bf16r(v0 * s[cm0]);
    if (has1) v1 = bf16r(v1 * s[cm1]);
  }
  if (o.flags & FQ3C_RESID) {
    const bf16* r = reinterpret_cast<const bf16*>(o.res) + (size_t)row * o.ldr + col;
    v0 = bf16r(v0 + __bfloat162float(r[0]));
    if (has1) v1 = bf16r(v1 + __bfloat162float(r[1]));
  }
  if (o.flags & FQ3C_CLAMP) { v0 = fminf(fmaxf(v0, -1.f), 1.f); v1 = fminf(fmaxf(v1, -1.f), 1.f); }
  if (o.flags & FQ3C_OUT_F32) {
    float* c = reinterpret_cast<float*>(o.C) + (size_t)row * o.ldc + col;
    c[0] = v0;
    if (has1) c[1] = v1;
  } else {
    bf16* c = reinterpret_cast<bf16*>(o.C) + (size_t)row * o.ldc + col;
    c[0] = __float2bfloat16_rn(v0);
    if (has1) c[1] = __float2bfloat16_rn(v1);
  }
  if (o.flags & FQ3C_SNAKE2) {
    const float* ea = reinterpret_cast<const float*>(o.p0);
    const float* ib = reinterpret_cast<const float*>(o.p1);
    bf16* c2 = reinterpret_cast<bf16*>(o.C2) + (size_t)row * o.ldc + col;
    c2[0] = __float2bfloat16_rn(v0 + ib[cm0] * sin_sq(v0 * ea[cm0]));
    if (has1) c2[1] = __float2bfloat16_rn(v1 + ib[cm1] * sin_sq(v1 * ea[cm1]));
  }
}

// Epilogue for eight consecutive columns of one row (the tcgen05 path: a thread owns a row of the accumulator, so it
// must move whole 16-byte pieces or every store is a partial sector).  Same arithmetic and order as epilogue_pair.
__device__ __forceinline__ void epilogue_row8(const fq3c_op& o, int row, int col, const float (&acc)[8]) {
  // the sequence models' products: unrounded f32 rows as two 16-byte stores (one whole sector), or an activation taken on the f32 sum
  // and rounded once
  if ((o.flags & FQ3C_NOROUND) && !(o.flags & ~(FQ3C_OUT_F32 | FQ3C_NOROUND | FQ3C_BIAS | FQ3C_GELU)) && col + 8 <= o.N &&
      (o.ldc & ((o.flags & FQ3C_OUT_F32) ? 3 : 7)) == 0 && o.col_mod == o.N && !(reinterpret_cast<uintptr_t>(o.C) & 15)) {
    if (row >= o.M) return;
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = acc[j];
    if (o.flags & FQ3C_BIAS) {
      const float* b = reinterpret_cast<const float*>(o.bias) + col;
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] += b[j];
    }
    if (o.flags & FQ3C_GELU) {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = gelu_f(v[j]);
    }
    if (!(o.flags & FQ3C_OUT_F32)) {
      uint32_t w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
        w[j] = *reinterpret_cast<const uint32_t*>(&h);
      }
      *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(o.C) + (size_t)row * o.ldc + col) = make_uint4(w[0], w[1], w[2], w[3]);
      return;
    }
    float4* c = reinterpret_cast<float4*>(reinterpret_cast<float*>(o.C) + (size_t)row * o.ldc + col);
    c[0] = make_float4(v[0], v[1], v[2], v[3]);
    c[1] = make_float4(v[4], v[5], v[6], v[7]);
    return;
  }
  // a gated unit on the unrounded sums: four outputs, one 8-byte store
  if ((o.flags & FQ3C_SWIGLU) && (o.flags & FQ3C_NOROUND) && !(o.flags & ~(FQ3C_SWIGLU | FQ3C_NOROUND | FQ3C_GELU_TANH)) && col + 8 <= o.N &&
      (o.ldc & 3) == 0 && !(reinterpret_cast<uintptr_t>(o.C) & 7)) {
    if (row >= o.M) return;
    float v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = glu_f(o.flags, acc[2 * j], acc[2 * j + 1]);
    const __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
    *reinterpret_cast<uint2*>(reinterpret_cast<bf16*>(o.C) + (size_t)row * o.ldc + (col >> 1)) =
        make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    return;
  }
  // the same on rounded sums (the talker's and the codec's feed-forward)
  if ((o.flags & FQ3C_SWIGLU) && !(o.flags & ~FQ3C_SWIGLU) && col + 8 <= o.N && (o.ldc & 3) == 0 && !(reinterpret_cast<uintptr_t>(o.C) & 7)) {
    if (row >= o.M) return;
    float v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = bf16r(silu_f(bf16r(acc[2 * j]))) * bf16r(acc[2 * j + 1]);
    const __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
    *reinterpret_cast<uint2*>(reinterpret_cast<bf16*>(o.C) + (size_t)row * o.ldc + (col >> 1)) =
        make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    return;
  }
  const bool vec = (col + 8 <= o.N) && !(o.flags & (FQ3C_SWIGLU | FQ3C_OUT_F32)) && ((o.ldc & 7) == 0) &&
                   (!(o.flags & FQ3C_RESID) || (o.ldr & 7) == 0);
  if (!vec) {
#pragma unroll
    for (int j = 0; j < 4; ++j) epilogue_pair(o, row, col + 2 * j, acc[2 * j], acc[2 * j + 1]);
    return;
  }
  if (row >= o.M) return;
  float v[8];
  int cm[8];
  {
    int c0 = col % o.col_mod;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      cm[j] = c0;
      if (++c0 == o.col_mod) c0 = 0;
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = acc[j];
  if (o.flags & FQ3C_BIAS) {
    const float* b = reinterpret_cast<const float*>(o.bias);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] += b[cm[j]];
  }
  if (o.flags & FQ3C_RELU2) {
#pragma unroll
    for (int j = 0; j < 8; ++j) { v[j] = fmaxf(v[j], 0.f); v[j] *= v[j]; }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = bf16r(v[j]);
  if (o.flags & FQ3C_GELU) {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = bf16r(gelu_f(v[j]));
  }
  if (o.flags & FQ3C_SILU) {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = bf16r(silu_f(v[j]));
  }
  if (o.flags & FQ3C_SCALE) {
    const float* sc = reinterpret_cast<const float*>(o.scale);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = bf16r(v[j] * sc[cm[j]]);
  }
  if (o.flags & FQ3C_RESID) {
    const uint4 rr = *reinterpret_cast<const uint4*>(reinterpret_cast<const bf16*>(o.res) + (size_t)row * o.ldr + col);
    const uint32_t rw[4] = {rr.x, rr.y, rr.z, rr.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[2 * j] = bf16r(v[2 * j] + __uint_as_float(rw[j] << 16));
      v[2 * j + 1] = bf16r(v[2 * j + 1] + __uint_as_float(rw[j] & 0xffff0000u));
    }
  }
  if (o.flags & FQ3C_CLAMP) {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = fminf(fmaxf(v[j], -1.f), 1.f);
  }
  {
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
      w[j] = *reinterpret_cast<const uint32_t*>(&h);
    }
    *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(o.C) + (size_t)row * o.ldc + col) = make_uint4(w[0], w[1], w[2], w[3]);
  }
  if (o.flags & FQ3C_SNAKE2) {
    const float* ea = reinterpret_cast<const float*>(o.p0);
    const float* ib = reinterpret_cast<const float*>(o.p1);
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * j] + ib[cm[2 * j]] * sin_sq(v[2 * j] * ea[cm[2 * j]]),
                                                     v[2 * j + 1] + ib[cm[2 * j + 1]] * sin_sq(v[2 * j + 1] * ea[cm[2 * j + 1]]));
      w[j] = *reinterpret_cast<const uint32_t*>(&h);
    }
    *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(o.C2) + (size_t)row * o.ldc + col) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// Implicit-GEMM convolution / linear layer on the bf16 tensor cores (mma.sync m16n8k16, fp32 accumulate).
__global__ void __launch_bounds__(128) fq3c_gemm_kernel(const fq3c_op o) {
  __shared__ __align__(16) bf16 As[2][BM][LDS];
  __shared__ __align__(16) bf16 Bs[2][BN][LDS];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wm = warp >> 1, wn = warp & 1;
  const int m0 = o.m_begin + blockIdx.y * BM, n0 = blockIdx.x * BN;
  const bf16* A = reinterpret_cast<const bf16*>(o.A);
  const bf16* B = reinterpret_cast<const bf16*>(o.B);
  const int KT = (o.K + BK - 1) / BK;

  auto load_stage = [&](int st, int kt) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int ch = tid + i * 128;  // 0..255
      const int r = ch >> 2, c = ch & 3;
      const int k0 = kt * BK + c * 8;
      // A: time-shifted row of the activation buffer
      {
        const int m = m0 + r;
        const int tap = k0 / o.cin, ci = k0 - tap * o.cin;
        const int srow = m + (tap < 8 ? o.tap_off[tap] : 0);
        const bool ok = (m < o.M) && (k0 < o.K) && (srow >= 0) && (srow < o.a_rows);
        const bf16* src = ok ? (A + (size_t)srow * o.lda + ci) : A;
        cp_async16(&As[st][r][c * 8], src, ok);
      }
      {
        const int n = n0 + r;
        const bool ok = (n < o.N) && (k0 < o.K);
        const bf16* src = ok ? (B + (size_t)n * o.K + k0) : B;
        cp_async16(&Bs[st][r][c * 8], src, ok);
      }
    }
    cp_async_commit();
  };

  float acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[i][j][k] = 0.f;

  load_stage(0, 0);
  for (int kt = 0; kt < KT; ++kt) {
    const int st = kt & 1;
    if (kt + 1 < KT) { load_stage(st ^ 1, kt + 1); cp_async_wait<1>(); } else { cp_async_wait<0>(); }
    __syncthreads();
#pragma unroll
    for (int ks = 0; ks < BK; ks += 16) {
      uint32_t af[2][4], bfr[4][2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int row = wm * 32 + i * 16 + (lane & 15);
        const int col = ks + (lane >> 4) * 8;
        ldmatrix_x4(af[i], &As[st][row][col]);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {  // each x4 covers two n8 tiles
        uint32_t r[4];
        const int row = wn * 32 + j * 16 + (lane & 7) + ((lane >> 4) << 3);
        const int col = ks + ((lane >> 3) & 1) * 8;
        ldmatrix_x4(r, &Bs[st][row][col]);
        bfr[2 * j][0] = r[0]; bfr[2 * j][1] = r[1]; bfr[2 * j + 1][0] = r[2]; bfr[2 * j + 1][1] = r[3];
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) mma16816(acc[i][j], af[i], bfr[j][0], bfr[j][1]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int row = m0 + wm * 32 + i * 16 + (lane >> 2);
      const int col = n0 + wn * 32 + j * 8 + (lane & 3) * 2;
      epilogue_pair(o, row, col, acc[i][j][0], acc[i][j][1]);
      epilogue_pair(o, row + 8, col, acc[i][j][2], acc[i][j][3]);
    }
}

// =================================================================================================
// tcgen05 path of the implicit GEMM (sm_100a): 128 x BN x 64 tiles, accumulator in tensor memory.
//
// A tile is K-major with the 128-byte swizzle the tensor core expects (the layout a TMA box with SWIZZLE_128B writes):
// row r of the tile is one 128-byte line (64 bf16), its 16-byte chunk c lives at r * 128 + ((c ^ (r & 7)) << 4).  The
// tiles are filled with cp.async so that the time-shifted (tap) rows of the implicit GEMM and the zero padding stay a
// per-chunk address computation; eight lanes cover one 128-byte line of a row, so global reads are coalesced and the
// swizzle makes the shared-memory writes conflict-free.  One thread issues tcgen05.mma (4 x k16 per stage) and commits to
// the stage's mbarrier; the epilogue reads the accumulator with tcgen05.ld (one TMEM lane = one output row per thread).
// =================================================================================================
constexpr int TM = 128, TK = 64, TSTAGES = 6;
constexpr int TLOADERS = 256;                 // warps 0-3 fill A, warps 4-7 fill B; warp 8 issues the MMAs
constexpr int TTHREADS = TLOADERS + 32;
constexpr int TMAXN = 128;
constexpr int T_A_BYTES = TM * TK * 2;        // 16 KB
constexpr int T_B_BYTES = TMAXN * TK * 2;     // 16 KB
constexpr int t_smem(int stages) { return stages * (T_A_BYTES + T_B_BYTES) + 1024 /*alignment*/ + 256 /*barriers + tmem pointer*/; }
constexpr int T_SMEM = t_smem(TSTAGES);

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ void mbar_wait(uint32_t bar, uint32_t parity) {
  while (!mbar_try_wait(bar, parity)) __nanosleep(20);
}
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr) {
  // K-major, SWIZZLE_128B: start address >> 4 | LBO (unused for swizzled K-major) = 1 | SBO = 1024 B (8 rows) | version 1 | layout 2
  return (uint64_t)((smem_addr & 0x3ffffu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
         ((uint64_t)2 << 61);
}

// Warp-specialised: the loader warps run up to TSTAGES k-blocks ahead of the tensor core (full / empty mbarriers per stage,
// cp.async completion counted straight into the full barrier), one thread issues the MMAs, all eight loader warps drain
// the accumulator.  No block-wide barrier inside the k loop.
// Split-K (splits > 1, short-and-wide problems that would leave most SMs idle): blockIdx.z takes a contiguous range of
// k-blocks and stores its raw fp32 tile into the workspace [split][M][Nw]; fq3c_splitk_reduce_kernel adds the splits in
// order and applies the fused epilogue.
// This kernel is left for c_in = 8 modulo 16 over several taps, where a 16-column MMA step would straddle two taps of a tensor map's row;
// everything else runs on fq3c_gemm_persist_kernel (fq3_gemm.cuh).
template <int MINB>  // CTAs per SM the register budget is planned for: 2 with three stages, 1 with six
__global__ void __launch_bounds__(TTHREADS, MINB) fq3c_gemm_tc5_kernel(const fq3c_op o, const int BN, const int splits, const int Nw, const int NST) {
  extern __shared__ unsigned char tsmem_raw[];
  const uint32_t raw = smem_u32(tsmem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;  // swizzle atoms are 1024-byte aligned
  unsigned char* gbase = tsmem_raw + (base - raw);
  const uint32_t a_smem = base, b_smem = base + NST * T_A_BYTES;
  const uint32_t bars = base + NST * (T_A_BYTES + T_B_BYTES);  // full[NST] | empty[NST] | done | tmem base address
  const uint32_t full = bars, empty = bars + 8u * NST, done = bars + 16u * NST;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gbase + NST * (T_A_BYTES + T_B_BYTES) + 16 * NST + 16);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = o.m_begin + blockIdx.y * TM, n0 = blockIdx.x * BN;
  const bf16* A = reinterpret_cast<const bf16*>(o.A);
  const bf16* B = reinterpret_cast<const bf16*>(o.B);
  const int KT_all = (o.K + TK - 1) / TK;
  const int kt_begin = (int)(((long)blockIdx.z * KT_all) / splits), kt_end = (int)(((long)(blockIdx.z + 1) * KT_all) / splits);
  const int KT = kt_end - kt_begin;  // k-blocks of this CTA; `it` below counts them from 0

  if (tid == 0) {
    for (int s = 0; s < NST; ++s) {
      mbar_init(full + 8u * s, TLOADERS);
      mbar_init(empty + 8u * s, 1);
    }
    mbar_init(done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMAXN) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  if (warp == 8) {
    // ------------------------------ MMA issuer ------------------------------
    if (lane == 0) {
      // instruction descriptor: D = F32, A = B = BF16, both K-major, N = BN, M = 128
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);
      for (int kt = 0; kt < KT; ++kt) {
        const int st = kt % NST;
        mbar_wait(full + 8u * st, (uint32_t)((kt / NST) & 1));
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // cp.async (generic proxy) writes -> tensor core (async proxy) reads
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a0 = a_smem + (uint32_t)st * T_A_BYTES, b0 = b_smem + (uint32_t)st * T_B_BYTES;
#pragma unroll
        for (int kk = 0; kk < TK / 16; ++kk) {
          const uint64_t da = umma_desc_sw128(a0 + kk * 32), db = umma_desc_sw128(b0 + kk * 32);
          const uint32_t acc = (kt > 0 || kk > 0) ? 1u : 0u;
          asm volatile(
              "{\n\t.reg .pred p;\n\t"
              "setp.ne.b32 p, %4, 0;\n\t"
              "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
              ::"r"(tmem), "l"(da), "l"(db), "r"(idesc), "r"(acc)
              : "memory");
        }
        // frees the stage once its MMAs have read it (implies tcgen05.fence::before_thread_sync)
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(empty + 8u * st) : "memory");
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(done) : "memory");
    }
  } else {
    // ------------------------------ loaders ------------------------------
    // warps 0-3: A rows r0 + 16 i (i < 8), chunk c; warps 4-7: B rows likewise.  Eight lanes cover one 128-byte line of a row.
    const int lt = tid & 127, c = lt & 7, r0 = lt >> 3;
    const bool is_a = warp < 4;
    for (int kt = 0; kt < KT; ++kt) {
      const int st = kt % NST;
      if (kt >= NST) {  // one lane per warp polls: 256 spinning threads would swamp the shared-memory pipe the copies need
        if (lane == 0) mbar_wait(empty + 8u * st, (uint32_t)(((kt / NST) - 1) & 1));
        __syncwarp();
      }
      const int k0 = (kt_begin + kt) * TK + c * 8;
      const bool kok = k0 < o.K;
      if (is_a) {
        const int tap = k0 / o.cin, ci = k0 - tap * o.cin;
        const int toff = (tap < 8) ? o.tap_off[tap] : 0;
        const uint32_t sbase = a_smem + (uint32_t)st * T_A_BYTES;
#pragma unroll
        for (int i = 0; i < TM / 16; ++i) {
          const int r = r0 + i * 16;
          const int m = m0 + r;
          const int srow = m + toff;
          const bool ok = kok && (m < o.M) && (srow >= 0) && (srow < o.a_rows);
          const bf16* src = ok ? (A + (size_t)srow * o.lda + ci) : A;
          const uint32_t dst = sbase + (uint32_t)r * 128u + (uint32_t)((c ^ (r & 7)) << 4);
          const int sz = ok ? 16 : 0;
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(sz) : "memory");
        }
      } else {
        const uint32_t sbase = b_smem + (uint32_t)st * T_B_BYTES;
        for (int r = r0; r < BN; r += 16) {
          const int n = n0 + r;
          const bool ok = kok && (n < o.N);
          const bf16* src = ok ? (B + (size_t)n * o.K + k0) : B;
          const uint32_t dst = sbase + (uint32_t)r * 128u + (uint32_t)((c ^ (r & 7)) << 4);
          const int sz = ok ? 16 : 0;
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(sz) : "memory");
        }
      }
      // counted as one arrival on the stage's full barrier when this thread's copies have landed
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(full + 8u * st) : "memory");
    }
    // ------------------------------ epilogue ------------------------------
    if (lane == 0) mbar_wait(done, 0u);
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // warp w reads TMEM lanes 32 * (w & 3) .. +31 (= output rows); warps 0-3 take the first half of the columns, 4-7 the second
    const int row = m0 + (warp & 3) * 32 + lane;
    const int chunks = (BN + 31) / 32;  // 32-column chunks in the tile
    const int per = (chunks + 1) / 2;
    const int c_begin = (warp >> 2) * per, c_end = min(chunks, c_begin + per);
    for (int cc = c_begin; cc < c_end; ++cc) {
      uint32_t v[32];
      const uint32_t taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(cc * 32);
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, "
          "%20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
          : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
            "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]),
            "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]),
            "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
          : "r"(taddr)
          : "memory");
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (cc * 32 + 8 * j < BN) {
          float a8[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) a8[q] = __uint_as_float(v[8 * j + q]);
          const int col = n0 + cc * 32 + 8 * j;
          if (splits > 1) {
            if (row < o.M && col < o.N) {
              float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(o.ws) + ((size_t)blockIdx.z * o.M + row) * Nw + col);
              dst[0] = make_float4(a8[0], a8[1], a8[2], a8[3]);
              dst[1] = make_float4(a8[4], a8[5], a8[6], a8[7]);
            }
          } else {
            epilogue_row8(o, row, col, a8);
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 8) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMAXN) : "memory");
}

// RVQ dequantiser front half: gather + sum codebook rows. C[m, 0:dim] = sum of the first i0 groups, C[m, dim:2dim] = rest.
// second half of a split-K GEMM: a thread owns eight consecutive columns of a row, adds the splits in order (deterministic)
// and runs the same fused epilogue the single-pass kernel would have run.  (Only behind fq3c_gemm_tc5_kernel: the persistent kernel sums in its cluster.)
__global__ void __launch_bounds__(256) fq3c_splitk_reduce_kernel(const fq3c_op o, const int splits, const int Nw) {
  const int groups = Nw >> 3;
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long)(o.M - o.m_begin) * groups) return;
  const int r_rel = (int)(idx / groups);
  const int row = o.m_begin + r_rel, col = (int)(idx - (long)r_rel * groups) * 8;
  float a8[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const float* ws = reinterpret_cast<const float*>(o.ws);
  for (int z = 0; z < splits; ++z) {
    const float4* src = reinterpret_cast<const float4*>(ws + ((size_t)z * o.M + row) * Nw + col);
    const float4 v0 = src[0], v1 = src[1];
    a8[0] += v0.x; a8[1] += v0.y; a8[2] += v0.z; a8[3] += v0.w;
    a8[4] += v1.x; a8[5] += v1.y; a8[6] += v1.z; a8[7] += v1.w;
  }
  epilogue_row8(o, row, col, a8);
}

__global__ void fq3c_rvq_kernel(const fq3c_op o) {
  grid_dep_begin();
  const long long* codes = reinterpret_cast<const long long*>(o.A);
  const bf16* cb = reinterpret_cast<const bf16*>(o.B);
  const int Q = o.i1, nsem = o.i0, dim = o.i2, cbsize = o.K;
  bf16* C = reinterpret_cast<bf16*>(o.C);
  const int m = blockIdx.x;
  for (int d = threadIdx.x; d < dim; d += blockDim.x) {
    float a = 0.f, b = 0.f;
    for (int g = 0; g < Q; ++g) {
      long long c = codes[(size_t)m * Q + g];
      c = c < 0 ? 0 : (c >= cbsize ? cbsize - 1 : c);
      const float v = __bfloat162float(cb[((size_t)g * cbsize + c) * dim + d]);
      if (g < nsem) a += v; else b += v;
    }
    C[(size_t)m * o.ldc + d] = __float2bfloat16_rn(a);
    C[(size_t)m * o.ldc + dim + d] = __float2bfloat16_rn(b);
  }
}

__device__ __forceinline__ float block_sum(float v, float* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float t = 0.f;
  for (int i = 0; i < nw; ++i) t += red[i];
  return t;
}

// RMSNorm of a row by a warp, eight entries a lane and load, with the sums of fq3c_rmsnorm_kernel's 256 threads in their order: lane l's pieces 8 l + 256 c .. + 7 are the
// entries of its threads 8 l .. 8 l + 7, and thread t of a warp of the block is entry t & 7 of lane t >> 3.  sq8 adds a piece to those eight sums; rms_of adds them as
// block_sum does (threads 16, 8, 4, 2, 1 apart, then the eight warps one by one) and gives the reciprocal root of the mean square.
__device__ __forceinline__ void sq8(const uint4 x, float (&ss)[8]) {
  const uint32_t u[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float a = __uint_as_float(u[q] << 16), b = __uint_as_float(u[q] & 0xffff0000u);
    ss[2 * q] = fmaf(a, a, ss[2 * q]);
    ss[2 * q + 1] = fmaf(b, b, ss[2 * q + 1]);
  }
}
__device__ __forceinline__ float rms_of(const float (&ss)[8], const int lane, const int N, const float eps) {
  const bool b4 = lane & 2, b3 = lane & 1;      // bits 4 and 3 of the lane's threads; each meeting keeps half of the entries
  float a[4], b[2];
#pragma unroll
  for (int i = 0; i < 4; ++i) a[i] = (b4 ? ss[i + 4] : ss[i]) + __shfl_xor_sync(0xffffffffu, b4 ? ss[i] : ss[i + 4], 2);      // 16 apart
#pragma unroll
  for (int i = 0; i < 2; ++i) b[i] = (b3 ? a[i + 2] : a[i]) + __shfl_xor_sync(0xffffffffu, b3 ? a[i] : a[i + 2], 1);          // 8 apart
  float t = (b4 ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, b4 ? b[0] : b[1], 2);      // entries 4 apart, between the lanes that kept them
  t += __shfl_xor_sync(0xffffffffu, t, 1);      // 2 apart
  t += __shfl_xor_sync(0xffffffffu, t, 2);      // 1 apart
  float sum = 0.f;
#pragma unroll
  for (int w = 0; w < 8; ++w) sum += __shfl_sync(0xffffffffu, t, 4 * w);
  return rsqrtf(sum / N + eps);
}
__device__ __forceinline__ uint4 norm8(const uint4 x, const float rs, const float* w) {
  const float4 a = *reinterpret_cast<const float4*>(w), b = *(reinterpret_cast<const float4*>(w) + 1);
  const float wv[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  const uint32_t u[4] = {x.x, x.y, x.z, x.w};
  uint32_t r[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(bf16r(__uint_as_float(u[q] << 16) * rs) * wv[2 * q], bf16r(__uint_as_float(u[q] & 0xffff0000u) * rs) * wv[2 * q + 1]);
    r[q] = *reinterpret_cast<const uint32_t*>(&h);
  }
  return make_uint4(r[0], r[1], r[2], r[3]);
}
// rows of whole 16-byte pieces
bool norm_vec_ok(const void* x, const void* y, const void* w, const int N, const int ldx, const int ldy) {
  return ((N | ldx | ldy) & 7) == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
}
// FQ3C_RMSNORM and the norm behind a product (fq3c_op.norm_out), the same bits either way.  Bound by latency for few rows (a launch, a trip to L2), by its bytes for
// many.  A block per row with two-byte loads and block-wide sums takes 2.6 us for 39 rows of 1024 and 5.5 for 1900, this 2.2 and 3.9.  (Normed by the product behind
// it instead, in each of its CTAs: a layer of a 39-row prompt 38.7 -> 43.3 us.)
constexpr int RN_WARPS = 4;
__global__ void __launch_bounds__(RN_WARPS * 32) fq3c_rownorm_vec_kernel(const bf16* x, const int ldx, bf16* y, const int ldy, const float* w, const float eps, const int row0, const int rows,
                                                                         const int N) {
  grid_dep_begin(rows > 512 || N > 1024);
  const int row = blockIdx.x * RN_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= rows) return;
  const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)(row0 + row) * ldx);
  uint4* yr = reinterpret_cast<uint4*>(y + (size_t)(row0 + row) * ldy);
  constexpr int C = 4;      // pieces of a lane kept from the sum to the norm; longer rows are read again
  uint4 v[C];
  float ss[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int c = 0; c < C; ++c)
    if (lane + 32 * c < N / 8) v[c] = xr[lane + 32 * c];
#pragma unroll
  for (int c = 0; c < C; ++c)
    if (lane + 32 * c < N / 8) sq8(v[c], ss);
  for (int p = lane + 32 * C; p < N / 8; p += 32) sq8(xr[p], ss);
  const float rs = rms_of(ss, lane, N, eps);
#pragma unroll
  for (int c = 0; c < C; ++c)
    if (lane + 32 * c < N / 8) yr[lane + 32 * c] = norm8(v[c], rs, w + 8 * (lane + 32 * c));
  for (int p = lane + 32 * C; p < N / 8; p += 32) yr[p] = norm8(xr[p], rs, w + 8 * p);
}
// rows without whole pieces
__global__ void fq3c_rmsnorm_kernel(const fq3c_op o) {
  grid_dep_begin();
  __shared__ float red[32];
  const bf16* x = reinterpret_cast<const bf16*>(o.A) + (size_t)blockIdx.x * o.lda;
  bf16* y = reinterpret_cast<bf16*>(o.C) + (size_t)blockIdx.x * o.ldc;
  const float* w = reinterpret_cast<const float*>(o.scale);
  float ss = 0.f;
  for (int c = threadIdx.x; c < o.N; c += blockDim.x) { const float v = __bfloat162float(x[c]); ss += v * v; }
  ss = block_sum(ss, red);
  const float rs = rsqrtf(ss / o.N + o.f0);
  for (int c = threadIdx.x; c < o.N; c += blockDim.x)
    y[c] = __float2bfloat16_rn(bf16r(bf16r(__bfloat162float(x[c]) * rs) * w[c]));
}

// RMSNorm of the rows a GEMM just finished in rows without whole pieces, with the arithmetic of fq3c_rmsnorm_kernel: same column-strided
// partial sums, same block tree, same rounding points — the fused form changes the launch count, not a bit of the result.
__device__ __forceinline__ void row_rmsnorm(const fq3c_op& o, int row, float* red) {
  const bf16* x = reinterpret_cast<const bf16*>(o.C) + (size_t)row * o.ldc;
  bf16* y = reinterpret_cast<bf16*>(o.norm_out) + (size_t)row * o.norm_ld;
  const float* w = reinterpret_cast<const float*>(o.norm_w);
  float ss = 0.f;
  for (int c = threadIdx.x; c < o.N; c += blockDim.x) { const float v = __bfloat162float(x[c]); ss += v * v; }
  ss = block_sum(ss, red);
  const float rs = rsqrtf(ss / o.N + o.norm_eps);
  for (int c = threadIdx.x; c < o.N; c += blockDim.x)
    y[c] = __float2bfloat16_rn(bf16r(bf16r(__bfloat162float(x[c]) * rs) * w[c]));
}
__global__ void __launch_bounds__(256) fq3c_rownorm_kernel(const fq3c_op o) {
  grid_dep_begin();
  __shared__ float red[32];
  row_rmsnorm(o, o.m_begin + blockIdx.x, red);
}
// split-K reduction + epilogue + RMSNorm, one CTA per output row: the row's eight-column groups are reduced and written by
// their threads, then the whole CTA reads the finished row back (it is in L1 / L2) for the norm
__global__ void __launch_bounds__(256) fq3c_splitk_reduce_norm_kernel(const fq3c_op o, const int splits, const int Nw) {
  __shared__ float red[32];
  const int row = o.m_begin + blockIdx.x;
  const float* ws = reinterpret_cast<const float*>(o.ws);
  for (int col = threadIdx.x * 8; col < Nw; col += blockDim.x * 8) {
    float a8[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int z = 0; z < splits; ++z) {
      const float4* src = reinterpret_cast<const float4*>(ws + ((size_t)z * o.M + row) * Nw + col);
      const float4 v0 = src[0], v1 = src[1];
      a8[0] += v0.x; a8[1] += v0.y; a8[2] += v0.z; a8[3] += v0.w;
      a8[4] += v1.x; a8[5] += v1.y; a8[6] += v1.z; a8[7] += v1.w;
    }
    epilogue_row8(o, row, col, a8);
  }
  __syncthreads();  // the row's global writes are visible to the whole block behind the barrier
  row_rmsnorm(o, row, red);
}

__global__ void fq3c_layernorm_kernel(const fq3c_op o) {
  grid_dep_begin();
  __shared__ float red[32];
  const bf16* x = reinterpret_cast<const bf16*>(o.A) + (size_t)blockIdx.x * o.lda;
  bf16* y = reinterpret_cast<bf16*>(o.C) + (size_t)blockIdx.x * o.ldc;
  const float* w = reinterpret_cast<const float*>(o.scale);
  const float* b = reinterpret_cast<const float*>(o.bias);
  float s = 0.f;
  for (int c = threadIdx.x; c < o.N; c += blockDim.x) s += __bfloat162float(x[c]);
  const float mean = block_sum(s, red) / o.N;
  float v = 0.f;
  for (int c = threadIdx.x; c < o.N; c += blockDim.x) { const float d = __bfloat162float(x[c]) - mean; v += d * d; }
  const float rs = rsqrtf(block_sum(v, red) / o.N + o.f0);
  for (int c = threadIdx.x; c < o.N; c += blockDim.x)
    y[c] = __float2bfloat16_rn((__bfloat162float(x[c]) - mean) * rs * w[c] + b[c]);
}

// RoPE in place on q and k inside the fused qkv buffer (HF rotate_half convention, bf16 rounding per product).
__global__ void fq3c_rope_kernel(const fq3c_op o) {
  grid_dep_begin();
  const int t = blockIdx.x, nheads = o.i0, d = o.i1, col0 = o.i2, half = d / 2;
  const int pos = t + (o.p0 ? *reinterpret_cast<const int*>(o.p0) : 0);
  bf16* row = reinterpret_cast<bf16*>(const_cast<void*>(o.A)) + (size_t)t * o.lda + col0;
  for (int idx = threadIdx.x; idx < nheads * half; idx += blockDim.x) {
    const int h = idx / half, i = idx - h * half;
    const float inv = powf(o.f0, -2.0f * i / d);
    const float ang = (float)pos * inv;
    const float c = bf16r(cosf(ang)), s = bf16r(sinf(ang));
    bf16* p = row + h * d;
    const float a = __bfloat162float(p[i]), b = __bfloat162float(p[i + half]);
    p[i] = __float2bfloat16_rn(bf16r(a * c) + bf16r(-b * s));
    p[i + half] = __float2bfloat16_rn(bf16r(b * c) + bf16r(a * s));
  }
}

// Sliding-window causal attention, one warp per (query, head); head_dim in {32, 64, 128}: a lane owns d/32 contiguous
// dims (one 2/4/8-byte load per K and V row), four keys are scored per step so their shuffle reductions overlap; the
// online-softmax updates are applied key by key in order.
template <int PER>
__device__ __forceinline__ void attn_load(const bf16* p, float (&v)[4]) {
  if (PER == 4) {
    const uint2 r = *reinterpret_cast<const uint2*>(p);
    v[0] = __uint_as_float(r.x << 16); v[1] = __uint_as_float(r.x & 0xffff0000u);
    v[2] = __uint_as_float(r.y << 16); v[3] = __uint_as_float(r.y & 0xffff0000u);
  } else if (PER == 2) {
    const uint32_t r = *reinterpret_cast<const uint32_t*>(p);
    v[0] = __uint_as_float(r << 16); v[1] = __uint_as_float(r & 0xffff0000u); v[2] = 0.f; v[3] = 0.f;
  } else {
    v[0] = __bfloat162float(p[0]); v[1] = 0.f; v[2] = 0.f; v[3] = 0.f;
  }
}
// A key's share p v joins a sum that shrinks by corr.  The product is rounded before the sum, in every kernel that adds key by key: their results are the same bits.
__device__ __forceinline__ float attn_add(const float acc, const float corr, const float p, const float v) { return fmaf(acc, corr, __fmul_rn(p, v)); }
template <int PER>
__device__ __forceinline__ void attn_warp(const fq3c_op& o, int t_out, int h, int lane) {
  const int nh = o.i0, nkv = o.i1, d = o.i2, win = o.K;
  const int kvh = h / (nh / nkv);
  const bf16* base = reinterpret_cast<const bf16*>(o.A);
  const int qoff = h * d + lane * PER, koff = nh * d + kvh * d + lane * PER, voff = nh * d + nkv * d + kvh * d + lane * PER;
  float q[4], acc[4] = {0.f, 0.f, 0.f, 0.f};
  const int hist = o.taps, t = t_out + hist;  // stateful decode: `hist` rows of earlier chunks sit in front of the query rows
  const int first = o.p0 ? hist - min(*reinterpret_cast<const int*>(o.p0), hist) : 0;
  attn_load<PER>(base + (size_t)t * o.lda + qoff, q);
  const float scale = rsqrtf((float)d);
  float m = -INFINITY, l = 0.f;
  const int j0 = max(first, t - win + 1);
  for (int jb = j0; jb <= t; jb += 4) {
    float s[4], v[4][4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int j = min(jb + u, t);
      float k[4];
      attn_load<PER>(base + (size_t)j * o.lda + koff, k);
      attn_load<PER>(base + (size_t)j * o.lda + voff, v[u]);
      s[u] = fmaf(q[0], k[0], __fmul_rn(q[1], k[1]));
      if (PER == 4) s[u] = fmaf(q[3], k[3], fmaf(q[2], k[2], s[u]));
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
      for (int u = 0; u < 4; ++u) s[u] += __shfl_xor_sync(0xffffffffu, s[u], off);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (jb + u <= t) {
        const float su = bf16r(bf16r(s[u]) * scale);
        const float mn = fmaxf(m, su), corr = expf(m - mn), p = expf(su - mn);
        l = fmaf(l, corr, p);
#pragma unroll
        for (int i = 0; i < PER; ++i) acc[i] = attn_add(acc[i], corr, p, v[u][i]);
        m = mn;
      }
    }
  }
  bf16* out = reinterpret_cast<bf16*>(o.C) + (size_t)t_out * o.ldc + h * d + lane * PER;
#pragma unroll
  for (int i = 0; i < PER; ++i) out[i] = __float2bfloat16_rn(acc[i] / l);
}
// any head_dim <= 128 (lane owns dims lane, lane + 32, ...): the small test configurations
__device__ __forceinline__ void attn_warp_generic(const fq3c_op& o, int t_out, int h, int lane) {
  const int nh = o.i0, nkv = o.i1, d = o.i2, win = o.K;
  const int kvh = h / (nh / nkv);
  const bf16* base = reinterpret_cast<const bf16*>(o.A);
  const int qoff = h * d, koff = nh * d + kvh * d, voff = nh * d + nkv * d + kvh * d;
  const int hist = o.taps, t = t_out + hist;
  const int first = o.p0 ? hist - min(*reinterpret_cast<const int*>(o.p0), hist) : 0;
  const int per = (d + 31) / 32;  // <= 4
  float q[4], acc[4] = {0.f, 0.f, 0.f, 0.f};
  for (int i = 0; i < per; ++i) {
    const int c = lane + i * 32;
    q[i] = c < d ? __bfloat162float(base[(size_t)t * o.lda + qoff + c]) : 0.f;
  }
  const float scale = rsqrtf((float)d);
  float m = -INFINITY, l = 0.f;
  const int j0 = max(first, t - win + 1);
  for (int j = j0; j <= t; ++j) {
    float s = 0.f;
    for (int i = 0; i < per; ++i) {
      const int c = lane + i * 32;
      if (c < d) s += q[i] * __bfloat162float(base[(size_t)j * o.lda + koff + c]);
    }
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    s = bf16r(bf16r(s) * scale);
    const float mn = fmaxf(m, s), corr = expf(m - mn), p = expf(s - mn);
    l = l * corr + p;
    for (int i = 0; i < per; ++i) {
      const int c = lane + i * 32;
      const float v = c < d ? __bfloat162float(base[(size_t)j * o.lda + voff + c]) : 0.f;
      acc[i] = acc[i] * corr + p * v;
    }
    m = mn;
  }
  bf16* out = reinterpret_cast<bf16*>(o.C) + (size_t)t_out * o.ldc + h * d;
  for (int i = 0; i < per; ++i) {
    const int c = lane + i * 32;
    if (c < d) out[c] = __float2bfloat16_rn(acc[i] / l);
  }
}
__global__ void fq3c_attn_kernel(const fq3c_op o) {
  grid_dep_begin();
  const int nh = o.i0, T = o.M;
  const int wpb = blockDim.x >> 5;
  const int gw = blockIdx.x * wpb + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (gw >= T * nh) return;
  const int t = gw / nh, h = gw - t * nh;
  const bool aligned = ((o.lda * 2) % 8 == 0) && ((o.ldc * 2) % 8 == 0);
  if (o.i2 == 128 && aligned) attn_warp<4>(o, t, h, lane);
  else if (o.i2 == 64 && aligned) attn_warp<2>(o, t, h, lane);
  else attn_warp_generic(o, t, h, lane);
}

// Causal attention of the dense prompt prefill (FQ3C_ATTN with flags bit 0: head_dim 128, no history rows, window >= M, M <= 2048):
// one warp per (query, head), two phases with different lane roles instead of the key-by-key online softmax above —
//   1. four lanes per KEY, eight keys per step: a lane multiplies 32 dims of its key (q from shared memory, four 16-byte loads of the
//      key row), two shuffles finish the dot product (against five per key in the kernel above); the score, rounded to bf16 exactly
//      where the kernel above rounds it, goes to shared memory, and after the warp's max is known the same lane replaces it by
//      p = exp(score - max) — once per key, not once per key and lane;
//   2. lanes take DIMS (four each): every lane walks the keys in order, p straight from shared memory, and accumulates l and its
//      four output dims — no rescaling, no shuffles.
// Same rounding points as attn_warp (score -> bf16 -> x scale -> bf16; fp32 softmax and accumulation; bf16 output); the fp32 sums run in
// another order, which the prefill tests bound against the oracle and the chunked prefill.  M = 240 (ICL prompt): 78 -> ~12 us per layer.
constexpr int APF_WARPS = 8;
__global__ void __launch_bounds__(APF_WARPS * 32) fq3c_attn_prefill_kernel(const fq3c_op o, const int tpad) {
  grid_dep_begin();
  extern __shared__ unsigned char apf_smem[];
  const int nh = o.i0, nkv = o.i1, T = o.M, win = o.K;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // heavy queries (many keys) first: the grid's tail then consists of the short ones.  (Warps of a CTA = the heads of one query;
  // consecutive queries of one head per CTA was measured: slower, 99 vs 66 us at M = 240.)
  const int gw = blockIdx.x * APF_WARPS + warp;
  if (gw >= T * nh) return;
  const int t = T - 1 - gw / nh, h = gw - (gw / nh) * nh;
  const int kvh = h / (nh / nkv);
  float* qs = reinterpret_cast<float*>(apf_smem) + warp * 128;
  float* sc = reinterpret_cast<float*>(apf_smem + APF_WARPS * 128 * 4) + (size_t)warp * tpad;
  const bf16* base = reinterpret_cast<const bf16*>(o.A);
  const size_t lda = (size_t)o.lda;
  const int koff = nh * 128 + kvh * 128, voff = (nh + nkv) * 128 + kvh * 128;
  {
    const uint2 r = *reinterpret_cast<const uint2*>(base + (size_t)t * lda + h * 128 + lane * 4);
    *reinterpret_cast<float4*>(qs + lane * 4) = make_float4(__uint_as_float(r.x << 16), __uint_as_float(r.x & 0xffff0000u),
                                                            __uint_as_float(r.y << 16), __uint_as_float(r.y & 0xffff0000u));
  }
  __syncwarp();
  const float scale = rsqrtf(128.f);
  const int j0 = max(0, t - win + 1);
  float mx = -INFINITY;
  // four lanes per key, eight keys per step: the four lanes of a key read 64 contiguous bytes per load instruction (a warp-wide
  // load touches 8 lines; one lane per key would touch 32 and the L1 tag stage, one line per cycle, becomes the bound: measured)
  const int sub = lane & 3, kq = lane >> 2;
  for (int jb = j0; jb <= t; jb += 16) {  // two groups of eight keys per step: sixteen rows in flight per L2 round trip
    uint4 kk[2][4];
    bool ok[2];
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      const int j = jb + g * 8 + kq;
      ok[g] = j <= t;
      const uint4* kr = reinterpret_cast<const uint4*>(base + (size_t)(ok[g] ? j : t) * lda + koff) + sub;
#pragma unroll
      for (int c = 0; c < 4; ++c) kk[g][c] = kr[c * 4];
    }
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      float d0 = 0.f, d1 = 0.f;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float* qp = qs + (c * 4 + sub) * 8;
        const float4 qa = *reinterpret_cast<const float4*>(qp), qb = *reinterpret_cast<const float4*>(qp + 4);
        d0 += qa.x * __uint_as_float(kk[g][c].x << 16) + qa.y * __uint_as_float(kk[g][c].x & 0xffff0000u) +
              qa.z * __uint_as_float(kk[g][c].y << 16) + qa.w * __uint_as_float(kk[g][c].y & 0xffff0000u);
        d1 += qb.x * __uint_as_float(kk[g][c].z << 16) + qb.y * __uint_as_float(kk[g][c].z & 0xffff0000u) +
              qb.z * __uint_as_float(kk[g][c].w << 16) + qb.w * __uint_as_float(kk[g][c].w & 0xffff0000u);
      }
      float dsum = d0 + d1;
      dsum += __shfl_xor_sync(0xffffffffu, dsum, 1);
      dsum += __shfl_xor_sync(0xffffffffu, dsum, 2);
      const float su = bf16r(bf16r(dsum) * scale);
      if (ok[g]) {
        if (sub == 0) sc[jb + g * 8 + kq - j0] = su;
        mx = fmaxf(mx, su);
      }
    }
  }
  for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  // the exponentials once per key (the lane that scored it), not once per key and lane: expf is ~20 instructions
  for (int j = j0 + lane; j <= t; j += 32) sc[j - j0] = expf(sc[j - j0] - mx);
  __syncwarp();
  float l = 0.f, acc[4] = {0.f, 0.f, 0.f, 0.f};
  const bf16* vp = base + voff + lane * 4;
  int j = j0;
  // sixteen keys per step: the step is one L2 round trip (the V rows of a prompt are not in L1), so all sixteen loads go out before
  // the first one is used; the accumulation itself stays in key order
  for (; j + 15 <= t; j += 16) {
    uint2 r[16];
    float pr[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) r[u] = *reinterpret_cast<const uint2*>(vp + (size_t)(j + u) * lda);
#pragma unroll
    for (int u = 0; u < 16; ++u) pr[u] = sc[j + u - j0];
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      l += pr[u];
      acc[0] += pr[u] * __uint_as_float(r[u].x << 16); acc[1] += pr[u] * __uint_as_float(r[u].x & 0xffff0000u);
      acc[2] += pr[u] * __uint_as_float(r[u].y << 16); acc[3] += pr[u] * __uint_as_float(r[u].y & 0xffff0000u);
    }
  }
  for (; j <= t; ++j) {
    const uint2 r0 = *reinterpret_cast<const uint2*>(vp + (size_t)j * lda);
    const float p0 = sc[j - j0];
    l += p0;
    acc[0] += p0 * __uint_as_float(r0.x << 16); acc[1] += p0 * __uint_as_float(r0.x & 0xffff0000u);
    acc[2] += p0 * __uint_as_float(r0.y << 16); acc[3] += p0 * __uint_as_float(r0.y & 0xffff0000u);
  }
  bf16* out = reinterpret_cast<bf16*>(o.C) + (size_t)t * o.ldc + h * 128 + lane * 4;
  const float inv = 1.f / l;
  uint2 w;
  w.x = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(acc[0] * inv)) | ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(acc[1] * inv)) << 16);
  w.y = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(acc[2] * inv)) | ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(acc[3] * inv)) << 16);
  *reinterpret_cast<uint2*>(out) = w;
}

// Dense prefill helper (talker): one warp per (row, head) of the fused qkv rows A [M, lda] = (q heads | k heads | v heads).
//   q / k heads: per-head RMSNorm with bf16 gamma (q: p0, k: p1), HF rounding points, then rotary embedding from the bf16
//                tables B (cos) / bias (sin) at position row + i2 (rotate-half), in place;
//   k / v heads: the finished row is also written to the static KV cache C (K) / C2 (V), laid out [kv_head][ldc][128].
// Same arithmetic as head_norm_rope / the KV append of the decode kernel (fq3_kernel.cuh), so decode steps can attend to it.
__global__ void fq3c_qknorm_rope_kv_kernel(const fq3c_op o) {
  grid_dep_begin(o.M > 512);
  const int nq = o.i0, nkv = o.i1, pos0 = o.i2, nheads = nq + 2 * nkv;
  const int wpb = blockDim.x >> 5;
  const int gw = blockIdx.x * wpb + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (gw >= o.M * nheads) return;
  const int t = gw / nheads, h = gw - t * nheads;
  bf16* row = reinterpret_cast<bf16*>(const_cast<void*>(o.A)) + (size_t)t * o.lda + (size_t)h * 128 + lane * 4;
  uint2 raw = *reinterpret_cast<const uint2*>(row);
  const int pos = pos0 + t;
  if (h < nq + nkv) {
    const bf16* gamma = reinterpret_cast<const bf16*>(h < nq ? o.p0 : o.p1) + lane * 4;
    const bf16* cosp = reinterpret_cast<const bf16*>(o.B) + (size_t)pos * 128 + lane * 4;
    const bf16* sinp = reinterpret_cast<const bf16*>(o.bias) + (size_t)pos * 128 + lane * 4;
    float x[4] = {__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u), __uint_as_float(raw.y << 16),
                  __uint_as_float(raw.y & 0xffff0000u)};
    float ss = x[0] * x[0] + x[1] * x[1] + x[2] * x[2] + x[3] * x[3];
    for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
    const float rs = rsqrtf(ss * (1.f / 128.f) + o.f0);
    float y[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) y[i] = bf16r(bf16r(x[i] * rs) * __bfloat162float(gamma[i]));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float partner = __shfl_xor_sync(0xffffffffu, y[i], 16);
      const float rot = (lane < 16) ? -partner : partner;
      x[i] = bf16r(bf16r(y[i] * __bfloat162float(cosp[i])) + bf16r(rot * __bfloat162float(sinp[i])));
    }
    const __nv_bfloat162 lo = __floats2bfloat162_rn(x[0], x[1]), hi = __floats2bfloat162_rn(x[2], x[3]);
    raw = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    *reinterpret_cast<uint2*>(row) = raw;
  }
  if (h >= nq) {
    const bool is_v = h >= nq + nkv;
    const int kvh = is_v ? h - nq - nkv : h - nq;
    bf16* dst = reinterpret_cast<bf16*>(is_v ? o.C2 : o.C) + ((size_t)kvh * o.ldc + pos) * 128 + lane * 4;
    *reinterpret_cast<uint2*>(dst) = raw;
  }
}

// Attention of a few rows or of a short window, FQ3C_ATTN with heads of D entries: a CTA takes RB query rows of one key / value head, stages the keys and values that they
// see in shared memory once, and then
//   scores: a warp per (row, head, 32 keys), a lane per key - q is a broadcast, keys lie 16 bytes apart in banks, no shuffles;
//   sums:   a warp per (row, head), the exponentials once per key, then a lane per D / 32 entries walks the keys in order.
// Its bits are those of the kernels with a warp per (row, head), infinities and NaN among them: fq3c_attn_kernel's, and with PROMPT fq3c_attn_prefill_kernel's.  A dot
// product is added up as their lanes and shuffles do, the running maximum of the one is a scan over the keys, its sums shrink key by key.  So a
// stream and the whole decode agree whichever kernel each of their sizes comes to.
// What bounds it is latency: one round trip to L2, a few thousand cycles of dependent work and a launch; the kernels with a warp per (row, head) make
// a round trip for every four to sixteen keys.
// PROMPT: `n` is the FQ3C_QKNORM_ROPE_KV op in front.  Every CTA norms and turns the keys it stages (again for each RB rows: 60 instructions a key), its queries, and
// writes its own rows of the cache: one launch in place of two, and the rows in `A` stay as the product left them.  39 rows of
// 16 heads 8.2 -> 5.6 us; the codec's attention (16 heads of 64, window 72) 33 rows 7.6 -> 3.8, 256 rows 32.0 -> 12.9, one row behind 71 others 14.4 -> 4.3.
constexpr int GP_SMS = 148;
constexpr int AR_WARPS = 16, AR_SMEM_MAX = 128 * 1024;
struct AttnRows { int rb, span, sp; size_t smem; };      // rows of a CTA, keys it may stage, pitch of its scores
__host__ __device__ constexpr int ar_k_pitch(int d) { return d * 2 + 16; }      // bytes
AttnRows attn_rows_plan(const fq3c_op& o, const bool prompt) {
  AttnRows r;
  const int hg = o.i0 / o.i1;
  r.rb = 1;      // as few rows as one CTA per SM allows: 100 rows of 16 heads with 160 CTAs 16.5 us
  while (r.rb < 16 && (long)((o.M + r.rb - 1) / r.rb) * o.i1 > GP_SMS) ++r.rb;
  r.span = (int)std::min<long>((long)o.K + r.rb - 1, (long)o.M + o.taps);
  r.sp = (r.span + 31) / 32 * 32;
  r.smem = (size_t)r.span * (ar_k_pitch(o.i2) + o.i2 * 2) + (size_t)r.rb * hg * (o.i2 + (prompt ? 1 : 2) * r.sp) * 4;
  return r;
}
// a head's row of 128, four entries a lane: RMSNorm and rotation with the rounding points of fq3c_qknorm_rope_kv_kernel
__device__ __forceinline__ uint2 norm_turn(const uint2 raw, const float eps, const uint2 gamma, const uint2 cosr, const uint2 sinr, const int lane) {
  float x[4] = {__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u), __uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xffff0000u)};
  const float ga[4] = {__uint_as_float(gamma.x << 16), __uint_as_float(gamma.x & 0xffff0000u), __uint_as_float(gamma.y << 16), __uint_as_float(gamma.y & 0xffff0000u)};
  const float co[4] = {__uint_as_float(cosr.x << 16), __uint_as_float(cosr.x & 0xffff0000u), __uint_as_float(cosr.y << 16), __uint_as_float(cosr.y & 0xffff0000u)};
  const float si[4] = {__uint_as_float(sinr.x << 16), __uint_as_float(sinr.x & 0xffff0000u), __uint_as_float(sinr.y << 16), __uint_as_float(sinr.y & 0xffff0000u)};
  float ss = x[0] * x[0] + x[1] * x[1] + x[2] * x[2] + x[3] * x[3];
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
  const float rs = rsqrtf(ss * (1.f / 128.f) + eps);
  float y[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) y[i] = bf16r(bf16r(x[i] * rs) * ga[i]);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float partner = __shfl_xor_sync(0xffffffffu, y[i], 16);
    x[i] = bf16r(y[i] * co[i]) + bf16r((lane < 16 ? -partner : partner) * si[i]);
  }
  const __nv_bfloat162 lo = __floats2bfloat162_rn(x[0], x[1]), hi = __floats2bfloat162_rn(x[2], x[3]);
  return make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}
__device__ __forceinline__ float dot2(const float x, const float y, const uint32_t a) { return fmaf(x, __uint_as_float(a << 16), __fmul_rn(y, __uint_as_float(a & 0xffff0000u))); }
__device__ __forceinline__ float dot4(const float4 q, const uint32_t a, const uint32_t b) {
  return fmaf(q.w, __uint_as_float(b & 0xffff0000u), fmaf(q.z, __uint_as_float(b << 16), dot2(q.x, q.y, a)));
}
// The D / 32 entries of each lane of attn_warp, summed in the order of its shuffles (lanes 16, 8, 4, 2, 1 apart): pieces of eight entries hold 256 / D lanes' shares, and
// here the pieces C, C + STRIDE, .. have met.  (Products of two bf16 are exact in f32 up to its largest value: only the order of the sums counts, and which product of a pair
// overflows by itself.)
template <int D, int C, int STRIDE>
__device__ __forceinline__ void lane_sums(const uint4* kp, const float4* qa, float (&sum)[256 / D]) {
  if constexpr (STRIDE == D / 8) {
    const uint4 k = kp[C];
    const float4 x = qa[2 * C], y = qa[2 * C + 1];
    if constexpr (D == 128) {
      sum[0] = dot4(x, k.x, k.y);
      sum[1] = dot4(y, k.z, k.w);
    } else {
      sum[0] = dot2(x.x, x.y, k.x);
      sum[1] = dot2(x.z, x.w, k.y);
      sum[2] = dot2(y.x, y.y, k.z);
      sum[3] = dot2(y.z, y.w, k.w);
    }
  } else {
    float far[256 / D];
    lane_sums<D, C, 2 * STRIDE>(kp, qa, sum);
    lane_sums<D, C + STRIDE, 2 * STRIDE>(kp, qa, far);
#pragma unroll
    for (int i = 0; i < 256 / D; ++i) sum[i] += far[i];
  }
}
template <int D, bool PROMPT>
__global__ void __launch_bounds__(AR_WARPS * 32) fq3c_attn_rows_kernel(const __grid_constant__ fq3c_op o, const __grid_constant__ fq3c_op n, const int RB, const int span_max, const int SP) {
  extern __shared__ __align__(16) unsigned char ar_raw[];
  constexpr int PER = D / 32, KP = ar_k_pitch(D);      // entries of a lane; bytes of a staged key
  typedef typename std::conditional<PER == 4, uint2, uint32_t>::type Vec;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nh = o.i0, G = o.i1, HG = nh / G, g = blockIdx.y, win = o.K, hist = PROMPT ? 0 : o.taps;
  const int r0 = blockIdx.x * RB, rows = min(RB, o.M - r0);
  grid_dep_begin();
  uint2 gk = make_uint2(0u, 0u), gq = make_uint2(0u, 0u);
  if (PROMPT) {
    gk = *reinterpret_cast<const uint2*>(reinterpret_cast<const bf16*>(n.p1) + lane * 4);
    gq = *reinterpret_cast<const uint2*>(reinterpret_cast<const bf16*>(n.p0) + lane * 4);
  }
  const int first = (!PROMPT && o.p0) ? hist - min(*reinterpret_cast<const int*>(o.p0), hist) : 0;
  const int j_lo = max(first, r0 + hist - win + 1), span = r0 + rows + hist - j_lo, items = span + rows * HG;
  unsigned char* ks = ar_raw;                                              // [span][KP]
  unsigned char* vs = ks + (size_t)span_max * KP;                          // [span][2 D]
  float* qs = reinterpret_cast<float*>(vs + (size_t)span_max * 2 * D);     // [RB HG][D]
  float* sc = qs + RB * HG * D;                                            // [RB HG][SP]
  const bf16* base = reinterpret_cast<const bf16*>(o.A) + lane * PER;
  const size_t lda = (size_t)o.lda;
  const bf16* cosp = reinterpret_cast<const bf16*>(n.B) + lane * 4;
  const bf16* sinp = reinterpret_cast<const bf16*>(n.bias) + lane * 4;
  // the keys with their values, then the queries: U of a warp's items on their way together
  constexpr int U = 4;
  for (int ib = warp; ib < items; ib += AR_WARPS * U) {
    Vec x[U], v[U];
    uint2 c[U], si[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = min(ib + u * AR_WARPS, items - 1), qi = i - span;
      const int row = qi < 0 ? j_lo + i : r0 + hist + qi / HG, head = qi < 0 ? nh + g : g * HG + qi % HG;
      x[u] = *reinterpret_cast<const Vec*>(base + row * lda + head * D);
      if (qi < 0) v[u] = *reinterpret_cast<const Vec*>(base + row * lda + (head + G) * D);
      if constexpr (PROMPT) {
        c[u] = *reinterpret_cast<const uint2*>(cosp + (size_t)(n.i2 + row) * 128);
        si[u] = *reinterpret_cast<const uint2*>(sinp + (size_t)(n.i2 + row) * 128);
      }
    }
    if constexpr (PROMPT) {
#pragma unroll
      for (int u = 0; u < U; ++u) x[u] = norm_turn(x[u], n.f0, ib + u * AR_WARPS < span ? gk : gq, c[u], si[u], lane);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = ib + u * AR_WARPS, qi = i - span;
      if (qi < 0) {
        *reinterpret_cast<Vec*>(ks + (size_t)i * KP + lane * PER * 2) = x[u];
        *reinterpret_cast<Vec*>(vs + (size_t)i * 2 * D + lane * PER * 2) = v[u];
        if constexpr (PROMPT) {
          if (j_lo + i >= r0) {
            const size_t at = ((size_t)g * n.ldc + n.i2 + j_lo + i) * 128 + lane * 4;
            *reinterpret_cast<uint2*>(reinterpret_cast<bf16*>(n.C) + at) = x[u];
            *reinterpret_cast<uint2*>(reinterpret_cast<bf16*>(n.C2) + at) = v[u];
          }
        }
      } else if (i < items) {
        float* q = qs + qi * D + lane * PER;
        if constexpr (PER == 4) *reinterpret_cast<float4*>(q) = make_float4(__uint_as_float(x[u].x << 16), __uint_as_float(x[u].x & 0xffff0000u), __uint_as_float(x[u].y << 16), __uint_as_float(x[u].y & 0xffff0000u));
        else *reinterpret_cast<float2*>(q) = make_float2(__uint_as_float(x[u] << 16), __uint_as_float(x[u] & 0xffff0000u));
      }
    }
  }
  __syncthreads();
  const float scale = rsqrtf((float)D);
  const int chunks = (span + 31) >> 5;
  for (int it = warp; it < rows * HG * chunks; it += AR_WARPS) {
    const int i = it / chunks, ch = it - i * chunks, j = ch * 32 + lane, t = r0 + i / HG + hist - j_lo;      // the row's own key
    if (ch * 32 > t || ch * 32 + 31 <= t - win) continue;
    const uint4* kp = reinterpret_cast<const uint4*>(ks + (size_t)min(j, span - 1) * KP);
    const float4* qa = reinterpret_cast<const float4*>(qs + i * D);
    float dot;
    if constexpr (PROMPT) {      // the shares of four lanes, every fourth piece each, its first and its last four entries apart
      float part[4];
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        float d0 = 0.f, d1 = 0.f;
#pragma unroll
        for (int c = l; c < D / 8; c += 4) {
          const uint4 k = kp[c];
          d0 += dot4(qa[2 * c], k.x, k.y);
          d1 += dot4(qa[2 * c + 1], k.z, k.w);
        }
        part[l] = d0 + d1;
      }
      dot = (part[0] + part[1]) + (part[2] + part[3]);
    } else {
      float sum[256 / D];
      lane_sums<D, 0, 1>(kp, qa, sum);
      if constexpr (D == 128) dot = sum[0] + sum[1];
      else dot = (sum[0] + sum[2]) + (sum[1] + sum[3]);
    }
    const float x = bf16r(bf16r(dot) * scale);
    if constexpr (PROMPT) sc[i * SP + j] = x;
    else reinterpret_cast<float2*>(sc)[i * SP + j].x = x;
  }
  __syncthreads();
  for (int i = warp; i < rows * HG; i += AR_WARPS) {
    const int row = i / HG, h = g * HG + i - row * HG, je = r0 + row + hist - j_lo, jb = max(0, je - win + 1);
    float l = 0.f, acc[PER];
#pragma unroll
    for (int e = 0; e < PER; ++e) acc[e] = 0.f;
    const unsigned char* vp = vs + lane * PER * 2;
    if constexpr (PROMPT) {
      float* s = sc + (size_t)i * SP;
      float mx = -INFINITY;
      for (int j = jb + lane; j <= je; j += 32) mx = fmaxf(mx, s[j]);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
      for (int j = jb + lane; j <= je; j += 32) s[j] = expf(s[j] - mx);
      __syncwarp();
#pragma unroll 8
      for (int j = jb; j <= je; ++j) {
        const float p = s[j];
        const Vec v = *reinterpret_cast<const Vec*>(vp + (size_t)j * 2 * D);
        l += p;
        acc[0] = fmaf(p, __uint_as_float(v.x << 16), acc[0]); acc[1] = fmaf(p, __uint_as_float(v.x & 0xffff0000u), acc[1]);
        acc[2] = fmaf(p, __uint_as_float(v.y << 16), acc[2]); acc[3] = fmaf(p, __uint_as_float(v.y & 0xffff0000u), acc[3]);
      }
    } else {
      // the highest score up to each key, four times 32 keys at a time: a key's weight, and what the sums in front of it shrink by
      float2* s = reinterpret_cast<float2*>(sc) + (size_t)i * SP;
      float m = -INFINITY;
      for (int b = jb + lane; b - lane <= je; b += 128) {
        float x[4], top[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) top[u] = x[u] = b + 32 * u <= je ? s[b + 32 * u].x : -INFINITY;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float y = __shfl_up_sync(0xffffffffu, top[u], d);
            if (lane >= d) top[u] = fmaxf(top[u], y);
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          top[u] = fmaxf(m, top[u]);
          float before = __shfl_up_sync(0xffffffffu, top[u], 1);
          if (lane == 0) before = m;
          m = __shfl_sync(0xffffffffu, top[u], 31);
          if (b + 32 * u <= je) s[b + 32 * u] = make_float2(expf(x[u] - top[u]), expf(before - top[u]));
        }
      }
      __syncwarp();
#pragma unroll 8
      for (int j = jb; j <= je; ++j) {
        const float2 w = s[j];
        const Vec v = *reinterpret_cast<const Vec*>(vp + (size_t)j * 2 * D);
        l = fmaf(l, w.y, w.x);
        if constexpr (PER == 4) {
          acc[0] = attn_add(acc[0], w.y, w.x, __uint_as_float(v.x << 16)); acc[1] = attn_add(acc[1], w.y, w.x, __uint_as_float(v.x & 0xffff0000u));
          acc[2] = attn_add(acc[2], w.y, w.x, __uint_as_float(v.y << 16)); acc[3] = attn_add(acc[3], w.y, w.x, __uint_as_float(v.y & 0xffff0000u));
        } else {
          acc[0] = attn_add(acc[0], w.y, w.x, __uint_as_float(v << 16)); acc[1] = attn_add(acc[1], w.y, w.x, __uint_as_float(v & 0xffff0000u));
        }
      }
    }
    if constexpr (PROMPT) {
      const float inv = 1.f / l;
#pragma unroll
      for (int e = 0; e < PER; ++e) acc[e] *= inv;
    } else {
#pragma unroll
      for (int e = 0; e < PER; ++e) acc[e] /= l;
    }
    bf16* out = reinterpret_cast<bf16*>(o.C) + (size_t)(r0 + row) * o.ldc + h * D + lane * PER;
    if constexpr (PER == 4) {
      const __nv_bfloat162 lo = __floats2bfloat162_rn(acc[0], acc[1]), hi = __floats2bfloat162_rn(acc[2], acc[3]);
      *reinterpret_cast<uint2*>(out) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    } else {
      *reinterpret_cast<__nv_bfloat162*>(out) = __floats2bfloat162_rn(acc[0], acc[1]);
    }
  }
}

__global__ void fq3c_dwconv_kernel(const fq3c_op o) {
  grid_dep_begin();
  const size_t n = (size_t)o.M * o.N;
  const bf16* x = reinterpret_cast<const bf16*>(o.A);
  const float* w = reinterpret_cast<const float*>(o.B);
  const float* b = reinterpret_cast<const float*>(o.bias);
  bf16* y = reinterpret_cast<bf16*>(o.C);
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int t = (int)(i / o.N), c = (int)(i - (size_t)t * o.N);
    float a = b[c];
    for (int j = 0; j < o.taps; ++j) {
      const int r = t - (o.taps - 1) + j;  // rows [-i0, 0) are the history rows of a stateful decode
      if (r >= -o.i0) a += w[c * o.taps + j] * __bfloat162float(x[(long)r * o.lda + c]);
    }
    y[(size_t)t * o.ldc + c] = __float2bfloat16_rn(a);
  }
}

__global__ void fq3c_copy_kernel(const fq3c_op o) {
  const int nv = o.N >> 3;  // 16-byte pieces per row (N, lda, ldc are multiples of 8)
  const size_t n = (size_t)o.M * nv;
  const bf16* x = reinterpret_cast<const bf16*>(o.A);
  bf16* y = reinterpret_cast<bf16*>(o.C);
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const size_t t = i / nv, c = (i - t * nv) * 8;
    *reinterpret_cast<uint4*>(y + t * o.ldc + c) = *reinterpret_cast<const uint4*>(x + t * o.lda + c);
  }
}
__global__ void fq3c_advance_kernel(int* counter, int by) { *counter += by; }

// A step's token ids and wanted rows, as the launch's own arguments: a copy from pageable memory first waits until the stream has nothing left to do, so that every decoded
// token's launches began some 40 us after the ones in front had ended (24 tokens behind a prompt of 203: 4920 us, this way 4130).
struct PutInts {
  static constexpr int MOST = 1000;      // with the two other fields within the 4 KB that a launch's arguments have everywhere
  int32_t* dst;
  int n;
  int32_t v[MOST];
};
__global__ void fq3c_put_ints_kernel(const __grid_constant__ PutInts p) {
  for (int i = threadIdx.x; i < p.n; i += blockDim.x) p.dst[i] = p.v[i];
}
// FQ3C_ROLL: blockIdx.x = history buffer, blockIdx.y = column slice (slices are independent).  dst row r <- src row r + new; when the
// ranges overlap (new < hist) the rows go in batches of `new`: a batch's sources are the next batch's destinations, so a block
// barrier separates them; within a batch sources and destinations are disjoint.
constexpr int ROLL_SLICES = 8;
__global__ void __launch_bounds__(256) fq3c_roll_kernel(const long long* desc, int* counter, int by) {
  const long long* d = desc + (size_t)blockIdx.x * 5;
  bf16* base = reinterpret_cast<bf16*>(d[0]);
  const int hist = (int)d[1], n_new = (int)d[2], cols = (int)d[3], ld = (int)d[4];
  const int nv = cols >> 3;
  const int p0 = (int)(((long)blockIdx.y * nv) / ROLL_SLICES), p1 = (int)(((long)(blockIdx.y + 1) * nv) / ROLL_SLICES);
  const int np = p1 - p0;
  const int batch = n_new >= hist ? hist : n_new;
  for (int r0 = 0; r0 < hist && np > 0; r0 += batch) {
    const int rows = min(batch, hist - r0);
    for (int i = threadIdx.x; i < rows * np; i += blockDim.x) {
      const int r = r0 + i / np, p = p0 + i % np;
      *reinterpret_cast<uint4*>(base + (size_t)r * ld + p * 8) = *reinterpret_cast<const uint4*>(base + (size_t)(r + n_new) * ld + p * 8);
    }
    __syncthreads();
  }
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && counter) *counter += by;
}

__global__ void fq3c_snake_kernel(const fq3c_op o) {
  const size_t n = (size_t)o.M * o.N;
  const bf16* x = reinterpret_cast<const bf16*>(o.A);
  const float* ea = reinterpret_cast<const float*>(o.p0);
  const float* ib = reinterpret_cast<const float*>(o.p1);
  bf16* y = reinterpret_cast<bf16*>(o.C);
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int t = (int)(i / o.N), c = (int)(i - (size_t)t * o.N);
    const float v = __bfloat162float(x[(size_t)t * o.lda + c]);
    y[(size_t)t * o.ldc + c] = __float2bfloat16_rn(v + ib[c] * sin_sq(v * ea[c]));
  }
}

// A convolution to ONE output channel (the vocoder's last layer: 7 taps x 96 channels): a dot product per row, not a matrix product.  A block stages the rows
// its 256 outputs see once (the 64 x 64 tensor-core tile read them once per tap and threw 63 of 64 columns away) and every thread forms one
// output, eight channels a step, f32 sums.  Bound by shared memory (one row's 16-byte pieces per lane).  491 520 rows: 178 -> 51 us.
constexpr int C1_ROWS = 256, C1_SPAN = 64, C1_CIN = 128;
__global__ void __launch_bounds__(C1_ROWS) fq3c_conv1_kernel(const fq3c_op o, const int lo, const int span) {
  grid_dep_begin();
  extern __shared__ __align__(16) unsigned char c1_raw[];
  const int cin = o.cin, pitch = cin + 8, m0 = o.m_begin + blockIdx.x * C1_ROWS, tid = threadIdx.x, cpr = cin >> 3;
  float* w = reinterpret_cast<float*>(c1_raw);                         // [taps][cin]
  bf16* xs = reinterpret_cast<bf16*>(w + o.taps * cin);                // [C1_ROWS + span][cin + 8]: rows 16 bytes apart in banks
  for (int i = tid; i < o.taps * cin; i += C1_ROWS) w[i] = __bfloat162float(reinterpret_cast<const bf16*>(o.B)[i]);
  const int rows = min(C1_ROWS, o.M - m0) + span;
  for (int i = tid; i < rows * cpr; i += C1_ROWS) {
    const int r = i / cpr, c = i - r * cpr, src = m0 + lo + r;
    const bool ok = src >= 0 && src < o.a_rows;
    cp_async16(xs + (size_t)r * pitch + c * 8, reinterpret_cast<const bf16*>(o.A) + (size_t)(ok ? src : 0) * o.lda + c * 8, ok);
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  const int row = m0 + tid;
  if (row >= o.M) return;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  for (int t = 0; t < o.taps; ++t) {
    const uint4* xr = reinterpret_cast<const uint4*>(xs + (size_t)(tid + o.tap_off[t] - lo) * pitch);
    const float4* wr = reinterpret_cast<const float4*>(w + t * cin);
#pragma unroll 4
    for (int c = 0; c < cpr; ++c) {
      const uint4 x = xr[c];
      const float4 a = wr[2 * c], b = wr[2 * c + 1];
      acc[0] = fmaf(__uint_as_float(x.x << 16), a.x, acc[0]); acc[1] = fmaf(__uint_as_float(x.x & 0xffff0000u), a.y, acc[1]);
      acc[2] = fmaf(__uint_as_float(x.y << 16), a.z, acc[2]); acc[3] = fmaf(__uint_as_float(x.y & 0xffff0000u), a.w, acc[3]);
      acc[0] = fmaf(__uint_as_float(x.z << 16), b.x, acc[0]); acc[1] = fmaf(__uint_as_float(x.z & 0xffff0000u), b.y, acc[1]);
      acc[2] = fmaf(__uint_as_float(x.w << 16), b.z, acc[2]); acc[3] = fmaf(__uint_as_float(x.w & 0xffff0000u), b.w, acc[3]);
    }
  }
  epilogue_pair(o, row, 0, (acc[0] + acc[1]) + (acc[2] + acc[3]), 0.f);
}

#include "fq3_seq.cuh"
#include "fq3_f32.cuh"
#include "fq3_gemm.cuh"
#include "fq3_ggemm.cuh"
#include "fq3_attn.cuh"

int fail(const std::string& m) { g_err = m; return -1; }

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link against libcuda)
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
    cudaGetLastError();
  }
  return fn;
}
// bf16 matrix [rows, inner] with a row pitch of ld elements, boxes of box_rows x 64 columns, 128-byte swizzle, zeros outside
bool make_map(CUtensorMap* m, const void* base, uint64_t inner, uint64_t rows, uint64_t ld, uint32_t box_rows) {
  EncodeTiledFn fn = encode_tiled();
  if (!fn || !base || inner == 0 || rows == 0) return false;
  if ((reinterpret_cast<uintptr_t>(base) & 15) || (ld * 2) % 16) return false;
  const cuuint64_t dims[2] = {inner, rows};
  const cuuint64_t strides[1] = {ld * 2};
  const cuuint32_t box[2] = {(cuuint32_t)TK, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// One launch; `after`: it may begin before the launches in front of it on the stream have ended (its kernel waits for them itself, with
// griddepcontrol.wait).  cluster: CTAs per cluster.
template <typename... P, typename... A>
void launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, bool after, int cluster, const A&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = s;
  cudaLaunchAttribute at[2];
  int n = 0;
  if (after) { at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[n].val.programmaticStreamSerializationAllowed = 1; ++n; }
  if (cluster > 1) { at[n].id = cudaLaunchAttributeClusterDimension; at[n].val.clusterDim.x = cluster; at[n].val.clusterDim.y = 1; at[n].val.clusterDim.z = 1; ++n; }
  cfg.attrs = at; cfg.numAttrs = n;
  cudaLaunchKernelEx(&cfg, kernel, args...);
}
// The sequence models' kernels wait (seq_dep_begin) only with few rows, so they are launched early by the same number that they test: the rows that their own arguments hold.
template <typename... A> int dep_rows(const fq3c_op& o, const A&...) { return o.M; }
template <typename... A> int dep_rows(const SeqGemm& g, const A&...) { return g.M; }
inline int dep_rows(const long long*, const int*, const int by) { return by; }      // fq3s_commit_kernel
// Walks over a cache in splits, whose blocks are large: not early with more of them than SMs, where they come up unevenly (one row of 32 heads over 4 behind 2000 positions 23.4 us, early
// 25.7).
inline bool blocks_fit(const dim3& grid) { return (long)grid.x * grid.y * grid.z <= GP_SMS; }
template <typename... P, typename... A>
void launch_seq(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, bool after, int cluster, const A&... args) {
  launch_after(kernel, grid, block, smem, s, after && seq_early(dep_rows(args...)), cluster, args...);
}

// the norm of a finished product's rows
void launch_rownorm(const fq3c_op& o, cudaStream_t s, const bool after) {
  const int rows = o.M - o.m_begin;
  if (norm_vec_ok(o.C, o.norm_out, o.norm_w, o.N, o.ldc, o.norm_ld))
    launch_after(fq3c_rownorm_vec_kernel, (unsigned)((rows + RN_WARPS - 1) / RN_WARPS), RN_WARPS * 32, 0, s, after, 1, reinterpret_cast<const bf16*>(o.C), o.ldc,
                 reinterpret_cast<bf16*>(o.norm_out), o.norm_ld, reinterpret_cast<const float*>(o.norm_w), o.norm_eps, o.m_begin, rows, o.N);
  else launch_after(fq3c_rownorm_kernel, (unsigned)rows, 256, 0, s, after, 1, o);
}

// ---- the tcgen05 GEMM: what a launch looks like ------------------------------------------------------------------------------
constexpr int GP_SMEM_MAX = 227 * 1024, GP_SMEM_HALF = 112 * 1024;
// Whether the epilogue may move whole 32-byte sectors (16 columns of bf16, 8 of f32).
bool gemm_vec16(const fq3c_op& o) {
  auto off = [](const void* p, int a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) != 0; };
  if (o.N % 16) return false;
  const bool f32 = (o.flags & FQ3C_OUT_F32) != 0;
  if (o.flags & FQ3C_SWIGLU) return o.ldc % 8 == 0 && !off(o.C, 32);
  if (o.ldc % (f32 && !(o.flags & FQ3C_SNAKE2) ? 8 : 16) || off(o.C, 32)) return false;
  if ((o.flags & FQ3C_RESID) && (o.ldr % 16 || off(o.res, 32))) return false;
  if ((o.flags & FQ3C_SNAKE2) && off(o.C2, 32)) return false;
  return true;
}
// A tile's epilogue, in cycles for 16 columns of its 128 rows with sixteen warps at work on an SM (two CTAs of eight or one of sixteen; fitted to 75776 x 384 x 64,
// where it is all there is: bf16 18 us, residual 34 - 42, GELU 43, gated units 38, residual and SnakeBeta 59 - 65).
long epilogue_piece(const int flags) {
  return 290 + (flags & FQ3C_RESID ? 310 : 0) + (flags & FQ3C_SNAKE2 ? 480 : 0) + (flags & (FQ3C_GELU | FQ3C_SILU) ? 560 : 0) + (flags & FQ3C_SWIGLU ? 510 : 0);
}
enum GemmShape { GS_WIDE, GS_FEW, GS_HALF };      // one CTA per SM with sixteen epilogue warps, one with eight, two with eight each
struct GemmLaunch { GemmPlan g; GemmShape shape; unsigned grid; size_t smem; };
GemmLaunch gemm_plan(const fq3c_op& o) {
  GemmLaunch L{};
  GemmPlan& g = L.g;
  const int rows = o.M - o.m_begin;
  g.mt = (rows + TM - 1) / TM;
  g.a_rows = g.mt == 1 ? (rows + 7) / 8 * 8 : TM;
  g.kpt = o.taps == 1 ? (o.K + TK - 1) / TK : (o.cin + TK - 1) / TK;
  g.kb = o.taps == 1 ? g.kpt : g.kpt * o.taps;
  const int last = (o.taps == 1 ? o.K : o.cin) - (g.kpt - 1) * TK;
  g.tail = (last + 15) / 16;
  // 64 rows and fewer: half of sixteen warps would have no rows, and the smaller block starts sooner (39 x 4096 x 1024: 5.0 and 5.3 us)
  const bool few = g.a_rows <= 64;
  L.shape = few ? GS_FEW : GS_WIDE;
  const int groups = few ? 2 : 4;
  // Sums in parts, where the tiles would cover less than half of the SMs and the reduction is long (the transformer's o / down projections of few rows): up to eight parts of
  // at least four k-blocks, as many as there are SMs for.  The parts are the order of the sums and their exactness: against float64, 39 x 1024 x 2048 is off by 2.4e-7 of its
  // norm in eight parts, by 4.7e-7 in four and by 2.1e-6 whole (the tensor pipe drops what lies below its accumulator's last place, once per product).  So they do not follow
  // what a launch costs, nor m_begin: a tail-only decode has to add the same partial sums in the same order.
  const int KT = (o.K + TK - 1) / TK;
  g.parts = 1;
  if ((o.ws || (o.reserved & 4)) && o.M <= 4 * TM && KT >= 8) {
    const int bn = o.N >= 64 ? 64 : 32;
    const int tiles = ((o.N + bn - 1) / bn) * ((o.M + TM - 1) / TM);
    const int sp = std::min(std::min(8, KT / 4), GP_SMS / std::max(1, tiles));
    if (sp > 1 && (long)KT * 430 - (long)((KT + sp - 1) / sp) * 440 > 3700 + 90L * std::min(o.M, TM)) {
      g.parts = sp;
      g.bn = bn;
      // Clusters of more than four CTAs, or of more than 128 in all, do not find room at the same time, nor beside the launches around them: their CTAs take two parts each
      // (eight parts in a prompt of 39 rows through 28 layers: clusters of eight 1203 us, of four 1125).  An SM's sixteen epilogue warps are of no use to a single tile: 73 x 1024 x
      // 3072 8.6 us, with eight 7.9; 200 rows 8.7 and 7.8.
      g.per = sp > 4 || tiles * sp > 128 ? 2 : 1;
      L.shape = GS_FEW;
    }
  }
  if (g.parts == 1) g.per = 1;
  g.splits = (g.parts + g.per - 1) / g.per;
  if (g.parts == 1) {
    // The width with the least waves x slower of (k loop, epilogue) + the other one once, in cycles.  A k-block takes what its instructions take (300), its four products
    // (two cycles a column), or its operand bytes at the 60 a cycle that L2 gives one SM.  The operand bytes of all tiles count a little by themselves: of two widths
    // that cost the same the wider one reads A less often (491520 x 96 x 96 with SnakeBeta: 16 columns 264 us, 96 columns 87).
    // Two CTAs per SM overlap their epilogues with each other's waits, but share the stages: only where a tile's few k-blocks fit in them (the same product over seven
    // taps: 143 us against 126).
    long best = -1;
    const long piece = epilogue_piece(o.flags);
    for (int cand = 256; cand >= 16; cand -= 16) {
      const int nt = (o.N + cand - 1) / cand;
      const int bn = std::min(256, ((o.N + nt - 1) / nt + 15) / 16 * 16), pieces = bn / 16;
      if (bn != cand && cand != 16) continue;
      const long tiles = (long)nt * g.mt, bytes = (g.a_rows + bn) * 128L, reads = tiles * g.kb * bytes / (4 * 60 * GP_SMS);
      auto cost = [&](const long rounds, const long k, const long e) { return rounds * std::max(k, e) + std::min(k, e) + reads; };
      const long c1 = cost((tiles + GP_SMS - 1) / GP_SMS, g.kb * std::max({300L, 2L * bn + 20, bytes / 60}), 700 + (pieces + groups - 1) / groups * groups * piece);
      const long c2 = cost(2 * ((tiles + 2 * GP_SMS - 1) / (2 * GP_SMS)), g.kb * std::max({160L, 2L * bn + 20, bytes / 60}), 500 + pieces * piece);
      const bool half = bn <= 128 && g.kb <= 4 && gp_stage_bytes(g.a_rows, bn) * std::max(2, g.kb) + GP_BAR_BYTES + 1024 <= GP_SMEM_HALF && c2 < c1;
      if (best < 0 || (half ? c2 : c1) < best) { best = half ? c2 : c1; g.bn = bn; L.shape = half ? GS_HALF : few ? GS_FEW : GS_WIDE; }
    }
  }
  g.nt = (o.N + g.bn - 1) / g.bn;
  g.acc_cols = 32;
  while (g.acc_cols < g.bn) g.acc_cols *= 2;
  g.early_b = o.reserved & 1;
  g.tries = o.reserved & 2 ? GP_TRIES_TEST : GP_TRIES;
  g.lost = o.reserved & 2 ? 0 : -1;
  // (few rows and a costly epilogue: 39 rows of gated units 8.3 -> 7.5 us; without one the extra meeting costs 1 us more than it saves)
  g.staged = g.parts > 1 || (g.mt == 1 && few && g.nt <= 2 * GP_SMS && (o.flags & (FQ3C_SWIGLU | FQ3C_GELU | FQ3C_SILU | FQ3C_SNAKE2)));
  g.vec16 = gemm_vec16(o) ? 1 : 0;
  const bool half = L.shape == GS_HALF;
  const int sb = gp_stage_bytes(g.a_rows, g.bn), tiles = g.mt * g.nt, n_kb = (g.kb + g.parts - 1) / g.parts * g.per;
  // The MMA reads 128 rows of A also where the box has fewer: the last stage's are inside the allocation.  One tile per CTA needs no more stages than k-blocks,
  // and a staged one's partial tiles have to fit in them.
  const int room = (half ? GP_SMEM_HALF : GP_SMEM_MAX) - 1024, fit = std::min((room - GP_BAR_BYTES) / sb, (room - T_A_BYTES) / sb + 1);
  const int part = (g.per * g.a_rows * gp_part_pitch(g.bn) * 4 + sb - 1) / sb;
  const bool once = g.staged || tiles <= GP_SMS * (half ? 2 : 1);
  g.stages = std::max(2, std::min(std::min(fit, 16), once ? std::max(n_kb, g.staged ? part : 0) : 16));
  L.smem = (size_t)std::max(g.stages * sb + GP_BAR_BYTES, (g.stages - 1) * sb + T_A_BYTES) + 1024;
  L.grid = g.staged ? (unsigned)(tiles * g.splits) : (unsigned)std::min(tiles, half ? 2 * GP_SMS : GP_SMS);
  return L;
}

// Which products go to the tensor pipe, and of those to the persistent kernel.  One k-block is enough: its vectorised epilogue beats the mma.sync kernel even at K = 96.
bool gemm_on_tc(const fq3c_op& o) {
  static const bool on = [] { const char* e = getenv("FQ3C_TCGEN05"); return e == nullptr || atoi(e) != 0; }();
  static const int min_k = [] { const char* e = getenv("FQ3C_TC5_MINK"); return e ? atoi(e) : TK; }();
  return on && o.N >= 16 && o.K >= min_k;
}
bool gemm_persists(const fq3c_op& o) { return gemm_on_tc(o) && (o.taps == 1 || o.cin % 16 == 0); }
// Columns behind N that are scratch make a width of whole 16-column pieces (B's missing rows arrive as zeros): the epilogue of any other width stores every
// entry by itself (1501 rows of 643 columns 31 us, of 656 9.3).
fq3c_op gemm_whole_pieces(const fq3c_op& o) {
  fq3c_op w = o;
  if ((o.reserved & 8) && !(o.flags & (FQ3C_BIAS | FQ3C_SCALE | FQ3C_RESID | FQ3C_SWIGLU | FQ3C_SNAKE2)) && o.ldc >= (o.N + 15) / 16 * 16 && !o.norm_out)
    w.N = (o.N + 15) / 16 * 16;
  return w;
}

// ---- attention of many queries on tcgen05 ---------------------------------------------------------------------------------------
bool attn_attrs_ready() {
  static bool done[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  auto room = [](auto kernel) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AT_SMEM) == cudaSuccess; };
  if (!done[dev])
    done[dev] = room(fq3c_attn_tc_kernel<AT_PROMPT, false>) && room(fq3c_attn_tc_kernel<AT_PROMPT, true>) && room(fq3c_attn_tc_kernel<AT_PLAIN, false>) &&
                room(fq3c_attn_tc_kernel<AT_PLAIN, true>) && room(fq3c_attn_tc_kernel<AT_CAP, false>) && room(fq3c_attn_tc_kernel<AT_CAP, true>) && room(fq3c_attn_tc_kernel<AT_DIST, false>);
  return done[dev];
}
// What the kernel's 8- and 16-byte accesses ask for.
bool attn_tc_takes(const AttnArgs& a, const int mode) {
  auto off = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; };
  return a.H % a.G == 0 && a.H / a.G <= 128 && a.ldk % 8 == 0 && a.ldv % 8 == 0 && a.ldq % 4 == 0 && a.ldo % (a.out_f32 ? 4 : 8) == 0 && !off(a.q) && !off(a.k) &&
         !off(a.v) && !off(a.out) && !(mode != AT_PROMPT && a.chunk > 0 && a.window > 0 && a.keep > 0) && attn_attrs_ready();
}
void launch_attn_tc(AttnArgs a, const int mode, cudaStream_t s, const bool after) {
  const int group = 128 / (a.H / a.G);
  const int rows_of = (a.M + group - 1) / group;      // row groups of a key head
  const long ctas = (long)rows_of * a.G;      // of one group each
  a.groups = ctas <= GP_SMS ? 1 : 2;
  a.two_from = a.ends = 0;
  // Up to twice as many row groups as SMs, and no window: a CTA's two groups are one from the end of the rows and one from their beginning, whose few tiles are among the other's, so
  // that no CTA has two of the longest (and the last one alone in the end).  Neighbours, ends (us of a layer, 16 heads over 4): 2048 rows with a cap 112 and 102, without 101 and 92,
  // 1700 behind 300 98 and 90; two layers of the talker (16 over 8), 1900 rows 366 and 354, 1500 318 and 307.  Under a window the neighbours share their tiles: 2048 rows of 256 63 and 69.
  // Of few more groups than SMs one to a CTA is faster still, as long as those that come last are short: blocks come up a key head behind the other, the longest group of each first, so
  // the last ones are the last key head's shortest, up to nine tenths of its groups (attention alone, one and ends, us: 1300 rows of 16 heads over 4, 16 groups over of a key head's 41, 36
  // and 42, with a cap 39 and 46; 1500, 40 of 47, 45 and 48; 1300 of 16 over 8, 20 of 21, 45 and 45; 1300 of 16 over 16, 28 of 11, 48 and 40).  Behind many positions all groups are long,
  // and the more so the more are over: with two_from the kernel then takes two (1300 of 16 over 4 behind 650 55 and 59, with a cap 61 and 69; of 16 over 8 73 and 62).  Over 170 sizes of
  // 15 head layouts at five positions each that is within 1 % of the better of the two on the average.
  if (a.groups == 2 && a.window <= 0 && a.chunk <= 0 && mode != AT_DIST && (ctas + 1) / 2 <= GP_SMS) {
    const long over = 10 * (ctas - GP_SMS);
    a.ends = 1;
    if (over <= 9L * rows_of) {
      a.groups = 1;
      if (a.p0) a.two_from = over <= 3L * rows_of ? a.M / 4 * 3 : mode == AT_CAP && over <= 7L * rows_of ? a.M / 2 : a.M / 4;
    }
  }
  const int per = a.groups * group;
  const dim3 grid((a.M + per - 1) / per, a.G);
  const bool ends = a.ends && (a.groups == 2 || a.two_from > 0);
  if (mode == AT_PROMPT && ends) launch_after(fq3c_attn_tc_kernel<AT_PROMPT, true>, grid, AT_THREADS, AT_SMEM, s, after, 1, a);
  else if (mode == AT_PROMPT) launch_after(fq3c_attn_tc_kernel<AT_PROMPT, false>, grid, AT_THREADS, AT_SMEM, s, after, 1, a);
  else if (mode == AT_PLAIN && ends) launch_after(fq3c_attn_tc_kernel<AT_PLAIN, true>, grid, AT_THREADS, AT_SMEM, s, after, 1, a);
  else if (mode == AT_PLAIN) launch_after(fq3c_attn_tc_kernel<AT_PLAIN, false>, grid, AT_THREADS, AT_SMEM, s, after, 1, a);
  else if (mode == AT_CAP && ends) launch_after(fq3c_attn_tc_kernel<AT_CAP, true>, grid, AT_THREADS, AT_SMEM, s, after, 1, a);
  else if (mode == AT_CAP) launch_after(fq3c_attn_tc_kernel<AT_CAP, false>, grid, AT_THREADS, AT_SMEM, s, after, 1, a);
  else launch_after(fq3c_attn_tc_kernel<AT_DIST, false>, grid, AT_THREADS, AT_SMEM, s, after, 1, a);
}

// FQ3C_ATTN_PREFILL=0: no kernel of its own for a prompt's attention (flags bit 0), nor one launch with the norm in front: the op by itself, as any other
bool prompt_kernels() {
  static const bool on = [] { const char* e = getenv("FQ3C_ATTN_PREFILL"); return e == nullptr || atoi(e) != 0; }();
  return on;
}

// ---- attention of few rows or a short window -----------------------------------------------------------------------------------
// What fq3c_attn_rows_kernel's vector accesses and shared memory ask for; grid.y is the head.  By itself it pays from nine keys in sight on: fq3c_attn_kernel fetches up to
// eight in two trips (16 heads of 64: 1 row 1.7 and 2.7 us, 8 rows 2.8 and 3.2, 9 rows 3.3 and 3.2; a window of 8, 33 rows 3.0 and 3.6, 600 rows 8.9 and 13.0), and from
// sixteen where the rows make more than one CTA per SM (600 rows, a window of 12 11.6 and 13.7, of 16 14.2 and 14.0).
bool attn_rows_takes(const fq3c_op& o, const bool prompt) {
  auto off = [](const void* p, int a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) != 0; };
  const int vec = o.i2 / 32;      // entries a lane moves at a time
  const long keys = std::min<long>(o.K, (long)o.M + o.taps);
  if (!prompt && (keys <= 8 || (keys < 16 && (long)((o.M + 15) / 16) * o.i1 > GP_SMS))) return false;
  return (o.i2 == 64 || o.i2 == 128) && o.i1 > 0 && o.i0 > 0 && o.i0 % o.i1 == 0 && o.i1 <= 65535 && o.K > 0 && o.taps >= 0 && o.lda % vec == 0 && o.ldc % vec == 0 &&
         !off(o.A, 2 * vec) && !off(o.C, 2 * vec) && attn_rows_plan(o, prompt).smem <= AR_SMEM_MAX && device_attrs_ready();
}
// The rows of a prompt from which its attention goes to tcgen05, where that takes the addresses.  Below them it is on the CUDA cores, by itself (fq3c_attn_prefill_kernel) or, where
// the rows are scratch, in one launch with the norm in front: the same bits, so that they do not depend on who else reads the rows.  One launch against the two with tcgen05:
// 64 rows of 16 heads over 8 8.0 and 10.8 us, 84 10.8 and 11.0, 90 11.0 and 11.0, 97 11.6 and 11.1, 112 14.5 and 11.3; of 32 over 8 64 rows 11.0 and 14.8 (the kernel by itself),
// 80 15.3 and 11.6; of 14 over 2 66 rows 8.8 and 10.3, 80 12.3 and 10.4 (15.2 by itself); of 8 112 rows 10.4 and 11.2, 128 12.5 and 11.6; of 4 112 rows 8.7 and 10.5.
bool attn_prompt_many(const fq3c_op& o) { return o.M > 112 || (o.M > 64 && (long)o.M * o.M * o.i0 > 115000); }
// `n` (q / k norm, rotation, cache rows) and the prompt attention `o` behind it, where the rows that `n` would rewrite are scratch to everyone else (reserved bit 0)
bool attn_rows_takes_prompt(const fq3c_op& n, const fq3c_op& o) {
  auto off = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 7) != 0; };
  return (n.reserved & 1) && o.kind == FQ3C_ATTN && (o.flags & 1) && o.A == n.A && o.lda == n.lda && o.M == n.M && o.i0 == n.i0 && o.i1 == n.i1 && o.i2 == 128 && o.taps == 0 && !o.p0 &&
         !attn_prompt_many(o) && !off(n.p0) && !off(n.p1) && !off(n.B) && !off(n.bias) && !off(n.C) && !off(n.C2) && attn_rows_takes(o, true);
}

// ---- sequence-model ops: launch logic ---------------------------------------------------------------------------------------
constexpr int SEQ_GEMM_FLAGS = FQ3C_BIAS | FQ3C_GELU | FQ3C_GELU_TANH | FQ3C_SIGMOID | FQ3C_OUT_F32 | FQ3C_F32 | FQ3C_NOROUND | FQ3C_A_F32 | FQ3C_SWIGLU | FQ3C_RELU2;

// a_f32 / b_f32: operand types.  exact: keep f32 A values as they are (CUDA cores) instead of rounding them onto the tensor cores.
// tail: ops that go on with the product's entries, where it takes the few-row kernel (gemv_tail).
bool takes_gemv(const SeqGemm& g) { return !g.seg && g.M <= 8 && (size_t)g.M * g.K * sizeof(float) <= 96 * 1024; }
int launch_seq_gemm(const SeqGemm& g, bool a_f32, bool b_f32, bool exact, int zcount, int row_tiles, cudaStream_t s, const bool after, const SeqTail* tail = nullptr) {
  if (g.flags & ~SEQ_GEMM_FLAGS) return fail("sequence product: unsupported epilogue flag");
  if (b_f32 && !a_f32) return fail("sequence product: f32 weights need f32 rows");
  if (g.M <= 0 || g.N <= 0 || g.K <= 0 || zcount <= 0) return 0;
  if ((g.flags & FQ3C_SWIGLU) && ((g.N & 1) || (g.flags & (FQ3C_BIAS | FQ3C_GELU | FQ3C_SIGMOID | FQ3C_RELU2)) || zcount != 1))
    return fail("sequence product: a gated-unit epilogue takes an even number of alternating gate / up columns and no other epilogue");
  const size_t gemv_smem = (size_t)g.M * g.K * sizeof(float);
  if (takes_gemv(g)) {
    static bool attr[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attr[dev]) {
      cudaFuncSetAttribute(fq3s_gemv_kernel<float, float>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
      cudaFuncSetAttribute(fq3s_gemv_kernel<float, bf16>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
      cudaFuncSetAttribute(fq3s_gemv_kernel<bf16, bf16>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
      cudaFuncSetAttribute(fq3s_gemv_kernel<float, float, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
      cudaFuncSetAttribute(fq3s_gemv_kernel<bf16, bf16, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
      attr[dev] = true;
    }
    dim3 grid((g.N + 7) / 8, 1, zcount);
    static const SeqTail none{};
    const int piece = b_f32 ? 4 : 8;
    const bool one = g.M == 1 && zcount == 1 && a_f32 == b_f32 && g.K % piece == 0 && g.ldb % piece == 0 && !((reinterpret_cast<uintptr_t>(g.A) | reinterpret_cast<uintptr_t>(g.B)) & 15);
    if (one) {
      const bool more = tail && tail->n > 0;
      if (more && b_f32) launch_seq(fq3s_gemv_kernel<float, float, true, true>, grid, 256, 0, s, after, 1, g, *tail);
      else if (more) launch_seq(fq3s_gemv_kernel<bf16, bf16, true, true>, grid, 256, 0, s, after, 1, g, *tail);
      else if (b_f32) launch_seq(fq3s_gemv_kernel<float, float, false, true>, grid, 256, 0, s, after, 1, g, none);
      else launch_seq(fq3s_gemv_kernel<bf16, bf16, false, true>, grid, 256, 0, s, after, 1, g, none);
      return 0;
    }
    if (tail && tail->n > 0 && a_f32 == b_f32) {
      if (b_f32) launch_seq(fq3s_gemv_kernel<float, float, true>, grid, 256, gemv_smem, s, after, 1, g, *tail);
      else launch_seq(fq3s_gemv_kernel<bf16, bf16, true>, grid, 256, gemv_smem, s, after, 1, g, *tail);
      return 0;
    }
    if (b_f32) launch_seq(fq3s_gemv_kernel<float, float>, grid, 256, gemv_smem, s, after, 1, g, none);
    else if (a_f32) launch_seq(fq3s_gemv_kernel<float, bf16>, grid, 256, gemv_smem, s, after, 1, g, none);
    else launch_seq(fq3s_gemv_kernel<bf16, bf16>, grid, 256, gemv_smem, s, after, 1, g, none);
    return 0;
  }
  if (g.seg && zcount == 1 && g.M <= 16 && (size_t)g.K * sizeof(float) <= 96 * 1024) {
    static bool gattr[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !gattr[dev]) {
      cudaFuncSetAttribute(fq3s_ggemv_kernel<float, float>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
      cudaFuncSetAttribute(fq3s_ggemv_kernel<float, bf16>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
      cudaFuncSetAttribute(fq3s_ggemv_kernel<bf16, bf16>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
      gattr[dev] = true;
    }
    dim3 grid((g.N + 7) / 8, g.M, 1);
    const size_t smem = (size_t)g.K * sizeof(float);
    if (b_f32) launch_seq(fq3s_ggemv_kernel<float, float>, grid, 256, smem, s, after, 1, g);
    else if (a_f32) launch_seq(fq3s_ggemv_kernel<float, bf16>, grid, 256, smem, s, after, 1, g);
    else launch_seq(fq3s_ggemv_kernel<bf16, bf16>, grid, 256, smem, s, after, 1, g);
    return 0;
  }
  // Experts on tcgen05: whole 16-byte pieces, each expert's weights behind the last one's, a k-block or more; at every number of rows that comes here faster than the mma.sync kernel
  // behind it, which keeps shorter sums (layers without a shared expert: 9 rows x 2 of 16 experts 48.5 and 41.3 us, 17 x 4 of 8 52.5 and 48.6, 100 x 1 of 16 54.6 and 46.4, 701 x 2 of 16
  // 81 and 51, 2048 x 4 of 32, 2048 wide, 527 and 245).
  if (g.seg && zcount == 1 && !a_f32 && !b_f32 && g.K >= TK && g.K % 8 == 0 && g.lda % 8 == 0 && g.ldb == g.K && g.b_estride == (long long)g.N * g.K && (long long)g.E * g.N < (1LL << 31) &&
      !((reinterpret_cast<uintptr_t>(g.A) | reinterpret_cast<uintptr_t>(g.B)) & 15) && device_attrs_ready()) {
    CUtensorMap tmB;
    if (make_map(&tmB, g.B, (uint64_t)g.K, (uint64_t)g.E * g.N, (uint64_t)g.K, GT_BN)) {
      const dim3 grid((g.N + GT_BN - 1) / GT_BN, (g.M + TM - 1) / TM + g.E);
      const bool glu = g.flags & FQ3C_SWIGLU;      // whole 32 bytes of a row (16 columns: of gated units 16 bytes)
      const int whole = !(reinterpret_cast<uintptr_t>(g.C) & (glu ? 15 : 31)) && g.ldc % (glu || (g.flags & FQ3C_OUT_F32) ? 8 : 16) == 0;
      if (glu) launch_seq(fq3s_ggemm_tc_kernel<true>, grid, GT_THREADS, GT_SMEM, s, after, 1, g, tmB, whole);
      else launch_seq(fq3s_ggemm_tc_kernel<false>, grid, GT_THREADS, GT_SMEM, s, after, 1, g, tmB, whole);
      return 0;
    }
  }
  // bf16 rows of whole 16-byte pieces (what its copies ask for), where the tcgen05 kernel has not taken them: experts with sums of 8 - 56, or weights that are not one behind the other
  if (!a_f32 && !b_f32 && !((g.K | g.lda | g.ldb | g.a_zstride) & 7) && !((g.b_zstride | g.b_estride) & 7) &&
      !((reinterpret_cast<uintptr_t>(g.A) | reinterpret_cast<uintptr_t>(g.B)) & 15)) {
    static bool pattr[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !pattr[dev]) {
      cudaFuncSetAttribute(fq3s_gemm_pipe_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, GQ_SMEM);
      cudaFuncSetAttribute(fq3s_gemm_pipe_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, GQ_SMEM);
      pattr[dev] = true;
    }
    const dim3 pgrid((g.N + GQ_BN - 1) / GQ_BN, (g.M + GQ_BM - 1) / GQ_BM + (g.seg ? g.E : 0), zcount);
    if (g.flags & FQ3C_SWIGLU) launch_seq(fq3s_gemm_pipe_kernel<true>, pgrid, 256, GQ_SMEM, s, after, 1, g);
    else launch_seq(fq3s_gemm_pipe_kernel<false>, pgrid, 256, GQ_SMEM, s, after, 1, g);
    return 0;
  }
  // tall bf16 products (many rows per block / per expert, wide enough outputs): 128 x 128 tiles
  if (!b_f32 && !(a_f32 && exact) && g.N >= 128 && (g.seg ? g.M >= 96 * g.E : g.M >= 256)) {
    dim3 grid128((g.N + 127) / 128, (g.M + 127) / 128 + (g.seg ? g.E : 0), zcount);
    const bool glu = (g.flags & FQ3C_SWIGLU) != 0;
    if (a_f32 && glu) launch_seq(fq3s_gemm_mma128_kernel<float, true>, grid128, 256, 0, s, after, 1, g);
    else if (a_f32) launch_seq(fq3s_gemm_mma128_kernel<float>, grid128, 256, 0, s, after, 1, g);
    else if (glu) launch_seq(fq3s_gemm_mma128_kernel<bf16, true>, grid128, 256, 0, s, after, 1, g);
    else launch_seq(fq3s_gemm_mma128_kernel<bf16>, grid128, 256, 0, s, after, 1, g);
    return 0;
  }
  dim3 grid((g.N + 63) / 64, row_tiles, zcount);
  // rows of whole 16-byte pieces: the pipelined product (the other one stages element by element)
  const bool pieces = !((g.K | g.lda | g.ldb | g.a_zstride) & 3) && !((g.b_zstride | g.b_estride) & 3) && !((reinterpret_cast<uintptr_t>(g.A) | reinterpret_cast<uintptr_t>(g.B)) & 15);
  if (b_f32 && pieces) {
    static bool attr[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attr[dev]) {
      cudaFuncSetAttribute(fq3s_gemm_f32_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, fg_smem(1));
      cudaFuncSetAttribute(fq3s_gemm_f32_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, fg_smem(4));
      attr[dev] = true;
    }
    // Four groups of threads where the tiles are a single wave of blocks, one group from there on (us, one and four; tiles x k): 64 rows of 1536 x 1024 (24 x 1024) 41.0 and 37.5, 384 (144)
    // 42.0 and 38.1, 500 (192) 70.3 and 73.9, 2048 (768) 198 and 218; 700 rows of 1024 x 64 (176 x 64) 10.2 and 12.1, 100 (32) 7.7 and 7.0.
    if ((long)grid.x * grid.y * grid.z <= GP_SMS) launch_seq(fq3s_gemm_f32_kernel<4>, grid, 256, fg_smem(4), s, after, 1, g);
    else launch_seq(fq3s_gemm_f32_kernel<1>, grid, 256, fg_smem(1), s, after, 1, g);
  }
  else if (b_f32) launch_seq(fq3s_gemm_kernel<float, float>, grid, 256, 0, s, after, 1, g);
  else if (a_f32 && exact) launch_seq(fq3s_gemm_kernel<float, bf16>, grid, 256, 0, s, after, 1, g);
  else if (a_f32 && (g.flags & FQ3C_SWIGLU)) launch_seq(fq3s_gemm_mma_kernel<float, true>, grid, 128, 0, s, after, 1, g);
  else if (a_f32) launch_seq(fq3s_gemm_mma_kernel<float>, grid, 128, 0, s, after, 1, g);
  else if (g.flags & FQ3C_SWIGLU) launch_seq(fq3s_gemm_mma_kernel<bf16, true>, grid, 128, 0, s, after, 1, g);
  else launch_seq(fq3s_gemm_mma_kernel<bf16>, grid, 128, 0, s, after, 1, g);
  return 0;
}

// threads of a block that works on one row of n entries: with a few rows (decoding) one per entry, so that the row's loads are one round trip
int row_threads(int rows, int n, int many) { return rows <= 8 ? std::max(32, std::min(1024, (n + 31) / 32 * 32)) : many; }

// the convolution over many rows of whole 16-byte pieces: four columns and TC_ROWS rows per thread
bool tconv_vec_ok(const fq3c_op& o) {
  return o.M >= 64 && o.taps > 1 && o.taps <= 8 && o.N % 4 == 0 && o.lda % 4 == 0 && o.ldc % 4 == 0 && !(o.flags & FQ3C_RESID) &&
         !((reinterpret_cast<uintptr_t>(o.A) | reinterpret_cast<uintptr_t>(o.C) | reinterpret_cast<uintptr_t>(o.p0) | reinterpret_cast<uintptr_t>(o.p1)) & 15) &&
         (!(o.flags & FQ3C_SILU) || o.i0 % 4 == 0);
}

// returns 1 when the kind is not a sequence-model op
const char* entry_op_error(const fq3c_op& o) {      // of DYT, DEPTH_MIX and XIELU
  if (o.kind == FQ3C_DYT) {
    if (!o.A || !o.scale || !o.C || ((o.flags & FQ3C_RESID) && !o.res)) return "dyt: missing operand";
    if (o.norm_out && (!o.norm_w || !(o.flags & FQ3C_OUT_F32))) return "dyt: a chained norm needs its weights and an f32 result";
  } else if (o.kind == FQ3C_DEPTH_MIX) {
    if (o.i0 < 1 || !o.A || !o.p0 || !o.C || (o.norm_out && !o.norm_w)) return "depth_mix: missing operand";
  } else if (!o.A || !o.p0 || !o.C) {
    return "xielu: missing operand";
  }
  return nullptr;
}
// Which of the ops behind a product of few rows go on with its entries in the same launch.  As launches of their own they see everything that the ones in front wrote; in one launch
// entry (m, n) sees what itself did, and nothing about other entries.  So no op may write what the product reads, and where an op writes what another one of them reads or
// writes, it has to be the same entry: the same rows (address, pitch, type), or memory apart.
void gemv_tail(const fq3c_op& o, const SeqGemm& g, const fq3c_op* next, const int n_next, SeqTail& t) {
  t.n = 0;
  if ((o.flags & ~(FQ3C_OUT_F32 | FQ3C_NOROUND | FQ3C_F32)) || !(o.flags & FQ3C_OUT_F32) || !takes_gemv(g) || o.N < 1 || o.K < 1) return;
  struct Rows { uintptr_t at, end; long pitch; int size; };
  const int M = o.M, N = o.N;
  auto rows = [&](const void* p, const long ld, const int size, const int cols) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    return p ? Rows{a, a + (uintptr_t)((long)(M - 1) * ld + cols) * size, M > 1 ? ld : 0, size} : Rows{0, 0, 0, 0};
  };
  auto apart = [](const Rows& a, const Rows& b) { return a.end <= b.at || b.end <= a.at; };
  auto same = [](const Rows& a, const Rows& b) { return a.at == b.at && a.pitch == b.pitch && a.size == b.size; };
  const int in = o.flags & FQ3C_F32 ? 4 : 2;
  const Rows from[2] = {rows(o.A, o.lda, in, o.K), Rows{reinterpret_cast<uintptr_t>(o.B), reinterpret_cast<uintptr_t>(o.B) + (uintptr_t)N * o.K * in, 0, in}};
  Rows reads[80], writes[8], fixed[16];      // entries read and written so far; parameters, which nothing may write
  int nr = 0, nw = 0, nf = 0;
  writes[nw++] = rows(o.C, o.ldc, 4, N);
  for (int k = 0; k < 2 && k < n_next; ++k) {
    const fq3c_op& q = next[k];
    const bool first = k == 0 && (q.kind == FQ3C_DYT || q.kind == FQ3C_XIELU), mix = k == 1 && next[0].kind == FQ3C_DYT && q.kind == FQ3C_DEPTH_MIX && q.i0 <= 64;
    if (!(first || mix) || q.M != M || q.N != N || entry_op_error(q)) return;
    if (first && (q.A != o.C || (M > 1 && q.lda != o.ldc))) return;
    int r = nr, w = nw, f = nf;
    auto param = [&](const void* p, const int n) {
      if (p) fixed[f++] = Rows{reinterpret_cast<uintptr_t>(p), reinterpret_cast<uintptr_t>(p) + (uintptr_t)n * 4, 0, 4};
    };
    if (mix) {
      for (int j = 0; j < q.i0; ++j) reads[r++] = rows(reinterpret_cast<const float*>(q.A) + (size_t)j * (size_t)q.K, q.lda, 4, N);
      param(q.p0, q.i0);
    } else if (q.kind == FQ3C_XIELU) {
      param(q.p0, 2);
    } else {
      if (q.flags & FQ3C_RESID) reads[r++] = rows(q.res, q.ldr, 4, N);
      param(q.scale, N);
      param(q.bias, N);
    }
    // What it reads is asked for in front of the product's sums, so nothing in front of it in this launch may have written that; but a mix gets the norm's result by hand.
    for (int a = 0; a < nw; ++a)
      for (int b = nr; b < r; ++b)
        if (!apart(writes[a], reads[b]) && !(mix && (next[0].flags & FQ3C_OUT_F32) && same(reads[b], rows(next[0].C, next[0].ldc, 4, N)) && same(writes[a], reads[b]))) return;
    const bool out32 = mix || (q.flags & FQ3C_OUT_F32);
    writes[w++] = rows(q.C, q.ldc, out32 ? 4 : 2, N);
    if (q.kind != FQ3C_XIELU && out32 && q.C2) writes[w++] = rows(q.C2, q.ldc, 2, N);
    if (q.kind != FQ3C_XIELU && out32 && q.norm_out) { writes[w++] = rows(q.norm_out, q.norm_ld, q.flags & FQ3C_F32 ? 4 : 2, N); param(q.norm_w, 2 * N); }
    for (int a = 0; a < w; ++a) {
      if (a >= nw && (!apart(writes[a], from[0]) || !apart(writes[a], from[1]))) return;
      for (int b = 0; b < r; ++b) if (!apart(writes[a], reads[b]) && !same(writes[a], reads[b])) return;
      for (int b = 0; b < a; ++b) if (!apart(writes[a], writes[b]) && !same(writes[a], writes[b])) return;
      for (int b = 0; b < f; ++b) if (!apart(writes[a], fixed[b])) return;
    }
    nr = r; nw = w; nf = f;
    t.op[k] = q;
    t.n = k + 1;
    if (q.kind == FQ3C_XIELU) return;
  }
}
// ---- attention over a cache, few rows ------------------------------------------------------------------------------------------
bool rot_append_ok(const fq3c_op& o) {
  return o.A && o.i0 >= 0 && o.i1 >= 0 && o.i2 >= 1 && o.taps >= 0 && !(o.taps & 1) && o.taps <= o.i2 && (o.taps == 0 || o.B) && (o.i1 == 0 || (o.C && (o.cin <= 0 || o.C2)));
}
const char* cache_attn_error(const fq3c_op& o) {
  if (o.i0 < 1 || o.i1 < 1 || o.i0 % o.i1 || o.i2 < 1 || o.cin < 1 || !o.A || !o.B || !o.p1 || !o.C) return "cache_attn: bad configuration";
  const int splits = std::max(1, o.m_begin);
  if (o.tap_off[1] > 0 && (o.K < 1 || !o.C2 || !o.norm_out || o.bias || o.tap_off[0] > 0 || o.a_rows > 0))
    return "cache_attn: pooled blocks go with a window and their pooled rows, not with kept first positions, a chunked mask or a distance penalty";
  if (splits > 64) return "cache_attn: at most 64 key splits";
  if (splits > 1 && (!o.ws || o.ws_bytes < (int64_t)o.M * o.i0 * splits * (o.cin + 2) * 4)) return "cache_attn: workspace too small for the splits";
  return nullptr;
}
// Which calls of few rows go to fq3s_attn_few_kernel: what its accesses and variants ask for, and as many keys as the eight CTAs of a cluster walk faster than up to 64 do with a second
// launch to merge them.  That is told by the keys that a row may see (the window, or what 32 per split say; 64 splits say nothing, so without a window 2016): one row behind 2000 positions,
// 4 heads a key head, 17.6 us by itself and 17.9 here; 8 heads a key head behind 1000 15.0 and 10.8, behind 2000 20.6 and 24; one head a key head behind 8000 63 and 24 (16 heads), 27 and 19 (one).
// And as many clusters (rows x key heads) as are on the GPU at a time, or nearly: 15 of the variants with one CTA an SM, 30 of those with two, which win with two rounds of them as well
// (8 rows of 32 heads over 8 behind 200 23.1 and 15.9; of 64 over 16, four rounds, 27.0 and 29.0; heads of 64, 32 over 32, behind 30 10.4 and 26.7).  Of the others two rounds are worth
// it where the kernels beside take two launches and the keys are few, or heads of 128 share them (32-bit caches: four rows of 8 heads over 8 behind 500 12.4 and 10.9, behind 1000 14.2 and
// 15.1, behind 4000 29 and 39; four of 32 over 8 behind 1980 45.2 and 39.0; two of 64 over 16 behind 30, one launch, 11.7 and 13.5).
bool attn_few_takes(const fq3c_op& o) {
  const int splits = std::max(1, o.m_begin);
  const long keys = o.K > 0 && o.a_rows <= 0 ? o.K : o.tap_off[0] > 0 ? o.tap_off[0] : splits < 64 ? 32L * splits : 1L << 30;
  auto off = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; };
  const int V = o.flags & FQ3C_F32 ? 4 : 8, HG = o.i1 > 0 ? o.i0 / o.i1 : 0;
  const long clusters = (long)o.M * o.i1;
  const bool fits = V == 8 && HG <= 4 ? clusters <= (o.i2 == 128 ? 64 : 32) : clusters <= 15 || (clusters <= 32 && splits > 1 && (keys <= 512 || (HG > 1 && o.i2 == 128)));
  return fits && o.M <= AF_ROWS && (HG == 1 || keys <= (HG == 8 ? 1024 : 2048)) && (o.i2 == 64 || o.i2 == 128) && o.cin == o.i2 && o.i0 >= 1 && o.i1 >= 1 && o.i0 % o.i1 == 0 && (HG <= 4 || HG == 8) && o.i1 <= 65535 && o.tap_off[1] <= 0 &&
         o.A && o.B && o.p1 && o.C && o.ldr % V == 0 && o.taps % V == 0 && !off(o.B) && !off(o.p1);
}
// `r` (rotation, cache rows) and the attention `o` of the same single row behind it
bool attn_few_takes_rot(const fq3c_op& r, const fq3c_op& o) {
  if (o.kind != FQ3C_CACHE_ATTN || r.M != 1 || o.M != 1 || r.m_begin > 0 || !attn_few_takes(o) || o.A != r.A || o.i0 != r.i0 || o.i2 != r.i2 || o.p0 != r.p0 || ((o.flags ^ r.flags) & FQ3C_F32)) return false;
  if (r.i1 > 0 && (r.i1 != o.i1 || r.cin != o.cin || r.C != o.B || r.ldc != o.ldr || r.C2 != o.p1 || r.ldr != o.taps || r.C == r.C2)) return false;
  // What one CTA writes early, others still read: the turned queries, the finished outputs
  auto apart = [](const void* a, const long na, const void* b, const long nb) {
    const uintptr_t x = reinterpret_cast<uintptr_t>(a), y = reinterpret_cast<uintptr_t>(b);
    return !a || !b || x + na <= y || y + nb <= x;
  };
  const long nq = 4L * o.i0 * o.i2, nk = 4L * r.i1 * r.i2, nout = (long)o.i0 * o.cin * (o.flags & FQ3C_OUT_F32 ? 4 : 2), ngate = 4L * (o.flags & FQ3C_GATE_ENTRY ? o.i0 * o.cin : o.i0);
  const float* krow = reinterpret_cast<const float*>(r.res ? r.res : r.A);
  const void* written[2] = {o.A, o.C};
  const long bytes[2] = {nq, nout};
  for (int w = 0; w < 2; ++w) {
    if (r.i1 > 0 && (!apart(written[w], bytes[w], krow + r.K, nk) || !apart(written[w], bytes[w], krow + r.a_rows, nk))) return false;
    if (!apart(written[w], bytes[w], o.res, ngate) || !apart(written[w], bytes[w], o.scale, 4L * o.i0) || !apart(written[w], bytes[w], o.bias, 8L * o.i0)) return false;
    if (!apart(written[w], bytes[w], r.B, 2L * r.taps) || !apart(written[w], bytes[w], r.p1, 2L * r.taps) || !apart(written[w], bytes[w], r.scale, 4L * r.i2) || !apart(written[w], bytes[w], r.bias, 4L * r.i2) ||
        !apart(written[w], bytes[w], o.p0, 4)) return false;
  }
  return apart(o.A, nq, o.C, nout);
}
template <typename TC, int D, bool ROT>
void launch_attn_few(const fq3c_op& o, const fq3c_op& r, cudaStream_t s, const bool after) {
  const int HG = o.i0 / o.i1;
  const dim3 grid(AF_RANKS, (unsigned)o.i1, (unsigned)o.M);
  const size_t smem = sizeof(float) * af_floats(HG, D);
  if (HG == 1) launch_seq(fq3s_attn_few_kernel<TC, D, 1, ROT>, grid, AF_WARPS * 32, smem, s, after, AF_RANKS, o, r);
  else if (HG == 2) launch_seq(fq3s_attn_few_kernel<TC, D, 2, ROT>, grid, AF_WARPS * 32, smem, s, after, AF_RANKS, o, r);
  else if (HG == 3) launch_seq(fq3s_attn_few_kernel<TC, D, 3, ROT>, grid, AF_WARPS * 32, smem, s, after, AF_RANKS, o, r);
  else if (HG == 4) launch_seq(fq3s_attn_few_kernel<TC, D, 4, ROT>, grid, AF_WARPS * 32, smem, s, after, AF_RANKS, o, r);
  else launch_seq(fq3s_attn_few_kernel<TC, D, 8, ROT>, grid, AF_WARPS * 32, smem, s, after, AF_RANKS, o, r);
}
// r: the ROT_APPEND in front that goes with it, or null
void launch_attn_few(const fq3c_op& o, const fq3c_op* r, cudaStream_t s, const bool after) {
  const bool f32 = (o.flags & FQ3C_F32) != 0;
  const fq3c_op& q = r ? *r : o;
  if (r) {
    if (f32) { if (o.i2 == 64) launch_attn_few<float, 64, true>(o, q, s, after); else launch_attn_few<float, 128, true>(o, q, s, after); }
    else { if (o.i2 == 64) launch_attn_few<bf16, 64, true>(o, q, s, after); else launch_attn_few<bf16, 128, true>(o, q, s, after); }
  } else {
    if (f32) { if (o.i2 == 64) launch_attn_few<float, 64, false>(o, q, s, after); else launch_attn_few<float, 128, false>(o, q, s, after); }
    else { if (o.i2 == 64) launch_attn_few<bf16, 64, false>(o, q, s, after); else launch_attn_few<bf16, 128, false>(o, q, s, after); }
  }
}

// ---- one decoded row of a delta-rule layer -------------------------------------------------------------------------------------
// c, o, n: convolution, recurrence and norm of one row that one launch can do: the convolution's channels are the head's queries, keys and values as they stand, the norm is per head,
// with a gate behind it or none.  In one launch a CTA reads what another one may have written already, so no op may write what it or an op in front of it reads, but for the entries it
// hands on: the convolution's result, the read-out, and the state, which is read and written by the same lanes.
bool delta_row_takes(const fq3c_op& c, const fq3c_op& o, const fq3c_op& n) {
  if (c.kind != FQ3C_TCONV || o.kind != FQ3C_MSTATE_SCAN || n.kind != FQ3C_GNORM || c.M != 1 || o.M != 1 || n.M != 1 || o.taps != 0) return false;
  const int H = o.i0, G = o.i1, dk = o.i2, dv = o.cin;
  if (H < 1 || G < 1 || H % G || H > 65535 || (dk != 64 && dk != 128 && dk != 256) || dv < 8 || dv > 128 || dv % 8) return false;
  if (!c.A || !c.B || !c.C || c.taps < 2 || c.taps > DS_TAPS || !c.p0 || !c.p1 || !(c.flags & FQ3C_OUT_F32) || ((c.flags & FQ3C_BIAS) && !c.bias)) return false;
  if (!o.A || !o.p0 || !o.C || !o.C2 || !o.res || !o.scale || !o.ws || o.ws_bytes < (int64_t)mstate_ws_cols(H, G, dk, true) * 4) return false;
  if (o.A != c.C || o.K != G * dk || o.a_rows != 2 * G * dk || c.N != 2 * G * dk + H * dv) return false;
  if (n.i0 != H || n.N != H * dv || n.A != o.C || !n.C || (n.flags & ~(FQ3C_GATE_POST | FQ3C_SIGMOID | FQ3C_OUT_F32)) || ((n.flags & FQ3C_GATE_POST) && !n.p1) || n.bias || n.C2 || n.p0) return false;
  struct Span { uintptr_t at, end; };
  auto span = [](const void* p, const int64_t bytes) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    return p ? Span{a, a + (uintptr_t)bytes} : Span{0, 0};
  };
  auto apart = [](const Span& a, const Span& b) { return a.end <= b.at || b.end <= a.at; };
  const int64_t conv = 4LL * c.N, hist = conv * (c.taps - 1), state = 4LL * H * dk * dv, out = 4LL * H * dv;
  const Span cv = span(c.C, conv), next = span(c.p1, hist), y = span(o.C, out), st = span(o.p0, state), st2 = span(o.C2, state), yn = span(n.C, n.flags & FQ3C_OUT_F32 ? out : out / 2);
  const Span reads[] = {span(c.A, conv), span(c.B, conv * c.taps), span(c.flags & FQ3C_BIAS ? c.bias : nullptr, conv), span(c.p0, hist), span(reinterpret_cast<const float*>(o.res) + o.col_mod, 4LL * H),
                        span(reinterpret_cast<const float*>(o.res) + o.m_begin, 4LL * H), span(o.scale, 4LL * H), span(o.bias, 4LL * H), span(n.scale, 4LL * (n.i2 > 0 ? n.i2 : n.N)),
                        span(n.flags & FQ3C_GATE_POST ? n.p1 : nullptr, out)};
  const Span writes[] = {cv, next, y, st2, yn};
  for (const Span& w : writes) {
    for (const Span& r : reads) if (!apart(w, r)) return false;
    if (!apart(w, st) && !(w.at == st2.at && w.end == st2.end && st.at == st2.at)) return false;
  }
  for (int a = 0; a < 5; ++a)
    for (int b = 0; b < a; ++b) if (!apart(writes[a], writes[b])) return false;
  return true;
}
void launch_delta_row(const fq3c_op& c, const fq3c_op& o, const fq3c_op& n, cudaStream_t s, const bool after) {
  const dim3 grid(DS_RANKS, (unsigned)o.i0);
  if (o.i2 == 64) launch_seq(fq3s_delta_row_kernel<8>, grid, 128, 0, s, after, DS_RANKS, c, o, n);
  else if (o.i2 == 128) launch_seq(fq3s_delta_row_kernel<16>, grid, 128, 0, s, after, DS_RANKS, c, o, n);
  else launch_seq(fq3s_delta_row_kernel<32>, grid, 128, 0, s, after, DS_RANKS, c, o, n);
}

int seq_run(const fq3c_op& o, cudaStream_t s, bool after) {
  switch (o.kind) {
    case FQ3C_EMBED:
      if (!o.A || !o.B || !o.C) return fail("embed: missing operand");
      if (o.i0 > 1 && o.K < o.N) return fail("embed: copies need a stride of at least N elements");
      if (o.C2 && o.ldr < o.N * std::max(o.i1, 1)) return fail("embed: the operand copies do not fit their pitch");
      if (o.flags & FQ3C_F32) launch_seq(fq3s_embed_kernel<float>, o.M, row_threads(o.M, o.N, 128), 0, s, after, 1, o);
      else launch_seq(fq3s_embed_kernel<bf16>, o.M, row_threads(o.M, o.N, 128), 0, s, after, 1, o);
      return 0;
    case FQ3C_TCONV:
      if (o.taps < 1 || !o.A || !o.B || !o.C || (o.taps > 1 && (!o.p0 || !o.p1))) return fail("tconv: missing operand");
      if (tconv_vec_ok(o)) {
        const dim3 grid((o.N / 4 + 127) / 128, (o.M + o.taps - 1 + TC_ROWS - 1) / TC_ROWS);
        if (o.taps <= 4) launch_seq(fq3s_tconv_vec_kernel<4>, grid, 128, 0, s, after, 1, o);
        else launch_seq(fq3s_tconv_vec_kernel<8>, grid, 128, 0, s, after, 1, o);
        return 0;
      }
      launch_seq(fq3s_tconv_kernel, dim3((o.N + 255) / 256, o.M + o.taps - 1), 256, 0, s, after, 1, o);
      return 0;
    case FQ3C_GNORM:
      if (o.i0 < 1 || o.N % o.i0 || ((o.flags & FQ3C_RESID) && !o.res)) return fail("gnorm: groups must divide N");
      if ((o.flags & (FQ3C_GATE_PRE | FQ3C_GATE_POST)) && !o.p1) return fail("gnorm: gate rows required");
      // many (row, group) pairs of a size a warp holds in registers, 16-byte rows: a warp per pair
      if ((int64_t)o.M * o.i0 >= 1024 && o.N / o.i0 % 4 == 0 && o.N / o.i0 <= 4 * 32 * GN_VECS && o.i2 % 4 == 0 && !((o.lda | o.ldc | o.ldr) & 3) &&
          (!(o.flags & (FQ3C_GATE_PRE | FQ3C_GATE_POST)) || o.i1 % 4 == 0) &&
          !((reinterpret_cast<uintptr_t>(o.A) | reinterpret_cast<uintptr_t>(o.C) | reinterpret_cast<uintptr_t>(o.C2) | reinterpret_cast<uintptr_t>(o.p1) |
             reinterpret_cast<uintptr_t>(o.res) | reinterpret_cast<uintptr_t>(o.scale)) & 15)) {
        const unsigned blocks = (unsigned)(((int64_t)o.M * o.i0 + 3) / 4);
        const int vecs = (o.N / o.i0 + 127) / 128;
        if (vecs == 1) launch_seq(fq3s_gnorm_warp_kernel<1>, blocks, 128, 0, s, after, 1, o);
        else if (vecs == 2) launch_seq(fq3s_gnorm_warp_kernel<2>, blocks, 128, 0, s, after, 1, o);
        else launch_seq(fq3s_gnorm_warp_kernel<GN_VECS>, blocks, 128, 0, s, after, 1, o);
        return 0;
      }
      launch_seq(fq3s_gnorm_kernel, dim3(o.M, o.i0), row_threads(o.M, o.N / o.i0, 128), 0, s, after, 1, o);
      return 0;
    case FQ3C_POLYNORM:
      if (!o.p0) return fail("polynorm: coefficients required");
      launch_seq(fq3s_polynorm_kernel, o.M, 256, 0, s, after, 1, o);
      return 0;
    case FQ3C_BDGEMM: {
      if (o.i0 < 1 || o.i1 < 1 || o.i2 < 1 || o.cin < 1) return fail("bdgemm: bad block shape");
      SeqGemm g{};
      g.A = o.A; g.B = o.B; g.bias = reinterpret_cast<const float*>(o.bias); g.C = o.C;
      g.M = o.M; g.N = o.i2; g.K = o.cin; g.lda = o.lda; g.ldb = o.cin; g.ldc = o.ldc; g.flags = o.flags;
      g.a_mod = o.i1; g.a_zstride = o.cin; g.c_zstride = o.i2; g.b_zstride = (long long)o.i2 * o.cin;
      return launch_seq_gemm(g, true, (o.flags & FQ3C_F32) != 0, (o.flags & FQ3C_NOROUND) != 0, o.i0, (o.M + 63) / 64, s, after);
    }
    case FQ3C_GGEMM: {
      if (o.i0 < 1 || !o.p0) return fail("ggemm: segment starts required");
      SeqGemm g{};
      g.A = o.A; g.B = o.B; g.bias = nullptr; g.C = o.C;
      g.M = o.M; g.N = o.N; g.K = o.K; g.lda = o.lda; g.ldb = o.K; g.ldc = o.ldc; g.flags = o.flags & ~FQ3C_BIAS;
      g.a_mod = 1; g.seg = reinterpret_cast<const int*>(o.p0); g.rows = reinterpret_cast<const int*>(o.p1); g.E = o.i0;
      g.b_estride = (long long)o.N * o.K; g.lost = (o.reserved >> 1) & 1;
      if (o.flags & FQ3C_SWIGLU) { g.rs_w = reinterpret_cast<const float*>(o.scale); g.rs_pos = reinterpret_cast<const int*>(o.ws); g.rs_top = o.i1; }
      if (g.rs_pos && (!g.rs_w || !g.rows || g.rs_top < 1)) return fail("ggemm: a router's weights need the choices' places, the row list and the choice count");
      const bool f32 = (o.flags & FQ3C_F32) != 0;
      return launch_seq_gemm(g, f32 || (o.flags & FQ3C_A_F32), f32, false, 1, (o.M + 63) / 64 + o.i0, s, after);
    }
    case FQ3C_LRU_SCAN: {
      if (!o.A || !o.B || !o.res || !o.scale || !o.p0 || !o.C || !o.C2) return fail("lru_scan: missing operand");
      int chunks = 1;
      if (o.M >= 256 && o.ws) chunks = std::min<int64_t>(std::min(64, o.M / 64), o.ws_bytes / ((int64_t)2 * o.N * 4));
      chunks = std::max(chunks, 1);
      const int per = (o.M + chunks - 1) / chunks;
      dim3 grid((o.N + 127) / 128, chunks);
      if (chunks > 1) {
        launch_seq(fq3s_lru_fold_kernel, grid, 128, 0, s, after, 1, o, chunks, per, reinterpret_cast<float*>(o.ws));
        count_launches(1);
      }
      launch_seq(fq3s_lru_scan_kernel, grid, 128, 0, s, after, 1, o, chunks, per, reinterpret_cast<const float*>(o.ws));
      return 0;
    }
    case FQ3C_ROUTER: {
      if (o.i0 < 1 || o.i0 > o.N || o.i1 < 1 || o.i1 > 64 || o.N % o.i1 || o.i2 < 1 || !o.C || !o.C2) return fail("router: bad configuration");
      int tpb = (int)std::min<size_t>(128, (48 * 1024) / ((size_t)o.N * 8));
      if (tpb < 1) return fail("router: too many experts");
      if (tpb >= 32) tpb &= ~31;
      if (o.ws && (o.M != 1 || o.i0 > 16 || !o.p0 || !o.p1 || o.K < 0)) return fail("router: grouping in the same launch takes one token with at most 16 choices");
      launch_seq(fq3s_router_kernel, (o.M + tpb - 1) / tpb, tpb, (size_t)o.N * tpb * 8, s, after, 1, o);
      return 0;
    }
    case FQ3C_MOE_SORT: {
      if (o.i1 < 1 || !o.A || !o.C || !o.C2 || !o.ws) return fail("moe_sort: missing operand");
      const int warps = std::min(std::min(32, ((48 * 1024) / 4 - o.i1 - 1) / o.i1), std::max(1, (o.M * o.i0 + 31) / 32));
      if (warps < 1) return fail("moe_sort: too many experts");
      launch_seq(fq3s_moe_sort_kernel, 1, warps * 32, (size_t)(o.i1 + 1 + warps * o.i1) * 4, s, after, 1, o);
      return 0;
    }
    case FQ3C_MOE_COMBINE:
      if (!o.A || !o.B || !o.p0 || !o.ws || !o.C) return fail("moe_combine: missing operand");
      launch_seq(fq3s_moe_combine_kernel, o.M, 256, 0, s, after, 1, o);
      return 0;
    case FQ3C_COMMIT:
      launch_seq(fq3s_commit_kernel, dim3(o.M, 8), 256, 0, s, after, 1, reinterpret_cast<const long long*>(o.A), reinterpret_cast<int*>(o.C), o.i0);
      return 0;
    case FQ3C_LATENT_ATTN: {
      if (o.i0 < 1 || o.i1 < 1 || !o.A || !o.B || !o.C) return fail("latent_attn: missing operand");
      if (o.cin < 0 || (o.cin > 0 && (!o.p1 || o.taps < o.i0 * o.cin)) || o.a_rows < 0 || (o.res && o.m_begin < o.i0))
        return fail("latent_attn: bad score-only part, window or gate");
      const int Dk = o.i1 + o.cin;      // a cache row: latent columns, then the score-only ones
      const int splits = std::max(1, o.K);
      if (splits > 64) return fail("latent_attn: at most 64 key splits");
      if (splits > 1 && (!o.ws || o.ws_bytes < (int64_t)o.M * o.i0 * splits * (o.i1 + 2) * 4)) return fail("latent_attn: workspace too small for the splits");
      // bf16 cache with a rank the MMA tiles divide: the tensor-core kernel (FQ3S_ATTN_MMA=0: CUDA cores everywhere)
      static int use_mma = -1;
      if (use_mma < 0) { const char* e6 = getenv("FQ3S_ATTN_MMA"); use_mma = (e6 == nullptr || atoi(e6) != 0) ? 1 : 0; }
      const int RS = (o.i1 + 255) / 256;
      if (use_mma && !(o.flags & FQ3C_F32) && RS <= 2 && o.i1 % 16 == 0 && o.i1 % (8 * RS) == 0 && o.cin % 16 == 0 && o.ldr % 8 == 0 &&
          !(reinterpret_cast<uintptr_t>(o.B) & 15)) {
        const int TJ = Dk > 256 ? 32 : 64;
        // one query (decoding): a block per split with all its warps on that query, R cut into up to eight 16-column-aligned slices
        int QB = LM_QB, RSk = RS;
        if (o.M == 1) {
          QB = 1;
          while (RSk < 8 && o.i1 % (32 * RSk) == 0) RSk *= 2;
        }
        const size_t smem = (size_t)(QB * 16 + 2 * TJ) * (Dk + 8) * 2;   // queries + two key tiles
        const int nt_o = (o.i1 / RSk) / 8;
        static bool mattr[64] = {};
        int dev = 0;
        cudaGetDevice(&dev);
        if (dev >= 0 && dev < 64 && !mattr[dev]) {
          cudaFuncSetAttribute(fq3s_latent_attn_mma_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
          cudaFuncSetAttribute(fq3s_latent_attn_mma_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
          cudaFuncSetAttribute(fq3s_latent_attn_mma_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
          mattr[dev] = true;
        }
        dim3 grid((o.M + QB - 1) / QB, (o.i0 + 15) / 16, splits);
        const int nth = 32 * QB * RSk;
        const bool early = after && blocks_fit(grid);
        if (nt_o <= 8) launch_seq(fq3s_latent_attn_mma_kernel<8>, grid, nth, smem, s, early, 1, o, RSk, splits, TJ, QB);
        else if (nt_o <= 16) launch_seq(fq3s_latent_attn_mma_kernel<16>, grid, nth, smem, s, early, 1, o, RSk, splits, TJ, QB);
        else launch_seq(fq3s_latent_attn_mma_kernel<32>, grid, nth, smem, s, early, 1, o, RSk, splits, TJ, QB);
        if (splits > 1) {
          launch_seq(fq3s_latent_merge_kernel, dim3(o.M, o.i0), 128, 0, s, after, 1, o, splits);
          count_launches(1);
        }
        return 0;
      }
      int HG = std::max(1, std::min(o.i0, o.i2 > 0 ? o.i2 : o.i0));
      while (HG > 1 && latent_attn_smem(HG, o.i1, o.cin) > 160 * 1024) --HG;
      const size_t smem = latent_attn_smem(HG, o.i1, o.cin);
      if (smem > 200 * 1024) return fail("latent_attn: latent rank too large for shared memory");
      static bool attr[64] = {};
      int dev = 0;
      cudaGetDevice(&dev);
      if (dev >= 0 && dev < 64 && !attr[dev]) {
        cudaFuncSetAttribute(fq3s_latent_attn_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        cudaFuncSetAttribute(fq3s_latent_attn_kernel<bf16>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        attr[dev] = true;
      }
      dim3 grid(o.M, (o.i0 + HG - 1) / HG, splits);
      // (never early: a token of four such layers in 32 bits behind 1000 positions 595 us, early 692)
      if (o.flags & FQ3C_F32) launch_seq(fq3s_latent_attn_kernel<float>, grid, 256, smem, s, false, 1, o, HG, splits);
      else launch_seq(fq3s_latent_attn_kernel<bf16>, grid, 256, smem, s, false, 1, o, HG, splits);
      if (splits > 1) {
        launch_seq(fq3s_latent_merge_kernel, dim3(o.M, o.i0), 128, 0, s, after, 1, o, splits);
        count_launches(1);
      }
      return 0;
    }
    case FQ3C_DYT:
    case FQ3C_DEPTH_MIX:
    case FQ3C_XIELU: {
      if (const char* e = entry_op_error(o)) return fail(e);
      const dim3 grid((o.N + 255) / 256, o.M);
      if (o.kind == FQ3C_DYT) launch_seq(fq3s_dyt_kernel, grid, 256, 0, s, after, 1, o);
      else if (o.kind == FQ3C_DEPTH_MIX) launch_seq(fq3s_depth_mix_kernel, grid, 256, 0, s, after, 1, o);
      else launch_seq(fq3s_xielu_kernel, grid, 256, 0, s, after, 1, o);
      return 0;
    }
    case FQ3C_ROT_APPEND: {
      if (!rot_append_ok(o)) return fail("rot_append: bad configuration");
      if (o.m_begin > 0 && (o.i1 < 1 || o.cin < 1 || !o.norm_out || !o.ws || !o.p0)) return fail("rot_append: pooled blocks need both caches, their pooled rows and a position");
      // what the flat kernel holds: no norm, no temperature, no pooled rows.  (Like the other one it turns queries in place while it reads keys and values: those lie in columns of their own.)
      if (o.M > 8 && o.m_begin <= 0 && !o.scale && !o.bias && !(o.flags & FQ3C_UNIT) && !(o.f3 > 0.f) && o.taps <= 4096) {
        const size_t smem = sizeof(float2) * (o.taps / 2);
        if (o.flags & FQ3C_F32) launch_seq(fq3s_rot_append_flat_kernel<float>, o.M, 256, smem, s, after, 1, o);
        else launch_seq(fq3s_rot_append_flat_kernel<bf16>, o.M, 256, smem, s, after, 1, o);
        return 0;
      }
      const int rth = o.M <= 8 ? std::max(256, std::min(1024, 32 * (o.i0 + o.i1))) : 256;      // few rows: a warp per head
      if (o.m_begin > 0 && o.M == 1 && (o.flags & FQ3C_F32)) launch_seq(fq3s_rot_append_kernel<float, true, 1024>, 1, rth, 0, s, after, 1, o);
      else if (o.m_begin > 0 && o.M == 1) launch_seq(fq3s_rot_append_kernel<bf16, true, 1024>, 1, rth, 0, s, after, 1, o);
      else if (rth > 256 && (o.flags & FQ3C_F32)) launch_seq(fq3s_rot_append_kernel<float, false, 1024>, o.M, rth, 0, s, after, 1, o);
      else if (rth > 256) launch_seq(fq3s_rot_append_kernel<bf16, false, 1024>, o.M, rth, 0, s, after, 1, o);
      else if (o.flags & FQ3C_F32) launch_seq(fq3s_rot_append_kernel<float>, o.M, 256, 0, s, after, 1, o);
      else launch_seq(fq3s_rot_append_kernel<bf16>, o.M, 256, 0, s, after, 1, o);
      if (o.m_begin > 0 && o.M > 1) {
        const dim3 grid(o.M / o.m_begin + 1, (o.i1 * std::max(o.i2, o.cin) + 255) / 256, 2);
        if (o.flags & FQ3C_F32) launch_seq(fq3s_pool_append_kernel<float>, grid, 256, 0, s, after, 1, o);
        else launch_seq(fq3s_pool_append_kernel<bf16>, grid, 256, 0, s, after, 1, o);
        count_launches(1);
      }
      return 0;
    }
    case FQ3C_CACHE_ATTN: {
      if (const char* e = cache_attn_error(o)) return fail(e);
      const int splits = std::max(1, o.m_begin), HG = o.i0 / o.i1;
      const bool pool = o.tap_off[1] > 0;
      if (attn_few_takes(o)) {
        launch_attn_few(o, nullptr, s, after);
        return 0;
      }
      // bf16 cache and a prompt portion: the tensor-core kernels (FQ3S_ATTN_MMA=0: CUDA cores everywhere).  Heads of 128 on tcgen05 from 9 rows on: against the
      // mma.sync kernel 9 rows of 16 heads over 4 behind 2000 positions 185 and 51 us, 1000 rows 303 and 76; only short portions at the very
      // beginning are slower (33-64 rows at position 0: 10.7-11.5 and 12.9), and the host does not know where a portion begins.
      static int use_mma = -1;
      if (use_mma < 0) { const char* e7 = getenv("FQ3S_ATTN_MMA"); use_mma = (e7 == nullptr || atoi(e7) != 0) ? 1 : 0; }
      if (use_mma && !(o.flags & FQ3C_F32) && o.M > 8 && o.i2 == 128 && o.cin == 128 && !pool) {
        AttnArgs a{};
        a.q = o.A; a.k = reinterpret_cast<const bf16*>(o.B); a.v = reinterpret_cast<const bf16*>(o.p1);
        a.tries = o.reserved & 2 ? GP_TRIES_TEST : GP_TRIES; a.lost = (o.reserved >> 1) & 1;
        a.ldq = o.lda; a.ldk = o.ldr; a.ldv = o.taps; a.H = o.i0; a.G = o.i1; a.M = o.M; a.p0 = reinterpret_cast<const int*>(o.p0);
        a.scale = o.f0; a.cap = o.f1; a.mult = o.f2; a.window = o.K; a.keep = o.a_rows; a.chunk = o.tap_off[0];
        a.r12 = reinterpret_cast<const float*>(o.bias); a.sink = reinterpret_cast<const float*>(o.scale); a.gate = reinterpret_cast<const float*>(o.res);
        a.gate_ld = o.col_mod; a.entry = o.res && (o.flags & FQ3C_GATE_ENTRY); a.out_f32 = (o.flags & FQ3C_OUT_F32) != 0; a.out = o.C; a.ldo = o.ldc;
        const int mode = o.bias ? AT_DIST : o.f1 > 0.f ? AT_CAP : AT_PLAIN;
        if (attn_tc_takes(a, mode)) {
          launch_attn_tc(a, mode, s, false);      // (many rows)
          return 0;
        }
      }
      // rows per block: a multiple of 16 (one MMA tile per warp) that whole queries fill, i.e. that the group size divides
      int mma_rows = 0;
      for (const int w : {4, 8, 3, 6, 5, 7, 2, 1})
        if (!mma_rows && (16 * w) % HG == 0) mma_rows = 16 * w;
      if (use_mma && mma_rows && !(o.flags & FQ3C_F32) && o.M > 8 && o.i2 % 16 == 0 && o.i2 <= 256 &&
          o.cin % 16 == 0 && o.cin <= 128 && o.ldr % 8 == 0 && o.taps % 8 == 0 && !(reinterpret_cast<uintptr_t>(o.B) & 15) &&
          !(reinterpret_cast<uintptr_t>(o.p1) & 15) && (!pool || !((reinterpret_cast<uintptr_t>(o.C2) | reinterpret_cast<uintptr_t>(o.norm_out)) & 15)) &&
          (o.ldc % 2 == 0 || (o.flags & FQ3C_OUT_F32))) {
        static bool mattr[64] = {};
        int dev = 0;
        cudaGetDevice(&dev);
        if (dev >= 0 && dev < 64 && !mattr[dev]) {
          cudaFuncSetAttribute(fq3s_cache_attn_mma_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
          cudaFuncSetAttribute(fq3s_cache_attn_mma_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
          cudaFuncSetAttribute(fq3s_cache_attn_mma_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
          cudaFuncSetAttribute(fq3s_cache_attn_mma_kernel<4, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
          cudaFuncSetAttribute(fq3s_cache_attn_mma_kernel<8, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
          cudaFuncSetAttribute(fq3s_cache_attn_mma_kernel<16, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
          mattr[dev] = true;
        }
        const int ROWS = (mma_rows == 64 && o.M * HG >= 8192 && cache_attn_mma_smem(128, o.i2, o.cin) <= 110 * 1024) ? 128 : mma_rows, QBLK = ROWS / HG;
        dim3 grid((o.M + QBLK - 1) / QBLK, o.i1);
        const size_t smem = cache_attn_mma_smem(ROWS, o.i2, o.cin);
        if (pool) {
          if (o.cin <= 32) launch_seq(fq3s_cache_attn_mma_kernel<4, true>, grid, ROWS * 2, smem, s, after, 1, o, ROWS);
          else if (o.cin <= 64) launch_seq(fq3s_cache_attn_mma_kernel<8, true>, grid, ROWS * 2, smem, s, after, 1, o, ROWS);
          else launch_seq(fq3s_cache_attn_mma_kernel<16, true>, grid, ROWS * 2, smem, s, after, 1, o, ROWS);
        } else if (o.cin <= 32) launch_seq(fq3s_cache_attn_mma_kernel<4>, grid, ROWS * 2, smem, s, after, 1, o, ROWS);
        else if (o.cin <= 64) launch_seq(fq3s_cache_attn_mma_kernel<8>, grid, ROWS * 2, smem, s, after, 1, o, ROWS);
        else launch_seq(fq3s_cache_attn_mma_kernel<16>, grid, ROWS * 2, smem, s, after, 1, o, ROWS);
        return 0;
      }
      // an f32 cache and more than a few queries, heads of 128: 32-row blocks with pipelined tiles
      if ((o.flags & FQ3C_F32) && o.M > 8 && o.i2 == 128 && o.cin == 128 && !pool && HG <= FA_R && !((o.lda | o.ldr | o.taps) & 3) &&
          !((reinterpret_cast<uintptr_t>(o.A) | reinterpret_cast<uintptr_t>(o.B) | reinterpret_cast<uintptr_t>(o.p1)) & 15)) {
        static bool fattr[64] = {};
        int dev = 0;
        cudaGetDevice(&dev);
        if (dev >= 0 && dev < 64 && !fattr[dev]) {
          cudaFuncSetAttribute(fq3s_attn_f32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FA_SMEM);
          fattr[dev] = true;
        }
        const int QB = FA_R / HG;
        launch_seq(fq3s_attn_f32_kernel, dim3((o.M + QB - 1) / QB, o.i1, splits), 128, FA_SMEM, s, after, 1, o);
        if (splits > 1) {
          launch_seq(fq3s_cache_attn_merge_kernel, dim3(o.M, o.i0), 128, 0, s, after, 1, o, splits);
          count_launches(1);
        }
        return 0;
      }
      int QB = o.M == 1 ? 1 : std::max(1, std::min(std::min(16, o.M), 16 / HG)), TJ = 32;
      while (cache_attn_smem(QB * HG, TJ, o.i2, o.cin) > 200 * 1024 && QB > 1) QB >>= 1;
      while (cache_attn_smem(QB * HG, TJ, o.i2, o.cin) > 200 * 1024 && TJ > 4) TJ >>= 1;
      const size_t smem = cache_attn_smem(QB * HG, TJ, o.i2, o.cin);
      if (smem > 200 * 1024) return fail("cache_attn: heads too large for shared memory");
      static bool attr[64] = {};
      int dev = 0;
      cudaGetDevice(&dev);
      if (dev >= 0 && dev < 64 && !attr[dev]) {
        cudaFuncSetAttribute(fq3s_cache_attn_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        cudaFuncSetAttribute(fq3s_cache_attn_kernel<bf16>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        cudaFuncSetAttribute(fq3s_cache_attn_kernel<float, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        cudaFuncSetAttribute(fq3s_cache_attn_kernel<bf16, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        attr[dev] = true;
      }
      dim3 grid((o.M + QB - 1) / QB, o.i1, splits);
      const bool early = after && blocks_fit(grid);
      if (pool && (o.flags & FQ3C_F32)) launch_seq(fq3s_cache_attn_kernel<float, true>, grid, 256, smem, s, early, 1, o, QB, TJ, splits);
      else if (pool) launch_seq(fq3s_cache_attn_kernel<bf16, true>, grid, 256, smem, s, early, 1, o, QB, TJ, splits);
      else if (o.flags & FQ3C_F32) launch_seq(fq3s_cache_attn_kernel<float>, grid, 256, smem, s, early, 1, o, QB, TJ, splits);
      else launch_seq(fq3s_cache_attn_kernel<bf16>, grid, 256, smem, s, early, 1, o, QB, TJ, splits);
      if (splits > 1) {
        launch_seq(fq3s_cache_attn_merge_kernel, dim3(o.M, o.i0), 128, 0, s, after, 1, o, splits);
        count_launches(1);
      }
      return 0;
    }
    case FQ3C_HYPER: {
      if (o.i0 < 1 || o.i0 > HY_MAX || !o.A || (o.i0 > 1 && o.K < o.N) || (o.res && (!o.p0 || !o.p1)) || (o.C && !o.bias) || (!o.C && !o.res))
        return fail("hyper: 1 to 16 streams; mixing and write weights with a sublayer output; read weights with an output");
      if ((size_t)o.N * 4 > 200 * 1024) return fail("hyper: row too wide for shared memory");
      static bool hattr[64] = {};
      int dev = 0;
      cudaGetDevice(&dev);
      if (dev >= 0 && dev < 64 && !hattr[dev]) {
        cudaFuncSetAttribute(fq3s_hyper_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        cudaFuncSetAttribute(fq3s_hyper_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        hattr[dev] = true;
      }
      if (o.i0 <= 8) launch_seq(fq3s_hyper_kernel<8>, o.M, 256, (size_t)o.N * 4, s, after, 1, o);
      else launch_seq(fq3s_hyper_kernel<16>, o.M, 256, (size_t)o.N * 4, s, after, 1, o);
      return 0;
    }
    case FQ3C_GLU:
      if (!o.A || !o.C || o.N < 1) return fail("glu: missing operand");
      launch_seq(fq3s_glu_kernel, dim3((o.N + 255) / 256, o.M), 256, 0, s, after, 1, o);
      return 0;
    case FQ3C_MSTATE_SCAN: {
      if (o.i0 < 1 || o.i1 < 1 || o.i0 % o.i1 || o.i2 < 1 || o.cin < 1 || !o.A || !o.p0 || !o.C || !o.C2) return fail("mstate_scan: bad configuration");
      if (o.taps < 0 || o.taps > 6)
        return fail("mstate_scan: taps selects the delta rule (0), the state-space scan (1), a decay per key channel (2), a fixed decay per head (3), a forget gate "
                    "per channel (4), exponential gates (5) or the delta rule with a decay per key channel (6)");
      if (o.i2 > 512) return fail("mstate_scan: at most 512 state rows per head");
      if (o.taps <= 1) {
        if (!o.res || !o.scale || !o.ws) return fail("mstate_scan: raw projections, A_log and a workspace required");
        if (o.ws_bytes < (int64_t)o.M * mstate_ws_cols(o.i0, o.i1, o.i2, o.taps == 0) * 4) return fail("mstate_scan: workspace too small");
      } else if (o.taps == 2) {
        if (!o.res || !o.ws || !o.B || o.i1 != o.i0 || o.m_begin < 1 || o.m_begin > MS_MAX_RANK)
          return fail("mstate_scan: channel decays need their latent rows, the up-projection (inner size 1 .. 1024), a workspace and one key head per head");
        if (o.ws_bytes < (int64_t)o.M * mstate_decay_cols(o.i0, o.i2) * 4) return fail("mstate_scan: workspace too small");
      } else if (o.taps == 6) {
        if (!o.res || !o.ws || !o.B || !o.scale || !o.bias || o.tap_off[0] < 1 || o.tap_off[0] > MS_MAX_RANK || o.tap_off[2] < 0 || o.tap_off[2] > MS_MAX_RANK ||
            (o.tap_off[2] > 0 && (!o.p1 || !o.norm_out || o.norm_ld < o.i0 * o.cin)))
          return fail("mstate_scan: channel decays of the delta rule need their latent rows, the up-projections (inner sizes 1 .. 1024), A_log, dt_bias and a workspace");
        if (o.ws_bytes < (int64_t)o.M * mstate_cdelta_cols(o.i0, o.i1, o.i2) * 4) return fail("mstate_scan: workspace too small");
      } else if (o.taps == 3) {
        if (!o.scale || o.i1 != o.i0) return fail("mstate_scan: fixed decays need one value and one key head per head");
      } else {
        if (!o.scale || o.i1 != o.i0 || (o.taps == 5 && (!o.res || !o.p1 || !o.norm_out || o.norm_ld < o.i0 || !(o.f1 > 0.f))))
          return fail("mstate_scan: gates need their bounds or maxima, one key head per head, and exponential gates a cap and room for the divisors");
        const int cols = o.taps == 4 ? mstate_gate_cols(o.i0, o.i2) : mstate_max_cols(o.i0);
        if (o.M > MS_CH && (!o.ws || o.ws_bytes < (int64_t)o.M * cols * 4)) return fail("mstate_scan: workspace too small");
      }
      // delta rules over many rows: blocks of tokens, when the workspace holds their records
      const bool blocks = (o.taps == 0 || o.taps == 6) && o.M >= CD_MIN_ROWS && o.i2 <= CD_MAX_DK &&
                          o.ws_bytes / 4 >= cd_ws_floats(o.M, o.i0, o.i2, o.taps == 6) && !(reinterpret_cast<uintptr_t>(o.ws) & 15);
      if (o.taps == 4 && o.M > MS_CH) {
        launch_seq(fq3s_mstate_gate_kernel, dim3(o.M, (o.i0 * o.i2 + 255) / 256), 256, 0, s, after, 1, o);
        count_launches(1);
      } else if (o.taps == 5 && o.M > MS_CH) {
        launch_seq(fq3s_mstate_max_kernel, o.i0, MM_THREADS, 0, s, after, 1, o);
        count_launches(1);
      } else if (o.taps == 6) {
        const int per = cdelta_prep_channels(o.M == 1 ? 1 : MS_PREP_ROWS);
        const dim3 grid((o.M + MS_PREP_ROWS - 1) / MS_PREP_ROWS, (o.i0 * o.i2 + per - 1) / per + (o.tap_off[2] > 0 ? (o.i0 * o.cin + per - 1) / per : 0) + (blocks ? 0 : 1));
        const size_t smem = sizeof(float) * MS_PREP_ROWS * (size_t)std::max(o.tap_off[0], o.tap_off[2]);
        if (o.M == 1) launch_seq(fq3s_mstate_cdelta_prep_kernel<1>, grid, 256, smem, s, after, 1, o, false);
        else launch_seq(fq3s_mstate_cdelta_prep_kernel<MS_PREP_ROWS>, grid, 256, smem, s, after, 1, o, blocks);
        count_launches(1);
      } else if (o.taps < 3 && !blocks) {
        launch_seq(fq3s_mstate_prep_kernel, o.taps == 2 ? (o.M + MS_PREP_ROWS - 1) / MS_PREP_ROWS : o.M, 128, 0, s, after, 1, o);
        count_launches(1);
      }
      static bool sattr[64] = {};
      int dev = 0;
      cudaGetDevice(&dev);
      if (dev >= 0 && dev < 64 && !sattr[dev]) {
        cudaFuncSetAttribute(fq3s_mstate_scan_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
        cudaFuncSetAttribute(fq3s_mstate_scan_kernel<32, 2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
        cudaFuncSetAttribute(fq3s_mstate_scan_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
        cudaFuncSetAttribute(fq3s_mstate_scan_kernel<64, 2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
        cudaFuncSetAttribute(fq3s_mstate_scan_kernel<16, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, 72 * 1024);
        cudaFuncSetAttribute(fq3s_mstate_scan_kernel<16, 3, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 72 * 1024);
        cudaFuncSetAttribute(fq3s_mstate_scan_kernel<32, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, 120 * 1024);
        cudaFuncSetAttribute(fq3s_mstate_scan_kernel<32, 3, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 120 * 1024);
        cudaFuncSetAttribute(fq3s_mstate_scan_kernel<64, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, 216 * 1024);
        cudaFuncSetAttribute(fq3s_mstate_scan_kernel<64, 3, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 216 * 1024);
        cudaFuncSetAttribute(fq3s_mstate_scan_kernel<16, 3, false, 1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 72 * 1024);
        cudaFuncSetAttribute(fq3s_mstate_scan_kernel<32, 3, false, 1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 120 * 1024);
        cudaFuncSetAttribute(fq3s_mstate_scan_kernel<64, 3, false, 1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 216 * 1024);
        sattr[dev] = true;
      }
      if (blocks) {
        static bool battr[64] = {};
        if (dev >= 0 && dev < 64 && !battr[dev]) {
          cudaFuncSetAttribute(fq3s_cdelta_record_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, cd_record_smem(CD_MAX_DK, true));
          cudaFuncSetAttribute(fq3s_cdelta_record_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, cd_record_smem(CD_MAX_DK, false));
          cudaFuncSetAttribute(fq3s_cdelta_walk_kernel<8, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, CD_WALK_SMEM);
          cudaFuncSetAttribute(fq3s_cdelta_walk_kernel<8, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, CD_WALK_SMEM);
          cudaFuncSetAttribute(fq3s_cdelta_walk_kernel<16, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, CD_WALK_SMEM);
          cudaFuncSetAttribute(fq3s_cdelta_walk_kernel<16, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, CD_WALK_SMEM);
          cudaFuncSetAttribute(fq3s_cdelta_walk_kernel<16, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, CD_WALK_SMEM);
          battr[dev] = true;
        }
        const dim3 rgrid((o.M + CD_C - 1) / CD_C, o.i0);
        if (o.taps == 6) launch_seq(fq3s_cdelta_record_kernel<true>, rgrid, CD_REC_THREADS, cd_record_smem(o.i2, true), s, after, 1, o);
        else launch_seq(fq3s_cdelta_record_kernel<false>, rgrid, CD_REC_THREADS, cd_record_smem(o.i2, false), s, after, 1, o);
        count_launches(1);
        // narrow state tiles while they do not outnumber the SMs, wide ones otherwise and for few state rows
        const bool narrow = o.i2 > 64 && o.i0 * ((o.cin + 7) / 8) <= 148;
        const dim3 grid((o.cin + (narrow ? 7 : 15)) / (narrow ? 8 : 16), o.i0);
        const int dvt = narrow ? 8 : 16, ring = cd_walk_floats(dvt, o.i2, 4) * 4 <= CD_WALK_SMEM ? 4 : 3;
        const size_t wsm = (size_t)cd_walk_floats(dvt, o.i2, ring) * 4;
        if (narrow && o.i2 <= 128) launch_seq(fq3s_cdelta_walk_kernel<8, 1>, grid, CD_WALK_THREADS, wsm, s, after, 1, o, ring);
        else if (narrow) launch_seq(fq3s_cdelta_walk_kernel<8, 2>, grid, CD_WALK_THREADS, wsm, s, after, 1, o, ring);
        else if (o.i2 <= 64) launch_seq(fq3s_cdelta_walk_kernel<16, 1>, grid, CD_WALK_THREADS, wsm, s, after, 1, o, ring);
        else if (o.i2 <= 128) launch_seq(fq3s_cdelta_walk_kernel<16, 2>, grid, CD_WALK_THREADS, wsm, s, after, 1, o, ring);
        else launch_seq(fq3s_cdelta_walk_kernel<16, 4>, grid, CD_WALK_THREADS, wsm, s, after, 1, o, ring);
        return 0;
      }
      // Long runs of a recurrence whose decays do not depend on the state: pieces walked twice (see the kernel), when the caller's
      // workspace has room behind the per-row coefficients for the pieces' states and decay products.
      const int sv = o.taps == 5 ? o.cin + 1 : o.cin;      // state columns (exponential gates: the normaliser is one more)
      const int coef = o.taps == 3 ? 0 : o.taps == 5 ? mstate_max_cols(o.i0) : o.taps == 4 ? mstate_gate_cols(o.i0, o.i2)
                     : o.taps == 2 ? mstate_decay_cols(o.i0, o.i2) : mstate_ws_cols(o.i0, o.i1, o.i2, false);
      const int64_t base = ((int64_t)o.M * coef + 3) & ~(int64_t)3;
      const int64_t per_piece = (int64_t)o.i0 * o.i2 * (sv + 1);
      int pieces = 1, piece = o.M;
      if (o.taps != 0 && o.taps != 6 && o.M >= 512 && o.ws) {
        pieces = (int)std::min<int64_t>(std::min(16, o.M / 128), (o.ws_bytes / 4 - base) / per_piece);
        if (pieces >= 2) {
          piece = (((o.M + pieces - 1) / pieces) + MS_CH - 1) / MS_CH * MS_CH;
          pieces = (o.M + piece - 1) / piece;
        }
        if (pieces < 2) { pieces = 1; piece = o.M; }
      }
      float* X = pieces > 1 ? reinterpret_cast<float*>(o.ws) + base : nullptr;
      float* P = pieces > 1 ? X + (int64_t)pieces * o.i0 * o.i2 * sv : nullptr;
      const int bound = o.i2 <= 32 ? 4 : o.i2 <= 64 ? 8 : o.i2 <= 128 ? 16 : o.i2 <= 256 ? 32 : 64;      // state rows a lane holds
      const bool cdelta = o.taps == 6, three = o.taps == 2 || o.taps == 4 || cdelta, gated = o.taps == 4 || o.taps == 5;
      const int cpt = pieces > 1 && bound <= 16 ? 2 : 1;                                                    // state columns a lane holds
      auto walk = [&](const int phase, const int nz) {
        const dim3 grid((sv + cpt * MS_COLS - 1) / (cpt * MS_COLS), o.i0, nz);
        const size_t smem = sizeof(float) * 2 * mstate_buf_floats(bound, three ? 3 : 2, cpt);
#define FQ3S_WALK(RPT, CPT) \
    if (three && gated) launch_seq(fq3s_mstate_scan_kernel<RPT, 3, true, CPT>, grid, 128, smem, s, after, 1, o, phase, piece, X, P); \
    else if (three) launch_seq(fq3s_mstate_scan_kernel<RPT, 3, false, CPT>, grid, 128, smem, s, after, 1, o, phase, piece, X, P); \
    else if (gated) launch_seq(fq3s_mstate_scan_kernel<RPT, 2, true, CPT>, grid, 128, smem, s, after, 1, o, phase, piece, X, P); \
    else launch_seq(fq3s_mstate_scan_kernel<RPT, 2, false, CPT>, grid, 128, smem, s, after, 1, o, phase, piece, X, P);
        if (cdelta) switch (bound) {
          case 4: launch_seq(fq3s_mstate_scan_kernel<4, 3, false, 1, true>, grid, 128, smem, s, after, 1, o, phase, piece, X, P); break;
          case 8: launch_seq(fq3s_mstate_scan_kernel<8, 3, false, 1, true>, grid, 128, smem, s, after, 1, o, phase, piece, X, P); break;
          case 16: launch_seq(fq3s_mstate_scan_kernel<16, 3, false, 1, true>, grid, 128, smem, s, after, 1, o, phase, piece, X, P); break;
          case 32: launch_seq(fq3s_mstate_scan_kernel<32, 3, false, 1, true>, grid, 128, smem, s, after, 1, o, phase, piece, X, P); break;
          default: launch_seq(fq3s_mstate_scan_kernel<64, 3, false, 1, true>, grid, 128, smem, s, after, 1, o, phase, piece, X, P); break;
        }
        else if (cpt == 2) switch (bound) {
          case 4: FQ3S_WALK(4, 2) break;
          case 8: FQ3S_WALK(8, 2) break;
          default: FQ3S_WALK(16, 2) break;
        }
        else switch (bound) {
          case 4: FQ3S_WALK(4, 1) break;
          case 8: FQ3S_WALK(8, 1) break;
          case 16: FQ3S_WALK(16, 1) break;
          case 32: FQ3S_WALK(32, 1) break;
          default: FQ3S_WALK(64, 1) break;
        }
#undef FQ3S_WALK
      };
      if (pieces == 1) {
        walk(0, 1);
        return 0;
      }
      walk(1, pieces - 1);
      const int64_t n = (int64_t)o.i0 * o.i2 * sv;
      launch_seq(fq3s_mstate_carry_kernel, (unsigned)((n + 255) / 256), 256, 0, s, after, 1, o, pieces, X, P, sv);
      walk(3, pieces);
      count_launches(2);
      return 0;
    }
    case FQ3C_SUM_NORM: {
      if (o.i0 < 1 || !o.A || !o.p0 || !o.C || (o.i0 > 1 && o.K < o.N) || ((o.flags & FQ3C_POST) && (!o.norm_w || o.C2))) return fail("sum_norm: missing operand");
      if ((size_t)o.N * 4 > 200 * 1024) return fail("sum_norm: row too wide for shared memory");
      static bool nattr[64] = {};
      int dev = 0;
      cudaGetDevice(&dev);
      if (dev >= 0 && dev < 64 && !nattr[dev]) {
        cudaFuncSetAttribute(fq3s_sum_norm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        nattr[dev] = true;
      }
      // rows of whole 16-byte pieces that a block of 256 holds in registers
      if (o.N % 4 == 0 && o.N <= 1024 * SN_VECS && !((o.lda | o.ldc | o.norm_ld | o.K) & 3) && !o.C2 &&
          !((reinterpret_cast<uintptr_t>(o.A) | reinterpret_cast<uintptr_t>(o.C) | reinterpret_cast<uintptr_t>(o.norm_out) | reinterpret_cast<uintptr_t>(o.norm_w) |
            reinterpret_cast<uintptr_t>(o.bias)) & 15)) {
        launch_seq(fq3s_sum_norm_vec_kernel, o.M, std::max(32, std::min(256, (o.N / 4 + 31) / 32 * 32)), 0, s, after, 1, o);
        return 0;
      }
      launch_seq(fq3s_sum_norm_kernel, o.M, row_threads(o.M, o.N, 256), (size_t)o.N * 4, s, after, 1, o);
      return 0;
    }
    default: return 1;
  }
}

}  // namespace

extern "C" {

int fq3c_abi_version(void) { return 12; }
const char* fq3c_last_error(void) { return g_err.c_str(); }
int64_t fq3c_launch_count(void) { return g_launches.load(); }
int fq3c_wait_errors(void) {
  int v = 0;
  return cudaMemcpyFromSymbol(&v, seq_wait_error, sizeof v) == cudaSuccess ? v : -1;
}

// The host's error words, one per device, made before a device's first launch (also when that one is captured: the calls are exempt from the capture).
static std::atomic<volatile int*> wait_words[64];
static bool wait_word_ready() {
  static std::mutex making;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  if (wait_words[dev].load(std::memory_order_acquire)) return true;
  std::lock_guard<std::mutex> lock(making);
  if (wait_words[dev].load(std::memory_order_relaxed)) return true;
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) return false;
  int* p = nullptr;
  cudaStream_t s = nullptr;
  bool ok = cudaHostAlloc(reinterpret_cast<void**>(&p), 64, cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess;
  if (ok) {
    *p = 0;
    ok = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) == cudaSuccess &&
         cudaMemcpyToSymbolAsync(seq_wait_host, &p, sizeof p, 0, cudaMemcpyHostToDevice, s) == cudaSuccess && cudaStreamSynchronize(s) == cudaSuccess;
    if (s) cudaStreamDestroy(s);
  }
  cudaThreadExchangeStreamCaptureMode(&mode);
  if (!ok) {
    if (p) cudaFreeHost(p);
    cudaGetLastError();
    return false;
  }
  wait_words[dev].store(p, std::memory_order_release);
  return true;
}
int fq3c_wait_failed(void) {
  for (auto& w : wait_words) {
    const volatile int* p = w.load(std::memory_order_acquire);
    if (p && *p) return 1;
  }
  return 0;
}

// Opt-in shared-memory sizes are a per-DEVICE function attribute: a process that serves several GPUs (server.py --gpus N: one scheduler
// thread per device) must set them on each device it launches on, not once per process.
static bool device_attrs_ready() {
  static bool done[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  if (done[dev]) return true;
  if (cudaFuncSetAttribute(fq3c_gemm_tc5_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, T_SMEM) != cudaSuccess ||
      cudaFuncSetAttribute(fq3c_gemm_tc5_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, t_smem(3)) != cudaSuccess ||
      cudaFuncSetAttribute(fq3c_gemm_persist_kernel<1, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, GP_SMEM_MAX) != cudaSuccess ||
      cudaFuncSetAttribute(fq3c_gemm_persist_kernel<1, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize, GP_SMEM_MAX) != cudaSuccess ||
      cudaFuncSetAttribute(fq3c_gemm_persist_kernel<2, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, GP_SMEM_HALF) != cudaSuccess ||
      cudaFuncSetAttribute(fq3s_ggemm_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, GT_SMEM) != cudaSuccess ||
      cudaFuncSetAttribute(fq3s_ggemm_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, GT_SMEM) != cudaSuccess ||
      cudaFuncSetAttribute(fq3c_attn_rows_kernel<128, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, AR_SMEM_MAX) != cudaSuccess ||
      cudaFuncSetAttribute(fq3c_attn_rows_kernel<128, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, AR_SMEM_MAX) != cudaSuccess ||
      cudaFuncSetAttribute(fq3c_attn_rows_kernel<64, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, AR_SMEM_MAX) != cudaSuccess ||
      cudaFuncSetAttribute(fq3c_attn_prefill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, APF_WARPS * (128 + 2048) * 4) != cudaSuccess)
    return false;
  done[dev] = true;
  return true;
}

// The side stream of FQ3C_BRANCH and its two events, per host thread and device: lists that run in several threads never share one.
struct SideStream { cudaStream_t stream = nullptr; cudaEvent_t begun = nullptr, done = nullptr; };
static SideStream* side_stream() {
  static thread_local SideStream sides[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  SideStream& e = sides[dev];
  if (e.done) return &e;
  if ((!e.stream && cudaStreamCreateWithFlags(&e.stream, cudaStreamNonBlocking) != cudaSuccess) ||
      (!e.begun && cudaEventCreateWithFlags(&e.begun, cudaEventDisableTiming) != cudaSuccess) ||
      cudaEventCreateWithFlags(&e.done, cudaEventDisableTiming) != cudaSuccess) {
    e.done = nullptr;
    cudaGetLastError();
    return nullptr;
  }
  return &e;
}
static int run_ops(const fq3c_op* ops, int n_ops, cudaStream_t main_stream, SideStream*& open);
int fq3c_gemm_plan(const fq3c_op* op, int32_t* out) {
  if (!op || !out || op->kind != FQ3C_GEMM || op->M <= 0 || op->m_begin < 0 || op->m_begin >= op->M || op->taps < 1 || op->taps > 8 || op->K % 8 || op->cin % 8 || !gemm_persists(*op))
    return fail("gemm_plan: not a product of the persistent kernel");
  const GemmLaunch L = gemm_plan(gemm_whole_pieces(*op));
  const int32_t v[8] = {L.shape, L.g.bn, L.g.mt, L.g.nt, L.g.parts, L.g.splits, L.g.stages, (int32_t)L.grid};
  std::copy(v, v + 8, out);
  return 0;
}
int fq3c_run(const fq3c_op* ops, int n_ops, void* stream) {
  if (!wait_word_ready()) return fail("cannot make the error word of bounded waits");
  SideStream* open = nullptr;
  const int rc = run_ops(ops, n_ops, (cudaStream_t)stream, open);
  if (open && (cudaEventRecord(open->done, open->stream) != cudaSuccess || cudaStreamWaitEvent((cudaStream_t)stream, open->done, 0) != cudaSuccess))
    return rc != 0 ? rc : fail("branch: join failed");      // a list (or an error) that left the side stream open
  return rc;
}
static int run_ops(const fq3c_op* ops, int n_ops, cudaStream_t main_stream, SideStream*& open) {
  cudaStream_t s = main_stream;
  // The codec's kernels wait for the launches in front themselves and may begin early, as long as the launch in front on their stream belongs to this list
  // (what ran before the list is complete when its first launch begins): a prompt of 39 rows through 28 layers 1676 -> 1497 us, a codec window 1059 -> 972.
  // The sequence models' own kernels, products of few rows among them, do so with one row alone (seq_early); their tcgen05 GEMMs always.
  bool chained = false;
  for (int i = 0; i < n_ops; ++i) {
    const fq3c_op& o = ops[i];
    if (o.M <= 0) continue;
    const bool after = chained;
    chained = o.kind != FQ3C_BRANCH;
    switch (o.kind) {
      case FQ3C_BRANCH: {
        if (o.i0 == 0) {
          if (open) return fail("branch: one side stream at a time");
          SideStream* side = side_stream();
          if (!side || cudaEventRecord(side->begun, main_stream) != cudaSuccess || cudaStreamWaitEvent(side->stream, side->begun, 0) != cudaSuccess)
            return fail("branch: cannot open the side stream");
          open = side;
          s = side->stream;
        } else if (o.i0 == 1) {
          s = main_stream;
        } else {
          s = main_stream;
          if (open) {
            SideStream* side = open;
            open = nullptr;
            if (cudaEventRecord(side->done, side->stream) != cudaSuccess || cudaStreamWaitEvent(main_stream, side->done, 0) != cudaSuccess)
              return fail("branch: join failed");
          }
        }
        continue;
      }
      case FQ3C_GEMM: {
        // True 32-bit operands, few rows (decode: weight streaming, one warp per output column) and shapes the tensor-core
        // kernels do not take (K not a multiple of 8, unaligned rows) go to the sequence-model product.
        if (o.taps == 1 && !(o.flags & ~SEQ_GEMM_FLAGS) && !o.norm_out &&
            ((o.flags & FQ3C_F32) || ((o.flags & FQ3C_NOROUND) && o.M <= 4) || o.K % 8 || o.lda % 8 ||
             (reinterpret_cast<uintptr_t>(o.A) & 15) || (reinterpret_cast<uintptr_t>(o.B) & 15))) {
          SeqGemm g{};
          g.A = o.A; g.B = o.B; g.bias = reinterpret_cast<const float*>(o.bias); g.C = o.C;
          g.M = o.M; g.N = o.N; g.K = o.K; g.lda = o.lda; g.ldb = o.K; g.ldc = o.ldc; g.flags = o.flags;
          g.a_mod = 1; g.early = o.reserved & 1;
          const bool f32 = (o.flags & FQ3C_F32) != 0;
          SeqTail tail{};
          gemv_tail(o, g, ops + i + 1, n_ops - i - 1, tail);
          if (launch_seq_gemm(g, f32, f32, true, 1, (o.M + 63) / 64, s, after, &tail) != 0) return -1;
          i += tail.n;
          break;
        }
        if (o.K % 8 || o.cin % 8 || o.taps > 8 || o.col_mod <= 0) return fail("gemm: K and cin must be multiples of 8, taps <= 8");
        if (o.m_begin < 0 || o.m_begin >= o.M) return fail("gemm: m_begin outside [0, M)");
        if (o.norm_out && ((o.flags & (FQ3C_SWIGLU | FQ3C_OUT_F32)) || !o.norm_w || o.norm_ld < o.N))
          return fail("gemm: a fused RMSNorm needs a bf16 [M, N] output, weights and norm_ld >= N");
        const bool use_tc5 = gemm_on_tc(o);
        if (use_tc5 && !device_attrs_ready()) return fail("cannot reserve shared memory for the tcgen05 GEMM / prefill attention");
        if (gemm_persists(o)) {
          const fq3c_op w = gemm_whole_pieces(o);
          const GemmLaunch L = gemm_plan(w);
          CUtensorMap tmA, tmB;
          if (make_map(&tmA, o.A, (uint64_t)o.cin, (uint64_t)o.a_rows, (uint64_t)o.lda, (uint32_t)L.g.a_rows) &&
              make_map(&tmB, o.B, (uint64_t)o.K, (uint64_t)o.N, (uint64_t)o.K, (uint32_t)L.g.bn)) {
            if (L.shape == GS_HALF) launch_after(fq3c_gemm_persist_kernel<2, 8>, L.grid, gp_threads(8), L.smem, s, after, L.g.splits, w, L.g, tmA, tmB);
            else if (L.shape == GS_FEW) launch_after(fq3c_gemm_persist_kernel<1, 8>, L.grid, gp_threads(8), L.smem, s, after, L.g.splits, w, L.g, tmA, tmB);
            else launch_after(fq3c_gemm_persist_kernel<1, 16>, L.grid, gp_threads(16), L.smem, s, after, L.g.splits, w, L.g, tmA, tmB);
            if (o.norm_out) {
              launch_rownorm(o, s, true);
              count_launches(1);
            }
            break;
          }
        }
        if (use_tc5) {
          // Tile width: a multiple of 16 columns (a legal UMMA N at M = 128), chosen so that the grid covers the SMs.
          // Tall operands (M >= 128) keep BN >= 64 (every column tile re-reads the A rows); short ones (the transformer at
          // 8-33 frames) are weight-streaming problems: the width that minimises waves x tile cost, down to 16 columns.
          const int mt = (o.M - o.m_begin + TM - 1) / TM;
          int bn = TMAXN;
          if (o.M >= TM) {
            if (((o.N + bn - 1) / bn) * mt < 100) bn = 64;
          } else {
            long best = -1;
            for (int cand = TMAXN; cand >= 16; cand >>= 1) {
              const long tiles = (long)((o.N + cand - 1) / cand) * mt;
              const long cost = ((tiles + 147) / 148) * (cand + 48);  // waves x (columns + fixed per-tile work)
              if (best < 0 || cost < best) { best = cost; bn = cand; }
            }
          }
          // Split-K when the tiles would cover less than half of the SMs and the reduction is long (the transformer's
          // o / down projections at 8-240 rows: 16-32 tiles each walking 32-96 k-blocks alone): wider tiles, every tile
          // split over up to eight CTAs, partial tiles through the caller's workspace.
          const int KT = (o.K + TK - 1) / TK;
          const int Nw = (o.N + 7) & ~7;
          int splits = 1;
          if (o.ws && o.M <= 4 * TM && KT >= 8) {
            const int bn_s = o.N >= 64 ? 64 : 32;
            // the split count must not depend on m_begin: a tail-only decode has to add the same partial sums in the same order
            const int tiles_s = ((o.N + bn_s - 1) / bn_s) * ((o.M + TM - 1) / TM);
            int sp = std::min(std::min(8, KT / 4), 148 / std::max(1, tiles_s));
            while (sp > 1 && (int64_t)sp * o.M * Nw * 4 > o.ws_bytes) --sp;
            if (sp > 1) { splits = sp; bn = bn_s; }
          }
          const int nt = (o.N + bn - 1) / bn;
          bn = std::min(TMAXN, (((o.N + nt - 1) / nt) + 15) / 16 * 16);
          dim3 grid((o.N + bn - 1) / bn, mt, splits);
          // Many tiles (the vocoder convolutions: hundreds of 128-row tiles with 2-11 k-blocks and a long SnakeBeta epilogue):
          // three stages instead of six so that two CTAs share an SM and one's epilogue overlaps the other's main loop.
          static int two_ctas = -1;
          if (two_ctas < 0) { const char* e2 = getenv("FQ3C_TWO_CTAS"); two_ctas = (e2 == nullptr || atoi(e2) != 0) ? 1 : 0; }
          const long n_ctas = (long)grid.x * grid.y * grid.z;
          const bool two = two_ctas && n_ctas >= 2 * 148 && KT <= 24;
          if (two) fq3c_gemm_tc5_kernel<2><<<grid, TTHREADS, t_smem(3), s>>>(o, bn, splits, Nw, 3);
          else fq3c_gemm_tc5_kernel<1><<<grid, TTHREADS, T_SMEM, s>>>(o, bn, splits, Nw, TSTAGES);
          if (splits > 1) {
            if (o.norm_out) {
              fq3c_splitk_reduce_norm_kernel<<<(unsigned)(o.M - o.m_begin), 256, 0, s>>>(o, splits, Nw);
            } else {
              const long n = (long)(o.M - o.m_begin) * (Nw >> 3);
              fq3c_splitk_reduce_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(o, splits, Nw);
            }
            count_launches(1);
          } else if (o.norm_out) {
            launch_rownorm(o, s, false);
            count_launches(1);
          }
          break;
        }
        // one output channel: rows, pitch and weights in whole 16-byte pieces, the rows a block sees within its shared memory
        if (o.N == 1 && o.cin % 8 == 0 && o.cin <= C1_CIN && !o.norm_out && !(o.flags & FQ3C_SWIGLU) && o.lda % 8 == 0 && !(reinterpret_cast<uintptr_t>(o.A) & 15)) {
          const int lo = *std::min_element(o.tap_off, o.tap_off + o.taps), span = *std::max_element(o.tap_off, o.tap_off + o.taps) - lo;
          if (span <= C1_SPAN) {
            const size_t smem = (size_t)o.taps * o.cin * 4 + (size_t)(C1_ROWS + span) * (o.cin + 8) * 2;
            static bool cattr[64] = {};
            int dev = 0;
            cudaGetDevice(&dev);
            if (dev >= 0 && dev < 64 && !cattr[dev]) {
              cudaFuncSetAttribute(fq3c_conv1_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 8 * C1_CIN * 4 + (C1_ROWS + C1_SPAN) * (C1_CIN + 8) * 2);
              cattr[dev] = true;
            }
            launch_after(fq3c_conv1_kernel, (unsigned)((o.M - o.m_begin + C1_ROWS - 1) / C1_ROWS), C1_ROWS, smem, s, after, 1, o, lo, span);
            break;
          }
        }
        dim3 grid((o.N + BN - 1) / BN, (o.M - o.m_begin + BM - 1) / BM);
        fq3c_gemm_kernel<<<grid, 128, 0, s>>>(o);
        if (o.norm_out) {
          launch_rownorm(o, s, false);
          count_launches(1);
        }
        break;
      }
      case FQ3C_RVQ: launch_after(fq3c_rvq_kernel, o.M, 128, 0, s, after, 1, o); break;
      case FQ3C_RMSNORM:
        if (norm_vec_ok(o.A, o.C, o.scale, o.N, o.lda, o.ldc))
          launch_after(fq3c_rownorm_vec_kernel, (unsigned)((o.M + RN_WARPS - 1) / RN_WARPS), RN_WARPS * 32, 0, s, after, 1, reinterpret_cast<const bf16*>(o.A), o.lda,
                       reinterpret_cast<bf16*>(o.C), o.ldc, reinterpret_cast<const float*>(o.scale), o.f0, 0, o.M, o.N);
        else launch_after(fq3c_rmsnorm_kernel, o.M, 256, 0, s, after, 1, o);
        break;
      case FQ3C_LAYERNORM: launch_after(fq3c_layernorm_kernel, o.M, 256, 0, s, after, 1, o); break;
      case FQ3C_ROPE: launch_after(fq3c_rope_kernel, o.M, 256, 0, s, after, 1, o); break;
      case FQ3C_ATTN: {
        if (o.i2 > 128) return fail("attn: head_dim > 128");
        const bool use_apf = prompt_kernels();
        if (use_apf && (o.flags & 1) && o.i2 == 128 && o.taps == 0 && !o.p0) {
          AttnArgs a{};
          a.q = o.A; a.k = reinterpret_cast<const bf16*>(o.A) + (size_t)o.i0 * 128; a.v = a.k + (size_t)o.i1 * 128;
          a.tries = o.reserved & 2 ? GP_TRIES_TEST : GP_TRIES; a.lost = (o.reserved >> 1) & 1;
          a.ldq = a.ldk = a.ldv = o.lda; a.H = o.i0; a.G = o.i1; a.M = o.M; a.scale = 0.08838834764831845f; a.window = o.K < o.M ? o.K : 0; a.out = o.C; a.ldo = o.ldc;
          if (attn_prompt_many(o) && attn_tc_takes(a, AT_PROMPT)) {
            launch_attn_tc(a, AT_PROMPT, s, after);
            break;
          }
        }
        if (use_apf && (o.flags & 1) && o.i2 == 128 && o.taps == 0 && !o.p0 && o.M <= 2048 && (o.lda % 8) == 0 && (o.ldc % 4) == 0 &&
            (o.i0 % o.i1) == 0) {
          const int tpad = (o.M + 7) & ~7;
          const size_t smem = (size_t)APF_WARPS * 128 * 4 + (size_t)APF_WARPS * tpad * 4;
          if (!device_attrs_ready()) return fail("cannot reserve shared memory for the prefill attention");
          const int warps = o.M * o.i0;
          launch_after(fq3c_attn_prefill_kernel, (warps + APF_WARPS - 1) / APF_WARPS, APF_WARPS * 32, smem, s, after, 1, o, tpad);
          break;
        }
        if (attn_rows_takes(o, false)) {
          const AttnRows r = attn_rows_plan(o, false);
          const dim3 grid((unsigned)((o.M + r.rb - 1) / r.rb), (unsigned)o.i1);
          if (o.i2 == 64) launch_after(fq3c_attn_rows_kernel<64, false>, grid, AR_WARPS * 32, r.smem, s, after, 1, o, o, r.rb, r.span, r.sp);
          else launch_after(fq3c_attn_rows_kernel<128, false>, grid, AR_WARPS * 32, r.smem, s, after, 1, o, o, r.rb, r.span, r.sp);
          break;
        }
        const int warps = o.M * o.i0;
        launch_after(fq3c_attn_kernel, (warps + 7) / 8, 256, 0, s, after, 1, o);
        break;
      }
      case FQ3C_DWCONV: {
        const size_t n = (size_t)o.M * o.N;
        launch_after(fq3c_dwconv_kernel, (unsigned)std::min<size_t>(2048, (n + 255) / 256), 256, 0, s, after, 1, o);
        break;
      }
      case FQ3C_QKNORM_ROPE_KV: {
        if (o.lda % 4 || !o.C || !o.C2 || !o.p0 || !o.p1 || !o.B || !o.bias) return fail("qknorm_rope_kv: missing operand");
        if (i + 1 < n_ops && prompt_kernels() && attn_rows_takes_prompt(o, ops[i + 1])) {      // with the attention behind it in one launch
          const fq3c_op& at = ops[++i];
          const AttnRows r = attn_rows_plan(at, true);
          launch_after(fq3c_attn_rows_kernel<128, true>, dim3((unsigned)((at.M + r.rb - 1) / r.rb), (unsigned)at.i1), AR_WARPS * 32, r.smem, s, after, 1, at, o, r.rb, r.span, r.sp);
          break;
        }
        const int warps = o.M * (o.i0 + 2 * o.i1);
        launch_after(fq3c_qknorm_rope_kv_kernel, (warps + 7) / 8, 256, 0, s, after, 1, o);
        break;
      }
      case FQ3C_SNAKE: {
        const size_t n = (size_t)o.M * o.N;
        fq3c_snake_kernel<<<(unsigned)std::min<size_t>(4096, (n + 255) / 256), 256, 0, s>>>(o);
        break;
      }
      case FQ3C_COPY: {
        if ((o.N % 8) || (o.lda % 8) || (o.ldc % 8) || !o.A || !o.C) return fail("copy: N, lda, ldc must be multiples of 8");
        const size_t n = (size_t)o.M * (o.N >> 3);
        fq3c_copy_kernel<<<(unsigned)std::min<size_t>(1024, (n + 255) / 256), 256, 0, s>>>(o);
        break;
      }
      case FQ3C_ROLL: {
        if (!o.A || o.M <= 0) return fail("roll: no descriptors");
        fq3c_roll_kernel<<<dim3((unsigned)o.M, ROLL_SLICES), 256, 0, s>>>(reinterpret_cast<const long long*>(o.A), reinterpret_cast<int*>(o.C), o.i0);
        break;
      }
      case FQ3C_ADVANCE: {
        if (!o.C) return fail("advance: null counter");
        fq3c_advance_kernel<<<1, 1, 0, s>>>(reinterpret_cast<int*>(o.C), o.i0);
        break;
      }
      case FQ3C_TCONV:
        if (i + 2 < n_ops && delta_row_takes(o, ops[i + 1], ops[i + 2])) {      // with the recurrence and the norm behind it in one launch
          launch_delta_row(o, ops[i + 1], ops[i + 2], s, after);
          i += 2;
          break;
        }
        [[fallthrough]];
      case FQ3C_ROT_APPEND:
        if (o.kind == FQ3C_ROT_APPEND && i + 1 < n_ops && rot_append_ok(o) && attn_few_takes_rot(o, ops[i + 1]) && !cache_attn_error(ops[i + 1])) {      // with the attention behind it in one launch
          ++i;
          launch_attn_few(ops[i], &o, s, after);
          break;
        }
        [[fallthrough]];
      default: {
        const int rc = seq_run(o, s, after);
        if (rc == 1) return fail("unknown op kind");
        if (rc != 0) return rc;
      }
    }
    count_launches(1);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(std::string("launch failed at op ") + std::to_string(i) + ": " + cudaGetErrorString(e));
  }
  return 0;
}


int fq3c_put_ints(const int32_t* values, int n, int32_t* dst, void* stream) {
  if (n < 0 || (n > 0 && (!values || !dst))) return fail("put_ints: bad arguments");
  for (int at = 0; at < n; at += PutInts::MOST) {
    PutInts p{dst + at, std::min(n - at, PutInts::MOST), {}};
    std::copy(values + at, values + at + p.n, p.v);
    fq3c_put_ints_kernel<<<1, p.n <= 32 ? 32 : 256, 0, (cudaStream_t)stream>>>(p);
    count_launches(1);
  }
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : fail(std::string("put_ints: ") + cudaGetErrorString(e));
}

/* A plan is static (same ops, same buffers for a given frame count): capture its launches once and replay them as one
 * CUDA graph (about a hundred short kernels per decode; the replay removes the per-launch CPU and scheduling gaps). */
struct fq3c_graph {
  cudaGraphExec_t exec;
  int n_kernels;
};
int fq3c_graph_create(const fq3c_op* ops, int n_ops, void** out) {
  if (!ops || !out || n_ops <= 0) return fail("graph: bad arguments");
  cudaStream_t cs;
  if (cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking) != cudaSuccess) return fail("graph: stream create failed");
  const int64_t before = t_launches;
  side_stream();      // made before the capture begins
  cudaGraph_t g = nullptr;
  cudaError_t e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
  int rc = 0;
  if (e == cudaSuccess) {
    rc = fq3c_run(ops, n_ops, cs);
    e = cudaStreamEndCapture(cs, &g);
  }
  const int n_kernels = (int)(t_launches - before);
  count_launches(-(int64_t)n_kernels);  // nothing ran yet
  cudaStreamDestroy(cs);
  if (rc != 0 || e != cudaSuccess || !g) {
    if (g) cudaGraphDestroy(g);
    return rc != 0 ? rc : fail(std::string("graph: capture failed: ") + cudaGetErrorString(e));
  }
  cudaGraphExec_t ex = nullptr;
  e = cudaGraphInstantiate(&ex, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) return fail(std::string("graph: instantiate failed: ") + cudaGetErrorString(e));
  *out = new fq3c_graph{ex, n_kernels};
  return 0;
}
int fq3c_graph_launch(void* graph, void* stream) {
  fq3c_graph* g = reinterpret_cast<fq3c_graph*>(graph);
  if (!g) return fail("graph: null handle");
  const cudaError_t e = cudaGraphLaunch(g->exec, (cudaStream_t)stream);
  if (e != cudaSuccess) return fail(std::string("graph: launch failed: ") + cudaGetErrorString(e));
  count_launches(g->n_kernels);
  return 0;
}
int fq3c_graph_destroy(void* graph) {
  fq3c_graph* g = reinterpret_cast<fq3c_graph*>(graph);
  if (g) {
    cudaGraphExecDestroy(g->exec);
    delete g;
  }
  return 0;
}

}  // extern "C"
