// fq3_f32.cuh — true 32-bit products and attention over many rows (the sequence models' `--dtype float32`), on the CUDA cores.
//
// Included by fq3_codec.cu behind fq3_seq.cuh.  Plain f32 multiply-adds, two to an instruction (fma.rn.f32x2), operands staged by cp.async; bound by the
// f32 pipe (128 multiply-adds a cycle and SM).
#pragma once

__device__ __forceinline__ ulonglong2 ld_pairs(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }   // four consecutive floats as two pairs

// C = A B^T like fq3s_gemm_kernel<float, float>, for rows of whole 16-byte pieces.  64 x 64 tiles, three stages of 32 k; a sum is kept as two (even and odd k) that are added at the end,
// so that both operands are read as they lie.  Shared memory and the f32 pipe bound it together.
// GROUPS = 1: a thread has 4 x 4 outputs, two or more blocks an SM.  GROUPS = 4: four groups of 64 threads take eight k of a stage each, a thread 8 x 8 outputs of its group's partial tile
// (16 floats loaded for 64 multiply-adds, half as many as with 4 x 4), the groups' four are added at the end; its registers make it one block an SM, so it is for tiles that are a single
// wave (figures where it is chosen).
constexpr int FG_BM = 64, FG_BN = 64, FG_BK = 32, FG_P = FG_BK + 4, FG_ST = 3, FG_CP = FG_BN + 8;
constexpr int fg_smem(const int groups) {
  const int stages = FG_ST * (FG_BM + FG_BN) * FG_P * 4, parts = groups > 1 ? groups * FG_BM * FG_CP * 4 : 0;
  return stages > parts ? stages : parts;
}
// a finished entry v of row r, column n (z's columns begin at ccol)
__device__ __forceinline__ void fg_store(const SeqGemm& g, const int r, const int row_end, const int ccol, const int n, float v) {
  if (g.flags & FQ3C_SWIGLU) {      // the unit's other column is the neighbouring lane's
    const float up = __shfl_down_sync(0xffffffffu, v, 1);
    if (r < row_end && n + 1 < g.N && !(n & 1)) sg_store_glu(g, r, ccol, n, v, up, sg_row_scale(g, r));
    return;
  }
  if (r >= row_end || n >= g.N) return;
  if (g.flags & FQ3C_BIAS) v += g.bias[ccol + n];
  if (g.flags & FQ3C_GELU) v = gelu_f(v);
  if (g.flags & FQ3C_GELU_TANH) v = gelu_tanh_f(v);
  if (g.flags & FQ3C_SIGMOID) v = sigmoid_f(v);
  if (g.flags & FQ3C_RELU2) { v = fmaxf(v, 0.f); v *= v; }
  const size_t ci = (size_t)r * g.ldc + ccol + n;
  if (g.flags & FQ3C_OUT_F32) reinterpret_cast<float*>(g.C)[ci] = v;
  else reinterpret_cast<bf16*>(g.C)[ci] = __float2bfloat16_rn(v);
}
template <int GROUPS>
__global__ void __launch_bounds__(256, GROUPS > 1 ? 1 : 2) fq3s_gemm_f32_kernel(const SeqGemm g) {
  seq_dep_begin(g.M);
  extern __shared__ __align__(16) float fg[];
  float (*As)[FG_BM][FG_P] = reinterpret_cast<float (*)[FG_BM][FG_P]>(fg);
  float (*Bs)[FG_BN][FG_P] = reinterpret_cast<float (*)[FG_BN][FG_P]>(fg + FG_ST * FG_BM * FG_P);
  const int tid = threadIdx.x, z = blockIdx.z;
  int row0, row_end;
  const float* Bp = reinterpret_cast<const float*>(g.B) + (size_t)z * g.b_zstride;
  if (g.seg) {
    int t = blockIdx.y, e = 0;
    row0 = -1; row_end = 0;
    for (; e < g.E; ++e) {
      const int s0 = g.seg[e], s1 = g.seg[e + 1], nt = (s1 - s0 + FG_BM - 1) / FG_BM;
      if (t < nt) { row0 = s0 + t * FG_BM; row_end = s1; break; }
      t -= nt;
    }
    if (row0 < 0) return;
    Bp += (size_t)e * g.b_estride;
  } else {
    row0 = blockIdx.y * FG_BM; row_end = g.M;
  }
  const int col0 = blockIdx.x * FG_BN;
  const float* Ap = reinterpret_cast<const float*>(g.A) + (size_t)(z % g.a_mod) * g.a_zstride;
  // a thread copies 16 bytes of rows lr and lr + 32 of both operands
  const int lr = tid >> 3, lk = (tid & 7) * 4;
  const float *ap[2], *bp[2];
  bool aok[2], bok[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = row0 + lr + 32 * i, n = col0 + lr + 32 * i;
    aok[i] = r < row_end;
    bok[i] = n < g.N;
    ap[i] = Ap + (size_t)(aok[i] ? (g.rows ? g.rows[r] : r) : 0) * g.lda;
    bp[i] = Bp + (size_t)(bok[i] ? n : 0) * g.ldb;
  }
  const int KT = (g.K + FG_BK - 1) / FG_BK;
  auto stage = [&](const int kt) {
    if (kt < KT) {
      const int st = kt % FG_ST, k = kt * FG_BK + lk;
      const bool in = k < g.K;      // (K is a multiple of four)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        cp_async16(&As[st][lr + 32 * i][lk], in ? ap[i] + k : ap[i], in && aok[i]);
        cp_async16(&Bs[st][lr + 32 * i][lk], in ? bp[i] + k : bp[i], in && bok[i]);
      }
    }
    cp_async_commit();
  };
  constexpr int E = GROUPS > 1 ? 8 : 4, L = 64 / E;      // outputs of a thread: E x E, rows and columns L apart
  const int kg = GROUPS > 1 ? tid >> 6 : 0, ty = tid / L % L, tx = tid % L;
  f32x2 acc[E][E];
#pragma unroll
  for (int i = 0; i < E; ++i)
#pragma unroll
    for (int j = 0; j < E; ++j) acc[i][j] = 0ull;
  stage(0);
  stage(1);
  for (int kt = 0; kt < KT; ++kt) {
    cp_async_wait<1>();
    __syncthreads();
    stage(kt + 2);
    const int st = kt % FG_ST;
#pragma unroll
    for (int k = 0; k < FG_BK / GROUPS; k += 4) {
      ulonglong2 a[E], b[E];
#pragma unroll
      for (int j = 0; j < E; ++j) b[j] = ld_pairs(&Bs[st][tx + L * j][kg * (FG_BK / GROUPS) + k]);
#pragma unroll
      for (int i = 0; i < E; ++i) a[i] = ld_pairs(&As[st][ty + L * i][kg * (FG_BK / GROUPS) + k]);
#pragma unroll
      for (int i = 0; i < E; ++i)
#pragma unroll
        for (int j = 0; j < E; ++j) acc[i][j] = fma2<true>(a[i].x, b[j].x, acc[i][j]);
#pragma unroll
      for (int i = 0; i < E; ++i)
#pragma unroll
        for (int j = 0; j < E; ++j) acc[i][j] = fma2<true>(a[i].y, b[j].y, acc[i][j]);
    }
  }
  const int ccol = z * g.c_zstride;
  if (GROUPS == 1) {
#pragma unroll
    for (int i = 0; i < E; ++i)
#pragma unroll
      for (int j = 0; j < E; ++j) fg_store(g, row0 + ty + L * i, row_end, ccol, col0 + tx + L * j, lo2(acc[i][j]) + hi2(acc[i][j]));
    return;
  }
  cp_async_wait<0>();
  __syncthreads();      // the stages become the groups' partial tiles
#pragma unroll
  for (int i = 0; i < E; ++i)
#pragma unroll
    for (int j = 0; j < E; ++j) fg[(kg * FG_BM + ty + L * i) * FG_CP + tx + L * j] = lo2(acc[i][j]) + hi2(acc[i][j]);
  __syncthreads();
#pragma unroll 4
  for (int i = tid >> 6; i < FG_BM; i += 4) {
    const float* p = fg + i * FG_CP + (tid & 63);
    fg_store(g, row0 + i, row_end, ccol, col0 + (tid & 63), (p[0] + p[FG_BM * FG_CP]) + (p[2 * FG_BM * FG_CP] + p[3 * FG_BM * FG_CP]));
  }
}

// Softmax attention over an f32 cache for many queries, heads of 128: fq3s_cache_attn_kernel's arithmetic (full-precision exponential, tanh, logarithm).  A block
// takes 32 (query, head of the group) rows of one key / value head and tiles of 64 positions: S [32 x 64] with 4 x 4 scores a thread, an online softmax over
// half-warps, O [32 x 128] += P V with 4 x 8 outputs a thread.  Keys of the next tile arrive while this one's weights and outputs are formed, values while
// its scores are.  384 rows of 8 heads behind 300 positions, window 512: 235 -> 56 us with three key splits and their merge.
// Eight columns (4 tx .. + 3 and 64 + 4 tx .. + 3) of an unnormalised output row over the keys first .. last that the row sees, and no others: formed again
// where the weight 0 of an unseen key met an infinite or NaN value of the tile.
__device__ __noinline__ void fa_row_again(const fq3c_op& o, const CacheAttnMask& mask, const int m, const int head, const int tx, const int pos, const int first, const int last,
                                          const float mx, float* out) {
  const int kvh = head / (o.i0 / o.i1);
  const float* q = reinterpret_cast<const float*>(o.A) + (size_t)m * o.lda + (size_t)head * 128;
  const float* r12 = reinterpret_cast<const float*>(o.bias);
  for (int j = 0; j < 8; ++j) out[j] = 0.f;
  for (int key = first; key <= min(last, pos); ++key) {
    if (!mask.sees(pos, key)) continue;
    const float* k = reinterpret_cast<const float*>(o.B) + (size_t)key * o.ldr + kvh * 128;
    float s = 0.f;
    for (int c = 0; c < 128; ++c) s = fmaf(q[c], k[c], s);
    s *= o.f0;
    if (o.f1 > 0.f) s = o.f1 * tanhf(s / o.f1);
    if (r12) s -= r12[head] * log1pf(r12[o.i0 + head] * (float)(pos - key));
    const float w = expf(s - mx);
    const float* v = reinterpret_cast<const float*>(o.p1) + (size_t)key * o.taps + kvh * 128 + 4 * tx;
    for (int j = 0; j < 8; ++j) out[j] = fmaf(w, v[(j >> 2) * 64 + (j & 3)], out[j]);
  }
}
constexpr int FA_R = 32, FA_T = 64, FA_P = 132, FA_PP = FA_T + 4;
constexpr int FA_SMEM = (FA_R * FA_P + 2 * FA_T * FA_P + FA_R * FA_PP) * 4;
__global__ void __launch_bounds__(128) fq3s_attn_f32_kernel(const fq3c_op o) {
  seq_dep_begin(o.M);
  extern __shared__ __align__(16) float fa[];
  float *qs = fa, *ks = qs + FA_R * FA_P, *vs = ks + FA_T * FA_P, *ps = vs + FA_T * FA_P;
  const int H = o.i0, HG = H / o.i1, QB = FA_R / HG, kvh = blockIdx.y, tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const int m0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * QB, P = o.p0 ? *reinterpret_cast<const int*>(o.p0) : 0;      // the most keys start first
  const int nq = min(QB, o.M - m0), ifirst = P + m0, ilast = ifirst + nq - 1;
  const CacheAttnMask mask{o.K, o.a_rows, o.tap_off[0], 0};
  const float* A = reinterpret_cast<const float*>(o.A);
  for (int i = tid; i < FA_R * 32; i += 128) {
    const int r = i >> 5, c = (i & 31) * 4, qi = r / HG, hh = r - qi * HG;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (qi < nq) v = *reinterpret_cast<const float4*>(A + (size_t)(m0 + qi) * o.lda + (size_t)(kvh * HG + hh) * 128 + c);
    *reinterpret_cast<float4*>(qs + r * FA_P + c) = v;
  }
  auto fetch = [&](const void* base, const int ld, float* dst, const int t) {
    const float* src = reinterpret_cast<const float*>(base) + (size_t)kvh * 128;
#pragma unroll 4
    for (int i = tid; i < FA_T * 32; i += 128) {
      const int r = i >> 5, c = (i & 31) * 4, j = t * FA_T + r;
      const bool ok = j <= ilast;
      cp_async16(dst + r * FA_P + c, src + (size_t)(ok ? j : 0) * ld + c, ok);
    }
    cp_async_commit();
  };
  const int ntiles = ilast / FA_T + 1, splits = gridDim.z;
  auto skip = [&](const int t) {      // nobody of the block sees it
    const int j0 = t * FA_T, j1 = j0 + FA_T;
    return (mask.window > 0 && j1 <= ifirst - mask.window + 1 && j0 >= mask.keep) || (mask.chunk > 0 && j1 <= ifirst - ifirst % mask.chunk);
  };
  auto next = [&](int t) { do ++t; while (t < ntiles && skip(t)); return t; };
  // this thread's rows ty + 8 e
  int pos[4], head[4];
  bool live[4];
  float r1[4] = {0.f, 0.f, 0.f, 0.f}, r2[4] = {0.f, 0.f, 0.f, 0.f};
  const float* r12 = reinterpret_cast<const float*>(o.bias);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int r = ty + 8 * e, qi = r / HG;
    live[e] = qi < nq;
    pos[e] = ifirst + qi;
    head[e] = kvh * HG + (r - qi * HG);
    if (r12 && live[e]) { r1[e] = r12[head[e]]; r2[e] = r12[H + head[e]]; }
  }
  const float cap = o.f1, icap = o.f1 > 0.f ? 1.f / o.f1 : 0.f;
  float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY}, sum[4] = {0.f, 0.f, 0.f, 0.f};
  f32x2 acc[4][4];      // columns 4 tx .. + 3 and 64 + 4 tx .. + 3 in pairs
#pragma unroll
  for (int e = 0; e < 4; ++e)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[e][j] = 0ull;
  // the splits share the tiles that somebody sees
  int count = 0, t = next(-1);
  if (splits > 1) {
    for (int u = t; u < ntiles; u = next(u)) ++count;
    const int u0 = (int)blockIdx.z * count / splits, u1 = ((int)blockIdx.z + 1) * count / splits;
    for (int i = 0; i < u0; ++i) t = next(t);
    count = u1 - u0;
  } else {
    count = ntiles;
  }
  if (count == 0) t = ntiles;
  const int tfirst = t;
  int tlast = t;
  if (t < ntiles) fetch(o.B, o.ldr, ks, t);
  if (t < ntiles) fetch(o.p1, o.taps, vs, t);
  while (t < ntiles) {
    const int tn = --count > 0 ? next(t) : ntiles, j0 = t * FA_T;
    cp_async_wait<1>();
    __syncthreads();
    f32x2 s2[4][4];
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
      for (int j = 0; j < 4; ++j) s2[e][j] = 0ull;
#pragma unroll 4
    for (int k = 0; k < 128; k += 4) {
      ulonglong2 a[4], b[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) a[e] = ld_pairs(qs + (ty + 8 * e) * FA_P + k);
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = ld_pairs(ks + (tx + 16 * j) * FA_P + k);
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int j = 0; j < 4; ++j) s2[e][j] = fma2<true>(a[e].y, b[j].y, fma2<true>(a[e].x, b[j].x, s2[e][j]));
    }
    __syncthreads();
    if (tn < ntiles) fetch(o.B, o.ldr, ks, tn);
    else cp_async_commit();
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float s[4], m = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int key = j0 + tx + 16 * j;
        float v = -INFINITY;
        if (live[e] && mask.sees(pos[e], key)) {
          v = (lo2(s2[e][j]) + hi2(s2[e][j])) * o.f0;
          if (cap > 0.f) v = cap * tanhf(v * icap);
          if (r12) v -= r1[e] * log1pf(r2[e] * (float)(pos[e] - key));
        }
        s[j] = v;
        m = fmaxf(m, v);
      }
#pragma unroll
      for (int w = 8; w > 0; w >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, w));      // the row's sixteen lanes
      const float mn = fmaxf(mx[e], m), al = mx[e] == -INFINITY ? 0.f : expf(mx[e] - mn);
      float add = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float p = s[j] == -INFINITY ? 0.f : expf(s[j] - mn);
        add += p;
        ps[(ty + 8 * e) * FA_PP + tx + 16 * j] = p;
      }
#pragma unroll
      for (int w = 8; w > 0; w >>= 1) add += __shfl_xor_sync(0xffffffffu, add, w);
      sum[e] = sum[e] * al + add;
      mx[e] = mn;
      const f32x2 al2 = pack2(al, al);
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[e][j] = mul2<true>(acc[e][j], al2);
    }
    cp_async_wait<1>();
    __syncthreads();
#pragma unroll 2
    for (int k = 0; k < FA_T; k += 4) {
      float4 p[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) p[e] = *reinterpret_cast<const float4*>(ps + (ty + 8 * e) * FA_PP + k);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const ulonglong2 v0 = ld_pairs(vs + (k + q) * FA_P + 4 * tx), v1 = ld_pairs(vs + (k + q) * FA_P + 64 + 4 * tx);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float w = q == 0 ? p[e].x : q == 1 ? p[e].y : q == 2 ? p[e].z : p[e].w;
          const f32x2 w2 = pack2(w, w);
          acc[e][0] = fma2<true>(w2, v0.x, acc[e][0]);
          acc[e][1] = fma2<true>(w2, v0.y, acc[e][1]);
          acc[e][2] = fma2<true>(w2, v1.x, acc[e][2]);
          acc[e][3] = fma2<true>(w2, v1.y, acc[e][3]);
        }
      }
    }
    __syncthreads();
    if (tn < ntiles) fetch(o.p1, o.taps, vs, tn);
    else cp_async_commit();
    tlast = t;
    t = tn;
  }
  cp_async_wait<0>();
  const float* sink = reinterpret_cast<const float*>(o.scale);
  const float* gate = reinterpret_cast<const float*>(o.res);
  const bool entry = gate && (o.flags & FQ3C_GATE_ENTRY);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    if (!live[e]) continue;
    const int m = pos[e] - P, h = head[e];
    f32x2 far = 0ull;      // NaN as soon as one of the sums is not finite
#pragma unroll
    for (int j = 0; j < 4; ++j) far = fma2<true>(acc[e][j], pack2(0.f, 0.f), far);
    if (lo2(far) + hi2(far) != 0.f && sum[e] < INFINITY) {
      float v[8];
      fa_row_again(o, mask, m, h, tx, pos[e], tfirst * FA_T, tlast * FA_T + FA_T - 1, mx[e], v);
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[e][j] = pack2(v[2 * j], v[2 * j + 1]);
    }
    if (splits > 1) {      // (maximum, sum, unnormalised output): fq3s_cache_attn_merge_kernel adds the splits
      float* dst = reinterpret_cast<float*>(o.ws) + (((size_t)m * H + h) * splits + blockIdx.z) * 130;
      if (tx == 0) { dst[0] = mx[e]; dst[1] = sum[e]; }
#pragma unroll
      for (int j = 0; j < 8; ++j) dst[2 + (j >> 2) * 64 + 4 * tx + (j & 3)] = j & 1 ? hi2(acc[e][j >> 1]) : lo2(acc[e][j >> 1]);
      continue;
    }
    float f = 1.f, den = sum[e];
    if (sink) {
      const float mm = fmaxf(mx[e], sink[h]);
      f = mx[e] == -INFINITY ? 0.f : expf(mx[e] - mm);
      den = den * f + expf(sink[h] - mm);
    }
    float g = gate && !entry ? sigmoid_f(gate[(size_t)m * o.col_mod + h]) : 1.f;
    if (o.f2 != 0.f) g *= o.f2;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int c = (j >> 2) * 64 + 4 * tx + (j & 3);
      float v = (j & 1 ? hi2(acc[e][j >> 1]) : lo2(acc[e][j >> 1])) * f / den * g;
      if (entry) v *= sigmoid_f(gate[(size_t)m * o.col_mod + (size_t)h * 128 + c]);
      const size_t at = (size_t)m * o.ldc + (size_t)h * 128 + c;
      if (o.flags & FQ3C_OUT_F32) reinterpret_cast<float*>(o.C)[at] = v;
      else reinterpret_cast<bf16*>(o.C)[at] = __float2bfloat16_rn(v);
    }
  }
}
