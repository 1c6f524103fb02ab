// The gated delta rule four tokens at a time, for steps that bring many tokens a sequence in bfloat16 storage.  Included by
// sequence_mix.cuh, whose walk (token by token) states the recurrence and stays for 32-bit storage, few tokens and heads of other
// sizes than 64 < dk <= 128.
//
// What bounds the walk is one link of its chain per token: two dot products with the state, a shuffle tree, the write (560
// cycles a token measured, of which 175 are instructions).  The state before a group of four tokens is enough for the whole
// group.  With c_i = g_1 .. g_i the decay up to token i (products of factors at most one: nothing overflows and nothing is
// divided), S0 the state before the group:
//   a_i = (c_i k_i)^T S0       p_i = (c_i q_i)^T S0
//   A_ij = k_i^T (g_{j+1} .. g_i) k_j  (j < i)      B_ij = q_i^T (g_{j+1} .. g_i) k_j  (j <= i)
//   u_i = beta_i (v_i - a_i - sum_{j<i} A_ij u_j)    o_i = p_i + sum_{j<=i} B_ij u_j
//   S   = c_4 S0 + sum_j ((g_{j+1} .. g_4) k_j) u_j
// which is the rule with the terms in another order, all of it 32-bit or more.  One link now serves four tokens: eight dot products side
// by side, one shuffle tree of eight values that halves what a lane holds at every level, a triangle of six multiply-adds, one
// write.  The multiply-adds of the state are 13 a number and group where the walk has 16, and pairs of rows share a packed
// instruction.
//
// The first kernel, a warp per (group, head), writes what does not depend on the state as one record: with a decay per key channel
// the vectors c_i k_i, c_i q_i, (g_{j+1} .. g_4) k_j and c_4; with one decay a head k_i and q_i (the decays are numbers then); and
// the coefficients.  The second walks the groups of a (sequence, head, tile of columns): KS neighbouring lanes share a
// column, R rows each in registers; records come through a ring in shared memory by cp.async, one barrier a group.
// Groups start at a step's first token of the sequence; a last group is filled up with tokens of zero keys and beta.
//
// 16 heads of 128 x 128 with a decay a channel, one sequence of 2,048 tokens: 630 us by the walk, 530 here (both kernels), 24 heads
// over 1,500 920 and 498, 8 heads with a decay a head 449 and 351; 61 sequences of which one brings 40 tokens 165 and 89.  Against
// 64-bit the outputs are off by 1.28e-7 of their norm by the walk, 1.16e-7 here.  A group is some 430 instructions a warp on its
// way to the next state, and the latency of the shuffles and of the triangle between them.  Heads of at most 64 rows and of
// more than 128 keep the walk: 4 x 64 over 700 tokens 148 us by the walk and 160 here, 3 x 32 over 131 35 and 57, 2 x 256 over 333 91
// and 92: a narrow head's link is short already, a wide one's 16 rows a lane are all instructions.
#pragma once

namespace {

constexpr int DG_TOKENS = 4;   // tokens a group
constexpr int DG_THREADS = 128;
constexpr int DG_STAGES = 6;
// floats of coefficients a record: beta 4, A 6 and two zeros, B 4 x 4 (zeros above its diagonal), c 4, (g_{j+1} .. g_4) 4 (a decay a head)
constexpr int DG_COEF = 36;

constexpr int DG_ROWS = 128;  // rows of a record's vectors, zeros from dk on
__host__ __device__ constexpr int dg_record(bool per_channel) { return (per_channel ? 13 : 8) * DG_ROWS + DG_COEF; }
// Where a sequence's records begin.  Its ceil(len / 4) groups fit before the next sequence's: floor(first / 4) + ceil(len / 4) <=
// floor((first + len) / 4) + 1.
__device__ __forceinline__ int dg_base(int first, int b) { return first / DG_TOKENS + b; }

__device__ __forceinline__ uint64_t dg_pack(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float dg_sum(uint64_t v) {
  float a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
  return a + b;
}
__device__ __forceinline__ uint64_t dg_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t dg_mul(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// ---- the records, a warp per (group, head); a lane owns rows 4 lane .. + 3
__device__ __forceinline__ void dg_load4(const bf16* src, int left, bool wide, float (&f)[4]) {
  if (wide && left >= 4) {
    const uint2 u = *reinterpret_cast<const uint2*>(src);
    const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x)), y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
    f[0] = x.x; f[1] = x.y; f[2] = y.x; f[3] = y.y;
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) f[e] = e < left ? to_float<bf16>(src[e]) : 0.f;
  }
}

__device__ __forceinline__ double dg_warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The norms and the products of decays are made in double, so that an entry of a record is rounded once: a walk token by token
// rounds a decayed state where a record holds decayed keys, and with float factors (one rounding more a token of the
// group) outputs were 0.2 to 7 % further off against 64 bits than the walk's, the state up to 14 %.  With what is taken from a value
// summed first (below) outputs are 0.82 to 1.02 of the walk's error, the state 0.86 to 1.00 (six seeds each of five shapes and three
// rates of decay; where a state hardly decays both sides are off by the decays' own rounding).  16 heads with a decay a channel over
// 2,048 tokens: 513 us with float factors, 530 so; with a decay a head 440 and 448.
template <bool CH>
__global__ void __launch_bounds__(128) delta_group_prepare_kernel(const DeltaParams p, int nseq) {
  pdl_launch();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const long long pair = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
  const long long at = pair / p.H;  // place among all records
  const int h = (int)(pair - at * p.H);
  int b = 0, hi = nseq - 1;  // the last sequence whose records begin at or before it
  while (b < hi) {
    const int mid = (b + hi + 1) >> 1;
    if (dg_base(p.qsl[mid], mid) <= at) b = mid; else hi = mid - 1;
  }
  const int first = p.qsl[b], q_len = p.qsl[b + 1] - first;
  const int grp = (int)(at - dg_base(first, b));
  const int t0 = grp * DG_TOKENS;
  if (t0 >= q_len) return;
  const int nt = min(DG_TOKENS, q_len - t0);
  const int dk = p.dk, kvh = h / (p.H / p.G);
  const size_t n0 = (size_t)(first + t0);
  const bf16* kbase = (const bf16*)p.k + n0 * p.qkv_stride + (size_t)kvh * dk;
  const bf16* qbase = (const bf16*)p.q + n0 * p.qkv_stride + (size_t)kvh * dk;
  const bool wide = (dk & 3) == 0 && (p.qkv_stride & 3) == 0 && ((((uintptr_t)p.k) | ((uintptr_t)p.q)) & 7) == 0;
  const float* abase = p.a + n0 * p.a_stride + (CH ? (size_t)h * dk : (size_t)h);
  const float neg_rate = -expf(p.A_log[h]);
  // a token past the sequence: zero keys, queries and beta, a decay of one
  const int r = 4 * lane;
  float k[DG_TOKENS][4], q[DG_TOKENS][4], g[DG_TOKENS][4];
  float bias[4] = {0.f, 0.f, 0.f, 0.f};
  if (CH)
#pragma unroll
    for (int e = 0; e < 4; ++e) bias[e] = r + e < dk ? p.dt_bias[(size_t)h * dk + r + e] : 0.f;
#pragma unroll
  for (int i = 0; i < DG_TOKENS; ++i) {
    const int left = i < nt ? dk - r : 0;
    dg_load4(kbase + (size_t)i * p.qkv_stride + r, left, wide, k[i]);
    dg_load4(qbase + (size_t)i * p.qkv_stride + r, left, wide, q[i]);
    if (CH)
#pragma unroll
      for (int e = 0; e < 4; ++e) g[i][e] = e < left ? decay_of<bf16>(neg_rate, abase[(size_t)i * p.a_stride + r + e] + bias[e]) : 1.f;
  }
  // lanes 0 .. 3 make a token's beta and (a decay a head) its decay; the logits may come as the slices of a split product, summed
  // in slice order
  float beta = 0.f, gl = 1.f;
  if (lane < nt) {
    const size_t n = n0 + lane;
    float bl = p.b[n * p.b_stride + h], al = CH ? 0.f : abase[(size_t)lane * p.a_stride];
    for (int sl = 1; sl < p.logit_slices; ++sl) {
      bl += p.b[(size_t)sl * p.logit_slice_stride + n * p.b_stride + h];
      if (!CH) al += abase[(size_t)sl * p.logit_slice_stride + (size_t)lane * p.a_stride];
    }
    beta = sigmoid_f(bl);
    if (!CH) gl = decay_of<bf16>(neg_rate, al + p.dt_bias[h]);
  }
  float gh[DG_TOKENS];
#pragma unroll
  for (int i = 0; i < DG_TOKENS; ++i) gh[i] = CH ? 1.f : __shfl_sync(0xffffffffu, gl, i);
  // sums over the rows: |k|^2, |q|^2 and the decayed products of every pair (a decay a head: the plain products)
  double sk[DG_TOKENS] = {}, sq[DG_TOKENS] = {};
  float pa[6] = {}, pb[10] = {};
#pragma unroll
  for (int e = 0; e < 4; ++e)
#pragma unroll
    for (int j = 0; j < DG_TOKENS; ++j) {
      sk[j] = fma((double)k[j][e], (double)k[j][e], sk[j]);
      sq[j] = fma((double)q[j][e], (double)q[j][e], sq[j]);
      float kd = k[j][e];  // (g_{j+1} .. g_i) k_j
      pb[j * (j + 1) / 2 + j] = fmaf(q[j][e], kd, pb[j * (j + 1) / 2 + j]);
#pragma unroll
      for (int i = j + 1; i < DG_TOKENS; ++i) {
        if (CH) kd *= g[i][e];
        pa[i * (i - 1) / 2 + j] = fmaf(k[i][e], kd, pa[i * (i - 1) / 2 + j]);
        pb[i * (i + 1) / 2 + j] = fmaf(q[i][e], kd, pb[i * (i + 1) / 2 + j]);
      }
    }
#pragma unroll
  for (int i = 0; i < DG_TOKENS; ++i) {
    sk[i] = 1.0 / sqrt(dg_warp_sum(sk[i]) + p.norm_eps);
    sq[i] = p.q_scale / sqrt(dg_warp_sum(sq[i]) + p.norm_eps);
  }
  float* rec = p.groups + ((size_t)(dg_base(first, b) + grp) * p.H + h) * dg_record(CH);
  double cp[DG_TOKENS], cs[DG_TOKENS];  // a decay a head: g_1 .. g_i and g_{j+1} .. g_4
  cp[0] = gh[0];
  cs[DG_TOKENS - 1] = 1.0;
#pragma unroll
  for (int i = 1; i < DG_TOKENS; ++i) {
    cp[i] = cp[i - 1] * gh[i];
    cs[DG_TOKENS - 1 - i] = cs[DG_TOKENS - i] * gh[DG_TOKENS - i];
  }
#pragma unroll
  for (int i = 0; i < DG_TOKENS; ++i) {
#pragma unroll
    for (int j = 0; j <= i; ++j) {
      double d = 1.0;
      if (!CH)
#pragma unroll
        for (int e = j + 1; e <= i; ++e) d *= gh[e];
      pb[i * (i + 1) / 2 + j] = (float)(warp_sum(pb[i * (i + 1) / 2 + j]) * (sq[i] * sk[j]) * d);
      if (j < i) pa[i * (i - 1) / 2 + j] = (float)(warp_sum(pa[i * (i - 1) / 2 + j]) * (sk[i] * sk[j]) * d);
    }
  }
  float* co = rec + (CH ? 13 : 8) * DG_ROWS;
  if (lane < DG_TOKENS) co[lane] = beta;
  if (lane == 0) {
#pragma unroll
    for (int i = 0; i < 8; ++i) co[4 + i] = i < 6 ? pa[i < 6 ? i : 0] : 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int j = 0; j < 4; ++j) co[12 + 4 * i + j] = j <= i ? pb[i * (i + 1) / 2 + (j <= i ? j : 0)] : 0.f;
      co[28 + i] = (float)cp[i];
      co[32 + i] = (float)cs[i];
    }
  }
  auto put = [&](int which, const float (&f)[4]) { *reinterpret_cast<float4*>(rec + which * DG_ROWS + r) = make_float4(f[0], f[1], f[2], f[3]); };
  double cc[4] = {1.0, 1.0, 1.0, 1.0}, ss[4] = {1.0, 1.0, 1.0, 1.0};
#pragma unroll
  for (int i = 0; i < DG_TOKENS; ++i) {
    float fk[4], fq[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (CH) cc[e] *= g[i][e];
      fk[e] = (float)(cc[e] * (k[i][e] * sk[i]));
      fq[e] = (float)(cc[e] * (q[i][e] * sq[i]));
    }
    put(i, fk);
    put(DG_TOKENS + i, fq);
    if (CH) {
      const int j = DG_TOKENS - 1 - i;
      float fs[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        fs[e] = (float)(ss[e] * (k[j][e] * sk[j]));
        ss[e] *= g[j][e];
      }
      put(2 * DG_TOKENS + j, fs);
    }
  }
  if (CH) {
    const float c4[4] = {(float)cc[0], (float)cc[1], (float)cc[2], (float)cc[3]};
    put(3 * DG_TOKENS, c4);
  }
}

// ---- the walk over the groups
// Four CTAs an SM: 124 to 128 registers a thread.  Without a bound the compiler takes 90 to 168 and, where it takes 90, puts the
// record's reads where the chain waits for them (16 heads of 128 with a decay a channel over 2,048 tokens 605 us, with it 530; 8 heads
// 438 and 363; 8 sequences of 256 tokens and 8 heads with a decay a head 211 and 166); a bound of one or two gives 136 to 186 and is
// 355 for those 8 heads, but 394 instead of 331 for 50 x 40 tokens, whose CTAs want to share an SM.
template <typename T, int KS, int R, bool CH>
__global__ void __launch_bounds__(DG_THREADS, 4) delta_groups_kernel(const DeltaParams p) {
  pdl_launch();
  pdl_wait();
  static_assert(KS * R == DG_ROWS && KS >= 8, "eight sums a column are shared out over the lanes");
  constexpr int COLS = DG_THREADS / KS, NJ = R / 4, REC = dg_record(CH);
  extern __shared__ __align__(16) float ring[];  // [DG_STAGES][REC]
  const int b = blockIdx.y, h = blockIdx.z;
  const int first = p.qsl[b], q_len = p.qsl[b + 1] - first;
  const int slot = p.state_slots[b];
  if (q_len <= 0 || slot < 0) return;
  const int dk = p.dk, dv = p.dv;
  const int n_groups = (q_len + DG_TOKENS - 1) / DG_TOKENS;
  const float* rec = p.groups + ((size_t)dg_base(first, b) * p.H + h) * REC + 4 * threadIdx.x;
  const size_t rec_step = (size_t)p.H * REC;
  float* const my_ring = ring + 4 * threadIdx.x;
  auto load = [&](int c, int stage) {
    if (c < n_groups) {
      float* dst = my_ring + stage * REC;
#pragma unroll
      for (int i = 0; i < (REC / 4 + DG_THREADS - 1) / DG_THREADS; ++i)
        if (i * DG_THREADS + (int)threadIdx.x < REC / 4) cp_async16(dst + 4 * DG_THREADS * i, rec + 4 * DG_THREADS * i);
      rec += rec_step;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int c = 0; c < DG_STAGES - 1; ++c) load(c, c);

  const int ks = threadIdx.x % KS, col = blockIdx.x * COLS + threadIdx.x / KS;
  const int lane0 = threadIdx.x & 31 & ~(KS - 1);  // the column's first lane
  const bool live = col < dv;
  // lane ks holds rows 4 (j KS + ks) + e: neighbouring lanes read neighbouring 16 bytes of a vector
  float* sg = p.state + (size_t)slot * p.state_stride + (size_t)h * dk * dv + col;
  uint64_t S[R / 2];
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    float s[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int r = 4 * (j * KS + ks) + e;
      s[e] = live && r < dk ? sg[(size_t)r * dv] : 0.f;
    }
    S[2 * j] = dg_pack(s[0], s[1]);
    S[2 * j + 1] = dg_pack(s[2], s[3]);
  }
  const T* vg = (const T*)p.v + (size_t)first * p.qkv_stride + (size_t)h * dv + col;
  float* og = p.out + (size_t)first * p.out_stride + (size_t)h * dv + col;
  // the values of a group are asked for two groups ahead (as they are stored: a conversion there would wait for the load)
  T v[3][DG_TOKENS];
  auto values = [&](int c, T (&dst)[DG_TOKENS]) {
    const bool whole = live && (c + 1) * DG_TOKENS <= q_len;
#pragma unroll
    for (int i = 0; i < DG_TOKENS; ++i) {
      const int t = c * DG_TOKENS + i;
      dst[i] = whole || (live && t < q_len) ? vg[(size_t)t * p.qkv_stride] : from_float<T>(0.f);
    }
  };
  values(0, v[0]);
  values(1, v[1]);

  // Eight sums a column (a_0 .. a_3, p_0 .. p_3): at every level of the tree a lane hands half of its values over, so that the
  // W lanes from i W on end with value i.
  constexpr int W = KS / 8;
  const int held = ks / W;
  int stage = 0;
  auto group = [&](int c, const T (&vv)[DG_TOKENS], T (&ahead)[DG_TOKENS]) {
    asm volatile("cp.async.wait_group %0;" ::"n"(DG_STAGES - 2) : "memory");
    __syncthreads();  // record c has landed for every thread; record c - 1 has been consumed
    load(c + DG_STAGES - 1, stage == 0 ? DG_STAGES - 1 : stage - 1);
    values(c + 2, ahead);
    const float* base = ring + stage * REC;
    stage = stage + 1 == DG_STAGES ? 0 : stage + 1;
    const float* mine = base + 4 * ks;
    const float* co = base + (CH ? 13 : 8) * DG_ROWS;
    auto pairs = [&](int which, int j) { return *reinterpret_cast<const ulonglong2*>(mine + which * DG_ROWS + j * 4 * KS); };
    uint64_t acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0ull;
    // (eight independent sums in turn: a multiply-add does not wait for the one before)
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      ulonglong2 w[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) w[i] = pairs(i, j);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = dg_fma(w[i].x, S[2 * j], acc[i]);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = dg_fma(w[i].y, S[2 * j + 1], acc[i]);
    }
    float sum[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) sum[i] = dg_sum(acc[i]);
#pragma unroll
    for (int st = 0; st < 3; ++st) {
      const int half = 4 >> st, d = KS >> (st + 1);
      const bool upper = (ks & d) != 0;
#pragma unroll
      for (int i = 0; i < half; ++i) {
        const float give = upper ? sum[i] : sum[i + half], keep = upper ? sum[i + half] : sum[i];
        sum[i] = keep + __shfl_xor_sync(0xffffffffu, give, d);
      }
    }
#pragma unroll
    for (int d = W >> 1; d > 0; d >>= 1) sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], d);
    float a[DG_TOKENS];
#pragma unroll
    for (int i = 0; i < DG_TOKENS; ++i) a[i] = __shfl_sync(0xffffffffu, sum[0], lane0 + i * W);
    const float4 beta = *reinterpret_cast<const float4*>(co), A0 = *reinterpret_cast<const float4*>(co + 4);
    const float2 A1 = *reinterpret_cast<const float2*>(co + 8);
    float4 cc = make_float4(1.f, 1.f, 1.f, 1.f), cs = cc;
    if (!CH) {
      cc = *reinterpret_cast<const float4*>(co + 28);
      cs = *reinterpret_cast<const float4*>(co + 32);
      a[0] *= cc.x; a[1] *= cc.y; a[2] *= cc.z; a[3] *= cc.w;
    }
    float u[DG_TOKENS];
    // what is taken from a value is summed first: the sums are small beside it, and so is what they are rounded by
    const float v0 = beta.x * to_float<T>(vv[0]), v1 = beta.y * to_float<T>(vv[1]), v2 = beta.z * to_float<T>(vv[2]), v3 = beta.w * to_float<T>(vv[3]);
    u[0] = fmaf(-beta.x, a[0], v0);
    const float a2 = fmaf(A0.y, u[0], a[2]), a3 = fmaf(A0.w, u[0], a[3]);
    u[1] = fmaf(-beta.y, fmaf(A0.x, u[0], a[1]), v1);
    u[2] = fmaf(-beta.z, fmaf(A0.z, u[1], a2), v2);
    u[3] = fmaf(-beta.w, fmaf(A1.y, u[2], fmaf(A1.x, u[1], a3)), v3);
    // the write: sums over the rows of different lanes and pairs, so the tokens go outside
    uint64_t uu[DG_TOKENS];
    uu[0] = dg_pack(u[0] * cs.x, u[0] * cs.x);
    uu[1] = dg_pack(u[1] * cs.y, u[1] * cs.y);
    uu[2] = dg_pack(u[2] * cs.z, u[2] * cs.z);
    uu[3] = dg_pack(u[3] * cs.w, u[3] * cs.w);
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      ulonglong2 d;
      if (CH)
        d = pairs(3 * DG_TOKENS, j);
      else
        d.x = d.y = dg_pack(cc.w, cc.w);
      S[2 * j] = dg_mul(S[2 * j], d.x);
      S[2 * j + 1] = dg_mul(S[2 * j + 1], d.y);
    }
#pragma unroll
    for (int i = 0; i < DG_TOKENS; ++i)
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const ulonglong2 k = pairs((CH ? 2 * DG_TOKENS : 0) + i, j);
        S[2 * j] = dg_fma(k.x, uu[i], S[2 * j]);
        S[2 * j + 1] = dg_fma(k.y, uu[i], S[2 * j + 1]);
      }
    // the lane that holds p_i finishes o_i; what a later token of the group brings (NaN, infinities) stays out of it
    const int tok = held - DG_TOKENS, t = c * DG_TOKENS + tok;
    if (tok >= 0 && (ks & (W - 1)) == 0 && live && t < q_len) {
      const float4 B = *reinterpret_cast<const float4*>(co + 12 + 4 * tok);
      float o = sum[0];
      if (!CH) o *= tok == 0 ? cc.x : tok == 1 ? cc.y : tok == 2 ? cc.z : cc.w;
      o = fmaf(B.x, u[0], o);
      if (tok >= 1) o = fmaf(B.y, u[1], o);
      if (tok >= 2) o = fmaf(B.z, u[2], o);
      if (tok >= 3) o = fmaf(B.w, u[3], o);
      og[(size_t)t * p.out_stride] = o;
    }
  };
  for (int c = 0; c < n_groups; c += 3) {
    group(c, v[0], v[2]);
    if (c + 1 < n_groups) group(c + 1, v[1], v[0]);
    if (c + 2 < n_groups) group(c + 2, v[2], v[1]);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    float s[4];
    asm("mov.b64 {%0, %1}, %2;" : "=f"(s[0]), "=f"(s[1]) : "l"(S[2 * j]));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(s[2]), "=f"(s[3]) : "l"(S[2 * j + 1]));
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int r = 4 * (j * KS + ks) + e;
      if (live && r < dk) sg[(size_t)r * dv] = s[e];
    }
  }
}

template <typename T, int KS, int R, bool CH>
int launch_delta_groups(const DeltaParams& p, int B, cudaStream_t st) {
  constexpr int COLS = DG_THREADS / KS;
  const dim3 grid((p.dv + COLS - 1) / COLS, B, p.H);
  const size_t smem = spread_smem((size_t)DG_STAGES * dg_record(CH) * sizeof(float), (long long)grid.x * grid.y * grid.z);
  auto kern = delta_groups_kernel<T, KS, R, CH>;
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  return launch(kern, grid, dim3(DG_THREADS), smem, st, p);
}

template <typename T, bool CH>
int dispatch_delta_groups(const DeltaParams& p, int B, cudaStream_t st) {
  static_assert(sizeof(T) == 2, "bfloat16 storage");
  const long long warps = ((long long)p.N / DG_TOKENS + B) * p.H;
  if ((unsigned)B > 65535u || (warps + 3) / 4 > 0x7fffffffll) return (int)cudaErrorInvalidValue;
  const dim3 grid((unsigned)((warps + 3) / 4));
  const int rc = launch(delta_group_prepare_kernel<CH>, grid, dim3(128), 0, st, p, B);
  if (rc) return rc;
  // (Figures here are from before the records' factors were double and the order of the sums below.)
  // What counts for a few long sequences is a short link (16 lanes a column: 16 heads of 128 x 128 over 2,048 tokens 513 us against
  // 506, 24 heads over 1,500 464 against 538, 8 x 256 tokens of 16 heads 348 against 388; with a decay a head 349 against 465 for
  // 8 heads); once every SM has more than a dozen CTAs to work off it is the number of instructions (8 lanes: 50 x 40 tokens of 16
  // heads 322 us against 384, 30 x 5 64 against 86).
  const bool few = (long long)B * p.H * ((p.dv + 15) / 16) <= 12 * 148;
  return few ? launch_delta_groups<T, 16, 8, CH>(p, B, st) : launch_delta_groups<T, 8, 16, CH>(p, B, st);
}

}  // namespace
