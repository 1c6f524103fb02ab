// The gated delta rule sixty-four tokens at a time, for steps that bring a sequence many tokens in bfloat16 storage.  Included by
// sequence_mix.cuh; the forms it stands beside are the walk (sequence_mix.cuh) and the groups of four (delta_groups.cuh), whose
// notation this is:
//   a_i = (c_i k_i)^T S0       p_i = (c_i q_i)^T S0
//   A_ij = k_i^T (g_{j+1} .. g_i) k_j  (j < i)      B_ij = q_i^T (g_{j+1} .. g_i) k_j  (j <= i)
//   u_i = beta_i (v_i - a_i - sum_{j<i} A_ij u_j)    o_i = p_i + sum_{j<=i} B_ij u_j
//   S   = c_n S0 + sum_j ((g_{j+1} .. g_n) k_j) u_j
// The u of a chunk are linear in S0: u = U - W S0, where U and W solve (1 + beta A) [U W] = beta [V  c k] by forward substitution.
// So everything but two products a chunk is done for all chunks at once, and a sequence's chain has one link for 64 tokens:
//   prepare : a CTA a (chunk, head): unit keys and queries, the products of decays, A, B, the solve;
//   chain   : a CTA a (sequence, head, tile of columns): u = U - W S, S <- c S + K^T u, chunk by chunk; it leaves every chunk's S0;
//   read    : a CTA a (chunk, head, 64 columns): o = (c q) S0 + B u.
// All of it is float on the FP32 pipes, packed two to an instruction; the norms and products of decays are double, as in the groups.
//
// Nothing overflows and nothing is divided, whatever the decays are: a chunk is four blocks of 16 tokens.  Inside a block A and B
// take the product of the very decays between the two tokens; between blocks J < I it is (decays from the start of I up to i) x (of
// the blocks between) x (from j to the end of J), all factors at most one.
//
// 16 heads of 128 x 128 with a decay a channel, one sequence of 2,048 tokens: 269 us (prepare 124, chain 98, read 45) against 525 by
// groups of four; 24 heads over 1,500 tokens 292 and 498, 8 heads with a decay a head over 2,048 187 and 351.  All three kernels are bound
// by what shared memory hands to registers, 4 bytes a lane and cycle: the broadcast of A in the solve (a word a multiply-add), 8 x 4 and
// 4 x 4 register tiles elsewhere.  A link of the chain is 3.1 us (of some 5,800 cycles 3,600 are
// its reads of W, S, K and u; with the rows of W S shared out over the warps instead of its tokens, and so with sums that go through
// shared memory and two barriers more, 3.3 us).
// Against 64 bits the outputs are off by 1.10e-7 of their norm there (groups 1.16e-7, walk 1.28e-7), the states by 0.89e-7 (0.91e-7,
// 0.96e-7); over three rates of decay and three seeds each outputs are 0.86 to 1.01 of the groups' error and at most the walk's.  That
// takes sums of A and B inside a block ended in double (those between blocks end in float), and beta x kept whole in the solve (without
// them 1.06).
#pragma once

namespace {

constexpr int DC_T = 64;          // tokens a chunk
constexpr int DC_ROWS = 128;      // rows of a state, zeros from dk on
constexpr int DC_THREADS = 256;
// a record, in floats: W^T [128][64], K [64][128] (decayed to the chunk's end; 16-byte words of odd tokens swapped in groups of four),
// (c q)^T [128][64], B^T [64 j][64 i], c_n [128]; then U [64][dv], which the chain overwrites by u, and S0 [128][dv]
constexpr int DC_WT = 0, DC_KH = 8192, DC_QT = 16384, DC_BT = 24576, DC_CT = 28672, DC_U = 28800;
__host__ __device__ constexpr long long dc_record(int dv) { return DC_U + (long long)(DC_T + DC_ROWS) * dv; }
// Where a sequence's records begin (as for the groups: ceil(len / 64) of them fit before the next sequence's).
__device__ __forceinline__ int dc_base(int first, int b) { return first / DC_T + b; }

// the sequence and chunk of a record; false for a record that nothing uses
__device__ __forceinline__ bool dc_find(const int* qsl, int nseq, int at, int& first, int& n) {
  int b = 0, hi = nseq - 1;  // the last sequence whose records begin at or before it
  while (b < hi) {
    const int mid = (b + hi + 1) >> 1;
    if (dc_base(qsl[mid], mid) <= at) b = mid; else hi = mid - 1;
  }
  const int q_len = qsl[b + 1] - qsl[b], t0 = (at - dc_base(qsl[b], b)) * DC_T;
  first = qsl[b] + t0;
  n = min(DC_T, q_len - t0);
  return t0 >= 0 && n > 0;
}

// float index of (token, number) in a [64][128] tile whose 16-byte words are swapped by the token's low bits
__device__ __forceinline__ int dc_at(int t, int d) { return t * DC_ROWS + ((((d >> 2) ^ (t & 7))) << 2) + (d & 3); }
__device__ __forceinline__ ulonglong2 dc_pairs(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }
__device__ __forceinline__ uint64_t dc_add(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// the sum of four neighbouring lanes' pairs
__device__ __forceinline__ double dc_sum4(uint64_t v) {
  float a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
  double d = (double)a + (double)b;
  d += __shfl_xor_sync(0xffffffffu, d, 1);
  return d + __shfl_xor_sync(0xffffffffu, d, 2);
}
__device__ __forceinline__ uint64_t dc_both(float a) { return dg_pack(a, a); }
__device__ __forceinline__ void dc_split(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
// block (J, I), J <= I, of the ten 16 x 16 blocks that A^T is kept as: [j][i]
__host__ __device__ constexpr int dc_block(int J, int I) { return (J * 4 - J * (J - 1) / 2 + (I - J)) * 256; }

constexpr int DC_SMEM_FLOATS = 3 * DC_T * DC_ROWS + 10 * 256 + DC_T;
constexpr size_t DC_PREPARE_SMEM = (size_t)DC_SMEM_FLOATS * 4 + (2 * DC_T + 4 * DC_ROWS) * 8;

// A and B between block I and the blocks before it: 16 rows of keys and 16 of queries by 16 I columns, 4 x 4 a thread, KS threads a tile.
template <int I>
__device__ __forceinline__ void dc_between(const float* K, const float* Q, const float* R, float* A, float* bt) {
  constexpr int KS = I == 1 ? 8 : I == 2 ? 4 : 2, CT = 4 * I;  // tiles: 8 of rows by CT of columns
  const int ks = threadIdx.x % KS, tile = threadIdx.x / KS, rt = tile & 7, ct = tile >> 3;
  const bool live = ct < CT;  // (whole warps except for I = 3, where the last two warps are out)
  uint64_t acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
  if (live) {
    const int t0 = 16 * I + rt;
#pragma unroll 2
    for (int m = 0; m < 32 / KS; ++m) {
      const int d = 4 * (ks + KS * m);
      ulonglong2 a[4], b[4];
      a[0] = dc_pairs(K + dc_at(t0, d));
      a[1] = dc_pairs(K + dc_at(t0 + 8, d));
      a[2] = dc_pairs(Q + dc_at(t0, d));
      a[3] = dc_pairs(Q + dc_at(t0 + 8, d));
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = dc_pairs(R + dc_at(ct + CT * j, d));
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = dc_add(dg_fma(a[i].y, b[j].y, dg_mul(a[i].x, b[j].x)), acc[i][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float s = dg_sum(acc[i][j]);
#pragma unroll
      for (int o = 1; o < KS; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (live && ks == 0) {
        const int jj = ct + CT * j, ii = rt + 8 * (i & 1);
        if (i < 2)
          A[dc_block(0, 0) + ((jj >> 4) * 4 - (jj >> 4) * ((jj >> 4) - 1) / 2 + (I - (jj >> 4))) * 256 + (jj & 15) * 16 + ii] = s;
        else
          bt[jj * DC_T + 16 * I + ii] = s;
      }
    }
}

template <bool CHANNEL>
__global__ void __launch_bounds__(DC_THREADS, 2) delta_chunk_prepare_kernel(const DeltaParams p, int nseq) {
  pdl_launch();
  pdl_wait();
  extern __shared__ __align__(16) float sm[];
  float* const K = sm;                       // raw keys, then decayed from their block's start
  float* const Q = K + DC_T * DC_ROWS;       // the same of the queries
  float* const G = Q + DC_T * DC_ROWS;       // decays, then keys decayed to their block's end (and on, block by block)
  float* const A = G + DC_T * DC_ROWS;       // A^T in blocks
  float* const beta = A + 10 * 256;
  double* const sk = reinterpret_cast<double*>(beta + DC_T);
  double* const sq = sk + DC_T;
  double* const PB = sq + DC_T;              // [4][128] a block's product of decays
  const int at = blockIdx.x / p.H, h = blockIdx.x - at * p.H;
  int first, n;
  if (!dc_find(p.qsl, nseq, at, first, n)) return;
  const int dk = p.dk, dv = p.dv, kvh = h / (p.H / p.G), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float* const rec = p.chunks + ((size_t)at * p.H + h) * dc_record(dv);

  // ---- keys, queries, decays: zero keys and queries and decays of one past the sequence and past dk
  {
    const bf16* kb = (const bf16*)p.k + (size_t)first * p.qkv_stride + (size_t)kvh * dk;
    const bf16* qb = (const bf16*)p.q + (size_t)first * p.qkv_stride + (size_t)kvh * dk;
    const bool wide = (dk & 3) == 0 && (p.qkv_stride & 3) == 0 && ((((uintptr_t)p.k) | ((uintptr_t)p.q)) & 7) == 0;
    const float* ab = p.a + (size_t)first * p.a_stride + (CHANNEL ? (size_t)h * dk : (size_t)h);
    const float neg_rate = -expf(p.A_log[h]);
    float bias[4] = {0.f, 0.f, 0.f, 0.f};
    const int r = 4 * lane;
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (CHANNEL) bias[e] = r + e < dk ? p.dt_bias[(size_t)h * dk + r + e] : 0.f;
    if (!CHANNEL) bias[0] = p.dt_bias[h];
    const bool awide = CHANNEL && (dk & 3) == 0 && (p.a_stride & 3) == 0 && (((uintptr_t)p.a) & 15) == 0;
    constexpr int WARPS = DC_THREADS / 32, PER = DC_T / WARPS;
    // (all of a warp's rows are asked for before any is used: a branch or a conversion between them would wait for each in turn)
    uint2 rk[PER], rq[PER];
    float4 ra[PER];
    const bool words = wide && (!CHANNEL || awide);  // of four numbers, dk a multiple of them
    if (words) {
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int t = warp + WARPS * i;
        const bool in = t < n && r < dk;
        rk[i] = in ? *reinterpret_cast<const uint2*>(kb + (size_t)t * p.qkv_stride + r) : make_uint2(0u, 0u);
        rq[i] = in ? *reinterpret_cast<const uint2*>(qb + (size_t)t * p.qkv_stride + r) : make_uint2(0u, 0u);
        if (CHANNEL) ra[i] = in ? *reinterpret_cast<const float4*>(ab + (size_t)t * p.a_stride + r) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int t = warp + WARPS * i, left = t < n ? dk - r : 0;
      float fk[4], fq[4], g[4] = {1.f, 1.f, 1.f, 1.f}, x[4] = {0.f, 0.f, 0.f, 0.f};
      if (words) {
        const uint32_t w[4] = {rk[i].x, rk[i].y, rq[i].x, rq[i].y};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          fk[e] = __uint_as_float((e & 1) ? w[e >> 1] & 0xffff0000u : w[e >> 1] << 16);
          fq[e] = __uint_as_float((e & 1) ? w[2 + (e >> 1)] & 0xffff0000u : w[2 + (e >> 1)] << 16);
        }
        if (CHANNEL) x[0] = ra[i].x, x[1] = ra[i].y, x[2] = ra[i].z, x[3] = ra[i].w;
      } else {
        dg_load4(kb + (size_t)t * p.qkv_stride + r, left, false, fk);
        dg_load4(qb + (size_t)t * p.qkv_stride + r, left, false, fq);
        if (CHANNEL)
#pragma unroll
          for (int e = 0; e < 4; ++e) x[e] = e < left ? ab[(size_t)t * p.a_stride + r + e] : 0.f;
      }
      if (CHANNEL) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float y = decay_of<bf16>(neg_rate, x[e] + bias[e]);
          g[e] = e < left ? y : 1.f;
        }
      } else if (t < n) {  // (the logits may come as the slices of a split product, summed in slice order)
        float al = ab[(size_t)t * p.a_stride];
        for (int sl = 1; sl < p.logit_slices; ++sl) al += ab[(size_t)sl * p.logit_slice_stride + (size_t)t * p.a_stride];
        g[0] = g[1] = g[2] = g[3] = decay_of<bf16>(neg_rate, al + bias[0]);
      }
      *reinterpret_cast<float4*>(K + dc_at(t, r)) = make_float4(fk[0], fk[1], fk[2], fk[3]);
      *reinterpret_cast<float4*>(Q + dc_at(t, r)) = make_float4(fq[0], fq[1], fq[2], fq[3]);
      *reinterpret_cast<float4*>(G + dc_at(t, r)) = make_float4(g[0], g[1], g[2], g[3]);
      double nk = 0.0, nq = 0.0;  // |k|^2, |q|^2
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        nk = fma((double)fk[e], (double)fk[e], nk);
        nq = fma((double)fq[e], (double)fq[e], nq);
      }
      nk = dg_warp_sum(nk);
      nq = dg_warp_sum(nq);
      if (lane == 0) {
        sk[t] = nk;
        sq[t] = nq;
      }
    }
    if (tid < DC_T) {
      float bl = 0.f;
      if (tid < n) {
        const float* br = p.b + (size_t)(first + tid) * p.b_stride + h;
        bl = br[0];
        for (int sl = 1; sl < p.logit_slices; ++sl) bl += br[(size_t)sl * p.logit_slice_stride];
        bl = sigmoid_f(bl);
      }
      beta[tid] = bl;
    }
  }
  __syncthreads();
  // (a thread a token: a warp that divides for its tokens in turn takes 30,000 cycles)
  if (tid < DC_T)
    sk[tid] = 1.0 / sqrt(sk[tid] + p.norm_eps);
  else if (tid < 2 * DC_T)
    sq[tid - DC_T] = p.q_scale / sqrt(sq[tid - DC_T] + p.norm_eps);
  __syncthreads();

  // ---- A and B inside the blocks: four threads (every fourth 16-byte word) two keys j and j + 8, which walk to the tokens after them;
  // half of the warps take A, half B
  {
    const int ds = tid & 3, j = (tid >> 2) & 7, blk = warp & 3, t0 = 16 * blk;
    const bool is_b = warp >= 4;
    const float* const X = is_b ? Q : K;
    uint64_t lo[16], hi[8];
#pragma unroll
    for (int i = 0; i < 16; ++i) lo[i] = 0ull;
#pragma unroll
    for (int i = 0; i < 8; ++i) hi[i] = 0ull;
#pragma unroll 1
    for (int m = 0; m < 8; ++m) {
      const int d = 4 * (ds + 4 * m);
      ulonglong2 k0 = dc_pairs(K + dc_at(t0 + j, d)), k1 = dc_pairs(K + dc_at(t0 + 8 + j, d));
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const ulonglong2 x = dc_pairs(X + dc_at(t0 + i, d));
        if (i > 0) {  // (what a token brings reaches none before it)
          const float4 g = *reinterpret_cast<const float4*>(G + dc_at(t0 + i, d));
          if (i < 8) {
            const bool on = i > j;
            k0.x = dg_mul(k0.x, dg_pack(on ? g.x : 1.f, on ? g.y : 1.f));
            k0.y = dg_mul(k0.y, dg_pack(on ? g.z : 1.f, on ? g.w : 1.f));
          } else {
            const bool on = i - 8 > j;
            k0.x = dg_mul(k0.x, dg_pack(g.x, g.y));
            k0.y = dg_mul(k0.y, dg_pack(g.z, g.w));
            k1.x = dg_mul(k1.x, dg_pack(on ? g.x : 1.f, on ? g.y : 1.f));
            k1.y = dg_mul(k1.y, dg_pack(on ? g.z : 1.f, on ? g.w : 1.f));
          }
        }
        lo[i] = dc_add(dg_fma(x.y, k0.y, dg_mul(x.x, k0.x)), lo[i]);
        if (i >= 8) hi[i - 8] = dc_add(dg_fma(x.y, k1.y, dg_mul(x.x, k1.x)), hi[i - 8]);
      }
    }
    const double* const sx = is_b ? sq : sk;
    const double c0 = sk[t0 + j], c1 = sk[t0 + 8 + j];
    float f0[16], f1[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      f0[i] = (float)(dc_sum4(lo[i]) * (sx[t0 + i] * c0));
      f1[i] = i < 8 ? 0.f : (float)(dc_sum4(hi[i < 8 ? 0 : i - 8]) * (sx[t0 + i] * c1));
      if (i < j + (is_b ? 0 : 1)) f0[i] = 0.f;
      if (i < j + 8 + (is_b ? 0 : 1)) f1[i] = 0.f;
    }
    float* const to = is_b ? rec + DC_BT + (size_t)(t0 + j) * DC_T + t0 : A + (blk * 4 - blk * (blk - 1) / 2) * 256 + j * 16;
    const int step = is_b ? 8 * DC_T : 8 * 16;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (ds == q) {
        *reinterpret_cast<float4*>(to + 4 * q) = make_float4(f0[4 * q], f0[4 * q + 1], f0[4 * q + 2], f0[4 * q + 3]);
        *reinterpret_cast<float4*>(to + step + 4 * q) = make_float4(f1[4 * q], f1[4 * q + 1], f1[4 * q + 2], f1[4 * q + 3]);
      }
  }
  __syncthreads();

  // ---- products of decays: two (block, channel) pairs a thread
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const int d = tid & 127, blk = (tid >> 7) + 2 * it;
    double c = 1.0;
#pragma unroll
    for (int i = 0; i < 16; ++i) c *= G[dc_at(16 * blk + i, d)];
    PB[blk * DC_ROWS + d] = c;
  }
  __syncthreads();
#pragma unroll 1
  for (int it = 0; it < 2; ++it) {
    const int d = tid & 127, blk = (tid >> 7) + 2 * it, t0 = 16 * blk;
    double pre = 1.0, post = 1.0;
#pragma unroll
    for (int J = 0; J < 4; ++J) {
      if (J < blk) pre *= PB[J * DC_ROWS + d];
      if (J > blk) post *= PB[J * DC_ROWS + d];
    }
    float g[16], k[16], q[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int x = dc_at(t0 + i, d);
      g[i] = G[x];
      k[i] = K[x];
      q[i] = Q[x];
    }
    double c = 1.0;
#pragma unroll
    for (int i4 = 0; i4 < 4; ++i4) {
      float kc[4], qc[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = 4 * i4 + e, x = dc_at(t0 + i, d);
        c *= g[i];
        const double fk = c * (k[i] * sk[t0 + i]), fq = c * (q[i] * sq[t0 + i]);
        K[x] = (float)fk;
        Q[x] = (float)fq;
        kc[e] = (float)(pre * fk);
        qc[e] = (float)(pre * fq);
      }
      // (c k goes where W will be: the solve reads it from there)
      *reinterpret_cast<float4*>(rec + DC_WT + (size_t)d * DC_T + t0 + 4 * i4) = make_float4(kc[0], kc[1], kc[2], kc[3]);
      *reinterpret_cast<float4*>(rec + DC_QT + (size_t)d * DC_T + t0 + 4 * i4) = make_float4(qc[0], qc[1], qc[2], qc[3]);
    }
    if (blk == 3) rec[DC_CT + d] = (float)(pre * c);
    double s = 1.0;
#pragma unroll
    for (int i = 15; i >= 0; --i) {
      const double fk = s * (k[i] * sk[t0 + i]);
      s *= g[i];
      G[dc_at(t0 + i, d)] = (float)fk;
      rec[DC_KH + (t0 + i) * DC_ROWS + ((((d >> 2) ^ ((i & 1) << 2))) << 2) + (d & 3)] = (float)(post * fk);
    }
  }
  __syncthreads();

  // ---- A and B between blocks; keys of blocks before I are carried through block I once it is done
  float* const bt = rec + DC_BT;
  auto carry = [&](int I) {
    __syncthreads();
    const int d = tid & 127;
    const float f = (float)PB[I * DC_ROWS + d];
    for (int t = tid >> 7; t < 16 * I; t += 2) G[dc_at(t, d)] *= f;
    __syncthreads();
  };
  dc_between<1>(K, Q, G, A, bt);
  carry(1);
  dc_between<2>(K, Q, G, A, bt);
  carry(2);
  dc_between<3>(K, Q, G, A, bt);
  __syncthreads();

  // ---- the solve: a thread a column, of c k (the first four warps) and of v; what is taken from a value is summed first
  for (int col = tid; col < DC_ROWS + dv; col += DC_THREADS) {
    const bool is_k = col < DC_ROWS;
    const int cv = col - DC_ROWS;
    float* const wt = rec + DC_WT + (size_t)(is_k ? col : 0) * DC_T;
    float* const ut = rec + DC_U + (is_k ? 0 : cv);
    const unsigned short* const vg = (const unsigned short*)p.v + (size_t)first * p.qkv_stride + (size_t)h * dv + (is_k ? 0 : cv);
    const int shift = is_k ? 0 : 16;  // a value of 16 bits is made a float where it is used: a conversion here would wait for it
    auto fetch = [&](int t, uint32_t (&x)[4]) {
      if (is_k) {
        const uint4 f = __ldcg(reinterpret_cast<const uint4*>(wt + t));
        x[0] = f.x; x[1] = f.y; x[2] = f.z; x[3] = f.w;
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) x[e] = t + e < n ? (uint32_t)vg[(size_t)(t + e) * p.qkv_stride] : 0u;
      }
    };
    uint64_t s[DC_T / 2];
#pragma unroll
    for (int i = 0; i < DC_T / 2; ++i) s[i] = 0ull;
    uint32_t x[4][4];  // asked for three words ahead
    fetch(0, x[0]);
    fetch(4, x[1]);
    fetch(8, x[2]);
#pragma unroll
    for (int jq = 0; jq < 16; ++jq) {
      if (jq + 3 < 16) fetch(4 * jq + 12, x[(jq + 3) & 3]);
      const float4 b4 = *reinterpret_cast<const float4*>(beta + 4 * jq);
      float u[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int j = 4 * jq + e;
        const float bj = e == 0 ? b4.x : e == 1 ? b4.y : e == 2 ? b4.z : b4.w;
        float lo, hi;
        dc_split(s[j >> 1], lo, hi);
        // beta x is kept whole: a chunk's u is rounded once more than a group's, when the chain takes W S from it
        const float xv = __uint_as_float(x[jq & 3][e] << shift), bx = bj * xv, rest = fmaf(bj, xv, -bx);
        u[e] = bx + fmaf(-bj, (j & 1) ? hi : lo, rest == rest ? rest : 0.f);  // (an infinite value has no rest)
        const uint64_t uu = dc_both(u[e]);
#pragma unroll
        for (int iq = (j + 1) / 4; iq < 16; ++iq) {
          const ulonglong2 a = dc_pairs(A + dc_block(j >> 4, iq >> 2) + (j & 15) * 16 + 4 * (iq & 3));
          s[2 * iq] = dg_fma(a.x, uu, s[2 * iq]);
          s[2 * iq + 1] = dg_fma(a.y, uu, s[2 * iq + 1]);
        }
        if (!is_k) ut[(size_t)j * dv] = u[e];
      }
      if (is_k) *reinterpret_cast<float4*>(wt + 4 * jq) = make_float4(u[0], u[1], u[2], u[3]);
    }
  }
}

// ---- the chain
template <int DVT> constexpr size_t dc_chain_smem() { return (size_t)(2 * (2 * 8192 + DC_T * DVT + DC_ROWS) + DC_ROWS * DVT) * 4; }

template <int DVT>
__global__ void __launch_bounds__(DC_THREADS, 1) delta_chunk_chain_kernel(const DeltaParams p) {
  pdl_launch();
  pdl_wait();
  static_assert(DVT == 16 || DVT == 32, "a thread's columns are one or two 16-byte words");
  constexpr int NQ = DVT / 16, STAGE = 2 * 8192 + DC_T * DVT + DC_ROWS;
  extern __shared__ __align__(16) float sm[];
  float* const S = sm + 2 * STAGE;            // [128][DVT]
  const int b = blockIdx.y, h = blockIdx.z, c0 = blockIdx.x * DVT;
  const int first = p.qsl[b], q_len = p.qsl[b + 1] - first;
  const int slot = p.state_slots[b];
  if (q_len <= 0 || slot < 0) return;
  const int dk = p.dk, dv = p.dv, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int chunks = (q_len + DC_T - 1) / DC_T;
  const size_t step = (size_t)p.H * dc_record(dv);
  float* const rec0 = p.chunks + ((size_t)dc_base(first, b) * p.H + h) * dc_record(dv);
  // place of a 16-byte word of columns in a row of u or S: odd rows' words lie elsewhere, so that two rows' reads do not collide
  // (as those of W^T do)
  auto word = [](int t, int q) { return DVT == 32 ? q ^ ((t & 1) << 2) : q; };
  auto load = [&](int c) {
    if (c < chunks) {
      const float* rec = rec0 + (size_t)c * step;
      float* dst = sm + (c & 1) * STAGE;
#pragma unroll
      for (int i = 0; i < 16; ++i) cp_async16(dst + 4 * ((i < 8 ? tid ^ ((tid >> 4) & 1) : tid) + 256 * i), rec + 4 * (tid + 256 * i));  // W^T, then K
      float* ud = dst + 2 * 8192;
#pragma unroll
      for (int i = 0; i < NQ; ++i) {
        const int idx = tid + 256 * i, t = idx / (DVT / 4), q = idx % (DVT / 4);
        float* to = ud + t * DVT + 4 * word(t, q);
        if (c0 + 4 * q < dv)
          cp_async16(to, rec + DC_U + (size_t)t * dv + c0 + 4 * q);
        else
          *reinterpret_cast<float4*>(to) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
      if (tid < DC_ROWS / 4) cp_async16(ud + DC_T * DVT + 4 * tid, rec + DC_CT + 4 * tid);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  load(0);
  float* const sg = p.state + (size_t)slot * p.state_stride + (size_t)h * dk * dv + c0;
  // a warp owns rows 16 warp .. + 15 of S throughout
  for (int idx = lane; idx < 16 * DVT; idx += 32) {
    const int r = 16 * warp + idx / DVT, c = idx % DVT;
    S[r * DVT + 4 * word(r, c >> 2) + (c & 3)] = r < dk && c0 + c < dv ? sg[(size_t)r * dv + c] : 0.f;
  }
  for (int c = 0; c < chunks; ++c) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // the stage is there, S is whole and the other stage has been read
    load(c + 1);
    const float* const W = sm + (c & 1) * STAGE;
    const float* const Kh = W + 8192;
    float* const U = sm + (c & 1) * STAGE + 2 * 8192;
    const float* const ct = U + DC_T * DVT;
    float* const rec = rec0 + (size_t)c * step;
#pragma unroll
    for (int i = 0; i < DVT / 8; ++i) {  // S0 for the read-out
      const int idx = lane + 32 * i, r = 16 * warp + idx / (DVT / 4), q = idx % (DVT / 4);
      if (c0 + 4 * q < dv)
        *reinterpret_cast<float4*>(rec + DC_U + (size_t)(DC_T + r) * dv + c0 + 4 * q) = *reinterpret_cast<const float4*>(S + r * DVT + 4 * word(r, q));
    }
    {  // u = U - W S for tokens 8 warp .. + 7: rows kg, kg + 8 .. of S, columns 4 cg .. + 3 (and 16 on); then the eight kg are summed
      const int cg = lane & 3, kg = lane >> 2;
      uint64_t acc[4][4 * NQ];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4 * NQ; ++j) acc[i][j] = 0ull;
      const float* const wp = W + kg * DC_T + 8 * warp;
      const int odd = kg & 1;
#pragma unroll
      for (int kk = 0; kk < 16; ++kk) {
        const ulonglong2 w0 = dc_pairs(wp + 8 * kk * DC_T + 4 * odd), w1 = dc_pairs(wp + 8 * kk * DC_T + 4 - 4 * odd);
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
          const float4 s4 = *reinterpret_cast<const float4*>(S + (kg + 8 * kk) * DVT + 4 * word(kg, 4 * q + cg));
          const uint64_t s[4] = {dc_both(s4.x), dc_both(s4.y), dc_both(s4.z), dc_both(s4.w)};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            acc[0][4 * q + j] = dg_fma(w0.x, s[j], acc[0][4 * q + j]);
            acc[1][4 * q + j] = dg_fma(w0.y, s[j], acc[1][4 * q + j]);
            acc[2][4 * q + j] = dg_fma(w1.x, s[j], acc[2][4 * q + j]);
            acc[3][4 * q + j] = dg_fma(w1.y, s[j], acc[3][4 * q + j]);
          }
        }
      }
      // a lane keeps half of what it has at each of three exchanges: the last is one token's four columns
      const int t = 8 * warp + kg;
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        float s[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint64_t two[2];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const uint64_t keep = (kg & 4) ? acc[2 + i][4 * q + j] : acc[i][4 * q + j], give = (kg & 4) ? acc[i][4 * q + j] : acc[2 + i][4 * q + j];
            two[i] = dc_add(keep, __shfl_xor_sync(0xffffffffu, give, 16));
          }
          const uint64_t keep = (kg & 2) ? two[1] : two[0], give = (kg & 2) ? two[0] : two[1];
          float lo, hi;
          dc_split(dc_add(keep, __shfl_xor_sync(0xffffffffu, give, 8)), lo, hi);
          s[j] = (odd ? hi : lo) + __shfl_xor_sync(0xffffffffu, odd ? lo : hi, 4);
        }
        float4* const at = reinterpret_cast<float4*>(U + t * DVT + 4 * word(t, 4 * q + cg));
        float4 u = *at;
        u.x -= s[0]; u.y -= s[1]; u.z -= s[2]; u.w -= s[3];
        *at = u;
        if (c0 + 16 * q + 4 * cg < dv) *reinterpret_cast<float4*>(rec + DC_U + (size_t)t * dv + c0 + 16 * q + 4 * cg) = u;
      }
    }
    __syncthreads();
    {  // S <- c S + K^T u on the warp's rows: every other token, rows 4 rg .. + 3, columns 4 cg .. + 3 (and 16 on)
      const int th = lane & 1, rg = (lane >> 1) & 3, cg = lane >> 3;
      uint64_t acc[2][4 * NQ];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4 * NQ; ++j) acc[i][j] = 0ull;
      const float* const kp = Kh + th * DC_ROWS + (((4 * warp + rg) ^ (th << 2)) << 2);
#pragma unroll 8
      for (int s = 0; s < 32; ++s) {
        const ulonglong2 k = dc_pairs(kp + 2 * s * DC_ROWS);
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
          const float4 u4 = *reinterpret_cast<const float4*>(U + (2 * s + th) * DVT + 4 * word(th, 4 * q + cg));
          const uint64_t u[4] = {dc_both(u4.x), dc_both(u4.y), dc_both(u4.z), dc_both(u4.w)};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            acc[0][4 * q + j] = dg_fma(k.x, u[j], acc[0][4 * q + j]);
            acc[1][4 * q + j] = dg_fma(k.y, u[j], acc[1][4 * q + j]);
          }
        }
      }
      const float4 c4 = *reinterpret_cast<const float4*>(ct + 16 * warp + 4 * rg);
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        // the two lanes of a pair share the sums out: the first keeps two columns, the second the others
        float v[2][4];  // [column kept][row]
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            float a0, a1, b0, b1;
            dc_split(acc[i][4 * q + j], a0, a1);
            dc_split(acc[i][4 * q + 2 + j], b0, b1);
            const float g0 = th ? a0 : b0, g1 = th ? a1 : b1, k0 = th ? b0 : a0, k1 = th ? b1 : a1;
            v[j][2 * i] = k0 + __shfl_xor_sync(0xffffffffu, g0, 1);
            v[j][2 * i + 1] = k1 + __shfl_xor_sync(0xffffffffu, g1, 1);
          }
        float* const at = S + (16 * warp + 4 * rg) * DVT + 2 * th;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          float2* const s2 = reinterpret_cast<float2*>(at + r * DVT + 4 * word(r, 4 * q + cg));
          const float cr = r == 0 ? c4.x : r == 1 ? c4.y : r == 2 ? c4.z : c4.w;
          const float2 old = *s2;
          *s2 = make_float2(fmaf(cr, old.x, v[0][r]), fmaf(cr, old.y, v[1][r]));
        }
      }
    }
  }
  __syncwarp();
  for (int idx = lane; idx < 16 * DVT; idx += 32) {
    const int r = 16 * warp + idx / DVT, c = idx % DVT;
    if (r < dk && c0 + c < dv) sg[(size_t)r * dv + c] = S[r * DVT + 4 * word(r, c >> 2) + (c & 3)];
  }
}

// ---- the read-out: o = (c q) S0 + B u for 64 tokens and 64 columns, 8 x 4 a thread
constexpr int DC_READ_THREADS = 128, DC_KT = 32;

__global__ void __launch_bounds__(DC_READ_THREADS, 4) delta_chunk_read_kernel(const DeltaParams p, int nseq) {
  pdl_launch();
  pdl_wait();
  __shared__ __align__(16) float As[2][DC_KT][DC_T], Bs[2][DC_KT][64];
  const int at = blockIdx.x / p.H, h = blockIdx.x - at * p.H, c0 = blockIdx.y * 64;
  int first, n;
  if (!dc_find(p.qsl, nseq, at, first, n)) return;
  const int dv = p.dv, tid = threadIdx.x;
  {  // a sequence without a slot has no read-out
    int b = 0, hi = nseq - 1;
    while (b < hi) {
      const int mid = (b + hi + 1) >> 1;
      if (dc_base(p.qsl[mid], mid) <= at) b = mid; else hi = mid - 1;
    }
    if (p.state_slots[b] < 0) return;
  }
  const float* const rec = p.chunks + ((size_t)at * p.H + h) * dc_record(dv);
  // tiles 0 .. 3: 32 rows of (c q)^T and of S0; 4 and 5: 32 rows of B^T and of u
  const int tiles = n > 32 ? 6 : 5;
  auto load = [&](int t) {
    if (t < tiles) {
      const float* a = t < 4 ? rec + DC_QT + t * DC_KT * DC_T : rec + DC_BT + (t - 4) * DC_KT * DC_T;
      const float* s = rec + DC_U + (size_t)(t < 4 ? DC_T + t * DC_KT : (t - 4) * DC_KT) * dv + c0;
      float* da = &As[t & 1][0][0];
      float* db = &Bs[t & 1][0][0];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int idx = tid + 128 * i, k = idx >> 4, q = idx & 15;
        cp_async16(da + 4 * idx, a + 4 * idx);
        if (c0 + 4 * q < dv)
          cp_async16(db + 4 * idx, s + (size_t)k * dv + 4 * q);
        else
          *reinterpret_cast<float4*>(db + 4 * idx) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int tg = tid & 7, cg = tid >> 3;
  uint64_t acc[4][4], sum[4][4];  // pairs of tokens 4 tg, 4 tg + 2, 32 + 4 tg, 32 + 4 tg + 2; columns 4 cg ..
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) sum[i][j] = 0ull;
  load(0);
#pragma unroll 1
  for (int t = 0; t < tiles; ++t) {
    load(t + 1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    const float(*const a)[DC_T] = As[t & 1];
    const float(*const s)[64] = Bs[t & 1];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
    auto half = [&](int hf, int k) {  // one row into the four tokens of a half
      const ulonglong2 w = dc_pairs(&a[k][32 * hf + 4 * tg]);
      const float4 s4 = *reinterpret_cast<const float4*>(&s[k][4 * cg]);
      const uint64_t x[4] = {dc_both(s4.x), dc_both(s4.y), dc_both(s4.z), dc_both(s4.w)};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[2 * hf][j] = dg_fma(w.x, x[j], acc[2 * hf][j]);
        acc[2 * hf + 1][j] = dg_fma(w.y, x[j], acc[2 * hf + 1][j]);
      }
    };
    auto triangle = [&](int hf) {  // rows up to each token's own; nothing of a later token is touched
#pragma unroll 4
      for (int k = 0; k < 4 * tg; ++k) half(hf, k);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int k = 4 * tg + e;
        const float4 w = *reinterpret_cast<const float4*>(&a[k][32 * hf + 4 * tg]);
        const float4 s4 = *reinterpret_cast<const float4*>(&s[k][4 * cg]);
        const float x[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float y0, y1, y2, y3;
          dc_split(acc[2 * hf][j], y0, y1);
          dc_split(acc[2 * hf + 1][j], y2, y3);
          if (e <= 0) y0 = fmaf(w.x, x[j], y0);
          if (e <= 1) y1 = fmaf(w.y, x[j], y1);
          if (e <= 2) y2 = fmaf(w.z, x[j], y2);
          y3 = fmaf(w.w, x[j], y3);
          acc[2 * hf][j] = dg_pack(y0, y1);
          acc[2 * hf + 1][j] = dg_pack(y2, y3);
        }
      }
    };
    if (t < 4) {
#pragma unroll 1
      for (int k8 = 0; k8 < DC_KT; k8 += 8) {
        uint64_t part[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) part[i][j] = 0ull;
#pragma unroll
      for (int k = k8; k < k8 + 8; ++k) {
        const ulonglong2 w0 = dc_pairs(&a[k][4 * tg]), w1 = dc_pairs(&a[k][32 + 4 * tg]);
        const float4 s4 = *reinterpret_cast<const float4*>(&s[k][4 * cg]);
        const uint64_t x[4] = {dc_both(s4.x), dc_both(s4.y), dc_both(s4.z), dc_both(s4.w)};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          part[0][j] = dg_fma(w0.x, x[j], part[0][j]);
          part[1][j] = dg_fma(w0.y, x[j], part[1][j]);
          part[2][j] = dg_fma(w1.x, x[j], part[2][j]);
          part[3][j] = dg_fma(w1.y, x[j], part[3][j]);
        }
      }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = dc_add(part[i][j], acc[i][j]);
      }
    } else if (t == 4) {
      triangle(0);
      if (tiles == 6)
#pragma unroll 8
        for (int k = 0; k < DC_KT; ++k) half(1, k);
    } else {
      triangle(1);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) sum[i][j] = dc_add(acc[i][j], sum[i][j]);
    __syncthreads();
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (c0 + 4 * cg >= dv) return;
  float* const og = p.out + (size_t)first * p.out_stride + (size_t)h * dv + c0 + 4 * cg;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = 32 * (i >> 1) + 4 * tg + 2 * (i & 1);
    float lo[4], hi[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) dc_split(sum[i][j], lo[j], hi[j]);
    if (t < n) *reinterpret_cast<float4*>(og + (size_t)t * p.out_stride) = make_float4(lo[0], lo[1], lo[2], lo[3]);
    if (t + 1 < n) *reinterpret_cast<float4*>(og + (size_t)(t + 1) * p.out_stride) = make_float4(hi[0], hi[1], hi[2], hi[3]);
  }
}

template <int DVT>
int launch_delta_chain(const DeltaParams& p, int B, cudaStream_t st) {
  const dim3 grid((p.dv + DVT - 1) / DVT, B, p.H);
  const size_t smem = dc_chain_smem<DVT>();
  const cudaError_t e = cudaFuncSetAttribute(delta_chunk_chain_kernel<DVT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  return launch(delta_chunk_chain_kernel<DVT>, grid, dim3(DC_THREADS), smem, st, p);
}

// dv, the read-out's rows and the records' buffer are multiples of four floats (checked by the caller).
template <bool CHANNEL>
int dispatch_delta_chunks(const DeltaParams& p, int B, cudaStream_t st) {
  const long long ctas = ((long long)p.N / DC_T + B) * p.H;
  if ((unsigned)B > 65535u || ctas > 0x7fffffffll || (p.dv + 63) / 64 > 65535) return (int)cudaErrorInvalidValue;
  const cudaError_t e = cudaFuncSetAttribute(delta_chunk_prepare_kernel<CHANNEL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DC_PREPARE_SMEM);
  if (e != cudaSuccess) return (int)e;
  int rc = launch(delta_chunk_prepare_kernel<CHANNEL>, dim3((unsigned)ctas), dim3(DC_THREADS), DC_PREPARE_SMEM, st, p, B);
  if (rc) return rc;
  rc = (long long)B * p.H * ((p.dv + 15) / 16) <= 148 ? launch_delta_chain<16>(p, B, st) : launch_delta_chain<32>(p, B, st);
  if (rc) return rc;
  return launch(delta_chunk_read_kernel, dim3((unsigned)ctas, (p.dv + 63) / 64), dim3(DC_READ_THREADS), 0, st, p, B);
}

}  // namespace
