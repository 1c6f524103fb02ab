// The state space of state_space.cu over many tokens of a sequence, 128 tokens a link of the chain, on the tcgen05 tensor cores;
// bfloat16 storage.  In the notation of decay_chunks.cuh (g_t the sum of the decays' logarithms up to token t of the chunk, d_t the step
// size), with the state as S [N][dv]:
//
//   o_t = e^(g_t) C_t S + sum_(s <= t) (C_t . B_s) e^(g_t - g_s) d_s x_s
//   S  <- e^(g_n) S + sum_s B_s (e^(g_n - g_s) d_s x_s)^T
//
// Every product of the second kernel has one operand that is a bfloat16 number as it is stored (B, C, x); the other (the state, the
// scores with their decays, the scaled x) is a float that goes in as three bfloat16 terms, whose sum is that float exactly.  Products of
// bfloat16 numbers are exact in float, so these are float products; sums in tensor memory are cut, not rounded, so no accumulator takes
// more than 64 terms of a sum (32 of the update's; its low terms first) and the parts are added in float.
//
//   scores : C_t . B_s of every chunk, once for the heads that share B and C, on the FP32 pipes, sixteen numbers at a time, what they
//            give added in double: a sum of 128 in one accumulator in tensor memory is off by 1.2e-7 to 1.7e-7 of its norm.
//   chunks : a CTA owns (sequence, head, 64 columns) and goes through the sequence's chunks.  Warps 0 .. 15 do what is between the
//            products: row r of the chunk (or of the state, which stays in registers) and a quarter of the columns a thread; a warp
//            issues the products; one brings the next chunk in and makes its exponentials.  Per chunk: the update, C S, the weights times
//            x, all with M = 128 and N = 64, 24 products each (of 55 cycles: 2.1 us a chunk).
//
// 64 heads of 128 x 64, one sequence of 2,048 tokens: 115 us with the two kernels before it, against 327 of the FP32 form (decay_chunks.cuh)
// and 516 of the walk; 96 heads 117 and 751; 8 sequences of 128 61 and 150.  A chunk takes 6.6 us, a chain of update, split of the state, C
// S, weights times x and read-out; the products alone are 2.3.
// Against 64 bits, in 1e-7 of the norm, this form / the FP32 form / the walk, averages over 16 heads and six seeds, x, B and C behind silu:
//   a_log about  0 : outputs 0.66 / 0.99 / 0.78, states 0.65 / 0.65 / 0.66      -2 : 0.67 / 0.90 / 1.26, 0.75 / 0.85 / 1.35
//                1 : outputs 0.63 / 0.97 / 0.73, states 0.56 / 0.57 / 0.58      -6 : 0.57 / 0.85 / 16.5, 0.59 / 0.94 / 22.2
// and as much nearer for normal ones (0: 0.69 / 1.04 / 1.00, 0.65 / 0.66 / 0.67).  With all of x, B and C positive and decays that leave
// only the last tokens (0 and 1) the state is further off, 0.64 / 0.56 / 0.61 and 0.61 / 0.53 / 0.55: there the tensor core cuts every
// term of a sum downwards.  It takes the sums of the scores in double (with floats 0.11 more for outputs at 0), 2^x to a unit in the last
// place (0.06), sums of 32 tokens for the update, and the three factors below.
//
// Between blocks of 32 tokens a decay is the product of the decays to and from a block's start; inside one it is the exponential of a
// difference of sums of two floats each (every exponent is at most zero).
#pragma once
#include "decay_walk.cuh"
#include "tcgen05.cuh"

namespace kvf {
namespace ssm {

using namespace kvf::tc;

constexpr int TOKENS = 128, N_MAX = 128, DV = 64;  // tokens a chunk, rows of a state, columns a CTA
constexpr int MMA_WARP = 16, LOADER_WARP = 17, THREADS = 576;
constexpr uint32_t HALF = TOKENS * 128;            // bytes of a [128][64] tile
constexpr uint32_t STAGE = 5 * HALF;          // C (two halves), B (two halves), x
constexpr uint32_t COL_P = 0, COL_R = 192, COL_U = 320, COL_L = 448;  // weights, C S, the update and then the weights times x, low terms of C S and of the update
// Tensor memory cuts what does not fit a float towards zero.  So much of a sum is given back, through its low terms: what C S (sums of four
// products), the update (of two) and the weights times x (of four, whose low and high terms share a sum) lose on the average of x, B
// and C of either sign and behind silu, a_log from -6 to 1.  With nothing given back to the update the state at 0 behind silu is off
// by 0.68, with six fifths of its share by 0.67; with a third less of the weights' share outputs are up to 0.07 further off, with a
// third more between 0.03 nearer and 0.03 further.  A sum whose terms are all positive loses up to 1.04e-7 of itself, others 0.65e-7.
constexpr float CUT = 0x1.4p-25f, CUT_U = 0x1.4p-25f, CUT_P = 0x1.8p-25f;
// what a chunk's logarithms become
struct Factors {
  float gh[TOKENS], gl[TOKENS];               // g_t in log2 units, as a float and the rest
  float d[TOKENS], eg[TOKENS], al[TOKENS];  // step, e^(g_t), e^(g_t - r) with r the sum at the start of t's block
  float wd[TOKENS], wr[TOKENS];      // e^(g_n - g_s) d_s and what it is rounded by
  float bd[3][96];                  // e^(r of block I + 1 - g_s) d_s for the tokens before that block
  float keep, pad[3];               // e^(g_n)
};
constexpr size_t SMEM = 2 * (size_t)STAGE + 3 * (size_t)HALF + 2 * sizeof(Factors) + 160;

struct Params {
  const bf16* x;  // rows of x [H*dv] | B [G*N] | C [G*N]
  long long ldx;
  const float* log_decay;  // [tokens][H]
  const float* step;       // [tokens][H]
  const float* raw;        // [tokens s][G][128 t]: C_t . B_s for the tokens t >= s of s's chunk
  float* state;
  long long state_stride;
  float* out;
  long long out_stride;
  const int* qsl;
  const int* state_slots;
  int* err;
  int H, G, ns, dv;
  int use_tma;  // whole chunks come as tensor-map boxes of [128 tokens][64]: 128 rows a state, columns a multiple of 64
};

// A x B with A either K-major or (bit 15) M-major, B K-major or (bit 16) N-major
constexpr uint32_t ID_OUT = idesc(DV, 1), ID_UPDATE = idesc(DV, 1) | (1u << 15);

// A whole warp waits (every lane sees the phase over itself: a shuffle of one lane's wait would hand on the answer, but not the order
// of what was written before it), or arrives once.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, int* err) {
  return __all_sync(0xffffffffu, bar_wait(bar, parity, err));
}
__device__ __forceinline__ void warp_arrive(uint32_t bar) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) bar_arrive(bar);
}
// Two floats' next bfloat16 term; what is left of them stays, and `more` times the term with it.
__device__ __forceinline__ uint32_t take(float& a, float& b, float more = 0.f) {
  const uint32_t w = pk(a, b);
  const uint64_t t = pack2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
  uint64_t rest = fma2(t, pack2(-1.f, -1.f), pack2(a, b));
  if (more != 0.f) rest = fma2(t, pack2(more, more), rest);
  unpack2(rest, a, b);
  return w;
}
// N floats as three bfloat16 terms, in pairs.  An infinity is its first term, with nothing left of it.  more(j): what number j has
// beyond its float.
template <int N, typename Put, typename More>
__device__ __forceinline__ void put_terms(float (&v)[N], float share, Put put, More more) {  // (`share` of the first term on top)
  uint32_t w[N / 2];
#pragma unroll
  for (int j = 0; j < N / 2; ++j) w[j] = take(v[2 * j], v[2 * j + 1], share);
  put(0, w);
  float odd = 0.f;  // no number if some rest is none
#pragma unroll
  for (int j = 0; j < N; ++j) {
    v[j] += more(j);
    odd += v[j];
  }
  if (odd != odd) {
#pragma unroll
    for (int j = 0; j < N; ++j) v[j] = v[j] == v[j] ? v[j] : 0.f;
  }
#pragma unroll
  for (int j = 0; j < N / 2; ++j) w[j] = take(v[2 * j], v[2 * j + 1]);
  put(1, w);
#pragma unroll
  for (int j = 0; j < N / 2; ++j) w[j] = pk(v[2 * j], v[2 * j + 1]);
  put(2, w);
}
// 2^(hi + lo) of two numbers of at most zero (|lo| far below one), to 0.6 units in the last place: 2^f over [-1/2, 1/2] is one and f times a
// polynomial of degree five through the Chebyshev points.  (With ex2.approx of the rounded hi + lo the outputs are off by a tenth more.)
__device__ __forceinline__ void exp2_pair(uint64_t hi, uint64_t lo, float& a, float& b) {
  constexpr float ROUND = 12582912.f;  // 1.5 x 2^23: the sum's last bits are the nearest whole number
  const uint64_t minus = pack2(-1.f, -1.f), t = add2(hi, pack2(ROUND, ROUND)), n = add2(t, pack2(-ROUND, -ROUND));
  const uint64_t f = add2(fma2(n, minus, hi), lo);
  uint64_t q = pack2(0x1.44400400p-13f, 0x1.44400400p-13f);
  q = fma2(q, f, pack2(0x1.5f089600p-10f, 0x1.5f089600p-10f));
  q = fma2(q, f, pack2(0x1.3b2a1c00p-7f, 0x1.3b2a1c00p-7f));
  q = fma2(q, f, pack2(0x1.c6af6c00p-5f, 0x1.c6af6c00p-5f));
  q = fma2(q, f, pack2(0x1.ebfbe000p-3f, 0x1.ebfbe000p-3f));
  q = fma2(q, f, pack2(0x1.62e43000p-1f, 0x1.62e43000p-1f));
  q = fma2(q, f, pack2(1.f, 1.f));
  float x0, x1, t0, t1;
  unpack2(q, a, b);
  unpack2(t, t0, t1);
  unpack2(hi, x0, x1);
  a = x0 < -126.f ? 0.f : a * __uint_as_float((__float_as_uint(t0) << 23) + 0x3f800000u);
  b = x1 < -126.f ? 0.f : b * __uint_as_float((__float_as_uint(t1) << 23) + 0x3f800000u);
}
__device__ __forceinline__ void put4(uint32_t at, const uint32_t* w) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
}
__device__ __forceinline__ void ld16(uint32_t at, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                 "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(at)
               : "memory");
}
// (naming the registers keeps the compiler from using them before the wait)
__device__ __forceinline__ void wait16(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                 "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :
               : "memory");
}
__device__ __forceinline__ void st16(uint32_t at, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(at),
               "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
               "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
               : "memory");
}

// The chunk of 128 tokens of a record, of which a sequence has at most floor(rows / 128) + 1; false for one that nothing uses.
__device__ __forceinline__ bool find_chunk(const int* qsl, int B, int at, int& first, int& n) {
  int b = 0, hi = B - 1;  // the last sequence whose records begin at or before it
  while (b < hi) {
    const int mid = (b + hi + 1) >> 1;
    if (qsl[mid] / TOKENS + mid <= at) b = mid; else hi = mid - 1;
  }
  const int t0 = (at - (qsl[b] / TOKENS + b)) * TOKENS;
  first = qsl[b] + t0;
  n = min(TOKENS, qsl[b + 1] - first);
  return t0 >= 0 && n > 0;
}

// raw[s][t] for 64 x 64 pairs of a chunk and group; blockIdx.y: tokens (s, t) from (0, 0), (0, 64), (64, 64) on.
static __global__ void __launch_bounds__(256) scores_kernel(const bf16* __restrict__ x, long long ldx, long long b_off, long long c_off,
                                                            const int* __restrict__ qsl, int B, int G, int ns, float* __restrict__ raw) {
  pdl_launch();
  pdl_wait();
  extern __shared__ __align__(16) float sm[];
  constexpr int LD = N_MAX + 4;
  int first, n;
  if (!find_chunk(qsl, B, blockIdx.x, first, n)) return;
  const int s0 = blockIdx.y == 2 ? 64 : 0, t0 = blockIdx.y == 0 ? 0 : 64, grp = blockIdx.z;
  if (s0 >= n || t0 >= n) return;
  float* const Bs = sm;
  float* const Cs = sm + 64 * LD;
  const int per = ns >> 3;
  for (int i = threadIdx.x; i < 64 * per; i += 256) {
    const int t = i / per, q = i - t * per;
    float f[8];
    auto put = [&](float* dst, int row, long long off) {
      const uint4 u = row < n ? *reinterpret_cast<const uint4*>(x + (long long)(first + row) * ldx + off + (long long)grp * ns + 8 * q) : make_uint4(0u, 0u, 0u, 0u);
      bf16x8_to_float(u, f);
      *reinterpret_cast<float4*>(dst + t * LD + 8 * q) = make_float4(f[0], f[1], f[2], f[3]);
      *reinterpret_cast<float4*>(dst + t * LD + 8 * q + 4) = make_float4(f[4], f[5], f[6], f[7]);
    };
    put(Bs, s0 + t, b_off);
    put(Cs, t0 + t, c_off);
  }
  __syncthreads();
  const int tg = threadIdx.x & 15, sg = threadIdx.x >> 4;  // rows tg + 16 i of C, sg + 16 j of B
  double sum[4][4] = {};
  for (int k0 = 0; k0 < ns; k0 += 16) {  // eight terms an accumulator: even and odd numbers of sixteen
    uint64_t acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
#pragma unroll
    for (int k = 0; k < 16; k += 4) {
      if (k0 + k >= ns) break;
      ulonglong2 c[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        c[i] = *reinterpret_cast<const ulonglong2*>(Cs + (tg + 16 * i) * LD + k0 + k);
        b[i] = *reinterpret_cast<const ulonglong2*>(Bs + (sg + 16 * i) * LD + k0 + k);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fma2(c[i].y, b[j].y, fma2(c[i].x, b[j].x, acc[i][j]));
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float lo, hi;
        unpack2(acc[i][j], lo, hi);
        sum[i][j] += (double)lo + (double)hi;
      }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int s = s0 + sg + 16 * j;
    if (s >= n) continue;
    float* const dst = raw + ((size_t)(first + s) * G + grp) * TOKENS + t0 + tg;
#pragma unroll
    for (int i = 0; i < 4; ++i) dst[16 * i] = (float)sum[i][j];
  }
}

static __global__ void __launch_bounds__(THREADS, 1) chunks_kernel(const __grid_constant__ CUtensorMap map, const Params p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const uint32_t base = sm32(smem_raw);
  const uint32_t terms = base + 2 * STAGE;  // three tiles: of the scaled x, then of the state
  Factors* const factors = reinterpret_cast<Factors*>(smem_raw + 2 * STAGE + 3 * HALF);
  const uint32_t bars = terms + 3 * HALF + 2 * (uint32_t)sizeof(Factors);
  const uint32_t full0 = bars, empty0 = bars + 16, read_done = bars + 40, update_done = bars + 48, out_done = bars + 56,
                 x_ready = bars + 64, p_ready = bars + 72, s_ready = bars + 80, r_free = bars + 88, drained = bars + 96, tmem_slot = bars + 104;
  // a bit for every token of a chunk (of even and odd chunks) whose x is an infinity or no number in some of the CTA's columns
  uint32_t* const odd_x = reinterpret_cast<uint32_t*>(smem_raw + (bars - base) + 112);
  pdl_launch();
  pdl_wait();
  const int b = blockIdx.z, h = blockIdx.y, c0 = blockIdx.x * DV;
  const int q_begin = p.qsl[b], q_len = p.qsl[b + 1] - q_begin, slot = p.state_slots[b];
  if (q_len <= 0 || slot < 0) return;
  if (base & 1023u) {  // as declared, else refuse rather than compute garbage
    if (threadIdx.x == 0 && p.err) atomicOr(p.err, 8);
    return;
  }
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int chunks = (q_len + TOKENS - 1) / TOKENS;
  if (tid == 0) {
    for (int i = 0; i < 8; ++i) odd_x[i] = 0u;
    for (int s = 0; s < 2; ++s) {
      bar_init(full0 + 8 * s, 1);
      bar_init(empty0 + 8 * s, 1 + MMA_WARP);
    }
    for (uint32_t bar : {read_done, update_done, out_done, drained}) bar_init(bar, 1);
    for (uint32_t bar : {x_ready, p_ready, s_ready, r_free}) bar_init(bar, MMA_WARP);  // the warps that work
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - base));

  if (warp >= LOADER_WARP) {
    // ---- loader: C, B and x of a chunk, and its factors
    const int gn = p.G * p.ns, grp = h / (p.H / p.G);
    const bf16* const rows = p.x + (size_t)q_begin * p.ldx;
    const long long xo = (long long)h * p.dv + c0, bo = (long long)p.H * p.dv + (long long)grp * p.ns, co = bo + gn;
    auto tile = [&](uint32_t dst, long long col, int width, int blocks, int t0, int n) {  // [128 tokens][64 blocks] of `width` numbers
      const int per = 8 * blocks;  // 16-byte words a row, a power of two
      const int c = lane & (per - 1);
      for (int t = lane / per; t < TOKENS; t += 32 / per) {
        const bool in = t < n && 8 * c < width;
        cpa16(dst + (uint32_t)(c >> 3) * HALF + sw128(t, c & 7), rows + (in ? (long long)(t0 + t) * p.ldx + col + 8 * c : 0), in);
      }
    };
    bool ok = true;
    int last = -1;
    float next_l[4], next_d[4];
    auto ask = [&](int c) {
      const int t0 = c * TOKENS, n = min(TOKENS, q_len - t0);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int t = 4 * lane + e;
        const size_t row = (size_t)(q_begin + t0 + min(t, n - 1)) * p.H + h;
        const float l = p.log_decay[row], d = p.step[row];
        next_l[e] = t < n ? l : 0.f;
        next_d[e] = t < n ? d : 0.f;
      }
    };
    ask(0);
    for (int c = 0; c < chunks && ok; ++c) {
      const int s = c & 1, t0 = c * TOKENS, n = min(TOKENS, q_len - t0);
      // ---- the factors, tokens 4 lane .. + 3: made before the stage is free, from numbers asked for a chunk ago
      double g[4], r[4];  // the sums up to each token; at the start of blocks 0 .. 3
      float d[4], w[4], al[4], eg[4], bd[3][4];
      double sum = 0.0;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        d[e] = next_d[e];
        sum += (double)next_l[e];
        g[e] = sum;
      }
      if (c + 1 < chunks) ask(c + 1);
      double incl = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
      }
      double before = __shfl_up_sync(0xffffffffu, incl, 1);
      if (lane == 0) before = 0.0;
      r[0] = 0.0;
      r[1] = __shfl_sync(0xffffffffu, incl, 7);
      r[2] = __shfl_sync(0xffffffffu, incl, 15);
      r[3] = __shfl_sync(0xffffffffu, incl, 23);
      const double total = __shfl_sync(0xffffffffu, incl, 31);
      const int blk = lane >> 3;
      const double start = blk == 0 ? r[0] : blk == 1 ? r[1] : blk == 2 ? r[2] : r[3];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        g[e] += before;
        eg[e] = expf((float)g[e]);
        w[e] = expf((float)(total - g[e]));
        al[e] = expf((float)(g[e] - start));
#pragma unroll
        for (int I = 1; I < 4; ++I) bd[I - 1][e] = expf((float)fmin(0.0, r[I] - g[e])) * d[e];  // (of the tokens before block I)
      }
      if (c >= 2) ok = warp_wait(empty0 + 8 * s, ((c >> 1) - 1) & 1, p.err);
      if (!ok) break;
      const uint32_t at = base + s * STAGE, bar = full0 + 8 * s;
      const bool boxes = p.use_tma && n == TOKENS;
      if (boxes) {
        if (lane == 0) bar_more_tx(bar, STAGE);
        __syncwarp();
        if (lane < 5) tma_load_2d(at + lane * HALF, &map, (int)(lane < 2 ? co + 64 * lane : lane < 4 ? bo + 64 * (lane - 2) : xo), q_begin + t0, bar);
      } else {
        tile(at, co, p.ns, 2, t0, n);
        tile(at + 2 * HALF, bo, p.ns, 2, t0, n);
        tile(at + 4 * HALF, xo, min(DV, p.dv - c0), 1, t0, n);
        cpa_commit();
      }
      Factors& f = factors[s];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int t = 4 * lane + e;
        const double g2 = g[e] * 1.4426950408889634;
        f.gh[t] = (float)g2;
        f.gl[t] = (float)(g2 - (double)(float)g2);
        f.d[t] = d[e];
        f.eg[t] = eg[e];
        f.wd[t] = w[e] * d[e];
        f.wr[t] = fmaf(w[e], d[e], -w[e] * d[e]);
        f.al[t] = al[e];
#pragma unroll
        for (int I = 1; I < 4; ++I)
          if (blk < I) f.bd[I - 1][t] = bd[I - 1][e];
      }
      if (lane == 0) f.keep = expf((float)total);
      cpa_wait<0>();
      fence_async_smem();
      __syncwarp();
      if (lane == 0) bar_arrive(bar);
      last = c;
    }
    // no copy outlives the CTA, whatever made the others leave
    if (last >= 0) bar_wait(full0 + 8 * (last & 1), (last >> 1) & 1, p.err);
    if (last >= 1) bar_wait(full0 + 8 * ((last - 1) & 1), ((last - 1) >> 1) & 1, p.err);
  } else if (warp == MMA_WARP) {
    if (elect_one()) {
      bool ok = true;
      const uint32_t k16 = (16 * 128) >> 4;  // 16 rows of a tile whose rows are walked
      const uint64_t td = sdesc(terms);
      for (int c = 0; c < chunks && ok; ++c) {
        const uint32_t ph = c & 1;
        const uint32_t at = base + ph * STAGE;
        const uint64_t cd = sdesc(at), bt = sdesc_mn(at + 2 * HALF, HALF), xd = sdesc(at + 4 * HALF);
        ok = bar_wait(full0 + 8 * ph, (c >> 1) & 1, p.err);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // the update, from the scaled x
        ok = bar_wait(x_ready, ph, p.err) && (c == 0 || bar_wait(r_free, ph ^ 1, p.err));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int i = 0; i < 24; ++i) {  // (one sum after another: products that take turns at two sums wait for one another)
          const int kk = i & 7, term = 2 - (i >> 3);
          umma(tmem + (term ? COL_L : (kk < 4 ? COL_U : COL_R) + DV * ((kk >> 1) & 1)), bt + kk * k16, td + ((term * HALF) >> 4) + kk * k16, ID_UPDATE,
               term ? i > 0 : (kk & 1) != 0);
        }
        umma_commit(update_done);
        // C S: the state's terms take the place of the scaled x's
        ok = bar_wait(s_ready, ph, p.err);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int i = 0; i < 24; ++i) {
          const int kk = i & 7, term = 2 - (i >> 3);
          umma(tmem + (term ? COL_L : COL_R + DV * (kk >> 2)), cd + (((kk >> 2) * HALF) >> 4) + 2 * (kk & 3), td + ((term * HALF) >> 4) + kk * k16, ID_OUT,
               term ? i > 0 : (kk & 3) != 0);
        }
        umma_commit(read_done);
        // the weights times x, where the update was
        ok = bar_wait(p_ready, ph, p.err);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int g = 0; g < 2; ++g)
#pragma unroll
          for (int term = 2; term >= 0; --term)
#pragma unroll
            for (int kk = 4 * g; kk < 4 * g + 4; ++kk)
              umma_ts(tmem + COL_U + DV * g, tmem + COL_P + 64 * term + 8 * kk, xd + kk * k16, ID_OUT, term < 2 || kk > 4 * g);
        umma_commit(out_done);
        umma_commit(empty0 + 8 * ph);
      }
      if (!ok) {  // no product outlives the tensor memory
        umma_commit(drained);
        bar_wait(drained, 0, p.err);
      }
    }
  } else {
    const int q4 = warp >> 2, blk = warp & 3, r = tid & 127;  // columns 16 q4 .. + 15 and the scores of block q4's tokens of row r
    const uint32_t mine = tmem + ((uint32_t)(blk * 32) << 16);
    float S[16];
    float* const sg = p.state + (size_t)slot * p.state_stride + ((size_t)h * p.ns + r) * p.dv + c0 + 16 * q4;
    const int left = r < p.ns ? min(16, p.dv - c0 - 16 * q4) : 0;  // columns that there are, a multiple of eight
#pragma unroll
    for (int j = 0; j < 16; j += 4) {
      const float4 v = j < left ? *reinterpret_cast<const float4*>(sg + j) : make_float4(0.f, 0.f, 0.f, 0.f);
      S[j] = v.x; S[j + 1] = v.y; S[j + 2] = v.z; S[j + 3] = v.w;
    }
    float* const og = p.out + (size_t)q_begin * p.out_stride + (size_t)h * p.dv + c0;
    const float* const raw = p.raw + ((size_t)q_begin * p.G + h / (p.H / p.G)) * TOKENS + r;
    auto put_row = [&](float (&v)[16], auto more) {  // the thread's 16 numbers of row r, in three tiles
      put_terms(v, 0.f, [&](int term, const uint32_t(&w)[8]) {
        put4(terms + term * HALF + sw128(r, 2 * q4), w);
        put4(terms + term * HALF + sw128(r, 2 * q4 + 1), w + 4);
      }, more);
      fence_async_smem();
    };
    // The scaled x of a chunk, for the update; its place is free once the chunk before's C S, which read the state there, is over.
    // What is infinite or no number is taken out of x itself: the weights of later tokens are zeros, and zero times it would reach the
    // tokens before it.  The read-out adds it to its own token and those after.
    auto scale_x = [&](int c) {
      const int s = c & 1;
      if (!warp_wait(full0 + 8 * s, (c >> 1) & 1, p.err)) return false;
      float x[16], v[16];
      const float w = factors[s].wd[r], rest = factors[s].wr[r];
      unsigned char* const row = smem_raw + s * STAGE + 4 * HALF;
      bf16x8_to_float(*reinterpret_cast<const uint4*>(row + sw128(r, 2 * q4)), x);
      bf16x8_to_float(*reinterpret_cast<const uint4*>(row + sw128(r, 2 * q4 + 1)), x + 8);
      float odd = 0.f;
#pragma unroll
      for (int j = 0; j < 16; ++j) odd = fmaf(x[j], 0.f, odd);
      if (odd != odd) {
        atomicOr(odd_x + 4 * s + (r >> 5), 1u << (r & 31));
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (x[j] * 0.f != 0.f) *reinterpret_cast<unsigned short*>(row + sw128(r, 2 * q4 + (j >> 3)) + 2 * (j & 7)) = 0;
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = x[j] * w;
      put_row(v, [&](int j) { return fmaf(x[j], rest, fmaf(x[j], w, -x[j] * w)); });
      warp_arrive(x_ready);
      return true;
    };
    // A sum is two sums of high terms (`b`, which is left, of the later tokens) and one of low terms; `part` of the first and the last
    // is given away.
    auto sums = [&](uint32_t col, uint32_t (&b)[16], auto part) {
      uint32_t a[16];
      ld16(mine + COL_L + 16 * q4, b);
      ld16(mine + col + 16 * q4, a);
      wait16(b);
      wait16(a);
#pragma unroll
      for (int j = 0; j < 16; ++j) part(j, __uint_as_float(a[j]) + fmaf(__uint_as_float(a[j]), CUT, __uint_as_float(b[j])));
      ld16(mine + col + DV + 16 * q4, b);
      wait16(b);
    };
    auto with = [](uint32_t b, float part) { return __uint_as_float(b) + fmaf(__uint_as_float(b), CUT, part); };
    auto ask = [&](int c, float (&v)[32]) {  // a chunk's scores
      const int n = min(TOKENS, q_len - c * TOKENS);
      const size_t step = (size_t)p.G * TOKENS;
      const float* const at = raw + (size_t)(c * TOKENS + 32 * q4) * step;
      if (q4 > blk) {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = 0.f;
      } else if (n == TOKENS) {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = at[j * step];
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = 32 * q4 + j < n && r < n ? at[j * step] : 0.f;
      }
    };
    auto weigh = [&](const Factors& f, float (&v)[32]) {
      if (q4 < blk) {
        const float* const bd = f.bd[blk - 1] + 32 * q4;
        const float al = f.al[r];
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          const float4 b4 = *reinterpret_cast<const float4*>(bd + j);
          v[j] *= al * b4.x;
          v[j + 1] *= al * b4.y;
          v[j + 2] *= al * b4.z;
          v[j + 3] *= al * b4.w;
        }
      } else if (q4 == blk) {
        const uint64_t gh = pack2(f.gh[r], f.gh[r]), gl = pack2(f.gl[r], f.gl[r]), minus = pack2(-1.f, -1.f);
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
          const uint64_t h2 = *reinterpret_cast<const uint64_t*>(f.gh + 32 * q4 + j), l2 = *reinterpret_cast<const uint64_t*>(f.gl + 32 * q4 + j);
          const float2 d2 = *reinterpret_cast<const float2*>(f.d + 32 * q4 + j);
          const uint64_t x = fma2(h2, minus, gh);  // what rounding takes from the difference goes to its low part (sums only fall)
          const uint64_t rest = fma2(add2(h2, fma2(gh, minus, x)), minus, fma2(l2, minus, gl));
          float e0, e1;
          exp2_pair(x, rest, e0, e1);
          v[j] = j <= lane ? v[j] * (e0 * d2.x) : 0.f;
          v[j + 1] = j + 1 <= lane ? v[j + 1] * (e1 * d2.y) : 0.f;
        }
      }  // (the others are zeros)
    };
    bool ok = scale_x(0);
    asm volatile("bar.sync 1, %0;" ::"n"(MMA_WARP * 32) : "memory");  // (the odd tokens of the first chunk are known to all)
    int met = 0;  // barriers of all the warps that work, of the chunks' read-outs
    float v[32];
    ask(0, v);
    for (int c = 0; c < chunks && ok; ++c) {
      const uint32_t ph = c & 1;
      const Factors& f = factors[ph];
      // ---- the state's terms for C S, where the scaled x was; S <- e^(g_n) S + the update
      ok = warp_wait(update_done, ph, p.err);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      uint32_t b[16];
      {
        float y[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) y[j] = S[j];
        put_row(y, [](int) { return 0.f; });
        const float keep = f.keep;
        ld16(mine + COL_U + 16 * q4, b);
        wait16(b);
#pragma unroll
        for (int j = 0; j < 16; ++j) y[j] = __uint_as_float(b[j]);
#pragma unroll
        for (uint32_t col : {COL_U + DV, COL_R, COL_R + DV}) {
          ld16(mine + col + 16 * q4, b);
          wait16(b);
#pragma unroll
          for (int j = 0; j < 16; ++j) y[j] += __uint_as_float(b[j]);
        }
        ld16(mine + COL_L + 16 * q4, b);
        wait16(b);
#pragma unroll
        for (int j = 0; j < 16; ++j) S[j] = fmaf(keep, S[j], y[j] + fmaf(y[j], CUT_U, __uint_as_float(b[j])));
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        warp_arrive(s_ready);  // (C S's low terms lie where the update's did)
      }
      // ---- the weights, under C S (the products with those of the chunk before are over)
      weigh(f, v);
      put_terms(v, CUT_P, [&](int term, const uint32_t(&w)[16]) { st16(mine + COL_P + 64 * term + 16 * q4, w); }, [](int) { return 0.f; });
      tmem_wait_st();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      warp_arrive(p_ready);
      // ---- the next chunk's scaled x, under the weights times x
      ok = warp_wait(read_done, ph, p.err);
      if (ok && c + 1 < chunks) ok = scale_x(c + 1);
      // ---- the read-out
      if (ok) ok = warp_wait(out_done, ph, p.err);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      float o[16];
      sums(COL_R, b, [&](int j, float x) { o[j] = x; });
      {
        const float eg = f.eg[r];
#pragma unroll
        for (int j = 0; j < 16; ++j) o[j] = eg * with(b[j], o[j]);
      }
      ld16(mine + COL_U + 16 * q4, b);
      wait16(b);
#pragma unroll
      for (int j = 0; j < 16; ++j) o[j] += __uint_as_float(b[j]);
      ld16(mine + COL_U + DV + 16 * q4, b);
      wait16(b);
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      warp_arrive(r_free);
#pragma unroll
      for (int j = 0; j < 16; ++j) o[j] += __uint_as_float(b[j]);
      const uint4 odd = *reinterpret_cast<const uint4*>(odd_x + 4 * ph);
      if (odd.x | odd.y | odd.z | odd.w) {
#pragma unroll 1
        for (int s = 0; s <= r; ++s) {
          if (!(odd_x[4 * ph + (s >> 5)] >> (s & 31) & 1u)) continue;
          const float wt = raw[(size_t)(c * TOKENS + s) * p.G * TOKENS] * (ex2((f.gh[r] - f.gh[s]) + (f.gl[r] - f.gl[s])) * f.d[s]);
          const bf16* const xs = p.x + (size_t)(q_begin + c * TOKENS + s) * p.ldx + (size_t)h * p.dv + c0 + 16 * q4;
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float x = c0 + 16 * q4 + j < p.dv ? __bfloat162float(xs[j]) : 0.f;
            if (x * 0.f != 0.f) o[j] = fmaf(wt, x, o[j]);
          }
        }
      }
      // By way of B's place, which the update has read: a warp then writes whole rows (straight from the registers a warp's 16 bytes a
      // row go to 32 rows at a time, which kept the path to memory busy for 3,000 cycles).
      unsigned char* const rows = smem_raw + ph * STAGE + 2 * HALF;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        *reinterpret_cast<float4*>(rows + r * 256 + (((4 * q4 + q) ^ (r & 7)) << 4)) = make_float4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
      asm volatile("bar.sync 1, %0;" ::"n"(MMA_WARP * 32) : "memory");
      ++met;
      if (tid < 4) odd_x[4 * ph + tid] = 0u;  // (before the chunk after the next's scaled x, which waits for this warp)
      const int n = min(TOKENS, q_len - c * TOKENS);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = warp * 8 + 2 * i + (lane >> 4), q = lane & 15;
        const float4 y = *reinterpret_cast<const float4*>(rows + t * 256 + ((q ^ (t & 7)) << 4));
        if (t < n && 4 * q < p.dv - c0) *reinterpret_cast<float4*>(og + (size_t)(c * TOKENS + t) * p.out_stride + 4 * q) = y;
      }
      fence_async_smem();  // the next copy into this place comes after
      warp_arrive(empty0 + 8 * ph);
      if (c + 1 < chunks) ask(c + 1, v);
    }
    // a warp whose wait ran out still meets the others at the barriers of the chunks left
    for (; met < chunks; ++met) asm volatile("bar.sync 1, %0;" ::"n"(MMA_WARP * 32) : "memory");
    if (ok) {
#pragma unroll
      for (int j = 0; j < 16; j += 4)
        if (j < left) *reinterpret_cast<float4*>(sg + j) = make_float4(S[j], S[j + 1], S[j + 2], S[j + 3]);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == MMA_WARP) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

// The rows of x as [rows][width] bfloat16 (a row stride of ldx numbers), in boxes of [128][64], 128-byte swizzle.
inline int rows_map(CUtensorMap* map, const void* x, long long ldx, long long width, long long rows) {
  EncodeTiledFn fn = encode_tiled();
  if (!fn) return (int)cudaErrorNotSupported;
  const cuuint64_t dims[2] = {(cuuint64_t)width, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ldx * 2};
  const cuuint32_t box[2] = {64u, (cuuint32_t)TOKENS};
  const cuuint32_t one[2] = {1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(x), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : (int)cudaErrorInvalidValue;
}

}  // namespace ssm
}  // namespace kvf
