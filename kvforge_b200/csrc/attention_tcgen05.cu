// Paged grouped-query attention for many queries (prompts, portions, mixed batches) on the
// tcgen05 tensor cores; bfloat16, head size 64 or 128.  Same contract as attention_generic.cu.
//
// One CTA serves 128 rows of one kv head of one sequence; a row is a (query token, head of the
// group) pair, so 128/g tokens.  Which tokens: an entry (sequence, first query) of a list made
// on the host with the step, longest walk over the keys first; without a list, the grid's y and
// z.  Keys are walked in tiles of 64 from position 0 (or from the tile that holds the window's
// first key).  Per tile t:
//   S = Q K^T      tcgen05.mma 128 x 64 x (head size), Q and the K tile in 128-byte-swizzled shared
//                  memory (K-major; a 128-wide tile as two 64-wide halves), S in tensor memory;
//   softmax        thread r owns row r (tensor-memory lane r): it reads the 64 scores once with
//                  tcgen05.ld, keeps the running maximum and sum in registers, and writes
//                  P = exp2(S * scale - m) as bfloat16 into shared memory in the swizzled K-major
//                  layout of an A operand (packed f32x2 fma and add, a three-input maximum);
//   O += P V       tcgen05.mma 128 x 64 x 64 per 64 output dims, the V tile [keys][64] as an
//                  MN-major B operand; O stays in tensor memory over all tiles.
// Two groups of four softmax warps take the even and the odd tiles, each with its own S buffer,
// P buffer, O accumulator, maximum and sum; at the end group 0 merges the two.
// The maximum m that P is scaled by follows the row's true maximum lazily: a thread raises it
// only when the true maximum has grown by more than 8 (in log2 units), so P <= 256; then the
// warp multiplies its rows of O by exp2(m_old - m_new) in tensor memory (tcgen05.ld / st) before
// the next P V.  The sum l carries the same factor, so O / l is the exact softmax average.
// Whether a thread rescales depends on its own row only: a row's result does not depend on the
// rows beside it.
// Warps 0-7 do the softmax.  Warp 8 brings Q in with cp.async and the K/V tiles as tensor-map
// boxes of a page's keys (16, 32 or 64 rows of 128 bytes; with pages that are no multiple of 16
// keys, and for a last tile that ends inside a page, key by key with cp.async) through a ring of
// 4 stages (5 at head size 128).  One thread of warp 9 issues the MMAs: when P(t) arrives, first
// S(t+2), which is all its group waits for, then P(t) V(t).  Two CTAs fit an SM at head size 64
// (112 KB of shared memory and 256 tensor-memory columns each), one at 128.
//
// Shaped scores (a soft cap, a bias by distance and head, kept first keys under a window; sinks beside them) are a form of their own:
// scores are finished in place before the maximum is taken, kept tiles are walked first, and a group stages the
// biases of its next tile (128 / g + 63 distances a head, in log2 units) in shared memory behind a barrier of its own, so that a
// score's bias is one conflict-free word; one stage of keys makes room for them.  2,048 tokens in two sequences, 32 heads of 64 on 8,
// a window of 1,024, a bias and 64 kept keys: 77 us against 149 us of the mma.sync tile kernel.
//
// Every mbarrier wait is bounded; if one runs out the kernel raises bit 4 of the error flag and
// winds down.  No cluster launch, no multicast.
#include "tcgen05.cuh"

using namespace kvf;
using namespace kvf::tc;

namespace {

// D: head size, 64 or 128.  A [rows][128] tile lies in shared memory as two [rows][64] halves of 128-byte
// swizzled rows; S = Q K^T then walks D/16 k-steps over the halves, and O += P V is one MMA of 64
// output columns per half of V.
constexpr int BM = 128;  // rows per CTA
constexpr int BN = 64;   // keys per tile
constexpr int SOFTMAX_WARPS = 8;                    // two groups of four: even and odd key tiles
constexpr int LOADER_WARP = SOFTMAX_WARPS, MMA_WARP = SOFTMAX_WARPS + 1;
constexpr int THREADS = (SOFTMAX_WARPS + 2) * 32;
// a tile's biases: 128 / g + 63 distances for each of g <= 8 heads, each head's padded to a multiple of 32 words plus 32 / g
constexpr int BIAS_WORDS = 800;
// SH: the form for shaped scores, which gives a stage of keys for two buffers of biases for either softmax group
template <int D, bool SH = false> struct Shape {
  static constexpr int HALVES = D / 64;
  static constexpr int KV_STAGES = (D == 64 ? 4 : 5) - (SH ? 1 : 0);
  // Tiles in flight behind the one being handed over, without boxes.  The place of tile t + LOOKAHEAD is free when P V of tile
  // t + LOOKAHEAD - KV_STAGES is done, which the issuer sends out after it has seen the keys two tiles further: those have to be
  // handed over by then.
  static constexpr int LOOKAHEAD = KV_STAGES >= 4 ? 2 : 1;
  static_assert(LOOKAHEAD - KV_STAGES + 2 <= 0, "the loader would wait for what waits for it");
  static constexpr int CTAS_PER_SM = D == 64 ? 2 : 1;  // 109 or 112 KB and 256 tensor-memory columns, or 204 or 224 KB and 512
  static constexpr uint32_t Q_BYTES = HALVES * 128 * 128;     // [128 rows][D] bfloat16
  static constexpr uint32_t KV_BYTES = HALVES * 64 * 128;     // a [64 keys][D] bfloat16 tile
  static constexpr uint32_t TMEM_COLS = D == 64 ? 256u : 512u;  // S: 2 x 64, O: 2 x D
  static constexpr size_t SMEM_BYTES = (size_t)Q_BYTES + (size_t)KV_STAGES * 2 * KV_BYTES + 2 * 128 * 128 + 256 + (SH ? 4 * BIAS_WORDS * 4 : 0);
};
constexpr uint32_t Q_HALF = BM * 128;        // [128 rows][64] bfloat16
constexpr uint32_t KV_HALF = BN * 128;       // [64 keys][64] bfloat16
constexpr uint32_t P_BYTES = BM * 128;       // [128 rows][64 keys] bfloat16

struct TcAttnParams {
  const bf16* q;
  bf16* out;
  const bf16* kcache;
  const bf16* vcache;
  const int* block_tables;
  const int* qsl;
  const int* ctx_lens;
  const int* work;  // n_work pairs (sequence or -1, first query of the tile), or null: the grid's y and z say which
  int* err;
  int num_seqs;  // a list entry that names a sequence beyond these is a dead tile
  int q_stride, out_stride, bt_stride;
  int nh, nkv, block_size, bs_shift;
  int window;
  float scale_log2;
  int use_tma;     // pages are multiples of 16 keys: K and V tiles come as tensor-map boxes of [box_rows][64]
  int box_rows;    // 16, 32 or 64: the largest of them that divides the page
  int total_rows;  // rows of the cache seen as [rows][64]: a box from this row reads zeros
};
// The form with sinks has its own parameters: the plain form stands at its register budget, and a longer parameter block alone
// makes it spill.
struct TcAttnSinkParams : TcAttnParams {
  const float* sinks;  // [nh] (natural-log units): a number a head whose exponential joins the denominator, without a key or a value
};
// Scores that are more than scaled dot products: a soft cap, a bias by distance and head, first keys that stay visible
// under a window; sinks too.
struct TcAttnShapedParams : TcAttnSinkParams {
  int keep_first;
  const float* bias;  // [nh][bias_far + 1]
  int bias_far;
  float cap_in, cap_out;  // scale / c and c * log2(e)
};
// What a kernel is made for: plain scores, sinks, or SHAPED plus which of a bias (1) and a cap (2) it takes.
enum { PLAIN = 0, SINKS = 1, SHAPED = 4 };
template <int MODE> struct ParamsOf { using type = TcAttnShapedParams; };
template <> struct ParamsOf<PLAIN> { using type = TcAttnParams; };
template <> struct ParamsOf<SINKS> { using type = TcAttnSinkParams; };

// One tile of the softmax for the thread's row.  v: the 64 raw scores (in place: not kept).
// MASK: some key of the tile may be hidden from some row of the warp.  Returns the tile's sum of
// P and stores P (bfloat16) into the row of the A-operand tile at p_row (a shared address of
// the row's first byte; chunk c of the row lies at p_row + ((c ^ (r & 7)) << 4)).
template <bool MASK>
__device__ __forceinline__ float softmax_tile(uint32_t (&va)[32], uint32_t (&vb)[32], float& m_ref, float& corr,
                                              float scale_log2, int first, int last, uint32_t p_row, int r7) {
  // first/last: the tile-local range of visible keys of this row (MASK only)
  float mx = -INFINITY;
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    const float a = (!MASK || (j >= first && j <= last)) ? __uint_as_float(va[j]) : -INFINITY;
    const float b = (!MASK || (j + 32 >= first && j + 32 <= last)) ? __uint_as_float(vb[j]) : -INFINITY;
    mx = fmaxf(mx, fmaxf(a, b));  // (a three-input maximum)
  }
  mx *= scale_log2;  // scale > 0
  corr = 1.f;
  if (mx > m_ref + RESCALE_STEP || (m_ref == -INFINITY && mx > -INFINITY)) {
    corr = ex2(m_ref - mx);  // 0 the first time
    m_ref = mx;
  }
  const float m_use = (m_ref == -INFINITY) ? 0.f : m_ref;
  const uint64_t scale2 = pack2(scale_log2, scale_log2), neg_m2 = pack2(-m_use, -m_use);
  uint64_t sum_a = pack2(0.f, 0.f), sum_b = sum_a;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    uint32_t(&v)[32] = half ? vb : va;
    uint32_t w[16];
#pragma unroll
    for (int j = 0; j < 32; j += 2) {
      const int c = half * 32 + j;
      float x0, x1;
      unpack2(fma2(pack2(__uint_as_float(v[j]), __uint_as_float(v[j + 1])), scale2, neg_m2), x0, x1);
      float e0 = ex2(x0), e1 = ex2(x1);
      if (MASK) {
        if (c < first || c > last) e0 = 0.f;
        if (c + 1 < first || c + 1 > last) e1 = 0.f;
      }
      if (j & 2)
        sum_b = add2(sum_b, pack2(e0, e1));
      else
        sum_a = add2(sum_a, pack2(e0, e1));
      w[j >> 1] = pk(e0, e1);
    }
#pragma unroll
    for (int q4 = 0; q4 < 4; ++q4) {
      const uint32_t dst = p_row + (uint32_t)(((half * 4 + q4) ^ r7) << 4);
      asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(w[4 * q4]), "r"(w[4 * q4 + 1]),
                   "r"(w[4 * q4 + 2]), "r"(w[4 * q4 + 3])
                   : "memory");
    }
  }
  float s0, s1;
  unpack2(add2(sum_a, sum_b), s0, s1);
  return s0 + s1;
}

// tanh(x) = 1 - 2 / (exp(2x) + 1): exact at both ends, absolute error of a few 1e-7 near zero.
__device__ __forceinline__ float fast_tanh(float x) { return 1.f - __fdividef(2.f, ex2(x * 2.8853900817779268f) + 1.f); }

// The same for shaped scores, which are made in place: s * scale, or with CAP c * tanh(s * scale / c), plus with BIAS the bias of
// the distance, `brow[-j]` for the tile's key j (a shared-memory row in log2 units).  Keys before `kept` are seen whatever
// `first` says.
template <bool BIAS, bool CAP>
__device__ __forceinline__ float softmax_shaped(uint32_t (&va)[32], uint32_t (&vb)[32], float& m_ref, float& corr, float scale_log2, float cap_in,
                                                float cap_out, const float* brow, bool mask, int first, int last, int kept, uint32_t p_row, int r7) {
  float mx = -INFINITY;
#pragma unroll
  for (int c = 0; c < 64; ++c) {
    uint32_t& v = c < 32 ? va[c & 31] : vb[c & 31];
    const float s = __uint_as_float(v);
    float x;
    if (CAP)
      x = BIAS ? fmaf(cap_out, fast_tanh(s * cap_in), brow[-c]) : cap_out * fast_tanh(s * cap_in);
    else
      x = BIAS ? fmaf(s, scale_log2, brow[-c]) : s * scale_log2;
    if (mask && (c > last || (c < first && c >= kept))) x = -INFINITY;
    v = __float_as_uint(x);
    mx = fmaxf(mx, x);
  }
  corr = 1.f;
  // The maximum is followed exactly, not in steps of RESCALE_STEP as plain scores do: the largest weight is then one, which no
  // rounding to bfloat16 changes.  Against 64 bits results are off by 0.98 to 1.00 of what they are on the mma.sync kernel, in
  // steps by 1.00 to 1.23, the more so the sharper the weights (2,048 tokens: 74.5 us in steps, 76.7 so).
  if (mx > m_ref) {
    corr = ex2(m_ref - mx);  // 0 the first time
    m_ref = mx;
  }
  const float m_use = (m_ref == -INFINITY) ? 0.f : m_ref;
  float sum_a = 0.f, sum_b = 0.f;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    uint32_t w[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int c = 8 * q + 2 * e;
      const float e0 = ex2(__uint_as_float(c < 32 ? va[c & 31] : vb[c & 31]) - m_use);
      const float e1 = ex2(__uint_as_float(c < 32 ? va[(c & 31) + 1] : vb[(c & 31) + 1]) - m_use);
      sum_a += e0;
      sum_b += e1;
      w[e] = pk(e0, e1);
    }
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(p_row + (uint32_t)((q ^ r7) << 4)), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
  }
  return sum_a + sum_b;
}

template <int D, int MODE>
__global__ void __launch_bounds__(THREADS, Shape<D, (MODE >= SHAPED)>::CTAS_PER_SM)
attn_tcgen05_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const typename ParamsOf<MODE>::type p) {
  constexpr bool SH = MODE >= SHAPED, BIAS = SH && (MODE & 1), CAP = SH && (MODE & 2);
  constexpr int HALVES = Shape<D, SH>::HALVES, KV_STAGES = Shape<D, SH>::KV_STAGES, LOOKAHEAD = Shape<D, SH>::LOOKAHEAD;
  constexpr uint32_t Q_BYTES = Shape<D>::Q_BYTES, KV_BYTES = Shape<D>::KV_BYTES;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // no slack for rounding up (two CTAs have to fit an SM): the base must be 1024-byte aligned
  // as declared, else the kernel refuses (bit 8 of the error flag) rather than compute garbage
  const uint32_t base = sm32(smem_raw);
  const uint32_t q_s = base;                                    // [128 rows][64]
  const uint32_t kv_s = q_s + Q_BYTES;                          // per stage: K [64 keys][64], V [64 keys][64]
  const uint32_t p_s = kv_s + KV_STAGES * 2 * KV_BYTES;         // two [128 rows][64 keys] buffers
  const uint32_t bars = p_s + 2 * P_BYTES;
  const uint32_t q_full = bars, kv_full0 = bars + 8, kv_empty0 = kv_full0 + 8 * KV_STAGES;
  const uint32_t s_full0 = kv_empty0 + 8 * KV_STAGES, p_full0 = s_full0 + 16, pv_done0 = p_full0 + 16;
  const uint32_t tmem_slot = pv_done0 + 16;
  [[maybe_unused]] float* const bias_s = reinterpret_cast<float*>(smem_raw + (p_s + 2 * P_BYTES + 256 - base));  // [group][2][BIAS_WORDS]
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - base));

  pdl_launch();
  if (base & 1023u) {
    if (threadIdx.x == 0 && p.err) atomicOr(p.err, 8);
    pdl_wait();
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // grid (kv heads, sequences, row blocks): CTAs start in the order of their index with x
  // fastest, so all heads of the longest walk start first, then the next longest, ...
  const int kvh = blockIdx.x;
  const int g = p.nh / p.nkv;
  const int tq = BM / g;
  // which tile of queries: from the list (made on the host, longest walk first), else from the grid
  int b = p.work ? p.work[2 * blockIdx.y] : (int)blockIdx.y;
  const int q0 = p.work ? p.work[2 * blockIdx.y + 1] : (int)(gridDim.z - 1 - blockIdx.z) * tq;  // the longest walks first
  if (b >= p.num_seqs) b = -1;  // whatever a list holds, nothing outside the step's arrays is read
  const int q_begin = b >= 0 ? p.qsl[b] : 0, q_len = b >= 0 ? p.qsl[b + 1] - q_begin : 0;
  const int ctx = b >= 0 ? p.ctx_lens[b] : 0;
  const bool live = q_len > 0 && ctx > 0 && q0 >= 0 && q0 < q_len;  // uniform over the CTA
  // A CTA without a tile leaves at once; the grid's first CTA stays for the dependency wait, so
  // the grid does not complete before its predecessor.
  if (!live && (blockIdx.x | blockIdx.y | blockIdx.z) != 0) return;
  const int n_tok = live ? min(tq, q_len - q0) : 0;
  const int p_first = ctx - q_len + q0;
  const int kv_hi = p_first + n_tok;
  const int kv_lo = live ? (first_key(p_first, p.window) / BN) * BN : 0;
  // kept first keys: their tiles come first, then the window's
  int n_kept = 0;
  if constexpr (SH) n_kept = live ? min((p.keep_first + BN - 1) / BN, kv_lo / BN) : 0;
  const int n_tiles = live ? (kv_hi - kv_lo + BN - 1) / BN + n_kept : 0;
  auto first_of = [&](int t) { return SH && t < n_kept ? t * BN : kv_lo + (t - (SH ? n_kept : 0)) * BN; };  // a tile's first key

  if (threadIdx.x == 0) {
    bar_init(q_full, 1);
    for (int s = 0; s < KV_STAGES; ++s) {
      bar_init(kv_full0 + 8 * s, 1);
      bar_init(kv_empty0 + 8 * s, 1);
    }
    for (int s = 0; s < 2; ++s) {
      bar_init(s_full0 + 8 * s, 1);
      bar_init(p_full0 + 8 * s, BM);
      bar_init(pv_done0 + 8 * s, 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(Shape<D>::TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot_ptr;
  // S of even and odd tiles: columns 0..63, 64..127; their O accumulators: 128..191, 192..255
  const uint32_t tmem_s = tmem_base, tmem_o = tmem_base + 2 * BN;

  pdl_wait();

  if (live && warp == LOADER_WARP) {
    // ---- loader: Q, then a K and a V tile per stage; 16-byte chunks into the swizzled layout
    const bf16* qg = p.q + (size_t)(q_begin + q0) * p.q_stride + (size_t)(kvh * g) * D;
    for (int idx = lane; idx < BM * (D / 8); idx += 32) {
      const int r = idx / (D / 8), c = idx % (D / 8);
      const int tok = r / g, hh = r - tok * g;
      const bool valid = tok < n_tok;
      cpa16(q_s + (c >> 3) * Q_HALF + sw128(r, c & 7), qg + (valid ? (size_t)tok * p.q_stride + (size_t)hh * D + c * 8 : 0), valid);
    }
    const int* bt = p.block_tables + (size_t)b * p.bt_stride;
    // A tile's 64 keys sit in up to 64 pages: lane l looks up keys l and l+32 (independent table
    // reads), and the copy loop, in which 8 lanes share a key, gets each key's row from the lane
    // that holds it.
    auto issue_tile = [&](int t) {
      const int s = t % KV_STAGES;
      const uint32_t ks = kv_s + s * 2 * KV_BYTES, vs = ks + KV_BYTES;
      const int t0 = first_of(t);
      long long row[2];  // element offset of the key's row in the cache, or -1
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int kp = t0 + lane + 32 * j;
        int blk = -1, off = 0;
        if (kp < ctx) {
          if (p.bs_shift >= 0) {
            blk = bt[kp >> p.bs_shift];
            off = kp & (p.block_size - 1);
          } else {
            blk = bt[kp / p.block_size];
            off = kp % p.block_size;
          }
        }
        row[j] = blk >= 0 ? (((long long)blk * p.nkv + kvh) * p.block_size + off) * D : -1;
      }
      const int c = lane & 7, sub = lane >> 3;
#pragma unroll
      for (int i = 0; i < BN / 4; ++i) {
        const int key = 4 * i + sub;  // held by lane key % 32 in slot key / 32 = i / 8
        const long long src = __shfl_sync(0xffffffffu, row[i >> 3], 4 * (i & 7) + sub);
        const bool valid = src >= 0;
#pragma unroll
        for (int h = 0; h < HALVES; ++h) {
          const long long at = valid ? src + h * 64 + c * 8 : 0;
          cpa16(ks + h * KV_HALF + sw128(key, c), p.kcache + at, valid);
          cpa16(vs + h * KV_HALF + sw128(key, c), p.vcache + at, valid);
        }
      }
    };
    if (p.use_tma) {
      // A tile is 64 / box_rows boxes of K and as many of V, one pair per lane, which the copy
      // engine lands in the swizzled layout and counts on the stage's barrier.  Only a tile that
      // reaches past the context inside a live page (whatever lies there must not be read: the
      // last tile of the sequence, at most) goes the slow way, which zero-fills by key.
      cpa_commit();  // Q
      bool ok = true, q_handed = false;
      for (int t = 0; t < n_tiles && ok; ++t) {
        const int s = t % KV_STAGES;
        if (t >= KV_STAGES) ok = __all_sync(0xffffffffu, bar_wait(kv_empty0 + 8 * s, ((t / KV_STAGES) - 1) & 1, p.err));
        if (!ok) break;
        const int t0 = first_of(t);
        const bool ragged = t0 + BN > ctx && (ctx & (p.box_rows - 1)) != 0;
        if (!ragged) {
          // lane j brings box j of the tile (box_rows keys of one page: a K box and a V box)
          const uint32_t bar = kv_full0 + 8 * s, ks = kv_s + s * 2 * KV_BYTES, vs = ks + KV_BYTES;
          if (lane == 0) bar_expect_tx(bar, 2 * KV_BYTES);
          __syncwarp();
          if (lane < BN / p.box_rows) {
            const int key0 = t0 + p.box_rows * lane;
            int blk = -1, off = 0;
            if (key0 < ctx) {
              if (p.bs_shift >= 0) {
                blk = bt[key0 >> p.bs_shift];
                off = key0 & (p.block_size - 1);
              } else {
                blk = bt[key0 / p.block_size];
                off = key0 % p.block_size;
              }
            }
            const int row = blk >= 0 ? (blk * p.nkv + kvh) * p.block_size + off : p.total_rows;
#pragma unroll
            for (int h = 0; h < HALVES; ++h) {
              tma_load_2d(ks + h * KV_HALF + lane * p.box_rows * 128, &map_k, 64 * h, row, bar);
              tma_load_2d(vs + h * KV_HALF + lane * p.box_rows * 128, &map_v, 64 * h, row, bar);
            }
          }
        } else {
          issue_tile(t);
          cpa_commit();
          cpa_wait<0>();
          fence_async_smem();
          __syncwarp();
          if (lane == 0) {
            if (!q_handed) bar_arrive(q_full);
            bar_arrive(kv_full0 + 8 * s);
          }
          q_handed = true;
        }
        if (!q_handed && (t + 1 >= KV_STAGES || t + 1 == n_tiles)) {
          // the first tiles are on their way: now wait for Q
          cpa_wait<0>();
          fence_async_smem();
          __syncwarp();
          if (lane == 0) bar_arrive(q_full);
          q_handed = true;
        }
      }
    } else {
    // groups: {Q, tile 0}, {tile 1}, ...; an empty group stands for a tile past the end
#pragma unroll
      for (int t = 0; t < LOOKAHEAD; ++t) {
        if (t < n_tiles) issue_tile(t);
        cpa_commit();
      }
      bool ok = true;
      for (int t = 0; t < n_tiles && ok; ++t) {
        // tile t (and, the first time, Q) has landed: hand it to the tensor core
        cpa_wait<LOOKAHEAD - 1>();
        fence_async_smem();
        __syncwarp();
        if (lane == 0) {
          if (t == 0) bar_arrive(q_full);
          bar_arrive(kv_full0 + 8 * (t % KV_STAGES));
        }
        const int nx = t + LOOKAHEAD;
        if (nx < n_tiles) {
          if (nx >= KV_STAGES) ok = bar_wait(kv_empty0 + 8 * (nx % KV_STAGES), ((nx / KV_STAGES) - 1) & 1, p.err);
          if (ok) issue_tile(nx);
        }
        cpa_commit();
      }
      cpa_wait<0>();
    }
  } else if (live && warp == MMA_WARP) {
    if (lane == 0) {
      // ---- MMA issuer.  When P(t) arrives its group waits for S(t+2) and for nothing else, so S(t+2)
      // goes out first (its buffer was read before P(t) was written) and P(t) V(t) after it; whether
      // K(t+2) has landed is asked while the softmax of tile t still runs.  Descriptors are made
      // once; a tile's differ from them by its stage and k-step (the address field counts 16-byte
      // units and cannot carry out of its 14 bits: shared memory ends below 256 KB).
      constexpr uint32_t id_s = idesc(BN, 0), id_o = idesc(64, 1);
      constexpr uint32_t STAGE_UNITS = (2 * KV_BYTES) >> 4;
      const uint64_t q_d = sdesc(q_s), k_d = sdesc(kv_s), v_d = sdesc(kv_s + KV_BYTES), p_d = sdesc(p_s);
      auto issue_s = [&](int t, int stage) {
        const uint32_t dst = tmem_s + (uint32_t)((t & 1) * BN);
        const uint64_t kd = k_d + (uint32_t)stage * STAGE_UNITS;
        umma_c<0>(dst, q_d, kd, id_s);
#pragma unroll
        for (int kk = 1; kk < D / 16; ++kk)  // k-steps 0..3 in the first half of the tiles, 4..7 in the second
          umma_c<1>(dst, q_d + (((kk >> 2) * Q_HALF) >> 4) + 2 * (kk & 3), kd + (((kk >> 2) * KV_HALF) >> 4) + 2 * (kk & 3), id_s);
        umma_commit(s_full0 + 8 * (t & 1));
      };
      bool ok = bar_wait(q_full, 0, p.err);
      if (ok) ok = bar_wait(kv_full0, 0, p.err);
      if (ok) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        issue_s(0, 0);
      }
      if (ok && n_tiles > 1) {
        ok = bar_wait(kv_full0 + 8, 0, p.err);
        if (ok) {
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          issue_s(1, 1);
        }
      }
      int st_s = 2 % KV_STAGES, st_pv = 0;  // the stages of tile t+2 and of tile t
      for (int t = 0; t < n_tiles && ok; ++t) {
        const bool more = t + 2 < n_tiles;
        if (more) ok = bar_wait(kv_full0 + 8 * st_s, ((t + 2) / KV_STAGES) & 1, p.err);
        if (ok) ok = bar_wait(p_full0 + 8 * (t & 1), (t >> 1) & 1, p.err);  // P(t) is in shared memory, O has been rescaled
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (more) {
          issue_s(t + 2, st_s);
          st_s = st_s + 1 == KV_STAGES ? 0 : st_s + 1;
        }
        const uint64_t vd = v_d + (uint32_t)st_pv * STAGE_UNITS, pd = p_d + (uint32_t)(t & 1) * (P_BYTES >> 4);
        const uint32_t od = tmem_o + (uint32_t)((t & 1) * D);
#pragma unroll
        for (int h = 0; h < HALVES; ++h) {  // 64 output dims per half of V
          // A: 16 keys of P = 32 bytes along the row; B: 16 keys of V = 16 rows of 128 bytes
          umma(od + 64 * h, pd, vd + ((h * KV_HALF) >> 4), id_o, t > 1 ? 1u : 0u);
#pragma unroll
          for (int kk = 1; kk < BN / 16; ++kk) umma_c<1>(od + 64 * h, pd + 2 * kk, vd + ((h * KV_HALF + kk * 16 * 128) >> 4), id_o);
        }
        umma_commit(pv_done0 + 8 * (t & 1));  // O[t&1] holds tiles t&1, .., t; P buffer t&1 may be rewritten
        umma_commit(kv_empty0 + 8 * st_pv);   // and the stage may be refilled
        st_pv = st_pv + 1 == KV_STAGES ? 0 : st_pv + 1;
      }
    }
  } else if (live && warp < SOFTMAX_WARPS) {
    // ---- softmax and output: thread r of each group owns row r; group 0 takes the even key tiles,
    // group 1 the odd ones, each with its S buffer, P buffer, O accumulator, maximum and sum
    const int grp = warp >> 2;
    const int r = threadIdx.x & 127;
    const int tok = r / g, hh = r - tok * g;
    const bool valid = tok < n_tok;
    const int pos = valid ? p_first + tok : -1;
    const int lo = first_key(pos, p.window);
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t my_s = tmem_s + lane_addr + (uint32_t)(grp * BN), my_o = tmem_o + lane_addr + (uint32_t)(grp * D);
    const uint32_t s_bar = s_full0 + 8 * grp, p_bar = p_full0 + 8 * grp, pv_bar = pv_done0 + 8 * grp;
    float m_ref = -INFINITY, l = 0.f;
    if constexpr (MODE != PLAIN) {
      bool sink = true;
      if constexpr (SH) sink = p.sinks != nullptr;
      if (sink && grp == 0 && valid) {  // the sink is where the first group starts: one in the sum at its own maximum
        m_ref = p.sinks[kvh * g + hh] * 1.4426950408889634f;
        l = 1.f;
      }
    }
    // a head's biases of a tile lie side by side by distance, p - key from -63 of the tile's first query on; heads a stride apart
    // that puts the lanes of a warp into other banks
    [[maybe_unused]] const int words = tq + BN - 1, b_stride = BIAS ? (words + 31) / 32 * 32 + (g <= 32 ? 32 / g : 1) % 32 : 0;
    bool ok = true;
    int i = 0;  // index among this group's tiles
    int t = grp;
    for (; t < n_tiles && ok; t += 2, ++i) {
      const int key0 = first_of(t);
      [[maybe_unused]] const float* brow = nullptr;
      if constexpr (BIAS) {
        float* dst = bias_s + (2 * grp + (i & 1)) * BIAS_WORDS;
        const int d0 = p_first - key0 - (BN - 1);
        for (int w = r; w < g * words; w += BM) {
          const int head = w / words, d = w - head * words;
          dst[head * b_stride + d] = __ldg(p.bias + (size_t)(kvh * g + head) * (p.bias_far + 1) + min(max(d0 + d, 0), p.bias_far)) * 1.4426950408889634f;
        }
        // one barrier a tile: the buffer written here was last read two tiles ago, before the barrier of the last one
        if (grp == 0)
          asm volatile("bar.sync 2, %0;" ::"n"(BM) : "memory");
        else
          asm volatile("bar.sync 3, %0;" ::"n"(BM) : "memory");
        brow = dst + hh * b_stride + min(tok, tq - 1) + BN - 1;
      }
      // (tcgen05.ld and st are warp-wide: the lanes of a warp leave the loop together)
      ok = __all_sync(0xffffffffu, bar_wait(s_bar, i & 1, p.err));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      uint32_t va[32], vb[32];
      tmem_ld32(my_s, va);
      tmem_ld32(my_s + 32, vb);
      // the group's last P V is done: its P buffer may be rewritten and its O may be rescaled
      if (i >= 1) ok = bar_wait(pv_bar, (i - 1) & 1, p.err);
      tmem_wait(va);
      tmem_wait(vb);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      bool need_mask = (key0 + BN - 1 > pos) || (key0 < lo);
      if constexpr (SH) need_mask = need_mask && !(key0 + BN - 1 <= pos && key0 + BN <= p.keep_first);
      const uint32_t p_row = p_s + (uint32_t)grp * P_BYTES + (uint32_t)r * 128u;
      float corr, sum;
      if constexpr (SH)
        sum = softmax_shaped<BIAS, CAP>(va, vb, m_ref, corr, p.scale_log2, p.cap_in, p.cap_out, brow, __any_sync(0xffffffffu, need_mask),
                                        max(lo, key0) - key0, min(pos, key0 + BN - 1) - key0, p.keep_first - key0, p_row, r & 7);
      else if (__any_sync(0xffffffffu, need_mask))
        sum = softmax_tile<true>(va, vb, m_ref, corr, p.scale_log2, max(lo, key0) - key0, min(pos, key0 + BN - 1) - key0, p_row, r & 7);
      else
        sum = softmax_tile<false>(va, vb, m_ref, corr, p.scale_log2, 0, BN - 1, p_row, r & 7);
      l = l * corr + sum;
      if (i > 0 && __any_sync(0xffffffffu, corr != 1.f)) {
#pragma unroll
        for (int c0 = 0; c0 < D; c0 += 32) {
          uint32_t v[32];
          tmem_ld32(my_o + (uint32_t)c0, v);
          tmem_wait(v);
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * corr);
          tmem_st32(my_o + (uint32_t)c0, v);
        }
        tmem_wait_st();
      }
      fence_async_smem();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      bar_arrive(p_bar);
    }
    if constexpr (BIAS) {
      // a warp whose wait ran out still meets the others of its group at the barriers of the tiles left
      if (!ok)
        for (t += 2; t < n_tiles; t += 2) {
          if (grp == 0)
            asm volatile("bar.sync 2, %0;" ::"n"(BM) : "memory");
          else
            asm volatile("bar.sync 3, %0;" ::"n"(BM) : "memory");
        }
    }
    if (ok && i > 0) ok = __all_sync(0xffffffffu, bar_wait(pv_bar, (i - 1) & 1, p.err));
    // ---- the two groups' results become one: group 1 hands its maximum and sum over (through its P
    // buffer, which its last P V has read), group 0 reads both accumulators
    float2* xch = reinterpret_cast<float2*>(smem_raw + (p_s + P_BYTES - base));
    if (grp == 1) xch[r] = make_float2(ok ? m_ref : -INFINITY, ok ? l : 0.f);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    asm volatile("bar.sync 1, %0;" ::"n"(SOFTMAX_WARPS * 32) : "memory");
    if (grp == 0 && ok) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const float2 other = xch[r];
      const float m_all = fmaxf(m_ref, other.x);
      const float w0 = (m_ref == -INFINITY) ? 0.f : ex2(m_ref - m_all), w1 = (other.x == -INFINITY) ? 0.f : ex2(other.x - m_all);
      const float l_all = l * w0 + other.y * w1;
      // a sum that is no number (a key that is none, an infinite score) shows in the result
      const float f0 = l_all != 0.f ? w0 / l_all : 0.f, f1 = l_all != 0.f ? w1 / l_all : 0.f;
      const bool seen1 = other.y != 0.f;                   // this row saw a key of group 1
      const bool use1 = __any_sync(0xffffffffu, seen1);  // group 1 saw a tile (else its accumulator was never written)
      bf16* dst = p.out + (size_t)(q_begin + q0 + (valid ? tok : 0)) * p.out_stride + (size_t)(kvh * g + hh) * D;
#pragma unroll
      for (int c0 = 0; c0 < D; c0 += 32) {
        uint32_t v[32], u[32];
        tmem_ld32(my_o + (uint32_t)c0, v);
        tmem_wait(v);
        if (use1) {
          tmem_ld32(my_o + (uint32_t)(D + c0), u);
          tmem_wait(u);
        }
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
          float f[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            f[e] = __uint_as_float(v[j + e]) * f0;
            if (use1 && seen1) f[e] += __uint_as_float(u[j + e]) * f1;
          }
          if (valid)
            *reinterpret_cast<uint4*>(dst + c0 + j) = make_uint4(pk(f[0], f[1]), pk(f[2], f[3]), pk(f[4], f[5]), pk(f[6], f[7]));
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(Shape<D>::TMEM_COLS) : "memory");
  }
}

}  // namespace

namespace {

template <int D, int MODE>
int launch_tc_attn(const CUtensorMap& mk, const CUtensorMap& mv, const typename ParamsOf<MODE>::type& p, dim3 grid, cudaStream_t st) {
  constexpr size_t smem = Shape<D, (MODE >= SHAPED)>::SMEM_BYTES;
  cudaError_t e = cudaFuncSetAttribute(attn_tcgen05_kernel<D, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  return launch(attn_tcgen05_kernel<D, MODE>, grid, dim3(THREADS), smem, st, mk, mv, p);
}

template <int D>
int launch_shaped(const CUtensorMap& mk, const CUtensorMap& mv, const TcAttnShapedParams& p, dim3 grid, cudaStream_t st) {
  switch ((p.bias ? 1 : 0) + (p.cap_out > 0.f ? 2 : 0)) {
    case 0: return launch_tc_attn<D, SHAPED>(mk, mv, p, grid, st);
    case 1: return launch_tc_attn<D, SHAPED + 1>(mk, mv, p, grid, st);
    case 2: return launch_tc_attn<D, SHAPED + 2>(mk, mv, p, grid, st);
    default: return launch_tc_attn<D, SHAPED + 3>(mk, mv, p, grid, st);
  }
}

}  // namespace

// bfloat16, head size 64 or 128, nh/nkv <= 128; out rows and q rows 16-byte aligned.  err: device flag.
// kcache/vcache: [num_blocks][nkv][block_size][d].
KVF_API int kvf_paged_attention_tcgen05_bf16(const void* q, void* out, const void* kcache, const void* vcache,
                                             const int* block_tables, const int* qsl, const int* ctx_lens, int B,
                                             int max_q_len, int q_stride, int out_stride, int bt_stride, int nh,
                                             int nkv, int d, int block_size, long long num_blocks, float scale,
                                             int window, const int* work, int n_work, int* err, const float* sinks,
                                             int keep_first, const float* bias, int bias_far, float softcap, cudaStream_t st) {
  if (B <= 0 || max_q_len <= 0) return 0;
  if ((d != 64 && d != 128) || nkv <= 0 || nh % nkv != 0 || nh / nkv > BM || block_size <= 0 || num_blocks <= 0) return (int)cudaErrorInvalidValue;
  if ((q_stride & 7) || (out_stride & 7) || ((((uintptr_t)q) | ((uintptr_t)out)) & 15)) return (int)cudaErrorInvalidValue;
  if ((unsigned)B > 65535u || (max_q_len + (BM / (nh / nkv)) - 1) / (BM / (nh / nkv)) > 65535) return (int)cudaErrorInvalidValue;
  if (keep_first < 0 || softcap < 0.f || (bias && (bias_far < 0 || nh / nkv > 8))) return (int)cudaErrorInvalidValue;
  if (window <= 0) keep_first = 0;  // without a window every key before the query is seen, or every one of its chunk
  TcAttnShapedParams p;
  p.keep_first = keep_first; p.bias = bias; p.bias_far = bias_far;
  p.cap_in = softcap > 0.f ? scale / softcap : 0.f;
  p.cap_out = softcap * 1.4426950408889634f;
  p.q = (const bf16*)q; p.out = (bf16*)out; p.kcache = (const bf16*)kcache; p.vcache = (const bf16*)vcache;
  p.block_tables = block_tables; p.qsl = qsl; p.ctx_lens = ctx_lens; p.err = err;
  p.work = work;
  p.sinks = sinks;
  p.num_seqs = B;
  p.q_stride = q_stride; p.out_stride = out_stride; p.bt_stride = bt_stride;
  p.nh = nh; p.nkv = nkv; p.block_size = block_size; p.window = window;
  p.bs_shift = -1;
  for (int sh = 0; sh < 31; ++sh)
    if ((1 << sh) == block_size) p.bs_shift = sh;
  p.scale_log2 = scale * 1.4426950408889634f;
  // pages of a multiple of 16 keys come in as tensor-map boxes; other page sizes key by key
  const long long rows = num_blocks * nkv * block_size;
  p.use_tma = (block_size % 16 == 0) && rows < (1ll << 31) - 64 && ((((uintptr_t)kcache) | ((uintptr_t)vcache)) & 15) == 0;
  p.total_rows = (int)(p.use_tma ? rows : 0);
  p.box_rows = block_size % 64 == 0 ? 64 : block_size % 32 == 0 ? 32 : 16;
  CUtensorMap mk, mv;
  memset(&mk, 0, sizeof(mk));
  memset(&mv, 0, sizeof(mv));
  if (p.use_tma) {
    if (cache_map(&mk, kcache, rows, d, p.box_rows) || cache_map(&mv, vcache, rows, d, p.box_rows)) p.use_tma = 0;
  }
  const int g = nh / nkv, tq = BM / g;
  if (work && (n_work <= 0 || n_work > 65535)) return (int)cudaErrorInvalidValue;
  const dim3 grid(nkv, work ? n_work : B, work ? 1 : (max_q_len + tq - 1) / tq);
  if (keep_first || bias || softcap > 0.f) return d == 64 ? launch_shaped<64>(mk, mv, p, grid, st) : launch_shaped<128>(mk, mv, p, grid, st);
  const TcAttnSinkParams& sunk = p;
  if (sinks) return d == 64 ? launch_tc_attn<64, SINKS>(mk, mv, sunk, grid, st) : launch_tc_attn<128, SINKS>(mk, mv, sunk, grid, st);
  const TcAttnParams& plain = p;
  return d == 64 ? launch_tc_attn<64, PLAIN>(mk, mv, plain, grid, st) : launch_tc_attn<128, PLAIN>(mk, mv, plain, grid, st);
}
