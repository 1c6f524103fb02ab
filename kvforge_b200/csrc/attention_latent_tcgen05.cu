// Attention of many queries (prompts, portions, mixed batches) over a paged cache of ONE row of d numbers per token shared by all
// heads (keys the whole row, values its first dv numbers), on the tcgen05 tensor cores; bfloat16.  Same contract as
// attention_latent.cu.
//
// A CTA serves 128 rows, a row being a (query token, head) pair (128 / nh tokens, every head), and up to 256 value columns: with
// values of 512 two CTAs share the rows' work, both making the scores.  That costs 2 x (d + 256) products a pair of row and key where
// d + 512 would do (1,664 and 1,088 for d = 576), but the accumulator of 128 x 512 alone is all of an SM's tensor memory.  Per tile
// of 128 keys:
//   S = Q K^T   tcgen05.mma 128 x 128 x 16, d/16 of them.  The first (up to four) blocks of 64 query numbers lie in tensor memory
//               as the A operand (128 columns): 80 KB of queries and 144 KB of keys are what an SM holds;
//   softmax     two groups of four warps, 64 keys of a row a thread, from tensor memory, as in attention_tcgen05.cu (the two
//               halves of a row exchange their maxima); P takes the place of S in tensor memory;
//   O += P V    P as the A operand from tensor memory, the value tile being the key tile's first dv columns, read as an
//               MN-major B operand of all the CTA's columns at once, blocks of 64 a stride apart (a product of its own for each block
//               of columns costs the issuing thread some 80 cycles, four of them 24 us of 184); O stays in tensor memory.
// The blocks of a key tile outside the CTA's value columns are free as soon as S is made, the others after P V: either part has a
// full and an empty barrier, so that the next tile's first part comes in under the softmax and its second under the first's products.
// Warps: eight softmax (which first bring the queries in), one loader (TMA boxes of 64 numbers x the keys of a page, 16-byte
// copies for the page that the context ends in), one issuer.  One CTA an SM.
// 2,048 tokens, 16 heads, d = 576, dv = 512 (73 GFLOP without what the two halves repeat, 46 us at the tensor peak): 161 us against 587 us
// of the mma.sync kernel, and the same error against 64-bit.  What bounds it is that scores, softmax, products and copies of a tile follow one
// another, for want of room for a second tile: with tiles of 64 keys in two stages and four softmax warps it took 233 us, with tiles of
// 128 and eight warps 220, 184 since those eight and not the loader alone bring the queries (147 KB a CTA), and 153 with one product
// for all value columns (pages of 16 tokens); the exact maximum (below) costs 8 of the 161.
// Every mbarrier wait is bounded; if one runs out the kernel raises bit 4 of the error flag and winds down.
#include "tcgen05.cuh"

using namespace kvf;
using namespace kvf::tc;

namespace {

constexpr int BM = 128, BN = 128, HALF = 64;  // rows, keys a tile, keys a softmax group takes of it
constexpr int SOFTMAX_THREADS = 2 * BM, LOADER_WARP = 8, MMA_WARP = 9, THREADS = 320;
constexpr int MAX_BLOCKS = 9;                // blocks of 64 numbers of a cache row (d <= 576)
constexpr int Q_TMEM = 4;                    // blocks of the queries that lie in tensor memory
constexpr uint32_t Q_BLOCK = BM * 128, K_BLOCK = BN * 128;  // bytes of a [rows][64] block
constexpr uint32_t COL_O = 0, COL_S = 256, COL_Q = 384;     // tensor-memory columns: O 256, S 128, Q 4 x 32

struct LatTcParams {
  const bf16* q;
  bf16* out;
  const bf16* cache;
  const int* block_tables;
  const int* qsl;
  const int* ctx_lens;
  const int* work;  // n_work pairs (sequence or -1, first query of the tile), or null: the grid's y and z say which
  int* err;
  int num_seqs;
  int q_stride, out_stride, bt_stride;
  int nh, d, dv, tq;
  int block_size, bs_shift, box_rows, total_rows;
  int window;
  int kb, qt;      // blocks of a row; how many of them lie in tensor memory for the queries
  int nvb;         // value blocks of a CTA
  float scale_log2;
};

// The maximum of the thread's 64 raw scores, of those from `first` to `last` with MASK.
template <bool MASK>
__device__ __forceinline__ float row_max(const uint32_t (&va)[32], const uint32_t (&vb)[32], int first, int last) {
  float mx = -INFINITY;
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    const float a = (!MASK || (j >= first && j <= last)) ? __uint_as_float(va[j]) : -INFINITY;
    const float b = (!MASK || (j + 32 >= first && j + 32 <= last)) ? __uint_as_float(vb[j]) : -INFINITY;
    mx = fmaxf(mx, fmaxf(a, b));
  }
  return mx;
}
// exp2(score * scale - m_ref) of the 64 scores as bfloat16 pairs; returns the (float) sum of what was stored, so that the
// division cancels a part of the rounding: a weight's error counts by how far its value lies from the result.
template <bool MASK>
__device__ __forceinline__ float weights(const uint32_t (&va)[32], const uint32_t (&vb)[32], uint32_t (&w)[32], float m_ref, float scale_log2, int first, int last) {
  const float m_use = (m_ref == -INFINITY) ? 0.f : m_ref;
  const uint64_t scale2 = pack2(scale_log2, scale_log2), neg_m2 = pack2(-m_use, -m_use);
  uint64_t sum_a = pack2(0.f, 0.f), sum_b = sum_a;
#pragma unroll
  for (int c = 0; c < 64; c += 2) {
    const uint32_t(&v)[32] = c < 32 ? va : vb;
    float x0, x1;
    unpack2(fma2(pack2(__uint_as_float(v[c & 31]), __uint_as_float(v[(c & 31) + 1])), scale2, neg_m2), x0, x1);
    float e0 = ex2(x0), e1 = ex2(x1);
    if (MASK) {
      if (c < first || c > last) e0 = 0.f;
      if (c + 1 < first || c + 1 > last) e1 = 0.f;
    }
    const uint32_t both = pk(e0, e1);
    w[c >> 1] = both;
    const uint64_t rounded = pack2(__uint_as_float(both << 16), __uint_as_float(both & 0xffff0000u));
    if (c & 2)
      sum_b = add2(sum_b, rounded);
    else
      sum_a = add2(sum_a, rounded);
  }
  float s0, s1;
  unpack2(add2(sum_a, sum_b), s0, s1);
  return s0 + s1;
}

__global__ void __launch_bounds__(THREADS, 1) latent_tcgen05_kernel(const __grid_constant__ CUtensorMap map, const LatTcParams p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const uint32_t base = sm32(smem_raw);
  const uint32_t q_s = base;                                             // [kb - qt] blocks of [128 rows][64]
  const uint32_t k_s = q_s + (uint32_t)(p.kb - p.qt) * Q_BLOCK;          // [kb] blocks of [128 keys][64]
  const uint32_t xch = k_s + (uint32_t)p.kb * K_BLOCK;                   // [2][2][128] floats: the halves' maxima, of even and odd tiles
  const uint32_t bars = xch + 4 * BM * 4;
  // part 0 of a key tile: the blocks outside this CTA's value columns; part 1: the others
  const uint32_t q_full = bars, kf0 = bars + 8, kf1 = bars + 16, ke0 = bars + 24, ke1 = bars + 32, s_full = bars + 40, p_full = bars + 48,
                 pv_done = bars + 56, drained = bars + 64, tmem_slot = bars + 72;
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - base));

  pdl_launch();
  if (base & 1023u) {  // as declared, else refuse rather than compute garbage
    if (threadIdx.x == 0 && p.err) atomicOr(p.err, 8);
    pdl_wait();
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int vb0 = blockIdx.x * p.nvb;  // first value block
  const int n0 = p.kb - p.nvb;         // blocks of part 0
  int b = p.work ? p.work[2 * blockIdx.y] : (int)blockIdx.y;
  const int q0 = p.work ? p.work[2 * blockIdx.y + 1] : (int)(gridDim.z - 1 - blockIdx.z) * p.tq;  // the longest walks first
  if (b >= p.num_seqs) b = -1;
  const int q_begin = b >= 0 ? p.qsl[b] : 0, q_len = b >= 0 ? p.qsl[b + 1] - q_begin : 0;
  const int ctx = b >= 0 ? p.ctx_lens[b] : 0;
  const bool live = q_len > 0 && ctx > 0 && q0 >= 0 && q0 < q_len;  // uniform over the CTA
  // a CTA without a tile leaves at once; the grid's first one stays for the dependency wait
  if (!live && (blockIdx.x | blockIdx.y | blockIdx.z) != 0) return;
  const int n_tok = live ? min(p.tq, q_len - q0) : 0;
  const int p_first = ctx - q_len + q0;
  const int kv_hi = p_first + n_tok;
  const int seen_lo = live ? first_key(p_first, p.window) : 0, kv_lo = (seen_lo / BN) * BN;
  const int n_tiles = live ? (kv_hi - kv_lo + BN - 1) / BN : 0;

  if (threadIdx.x == 0) {
    bar_init(q_full, SOFTMAX_THREADS);
    bar_init(kf0, 1);
    bar_init(kf1, 1);
    bar_init(ke0, 1);
    bar_init(ke1, 1);
    bar_init(s_full, 1);
    bar_init(p_full, SOFTMAX_THREADS);
    bar_init(pv_done, 1);
    bar_init(drained, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot_ptr;

  pdl_wait();

  if (live && warp == LOADER_WARP) {
    // ---- loader: the key tiles
    const int* bt = p.block_tables + (size_t)b * p.bt_stride;
    auto page_of = [&](int key, int& off) {  // the page of a key (-1: past the context or given back)
      off = 0;
      if (key >= ctx) return -1;
      if (p.bs_shift >= 0) {
        off = key & (p.block_size - 1);
        return bt[key >> p.bs_shift];
      }
      off = key % p.block_size;
      return bt[key / p.block_size];
    };
    const int boxes = BN / p.box_rows;
    bool ok = true;
    int last0 = -1, last1 = -1;  // the last tile whose part 0, whose part 1 was asked for
    for (int t = 0; t < n_tiles && ok; ++t) {
      const int t0 = kv_lo + t * BN;
      const bool ragged = t0 + BN > ctx && (ctx & (p.box_rows - 1)) != 0;
      if (!ragged) {
        // lane j looks up box j (box_rows keys of one page); then the lanes share out the boxes of the part's blocks
        int off;
        const int blk = page_of(t0 + p.box_rows * (lane % boxes), off);
        const int row = blk >= 0 ? blk * p.block_size + off : p.total_rows;  // past the end: zeros
        for (int part = 0; part < 2; ++part) {
          const int nb = part ? p.nvb : n0;
          if (nb == 0) continue;
          if (t >= 1) ok = __all_sync(0xffffffffu, bar_wait(part ? ke1 : ke0, (t - 1) & 1, p.err));
          if (!ok) break;
          const uint32_t bar = part ? kf1 : kf0;
          if (lane == 0) bar_expect_tx(bar, (uint32_t)nb * K_BLOCK);
          __syncwarp();
          (part ? last1 : last0) = t;
          for (int i = lane; i < nb * boxes; i += 32) {  // boxes divides 32: a lane keeps its box
            const int j = i / boxes;
            const int kb = part ? vb0 + j : (j < vb0 ? j : j + p.nvb);
            tma_load_2d(k_s + (uint32_t)kb * K_BLOCK + (uint32_t)((lane % boxes) * p.box_rows) * 128u, &map, 64 * kb, row, bar);
          }
        }
      } else {
        // the sequence's last tile ends inside a page, whose other keys must not be read: that page's box comes key by key, with
        // zeros past the context, the others as above
        if (t >= 1) {
          ok = __all_sync(0xffffffffu, (n0 == 0 || bar_wait(ke0, (t - 1) & 1, p.err)) && bar_wait(ke1, (t - 1) & 1, p.err));
          if (!ok) break;
        }
        int off;
        const int blk = page_of(t0 + p.box_rows * (lane % boxes), off);
        const int row = blk >= 0 ? blk * p.block_size + off : p.total_rows;
        const int cut = (ctx - t0) / p.box_rows;  // the box that the context ends in
        const uint32_t others = (uint32_t)((boxes - 1) * p.box_rows) * 128u;
        if (lane == 0) {
          if (n0) bar_more_tx(kf0, (uint32_t)n0 * others);
          bar_more_tx(kf1, (uint32_t)p.nvb * others);
        }
        __syncwarp();
        for (int i = lane; i < p.kb * boxes; i += 32) {  // boxes divides 32: a lane keeps its box
          const int kb = i / boxes;
          if (lane % boxes != cut)
            tma_load_2d(k_s + (uint32_t)kb * K_BLOCK + (uint32_t)((lane % boxes) * p.box_rows) * 128u, &map, 64 * kb, row, kb >= vb0 && kb < vb0 + p.nvb ? kf1 : kf0);
        }
        int cut_off;
        const int cut_blk = page_of(t0 + cut * p.box_rows, cut_off);
        const bf16* const src = p.cache + (cut_blk >= 0 ? ((size_t)cut_blk * p.block_size + cut_off) * p.d : 0);
        const int keys = cut_blk >= 0 ? ctx - t0 - cut * p.box_rows : 0, chunks = p.kb * 8;
        for (int key = 0; key < p.box_rows; ++key)
          for (int c = lane; c < chunks; c += 32) {
            const bool valid = key < keys && c * 8 < p.d;
            cpa16(k_s + (uint32_t)(c >> 3) * K_BLOCK + sw128(cut * p.box_rows + key, c & 7), src + (valid ? (size_t)key * p.d + c * 8 : 0), valid);
          }
        cpa_commit();
        cpa_wait<0>();
        fence_async_smem();
        __syncwarp();
        if (lane == 0) {
          if (n0) bar_arrive(kf0);
          bar_arrive(kf1);
        }
        if (n0) last0 = t;
        last1 = t;
      }
    }
    // no copy outlives the CTA, whatever made the others leave
    if (last0 >= 0) bar_wait(kf0, last0 & 1, p.err);
    if (last1 >= 0) bar_wait(kf1, last1 & 1, p.err);
  } else if (live && warp == MMA_WARP) {
    if (lane == 0) {
      const uint32_t id_s = idesc(BN, 0), id_o = idesc(64 * p.nvb, 1);
      const uint64_t q_d = sdesc(q_s), k_d = sdesc(k_s), v_d = sdesc_mn(k_s + (uint32_t)vb0 * K_BLOCK, K_BLOCK);
      const uint32_t s_t = tmem + COL_S, o_t = tmem + COL_O;
      bool ok = bar_wait(q_full, 0, p.err);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int t = 0; t < n_tiles && ok; ++t) {
        if (t > 0) ok = bar_wait(pv_done, (t - 1) & 1, p.err);  // S(t) goes where P(t-1) lies
        uint32_t acc = 0;
        for (int part = 0; part < 2 && ok; ++part) {
          const int nb = part ? p.nvb : n0;
          if (nb == 0) continue;
          ok = bar_wait(part ? kf1 : kf0, t & 1, p.err);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          for (int j = 0; j < nb; ++j) {
            const int kb = part ? vb0 + j : (j < vb0 ? j : j + p.nvb);
            const uint64_t bd = k_d + (uint64_t)((uint32_t)kb * (K_BLOCK >> 4));
            if (kb < p.qt) {
              const uint32_t a = tmem + COL_Q + (uint32_t)kb * 32u;
#pragma unroll
              for (int kk = 0; kk < 4; ++kk) {
                umma_ts(s_t, a + 8u * kk, bd + 2 * kk, id_s, acc);
                acc = 1;
              }
            } else {
              const uint64_t ad = q_d + (uint64_t)((uint32_t)(kb - p.qt) * (Q_BLOCK >> 4));
#pragma unroll
              for (int kk = 0; kk < 4; ++kk) {
                umma(s_t, ad + 2 * kk, bd + 2 * kk, id_s, acc);
                acc = 1;
              }
            }
          }
          umma_commit(part ? s_full : ke0);  // S is made; what is not a value is free again
        }
        if (ok) ok = bar_wait(p_full, t & 1, p.err);  // P(t) is in tensor memory, O has been rescaled
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // Only the keys that some row of the CTA may see: a weight of zero times a value that is no number is none, and a tile
        // reaches up to 127 keys beyond the last query (and before the first one's window).
        const int key0 = kv_lo + t * BN, kk_lo = max(0, seen_lo - key0) / 16, kk_hi = min(BN, kv_hi - key0 + 15) / 16;
#pragma unroll
        for (int kk = 0; kk < BN / 16; ++kk)  // A: 16 keys of P = 8 columns; B: 16 keys = 16 rows of 128 bytes in each block
          if (kk >= kk_lo && kk < kk_hi) umma_ts(o_t, s_t + 8u * kk, v_d + (uint64_t)(kk * (16 * 128 >> 4)), id_o, (t > 0 || kk > kk_lo) ? 1u : 0u);
        umma_commit(pv_done);
        umma_commit(ke1);
      }
      if (!ok) {  // no product outlives the tensor memory
        umma_commit(drained);
        bar_wait(drained, 0, p.err);
      }
    }
  } else if (live && warp < LOADER_WARP) {
    // ---- softmax and output: thread r of either group owns row r, group 0 the first 64 keys of a tile, group 1 the others
    const int grp = warp >> 2, r = threadIdx.x & (BM - 1);
    const int tok = r / p.nh, hh = r - tok * p.nh;
    const bool valid = tok < n_tok;
    const int pos = valid ? p_first + tok : -1;
    const int lo = first_key(pos, p.window);
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t my_s = tmem + lane_addr + COL_S, my_o = tmem + lane_addr + COL_O;
    float* const mine = reinterpret_cast<float*>(smem_raw + (xch - base)) + grp * BM + r;
    const float* const theirs = reinterpret_cast<const float*>(smem_raw + (xch - base)) + (grp ^ 1) * BM + r;
    {
      // the queries: blocks from qt on to shared memory by all 256 threads, then either group writes half of the others to tensor memory
      const int qc = (p.kb - p.qt) * 8;  // 16-byte chunks of a row
      const bf16* const rows = p.q + (size_t)(q_begin + q0) * p.q_stride;
      if (qc) {
        int rr = (int)threadIdx.x / qc, c = (int)threadIdx.x - rr * qc;
        const int dr = SOFTMAX_THREADS / qc, dc = SOFTMAX_THREADS - dr * qc;
        while (rr < BM) {
          const int tk = rr / p.nh, at = (p.qt * 8 + c) * 8;
          const bool in = tk < n_tok && at < p.d;
          cpa16(q_s + (uint32_t)(c >> 3) * Q_BLOCK + sw128(rr, c & 7), rows + (in ? (size_t)tk * p.q_stride + (size_t)(rr - tk * p.nh) * p.d + at : 0), in);
          rr += dr;
          c += dc;
          if (c >= qc) {
            c -= qc;
            ++rr;
          }
        }
        cpa_commit();
      }
      const uint4* src = reinterpret_cast<const uint4*>(rows + (valid ? (size_t)tok * p.q_stride + (size_t)hh * p.d : 0));
      for (int blk = grp; blk < p.qt; blk += 2) {
        uint32_t v[32];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const uint4 u = valid ? src[blk * 8 + c] : make_uint4(0u, 0u, 0u, 0u);
          v[4 * c] = u.x; v[4 * c + 1] = u.y; v[4 * c + 2] = u.z; v[4 * c + 3] = u.w;
        }
        tmem_st32(tmem + lane_addr + COL_Q + (uint32_t)blk * 32u, v);
      }
      tmem_wait_st();
      cpa_wait<0>();
      fence_async_smem();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      bar_arrive(q_full);
    }
    float m_ref = -INFINITY, l = 0.f;
    bool ok = true;
    int t = 0;
    for (; t < n_tiles; ++t) {
      const int key0 = kv_lo + t * BN + grp * HALF;
      // (tcgen05.ld and st are warp-wide: the lanes of a warp leave the loop together)
      ok = __all_sync(0xffffffffu, bar_wait(s_full, t & 1, p.err));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      uint32_t va[32], vb[32];
      tmem_ld32(my_s + (uint32_t)(grp * HALF), va);
      tmem_ld32(my_s + (uint32_t)(grp * HALF) + 32u, vb);
      tmem_wait(va);
      tmem_wait(vb);
      const bool mask = __any_sync(0xffffffffu, (key0 + HALF - 1 > pos) || (key0 < lo));
      const int first = max(lo, key0) - key0, last = min(pos, key0 + HALF - 1) - key0;
      float mx = mask ? row_max<true>(va, vb, first, last) : row_max<false>(va, vb, 0, HALF - 1);
      mine[(t & 1) * 2 * BM] = mx;
      // both halves of every row are in registers: their maxima can be exchanged, and P may take the place of S
      asm volatile("bar.sync 1, %0;" ::"n"(SOFTMAX_THREADS) : "memory");
      mx = fmaxf(mx, theirs[(t & 1) * 2 * BM]) * p.scale_log2;  // scale > 0
      float corr = 1.f;
      // Followed exactly, so that the largest weight is one, which no rounding changes (rises of less than a factor of 2^8 left
      // alone and the weights summed before they are rounded: results are 1.01 to 1.24 times as far off against 64 bits as on the
      // mma.sync kernel, with both 0.995 to 1.004; 2,048 tokens 153 us and 161).
      if (mx > m_ref) {
        corr = ex2(m_ref - mx);  // 0 the first time
        m_ref = mx;
      }
      uint32_t w[32];
      const float sum = mask ? weights<true>(va, vb, w, m_ref, p.scale_log2, first, last) : weights<false>(va, vb, w, m_ref, p.scale_log2, 0, HALF - 1);
      l = l * corr + sum;
      tmem_st32(my_s + (uint32_t)(grp * 32), w);  // 64 weights = 32 columns
      // P V of the tile before is over (S(t) was made after it): either group rescales half of O
      if (t > 0 && __any_sync(0xffffffffu, corr != 1.f)) {
        for (int c0 = 32 * grp; c0 < 64 * p.nvb; c0 += 64) {
          uint32_t v[32];
          tmem_ld32(my_o + (uint32_t)c0, v);
          tmem_wait(v);
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * corr);
          tmem_st32(my_o + (uint32_t)c0, v);
        }
      }
      tmem_wait_st();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      bar_arrive(p_full);
    }
    // a warp whose wait ran out still meets the others at the barriers of the tiles left
    if (!ok)
      for (; t < n_tiles; ++t) asm volatile("bar.sync 1, %0;" ::"n"(SOFTMAX_THREADS) : "memory");
    if (ok) ok = __all_sync(0xffffffffu, bar_wait(pv_done, (n_tiles - 1) & 1, p.err));
    // (the sums take the place that the maxima of the tile before the last had)
    mine[(n_tiles & 1) * 2 * BM] = l;
    asm volatile("bar.sync 1, %0;" ::"n"(SOFTMAX_THREADS) : "memory");
    l += theirs[(n_tiles & 1) * 2 * BM];
    if (ok) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const float inv = l > 0.f ? 1.f / l : 0.f;
      bf16* dst = p.out + (size_t)(q_begin + q0 + (valid ? tok : 0)) * p.out_stride + (size_t)hh * p.dv + vb0 * 64;
      for (int c0 = 32 * grp; c0 < 64 * p.nvb; c0 += 64) {
        uint32_t v[32];
        tmem_ld32(my_o + (uint32_t)c0, v);
        tmem_wait(v);
        if (valid) {
#pragma unroll
          for (int j = 0; j < 32; j += 8)
            *reinterpret_cast<uint4*>(dst + c0 + j) =
                make_uint4(pk(__uint_as_float(v[j]) * inv, __uint_as_float(v[j + 1]) * inv), pk(__uint_as_float(v[j + 2]) * inv, __uint_as_float(v[j + 3]) * inv),
                           pk(__uint_as_float(v[j + 4]) * inv, __uint_as_float(v[j + 5]) * inv), pk(__uint_as_float(v[j + 6]) * inv, __uint_as_float(v[j + 7]) * inv));
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

}  // namespace

// q: rows of q_stride elements whose first nh * d are the query heads; out [N, nh * dv], 16-byte aligned rows; cache
// [num_blocks][1][block_size][d].  Shapes this kernel does not take are refused with cudaErrorInvalidValue.
KVF_API int kvf_latent_attention_tcgen05_bf16(const void* q, void* out, const void* cache, const int* block_tables, const int* qsl,
                                              const int* ctx_lens, int B, int max_q_len, int q_stride, int out_stride, int bt_stride,
                                              int nh, int d, int dv, int block_size, long long num_blocks, float scale, int window,
                                              const int* work, int n_work, int* err, cudaStream_t st) {
  if (B <= 0 || max_q_len <= 0) return 0;
  if (d <= 0 || d > 64 * MAX_BLOCKS || (d % 16) || dv > d || (dv != 64 && dv != 128 && dv != 256 && dv != 512)) return (int)cudaErrorInvalidValue;
  if (nh <= 0 || nh > BM || block_size <= 0 || (block_size % 16) || num_blocks <= 0 || window < 0 || !(scale > 0.f)) return (int)cudaErrorInvalidValue;
  if ((q_stride & 7) || (out_stride & 7) || ((((uintptr_t)q) | ((uintptr_t)out) | ((uintptr_t)cache)) & 15)) return (int)cudaErrorInvalidValue;
  const long long rows = num_blocks * block_size;
  if (rows >= (1ll << 31) - 64) return (int)cudaErrorInvalidValue;
  LatTcParams p;
  p.q = (const bf16*)q; p.out = (bf16*)out; p.cache = (const bf16*)cache;
  p.block_tables = block_tables; p.qsl = qsl; p.ctx_lens = ctx_lens; p.work = work; p.err = err;
  p.num_seqs = B;
  p.q_stride = q_stride; p.out_stride = out_stride; p.bt_stride = bt_stride;
  p.nh = nh; p.d = d; p.dv = dv; p.tq = BM / nh;
  p.block_size = block_size;
  p.bs_shift = -1;
  for (int sh = 0; sh < 31; ++sh)
    if ((1 << sh) == block_size) p.bs_shift = sh;
  p.box_rows = block_size % 64 == 0 ? 64 : block_size % 32 == 0 ? 32 : 16;
  p.total_rows = (int)rows;
  p.window = window;
  p.kb = (d + 63) / 64;
  p.qt = p.kb - 1 < Q_TMEM ? p.kb - 1 : Q_TMEM;
  p.nvb = dv >= 256 ? 4 : dv / 64;
  p.scale_log2 = scale * 1.4426950408889634f;
  const int tiles = (max_q_len + p.tq - 1) / p.tq;
  if (work ? (n_work <= 0 || n_work > 65535) : (B > 65535 || tiles > 65535)) return (int)cudaErrorInvalidValue;
  CUtensorMap map;
  memset(&map, 0, sizeof(map));
  const int rc = cache_map(&map, cache, rows, d, p.box_rows);
  if (rc) return rc;
  const size_t smem = (size_t)(p.kb - p.qt) * Q_BLOCK + (size_t)p.kb * K_BLOCK + 4 * BM * 4 + 96;
  const cudaError_t e = cudaFuncSetAttribute(latent_tcgen05_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  return launch(latent_tcgen05_kernel, dim3(dv / (64 * p.nvb), work ? n_work : B, work ? 1 : tiles), dim3(THREADS), smem, st, map, p);
}
