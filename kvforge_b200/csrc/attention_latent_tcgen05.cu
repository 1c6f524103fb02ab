// Attention of many queries (prompts, portions, mixed batches) over a paged cache of ONE row of d numbers per token shared by all
// heads (keys the whole row, values its first dv numbers), on the tcgen05 tensor cores; bfloat16.  Same contract as
// attention_latent.cu.
//
// A CTA serves 128 rows, a row being a (query token, head) pair (128 / nh tokens, every head), and up to 256 value columns: with
// values of 512 two CTAs share the rows' work, both making the scores.  That costs (d + 256) products a pair of row and key
// where 2 x (d + 512) / 2 would do, but the accumulator of 128 x 512 alone is all of an SM's tensor memory.  Per tile of 64 keys:
//   S = Q K^T   tcgen05.mma 128 x 64 x 16, d/16 of them.  What bounds it is shared memory: a product that reads both operands
//               there takes in 6 KB for 32 cycles of arithmetic, 48 cycles at 128 bytes a cycle.  So the first (up to four) blocks of
//               64 query numbers lie in tensor memory as the A operand (128 columns), which also leaves room for a second
//               stage of keys: 80 KB of queries + 2 x 72 KB of keys at d = 576;
//   softmax     one thread a row, from tensor memory, as in attention_tcgen05.cu (running maximum raised lazily); P takes the place
//               of S in tensor memory;
//   O += P V    P as the A operand from tensor memory, the value tile being the key tile's first dv columns, read as an
//               MN-major B operand; O stays in tensor memory.
// S has two buffers: S(t+1) is made while the softmax of tile t runs.  The blocks of a key tile outside the CTA's value
// columns are free as soon as S is made, the others after P V: each stage has a full and an empty barrier for either part, so
// that the next tile but one comes in early.  P V has a barrier for the even and one for the odd tiles: a thread that does not
// wait for every tile's product would mistake the phase before the last for the one it means on a single barrier.  P(t) V(t) has to be over before S(t+2) takes its buffer.
// Warps: four softmax (thread r owns row r), one loader (TMA boxes of 64 numbers x the keys of a page, 16-byte copies for a last tile
// that ends inside a page), one issuer.  One CTA an SM.
// 2,048 tokens, 16 heads, d = 576, dv = 512 (73 GFLOP without what the two halves repeat, 46 us at the tensor peak): 240 us against 591 us
// of the mma.sync kernel, and the same error against 64-bit (the layer around it 717 -> 367 us).
// Every mbarrier wait is bounded; if one runs out the kernel raises bit 4 of the error flag and winds down.
#include "tcgen05.cuh"

using namespace kvf;
using namespace kvf::tc;

namespace {

constexpr int BM = 128, BN = 64;
constexpr int LOADER_WARP = 4, MMA_WARP = 5, THREADS = 192;
constexpr int MAX_BLOCKS = 9;                // blocks of 64 numbers of a cache row (d <= 576)
constexpr int Q_TMEM = 4;                    // blocks of the queries that lie in tensor memory
constexpr uint32_t Q_BLOCK = BM * 128, K_BLOCK = BN * 128;  // bytes of a [rows][64] block
constexpr uint32_t COL_O = 0, COL_S = 256, COL_Q = 384;     // tensor-memory columns: O 256, S 2 x 64, Q 4 x 32

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

__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t b, uint32_t id, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(b), "r"(id), "r"(accumulate)
      : "memory");
}

// One tile of the softmax for the thread's row: va, vb the 64 raw scores, w the 64 weights as bfloat16 pairs.  Returns their sum.
template <bool MASK>
__device__ __forceinline__ float softmax_row(const uint32_t (&va)[32], const uint32_t (&vb)[32], uint32_t (&w)[32], float& m_ref,
                                             float& corr, float scale_log2, int first, int last) {
  float mx = -INFINITY;
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    const float a = (!MASK || (j >= first && j <= last)) ? __uint_as_float(va[j]) : -INFINITY;
    const float b = (!MASK || (j + 32 >= first && j + 32 <= last)) ? __uint_as_float(vb[j]) : -INFINITY;
    mx = fmaxf(mx, fmaxf(a, b));
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
  for (int c = 0; c < 64; c += 2) {
    const uint32_t(&v)[32] = c < 32 ? va : vb;
    float x0, x1;
    unpack2(fma2(pack2(__uint_as_float(v[c & 31]), __uint_as_float(v[(c & 31) + 1])), scale2, neg_m2), x0, x1);
    float e0 = ex2(x0), e1 = ex2(x1);
    if (MASK) {
      if (c < first || c > last) e0 = 0.f;
      if (c + 1 < first || c + 1 > last) e1 = 0.f;
    }
    if (c & 2)
      sum_b = add2(sum_b, pack2(e0, e1));
    else
      sum_a = add2(sum_a, pack2(e0, e1));
    w[c >> 1] = pk(e0, e1);
  }
  float s0, s1;
  unpack2(add2(sum_a, sum_b), s0, s1);
  return s0 + s1;
}

__global__ void __launch_bounds__(THREADS, 1) latent_tcgen05_kernel(const __grid_constant__ CUtensorMap map, const LatTcParams p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const uint32_t base = sm32(smem_raw);
  const uint32_t q_s = base;                                             // [kb - qt] blocks of [128 rows][64]
  const uint32_t k_s = q_s + (uint32_t)(p.kb - p.qt) * Q_BLOCK;          // per stage [kb] blocks of [64 keys][64]
  const uint32_t k_stage = (uint32_t)p.kb * K_BLOCK;
  const uint32_t bars = k_s + 2 * k_stage;
  // part 0 of a key tile: the blocks outside this CTA's value columns; part 1: the others
  const uint32_t q_full = bars, kf0 = bars + 8, kf1 = bars + 24, ke0 = bars + 40, ke1 = bars + 56, s_full = bars + 72, p_full = bars + 88,
                 pv_done = bars + 104, drained = bars + 120, tmem_slot = bars + 128;
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
  const int kv_lo = live ? (first_key(p_first, p.window) / BN) * BN : 0;
  const int n_tiles = live ? (kv_hi - kv_lo + BN - 1) / BN : 0;

  if (threadIdx.x == 0) {
    bar_init(q_full, BM + 1);
    for (int s = 0; s < 2; ++s) {
      bar_init(kf0 + 8 * s, 1);
      bar_init(kf1 + 8 * s, 1);
      bar_init(ke0 + 8 * s, 1);
      bar_init(ke1 + 8 * s, 1);
      bar_init(s_full + 8 * s, 1);
      bar_init(p_full + 8 * s, BM);
      bar_init(pv_done + 8 * s, 1);
    }
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
    // ---- loader: the queries' blocks that lie in shared memory, then the key tiles
    const int qc = (p.kb - p.qt) * 8;  // 16-byte chunks of a row
    for (int idx = lane; idx < BM * qc; idx += 32) {
      const int r = idx / qc, c = idx - r * qc;
      const int tok = r / p.nh, hh = r - tok * p.nh;
      const int at = (p.qt * 8 + c) * 8;
      const bool valid = tok < n_tok && at < p.d;
      cpa16(q_s + (uint32_t)(c >> 3) * Q_BLOCK + sw128(r, c & 7),
            p.q + (valid ? (size_t)(q_begin + q0 + tok) * p.q_stride + (size_t)hh * p.d + at : 0), valid);
    }
    cpa_commit();
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
    int last0 = -1, last1 = -1;  // the last tile whose part 0, whose part 1 was asked for
    bool ok = true, q_handed = false;
    for (int t = 0; t < n_tiles && ok; ++t) {
      const int s = t & 1;
      const uint32_t ks = k_s + (uint32_t)s * k_stage;
      const int t0 = kv_lo + t * BN;
      const bool ragged = t0 + BN > ctx && (ctx & (p.box_rows - 1)) != 0;
      const uint32_t par = ((t >> 1) - 1) & 1;
      if (!ragged) {
        // lane j looks up box j (box_rows keys of one page); then the lanes share out the boxes of the part's blocks
        int off;
        const int blk = page_of(t0 + p.box_rows * (lane % boxes), off);
        const int row = blk >= 0 ? blk * p.block_size + off : p.total_rows;  // past the end: zeros
        for (int part = 0; part < 2; ++part) {
          const int nb = part ? p.nvb : n0;
          if (nb == 0) continue;
          if (t >= 2) ok = __all_sync(0xffffffffu, bar_wait((part ? ke1 : ke0) + 8 * s, par, p.err));
          if (!ok) break;
          const uint32_t bar = (part ? kf1 : kf0) + 8 * s;
          if (lane == 0) bar_expect_tx(bar, (uint32_t)nb * K_BLOCK);
          __syncwarp();
          (part ? last1 : last0) = t;
          for (int i = lane; i < nb * boxes; i += 32) {  // boxes divides 32: a lane keeps its box
            const int j = i / boxes;
            const int kb = part ? vb0 + j : (j < vb0 ? j : j + p.nvb);
            tma_load_2d(ks + (uint32_t)kb * K_BLOCK + (uint32_t)((lane % boxes) * p.box_rows) * 128u, &map, 64 * kb, row, bar);
          }
        }
      } else {
        // the sequence's last tile ends inside a page, whose other keys must not be read: key by key, zeros past the context
        if (t >= 2) {
          ok = __all_sync(0xffffffffu, (n0 == 0 || bar_wait(ke0 + 8 * s, par, p.err)) && bar_wait(ke1 + 8 * s, par, p.err));
          if (!ok) break;
        }
        const int chunks = p.kb * 8;
        for (int key = 0; key < BN; ++key) {
          int off;
          const int blk = page_of(t0 + key, off);
          const bf16* src = p.cache + (blk >= 0 ? ((size_t)blk * p.block_size + off) * p.d : 0);
          for (int c = lane; c < chunks; c += 32) {
            const bool valid = blk >= 0 && c * 8 < p.d;
            cpa16(ks + (uint32_t)(c >> 3) * K_BLOCK + sw128(key, c & 7), src + (valid ? c * 8 : 0), valid);
          }
        }
        cpa_commit();
        cpa_wait<0>();
        fence_async_smem();
        __syncwarp();
        if (lane == 0) {
          if (!q_handed) bar_arrive(q_full);
          if (n0) bar_arrive(kf0 + 8 * s);
          bar_arrive(kf1 + 8 * s);
        }
        q_handed = true;
        if (n0) last0 = t;
        last1 = t;
      }
      if (ok && !q_handed && (t == 1 || t + 1 == n_tiles)) {  // the first tiles are on their way: now wait for the queries
        cpa_wait<0>();
        fence_async_smem();
        __syncwarp();
        if (lane == 0) bar_arrive(q_full);
        q_handed = true;
      }
    }
    cpa_wait<0>();
    // no copy outlives the CTA, whatever made the others leave
    for (int back = 0; back < 2; ++back) {
      if (last0 - back >= 0) bar_wait(kf0 + 8 * ((last0 - back) & 1), ((last0 - back) >> 1) & 1, p.err);
      if (last1 - back >= 0) bar_wait(kf1 + 8 * ((last1 - back) & 1), ((last1 - back) >> 1) & 1, p.err);
    }
  } else if (live && warp == MMA_WARP) {
    if (lane == 0) {
      const uint32_t id_s = idesc(BN, 0), id_o = idesc(64, 1);
      const uint64_t q_d = sdesc(q_s), k_d = sdesc(k_s);
      bool ok = bar_wait(q_full, 0, p.err);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      auto issue_s = [&](int t) {
        const int s = t & 1;
        const uint32_t dst = tmem + COL_S + (uint32_t)s * BN, par = (t >> 1) & 1;
        const uint64_t kd = k_d + (uint64_t)(((uint32_t)s * k_stage) >> 4);
        uint32_t acc = 0;
        for (int part = 0; part < 2; ++part) {
          const int nb = part ? p.nvb : n0;
          if (nb == 0) continue;
          if (!bar_wait((part ? kf1 : kf0) + 8 * s, par, p.err)) return false;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          for (int j = 0; j < nb; ++j) {
            const int kb = part ? vb0 + j : (j < vb0 ? j : j + p.nvb);
            const uint64_t bd = kd + (uint64_t)((uint32_t)kb * (K_BLOCK >> 4));
            if (kb < p.qt) {
              const uint32_t a = tmem + COL_Q + (uint32_t)kb * 32u;
#pragma unroll
              for (int kk = 0; kk < 4; ++kk) {
                umma_ts(dst, a + 8u * kk, bd + 2 * kk, id_s, acc);
                acc = 1;
              }
            } else {
              const uint64_t ad = q_d + (uint64_t)((uint32_t)(kb - p.qt) * (Q_BLOCK >> 4));
#pragma unroll
              for (int kk = 0; kk < 4; ++kk) {
                umma(dst, ad + 2 * kk, bd + 2 * kk, id_s, acc);
                acc = 1;
              }
            }
          }
          if (part == 0) umma_commit(ke0 + 8 * s);  // what is not a value is free again
        }
        umma_commit(s_full + 8 * s);
        return true;
      };
      if (ok) ok = issue_s(0);
      if (ok && n_tiles > 1) ok = issue_s(1);
      for (int t = 0; t < n_tiles && ok; ++t) {
        const int s = t & 1;
        ok = bar_wait(p_full + 8 * s, (t >> 1) & 1, p.err);  // P(t) is in tensor memory, O has been rescaled
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a = tmem + COL_S + (uint32_t)s * BN;
        const uint64_t vd = k_d + (uint64_t)(((uint32_t)s * k_stage + (uint32_t)vb0 * K_BLOCK) >> 4);
        for (int j = 0; j < p.nvb; ++j) {
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)  // A: 16 keys of P = 8 columns; B: 16 keys = 16 rows of 128 bytes
            umma_ts(tmem + COL_O + 64u * j, a + 8u * kk, vd + (uint64_t)((uint32_t)j * (K_BLOCK >> 4) + kk * (16 * 128 >> 4)), id_o,
                    (t > 0 || kk > 0) ? 1u : 0u);
        }
        umma_commit(pv_done + 8 * s);
        umma_commit(ke1 + 8 * s);
        if (t + 2 < n_tiles) {
          ok = bar_wait(pv_done + 8 * s, (t >> 1) & 1, p.err);  // S(t+2) goes where P(t) lies
          if (ok) ok = issue_s(t + 2);
        }
      }
      if (!ok) {  // no product outlives the tensor memory
        umma_commit(drained);
        bar_wait(drained, 0, p.err);
      }
    }
  } else if (live && warp < 4) {
    // ---- softmax and output: thread r owns row r
    const int r = threadIdx.x;
    const int tok = r / p.nh, hh = r - tok * p.nh;
    const bool valid = tok < n_tok;
    const int pos = valid ? p_first + tok : -1;
    const int lo = first_key(pos, p.window);
    const uint32_t lane_addr = (uint32_t)(warp * 32) << 16;
    const uint32_t my_s = tmem + lane_addr + COL_S, my_o = tmem + lane_addr + COL_O;
    {
      const uint4* src = reinterpret_cast<const uint4*>(p.q + (valid ? (size_t)(q_begin + q0 + tok) * p.q_stride + (size_t)hh * p.d : 0));
      for (int blk = 0; blk < p.qt; ++blk) {
        uint32_t v[32];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const uint4 u = valid ? src[blk * 8 + c] : make_uint4(0u, 0u, 0u, 0u);
          v[4 * c] = u.x; v[4 * c + 1] = u.y; v[4 * c + 2] = u.z; v[4 * c + 3] = u.w;
        }
        tmem_st32(tmem + lane_addr + COL_Q + (uint32_t)blk * 32u, v);
      }
      tmem_wait_st();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      bar_arrive(q_full);
    }
    float m_ref = -INFINITY, l = 0.f;
    bool ok = true;
    int t = 0;
    for (; t < n_tiles && ok; ++t) {
      const int s = t & 1, key0 = kv_lo + t * BN;
      // (tcgen05.ld and st are warp-wide: the lanes of a warp leave the loop together)
      ok = __all_sync(0xffffffffu, bar_wait(s_full + 8 * s, (t >> 1) & 1, p.err));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      uint32_t va[32], vb[32], w[32];
      tmem_ld32(my_s + (uint32_t)s * BN, va);
      tmem_ld32(my_s + (uint32_t)s * BN + 32u, vb);
      tmem_wait(va);
      tmem_wait(vb);
      const bool need_mask = (key0 + BN - 1 > pos) || (key0 < lo);
      float corr, sum;
      if (__any_sync(0xffffffffu, need_mask))
        sum = softmax_row<true>(va, vb, w, m_ref, corr, p.scale_log2, max(lo, key0) - key0, min(pos, key0 + BN - 1) - key0);
      else
        sum = softmax_row<false>(va, vb, w, m_ref, corr, p.scale_log2, 0, BN - 1);
      l = l * corr + sum;
      tmem_st32(my_s + (uint32_t)s * BN, w);  // 64 weights = 32 columns, where the thread's scores were
      if (t > 0 && __any_sync(0xffffffffu, corr != 1.f)) {
        ok = __all_sync(0xffffffffu, bar_wait(pv_done + 8 * (s ^ 1), ((t - 1) >> 1) & 1, p.err));  // O holds tiles 0 .. t-1
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int c0 = 0; c0 < 64 * p.nvb; c0 += 32) {
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
      bar_arrive(p_full + 8 * s);
    }
    if (ok) ok = __all_sync(0xffffffffu, bar_wait(pv_done + 8 * ((n_tiles - 1) & 1), ((n_tiles - 1) >> 1) & 1, p.err));
    if (ok) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const float inv = l > 0.f ? 1.f / l : 0.f;
      bf16* dst = p.out + (size_t)(q_begin + q0 + (valid ? tok : 0)) * p.out_stride + (size_t)hh * p.dv + vb0 * 64;
      for (int c0 = 0; c0 < 64 * p.nvb; c0 += 32) {
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
  const size_t smem = (size_t)(p.kb - p.qt) * Q_BLOCK + (size_t)2 * p.kb * K_BLOCK + 144;
  const cudaError_t e = cudaFuncSetAttribute(latent_tcgen05_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  return launch(latent_tcgen05_kernel, dim3(dv / (64 * p.nvb), work ? n_work : B, work ? 1 : tiles), dim3(THREADS), smem, st, map, p);
}
