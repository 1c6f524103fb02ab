// Attention whose heads talk before the softmax, many queries (prompts, portions), on the tcgen05 tensor cores; bfloat16, heads of 64 or
// 128 numbers with values as wide as keys, at most 512 numbers in a token's keys.  Same contract as attention_talking.cuh.
//
// The mixing is linear, so it can be done to the queries instead of to every score:
//   s'_h = sum_g talk[h][g] q_g . k_c(g) = sum_c q'_hc . k_c     with  q'_hc = sum over c's query heads g of talk[h][g] q_g
// and a head's scores are one product of all the kv heads' keys side by side (nkv x d numbers) with a long query of its own.  That is
// nkv times the products of plain attention, 69 GFLOP a term for 2,048 tokens, 32 heads of 64 on 8, and none of the 4.3 GFLOP a
// prompt that the mixing takes on the FP32 pipes, nor the scores' way through shared memory before and after it.  The long queries are
// made in float and go into the product as two bfloat16 terms (16 bits of them), like the weights in their product with the values.
//
// A CTA serves 128 rows of one kv head's query heads (a row a query token and head: 128 / g tokens).  Per tile of 96 keys (heads of
// 128: 64), which is what two score buffers leave room for in tensor memory and nearly the products' full rate (57.8 cycles a product
// 96 wide, 68.7 at 128, 55.4 at 64):
//   S = Q' K^T  the high terms lie in tensor memory as the A operand (256 columns), the low ones in shared memory (128 KB); the keys
//               come in blocks of 64 numbers through a ring of six, each used by eight products and given back;
//   softmax     two groups of four warps, half of a row's keys a thread, as in attention_latent_tcgen05.cu, under the next tile's
//               scores; the weights, two terms, take the place of the scores in tensor memory;
//   O += P V    the value tile as an MN-major operand; O stays in tensor memory.
// 2,048 tokens, 32 heads of 64 on 8: 147 us against 390 of the mma.sync kernel (8 single CTAs over 1,000 keys: 43 and 156), with the same
// error against 64 bits to four places (1.6596e-3 of the norm, of which all but 2e-6 is the result's rounding).  What it took: two score
// buffers (205 us with one and tiles of 128), a thread that the compiler knows to be alone issuing the products (194 -> 188), and three
// warps asking for boxes instead of one (188 -> 151: a warp asks for a box of 2 KB every 60 cycles or so).  A token's keys of all heads
// are read from L2 for every 32 tokens and kv head, 0.6 GB in all, 4 GB/ms an SM; the products alone are 93 us.
// The sink is where a row's maximum and the first group's sum start.
// Warps: eight softmax (which first make the long queries), three loaders (TMA boxes, 16-byte copies for the page that the context ends
// in), one issuer.  One CTA an SM.  Every mbarrier wait is bounded; if one runs out the kernel raises bit 4 of the error flag and winds
// down.
#include "tcgen05.cuh"

using namespace kvf;
using namespace kvf::tc;

namespace {

constexpr int BM = 128;  // rows
constexpr int SOFTMAX_THREADS = 2 * BM, MMA_WARP = 8, LOADER_WARP = 9, LOADERS = 3, THREADS = 384;
constexpr int MAX_BLOCKS = 8, RING = 6;       // blocks of 64 numbers of a token's keys; key blocks in flight
constexpr uint32_t Q_BLOCK = BM * 128;        // bytes of a [128 rows][64] block
template <int D> struct Shape {
  static constexpr int BN = D == 64 ? 96 : 64, HALF = BN / 2;  // keys a tile, keys a softmax group takes of it
  static constexpr int DVB = D / 64;                           // blocks of a head's values
  static constexpr uint32_t BLOCK = BN * 128;                  // bytes of a [BN keys][64] block
  static size_t smem(int kb) { return (size_t)kb * Q_BLOCK + (size_t)(RING + 2 * DVB) * BLOCK + 4 * BM * 4 + 192; }
};
constexpr uint32_t COL_Q = 0, COL_O = 256;  // the scores' two buffers lie behind O

struct TalkTcParams {
  const bf16* q;
  bf16* out;
  const bf16* kcache;
  const bf16* vcache;
  const int* block_tables;
  const int* qsl;
  const int* ctx_lens;
  const float* talk;  // [nh][nh] (target head, source head)
  const float* sink;  // [nh] or null
  const int* work;    // n_work pairs (sequence or -1, first query of the tile), or null: the grid's y and z say which
  int* err;
  int num_seqs;
  int q_stride, out_stride, bt_stride;
  int nh, nkv, gs, d, tq;
  int block_size, bs_shift, box_rows, total_rows;
  int window;
  int kb;   // blocks of 64 numbers of all kv heads' keys
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
// two floats' first bfloat16 term; what is left of them stays
__device__ __forceinline__ uint32_t take(float& a, float& b) {
  const uint32_t w = pk(a, b);
  a -= __uint_as_float(w << 16);
  b -= __uint_as_float(w & 0xffff0000u);
  return w;
}

// The maximum of N raw scores, of those from `first` to `last` with MASK.
template <bool MASK, int N>
__device__ __forceinline__ float row_max(const uint32_t (&v)[N], int first, int last) {
  float mx = -INFINITY;
#pragma unroll
  for (int j = 0; j < N; j += 2) {
    const float a = (!MASK || (j >= first && j <= last)) ? __uint_as_float(v[j]) : -INFINITY;
    const float b = (!MASK || (j + 1 >= first && j + 1 <= last)) ? __uint_as_float(v[j + 1]) : -INFINITY;
    mx = fmaxf(mx, fmaxf(a, b));
  }
  return mx;
}
// exp2(score * scale - m_ref) of N scores as bfloat16 pairs: the rounded weights in `hi`, the rounded rests in the first half of `v`;
// returns their sum.
template <bool MASK, int N>
__device__ __forceinline__ float weights(uint32_t (&v)[N], uint32_t (&hi)[N / 2], float m_use, float scale_log2, int first, int last) {
  const uint64_t scale2 = pack2(scale_log2, scale_log2), neg_m2 = pack2(-m_use, -m_use);
  uint64_t sum = pack2(0.f, 0.f);
#pragma unroll
  for (int c = 0; c < N; c += 2) {
    float x0, x1;
    unpack2(fma2(pack2(__uint_as_float(v[c]), __uint_as_float(v[c + 1])), scale2, neg_m2), x0, x1);
    float e0 = ex2(x0), e1 = ex2(x1);
    if (MASK) {
      if (c < first || c > last) e0 = 0.f;
      if (c + 1 < first || c + 1 > last) e1 = 0.f;
    }
    sum = add2(sum, pack2(e0, e1));
    hi[c >> 1] = take(e0, e1);
    v[c >> 1] = pk(e0, e1);
  }
  float s0, s1;
  unpack2(sum, s0, s1);
  return s0 + s1;
}
__device__ __forceinline__ void ld16(uint32_t at, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                 "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(at)
               : "memory");
}
__device__ __forceinline__ void wait16(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                 "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :
               : "memory");
}
__device__ __forceinline__ void st8(uint32_t at, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(at), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]),
               "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void st16(uint32_t at, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(at),
               "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
               "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
               : "memory");
}

template <int D>
__global__ void __launch_bounds__(THREADS, 1)
talking_tcgen05_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const TalkTcParams p) {
  constexpr int BN = Shape<D>::BN, HALF = Shape<D>::HALF, DVB = Shape<D>::DVB;
  constexpr uint32_t BLOCK = Shape<D>::BLOCK, COL_S = COL_O + D;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const uint32_t base = sm32(smem_raw);
  const uint32_t q_s = base;                                // [kb] blocks of [128 rows][64]: the long queries' low terms
  const uint32_t k_s = q_s + (uint32_t)p.kb * Q_BLOCK;      // [RING] blocks of [BN keys][64]
  const uint32_t v_s = k_s + RING * BLOCK;                  // two tiles of values
  const uint32_t xch = v_s + 2 * DVB * BLOCK;               // [2][2][128] floats: the halves' maxima, of even and odd tiles
  const uint32_t bars = xch + 4 * BM * 4;
  const uint32_t q_full = bars, kf0 = bars + 8, ke0 = kf0 + 8 * RING, vf0 = ke0 + 8 * RING, ve0 = vf0 + 16, s_full0 = ve0 + 16, p_full0 = s_full0 + 16,
                 pv_done = p_full0 + 16, drained = pv_done + 8, tmem_slot = drained + 8;
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - base));

  pdl_launch();
  if (base & 1023u) {  // as declared, else refuse rather than compute garbage
    if (threadIdx.x == 0 && p.err) atomicOr(p.err, 8);
    pdl_wait();
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kvh = blockIdx.x;
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
    for (int s = 0; s < RING; ++s) {
      bar_init(kf0 + 8 * s, 1);
      bar_init(ke0 + 8 * s, 1);
    }
    for (int s = 0; s < 2; ++s) {
      bar_init(vf0 + 8 * s, 1);
      bar_init(ve0 + 8 * s, 1);
      bar_init(s_full0 + 8 * s, 1);
      bar_init(p_full0 + 8 * s, SOFTMAX_THREADS);
    }
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

  if (live && warp >= LOADER_WARP) {
    // ---- loaders: every third block of keys each, the last the values too
    const int mine = warp - LOADER_WARP;
    const bool has_values = mine == LOADERS - 1;
    const int* bt = p.block_tables + (size_t)b * p.bt_stride;
    const int boxes = BN / p.box_rows;
    bool ok = true;
    int k_last = -1, v_last = -1;  // the last block of keys, tile of values asked for
    for (int t = 0; t < n_tiles && ok; ++t) {
      const int t0 = kv_lo + t * BN;
      // lane j looks up box j (box_rows keys of one page)
      const int key0 = t0 + p.box_rows * lane;
      int blk = -1, off = 0;
      if (lane < boxes && key0 < ctx) {
        if (p.bs_shift >= 0) {
          blk = bt[key0 >> p.bs_shift];
          off = key0 & (p.block_size - 1);
        } else {
          blk = bt[key0 / p.block_size];
          off = key0 % p.block_size;
        }
      }
      // a tile that ends inside a page, whose other keys must not be read: that page's box comes key by key, with zeros past the context
      const bool ragged = t0 + BN > ctx && (ctx & (p.box_rows - 1)) != 0;
      const int cut = ragged ? (ctx - t0) / p.box_rows : -1;
      const int cut_blk = __shfl_sync(0xffffffffu, blk, ragged ? cut : 0), cut_off = __shfl_sync(0xffffffffu, off, ragged ? cut : 0);
      const int cut_keys = ragged && cut_blk >= 0 ? ctx - t0 - cut * p.box_rows : 0;
      auto announce = [&](uint32_t bar, uint32_t bytes) {
        if (!ragged && lane == 0) bar_expect_tx(bar, bytes);
        __syncwarp();
      };
      auto block = [&](uint32_t dst, const CUtensorMap* map, const bf16* cache, int head, int half, uint32_t bar) {
        const int row = blk >= 0 ? (blk * p.nkv + head) * p.block_size + off : p.total_rows;  // past the end: zeros
        if (ragged) {
          if (lane == 0) bar_more_tx(bar, (uint32_t)((boxes - 1) * p.box_rows) * 128u);
          __syncwarp();
        }
        if (lane < boxes && lane != cut) tma_load_2d(dst + (uint32_t)(lane * p.box_rows) * 128u, map, 64 * half, row, bar);
        if (ragged) {
          const bf16* const src = cache + (((size_t)(cut_blk >= 0 ? cut_blk : 0) * p.nkv + head) * p.block_size + cut_off) * p.d + 64 * half;
          for (int i = lane; i < p.box_rows * 8; i += 32) {
            const int key = i >> 3, c = i & 7;
            const bool in = key < cut_keys;
            cpa16(dst + sw128(cut * p.box_rows + key, c), in ? src + (size_t)key * p.d + c * 8 : cache, in);
          }
          cpa_commit();
          cpa_wait<0>();
          fence_async_smem();
          __syncwarp();
        }
      };
      auto hand_over = [&](uint32_t bar) {
        if (ragged && lane == 0) bar_arrive(bar);
      };
      auto values = [&]() {
        const int s = t & 1;
        if (t >= 2) ok = __all_sync(0xffffffffu, bar_wait(ve0 + 8 * s, ((t >> 1) - 1) & 1, p.err));
        if (!ok) return;
        announce(vf0 + 8 * s, (uint32_t)DVB * BLOCK);
        for (int hf = 0; hf < DVB; ++hf) block(v_s + (uint32_t)(s * DVB + hf) * BLOCK, &map_v, p.vcache, kvh, hf, vf0 + 8 * s);
        hand_over(vf0 + 8 * s);
        v_last = t;
      };
      int asked = 0;  // of this tile's blocks
      for (int i = 0; i < p.kb && ok; ++i) {
        const int g = t * p.kb + i, s = g % RING;
        if (g % LOADERS != mine) continue;
        if (g >= RING) ok = __all_sync(0xffffffffu, bar_wait(ke0 + 8 * s, ((g / RING) - 1) & 1, p.err));
        if (!ok) break;
        announce(kf0 + 8 * s, BLOCK);
        block(k_s + (uint32_t)s * BLOCK, &map_k, p.kcache, i / DVB, i % DVB, kf0 + 8 * s);
        hand_over(kf0 + 8 * s);
        k_last = g;
        if (has_values && ++asked == RING / LOADERS) values();  // behind the blocks that find the ring free
      }
      if (ok && has_values && v_last < t) values();
    }
    // no copy outlives the CTA, whatever made the others leave
    for (int g = k_last; g >= 0 && g > k_last - RING; g -= LOADERS) bar_wait(kf0 + 8 * (g % RING), (g / RING) & 1, p.err);
    for (int i = v_last; i >= 0 && i > v_last - 2; --i) bar_wait(vf0 + 8 * (i & 1), (i >> 1) & 1, p.err);
  } else if (live && warp == MMA_WARP) {
    if (elect_one()) {
      constexpr uint32_t id_s = idesc(BN, 0), id_o = idesc(D, 1);
      const uint64_t q_d = sdesc(q_s), k_d = sdesc(k_s), v_d = sdesc_mn(v_s, BLOCK);
      const uint32_t o_t = tmem + COL_O;
      int i = 0;
      auto scores = [&](int t) {
        const uint32_t s_t = tmem + COL_S + (uint32_t)((t & 1) * BN);
        for (int kb = 0; kb < p.kb; ++kb, ++i) {
          const int s = i % RING;
          if (!bar_wait(kf0 + 8 * s, (i / RING) & 1, p.err)) return false;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t kd = k_d + (uint64_t)((uint32_t)s * (BLOCK >> 4)), qd = q_d + (uint64_t)((uint32_t)kb * (Q_BLOCK >> 4));
          const uint32_t qt = tmem + COL_Q + 32u * kb;
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) umma(s_t, qd + 2 * kk, kd + 2 * kk, id_s, (kb > 0 || kk > 0) ? 1u : 0u);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) umma_ts(s_t, qt + 8u * kk, kd + 2 * kk, id_s, 1u);
          umma_commit(ke0 + 8 * s);
        }
        umma_commit(s_full0 + 8 * (t & 1));
        return true;
      };
      bool ok = bar_wait(q_full, 0, p.err);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (ok) ok = scores(0);
      for (int t = 0; t < n_tiles && ok; ++t) {
        if (t + 1 < n_tiles) {
          if (t > 0) ok = bar_wait(pv_done, (t - 1) & 1, p.err);  // S(t+1) goes where P(t-1) lies
          if (ok) ok = scores(t + 1);
        }
        const int v = t & 1;
        if (ok) ok = bar_wait(vf0 + 8 * v, (t >> 1) & 1, p.err) && bar_wait(p_full0 + 8 * v, (t >> 1) & 1, p.err);  // P(t) is there, O has been rescaled
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // only the keys that some row of the CTA may see: a weight of zero times a value that is no number is none
        const int key0 = kv_lo + t * BN, kk_lo = max(0, seen_lo - key0) / 16, kk_hi = min(BN, kv_hi - key0 + 15) / 16;
        const uint64_t vd = v_d + (uint64_t)((uint32_t)(v * DVB) * (BLOCK >> 4));
        const uint32_t p_t = tmem + COL_S + (uint32_t)(v * BN);
#pragma unroll
        for (int kk = 0; kk < BN / 16; ++kk)
          if (kk >= kk_lo && kk < kk_hi) {
            umma_ts(o_t, p_t + BN / 2 + 8u * kk, vd + (uint64_t)(kk * (16 * 128 >> 4)), id_o, (t > 0 || kk > kk_lo) ? 1u : 0u);
            umma_ts(o_t, p_t + 8u * kk, vd + (uint64_t)(kk * (16 * 128 >> 4)), id_o, 1u);
          }
        umma_commit(pv_done);
        umma_commit(ve0 + 8 * v);
      }
      if (!ok) {  // no product outlives the tensor memory
        umma_commit(drained);
        bar_wait(drained, 0, p.err);
      }
    }
  } else if (live && warp < MMA_WARP) {
    // ---- softmax and output: thread r of either group owns row r, group 0 the first half of a tile's keys, group 1 the others
    const int grp = warp >> 2, r = threadIdx.x & (BM - 1);
    const int tok = r / p.gs, hh = r - tok * p.gs, head = kvh * p.gs + hh;
    const bool valid = tok < n_tok;
    const int pos = valid ? p_first + tok : -1;
    const int lo = first_key(pos, p.window);
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t my_s0 = tmem + lane_addr + COL_S, my_o = tmem + lane_addr + COL_O;
    float* const mine = reinterpret_cast<float*>(smem_raw + (xch - base)) + grp * BM + r;
    const float* const theirs = reinterpret_cast<const float*>(smem_raw + (xch - base)) + (grp ^ 1) * BM + r;
    {
      // the long queries: either group makes every other block of 64 numbers of all rows
      const bf16* const q = p.q + (size_t)(q_begin + q0 + (valid ? tok : 0)) * p.q_stride;
      const float* const talk = p.talk + (size_t)(valid ? head : 0) * p.nh;
      for (int kb = grp; kb < p.kb; kb += 2) {
        const int c = kb / DVB, half = kb - c * DVB;
        uint64_t acc[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) acc[j] = 0ull;
        for (int g = 0; g < p.gs; ++g) {
          const float w = valid ? __ldg(talk + c * p.gs + g) : 0.f;
          const uint64_t w2 = pack2(w, w);
          const uint4* const src = reinterpret_cast<const uint4*>(q + (size_t)(c * p.gs + g) * D + 64 * half);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint4 u = valid ? src[i] : make_uint4(0u, 0u, 0u, 0u);
            const uint32_t x[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[4 * i + e] = fma2(pack2(__uint_as_float(x[e] << 16), __uint_as_float(x[e] & 0xffff0000u)), w2, acc[4 * i + e]);
          }
        }
        uint32_t hi[32];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          uint32_t rest[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            float x, y;
            unpack2(acc[4 * i + e], x, y);
            hi[4 * i + e] = take(x, y);
            rest[e] = pk(x, y);
          }
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(q_s + (uint32_t)kb * Q_BLOCK + sw128(r, i)), "r"(rest[0]), "r"(rest[1]), "r"(rest[2]),
                       "r"(rest[3])
                       : "memory");
        }
        tmem_st32(tmem + lane_addr + COL_Q + 32u * kb, hi);
      }
      tmem_wait_st();
      fence_async_smem();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      bar_arrive(q_full);
    }
    float m_ref = -INFINITY, l = 0.f;
    if (p.sink && valid) {
      m_ref = p.sink[head] * 1.4426950408889634f;
      l = grp == 0 ? 1.f : 0.f;
    }
    bool ok = true;
    int t = 0;
    for (; t < n_tiles; ++t) {
      const int key0 = kv_lo + t * BN + grp * HALF;
      // (tcgen05.ld and st are warp-wide: the lanes of a warp leave the loop together)
      ok = __all_sync(0xffffffffu, bar_wait(s_full0 + 8 * (t & 1), (t >> 1) & 1, p.err));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t my_s = my_s0 + (uint32_t)((t & 1) * BN);
      uint32_t va[32], vb[16];
      tmem_ld32(my_s + (uint32_t)(grp * HALF), va);
      if (HALF > 32) ld16(my_s + (uint32_t)(grp * HALF) + 32u, vb);
      tmem_wait(va);
      if (HALF > 32) wait16(vb);
      const bool mask = __any_sync(0xffffffffu, (key0 + HALF - 1 > pos) || (key0 < lo));
      const int first = max(lo, key0) - key0, last = min(pos, key0 + HALF - 1) - key0;
      float mx = mask ? row_max<true, 32>(va, first, last) : row_max<false, 32>(va, 0, 31);
      if (HALF > 32) mx = fmaxf(mx, mask ? row_max<true, 16>(vb, first - 32, last - 32) : row_max<false, 16>(vb, 0, 15));
      mine[(t & 1) * 2 * BM] = mx;
      // both halves of every row are in registers: their maxima can be exchanged, and P may take the place of S
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      asm volatile("bar.sync 1, %0;" ::"n"(SOFTMAX_THREADS) : "memory");
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      mx = fmaxf(mx, theirs[(t & 1) * 2 * BM]) * p.scale_log2;  // scale > 0
      float corr = 1.f;
      if (mx > m_ref) {  // followed exactly, as on the mma.sync kernel
        corr = ex2(m_ref - mx);  // 0 the first time without a sink
        m_ref = mx;
      }
      const float m_use = (m_ref == -INFINITY) ? 0.f : m_ref;
      // half of the weights: HALF / 2 columns of first terms, as many of rests BN / 2 columns on
      const uint32_t my_p = my_s + (uint32_t)(grp * (HALF / 2));
      uint32_t hi[16], hi8[8];
      float sum = mask ? weights<true, 32>(va, hi, m_use, p.scale_log2, first, last) : weights<false, 32>(va, hi, m_use, p.scale_log2, 0, 31);
      st16(my_p, hi);
      st16(my_p + BN / 2, va);
      if (HALF > 32) {
        sum += mask ? weights<true, 16>(vb, hi8, m_use, p.scale_log2, first - 32, last - 32) : weights<false, 16>(vb, hi8, m_use, p.scale_log2, 0, 15);
        st8(my_p + 16u, hi8);
        st8(my_p + BN / 2 + 16u, vb);
      }
      l = l * corr + sum;
      // once P V of the tile before is over either group rescales half of O
      if (t > 0) {
        ok = __all_sync(0xffffffffu, bar_wait(pv_done, (t - 1) & 1, p.err));
        if (ok && __any_sync(0xffffffffu, corr != 1.f)) {
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          for (int c0 = 32 * grp; c0 < D; c0 += 64) {
            uint32_t v[32];
            tmem_ld32(my_o + (uint32_t)c0, v);
            tmem_wait(v);
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * corr);
            tmem_st32(my_o + (uint32_t)c0, v);
          }
        }
      }
      tmem_wait_st();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      if (!ok) {
        ++t;
        break;
      }
      bar_arrive(p_full0 + 8 * (t & 1));
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
      const float inv = l > 0.f ? 1.f / l : (l == l ? 0.f : l);  // a sum that is no number shows in the result
      bf16* dst = p.out + (size_t)(q_begin + q0 + (valid ? tok : 0)) * p.out_stride + (size_t)head * D;
      for (int c0 = 32 * grp; c0 < D; c0 += 64) {
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

template <int D>
int launch_talking(const CUtensorMap& mk, const CUtensorMap& mv, const TalkTcParams& p, int B, int tiles, int n_work, cudaStream_t st) {
  const size_t smem = Shape<D>::smem(p.kb);
  const cudaError_t e = cudaFuncSetAttribute(talking_tcgen05_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  return launch(talking_tcgen05_kernel<D>, dim3(p.nkv, p.work ? n_work : B, p.work ? 1 : tiles), dim3(THREADS), smem, st, mk, mv, p);
}

}  // namespace

// Shapes this kernel does not take are refused with cudaErrorInvalidValue.
KVF_API int kvf_talking_attention_tcgen05_bf16(const void* q, void* out, const void* kcache, const void* vcache, const int* block_tables,
                                               const int* qsl, const int* ctx_lens, const float* talk, const float* sink, int B, int max_q_len,
                                               int q_stride, int out_stride, int bt_stride, int nh, int nkv, int d, int block_size,
                                               long long num_blocks, float scale, int window, const int* work, int n_work, int* err,
                                               cudaStream_t st) {
  if (B <= 0 || max_q_len <= 0) return 0;
  if ((d != 64 && d != 128) || nkv <= 0 || nkv * d > 64 * MAX_BLOCKS || nh % nkv || nh / nkv > BM || !talk) return (int)cudaErrorInvalidValue;
  if (block_size <= 0 || (block_size % 16) || num_blocks <= 0 || window < 0 || !(scale > 0.f)) return (int)cudaErrorInvalidValue;
  if ((q_stride & 7) || (out_stride & 7) || ((((uintptr_t)q) | ((uintptr_t)out) | ((uintptr_t)kcache) | ((uintptr_t)vcache)) & 15)) return (int)cudaErrorInvalidValue;
  const long long rows = num_blocks * nkv * block_size;
  if (rows >= (1ll << 31) - 64) return (int)cudaErrorInvalidValue;
  TalkTcParams p;
  p.q = (const bf16*)q; p.out = (bf16*)out; p.kcache = (const bf16*)kcache; p.vcache = (const bf16*)vcache;
  p.block_tables = block_tables; p.qsl = qsl; p.ctx_lens = ctx_lens; p.talk = talk; p.sink = sink; p.work = work; p.err = err;
  p.num_seqs = B;
  p.q_stride = q_stride; p.out_stride = out_stride; p.bt_stride = bt_stride;
  p.nh = nh; p.nkv = nkv; p.gs = nh / nkv; p.d = d; p.tq = BM / p.gs;
  p.block_size = block_size;
  p.bs_shift = -1;
  for (int sh = 0; sh < 31; ++sh)
    if ((1 << sh) == block_size) p.bs_shift = sh;
  p.box_rows = d == 128 && block_size % 64 == 0 ? 64 : block_size % 32 == 0 ? 32 : 16;  // divides a tile
  p.total_rows = (int)rows;
  p.window = window;
  p.kb = nkv * d / 64;
  p.scale_log2 = scale * 1.4426950408889634f;
  const int tiles = (max_q_len + p.tq - 1) / p.tq;
  if (work ? (n_work <= 0 || n_work > 65535) : (B > 65535 || tiles > 65535)) return (int)cudaErrorInvalidValue;
  CUtensorMap mk, mv;
  memset(&mk, 0, sizeof(mk));
  memset(&mv, 0, sizeof(mv));
  int rc = cache_map(&mk, kcache, rows, d, p.box_rows);
  if (!rc) rc = cache_map(&mv, vcache, rows, d, p.box_rows);
  if (rc) return rc;
  return d == 64 ? launch_talking<64>(mk, mv, p, B, tiles, n_work, st) : launch_talking<128>(mk, mv, p, B, tiles, n_work, st);
}
