// True 32-bit matrix product on the FP32 pipes:  C[M,N] = A[M,K] * W[N,K]^T.
//
// No tensor cores and no reduced-precision mode: every product is an FFMA.  Each output
// element is accumulated by one thread over k = 0..K-1 in order, so its value does not
// depend on M, on the tile it falls in or on the rest of the batch.
#include "common.cuh"

namespace {

constexpr int LK = 16, LPAD = 4;

__device__ __forceinline__ uint64_t pair(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma_pair(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// Tiles of BM x BN outputs, TM x TN per thread (as blocks of 4 x 4, so that a thread's reads of shared memory are
// whole float4s), the next tile's operands fetched into registers while this one is multiplied, two buffers in
// shared memory.  Two neighbouring columns share a packed multiply-add (each half rounds as fmaf does), which halves
// the instructions beside the reads of shared memory.  An output is one accumulator that walks k = 0..K-1 in order,
// so every tile shape gives the same bits, and so does the kernel of few rows below.
template <int BM, int BN, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), 512 / ((BM / TM) * (BN / TN)))
sgemm_nt_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M,
                int N, int K, int lda, int ldw, int ldc, int vec_ok) {
  constexpr int TX = BN / TN, THREADS = (BM / TM) * TX;
  constexpr int MB = TM / 4, NB = TN / 4;        // blocks of four rows, of four columns a thread
  constexpr int ROWS = THREADS / 4;              // rows a pass of the loader covers: four quads of k a row
  constexpr int PA = BM / ROWS, PW = BN / ROWS;  // its passes over A and over W
  static_assert(BM % ROWS == 0 && BN % ROWS == 0, "whole passes");
  __shared__ __align__(16) float As[2][LK][BM + LPAD];
  __shared__ __align__(16) float Ws[2][LK][BN + LPAD];
  const int t = threadIdx.x;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  // a warp's lanes lie 4 x 8 in the tile: the fewest distinct words of shared memory a read asks for
  const int warp = t >> 5, lane = t & 31;
  const int tx = (warp % (TX / 8)) * 8 + (lane & 7), ty = (warp / (TX / 8)) * 4 + (lane >> 3);
  const int lrow = t >> 2, lk = (t & 3) * 4;
  uint64_t acc[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) acc[i][j] = pair(0.f, 0.f);
  float ra[PA][4], rw[PW][4];
  auto row_quad = [&](float (&r)[4], const float* base, int row, int rows, int ld, int k) {
#pragma unroll
    for (int i = 0; i < 4; ++i) r[i] = 0.f;
    if (row >= rows) return;
    const float* p = base + (size_t)row * ld + k;
    if (vec_ok && k + 3 < K) {
      const float4 v = *reinterpret_cast<const float4*>(p);
      r[0] = v.x; r[1] = v.y; r[2] = v.z; r[3] = v.w;
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (k + i < K) r[i] = p[i];
    }
  };
  auto fetch = [&](int k0) {
#pragma unroll
    for (int h = 0; h < PA; ++h) row_quad(ra[h], A, m0 + lrow + ROWS * h, M, lda, k0 + lk);
#pragma unroll
    for (int h = 0; h < PW; ++h) row_quad(rw[h], W, n0 + lrow + ROWS * h, N, ldw, k0 + lk);
  };
  auto stash = [&](int buf) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int h = 0; h < PA; ++h) As[buf][lk + i][lrow + ROWS * h] = ra[h][i];
#pragma unroll
      for (int h = 0; h < PW; ++h) Ws[buf][lk + i][lrow + ROWS * h] = rw[h][i];
    }
  };
  fetch(0);
  stash(0);
  __syncthreads();
  int buf = 0;
  for (int k0 = 0; k0 < K; k0 += LK) {
    const bool more = k0 + LK < K;
    if (more) fetch(k0 + LK);  // on its way while this tile is multiplied
#pragma unroll
    for (int k = 0; k < LK; ++k) {
      float ar[TM];
      uint64_t wr[TN / 2];
#pragma unroll
      for (int b = 0; b < MB; ++b) {
        const float4 v = *reinterpret_cast<const float4*>(&As[buf][k][b * (BM / MB) + ty * 4]);
        ar[4 * b] = v.x; ar[4 * b + 1] = v.y; ar[4 * b + 2] = v.z; ar[4 * b + 3] = v.w;
      }
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&Ws[buf][k][b * (BN / NB) + tx * 4]);
        wr[2 * b] = v.x; wr[2 * b + 1] = v.y;
      }
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const uint64_t aa = pair(ar[i], ar[i]);
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = fma_pair(aa, wr[j], acc[i][j]);
      }
    }
    if (more) {
      stash(buf ^ 1);  // the other buffer: its last readers passed the barrier below one tile ago
      __syncthreads();
      buf ^= 1;
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + (i >> 2) * (BM / MB) + ty * 4 + (i & 3);
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) {
      const int gn = n0 + (j >> 1) * (BN / NB) + tx * 4 + 2 * (j & 1);
      float lo, hi;
      asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(acc[i][j]));
      if (gn < N) C[(size_t)gm * ldc + gn] = lo;
      if (gn + 1 < N) C[(size_t)gm * ldc + gn + 1] = hi;
    }
  }
}

template <int BM, int BN, int TM, int TN>
int launch_tiles(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int vec_ok, cudaStream_t st) {
  const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  if (grid.y > 65535) return (int)cudaErrorInvalidValue;
  sgemm_nt_kernel<BM, BN, TM, TN><<<grid, (BM / TM) * (BN / TN), 0, st>>>(A, W, C, M, N, K, lda, ldw, ldc, vec_ok);
  return KVF_LAUNCH_STATUS();
}

// Time of the SM with the most tiles, in units of an output of a 128 x 128 tile on a full SM: `cost` is what an output of
// the shape costs beside that, and an SM that holds few warps (four warps a scheduler hide everything, one little) takes longer.
double busiest(int M, int N, int bm, int bn, int warps, int resident, double cost) {
  const long long tiles = (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn), per_sm = (tiles + 147) / 148;
  const long long held = (per_sm < resident ? per_sm : resident) * warps;
  return (double)per_sm * bm * bn * cost * (held <= 4 ? 1.55 : held <= 8 ? 1.16 : held <= 12 ? 1.06 : 1.0);
}

// The same sums for a handful of rows (decoding): with M <= 16 the tiles above are nearly empty and
// a product with a narrow output (N = 2,048: 32 CTAs) leaves most SMs idle.  Here a CTA of 64
// threads takes MR rows of A (8 or 16) and 256 / MR rows of W, four outputs per thread (two rows of
// A by two rows of W); W and A come in through a cp.async pipeline, k contiguous in shared memory,
// and each output is one accumulator that walks k = 0..K-1 in order, exactly as above: the bits are
// the same whichever of the kernels runs.  (Entries past K are filled with zeros and add
// nothing.)  What bounds a warp is its chains of dependent FMAs, so a thread has four of them.
// Needs K % 4 == 0 and 16-byte aligned rows.
constexpr int SBK = 64, SSTAGES = 6, SLD = SBK + 4, STHREADS = 64;

template <int MR>
__global__ void __launch_bounds__(STHREADS)
sgemm_nt_small_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M,
                      int N, int K, int lda, int ldw, int ldc) {
  constexpr int SBN = 256 / MR, HN = SBN / 2, HM = MR / 2;
  constexpr int STAGE = (SBN + MR) * SLD;  // floats: the rows of W, then the rows of A
  extern __shared__ __align__(16) float small_smem[];
  const int t = threadIdx.x;
  const int n0 = blockIdx.x * SBN;
  const int nl = t % HN, mr = t / HN;  // outputs: rows mr and mr + HM, columns n0 + nl and n0 + nl + HN
  const int n_tiles = (K + SBK - 1) / SBK;
  auto load = [&](int stage, int tile) {
    const int k0 = tile * SBK;
    float* ws = small_smem + stage * STAGE;
    float* as = ws + SBN * SLD;
#pragma unroll
    for (int i = t; i < SBN * 16; i += STHREADS) {  // rows of W x 16 chunks of 4 floats
      const int row = i >> 4, c = (i & 15) * 4;
      const bool ok = n0 + row < N && k0 + c < K;
      const float* src = ok ? W + (size_t)(n0 + row) * ldw + k0 + c : W;
      const unsigned dst = (unsigned)__cvta_generic_to_shared(ws + row * SLD + c);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0));
    }
#pragma unroll
    for (int i = t; i < MR * 16; i += STHREADS) {
      const int row = i >> 4, c = (i & 15) * 4;
      const bool ok = row < M && k0 + c < K;
      const float* src = ok ? A + (size_t)row * lda + k0 + c : A;
      const unsigned dst = (unsigned)__cvta_generic_to_shared(as + row * SLD + c);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0));
    }
  };
#pragma unroll
  for (int s = 0; s < SSTAGES - 1; ++s) {
    if (s < n_tiles) load(s, s);
    asm volatile("cp.async.commit_group;" ::);
  }
  float c00 = 0.f, c01 = 0.f, c10 = 0.f, c11 = 0.f;  // c[row][column]
  for (int tile = 0; tile < n_tiles; ++tile) {
    asm volatile("cp.async.wait_group %0;" ::"n"(SSTAGES - 2));
    __syncthreads();  // tile `tile` has landed for every thread; tile - 1 has been consumed
    if (tile + SSTAGES - 1 < n_tiles) load((tile + SSTAGES - 1) % SSTAGES, tile + SSTAGES - 1);
    asm volatile("cp.async.commit_group;" ::);
    const float* ws = small_smem + (tile % SSTAGES) * STAGE;
    const float* a0 = ws + SBN * SLD + mr * SLD;
    const float* a1 = a0 + HM * SLD;
    const float* w0 = ws + nl * SLD;
    const float* w1 = w0 + HN * SLD;
#pragma unroll
    for (int k = 0; k < SBK; k += 4) {
      const float4 p = *reinterpret_cast<const float4*>(a0 + k);
      const float4 q = *reinterpret_cast<const float4*>(a1 + k);
      const float4 u = *reinterpret_cast<const float4*>(w0 + k);
      const float4 v = *reinterpret_cast<const float4*>(w1 + k);
      c00 = fmaf(p.x, u.x, c00); c01 = fmaf(p.x, v.x, c01); c10 = fmaf(q.x, u.x, c10); c11 = fmaf(q.x, v.x, c11);
      c00 = fmaf(p.y, u.y, c00); c01 = fmaf(p.y, v.y, c01); c10 = fmaf(q.y, u.y, c10); c11 = fmaf(q.y, v.y, c11);
      c00 = fmaf(p.z, u.z, c00); c01 = fmaf(p.z, v.z, c01); c10 = fmaf(q.z, u.z, c10); c11 = fmaf(q.z, v.z, c11);
      c00 = fmaf(p.w, u.w, c00); c01 = fmaf(p.w, v.w, c01); c10 = fmaf(q.w, u.w, c10); c11 = fmaf(q.w, v.w, c11);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::);
  const int col0 = n0 + nl, col1 = n0 + nl + HN;
  if (mr < M) {
    if (col0 < N) C[(size_t)mr * ldc + col0] = c00;
    if (col1 < N) C[(size_t)mr * ldc + col1] = c01;
  }
  if (mr + HM < M) {
    if (col0 < N) C[(size_t)(mr + HM) * ldc + col0] = c10;
    if (col1 < N) C[(size_t)(mr + HM) * ldc + col1] = c11;
  }
}

template <int MR>
int launch_small(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, cudaStream_t st) {
  constexpr int SBN = 256 / MR;
  const size_t smem = (size_t)SSTAGES * (SBN + MR) * SLD * sizeof(float);
  cudaError_t e = cudaFuncSetAttribute(sgemm_nt_small_kernel<MR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  sgemm_nt_small_kernel<MR><<<dim3((N + SBN - 1) / SBN), STHREADS, smem, st>>>(A, W, C, M, N, K, lda, ldw, ldc);
  return KVF_LAUNCH_STATUS();
}

}  // namespace

// A: [M,K] row stride lda; W: [N,K] row stride ldw; C: [M,N] row stride ldc; all float.
KVF_API int kvf_gemm_nt_f32(const float* A, const float* W, float* C, int M, int N, int K, int lda,
                            int ldw, int ldc, cudaStream_t st) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return (int)cudaErrorInvalidValue;
  const int vec_ok = ((lda & 3) == 0) && ((ldw & 3) == 0) && ((((uintptr_t)A) & 15) == 0) &&
                     ((((uintptr_t)W) & 15) == 0);
  if (M <= 16 && vec_ok && (K & 3) == 0) {
    if (M <= 8) return launch_small<8>(A, W, C, M, N, K, lda, ldw, ldc, st);
    return launch_small<16>(A, W, C, M, N, K, lda, ldw, ldc, st);
  }
  // Large tiles read shared memory least per output, small ones leave fewer outputs to rows and SMs that have none.  Costs and
  // the factor for few warps were measured (B200; the four shapes in turn, one kernel of 128 x 128 or 64 x 64 tiles before):
  // 515 x 16,384 x 2,048: 907, 788, 871, 1,159 us (1,022 before); 515 x 2,048 x 8,192: 829, 612, 504, 655 us (954);
  // 2,048 x 16,384 x 2,048: 2,530, 2,665, 2,995, 4,258 us (2,855: 48 TFLOP/s, now 54); 48 x 2,048 x 2,048: 201, 152, 82, 62 us (103).
  const double t0 = busiest(M, N, 128, 128, 8, 2, 1.0), t1 = busiest(M, N, 64, 128, 4, 4, 1.08), t2 = busiest(M, N, 64, 64, 4, 4, 1.18),
               t3 = busiest(M, N, 32, 64, 4, 4, 1.68);
  // (a grid's second dimension ends at 65,535: beyond two million rows only the highest tiles remain)
  if (M > 65535 * 32 || (t0 <= t1 && t0 <= t2 && t0 <= t3)) return launch_tiles<128, 128, 8, 8>(A, W, C, M, N, K, lda, ldw, ldc, vec_ok, st);
  if (t1 <= t2 && t1 <= t3) return launch_tiles<64, 128, 8, 8>(A, W, C, M, N, K, lda, ldw, ldc, vec_ok, st);
  if (t2 <= t3) return launch_tiles<64, 64, 8, 4>(A, W, C, M, N, K, lda, ldw, ldc, vec_ok, st);
  return launch_tiles<32, 64, 4, 4>(A, W, C, M, N, K, lda, ldw, ldc, vec_ok, st);
}
