// Heads of a bfloat16 row, eight numbers a thread: what the kernels that norm and turn the heads of many tokens share.  A head of d numbers
// (d / 8 a power of two up to 32) is d / 8 neighbouring lanes' 16-byte words.
#pragma once
#include <initializer_list>

#include "common.cuh"

namespace kvf {

constexpr int HEAD_VEC_THREADS = 128;
// Steps of fewer tokens stay with a warp a head: a CTA a token leaves too few warps in flight there.  A warp a head and this form, us:
//   rotation and head norm (qk_prepare)  32 query heads on 8 of 64: 128 tokens 4.0 and 4.6, 192 5.6 and 4.7, 256 6.3 and 4.7, 2,048 33 and 11
//                                        24 on 8 of 128: 128 4.6 and 5.4, 192 5.5 and 5.7, 256 7.3 and 5.7, 2,048 35 and 15
//   head norm with rotation and cache write  32 on 8 of 64: 128 3.9 and 5.0, 256 5.8 and 5.2, 384 7.1 and 5.4, 2,048 21 and 12
//                                        24 on 8 of 128: 128 4.0 and 6.0, 256 5.9 and 6.4, 384 7.8 and 7.0, 2,048 22 and 18
//                                        8 on 2 of 128: 256 3.7 and 4.4, 384 4.5 and 4.6, 512 4.8 and 4.9, 1,024 7.8 and 5.8
constexpr int HEAD_VEC_PREPARE = 256, HEAD_VEC_NORM = 384;

__device__ __forceinline__ void store8(bf16* p, const float (&f)[8]) {
  uint4 u;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  *reinterpret_cast<uint4*>(p) = u;
}
// The sum over a head's `lanes` lanes; every lane of the warp takes part.
__device__ __forceinline__ float head_sum(float v, int lanes) {
  for (int o = 1; o < lanes; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// Turns the first 2 * half numbers of a head, of which the thread holds word `w` of eight, by the cosines turn[0 .. half) and sines
// turn[half .. 2 half): split pairs (i, i + half), half / 8 a power of two, or neighbouring ones.  Every lane takes part.
__device__ __forceinline__ void turn_head(float (&x)[8], int w, int half, bool split, const float* turn) {
  if (half == 0) return;
  if (split) {
    const int words = half >> 3;
    const bool turns = w < 2 * words, second = (w & words) != 0;
    const int at = turns ? 8 * (w & (words - 1)) : 0;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float other = __shfl_xor_sync(0xffffffffu, x[e], words);
      const float cs = turn[at + e], sn = turn[half + at + e];
      float y1, y2;
      rotate_pair(second ? other : x[e], second ? x[e] : other, cs, sn, y1, y2);
      if (turns) x[e] = second ? y2 : y1;
    }
  } else {
#pragma unroll
    for (int e = 0; e < 8; e += 2) {
      const int i = 4 * w + (e >> 1);
      if (i < half) {
        float y1, y2;
        rotate_pair(x[e], x[e + 1], turn[i], turn[half + i], y1, y2);
        x[e] = y1;
        x[e + 1] = y2;
      }
    }
  }
}
// Whether heads of d numbers whose first `rot` turn come in such words.
inline bool head_vec_ok(int d, int rot, bool split) {
  const int lanes = d / 8, words = rot / 16;
  if (d % 8 || lanes < 1 || lanes > 32 || (lanes & (lanes - 1))) return false;
  return rot == 0 || !split || (rot % 16 == 0 && (words & (words - 1)) == 0);
}
inline bool aligned16(std::initializer_list<const void*> ptrs) {
  for (const void* p : ptrs)
    if ((uintptr_t)p & 15) return false;
  return true;
}

}  // namespace kvf
