// gl_dice.cuh -- the load of one complex point in the forward column passes (FP64 and
// integer form): dice the previous products into balanced digits and carries, add the
// carry of the word below.
#pragma once
#include "gl_device.cuh"
#include "gl_internal.h"

namespace gl {

// The words j0, j0+1 from the products P[k] of the words j0+1-k, k = 0 .. NC+2, and the
// flags of the words j0-1, j0, j0+1: their digits plus the carry of the word below.
template <int NC>
__device__ __forceinline__ void dice_pair(const long long* P, int LO, uint32_t fm, uint32_t f0, uint32_t f1, int* v0,
                                          int* v1) {
  int dm, hm, d0, h0, d1, h1;
  if (NC <= 3) {
    // words of 16 bits or more: in 32-bit arithmetic, from sign and magnitude of each
    // product taken once
    uint32_t lo[NC + 3], hi[NC + 3], sg[NC + 3];
#pragma unroll
    for (int k = 0; k < NC + 3; ++k) {
      const unsigned long long g = (unsigned long long)(P[k] >> 63);
      const unsigned long long m = ((unsigned long long)P[k] ^ g) - g;
      lo[k] = (uint32_t)m;
      hi[k] = (uint32_t)(m >> 32);
      sg[k] = (uint32_t)g;
    }
    auto dice_at = [&](uint32_t f, int off) {
      const uint32_t mask = (1u << (LO + (int)(f & 1))) - 1;
      uint32_t sum = ((lo[off] & mask) ^ sg[off]) - sg[off];
      int shift = 0;
#pragma unroll
      for (int i = 1; i <= NC; ++i) {
        shift += LO + (int)((f >> i) & 1);
        const int k = off + i;  // shift < 32 for i = 1, >= 32 beyond
        const uint32_t w = (i == 1 ? __funnelshift_r(lo[k], hi[k], shift) : hi[k] >> (shift - 32)) & mask;
        sum += (w ^ sg[k]) - sg[k];
      }
      return (int)sum;
    };
    balanced_split32(dice_at(fm, 2), LO + (int)(fm & 1), &dm, &hm);
    balanced_split32(dice_at(f0, 1), LO + (int)(f0 & 1), &d0, &h0);
    balanced_split32(dice_at(f1, 0), LO + (int)(f1 & 1), &d1, &h1);
  } else {
    auto dice_at = [&](uint32_t f, int off) {
      const long long mask = (1ll << (LO + (int)(f & 1))) - 1;
      const long long v = P[off];
      long long sum = v < 0 ? -((-v) & mask) : (v & mask);
      int shift = 0;
#pragma unroll
      for (int i = 1; i <= NC; ++i) {
        shift += LO + (int)((f >> i) & 1);
        const long long w = P[off + i];
        sum += shift >= 63 ? 0 : (w < 0 ? -(((-w) >> shift) & mask) : ((w >> shift) & mask));
      }
      return sum;
    };
    balanced_split(dice_at(fm, 2), LO + (int)(fm & 1), &dm, &hm);
    balanced_split(dice_at(f0, 1), LO + (int)(f0 & 1), &d0, &h0);
    balanced_split(dice_at(f1, 0), LO + (int)(f1 & 1), &d1, &h1);
  }
  *v0 = d0 + hm;
  *v1 = d1 + h0;
}

// Words j0 = 2m, j0+1 of point m = m1 + W m2 as (v0, v1): from the carry-save state, or by
// dicing the products with carry depth NC (llintToIrrBal<n>).  The digit sums of j0-1, j0,
// j0+1 need the products of words j0-1-NC .. j0+1: P[k] = product of word j0+1-k,
// k = 0 .. NC+2.  Words j0+1-2d and j0-2d are the two words of point m-d, column m1-d of
// the same row (the previous row, from the last columns, when m1 < d), adjacent in the
// column-major layout: one 16-byte load per point, and no division to find it.
// EARLY: the kernel may become resident while the pass that writes the products still runs
// (a programmatic dependent), so they are read with ordinary loads; the non-coherent path
// is for memory that nothing writes during the kernel's whole life.
template <bool EARLY, typename T>
__device__ __forceinline__ T load_product(const T* p) {
  if constexpr (EARLY) return *p;
  else return __ldg(p);
}
template <bool FROM_STATE, int NC, bool EARLY = false>
__device__ __forceinline__ void load_point(const IterArgs& a, const int m1, const int m2, int* v0, int* v1) {
  const int H = a.H, W = a.W, N = a.N, LO = a.LO;
  constexpr int D = (NC + 2) / 2;  // points m-1 .. m-D hold the words j0-1 .. j0+1-(NC+2)
  const int s0 = 2 * (m1 * H + m2);
  if (FROM_STATE) {
    const int j0 = 2 * (m1 + W * m2);
    *v0 = a.digit[j0] + (int)a.hi[j0 == 0 ? N - 1 : j0 - 1];
    *v1 = a.digit[j0 + 1] + (int)a.hi[j0];
  } else {
    long long P[NC + 3];
    const longlong2 own = load_product<EARLY>(reinterpret_cast<const longlong2*>(a.ll + s0));
    P[0] = own.y;
    P[1] = own.x;
    uint32_t fm = 0;  // flags of word j0-1 (the upper word of point m-1)
#pragma unroll
    for (int d = 1; d <= D; ++d) {
      int c = m1 - d, r = m2;
      if (c < 0) {  // one wrap suffices: layouts have W >= 4 >= D
        c += W;
        r = r == 0 ? H - 1 : r - 1;
      }
      const int sd = 2 * (c * H + r);
      if (d == 1) fm = __ldg(a.flags + sd + 1);
      if (2 * d + 1 < NC + 3) {
        const longlong2 v = load_product<EARLY>(reinterpret_cast<const longlong2*>(a.ll + sd));
        P[2 * d] = v.y;
        P[2 * d + 1] = v.x;
      } else {  // only the upper word of the farthest point
        P[2 * d] = load_product<EARLY, long long>(a.ll + sd + 1);
      }
    }
    const uchar2 ff = __ldg(reinterpret_cast<const uchar2*>(a.flags + s0));
    const uint32_t f0 = ff.x, f1 = ff.y;
    dice_pair<NC>(P, LO, fm, f0, f1, v0, v1);
  }
}

}  // namespace gl
