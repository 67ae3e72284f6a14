// gl_int_stage.cuh -- line DFTs of the integer form in shared memory (gl_int_kernels.cu,
// gl_int_resident.cu).
#pragma once
#include "gl_gf61.cuh"
#include "gl_internal.h"

namespace gl {

using gf::g2;

// whether a line plan needs the kernels compiled with radices 5 and 7
inline bool has57(const LinePlan& lp) {
  for (int i = 0; i < lp.nst; ++i)
    if (lp.radix[i] == 5 || lp.radix[i] == 7) return true;
  return false;
}

__device__ __forceinline__ int ipad(int i) { return i + (i >> 3); }

// a stage value from the global table (read-only path) or from a shared-memory copy
template <bool SHARED>
__device__ __forceinline__ int4 slot_at(const int4* p) {
  return SHARED ? *p : __ldg(p);
}

// Stockham DIT stage, out of place, as in the FP64 form: butterfly j of a line reads
// x[j + q L/R], multiplies by w^q and writes x[(j - k) R + k + p Ns], k = j mod Ns.
// The position k needs no division in the first stages (Ns a power of two) or the last
// (Ns = L/R > j).
template <int R, int S, bool SHARED>
__device__ __forceinline__ void int_stage(const g2* __restrict__ src, g2* __restrict__ dst, int nlines, int ls,
                                          int L, int Ns, const int4* __restrict__ tw) {
  const int LR = L / R;
  const int nb = nlines * LR;
  const bool last = Ns == LR, pow2 = (Ns & (Ns - 1)) == 0;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) {
    int l = 0;
    if (nlines == 2) l = b >= LR;
    else if (nlines > 2) l = b / LR;
    const int j = b - l * LR;
    const int k = last ? j : pow2 ? (j & (Ns - 1)) : j % Ns;
    const g2* s = src + l * ls;
    g2 v[R];
    gf::butterfly<R, S>(
        v, Ns > 1, [&](int q) { return s[ipad(j + q * LR)]; }, [&](int i) { return slot_at<SHARED>(tw + (k + i * Ns)); });
    g2* d = dst + l * ls;
    const int base = (j - k) * R + k;
#pragma unroll
    for (int q = 0; q < R; ++q) d[ipad(base + q * Ns)] = v[q];
  }
  __syncthreads();
}

// B57: the plan may have radices 5 and 7 (compiled apart: a kernel's registers are set by
// its largest stage, and without them three CTAs of 256 threads fit an SM).
template <int S, bool B57, bool SHARED = false>
__device__ __forceinline__ g2* int_line_fft(g2* a, g2* b, int nlines, int ls, const LinePlan& lp, const int4* tw) {
  int Ns = 1;
  for (int s = 0; s < lp.nst; ++s) {
    const int4* st = tw + lp.off[s];
    switch (lp.radix[s]) {
      case 8: int_stage<8, S, SHARED>(a, b, nlines, ls, lp.L, Ns, st); break;
      case 4: int_stage<4, S, SHARED>(a, b, nlines, ls, lp.L, Ns, st); break;
      case 2: int_stage<2, S, SHARED>(a, b, nlines, ls, lp.L, Ns, st); break;
      case 3: int_stage<3, S, SHARED>(a, b, nlines, ls, lp.L, Ns, st); break;
      default:
        if constexpr (B57) {
          if (lp.radix[s] == 5) int_stage<5, S, SHARED>(a, b, nlines, ls, lp.L, Ns, st);
          else int_stage<7, S, SHARED>(a, b, nlines, ls, lp.L, Ns, st);
        }
        break;
    }
    Ns *= lp.radix[s];
    g2* t = a;
    a = b;
    b = t;
  }
  return a;
}

// The product's range checks, as round_word of the FP64 form.  Where n + 1 words always
// hold 51 bits (all but words of a few bits), the first check implies the second.
__device__ __forceinline__ long long check_word(long long r, unsigned* fl) {
  const unsigned long long mag = (unsigned long long)(r < 0 ? -r : r);
  if (mag >> 51) {
    *fl |= kStatusBig;
    return 0;
  }
  return r;
}
__device__ __forceinline__ void check_span(long long r, int span, unsigned* fl) {
  const unsigned long long mag = (unsigned long long)(r < 0 ? -r : r);
  if (span < 63 && (mag >> span) != 0ull) *fl |= kStatusSlice;
}

}  // namespace gl
