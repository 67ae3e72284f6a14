// gl_hostcheck.cu -- the device arithmetic helpers (small DFTs, integer-domain
// rounding and conversion, dicing) compiled for the host, so the CPU test suite can
// check them against numpy and the oracle without a GPU.  Not used by the product.
#include <algorithm>
#include <cstdint>

#include "gl_device.cuh"

using namespace gl;

template <int S>
static void run_dft(int R, cplx* x) {
  switch (R) {
    case 2: dft<2, S>(x); break;
    case 3: dft<3, S>(x); break;
    case 4: dft<4, S>(x); break;
    case 5: dft<5, S>(x); break;
    case 7: dft<7, S>(x); break;
    case 8: dft<8, S>(x); break;
    case 16: dft<16, S>(x); break;
    default: break;
  }
}

extern "C" {

// in-place DFT of R interleaved complex doubles; sign -1 forward, +1 inverse
int hc_dft(int R, int sign, double* xy) {
  if (R != 2 && R != 3 && R != 4 && R != 5 && R != 7 && R != 8 && R != 16) return -1;
  cplx* x = reinterpret_cast<cplx*>(xy);
  if (sign < 0) run_dft<-1>(R, x);
  else run_dft<1>(R, x);
  return 0;
}

long long hc_round(double x, unsigned long long* err64, int* big) {
  *big = 0;
  return round_ll_bits(x, err64, big);
}

double hc_dbl_from_int(int v) { return dbl_from_int(v); }

// dice one word j from products ll (cyclic, length N) with flags
struct CyclicProducts {
  const long long* ll;
  int N, j;
  __host__ __device__ long long operator()(int i) const {
    const int k = j - i;
    return ll[k < 0 ? k + N : k];
  }
};

long long hc_dice_sum(int LO, int n, unsigned f, const long long* ll, int N, int j) {
  return dice_sum(LO, n, f, CyclicProducts{ll, N, j});
}

void hc_balanced_split(long long sum, int bits, int* digit, int* hi) { balanced_split(sum, bits, digit, hi); }
void hc_balanced_split32(int sum, int bits, int* digit, int* hi) { balanced_split32(sum, bits, digit, hi); }

}  // extern "C"

// The product's host tables (gl_tables.cpp), for pinning against the golden values.
#include <vector>

#include "gl_tables.h"

extern "C" {

void hc_weights(int p, int N, double* A, double* Ainv) {
  std::vector<double> a, ai;
  gl::weight_tables(p, N, (double)N, a, ai);
  for (int j = 0; j < N; ++j) {
    A[j] = a[j];
    Ainv[j] = ai[j];
  }
}

void hc_twiddles(int L, double* re, double* im) {
  for (int t = 0; t < L; ++t) {
    gl::HostCplx w = gl::twiddle(t, L);
    re[t] = w.re;
    im[t] = w.im;
  }
}

void hc_word_tables(int p, int N, int* bits, unsigned char* flags) {
  std::vector<int32_t> b;
  std::vector<uint8_t> f;
  gl::word_tables(p, N, b, f);
  for (int j = 0; j < N; ++j) {
    bits[j] = b[j];
    flags[j] = f[j];
  }
}

}  // extern "C"

extern "C" {

// layered radix-2^k DIT of R points (interleaved complex), external-twiddle values
// tv (R/2 complex, or 1 for R = 2) when with_tw, else the constant first-stage form
int hc_layered(int R, int sign, int with_tw, const double* tv, double* xy) {
  cplx* x = reinterpret_cast<cplx*>(xy);
  const cplx* t = reinterpret_cast<const cplx*>(tv);
  if (sign < 0) {
    switch (R) {
      case 2: with_tw ? layered_dit<2, -1, true>(x, t) : layered_dit<2, -1, false>(x, t); break;
      case 4: with_tw ? layered_dit<4, -1, true>(x, t) : layered_dit<4, -1, false>(x, t); break;
      case 8: with_tw ? layered_dit<8, -1, true>(x, t) : layered_dit<8, -1, false>(x, t); break;
      case 16: with_tw ? layered_dit<16, -1, true>(x, t) : layered_dit<16, -1, false>(x, t); break;
      default: return -1;
    }
  } else {
    switch (R) {
      case 2: with_tw ? layered_dit<2, 1, true>(x, t) : layered_dit<2, 1, false>(x, t); break;
      case 4: with_tw ? layered_dit<4, 1, true>(x, t) : layered_dit<4, 1, false>(x, t); break;
      case 8: with_tw ? layered_dit<8, 1, true>(x, t) : layered_dit<8, 1, false>(x, t); break;
      case 16: with_tw ? layered_dit<16, 1, true>(x, t) : layered_dit<16, 1, false>(x, t); break;
      default: return -1;
    }
  }
  return 0;
}

}  // extern "C"

extern "C" {

// the product's stage-ordered twiddle table for a line of length L (returns the size;
// out may be NULL to query it), offsets per stage into off
int hc_stage_twiddles(int L, const int* radices, int nst, double* out, int* off) {
  std::vector<int> r(radices, radices + nst);
  std::vector<gl::HostCplx> tw;
  gl::stage_twiddles(L, r, tw, off);
  if (out)
    for (size_t i = 0; i < tw.size(); ++i) {
      out[2 * i] = tw[i].re;
      out[2 * i + 1] = tw[i].im;
    }
  return (int)tw.size();
}

void hc_pair_coeff(int k, int M, double* c) {
  gl::HostCplx v = gl::pair_coeff(k, M);
  c[0] = v.re;
  c[1] = v.im;
}

}  // extern "C"

// One line DFT of length L with the given radices, run on the host through the device
// butterfly (stage_dft) and the product's stage-ordered table, in the Stockham order of
// the kernels' shared-memory stages (without the padding).  sign -1 forward, +1 inverse
// (unscaled).  Returns 0, or -1 for an unsupported radix.
namespace {
struct TableSlot {
  const cplx* tw;
  int Ns, k;
  __host__ __device__ cplx operator()(int i) const { return tw[(size_t)i * Ns + k]; }
};

template <int S>
int host_stage(int R, const cplx* src, cplx* dst, int L, int Ns, const cplx* tw) {
  const int LR = L / R;
  for (int j = 0; j < LR; ++j) {
    const int k = j % Ns;
    cplx v[16];
    for (int q = 0; q < R; ++q) v[q] = src[j + q * LR];
    const TableSlot slot{tw, Ns, k};
    const bool t = Ns > 1;
    switch (R) {
      case 2: stage_dft<2, S>(v, t, slot); break;
      case 3: stage_dft<3, S>(v, t, slot); break;
      case 4: stage_dft<4, S>(v, t, slot); break;
      case 5: stage_dft<5, S>(v, t, slot); break;
      case 7: stage_dft<7, S>(v, t, slot); break;
      case 8: stage_dft<8, S>(v, t, slot); break;
      case 16: stage_dft<16, S>(v, t, slot); break;
      default: return -1;
    }
    const int base = (j - k) * R + k;
    for (int q = 0; q < R; ++q) dst[base + q * Ns] = v[q];
  }
  return 0;
}
}  // namespace

extern "C" int hc_line_fft(int L, const int* radices, int nst, int sign, double* xy) {
  std::vector<int> r(radices, radices + nst);
  std::vector<gl::HostCplx> tw;
  int off[16];
  if (nst > 16) return -1;
  gl::stage_twiddles(L, r, tw, off);
  std::vector<cplx> a(reinterpret_cast<cplx*>(xy), reinterpret_cast<cplx*>(xy) + L), b((size_t)L);
  const cplx* t = reinterpret_cast<const cplx*>(tw.data());
  int Ns = 1;
  for (int s = 0; s < nst; ++s) {
    const int st = sign < 0 ? host_stage<-1>(r[s], a.data(), b.data(), L, Ns, t + off[s])
                            : host_stage<1>(r[s], a.data(), b.data(), L, Ns, t + off[s]);
    if (st) return st;
    Ns *= r[s];
    a.swap(b);
  }
  for (int i = 0; i < L; ++i) {
    xy[2 * i] = a[i].re;
    xy[2 * i + 1] = a[i].im;
  }
  return 0;
}

// ---------------------------------------------------------------------------
// The integer form's field arithmetic and tables (gl_gf61.cuh, gl_tables.cpp)
// ---------------------------------------------------------------------------
#include "gl_gf61.cuh"

namespace {
using gl::gf::g2;

__host__ __device__ int4 tw4(const gl::HostTw& w) { return make_int4(w.c0, w.c1, w.d0, w.d1); }

struct GfIn {
  const g2* a;
  int step;
  __host__ __device__ g2 operator()(int q) const { return a[q * step]; }
};
struct GfSlot {
  const gl::HostTw* tw;
  int step;
  __host__ __device__ int4 operator()(int q) const { return tw4(tw[q * step]); }
};

struct PolyGet {
  const int4* l;
  __host__ __device__ int4 operator()(int i) const { return l[i]; }
};

// One line of L points, stride st, transformed as the integer form's stages do; *peak: the
// largest magnitude of a stage's output.
template <int S>
void gf_line(g2* x, int st, int L, const std::vector<int>& radices, int64_t* peak) {
  std::vector<gl::HostTw> tw;
  std::vector<int> off(radices.size() + 1);
  gl::gf_stage_twiddles(radices.data(), (int)radices.size(), S > 0, tw, off.data());
  std::vector<g2> a((size_t)L), b((size_t)L);
  for (int i = 0; i < L; ++i) a[i] = x[(size_t)i * st];
  int Ns = 1;
  for (size_t s = 0; s < radices.size(); ++s) {
    const int R = radices[s], LR = L / R;
    for (int j = 0; j < LR; ++j) {
      const int k = j % Ns;
      g2 v[8];
      const GfIn in{a.data() + j, LR};
      const GfSlot slot{tw.data() + off[s] + k, Ns};
      switch (R) {
        case 2: gl::gf::butterfly<2, S>(v, Ns > 1, in, slot); break;
        case 3: gl::gf::butterfly<3, S>(v, Ns > 1, in, slot); break;
        case 4: gl::gf::butterfly<4, S>(v, Ns > 1, in, slot); break;
        case 5: gl::gf::butterfly<5, S>(v, Ns > 1, in, slot); break;
        case 7: gl::gf::butterfly<7, S>(v, Ns > 1, in, slot); break;
        default: gl::gf::butterfly<8, S>(v, Ns > 1, in, slot); break;
      }
      for (int q = 0; q < R; ++q) {
        b[(j - k) * R + k + q * Ns] = v[q];
        for (int64_t m : {v[q].re, v[q].im}) *peak = std::max(*peak, m < 0 ? -m : m);
      }
    }
    std::swap(a, b);
    Ns *= R;
  }
  for (int i = 0; i < L; ++i) x[(size_t)i * st] = a[i];
}
}  // namespace

extern "C" {

// out = the unweighted products of the words v (N = 2 W H of them) by the integer form's
// passes on an H x W layout; returns 0, or -1 where the field lacks the roots.  *peak: the
// largest magnitude of a transform stage's output.
int hc_gf_square(int p, int W, int H, const int* v, long long* out, long long* peak) {
  const int M = W * H, N = 2 * M;
  if (gl::gf_excess(M) != 1) return -1;
  std::vector<uint8_t> e;
  std::vector<gl::HostTw> k1, pair, k2;
  std::vector<gl::RowPair> rows;
  gl::gf_weights(p, N, e);
  gl::gf_pass_tables(W, H, 1, k1, pair, k2);
  gl::gf_row_pairs(W, H, rows);
  const std::vector<int> rw = gl::radix_plan(W, 8), rh = gl::radix_plan(H, 8);
  int64_t pk = 0;
  std::vector<g2> z((size_t)M);
  for (int m = 0; m < M; ++m)
    z[m] = g2{gl::gf::weighted(v[2 * m], e[2 * m]), gl::gf::weighted(v[2 * m + 1], e[2 * m + 1])};
  for (int m1 = 0; m1 < W; ++m1) {
    gf_line<-1>(&z[m1], W, H, rh, &pk);
    for (int k = 0; k < H; ++k) z[k * W + m1] = gl::gf::cmul(z[k * W + m1], tw4(k1[m1 * H + k]));
  }
  const int qW = (int)(gl::gf::kQ % (uint64_t)W);
  for (const gl::RowPair& r : rows) {
    g2 *za = &z[(size_t)r.a * W], *zb = &z[(size_t)r.b * W];
    gf_line<-1>(za, 1, W, rw, &pk);
    if (za != zb) gf_line<-1>(zb, 1, W, rw, &pk);
    for (int t = 0; t < W; ++t) {
      const int u = (int)(((int64_t)qW * t + r.shift) % W);
      if (za == zb && u < t) continue;
      g2 vk, vkp;
      gl::gf::pair_square(za[t], zb[u], tw4(pair[r.a * W + t]), &vk, &vkp);
      za[t] = vk;
      if (za != zb || t != u) zb[u] = vkp;
    }
    gf_line<+1>(za, 1, W, rw, &pk);
    if (za != zb) gf_line<+1>(zb, 1, W, rw, &pk);
    for (int t = 0; t < W; ++t) {
      za[t] = gl::gf::cmul(za[t], tw4(k2[r.a * W + t]));
      if (za != zb) zb[t] = gl::gf::cmul(zb[t], tw4(k2[r.b * W + t]));
    }
  }
  for (int m1 = 0; m1 < W; ++m1) gf_line<+1>(&z[m1], W, H, rh, &pk);
  for (int m = 0; m < M; ++m) {
    out[2 * m] = gl::gf::unweighted(z[m].re, e[2 * m]);
    out[2 * m + 1] = gl::gf::unweighted(z[m].im, e[2 * m + 1]);
  }
  *peak = pk;
  return 0;
}

// (re, im) x (c + i d) as the kernels compute it (|re|, |im| < 2^62; c, d residues)
void hc_gf_cmul(const long long* x, const unsigned long long* w, long long* out) {
  const g2 r = gl::gf::cmul(g2{x[0], x[1]}, tw4(gl::gf_pack(w[0], w[1])));
  out[0] = r.re;
  out[1] = r.im;
}
long long hc_gf_red(long long x) { return gl::gf::red(x); }
long long hc_gf_weighted(int v, int e) { return gl::gf::weighted(v, e); }
long long hc_gf_unweighted(long long x, int e) { return gl::gf::unweighted(x, e); }

// One value within R in limbs (c0, c1 of each part).
void hc_gf_as_limbs(const long long* x, int* out) {
  const int4 w = gl::gf::as_limbs(g2{x[0], x[1]});
  out[0] = w.x, out[1] = w.y, out[2] = w.z, out[3] = w.w;
}
// u(y)^2 mod y^t - z for coefficients u within R, as the polynomial row pass computes it;
// z as residues.
void hc_gf_poly_square(int t, const long long* u, const unsigned long long* z, long long* out) {
  std::vector<int4> l((size_t)t);
  for (int i = 0; i < t; ++i) l[i] = gl::gf::as_limbs(g2{u[2 * i], u[2 * i + 1]});
  const PolyGet get{l.data()};
  for (int b = 0; b < t; ++b) {
    const g2 r = gl::gf::poly_square(get, t, b, tw4(gl::gf_pack(z[0], z[1])));
    out[2 * b] = r.re;
    out[2 * b + 1] = r.im;
  }
}

}  // extern "C"
