// gl_tables.h -- host precompute of a test's word sizes, IBDWT weights and FFT
// twiddles.  All floating point here is IEEE double / double-double with explicit
// fma and -ffp-contract=off, so the tables are bit-identical on x86_64 and aarch64.
#pragma once
#include <cstdint>
#include <vector>

#include <functional>

namespace gl {

// Run body(i) for i in [0, n) on the host's cores (std::thread, static chunks).
void parallel_for(int64_t n, const std::function<void(int64_t, int64_t)>& chunk);

struct HostCplx {
  double re, im;
};

// setSliceAndDice (gpuLucas.cu:323-343) extended to ratio 21; -1 when refused.
int slice_depth(int p, int N);

// bits[j] = ceil(p(j+1)/N) - ceil(pj/N) (computeBitsPerWord, gpuLucas.cu:688-694, in
// exact integer arithmetic); flags[j] bit i = word (j-i) mod N has LO+1 bits, i < 8
// (computeBitsPerWordVectors, gpuLucas.cu:700-714).
void word_tables(int p, int N, std::vector<int32_t>& bits, std::vector<uint8_t>& flags);
// One entry of each: bits[j] and flags[j] of word_tables (no containers).
int word_bits(int p, int N, int j);
uint8_t word_flags(int p, int N, int j);

// A[j] = 2^(ceil(jp/N) - jp/N) and Ainv[j] = 2^-(ceil(jp/N) - jp/N) * scale, computed in
// double-double and rounded once (computeWeightVectors, gpuLucas.cu:673-686, uses
// scale = 1/N; the fused kernels need 1/(2N)).
void weight_tables(int p, int N, double inv_scale_den, std::vector<double>& A, std::vector<double>& Ainv);

// One entry of weight_tables: A[j] and Ainv[j] (same rounding), no containers.
void weight_entry(int p, int N, int j, double inv_scale_den, double* A, double* Ainv);

// exp(-2 pi i t / L) for t in [0, L), correctly rounded from double-double.
void twiddle_table(int64_t L, std::vector<HostCplx>& tw);
HostCplx twiddle(int64_t t, int64_t L);

// Stage-ordered values of one Stockham line DFT of length L with the given radix
// sequence.  Stage s (span Ns, radix R, external twiddle w = w_L^(k L/(Ns R)) for
// butterfly position k < Ns) stores its 16-byte slots v-major at off[s] + v*Ns + k, so
// lanes with consecutive k read consecutive slots:
//  - R = 8, 4, 3: the ratio form of w^q = i^f rho_q (1 + i tau_q) (8, 4, 4 slots of two
//    doubles: tau, ratios of rho, flags; the order is the device butterflies', ratio_r8,
//    ratio_r4, ratio_r3 in gl_device.cuh);
//  - R = 2, 16: the layered radix-2 DIT needs, at level l = 1..log2 R, the values
//    w^(R/2^l) * W_(2^l)^p for p < max(1, 2^(l-2)) (the other half are the same times
//    +-i): v runs over (l=1,p=0), (l=2,p=0), (l=3,p=0..1), (l=4,p=0..3);
//  - R = 5, 7: w^q for q = 1..R-1.
// The first stage (Ns = 1) needs no table.  Returns the table (at least one entry)
// and fills off[] (offset of each stage).
void stage_twiddles(int L, const std::vector<int>& radices, std::vector<HostCplx>& tw, int* off);
// number of stored 16-byte slots per butterfly position for a stage of radix R
int stage_values(int R);

// -(1 + w_M^k)/4 from double-double cos/sin, rounded once: the coefficient of the
// real-signal square V_k = U_k^2 + c_k (U_k - conj(U_{M-k}))^2.
HostCplx pair_coeff(int64_t k, int64_t M);

// ---- tables of the integer form (gl_gf61.cuh): everything is exact in GF(q^2), q = 2^61 - 1

// a table entry (c, d) for c + i d, each as two limbs c0 + c1 2^31
struct HostTw {
  int32_t c0, c1, d0, d1;
};
// GF(q^2) has roots of unity of order M for odd parts of M that divide 3^2 5^2 7.  For
// other M the transform is of length M/t, t the excess odd part, over polynomials of degree
// below t: u[b + t a] is coefficient b of element a, and frequency k holds a polynomial mod
// y^t - root(k, M/t).  Returns t (1: a plain transform).  N = 2 M is prime to 61, so the
// weights are powers of two.
int gf_excess(int M);
// the entry of c + i d, 0 <= c, d < q
HostTw gf_pack(uint64_t c, uint64_t d);
// Values of one Stockham line DFT: for every stage after the first, span Ns and radix R, w^q
// (q = 1..R-1) of w = root(+-k, Ns R) at off[s] + (q-1) Ns + k, where root(t, L) is a fixed
// family of roots of unity with root(t, L) root(u, L) = root(t + u, L) and root(t k, L k) =
// root(t, L).
void gf_stage_twiddles(const int* radices, int nst, bool inverse, std::vector<HostTw>& tw, int* off);
// For t = gf_excess(W H), W = t V, L = V H (t = 1: V = W, L = M):
// k1[m1 H + k2] = root((m1/t) k2, L); k2t[k2 W + m1] = root(-(m1/t) k2, L) / L;
// pair[k2 V + k1] = -(1 + root(k2 + H k1, L)) / 4 for t = 1, root(k2 + H k1, L) for t > 1
void gf_pass_tables(int W, int H, int t, std::vector<HostTw>& k1, std::vector<HostTw>& pair, std::vector<HostTw>& k2t);
// The row pairs of the row pass.  Frequency k = k2 + H k1 pairs with q k mod L, so row k2
// pairs with row q k2 mod H, and in it position k1 with q k1 + shift mod V.
struct RowPair {
  int32_t a, b, shift, pad;  // rows a <= b (a == b: a row paired with itself)
};
void gf_row_pairs(int V, int H, std::vector<RowPair>& rows);
// weight exponent of word j: A[j] = 2^(r/N) = 2^e with r = ceil(jp/N) N - jp, e = r N^-1 mod 61
void gf_weights(int p, int N, std::vector<uint8_t>& e);

// factor n into the allowed radices (16, 8, 4, 2, 3, 5, 7; powers of two up to
// max_radix), largest power of two first, then 3, 5, 7; empty if n has another prime
// factor.
std::vector<int> radix_plan(int n, int max_radix);
// The same into out[0..cap): returns the number of stages, or -1 if n has another prime
// factor or needs more than cap stages.
int radix_plan_into(int n, int max_radix, int* out, int cap);

}  // namespace gl
