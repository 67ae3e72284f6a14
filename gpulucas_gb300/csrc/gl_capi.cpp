// gl_capi.cpp -- the C ABI (include/gpulucas.h): plans, iteration, residues and the
// reference-named entry points errorTest / mersenneTest / setSliceAndDice.
#include <algorithm>
#include <array>
#include <cmath>
#include <cstdio>
#include <map>
#include <mutex>
#include <cstdlib>
#include <cstring>
#include <new>
#include <type_traits>
#include <vector>

#include "gl_gf61.cuh"
#include "gl_internal.h"
#include "gl_plan.h"
#include "gl_tables.h"

using namespace gl;

namespace {

constexpr int kGraphBatch = 64;
// An integer-form plan runs one iteration in this many in FP64: the same products, with
// the round-off measured.
constexpr int kFp64Every = 64;
static_assert(kFp64Every == kGraphBatch, "a captured batch ends with its FP64 iteration");

int cuda_status(cudaError_t e) { return e == cudaSuccess ? GL_OK : GL_ERR_CUDA; }

#define GL_CUDA(call)                                \
  do {                                               \
    cudaError_t e_ = (call);                         \
    if (e_ != cudaSuccess) return GL_ERR_CUDA;       \
  } while (0)

template <typename T>
int dev_alloc(gl_plan* pl, T** ptr, size_t count) {
  void* p = nullptr;
  size_t bytes = sizeof(T) * count;
  if (cudaMalloc(&p, bytes) != cudaSuccess) {
    cudaGetLastError();  // the next launch would return it as its own
    return GL_ERR_NOMEM;
  }
  pl->allocs.push_back(p);
  pl->device_bytes += bytes;
  *ptr = static_cast<T*>(p);
  return GL_OK;
}

bool fill_line_plan(int L, LinePlan* lp, int max_radix = kMaxRadix) {
  std::vector<int> r = radix_plan(L, max_radix);
  if (r.empty() || r.size() > 8) return false;
  lp->L = L;
  lp->nst = (int)r.size();
  for (int i = 0; i < 8; ++i) lp->radix[i] = i < lp->nst ? r[i] : 0;
  return true;
}

int round_up32(int x) { return (x + 31) / 32 * 32; }

// FP64 instructions per point of one stage of radix r of a line DFT.  First stage:
// constant twiddles only (layered DIT, DFT_R).  Later stages: radices 8, 4, 3 in ratio
// form (66, 22, 16 instructions per butterfly), 2 and 16 the layered DIT (3 per point and
// bit), 5 and 7 DFT_R plus one complex product per input.
double stage_ops(int r, bool first) {
  const bool pow2 = (r & (r - 1)) == 0;
  int lg = 0;
  while ((1 << lg) < r) ++lg;
  if (!first && (r == 8 || r == 4 || r == 3)) return (r == 8 ? 66.0 : r == 4 ? 22.0 : 16.0) / r;
  if (pow2) {
    if (!first) return 3.0 * lg;
    return r == 2 ? 2.0 : r == 4 ? 4.0 : r == 8 ? 6.5 : 9.25;  // 16
  }
  const double odd = r == 3 ? 14.0 : r == 5 ? 36.0 : 72.0;  // 7
  return odd / r + (first ? 0.0 : 4.0 * (r - 1) / r);
}

// FP64 instructions per point of one line DFT with the given radices.
double line_ops(const LinePlan& lp) {
  double ops = 0.0;
  for (int s = 0; s < lp.nst; ++s) ops += stage_ops(lp.radix[s], s == 0);
  return ops;
}

// FP64 instructions issued per point of one line DFT when a CTA transforms `nlines` lines
// of the plan together: a stage of radix r has nlines L / r butterflies, one per lane, and
// a warp issues each instruction for all 32 lanes, so the stage costs round_up32(its
// butterflies) / its butterflies times its work.
double line_issue_ops(const LinePlan& lp, int nlines) {
  double ops = 0.0;
  for (int s = 0; s < lp.nst; ++s) {
    const int nb = nlines * lp.L / lp.radix[s];
    ops += stage_ops(lp.radix[s], s == 0) * (double)((nb + 31) / 32 * 32) / nb;
  }
  return ops;
}

// Line plan that issues the fewest FP64 instructions with `nlines` lines per CTA, for
// a batch member (lines short enough that partly filled warps matter): L = 2^a 3^b 5^c 7^d
// with the power of two split into radices 8, 4 and 2 (8 and 4 up to max_radix) in every
// way, and each distinct radix tried as the first stage (the one with constant twiddles);
// the other stages keep the order 8, 4, 2, 3, 5, 7.  At most 8 stages.
bool fill_line_plan_issue(int L, int nlines, int max_radix, LinePlan* lp) {
  if (L < 2) return false;
  int m = L, e[4] = {0, 0, 0, 0};
  const int primes[4] = {2, 3, 5, 7};
  for (int i = 0; i < 4; ++i)
    while (m % primes[i] == 0) {
      m /= primes[i];
      ++e[i];
    }
  if (m != 1) return false;
  double best = 1e300;
  LinePlan out{};
  for (int n8 = 0; 3 * n8 <= e[0]; ++n8) {
    if (n8 && max_radix < 8) break;
    for (int n4 = 0; 3 * n8 + 2 * n4 <= e[0]; ++n4) {
      if (n4 && max_radix < 4) break;
      const int n2 = e[0] - 3 * n8 - 2 * n4;
      const int counts[6] = {n8, n4, n2, e[1], e[2], e[3]};
      const int radices[6] = {8, 4, 2, 3, 5, 7};
      const int nst = n8 + n4 + n2 + e[1] + e[2] + e[3];
      if (nst < 1 || nst > 8) continue;
      for (int f = 0; f < 6; ++f) {
        if (!counts[f]) continue;
        LinePlan c{};
        c.L = L;
        c.nst = nst;
        int k = 0;
        c.radix[k++] = radices[f];
        for (int i = 0; i < 6; ++i)
          for (int j = 0; j < counts[i] - (i == f ? 1 : 0); ++j) c.radix[k++] = radices[i];
        const double cost = line_issue_ops(c, nlines);
        if (cost < best - 1e-9) {
          best = cost;
          out = c;
        }
      }
    }
  }
  if (best >= 1e300) return false;
  *lp = out;
  return true;
}

int padded_stride(int L) { return L + (L >> 4) + 1; }

// FP64-instruction equivalent of one CTA's fixed cost in a batch launch
constexpr double kBatchUnitOverhead = 2000.0;

int stage_offsets(const LinePlan& lp, int* off);

// Shared memory of a row-pass CTA: four line buffers (the pair, ping-pong) and the copy of
// the length-W line DFT's stage values.
size_t row_smem(int W, const LinePlan& pw) {
  int off[8];
  return (size_t)4 * padded_stride(W) * 16 + (size_t)stage_offsets(pw, off) * sizeof(DevCplx);
}

// Radix caps of a layout chosen without timing: below 2^17 complex points a single test
// cannot fill the device with one thread per radix-8 butterfly, and the timed search
// picks radix-4 caps there (more warps per line); a batch member keeps radix 8 (the batch
// fills the device).  Explicit options win.
void model_caps(int M, const gl_plan_opts& o, int sms_override, int* rc, int* rr) {
  const bool small = M < (1 << 17) && !sms_override && !o.fft_h;
  *rc = o.max_radix_col ? o.max_radix_col : (small ? 4 : kMaxRadix);
  *rr = o.max_radix_row ? o.max_radix_row : (small ? 4 : kMaxRadix);
}

// Pick M = W * H for `sms` SMs.  Work units: W columns (column passes, one per CTA)
// and H/2+1 row pairs (row pass).  With equal units per kernel the busiest SM runs
// ceil(units / sms) of them, so the modelled time is the sum over the three kernels
// of ceil(units/sms) * FP64 instructions per unit.  Shared memory per CTA must fit
// twice (two CTAs per SM at least) and blocks stay <= kMaxThreads.
// Every usable column length H of M = W * H with its modelled cost, cheapest first.
std::vector<std::pair<double, int>> ranked_layouts(int M, int sms) {
  if (sms <= 0) sms = 152;
  std::vector<std::pair<double, int>> out;
  for (int H = 2; H <= M / 2; ++H) {
    if (M % H) continue;
    const int W = M / H;
    if (W < 4) continue;  // the forward column pass finds the words below a column with one wrap
    LinePlan a, b;
    // a batch member: line plans and costs by the FP64 instructions issued (a CTA takes
    // one column or one row pair), since its short lines leave warps partly filled
    const bool member = sms == 1;
    if (member ? !fill_line_plan_issue(W, 2, kMaxRadix, &a) || !fill_line_plan_issue(H, 1, kMaxRadix, &b)
               : !fill_line_plan(W, &a) || !fill_line_plan(H, &b))
      continue;
    const size_t smc = (size_t)2 * padded_stride(H) * 16, smr = row_smem(W, a);
    if (smc > (size_t)kMaxDynSmem || smr > (size_t)kMaxDynSmem) continue;
    if ((H + kElemsPerThread - 1) / kElemsPerThread > 4 * kMaxThreads) continue;
    const double col_ops = member ? line_issue_ops(b, 1) : line_ops(b);
    const double row_ops = member ? line_issue_ops(a, 2) : line_ops(a);
    double col = std::ceil((double)W / sms) * H * (col_ops + 6.0);
    double row = std::ceil((double)(H / 2 + 1) / sms) * 2.0 * W * (2.0 * row_ops + 16.0);
    if (member) {
      // its units share the device with the batch's other units, so the fixed cost of a
      // CTA (launch, descriptor copy, barriers, global round trips) is charged per unit,
      // which keeps the lines long enough to amortise it
      col += (double)W * kBatchUnitOverhead;
      row += (double)(H / 2 + 1) * kBatchUnitOverhead;
    }
    double cost = 2.0 * col + row;
    // prefer smaller shared-memory footprints (more resident CTAs) on ties
    cost *= 1.0 + 0.02 * (double)(smc + smr) / (64.0 * 1024);
    out.emplace_back(cost, H);
  }
  std::sort(out.begin(), out.end());
  return out;
}

// Block size of the row pass (two lines of W points): from t0 (one thread per butterfly of
// the largest-radix stage) up to kRowThreads, the smallest multiple of 32 that minimises
// the stages' rounds of butterflies weighted by radix, so that a stage with more, smaller
// butterflies (radix 3 after radix 8) does not leave most warps waiting at its barrier
// while a few run one more round.  W = 576 (8, 8, 3, 3): 160 -> 192 threads.
int row_threads(int W, const LinePlan& pw, int t0) {
  int best = t0;
  long best_cost = -1;
  for (int t = t0; t <= kRowThreads; t += 32) {
    long cost = 0;
    for (int s = 0; s < pw.nst; ++s) {
      const int R = pw.radix[s];
      const int nb = 2 * W / R;
      cost += (long)((nb + t - 1) / t) * R;
    }
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best = t;
    }
  }
  return best;
}

// Layout for M: column length `force_h` (0: the model's best) with line plans whose
// largest radix is rc (columns) / rr (rows); each column gets one thread per butterfly
// of its largest-radix stage, each row pair row_threads().
int choose_fused_geom(int M, int force_h, int sms, FusedGeom* g, int rc = kMaxRadix, int rr = kMaxRadix,
                      bool ip = false, bool pf = false, bool ws = false, int row = 0) {
  if ((rc != 8 && rc != 4 && rc != 2) || (rr != 8 && rr != 4 && rr != 2)) return GL_ERR_ARG;
  int bestH = 0;
  for (const auto& c : ranked_layouts(M, sms))
    if (!force_h || c.second == force_h) {
      bestH = c.second;
      break;
    }
  if (!bestH) return GL_ERR_SIZE;
  g->H = bestH;
  g->W = M / bestH;
  g->G = 1;
  g->rc = rc;
  g->rr = rr;
  if (sms == 1) {  // a batch member: the plans that issue the fewest FP64 instructions
    if (!fill_line_plan_issue(g->W, 2, rr, &g->pw) || !fill_line_plan_issue(g->H, 1, rc, &g->ph)) return GL_ERR_SIZE;
  } else if (!fill_line_plan(g->W, &g->pw, rr) || !fill_line_plan(g->H, &g->ph, rc)) {
    return GL_ERR_SIZE;
  }
  g->ls_col = padded_stride(g->H);
  g->ls_row = padded_stride(g->W);
  g->sm_col = (size_t)2 * g->ls_col * 16;
  g->sm_cinv = g->sm_col;
  g->sm_row = row_smem(g->W, g->pw);
  auto threads = [](int points, int per_thread, int cap) {
    int t = round_up32((points + per_thread - 1) / per_thread);
    return t < 64 ? 64 : (t > cap ? cap : t);
  };
  g->t_col = threads(g->H, rc, kMaxThreads);
  g->t_row = row_threads(g->W, g->pw, threads(2 * g->W, rr, kRowThreads));
  g->row_var = 0;
  if (row < 0 || row > 2) return GL_ERR_ARG;
  if (row > 0) {
    for (int s = 0; s < g->pw.nst; ++s) {
      const int R = g->pw.radix[s];
      if (R != 2 && R != 3 && R != 4) return GL_ERR_SIZE;
    }
    g->row_var = row;
    if (row == 2) g->sm_row = (size_t)4 * g->ls_row * 16;  // stage values read through L1
  }
  g->col_ip = 0;
  g->col_pf = 0;
  g->col_ws = 0;
  if (ip || ws) {
    // in place: every column stage has at most (8 / R for radix R = 2^k, 1 for odd R)
    // butterflies per thread, held in registers across the stage's first barrier
    for (int s = 0; s < g->ph.nst; ++s) {
      const int R = g->ph.radix[s];
      const int per = (R & (R - 1)) == 0 ? 8 / R : 1;
      if (g->H / R > per * g->t_col) return GL_ERR_SIZE;
    }
    g->col_ip = 1;
    g->sm_col = g->sm_cinv = (size_t)g->ls_col * 16;
    if (ws) {
      // two columns per CTA: two in-place line buffers; the inverse pass too, unless it
      // prefetches its weights (then it keeps one column per CTA)
      if (g->W < 2 || g->t_col != kMaxThreads) return GL_ERR_SIZE;
      g->col_ws = 1;
      g->sm_col = g->sm_cinv = (size_t)2 * g->ls_col * 16;
      if (g->sm_col > (size_t)kMaxDynSmem) return GL_ERR_SIZE;
    }
    if (pf) {
      if (g->H % 8) return GL_ERR_SIZE;  // bulk copies of 2H bytes must be 16-byte multiples
      g->col_pf = 1;
      g->sm_cinv = (size_t)g->ls_col * 16 + (size_t)18 * g->H;
    }
  }
  return GL_OK;
}

int choose_plain_geom(int M, PlainGeom* g) {
  const int nst = radix_plan_into(M, 4, g->radix, 40);
  if (nst <= 0) return GL_ERR_SIZE;
  g->nst = nst;
  g->threads = 256;
  return GL_OK;
}

// offsets of each stage in a stage-ordered twiddle table (gl_tables.cpp layout) and
// the table length, without computing the values
int stage_offsets(const LinePlan& lp, int* off) {
  int size = 1, Ns = 1;
  for (int s = 0; s < lp.nst; ++s) {
    off[s] = size;
    if (Ns > 1) size += stage_values(lp.radix[s]) * Ns;
    Ns *= lp.radix[s];
  }
  return size;
}

int int_stage_offsets(LinePlan* lp) {
  int size = 1, Ns = 1;
  for (int s = 0; s < lp->nst; ++s) {
    lp->off[s] = size;
    if (Ns > 1) size += (lp->radix[s] - 1) * Ns;
    Ns *= lp->radix[s];
  }
  return size;
}

// Largest polynomial length (gf_excess) the integer form is used at.  Squaring takes about
// t/2 products per coefficient, but a test alone waits on latencies more than it computes
// (us per iteration, integer/FP64: t = 7, N = 44100, 24.9/35.2, 78400, 26.1/39.2; t = 25,
// 52500, 27.0/35.7; t = 27, 54432, 28.8/31.6, 62208, 28.0/27.0, 124416, 29.7/32.9, 995328,
// 96.8/140; t = 35, 98000, 34.3/43.1; t = 49, 43904, 28.7/34.6, 351232, 68.2/75.6).
constexpr int kMaxIntPoly = 49;
// Longer polynomials than this pay at some lengths only (t = 45: 40500, 28.3/30.5; 81000,
// 36.0/33.5; 324000, 74.3/65.9; 648000, 123/117; 1296000, 211/223; 2592000, 386/434; t = 49:
// 82320, 37.6/40.1; 98784, 43.8/39.7; 137200, 49.2/47.5), so there both forms are timed; from
// 2^14 points, since below launches take most of either's time and the integer form is faster.
constexpr int kMaxSurePoly = 27;
constexpr int kMinTimedFormM = 1 << 14;

// Geometry of the integer form on an H x W layout; false where its polynomials do not fit
// the rows or a CTA's lines its shared memory.
// in_place, wide, rc, rr: the variants autotune_int_layout times.
struct IntVariant {
  bool in_place = false;  // column passes in place
  bool wide = false;      // a thread per two points instead of one per butterfly
  int rc = kMaxRadix, rr = kMaxRadix;  // largest radix of the columns and rows
};
bool choose_int_geom(int H, int W, IntGeom* g, const IntVariant& var = IntVariant()) {
  g->t = gf_excess(H * W);
  if (g->t > kMaxIntPoly || W % g->t) return false;
  const int V = W / g->t;
  if (!fill_line_plan(V, &g->pw, var.rr) || !fill_line_plan(H, &g->ph, var.rc)) return false;
  int_stage_offsets(&g->pw);
  int_stage_offsets(&g->ph);
  auto threads = [](int n) {
    const int t = round_up32(n);
    return t < 64 ? 64 : (t > kMaxThreads ? kMaxThreads : t);
  };
  g->col_p = var.in_place;
  g->t_col = threads(var.wide ? H / 2 : (H + var.rc - 1) / var.rc);
  g->t_row = var.wide || g->t > 1 ? threads(W) : row_threads(W, g->pw, threads((2 * W + var.rr - 1) / var.rr));
  for (int s = 0; s < g->ph.nst && var.in_place; ++s) {
    // radices 8, 4, 2, 3 only, and no more butterflies than the threads hold
    const int R = g->ph.radix[s];
    if (R == 5 || R == 7 || H / R > kIntHeld / R * g->t_col) return false;
  }
  g->sm_col = (size_t)(var.in_place ? 1 : 2) * int_stride(H) * 16;
  g->sm_row = (size_t)int_row_slots(V, g->t) * 16;
  return g->sm_col <= (size_t)kMaxIntSmem && g->sm_row <= (size_t)kMaxIntSmem;
}

// The variant for a layout chosen without timing, what the search usually picks: radix 4 and
// wide blocks below 2^17 points, above in-place columns where they fit (N = 2359296:
// 134 us per iteration against 142 with two buffers).
IntVariant untimed_variant(int H, int W) {
  IntVariant v;
  IntGeom g{};
  if ((int64_t)H * W < (1 << 17)) {
    v.rc = v.rr = 4;
    v.wide = true;
  } else {
    v.in_place = true;
    if (!choose_int_geom(H, W, &g, v)) v.in_place = false;
  }
  return v;
}

// Whether the integer form is worth its while at M points, where nothing is timed: not at
// t = 45 (see kMaxSurePoly; the FP64 form's radices 3 and 5 lose little there) below 2^19.
bool int_pays_untimed(int M) {
  const int t = gf_excess(M);
  return t <= kMaxSurePoly || t % 7 == 0 || M < kMinTimedFormM || M >= (1 << 19);
}

// Column length of the first layout of the cost model that the integer form can run, or 0.
int first_int_layout(int M, int sms) {
  IntGeom g{};
  for (const auto& c : ranked_layouts(M, sms))
    if (choose_int_geom(c.second, M / c.second, &g)) return c.second;
  return 0;
}

// Whether the passes touch the tables they will read at their start (IntArgs::touch): where
// at most two CTAs run per SM, its L1 is empty and has room for all of them.
int int_touch(int H, int W) { return W <= 2 * kSms && H / 2 < 2 * kSms; }

// Whether the products of (p, N) are determined by their residues mod q = 2^61 - 1 for
// every state the iteration can reach: words are at most 2^LO plus a carry in magnitude,
// an unweighted product sums N of their products times at most 2, and must stay within
// gf::kMaxProduct.  *vmax: the bound on a word used here (a loaded state is checked against it).
constexpr double kProductBound = 1152921504606846976.0 - 1024.0;  // 2^60, less the rounding of the sum
bool int_range_ok(int p, int N, int* vmax) {
  const int LO = p / N;
  if (LO > 28) return false;
  const double v = (double)(1 << LO) + 256.0;
  *vmax = (1 << LO) + 256;
  static_assert((int64_t)kProductBound <= gf::kMaxProduct, "the sum below is rounded");
  return 2.0 * N * v * v <= kProductBound;
}

// The integer form has no round-off to watch, so it is used where the FP64 form's stays
// below the default limit and with a limit that is not tightened; elsewhere every iteration
// measures its round-off.  The line is gl_safe_signal_size's (round-off <= 0.125) plus 0.3
// bits per word: the round-off doubles every 0.45 bits or so, so <= 0.2 there (measured on
// the line, 1500 to 30000 iterations at 18 lengths from 4200 to 4194304: 0.14 to 0.19).  At
// the resident lengths, which a full test of p - 2 iterations is short at, the line is closer
// to the limit: plus 0.9 up to N = 2048, plus 0.75 up to 4096.  Measured on it, 60000
// iterations each: N = 2048 0.34, 2000 and 1920 0.38, 1536 and 1280 0.31, 4096 0.27, 3840 0.31,
// 3072 0.28, 2560 0.31.  From N = 1024 down the carry table's 22 bits come before the line:
// 0.31 at 1024 and 960, 0.38 at 1000, 0.27 at 768, 0.19 at 512, 0.06 at 128.
bool int_roundoff_ok(int p, int N, double error_limit) {
  const double over = N <= 2048 ? 0.9 : N <= kResidentAutoN ? 0.75 : 0.3;
  return error_limit >= 0.4 && (double)p / N <= 19.2 + over - 0.26 * std::log2(N / 163840.0);
}

// Device buffers of a layout search, kept from one variant to the next: allocated
// zero-filled, grown where a variant needs more.
struct SearchBuffers {
  static constexpr int kMax = 16;
  void* ptr[kMax] = {};
  size_t cap[kMax] = {};
  ~SearchBuffers() {
    for (void* p : ptr)
      if (p) cudaFree(p);
  }
  bool get(int i, size_t bytes, cudaStream_t s) {
    if (cap[i] >= bytes) return true;
    if (ptr[i]) cudaFree(ptr[i]);
    ptr[i] = nullptr;
    cap[i] = 0;
    if (cudaMalloc(&ptr[i], bytes) != cudaSuccess) {
      cudaGetLastError();  // the next launch would return it as its own
      ptr[i] = nullptr;
      return false;
    }
    cap[i] = bytes;
    return cudaMemsetAsync(ptr[i], 0, bytes, s) == cudaSuccess;
  }
};

// Device time of one fused iteration with column length H, measured on zero-filled
// buffers (the kernels' time does not depend on the values).  Returns ms, or -1.
double time_layout(int M, int H, int rc, int rr, bool ip, bool pf, bool ws, int row, int n, int sms, int iters,
                   SearchBuffers& sb, cudaStream_t s) {
  FusedGeom g{};
  if (choose_fused_geom(M, H, sms, &g, rc, rr, ip, pf, ws, row) != GL_OK) return -1.0;
  const int N = 2 * M;
  const int szw = stage_offsets(g.pw, g.pw.off), szh = stage_offsets(g.ph, g.ph.off);
  const size_t bytes[] = {sizeof(long long) * N, (size_t)N, (size_t)N, sizeof(double) * N, sizeof(double) * N,
                          16 * (size_t)M, 16 * (size_t)M, 16 * (size_t)M, 16 * (size_t)M,
                          16 * (size_t)szw, 16 * (size_t)szh, sizeof(int) * N, (size_t)N, sizeof(Status),
                          16 * (size_t)M};
  constexpr int nb = sizeof(bytes) / sizeof(bytes[0]);
  static_assert(nb <= SearchBuffers::kMax, "buffers of a search");
  void* const* buf = sb.ptr;
  double ms = -1.0;
  bool ok = true;
  for (int i = 0; i < nb && ok; ++i) ok = sb.get(i, bytes[i], s);
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (ok) ok = cudaEventCreate(&e0) == cudaSuccess && cudaEventCreate(&e1) == cudaSuccess;
  if (ok) ok = set_fused_smem_limits(g) == cudaSuccess;
  if (ok) {
    IterArgs a{};
    a.N = N; a.M = M; a.W = g.W; a.H = g.H; a.G = 1; a.LO = 18; a.n = n;
    a.ls_col = g.ls_col; a.ls_row = g.ls_row; a.pw = g.pw; a.ph = g.ph;
    a.ll = (long long*)buf[0]; a.flags = (const unsigned char*)buf[1]; a.span = (const unsigned char*)buf[2];
    a.A = (const double*)buf[3]; a.Ainv = (const double*)buf[4]; a.Z = (DevCplx*)buf[5];
    a.twK1 = (const DevCplx*)buf[6]; a.twPair = (const DevCplx*)buf[7]; a.twK2 = (const DevCplx*)buf[8];
    a.twW = (const DevCplx*)buf[9]; a.twH = (const DevCplx*)buf[10]; a.twW_n = szw;
    a.digit = (int*)buf[11]; a.hi = (signed char*)buf[12]; a.status = (Status*)buf[13];
    a.Z2 = (DevCplx*)buf[14];
    for (int i = 0; i < 2 && ok; ++i) ok = launch_fused_iteration(a, g, s, false) == cudaSuccess;
    ok = ok && cudaEventRecord(e0, s) == cudaSuccess;
    for (int i = 0; i < iters && ok; ++i) ok = launch_fused_iteration(a, g, s, false) == cudaSuccess;
    ok = ok && cudaEventRecord(e1, s) == cudaSuccess && cudaEventSynchronize(e1) == cudaSuccess;
    float t = 0.f;
    if (ok && cudaEventElapsedTime(&t, e0, e1) == cudaSuccess) ms = t / iters;
  }
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  cudaStreamSynchronize(s);
  return ms;
}

// Autotuned layout for M on this device: the cheapest few column lengths of the cost
// model are timed and the fastest kept, once per (M, SM count) per process.  Below
// 2^17 complex points the lines are too short to fill the GPU with one thread per
// radix-8 butterfly, so the three best lengths are also timed with radix-4 and radix-2
// caps.  The column-pass variants (two buffers, in place, in place with prefetched
// weights, two columns per CTA) are timed on the best lengths, and the winner once more
// with radix-4 rows: a radix-8 row stage of W/8 butterflies per line leaves part of a warp
// idle when 2W/8 is not a multiple of 32 (W = 576: 144 butterflies on 192 threads), while
// radix-4 stages fill whole warps.  only_h: that column length alone (an integer-form plan's,
// whose FP64 iterations run on the layout the integer search picked).
struct TunedLayout {
  int H = 0, rc = kMaxRadix, rr = kMaxRadix, row = 0;
  bool ip = false, pf = false, ws = false;
  double ms = 0.0;
};
std::mutex g_tune_mutex;
std::map<std::array<int, 3>, TunedLayout> g_tune_cache;

TunedLayout autotune_layout(int M, int n, int sms, cudaStream_t s, double* ms_out, int only_h = 0) {
  {
    std::lock_guard<std::mutex> lock(g_tune_mutex);
    auto it = g_tune_cache.find({M, sms, only_h});
    if (it != g_tune_cache.end()) {
      if (ms_out) *ms_out = it->second.ms;
      return it->second;
    }
  }
  auto ranked = ranked_layouts(M, sms);
  if (only_h)
    ranked.erase(std::remove_if(ranked.begin(), ranked.end(), [&](const auto& c) { return c.second != only_h; }),
                 ranked.end());
  TunedLayout best;
  double best_ms = 1e300;
  const int iters = M >= (1 << 18) ? 10 : 40;
  SearchBuffers sb;
  auto consider = [&](int H, int rc, int rr, bool ip, bool pf = false, bool ws = false, int row = 0) {
    const double ms = time_layout(M, H, rc, rr, ip, pf, ws, row, n, sms, iters, sb, s);
    if (ms > 0.0 && ms < best_ms) {
      best_ms = ms;
      best.H = H;
      best.rc = rc;
      best.rr = rr;
      best.ip = ip;
      best.pf = pf;
      best.ws = ws;
      best.row = row;
    }
  };
  for (size_t i = 0; i < ranked.size() && i < 6; ++i) {
    consider(ranked[i].second, kMaxRadix, kMaxRadix, false);
    // the in-place column passes (half the shared memory, 4 CTAs per SM); long columns
    // also with prefetched weights and two per CTA
    consider(ranked[i].second, kMaxRadix, kMaxRadix, true);
    if (M >= (1 << 17)) {
      consider(ranked[i].second, kMaxRadix, kMaxRadix, true, true);
      consider(ranked[i].second, kMaxRadix, kMaxRadix, true, false, true);
      consider(ranked[i].second, kMaxRadix, kMaxRadix, true, true, true);
    }
  }
  if (M >= (1 << 17) && best.H) {
    const TunedLayout b = best;
    consider(b.H, b.rc, 4, b.ip, b.pf, b.ws);
  }
  if (best.H) {
    // the row pass compiled for radices 4, 3, 2 only, with its stage values in shared
    // memory or read through L1 (where the row plan allows it; otherwise not timed)
    const TunedLayout b = best;
    consider(b.H, b.rc, b.rr, b.ip, b.pf, b.ws, 1);
    consider(b.H, b.rc, b.rr, b.ip, b.pf, b.ws, 2);
  }
  if (M < (1 << 17))
    for (size_t i = 0; i < ranked.size() && i < 3; ++i) {
      consider(ranked[i].second, 4, kMaxRadix, false);
      consider(ranked[i].second, kMaxRadix, 4, false);
      consider(ranked[i].second, 4, 4, false);
      consider(ranked[i].second, 4, 4, true);
      consider(ranked[i].second, 4, kMaxRadix, true);
      // radix-2 stages: a little more FP64 work per point and bit (3 against 2.75 for
      // radix 4 in ratio form), twice the butterflies per stage, so twice the warps to hide
      // FP64 latency on short lines
      consider(ranked[i].second, 2, 4, false);
      consider(ranked[i].second, 4, 2, false);
      consider(ranked[i].second, 2, 2, false);
    }
  if (!best.H) return best;
  best.ms = best_ms;
  std::lock_guard<std::mutex> lock(g_tune_mutex);
  g_tune_cache[{M, sms, only_h}] = best;
  if (ms_out) *ms_out = best_ms;
  return best;
}

// Device time of one integer-form iteration on the H x (M / H) layout, or -1.  The best of
// three runs, since variants of short lengths lie within a few per cent; of fewer, once it is
// a third above best_ms, the fastest variant so far (a hiccup of the host makes up a tenth).
// replay: the iterations of a run as one captured graph, as a plan replays them.
double time_int_layout(int M, int H, const IntVariant& var, int n, int iters, double best_ms, SearchBuffers& sb,
                       cudaStream_t s, bool replay = false) {
  IntGeom g{};
  const int W = M / H, N = 2 * M;
  if (!choose_int_geom(H, W, &g, var)) return -1.0;
  std::vector<RowPair> rows;
  gf_row_pairs(W / g.t, H, rows);
  LinePlan pw = g.pw, ph = g.ph;
  const size_t szw = (size_t)int_stage_offsets(&pw) * 16, szh = (size_t)int_stage_offsets(&ph) * 16;
  const size_t m16 = 16 * (size_t)M;
  const size_t bytes[] = {8 * (size_t)N, (size_t)N, (size_t)N, (size_t)N, m16, m16, m16, m16, m16,
                          szw, szw, szh, szh, rows.size() * sizeof(RowPair), sizeof(Status)};
  constexpr int nb = sizeof(bytes) / sizeof(bytes[0]);
  static_assert(nb <= SearchBuffers::kMax, "buffers of a search");
  void* const* buf = sb.ptr;
  double ms = -1.0;
  bool ok = true;
  for (int i = 0; i < nb && ok; ++i) ok = sb.get(i, bytes[i], s);
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (ok) ok = cudaEventCreate(&e0) == cudaSuccess && cudaEventCreate(&e1) == cudaSuccess;
  if (ok) ok = set_int_smem_limits(g, n, (int)rows.size(), false) == cudaSuccess;
  if (ok)
    ok = cudaMemcpyAsync(buf[13], rows.data(), rows.size() * sizeof(RowPair), cudaMemcpyHostToDevice, s) == cudaSuccess &&
         cudaStreamSynchronize(s) == cudaSuccess;
  if (ok) {
    IterArgs a{};
    a.N = N; a.M = M; a.W = W; a.H = H; a.G = 1; a.LO = 18; a.n = n;
    a.ll = (long long*)buf[0]; a.flags = (const unsigned char*)buf[1]; a.span = (const unsigned char*)buf[2];
    a.in.e = (const unsigned char*)buf[3]; a.Z = (DevCplx*)buf[4]; a.Z2 = (DevCplx*)buf[5];
    a.in.k1 = (const int4*)buf[6]; a.in.pair = (const int4*)buf[7]; a.in.k2 = (const int4*)buf[8];
    a.in.wf = (const int4*)buf[9]; a.in.wi = (const int4*)buf[10];
    a.in.hf = (const int4*)buf[11]; a.in.hi = (const int4*)buf[12];
    a.in.rows = (const int4*)buf[13]; a.status = (Status*)buf[14];
    gl_int_args(H, W, g, (int)rows.size(), &a.in);
    cudaStream_t q = s;
    cudaGraphExec_t exec = nullptr;
    auto launch = [&](int k) {
      bool fine = true;
      for (int i = 0; i < k && fine; ++i) fine = launch_int_iteration(a, g, q, false) == cudaSuccess;
      return fine;
    };
    if (replay) {  // (the default stream cannot be captured)
      q = nullptr;
      cudaGraph_t graph = nullptr;
      ok = cudaStreamCreateWithFlags(&q, cudaStreamNonBlocking) == cudaSuccess &&
           cudaStreamBeginCapture(q, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
      if (ok) {
        ok = launch(iters);
        ok = cudaStreamEndCapture(q, &graph) == cudaSuccess && ok && graph &&
             cudaGraphInstantiate(&exec, graph, 0) == cudaSuccess;
      }
      if (graph) cudaGraphDestroy(graph);
      ok = ok && cudaGraphLaunch(exec, q) == cudaSuccess;
    } else {
      ok = launch(2);
    }
    for (int round = 0; round < 3 && ok && !(ms > 1.33 * best_ms); ++round) {
      ok = cudaEventRecord(e0, q) == cudaSuccess;
      ok = ok && (exec ? cudaGraphLaunch(exec, q) == cudaSuccess : launch(iters));
      ok = ok && cudaEventRecord(e1, q) == cudaSuccess && cudaEventSynchronize(e1) == cudaSuccess;
      float t = 0.f;
      if (ok && cudaEventElapsedTime(&t, e0, e1) == cudaSuccess && (ms < 0.0 || t / iters < ms)) ms = t / iters;
    }
    if (replay && q) {
      cudaStreamSynchronize(q);
      cudaStreamDestroy(q);
    }
    if (exec) cudaGraphExecDestroy(exec);
  }
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  cudaStreamSynchronize(s);
  return ms;
}

// Layout of the integer form for M complex points on this device: the candidates of the
// layout model that it can run are timed, with two line buffers per column and in place,
// and the fastest kept, once per (M, SM count) per process.  Below 2^17 points lines are
// too few to fill the device and a pass is its chain of latencies: there the three fastest
// are also timed with radix-4 stages (more threads, shorter butterflies) and with a thread
// per two points (the loads, dicing and twiddles of a line side by side).  There launches one
// by one also hide up to 3 % between variants (N = 163840, rows of radices 4,4,4,4 and 8,8,4:
// both 28.7 us, replayed 23.1 and 23.7), and which of them a process ran was chance; so the
// best five within 4 % are timed again as replayed graphs.  H = 0: no layout.
struct IntTuned {
  int H = 0;
  IntVariant var;
  double ms = 1e300;
};
std::map<std::pair<int, int>, IntTuned> g_int_tune_cache;
constexpr int kIntLayoutsTimed = 8;

IntTuned autotune_int_layout(int M, int n, int sms, cudaStream_t s) {
  {
    std::lock_guard<std::mutex> lock(g_tune_mutex);
    auto it = g_int_tune_cache.find({M, sms});
    if (it != g_int_tune_cache.end()) return it->second;
  }
  IntTuned best;
  SearchBuffers sb;
  std::vector<std::pair<double, int>> timed;  // column lengths by their best time
  std::vector<IntTuned> tried;
  auto consider = [&](int H, const IntVariant& var) {
    const double ms = time_int_layout(M, H, var, n, M >= (1 << 18) ? 10 : 40, best.ms, sb, s);
    if (ms > 0.0) tried.push_back(IntTuned{H, var, ms});
    if (ms > 0.0 && ms < best.ms) best = tried.back();
    return ms;
  };
  for (const auto& c : ranked_layouts(M, sms)) {
    if (timed.size() == (size_t)kIntLayoutsTimed) break;
    double ms = -1.0;
    for (bool p : {false, true}) {
      IntVariant v;
      v.in_place = p;
      const double t = consider(c.second, v);
      if (t > 0.0 && (ms <= 0.0 || t < ms)) ms = t;
    }
    if (ms > 0.0) timed.emplace_back(ms, c.second);
  }
  std::sort(timed.begin(), timed.end());
  for (size_t i = 0; i < timed.size() && i < 3 && M < (1 << 17); ++i)
    for (int rc : {8, 4})
      for (int rr : {8, 4})
        for (bool wide : {false, true}) {
          if (rc == 8 && rr == 8 && !wide) continue;
          IntVariant v;
          v.rc = rc;
          v.rr = rr;
          v.wide = wide;
          consider(timed[i].second, v);
        }
  if (!best.H) return best;
  if (M < (1 << 17)) {
    std::sort(tried.begin(), tried.end(), [](const IntTuned& a, const IntTuned& b) { return a.ms < b.ms; });
    const double near = 1.04 * best.ms;
    double best_replay = 1e300;
    for (size_t i = 0; i < tried.size() && i < 5 && tried[i].ms <= near; ++i) {
      const double ms = time_int_layout(M, tried[i].H, tried[i].var, n, 16, 1e300, sb, s, true);
      if (ms > 0.0 && ms < best_replay) {
        best_replay = ms;
        best = tried[i];
      }
    }
  }
  std::lock_guard<std::mutex> lock(g_tune_mutex);
  g_int_tune_cache[{M, sms}] = best;
  return best;
}

// The integer form's layout for a plan whose layouts are timed; H = 0 where the FP64 form is
// faster.  The forms are compared as launched one by one, each search's winner timed three
// times more (a search times a variant once or a few times, and a hiccup of the host is 3 %);
// 2 % is what the FP64 form gains more from a captured graph at most.  Once per (M, SM count)
// per process.
std::map<std::pair<int, int>, bool> g_fp64_faster;
IntTuned timed_int_layout(int M, int n, int sms, cudaStream_t s) {
  IntTuned it = autotune_int_layout(M, n, sms, s);
  if (!it.H || M < kMinTimedFormM || gf_excess(M) <= kMaxSurePoly) return it;
  {
    std::lock_guard<std::mutex> lock(g_tune_mutex);
    auto known = g_fp64_faster.find({M, sms});
    if (known != g_fp64_faster.end()) {
      if (known->second) it.H = 0;
      return it;
    }
  }
  const TunedLayout t = autotune_layout(M, n, sms, s, nullptr);
  if (!t.H) return it;
  const int iters = M >= (1 << 18) ? 10 : 40;
  SearchBuffers sb;
  double fp64 = t.ms, integer = it.ms;
  for (int i = 0; i < 3; ++i) {
    const double f = time_layout(M, t.H, t.rc, t.rr, t.ip, t.pf, t.ws, t.row, n, sms, iters, sb, s);
    if (f > 0.0 && f < fp64) fp64 = f;
    const double k = time_int_layout(M, it.H, it.var, n, iters, 1e300, sb, s);
    if (k > 0.0 && k < integer) integer = k;
  }
  const bool faster = fp64 < 0.98 * integer;
  if (faster) it.H = 0;
  std::lock_guard<std::mutex> lock(g_tune_mutex);
  g_fp64_faster[{M, sms}] = faster;
  return it;
}

void free_plan(gl_plan* pl) {
  if (!pl) return;
  if (pl->device >= 0) cudaSetDevice(pl->device);
  if (pl->gexec) cudaGraphExecDestroy(pl->gexec);
  for (cudaGraphExec_t g : pl->hw_exec)
    if (g) cudaGraphExecDestroy(g);
  for (void* p : pl->allocs) cudaFree(p);
  if (pl->h_status) cudaFreeHost(pl->h_status);
  if (pl->h_res) cudaFreeHost(pl->h_res);
  if (pl->ev0) cudaEventDestroy(pl->ev0);
  if (pl->ev1) cudaEventDestroy(pl->ev1);
  if (pl->stream) cudaStreamDestroy(pl->stream);
  delete pl;
}

// One iteration on the plan's stream.  fp64: the FP64 form (its round-off is measured);
// else the integer form, for plans that have it.  A state loaded by the caller
// (from_state) may hold words the integer form has no bound for, and runs in FP64.
int launch_iteration(gl_plan* pl, bool fp64) {
  cudaError_t e;
  if (pl->mode == GL_MODE_PLAIN) {
    e = launch_plain_iteration(pl->args, pl->pg, pl->stream);
  } else if (pl->int_form && !fp64 && !pl->from_state) {
    e = launch_int_iteration(pl->args, pl->ig, pl->stream, false);
  } else {
    e = launch_fused_iteration(pl->args, pl->fg, pl->stream, pl->from_state);
    pl->from_state = false;
  }
  return e == cudaSuccess ? GL_OK : GL_ERR_CUDA;
}

// k iterations; an integer-form plan runs one in kFp64Every in FP64
int launch_iterations(gl_plan* pl, int64_t k) {
  for (int64_t i = 0; i < k; ++i) {
    const bool fp64 = pl->from_state || ++pl->since_fp64 >= kFp64Every;
    const int rc = launch_iteration(pl, fp64);
    if (rc != GL_OK) return rc;
    if (fp64) pl->since_fp64 = 0;
  }
  return GL_OK;
}

// Enqueue k iterations, with batches of kGraphBatch replayed from one CUDA graph (in an
// integer-form plan the last of the batch is the FP64 one).
int enqueue(gl_plan* pl, int64_t k) {
  if (k <= 0) return GL_OK;
  int rc;
  if (pl->from_state) {  // the state-loading first pass is never captured
    if ((rc = launch_iterations(pl, 1)) != GL_OK) return rc;
    --k;
  }
  if (pl->resident) {  // one cluster launch runs them all, or all up to the next FP64 one
    while (k > 0) {
      const int left = kFp64Every - 1 - pl->since_fp64;
      if (pl->int_form && left > 0) {
        const int chunk = (int)std::min<int64_t>(k, left);
        GL_CUDA(launch_int_resident(pl->args, pl->irg, chunk, pl->stream));
        pl->since_fp64 += chunk;
        k -= chunk;
        continue;
      }
      const int chunk = pl->int_form ? 1 : (int)std::min<int64_t>(k, 1 << 30);
      GL_CUDA(launch_resident(pl->args, pl->rg, chunk, pl->stream));
      pl->since_fp64 = 0;
      k -= chunk;
    }
    return GL_OK;
  }
  if (pl->use_graphs && k >= kGraphBatch) {
    if (!pl->gexec) {
      cudaGraph_t graph = nullptr;
      GL_CUDA(cudaStreamBeginCapture(pl->stream, cudaStreamCaptureModeThreadLocal));
      int lrc = GL_OK;
      for (int i = 0; i < kGraphBatch && lrc == GL_OK; ++i) lrc = launch_iteration(pl, i == kGraphBatch - 1);
      cudaError_t ec = cudaStreamEndCapture(pl->stream, &graph);
      if (lrc != GL_OK || ec != cudaSuccess) {
        if (graph) cudaGraphDestroy(graph);
        return GL_ERR_CUDA;
      }
      cudaError_t ei = cudaGraphInstantiate(&pl->gexec, graph, 0);
      cudaGraphDestroy(graph);
      if (ei != cudaSuccess) {
        pl->gexec = nullptr;
        return GL_ERR_CUDA;
      }
      pl->gexec_iters = kGraphBatch;
    }
    while (k >= pl->gexec_iters) {
      GL_CUDA(cudaGraphLaunch(pl->gexec, pl->stream));
      k -= pl->gexec_iters;
      pl->since_fp64 = 0;
    }
  }
  return launch_iterations(pl, k);
}

// Wait for the stream and fold the device status into the plan.
int read_status(gl_plan* pl, double* maxerr_out) {
  GL_CUDA(cudaMemcpyAsync(pl->h_status, pl->args.status, sizeof(Status), cudaMemcpyDeviceToHost, pl->stream));
  GL_CUDA(cudaStreamSynchronize(pl->stream));
  const double e = std::ldexp((double)pl->h_status->maxerr64, -64);
  if (e > pl->run_maxerr) pl->run_maxerr = e;
  if (maxerr_out) *maxerr_out = e;
  if (pl->h_status->flags & kStatusTimeout) return GL_ERR_TIMEOUT;
  if (pl->h_status->flags) return GL_ERR_OVERFLOW;
  if (e >= pl->error_limit) return GL_ERR_ROUNDOFF;
  return GL_OK;
}

}  // namespace

extern "C" {

int gl_version(void) { return 100; }

const char* gl_error_string(int s) {
  switch (s) {
    case GL_OK: return "ok";
    case GL_ERR_ARG: return "bad argument";
    case GL_ERR_RATIO: return "p/N outside the carry-depth table (ratio >= 22)";
    case GL_ERR_SIZE: return "N must be even with N/2 = 2^a 3^b 5^c 7^d and a usable FFT layout";
    case GL_ERR_CUDA: return "CUDA runtime error";
    case GL_ERR_NOMEM: return "out of memory";
    case GL_ERR_ROUNDOFF: return "round-off error reached the limit";
    case GL_ERR_OVERFLOW: return "product out of the exactly representable / sliced range";
    case GL_ERR_NODEVICE: return "no CUDA device";
    case GL_ERR_IO: return "checkpoint I/O error";
    case GL_ERR_CHECKPOINT: return "checkpoint does not match the test";
    case GL_ERR_STATE: return "call not valid in this state";
    case GL_ERR_TOO_LARGE: return "N exceeds 65536, the limit of gl_iterate_noalloc";
    case GL_ERR_TIMEOUT: return "a bounded device-side wait ran out";
    default: return "unknown status";
  }
}

int gl_default_opts(gl_plan_opts* o) {
  if (!o) return GL_ERR_ARG;
  std::memset(o, 0, sizeof(*o));
  o->mode = GL_MODE_FUSED;
  o->device = 0;
  o->error_limit = 0.4;
  o->check_every = 1000;
  o->use_graphs = 1;
  o->autotune = 1;
  return GL_OK;
}

int setSliceAndDice(int testPrime, int signalSize) {
  if (testPrime <= 2 || signalSize <= 0) return GL_ERR_ARG;
  int n = slice_depth(testPrime, signalSize);
  return n < 0 ? GL_ERR_RATIO : n;
}

int gl_plan_create(int p, int N, const gl_plan_opts* opts, gl_plan** out) {
  return gl_plan_create_ex(p, N, opts, opts && opts->batch_layout ? 1 : 0, out);
}

}  // extern "C"

cudaError_t gl_make_stream(cudaStream_t* s, int level) {
  int least = 0, greatest = 0;
  if (level) {
    const cudaError_t e = cudaDeviceGetStreamPriorityRange(&least, &greatest);
    if (e != cudaSuccess) return e;
  }
  const int prio = level == 1 ? greatest : (level == 2 ? (greatest + least) / 2 : least);
  return cudaStreamCreateWithPriority(s, cudaStreamNonBlocking, prio);
}

void gl_int_args(int H, int W, const IntGeom& g, int nrows, IntArgs* in) {
  in->nrows = nrows;
  in->touch = int_touch(H, W);
  in->t = g.t;
  in->V = W / g.t;
  in->qV = (int)(((1ull << 61) - 1) % (uint64_t)in->V);
  in->ls_col = int_stride(H);
  in->ls_row = int_stride(in->V);
  in->pw = g.pw;
  in->ph = g.ph;
}

bool gl_int_layout(int p, int N, int* H, IntGeom* g) {
  int vmax = 0;
  if (!int_range_ok(p, N, &vmax) || !int_roundoff_ok(p, N, 0.4)) return false;
  const int M = N / 2;
  if (!(*H = first_int_layout(M, kSms))) return false;
  return choose_int_geom(*H, M / *H, g, untimed_variant(*H, M / *H));
}

void gl_plan_note_external_iterations(gl_plan* pl, int64_t iters) {
  pl->iters_done += iters;
  pl->from_state = false;
  pl->carry_valid = pl->mode == GL_MODE_PLAIN;
}

double gl_model_iteration_cost(int M, int sms) {
  const auto r = ranked_layouts(M, sms);
  return r.empty() ? HUGE_VAL : r.front().first;
}

double gl_plan_unit_cost(const gl_plan* pl, bool row) {
  if (row) return 2.0 * pl->fg.W * (2.0 * line_ops(pl->fg.pw) + 16.0);
  return pl->fg.H * (line_ops(pl->fg.ph) + 6.0);
}

// Options that choose among the FP64 form's layouts and kernels: such a plan runs them in
// every iteration.
static bool names_fp64_variant(const gl_plan_opts& o) {
  return o.fft_h || o.cols_per_cta || o.max_radix_col || o.max_radix_row || o.resident > 0 || o.col_inplace ||
         o.row_pass;
}

// Whether a plan of (p, N) with these options is to run the integer form (where a layout
// for it is found).
static bool wants_int_form(int p, int N, const gl_plan_opts& o, int* vmax) {
  return o.mode == GL_MODE_FUSED && !o.batch_layout && !names_fp64_variant(o) && int_range_ok(p, N, vmax) &&
         int_roundoff_ok(p, N, o.error_limit);
}

// Device bytes of the integer form's tables for an H x W layout.
static size_t int_table_bytes(int H, int W, const IntGeom& g) {
  LinePlan pw = g.pw, ph = g.ph;
  const size_t M = (size_t)H * W;
  std::vector<RowPair> rows;
  gf_row_pairs(W / g.t, H, rows);
  return (2 * M + M / g.t) * 16 + 2 * M /* exponents */ + 2 * 16 * ((size_t)int_stage_offsets(&pw) + int_stage_offsets(&ph)) +
         rows.size() * sizeof(RowPair);
}

static int build_int_tables(gl_plan* pl, int vmax) {
  const int W = pl->fg.W, H = pl->fg.H, N = pl->N, t = pl->ig.t, V = W / t;
  std::vector<HostTw> k1, pair, k2, wf, wi, hf, hi;
  std::vector<RowPair> rows;
  std::vector<uint8_t> e, e_c((size_t)N);
  int off[8];
  gf_pass_tables(W, H, t, k1, pair, k2);
  gf_row_pairs(V, H, rows);
  gf_weights(pl->p, N, e);
  gf_stage_twiddles(pl->ig.pw.radix, pl->ig.pw.nst, false, wf, off);
  gf_stage_twiddles(pl->ig.pw.radix, pl->ig.pw.nst, true, wi, off);
  gf_stage_twiddles(pl->ig.ph.radix, pl->ig.ph.nst, false, hf, off);
  gf_stage_twiddles(pl->ig.ph.radix, pl->ig.ph.nst, true, hi, off);
  for (int m1 = 0, c = 0; m1 < W; ++m1)  // column-major, as the other per-word tables
    for (int m2 = 0; m2 < H; ++m2, c += 2) {
      e_c[c] = e[2 * (m1 + (size_t)W * m2)];
      e_c[c + 1] = e[2 * (m1 + (size_t)W * m2) + 1];
    }
  IntArgs& in = pl->args.in;
  auto up = [&](auto** dst, const void* src, size_t count) {
    using T = std::remove_const_t<std::remove_pointer_t<std::remove_pointer_t<decltype(dst)>>>;
    T* d = nullptr;
    const int rc = dev_alloc(pl, &d, count);
    if (rc != GL_OK) return rc;
    *dst = d;
    return cuda_status(cudaMemcpyAsync(d, src, count * sizeof(T), cudaMemcpyHostToDevice, pl->stream));
  };
  static_assert(sizeof(HostTw) == sizeof(int4) && sizeof(RowPair) == sizeof(int4), "table entries");
  int rc;
  if ((rc = up(&in.k1, k1.data(), k1.size())) || (rc = up(&in.pair, pair.data(), pair.size())) ||
      (rc = up(&in.k2, k2.data(), k2.size())) || (rc = up(&in.wf, wf.data(), wf.size())) ||
      (rc = up(&in.wi, wi.data(), wi.size())) || (rc = up(&in.hf, hf.data(), hf.size())) ||
      (rc = up(&in.hi, hi.data(), hi.size())) || (rc = up(&in.rows, rows.data(), rows.size())) ||
      (rc = up(&in.e, e_c.data(), e_c.size())))
    return rc;
  GL_CUDA(cudaStreamSynchronize(pl->stream));  // host tables go out of scope
  gl_int_args(H, W, pl->ig, (int)rows.size(), &in);
  in.vmax = vmax;
  in.check_span = (pl->n + 1) * pl->LO < 51;
  GL_CUDA(set_int_smem_limits(pl->ig, pl->n, (int)rows.size(), true));
  pl->int_form = true;
  return GL_OK;
}

int gl_plan_create_ex(int p, int N, const gl_plan_opts* opts, int sms_override, gl_plan** out, bool fp64_only) {
  if (!out) return GL_ERR_ARG;
  *out = nullptr;
  gl_plan_opts o;
  if (opts) o = *opts;
  else gl_default_opts(&o);
  if (N == 0 && p >= 3) {
    int rc0 = gl_find_signal_size(p, &o, &N, nullptr, nullptr);
    if (rc0 != GL_OK) return rc0;
  }
  if (p < 3 || N < 16 || (N & 1) || N > p) return GL_ERR_ARG;
  if (o.mode != GL_MODE_FUSED && o.mode != GL_MODE_PLAIN) return GL_ERR_ARG;
  if (!(o.error_limit > 0.0 && o.error_limit <= 0.5) || o.check_every < 1) return GL_ERR_ARG;
  if (o.high_priority < 0 || o.high_priority > 2) return GL_ERR_ARG;
  const int n = slice_depth(p, N);
  if (n < 0) return GL_ERR_RATIO;
  const int M = N / 2;
  FusedGeom fg{};
  PlainGeom pg{};
  if (o.cols_per_cta > 1) return GL_ERR_ARG;  // the column passes take one column per CTA
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return GL_ERR_NODEVICE;
  if (o.device < 0 || o.device >= ndev) return GL_ERR_ARG;
  if (cudaSetDevice(o.device) != cudaSuccess) return GL_ERR_CUDA;
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, o.device) != cudaSuccess) return GL_ERR_CUDA;
  if (sms_override > 0) sms = sms_override;
  int force_h = o.fft_h, cap_c = kMaxRadix, cap_r = kMaxRadix;
  model_caps(M, o, sms_override, &cap_c, &cap_r);
  // Short lengths: the resident form (one cluster, the whole test in shared memory) when
  // a layout with W divisible by the cluster size fits; it replaces the layout search.
  bool resident = false;
  ResidentGeom rg{};
  int vmax = 0;
  // The integer form, unless an option names a variant of the FP64 kernels.
  bool int_form = !fp64_only && !sms_override && wants_int_form(p, N, o, &vmax);
  IntGeom ig{};
  IntVariant int_var;
  IntResidentGeom irg{};
  if (o.mode == GL_MODE_FUSED && !sms_override && !force_h &&
      (o.resident > 0 ? N <= kResidentMaxN : (o.resident == 0 && N <= kResidentAutoN))) {
    // radix 4: each CTA's lines are short, and more, shorter butterflies keep more warps
    // issuing FP64 work (measured: 13.8 us at N = 2048 against 16.6 us with radix 8)
    const int rcap = o.max_radix_col ? o.max_radix_col : 4, wcap = o.max_radix_row ? o.max_radix_row : 4;
    IntVariant var;
    var.rc = var.rr = 8;
    // a layout both forms can run; failing that, any for FP64 alone
    bool int_resident = int_form;
    auto ranked = ranked_layouts(M, sms);
    if (int_form) {
      const auto all = ranked;
      ranked.insert(ranked.end(), all.begin(), all.end());
    }
    size_t tried = 0;
    const size_t first_round = int_form ? ranked.size() / 2 : 0;
    for (const auto& c : ranked) {
      int_resident = int_form && tried++ < first_round;
      FusedGeom t{};
      if (choose_fused_geom(M, c.second, sms, &t, rcap, wcap) != GL_OK) continue;
      if (int_resident) {
        if (!choose_int_geom(t.H, t.W, &ig, var)) continue;
        LinePlan pw = ig.pw, ph = ig.ph;
        const int hn = int_stage_offsets(&ph), wn = int_stage_offsets(&pw);
        if (int_resident_geom(t.H, t.W, ig, hn, wn, n, &irg) != cudaSuccess) continue;
      }
      int offh[8], offw[8];
      const int nh = stage_offsets(t.ph, offh), nw = stage_offsets(t.pw, offw);
      if (resident_geom(t, nh, nw, n, &rg) == cudaSuccess) {
        resident = true;
        int_form = int_resident;
        int_var = var;
        force_h = c.second;
        cap_c = rcap;
        cap_r = wcap;
        break;
      }
    }
    cudaGetLastError();
  }
  if (o.resident > 0 && !resident) return GL_ERR_SIZE;
  if (int_form && !resident) {
    IntTuned it;
    if (o.autotune && !sms_override) it = timed_int_layout(M, n, sms, 0);
    else if (int_pays_untimed(M)) {
      it.H = first_int_layout(M, sms);
      if (it.H) it.var = untimed_variant(it.H, M / it.H);
    }
    force_h = it.H;
    int_var = it.var;
    int_form = it.H != 0;
  }
  bool col_ip = false, col_pf = false, col_ws = false;
  int row_var = 0;
  if (o.mode == GL_MODE_FUSED && (!force_h || (int_form && !resident)) && o.autotune && !sms_override) {
    const TunedLayout t = autotune_layout(M, n, sms, 0, nullptr, force_h);
    if (t.H) {
      force_h = t.H;
      if (!o.max_radix_col) cap_c = t.rc;
      if (!o.max_radix_row) cap_r = t.rr;
      col_ip = t.ip && !resident;
      col_pf = col_ip && t.pf;
      col_ws = col_ip && t.ws;
      row_var = resident ? 0 : t.row;
    }
  }
  if (o.row_pass) {
    if (o.row_pass < -1 || o.row_pass > 2) return GL_ERR_ARG;
    row_var = o.row_pass > 0 && !resident ? o.row_pass : 0;
  }
  if (o.col_inplace) {
    if (o.col_inplace > 4) return GL_ERR_ARG;
    col_ip = o.col_inplace > 0 && !resident && !sms_override;
    col_pf = col_ip && (o.col_inplace == 2 || o.col_inplace == 4);
    col_ws = col_ip && (o.col_inplace == 3 || o.col_inplace == 4);
  }
  int rc = o.mode == GL_MODE_FUSED
               ? choose_fused_geom(M, force_h, sms, &fg, cap_c, cap_r, col_ip, col_pf, col_ws, row_var)
               : choose_plain_geom(M, &pg);
  if (rc == GL_ERR_SIZE && col_ip && o.col_inplace <= 0)  // the searched layout cannot: two buffers
    rc = choose_fused_geom(M, force_h, sms, &fg, cap_c, cap_r, false);
  if (rc != GL_OK) return rc;
  int_form = int_form && choose_int_geom(fg.H, fg.W, &ig, int_var);

  gl_plan* pl = new (std::nothrow) gl_plan();
  if (!pl) return GL_ERR_NOMEM;
  pl->p = p; pl->N = N; pl->M = M; pl->LO = p / N; pl->n = n;
  pl->mode = o.mode; pl->device = o.device;
  pl->error_limit = o.error_limit; pl->check_every = o.check_every; pl->use_graphs = o.use_graphs;
  pl->fg = fg; pl->pg = pg; pl->ig = ig; pl->irg = irg;

#define GL_TRY(x)             \
  do {                        \
    int r_ = (x);             \
    if (r_ != GL_OK) {        \
      free_plan(pl);          \
      return r_;              \
    }                         \
  } while (0)
#define GL_TRYC(x) GL_TRY(cuda_status(x))

  GL_TRYC(gl_make_stream(&pl->stream, o.high_priority));
  GL_TRYC(cudaEventCreate(&pl->ev0));
  GL_TRYC(cudaEventCreate(&pl->ev1));
  GL_TRYC(cudaMallocHost((void**)&pl->h_status, sizeof(Status)));

  std::vector<int32_t> bits;
  std::vector<uint8_t> flags;
  std::vector<double> A, Ainv;
  std::vector<HostCplx> twM;
  word_tables(p, N, bits, flags);
  // the row pass produces V = DFT_M(z_even + i z_odd) exactly, so the unnormalized
  // inverse returns M z: Ainv = 1/(M A) (the reference's (1/A)/N with N = 2M)
  weight_tables(p, N, (double)M, A, Ainv);
  twiddle_table(M, twM);

  IterArgs& a = pl->args;
  a.N = N; a.M = M; a.LO = pl->LO; a.n = n;
  long long* ll;
  unsigned char *fl, *span = nullptr;
  double *dA, *dAi;
  DevCplx *Z, *Z2 = nullptr, *dtwM = nullptr, *dtwW = nullptr, *dtwH = nullptr;
  DevCplx *dK1 = nullptr, *dPair = nullptr, *dK2 = nullptr;
  int* digit;
  signed char* hi;
  Status* status;
  GL_TRY(dev_alloc(pl, &ll, N));
  GL_TRY(dev_alloc(pl, &fl, N));
  GL_TRY(dev_alloc(pl, &dA, N));
  GL_TRY(dev_alloc(pl, &dAi, N));
  GL_TRY(dev_alloc(pl, &Z, M));
  GL_TRY(dev_alloc(pl, &digit, N));
  GL_TRY(dev_alloc(pl, &hi, N));
  GL_TRY(dev_alloc(pl, &status, 1));
  GL_TRY(dev_alloc(pl, &pl->rscratch, residue_scratch_bytes(N)));
  GL_TRYC(cudaMallocHost((void**)&pl->h_res, sizeof(int32_t) * 72));
  if (o.mode == GL_MODE_PLAIN) {
    std::vector<HostCplx> pc((size_t)M);
    parallel_for(M, [&](int64_t b, int64_t e) {
      for (int64_t k = b; k < e; ++k) pc[k] = pair_coeff(k, M);
    });
    GL_TRY(dev_alloc(pl, &Z2, M));
    GL_TRY(dev_alloc(pl, &dtwM, M));
    GL_TRY(dev_alloc(pl, &dPair, M));
    GL_TRYC(cudaMemcpyAsync(dtwM, twM.data(), sizeof(DevCplx) * M, cudaMemcpyHostToDevice, pl->stream));
    GL_TRYC(cudaMemcpyAsync(dPair, pc.data(), sizeof(DevCplx) * M, cudaMemcpyHostToDevice, pl->stream));
    GL_TRYC(cudaMemcpyAsync(fl, flags.data(), N, cudaMemcpyHostToDevice, pl->stream));
    GL_TRYC(cudaMemcpyAsync(dA, A.data(), sizeof(double) * N, cudaMemcpyHostToDevice, pl->stream));
    GL_TRYC(cudaMemcpyAsync(dAi, Ainv.data(), sizeof(double) * N, cudaMemcpyHostToDevice, pl->stream));
    GL_TRYC(cudaStreamSynchronize(pl->stream));  // host tables go out of scope
  } else {
    const int W = fg.W, H = fg.H;
    // per-word tables in column-major order: word j = 2(m1 + W m2) + e -> 2(m1 H + m2) + e
    std::vector<uint8_t> fl_c(N), span_c(N);
    std::vector<double> A_c(N), Ai_c(N);
    for (int j = 0; j < N; ++j) {
      const int m = j >> 1, m1 = m % W, m2 = m / W;
      const int c = 2 * (m1 * H + m2) + (j & 1);
      fl_c[c] = flags[j];
      A_c[c] = A[j];
      Ai_c[c] = Ainv[j];
      int tot = 0;
      for (int i = 0; i <= n; ++i) tot += bits[(j + i) % N];
      span_c[c] = (uint8_t)(tot > 255 ? 255 : tot);
    }
    std::vector<int> rw(fg.pw.radix, fg.pw.radix + fg.pw.nst), rh(fg.ph.radix, fg.ph.radix + fg.ph.nst);
    std::vector<HostCplx> twW, twH, tK1((size_t)M), tPair((size_t)M), tK2((size_t)M);
    stage_twiddles(W, rw, twW, fg.pw.off);
    stage_twiddles(H, rh, twH, fg.ph.off);
    parallel_for(H, [&](int64_t b, int64_t e) {
      for (int64_t k2 = b; k2 < e; ++k2)
        for (int m1 = 0; m1 < W; ++m1) {
          const HostCplx w = twM[(size_t)m1 * k2];   // m1 * k2 < M
          tK1[(size_t)m1 * H + k2] = w;
          tK2[(size_t)k2 * W + m1] = w;
          tPair[(size_t)k2 * W + m1] = pair_coeff(k2 + (int64_t)H * m1, M);
        }
    });
    pl->fg = fg;
    GL_TRY(dev_alloc(pl, &Z2, M));  // the row pass's output, column-major
    GL_TRY(dev_alloc(pl, &span, N));
    GL_TRY(dev_alloc(pl, &dtwW, twW.size()));
    GL_TRY(dev_alloc(pl, &dtwH, twH.size()));
    GL_TRY(dev_alloc(pl, &dK1, M));
    GL_TRY(dev_alloc(pl, &dPair, M));
    GL_TRY(dev_alloc(pl, &dK2, M));
    GL_TRYC(cudaMemcpyAsync(fl, fl_c.data(), N, cudaMemcpyHostToDevice, pl->stream));
    GL_TRYC(cudaMemcpyAsync(span, span_c.data(), N, cudaMemcpyHostToDevice, pl->stream));
    GL_TRYC(cudaMemcpyAsync(dA, A_c.data(), sizeof(double) * N, cudaMemcpyHostToDevice, pl->stream));
    GL_TRYC(cudaMemcpyAsync(dAi, Ai_c.data(), sizeof(double) * N, cudaMemcpyHostToDevice, pl->stream));
    GL_TRYC(cudaMemcpyAsync(dtwW, twW.data(), sizeof(DevCplx) * twW.size(), cudaMemcpyHostToDevice, pl->stream));
    GL_TRYC(cudaMemcpyAsync(dtwH, twH.data(), sizeof(DevCplx) * twH.size(), cudaMemcpyHostToDevice, pl->stream));
    GL_TRYC(cudaMemcpyAsync(dK1, tK1.data(), sizeof(DevCplx) * M, cudaMemcpyHostToDevice, pl->stream));
    GL_TRYC(cudaMemcpyAsync(dPair, tPair.data(), sizeof(DevCplx) * M, cudaMemcpyHostToDevice, pl->stream));
    GL_TRYC(cudaMemcpyAsync(dK2, tK2.data(), sizeof(DevCplx) * M, cudaMemcpyHostToDevice, pl->stream));
    GL_TRYC(cudaStreamSynchronize(pl->stream));  // host tables go out of scope
    a.W = W; a.H = H; a.G = 1; a.pw = pl->fg.pw; a.ph = pl->fg.ph; a.ls_col = fg.ls_col; a.ls_row = fg.ls_row;
    a.twW_n = (int)twW.size();
    // the row pass copies the whole table behind its four line buffers (unless it reads
    // the table through L1)
    if ((size_t)4 * fg.ls_row * 16 + (fg.row_var == 2 ? 0 : twW.size() * sizeof(DevCplx)) != fg.sm_row)
      GL_TRY(GL_ERR_SIZE);
    GL_TRYC(set_fused_smem_limits(fg));
    if (resident) {
      if (rg.twH_n != (int)twH.size() || rg.twW_n != (int)twW.size()) GL_TRY(GL_ERR_SIZE);
      pl->resident = true;
      pl->rg = rg;
    }
  }
  a.ll = ll; a.flags = fl; a.span = span; a.A = dA; a.Ainv = dAi; a.Z = Z; a.Z2 = Z2;
  a.twM = dtwM; a.twW = dtwW; a.twH = dtwH; a.twK1 = dK1; a.twPair = dPair; a.twK2 = dK2;
  a.digit = digit; a.hi = hi; a.status = status;
  if (int_form) {
    const size_t held = pl->allocs.size(), bytes = pl->device_bytes;
    const int ri = build_int_tables(pl, vmax);
    if (ri == GL_ERR_NOMEM) {  // its tables do not fit beside the FP64 form's: FP64 alone
      for (; pl->allocs.size() > held; pl->allocs.pop_back()) cudaFree(pl->allocs.back());
      pl->device_bytes = bytes;
      a.in = IntArgs{};
    } else {
      GL_TRY(ri);
    }
  }
  *out = pl;
  int r = gl_reset(pl);
  if (r != GL_OK) {
    free_plan(pl);
    *out = nullptr;
    return r;
  }
  return GL_OK;
#undef GL_TRY
#undef GL_TRYC
}

int gl_plan_describe_ex(int p, int N, const gl_plan_opts* opts, gl_plan_info* info, bool fp64_only) {
  if (!info) return GL_ERR_ARG;
  gl_plan_opts o;
  if (opts) o = *opts;
  else gl_default_opts(&o);
  if (p < 3 || N < 16 || (N & 1) || N > p) return GL_ERR_ARG;
  if (o.mode != GL_MODE_FUSED && o.mode != GL_MODE_PLAIN) return GL_ERR_ARG;
  const int n = slice_depth(p, N);
  if (n < 0) return GL_ERR_RATIO;
  gl_plan tmp;
  tmp.p = p; tmp.N = N; tmp.M = N / 2; tmp.LO = p / N; tmp.n = n; tmp.mode = o.mode;
  if (o.cols_per_cta > 1) return GL_ERR_ARG;
  int sms = 0, ndev = 0;
  if (cudaGetDeviceCount(&ndev) == cudaSuccess && ndev > 0 && o.device >= 0 && o.device < ndev)
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, o.device);
  if (sms <= 0) sms = 152;  // GB300
  if (o.batch_layout) sms = 1;
  int cap_c = kMaxRadix, cap_r = kMaxRadix;
  model_caps(tmp.M, o, o.batch_layout ? 1 : 0, &cap_c, &cap_r);
  int vmax = 0;
  const bool int_form = !fp64_only && wants_int_form(p, N, o, &vmax);
  const int int_h = int_form && int_pays_untimed(tmp.M) ? first_int_layout(tmp.M, sms) : 0;
  int rc = o.mode == GL_MODE_FUSED ? choose_fused_geom(tmp.M, int_h ? int_h : o.fft_h, sms, &tmp.fg, cap_c, cap_r)
                                   : choose_plain_geom(tmp.M, &tmp.pg);
  if (rc != GL_OK) return rc;
  tmp.device = -1;
  int r = gl_plan_get_info(&tmp, info);
  if (o.mode == GL_MODE_FUSED) {
    const size_t M = tmp.M, N8 = (size_t)N * 8;
    const size_t stages = (size_t)stage_offsets(tmp.fg.pw, tmp.fg.pw.off) + stage_offsets(tmp.fg.ph, tmp.fg.ph.off);
    info->device_bytes = N8 /*ll*/ + 2 * (size_t)N /*flags, span*/ + 2 * N8 /*A, Ainv*/ +
                         5 * M * 16 /*Z, Z2, 3 twiddle tables*/ + stages * 16 + (size_t)N * 5 /*digit, hi*/ +
                         sizeof(Status) + residue_scratch_bytes(N);
    IntGeom ig{};
    if (int_h && choose_int_geom(tmp.fg.H, tmp.fg.W, &ig))
      info->device_bytes += int_table_bytes(tmp.fg.H, tmp.fg.W, ig);
  }
  return r;
}

extern "C" {

int gl_plan_describe(int p, int N, const gl_plan_opts* opts, gl_plan_info* info) {
  return gl_plan_describe_ex(p, N, opts, info, false);
}

int gl_plan_destroy(gl_plan* plan) {
  if (!plan) return GL_ERR_ARG;
  free_plan(plan);
  return GL_OK;
}

int gl_plan_get_info(const gl_plan* pl, gl_plan_info* info) {
  if (!pl || !info) return GL_ERR_ARG;
  std::memset(info, 0, sizeof(*info));
  info->p = pl->p; info->N = pl->N;
  info->lo_bits = pl->LO; info->hi_bits = pl->LO + 1;
  info->carry_depth = pl->n; info->mode = pl->mode;
  if (pl->mode == GL_MODE_FUSED) {
    info->fft_w = pl->fg.W; info->fft_h = pl->fg.H; info->cols_per_cta = pl->fg.col_ws ? 2 : pl->fg.G;
    info->col_variant = !pl->fg.col_ip ? -1 : pl->fg.col_ws ? (pl->fg.col_pf ? 4 : 3) : (pl->fg.col_pf ? 2 : 1);
    info->row_variant = pl->fg.row_var ? pl->fg.row_var : -1;
    for (int i = 0; i < pl->fg.pw.nst; ++i) info->radix_w[i] = pl->fg.pw.radix[i];
    for (int i = 0; i < pl->fg.ph.nst; ++i) info->radix_h[i] = pl->fg.ph.radix[i];
    info->threads_col = pl->fg.t_col; info->threads_row = pl->fg.t_row;
    info->smem_col = (int)pl->fg.sm_col; info->smem_row = (int)pl->fg.sm_row;
  } else {
    info->fft_w = pl->M; info->fft_h = 1;
    for (int i = 0; i < pl->pg.nst && i < 8; ++i) info->radix_w[i] = pl->pg.radix[i];
  }
  info->device_bytes = pl->device_bytes;
  info->resident_ctas = pl->resident ? pl->rg.C : 0;
  info->resident_smem = pl->resident ? pl->rg.smem : 0;
  return GL_OK;
}

int gl_plan_int_info(const gl_plan* pl, gl_int_info* info) {
  if (!pl || !info) return GL_ERR_ARG;
  std::memset(info, 0, sizeof(*info));
  if (!pl->int_form) return GL_OK;
  const IntGeom& g = pl->ig;
  info->integer = 1;
  info->fp64_every = kFp64Every;
  info->poly = g.t;
  info->col_inplace = g.col_p;
  for (int i = 0; i < g.pw.nst; ++i) info->radix_w[i] = g.pw.radix[i];
  for (int i = 0; i < g.ph.nst; ++i) info->radix_h[i] = g.ph.radix[i];
  info->threads_col = g.t_col; info->threads_row = g.t_row;
  info->smem_col = (int)g.sm_col; info->smem_row = (int)g.sm_row;
  info->resident_ctas = pl->resident ? pl->irg.C : 0;
  info->resident_smem = pl->resident ? pl->irg.smem : 0;
  return GL_OK;
}

int gl_reset(gl_plan* pl) {
  if (!pl) return GL_ERR_ARG;
  GL_CUDA(cudaSetDevice(pl->device));
  GL_CUDA(launch_set_initial(pl->args, pl->mode, pl->stream));
  GL_CUDA(cudaMemsetAsync(pl->args.status, 0, sizeof(Status), pl->stream));
  GL_CUDA(cudaStreamSynchronize(pl->stream));
  pl->iters_done = 0;
  pl->since_fp64 = 0;
  pl->run_maxerr = 0.0;
  pl->from_state = false;
  pl->carry_valid = true;
  return GL_OK;
}

int gl_iterate(gl_plan* pl, int64_t iters, gl_iter_report* rep) {
  if (!pl || iters < 0) return GL_ERR_ARG;
  GL_CUDA(cudaSetDevice(pl->device));
  double call_max = 0.0;
  int status = GL_OK;
  int64_t done = 0;
  GL_CUDA(cudaEventRecord(pl->ev0, pl->stream));
  if (pl->mode == GL_MODE_PLAIN && !pl->carry_valid && iters > 0) {
    GL_CUDA(launch_dice(pl->args, pl->stream));
    pl->carry_valid = true;
  }
  while (done < iters) {
    const int64_t b = iters - done < pl->check_every ? iters - done : pl->check_every;
    int rc = enqueue(pl, b);
    if (rc != GL_OK) return rc;
    done += b;
    pl->iters_done += b;
    pl->carry_valid = pl->mode == GL_MODE_PLAIN;
    double e = 0.0;
    status = read_status(pl, &e);
    if (status == GL_ERR_CUDA) return status;
    if (e > call_max) call_max = e;
    if (status != GL_OK) break;
  }
  GL_CUDA(cudaEventRecord(pl->ev1, pl->stream));
  GL_CUDA(cudaEventSynchronize(pl->ev1));
  float ms = 0.f;
  GL_CUDA(cudaEventElapsedTime(&ms, pl->ev0, pl->ev1));
  if (rep) {
    rep->iterations = done;
    rep->total_iterations = pl->iters_done;
    rep->max_roundoff = call_max;
    rep->ms = ms;
    rep->status = status;
  }
  return status;
}

int gl_plan_stream(gl_plan* pl, void** cuda_stream) {
  if (!pl || !cuda_stream) return GL_ERR_ARG;
  *cuda_stream = (void*)pl->stream;
  return GL_OK;
}

int gl_enqueue(gl_plan* pl, int64_t iters) {
  if (!pl || iters < 0) return GL_ERR_ARG;
  GL_CUDA(cudaSetDevice(pl->device));
  if (pl->mode == GL_MODE_PLAIN && !pl->carry_valid && iters > 0) {
    GL_CUDA(launch_dice(pl->args, pl->stream));
    pl->carry_valid = true;
  }
  int rc = enqueue(pl, iters);
  if (rc != GL_OK) return rc;
  pl->iters_done += iters;
  if (iters > 0) pl->carry_valid = pl->mode == GL_MODE_PLAIN;
  return GL_OK;
}

int gl_sync_status(gl_plan* pl, gl_iter_report* rep) {
  if (!pl) return GL_ERR_ARG;
  GL_CUDA(cudaSetDevice(pl->device));
  double e = 0.0;
  int st = read_status(pl, &e);
  if (rep) {
    std::memset(rep, 0, sizeof(*rep));
    rep->total_iterations = pl->iters_done;
    rep->max_roundoff = e;
    rep->status = st;
  }
  return st;
}

int gl_launches_per_iteration(const gl_plan* pl) {
  if (!pl) return GL_ERR_ARG;
  if (pl->mode == GL_MODE_FUSED) return 3;
  return 2 * pl->pg.nst + 4;
}

int gl_profile_kernels(gl_plan* pl, int iters, double* ms_out, const char** names, int* nk) {
  if (!pl || !ms_out || iters < 1) return GL_ERR_ARG;
  if (pl->mode != GL_MODE_FUSED) return GL_ERR_STATE;
  GL_CUDA(cudaSetDevice(pl->device));
  static const char* const kFp64Names[3] = {"k_col_fwd", "k_row_sq", "k_col_inv"};
  static const char* const kIntNames[3] = {"ki_col_fwd", "ki_row_sq", "ki_col_inv"};
  if (pl->from_state) {  // consume a pending state load first
    int rc = launch_iterations(pl, 1);
    if (rc != GL_OK) return rc;
    pl->iters_done += 1;
  }
  cudaEvent_t ev[4];
  for (auto& e : ev) GL_CUDA(cudaEventCreate(&e));
  double acc[3] = {0, 0, 0};
  int rc = GL_OK;
  for (int it = 0; it < iters && rc == GL_OK; ++it) {
    for (int k = 0; k < 3; ++k) {
      if (cudaEventRecord(ev[k], pl->stream) != cudaSuccess) { rc = GL_ERR_CUDA; break; }
      if ((pl->int_form ? launch_int_kernel(pl->args, pl->ig, pl->stream, k)
                        : launch_fused_kernel(pl->args, pl->fg, pl->stream, k)) != cudaSuccess) { rc = GL_ERR_CUDA; break; }
    }
    if (rc != GL_OK) break;
    if (cudaEventRecord(ev[3], pl->stream) != cudaSuccess || cudaEventSynchronize(ev[3]) != cudaSuccess) {
      rc = GL_ERR_CUDA;
      break;
    }
    for (int k = 0; k < 3; ++k) {
      float ms = 0.f;
      cudaEventElapsedTime(&ms, ev[k], ev[k + 1]);
      acc[k] += ms;
    }
  }
  for (auto& e : ev) cudaEventDestroy(e);
  if (rc != GL_OK) return rc;
  pl->iters_done += iters;
  pl->carry_valid = false;
  for (int k = 0; k < 3; ++k) {
    ms_out[k] = acc[k] / iters;
    if (names) names[k] = !pl->int_form ? kFp64Names[k] : k == 1 && pl->ig.t > 1 ? "ki_row_poly" : kIntNames[k];
  }
  if (nk) *nk = 3;
  return GL_OK;
}

int gl_get_products(gl_plan* pl, int64_t* ll_out) {
  if (!pl || !ll_out) return GL_ERR_ARG;
  GL_CUDA(cudaSetDevice(pl->device));
  const long long* src = pl->args.ll;
  if (pl->mode == GL_MODE_FUSED) {  // un-permute into the (idle) work array
    long long* tmp = reinterpret_cast<long long*>(pl->args.Z);
    GL_CUDA(launch_permute_words(pl->args, pl->args.ll, tmp, false, pl->stream));
    src = tmp;
  }
  GL_CUDA(cudaMemcpyAsync(ll_out, src, sizeof(int64_t) * pl->N, cudaMemcpyDeviceToHost, pl->stream));
  GL_CUDA(cudaStreamSynchronize(pl->stream));
  return GL_OK;
}

static int ensure_carry(gl_plan* pl) {
  if (!pl->carry_valid) {
    if (pl->mode == GL_MODE_FUSED) GL_CUDA(launch_dice_perm(pl->args, pl->stream));
    else GL_CUDA(launch_dice(pl->args, pl->stream));
    pl->carry_valid = true;
  }
  return GL_OK;
}

// The device address of pinned (page-locked, mapped) host memory, or null for any other
// pointer.
static void* mapped_host(const void* p) {
  cudaPointerAttributes at{};
  const bool ok = cudaPointerGetAttributes(&at, p) == cudaSuccess && at.type == cudaMemoryTypeHost;
  cudaGetLastError();  // a failed query leaves no error behind
  return ok ? at.devicePointer : nullptr;
}

// One host-state step of one fused iteration between pinned host buffers.  kind 1: the
// state as carry-added words (in[0] -> out[0]); kind 2: as the carry-save pair (digit
// in[0], carry in[1] -> out[0], out[1]).  out_dev: device addresses of the outputs'
// mappings.
struct HostStep {
  int kind;
  const void* in[2];
  void* out[2];
  void* out_dev[2];
};

// Copies in, the state-loading iteration, and the dicing, which also stores the state and
// the status into the mapped host buffers, so that transfer runs under the kernel instead
// of as copies after it.  Enqueued on the plan's stream (captured into a graph by the
// caller).
static cudaError_t enqueue_host_step(gl_plan* pl, const HostStep& hs, Status* status_dev, bool integer) {
  const size_t N = (size_t)pl->N;
  cudaError_t e;
  if ((e = cudaMemcpyAsync(pl->args.digit, hs.in[0], sizeof(int32_t) * N, cudaMemcpyHostToDevice, pl->stream)))
    return e;
  if (hs.kind == 1) e = cudaMemsetAsync(pl->args.hi, 0, N, pl->stream);
  else e = cudaMemcpyAsync(pl->args.hi, hs.in[1], N, cudaMemcpyHostToDevice, pl->stream);
  if (e) return e;
  if ((e = cudaMemsetAsync(pl->args.status, 0, sizeof(Status), pl->stream))) return e;
  // the integer form's load checks the words against its bound, and the dicing below leaves
  // the buffers alone if one is beyond it
  e = integer ? launch_int_iteration(pl->args, pl->ig, pl->stream, true)
              : launch_fused_iteration(pl->args, pl->fg, pl->stream, true);
  if (e) return e;
  if (hs.kind == 1) return launch_dice_words(pl->args, true, pl->stream, (int32_t*)hs.out_dev[0], status_dev);
  return launch_dice_perm(pl->args, pl->stream, (int*)hs.out_dev[0], (signed char*)hs.out_dev[1], status_dev);
}

// Whether this call runs as the captured step: one iteration of a fused (not resident)
// plan with graphs, every buffer pinned and mapped.  Fills hs->out_dev and *status_dev.
static bool host_step_mapped(gl_plan* pl, int64_t iters, HostStep* hs, Status** status_dev) {
  if (iters != 1 || pl->mode != GL_MODE_FUSED || pl->resident || !pl->use_graphs) return false;
  for (int i = 0; i < (hs->kind == 1 ? 1 : 2); ++i)
    if (!mapped_host(hs->in[i]) || !(hs->out_dev[i] = mapped_host(hs->out[i]))) return false;
  return (*status_dev = (Status*)mapped_host(pl->h_status)) != nullptr;
}

// Launches the step between ev0 and ev1 as one graph (about ten calls fewer per
// step), built on the first call for these buffers and kept by the plan: one graph in FP64,
// one in the integer form.
static int launch_host_step(gl_plan* pl, const HostStep& hs, Status* status_dev, bool integer) {
  bool same = pl->hw_kind == hs.kind;
  for (int i = 0; i < 2; ++i)
    same = same && pl->hw_in[i] == hs.in[i] && pl->hw_out[i] == hs.out[i] && pl->hw_out_dev[i] == hs.out_dev[i];
  if (!same) {
    for (cudaGraphExec_t& g : pl->hw_exec) {
      if (g) cudaGraphExecDestroy(g);
      g = nullptr;
    }
    pl->hw_kind = hs.kind;
    for (int i = 0; i < 2; ++i) {
      pl->hw_in[i] = hs.in[i];
      pl->hw_out[i] = hs.out[i];
      pl->hw_out_dev[i] = hs.out_dev[i];
    }
  }
  cudaGraphExec_t& exec = pl->hw_exec[integer ? 1 : 0];
  if (!exec) {
    cudaGraph_t graph = nullptr;
    GL_CUDA(cudaStreamBeginCapture(pl->stream, cudaStreamCaptureModeThreadLocal));
    const cudaError_t es = enqueue_host_step(pl, hs, status_dev, integer);
    const cudaError_t ec = cudaStreamEndCapture(pl->stream, &graph);
    if (es != cudaSuccess || ec != cudaSuccess || !graph) {
      if (graph) cudaGraphDestroy(graph);
      return GL_ERR_CUDA;
    }
    const cudaError_t ei = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ei != cudaSuccess) {
      exec = nullptr;
      return GL_ERR_CUDA;
    }
  }
  GL_CUDA(cudaEventRecord(pl->ev0, pl->stream));
  GL_CUDA(cudaGraphLaunch(exec, pl->stream));
  GL_CUDA(cudaEventRecord(pl->ev1, pl->stream));
  return GL_OK;
}

// Report of a host-state call whose work lies between ev0 and ev1: wait for it, read the
// status it left in pl->h_status.
static int report_host_step(gl_plan* pl, int64_t iters, gl_iter_report* rep) {
  GL_CUDA(cudaEventSynchronize(pl->ev1));
  const double e = std::ldexp((double)pl->h_status->maxerr64, -64);
  if (e > pl->run_maxerr) pl->run_maxerr = e;
  int st = GL_OK;
  if (pl->h_status->flags & kStatusTimeout) st = GL_ERR_TIMEOUT;
  else if (pl->h_status->flags) st = GL_ERR_OVERFLOW;
  else if (e >= pl->error_limit) st = GL_ERR_ROUNDOFF;
  float ms = 0.f;
  GL_CUDA(cudaEventElapsedTime(&ms, pl->ev0, pl->ev1));
  if (rep) {
    rep->iterations = iters;
    rep->total_iterations = pl->iters_done;
    rep->max_roundoff = e;
    rep->ms = ms;
    rep->status = st;
  }
  return st;
}

static int finish_host_step(gl_plan* pl, int64_t iters, gl_iter_report* rep) {
  GL_CUDA(cudaEventRecord(pl->ev1, pl->stream));
  return report_host_step(pl, iters, rep);
}

// The captured step from launch to report.  A state with a word beyond the integer form's
// bound has left the buffers as they were, and the step runs again in FP64.
static int run_host_step(gl_plan* pl, const HostStep& hs, Status* status_dev, gl_iter_report* rep) {
  bool integer = pl->int_form && ++pl->since_fp64 < kFp64Every;
  int rc = launch_host_step(pl, hs, status_dev, integer);
  if (rc == GL_OK && integer) {
    GL_CUDA(cudaEventSynchronize(pl->ev1));
    if (pl->h_status->flags & kStatusWide) rc = launch_host_step(pl, hs, status_dev, integer = false);
  }
  if (rc != GL_OK) return rc;
  if (!integer) pl->since_fp64 = 0;
  pl->from_state = false;
  pl->iters_done += 1;
  pl->carry_valid = true;  // the device (digit, hi) is the state the host received
  return report_host_step(pl, 1, rep);
}

int gl_iterate_host(gl_plan* pl, const int32_t* digit_in, const int8_t* hi_in, int64_t iters, int32_t* digit_out,
                    int8_t* hi_out, gl_iter_report* rep) {
  if (!pl || !digit_in || !hi_in || !digit_out || !hi_out || iters < 0) return GL_ERR_ARG;
  GL_CUDA(cudaSetDevice(pl->device));
  const size_t N = (size_t)pl->N;
  HostStep hs{2, {digit_in, hi_in}, {digit_out, hi_out}, {nullptr, nullptr}};
  Status* status_dev = nullptr;
  if (host_step_mapped(pl, iters, &hs, &status_dev)) return run_host_step(pl, hs, status_dev, rep);
  GL_CUDA(cudaEventRecord(pl->ev0, pl->stream));
  GL_CUDA(cudaMemcpyAsync(pl->args.digit, digit_in, sizeof(int32_t) * N, cudaMemcpyHostToDevice, pl->stream));
  GL_CUDA(cudaMemcpyAsync(pl->args.hi, hi_in, N, cudaMemcpyHostToDevice, pl->stream));
  GL_CUDA(cudaMemsetAsync(pl->args.status, 0, sizeof(Status), pl->stream));
  pl->from_state = pl->mode == GL_MODE_FUSED;
  pl->carry_valid = true;
  if (iters > 0) {
    const int rc = enqueue(pl, iters);
    if (rc != GL_OK) return rc;
    pl->iters_done += iters;
    pl->carry_valid = pl->mode == GL_MODE_PLAIN;
  }
  const int rc = ensure_carry(pl);
  if (rc != GL_OK) return rc;
  GL_CUDA(cudaMemcpyAsync(digit_out, pl->args.digit, sizeof(int32_t) * N, cudaMemcpyDeviceToHost, pl->stream));
  GL_CUDA(cudaMemcpyAsync(hi_out, pl->args.hi, N, cudaMemcpyDeviceToHost, pl->stream));
  GL_CUDA(cudaMemcpyAsync(pl->h_status, pl->args.status, sizeof(Status), cudaMemcpyDeviceToHost, pl->stream));
  return finish_host_step(pl, iters, rep);
}

int gl_iterate_host_words(gl_plan* pl, const int32_t* words_in, int64_t iters, int32_t* words_out,
                          gl_iter_report* rep) {
  if (!pl || !words_in || !words_out || iters < 0) return GL_ERR_ARG;
  GL_CUDA(cudaSetDevice(pl->device));
  const size_t N = (size_t)pl->N;
  HostStep hs{1, {words_in, nullptr}, {words_out, nullptr}, {nullptr, nullptr}};
  Status* status_dev = nullptr;
  if (host_step_mapped(pl, iters, &hs, &status_dev)) return run_host_step(pl, hs, status_dev, rep);
  GL_CUDA(cudaEventRecord(pl->ev0, pl->stream));
  GL_CUDA(cudaMemcpyAsync(pl->args.digit, words_in, sizeof(int32_t) * N, cudaMemcpyHostToDevice, pl->stream));
  GL_CUDA(cudaMemsetAsync(pl->args.hi, 0, N, pl->stream));
  GL_CUDA(cudaMemsetAsync(pl->args.status, 0, sizeof(Status), pl->stream));
  pl->from_state = pl->mode == GL_MODE_FUSED;
  pl->carry_valid = true;
  if (iters > 0) {
    const int rc = enqueue(pl, iters);
    if (rc != GL_OK) return rc;
    pl->iters_done += iters;
    pl->carry_valid = pl->mode == GL_MODE_PLAIN;
  }
  if (pl->carry_valid) GL_CUDA(launch_add_carry(pl->args, pl->stream));
  else GL_CUDA(launch_dice_words(pl->args, pl->mode == GL_MODE_FUSED, pl->stream));
  pl->carry_valid = true;  // (words, 0) is the carry-save state
  GL_CUDA(cudaMemcpyAsync(words_out, pl->args.digit, sizeof(int32_t) * N, cudaMemcpyDeviceToHost, pl->stream));
  GL_CUDA(cudaMemcpyAsync(pl->h_status, pl->args.status, sizeof(Status), cudaMemcpyDeviceToHost, pl->stream));
  return finish_host_step(pl, iters, rep);
}

int gl_get_carry_state(gl_plan* pl, int32_t* digit_out, int8_t* hi_out) {
  if (!pl || !digit_out || !hi_out) return GL_ERR_ARG;
  GL_CUDA(cudaSetDevice(pl->device));
  int rc = ensure_carry(pl);
  if (rc != GL_OK) return rc;
  GL_CUDA(cudaMemcpyAsync(digit_out, pl->args.digit, sizeof(int32_t) * pl->N, cudaMemcpyDeviceToHost, pl->stream));
  GL_CUDA(cudaMemcpyAsync(hi_out, pl->args.hi, pl->N, cudaMemcpyDeviceToHost, pl->stream));
  GL_CUDA(cudaStreamSynchronize(pl->stream));
  return GL_OK;
}

int gl_set_products(gl_plan* pl, const int64_t* ll, int64_t iterations) {
  if (!pl || !ll || iterations < 0) return GL_ERR_ARG;
  GL_CUDA(cudaSetDevice(pl->device));
  if (pl->mode == GL_MODE_FUSED) {
    long long* tmp = reinterpret_cast<long long*>(pl->args.Z);
    GL_CUDA(cudaMemcpyAsync(tmp, ll, sizeof(int64_t) * pl->N, cudaMemcpyHostToDevice, pl->stream));
    GL_CUDA(launch_permute_words(pl->args, tmp, pl->args.ll, true, pl->stream));
  } else {
    GL_CUDA(cudaMemcpyAsync(pl->args.ll, ll, sizeof(int64_t) * pl->N, cudaMemcpyHostToDevice, pl->stream));
  }
  GL_CUDA(cudaStreamSynchronize(pl->stream));
  pl->iters_done = iterations;
  pl->from_state = false;
  pl->carry_valid = false;
  return GL_OK;
}

int gl_set_carry_state(gl_plan* pl, const int32_t* digit, const int8_t* hi, int64_t iterations) {
  if (!pl || !digit || !hi || iterations < 0) return GL_ERR_ARG;
  GL_CUDA(cudaSetDevice(pl->device));
  GL_CUDA(cudaMemcpyAsync(pl->args.digit, digit, sizeof(int32_t) * pl->N, cudaMemcpyHostToDevice, pl->stream));
  GL_CUDA(cudaMemcpyAsync(pl->args.hi, hi, pl->N, cudaMemcpyHostToDevice, pl->stream));
  GL_CUDA(cudaStreamSynchronize(pl->stream));
  pl->iters_done = iterations;
  pl->from_state = pl->mode == GL_MODE_FUSED;
  pl->carry_valid = true;
  return GL_OK;
}

int gl_get_residue(gl_plan* pl, int32_t* digits_out, uint64_t* res64, int* is_zero) {
  if (!pl) return GL_ERR_ARG;
  GL_CUDA(cudaSetDevice(pl->device));
  int rc = ensure_carry(pl);
  if (rc != GL_OK) return rc;
  // the work array is idle between iterations: it holds the balanced digits
  int32_t* balanced = reinterpret_cast<int32_t*>(pl->args.Z);
  GL_CUDA(launch_residue(pl->args, pl->mode == GL_MODE_FUSED, balanced, pl->rscratch, pl->stream));
  GL_CUDA(cudaMemcpyAsync(pl->h_res, pl->rscratch + residue_head_offset(pl->N), sizeof(int32_t) * 69,
                          cudaMemcpyDeviceToHost, pl->stream));
  if (digits_out)
    GL_CUDA(cudaMemcpyAsync(digits_out, balanced, sizeof(int32_t) * pl->N, cudaMemcpyDeviceToHost, pl->stream));
  GL_CUDA(cudaStreamSynchronize(pl->stream));
  const int32_t* head = pl->h_res;
  const int32_t* scal = head + 64;
  const int flags = head[68];
  if (scal[2] != scal[3]) return GL_ERR_STATE;  // the end-around carry has no fixed point
  const bool all0 = !(flags & 1), allmax = !(flags & 2);
  // low 64 bits of the canonical digits; word j holds ceil(p(j+1)/N) - ceil(pj/N) bits
  uint64_t r = 0;
  int pos = 0;
  for (int j = 0; j < pl->N && j < 64 && pos < 64; ++j) {
    const int64_t lo = ((int64_t)pl->p * j + pl->N - 1) / pl->N;
    const int64_t hi = ((int64_t)pl->p * (j + 1) + pl->N - 1) / pl->N;
    r |= (uint64_t)(uint32_t)head[j] << pos;  // bits above 64 fall off
    pos += (int)(hi - lo);
  }
  if (allmax) r = 0;  // 2^p - 1 == 0
  if (res64) *res64 = r;
  if (is_zero) *is_zero = (all0 || allmax) ? 1 : 0;
  return GL_OK;
}

int gl_mersenne_test(gl_plan* pl, int64_t iters, gl_result* res) {
  if (!pl) return GL_ERR_ARG;
  const bool full = iters == 0;
  if (full) {
    int rc = gl_reset(pl);
    if (rc != GL_OK) return rc;
    iters = (int64_t)pl->p - 2;
  }
  gl_iter_report rep{};
  int st = gl_iterate(pl, iters, &rep);
  if (st == GL_ERR_CUDA || st == GL_ERR_ARG) return st;
  uint64_t r = 0;
  int z = 0;
  int rc = gl_get_residue(pl, nullptr, &r, &z);
  if (rc != GL_OK) return rc;
  if (res) {
    res->p = pl->p;
    res->N = pl->N;
    res->iterations = pl->iters_done;
    res->is_zero = z;
    res->is_prime = (pl->iters_done == (int64_t)pl->p - 2 && z && st == GL_OK) ? 1 : 0;
    res->res64 = r;
    res->max_roundoff = pl->run_maxerr;
    res->ms = rep.ms;
  }
  return st;
}

int gl_error_test(int p, int N, const gl_plan_opts* opts, int iters, gl_iter_report* rep) {
  gl_plan* pl = nullptr;
  // a round-off trial: FP64 in every iteration
  int rc = gl_plan_create_ex(p, N, opts, opts && opts->batch_layout ? 1 : 0, &pl, true);
  if (rc != GL_OK) return rc;
  if (iters <= 0) {
    iters = p / 10000;
    if (iters < 100) iters = 100;
    if (iters > 2500) iters = 2500;
  }
  rc = gl_iterate(pl, iters, rep);
  gl_plan_destroy(pl);
  return rc;
}

int gl_find_signal_size(int p, const gl_plan_opts* opts, int* N_out, double* ms_per_iter, double* max_roundoff) {
  if (!N_out || p < 64) return GL_ERR_ARG;
  gl_plan_opts o;
  if (opts) o = *opts;
  else gl_default_opts(&o);
  o.mode = GL_MODE_FUSED;
  const gl_plan_opts want = o;  // the plan that the caller will make
  o.fft_h = 0;
  o.error_limit = 0.5;
  o.check_every = 100;
  // candidate lengths, smallest first
  std::vector<int> cand;
  for (int64_t p2 = 2; p2 <= (1 << 26); p2 *= 2)
    for (int64_t p3 = 1, b = 0; b <= 5; p3 *= 3, ++b)
      for (int64_t p5 = 1, c = 0; c <= 3; p5 *= 5, ++c)
        for (int64_t p7 = 1, d = 0; d <= 2; p7 *= 7, ++d) {
          const int64_t N = p2 * p3 * p5 * p7;
          if (N < 64 || N > p / 8 || N > (1 << 27)) continue;
          if (slice_depth(p, (int)N) < 0) continue;
          cand.push_back((int)N);
        }
  std::sort(cand.begin(), cand.end());
  cand.erase(std::unique(cand.begin(), cand.end()), cand.end());
  int best = 0, first = 0;
  double best_ms = 1e300, best_err = 0.0;
  for (int N : cand) {
    if (first && N > first + first / 7) break;  // within ~15 % of the smallest accepted
    // The trial measures the round-off, in FP64; its own layout search is left out where the
    // plan will run the integer form.
    int vmax = 0;
    const bool integer = wants_int_form(p, N, want, &vmax);
    gl_plan_opts trial = o;
    if (integer) trial.autotune = 0;
    gl_plan* pl = nullptr;
    int rc = gl_plan_create_ex(p, N, &trial, o.batch_layout ? 1 : 0, &pl, true);
    if (rc == GL_ERR_NOMEM || rc == GL_ERR_NODEVICE || rc == GL_ERR_CUDA) return rc;
    if (rc != GL_OK) continue;
    gl_iter_report rep{};
    rc = gl_iterate(pl, 100, &rep);
    // ranked by the time of the form the plan will run
    double ms = -1.0;
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, pl->device);
    if (integer) {
      const IntTuned it = timed_int_layout(N / 2, pl->n, sms, 0);
      double fp64 = -1.0;
      if (it.H) autotune_layout(N / 2, pl->n, sms, 0, &fp64, it.H);
      if (fp64 > 0.0) ms = ((kFp64Every - 1) * it.ms + fp64) / kFp64Every;
    }
    if (ms <= 0.0) autotune_layout(N / 2, pl->n, sms, 0, &ms);
    gl_plan_destroy(pl);
    if (rc == GL_ERR_CUDA) return rc;
    if (rc != GL_OK || rep.max_roundoff >= 0.30 || ms <= 0.0) continue;
    if (!first) first = N;
    if (ms < best_ms) {
      best_ms = ms;
      best = N;
      best_err = rep.max_roundoff;
    }
  }
  if (!best) return GL_ERR_SIZE;
  if (ms_per_iter) {  // measured on the plan itself: its graphs, its resident form
    gl_plan* pl = nullptr;
    gl_iter_report rep{};
    const int rc = gl_plan_create_ex(p, best, &want, want.batch_layout ? 1 : 0, &pl);
    if (rc == GL_OK) {
      gl_iterate(pl, kGraphBatch, &rep);
      if (gl_iterate(pl, 4 * kGraphBatch, &rep) == GL_OK && rep.ms > 0.0) best_ms = rep.ms / (4 * kGraphBatch);
      gl_plan_destroy(pl);
    }
    *ms_per_iter = best_ms;
  }
  *N_out = best;
  if (max_roundoff) *max_roundoff = best_err;
  return GL_OK;
}

float errorTest(int testPrime, int signalSize) {
  gl_iter_report rep{};
  int rc = gl_error_test(testPrime, signalSize, nullptr, 0, &rep);
  if (rc != GL_OK || rep.iterations <= 0) return -1.0f;
  return (float)(rep.ms / (double)rep.iterations);
}

int mersenneTest(int testPrime, int signalSize) {
  gl_plan* pl = nullptr;
  int rc = gl_plan_create(testPrime, signalSize, nullptr, &pl);
  if (rc != GL_OK) return rc;
  gl_result res{};
  rc = gl_mersenne_test(pl, 0, &res);
  gl_plan_destroy(pl);
  if (rc != GL_OK) return rc;
  if (res.is_prime)
    std::printf("M( %d )P, n = %d, gpulucas_gb300 v%d.%d.%d\n", testPrime, signalSize, 0, 1, 0);
  else
    std::printf("M( %d )C, 0x%016llx, n = %d, gpulucas_gb300 v%d.%d.%d\n", testPrime,
                (unsigned long long)res.res64, signalSize, 0, 1, 0);
  std::fflush(stdout);
  return res.is_prime;
}

int gl_selftest_bounded_wait(int device, int tries) {
  if (tries < 1) return GL_ERR_ARG;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return GL_ERR_NODEVICE;
  if (device < 0 || device >= ndev || cudaSetDevice(device) != cudaSuccess) return GL_ERR_ARG;
  Status* d = nullptr;
  Status h{};
  if (cudaMalloc(&d, sizeof(Status)) != cudaSuccess) return GL_ERR_NOMEM;
  int rc = GL_OK;
  if (cudaMemset(d, 0, sizeof(Status)) != cudaSuccess || launch_wait_selftest(d, tries, 0) != cudaSuccess ||
      cudaMemcpy(&h, d, sizeof(Status), cudaMemcpyDeviceToHost) != cudaSuccess)
    rc = GL_ERR_CUDA;
  cudaFree(d);
  if (rc != GL_OK) return rc;
  return (h.flags & kStatusTimeout) ? GL_ERR_TIMEOUT : GL_OK;
}

// Runs probe(blocks, threads, iters) with iters doubling until one launch takes >= ms;
// returns its milliseconds and the iteration count.
}  // extern "C"
template <typename Probe>
static int timed_probe(int device, double ms, Probe probe, float* el_out, long long* iters_out, int* blocks_out) {
  GL_CUDA(cudaSetDevice(device));
  int nsm = 0;
  GL_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device));
  const int threads = 256, blocks = nsm * 4;
  double* buf = nullptr;
  GL_CUDA(cudaMalloc(&buf, sizeof(double) * threads * blocks));
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  long long iters = 1024;
  float el = 0.f;
  int rc = GL_OK;
  for (int rep = 0; rep < 12; ++rep) {
    cudaEventRecord(a, 0);
    if (probe(blocks, threads, iters, buf, (cudaStream_t)0) != cudaSuccess) { rc = GL_ERR_CUDA; break; }
    cudaEventRecord(b, 0);
    if (cudaEventSynchronize(b) != cudaSuccess) { rc = GL_ERR_CUDA; break; }
    cudaEventElapsedTime(&el, a, b);
    if (el >= ms) break;
    iters *= 2;
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  cudaFree(buf);
  *el_out = el;
  *iters_out = iters;
  *blocks_out = blocks;
  return rc;
}
extern "C" {

int gl_probe_fp64_peak(int device, double ms, double* tflops) {
  if (!tflops || ms <= 0) return GL_ERR_ARG;
  float el = 0.f;
  long long iters = 0;
  int blocks = 0;
  const int rc = timed_probe(device, ms, probe_fp64, &el, &iters, &blocks);
  if (rc == GL_OK) {
    const double fmas = (double)blocks * 256 * 8.0 * (double)iters;
    *tflops = 2.0 * fmas / (el * 1e-3) / 1e12;
  }
  return rc;
}

int gl_probe_fp64_butterfly(int device, double ms, double* instr_per_s) {
  if (!instr_per_s || ms <= 0) return GL_ERR_ARG;
  float el = 0.f;
  long long iters = 0;
  int blocks = 0;
  const int rc = timed_probe(device, ms, probe_butterfly, &el, &iters, &blocks);
  if (rc == GL_OK) *instr_per_s = (double)blocks * 256 * kProbeButterflyInstr * (double)iters / (el * 1e-3);
  return rc;
}

}  // extern "C"
