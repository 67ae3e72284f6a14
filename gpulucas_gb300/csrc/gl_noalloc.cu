// gl_noalloc.cu -- Lucas-Lehmer iterations for callers that cannot allocate device
// memory.
//
// Some callers may not call cudaMalloc at all: code that runs inside a framework
// whose memory pool owns every device allocation, code that must not grow its
// footprint once a service is running, or code whose allocation calls would
// synchronise a device it shares with latency-sensitive work.  gl_iterate_noalloc
// serves them: the caller passes device buffers for the input and output products,
// and everything else the iterations need -- the two FFT work arrays, the weight,
// flag and twiddle tables of the test, the carry-save digits and the round-off
// status word -- lives in one file-scope __device__ array below.  It is sized for
// N <= kNoAllocMaxN (65536 words, about 5.9 MiB) and stays resident on every GPU that
// loads this library until the process exits.
//
// The iterations are the integer form (gl_int_kernels.cu) where a plan of (p, N) would use
// it, one in 64 and the last of a call in FP64; elsewhere all are FP64.  FP64 iterations
// are the plain form (one kernel per reference step), launched through the same launchers
// as a plan of GL_MODE_PLAIN.  The products equal those of gl_iterate bit for bit.
// N = 65536: 110.7 us per iteration in the plain form, whose twenty launches each read and
// write the whole signal, against 20.6 in the integer form's three.
#include <cstring>
#include <mutex>
#include <vector>

#include "gl_internal.h"
#include "gl_plan.h"
#include "gl_tables.h"

namespace gl {
namespace {

constexpr int kNoAllocMaxN = 65536;
constexpr int kNoAllocMaxM = kNoAllocMaxN / 2;
constexpr int kMaxDevices = 64;

constexpr size_t align256(size_t x) { return (x + 255) / 256 * 256; }
// byte offsets of the sub-buffers inside the scratch array
constexpr size_t kOffZ = 0;
constexpr size_t kOffZ2 = kOffZ + align256(sizeof(DevCplx) * kNoAllocMaxM);
constexpr size_t kOffTwM = kOffZ2 + align256(sizeof(DevCplx) * kNoAllocMaxM);
constexpr size_t kOffPair = kOffTwM + align256(sizeof(DevCplx) * kNoAllocMaxM);
constexpr size_t kOffA = kOffPair + align256(sizeof(DevCplx) * kNoAllocMaxM);
constexpr size_t kOffAinv = kOffA + align256(sizeof(double) * kNoAllocMaxN);
constexpr size_t kOffDigit = kOffAinv + align256(sizeof(double) * kNoAllocMaxN);
constexpr size_t kOffHi = kOffDigit + align256(sizeof(int) * kNoAllocMaxN);
constexpr size_t kOffFlags = kOffHi + align256(kNoAllocMaxN);
constexpr size_t kOffStatus = kOffFlags + align256(kNoAllocMaxN);
// the integer form's state and tables
constexpr int kNoAllocMaxLine = 4096;  // points of a line, and rows
constexpr size_t kOffLl = kOffStatus + align256(sizeof(Status));
constexpr size_t kOffFlagsC = kOffLl + align256(sizeof(long long) * kNoAllocMaxN);
constexpr size_t kOffSpan = kOffFlagsC + align256(kNoAllocMaxN);
constexpr size_t kOffExp = kOffSpan + align256(kNoAllocMaxN);
constexpr size_t kOffK1 = kOffExp + align256(kNoAllocMaxN);
constexpr size_t kOffK2 = kOffK1 + align256(sizeof(HostTw) * kNoAllocMaxM);
constexpr size_t kOffIntPair = kOffK2 + align256(sizeof(HostTw) * kNoAllocMaxM);
constexpr size_t kOffStages = kOffIntPair + align256(sizeof(HostTw) * kNoAllocMaxM);  // wf, wi, hf, hi
constexpr size_t kOffRows = kOffStages + 4 * align256(sizeof(HostTw) * kNoAllocMaxLine);
constexpr size_t kScratchBytes = kOffRows + align256(sizeof(RowPair) * kNoAllocMaxLine);

// The scratch.  In host code this name is only a host-side stand-in for the symbol,
// never a device address: the address comes from cudaGetSymbolAddress below.
static __device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

// Host staging for the per-test tables, reused by every call.  The FP64 tables' is static;
// the integer form's is allocated on the host, with the first test that needs it.
static DevCplx h_twM[kNoAllocMaxM];
static DevCplx h_pair[kNoAllocMaxM];
static double h_A[kNoAllocMaxN];
static double h_Ainv[kNoAllocMaxN];
static unsigned char h_flags[kNoAllocMaxN];
static Status h_status;

// The integer form of the test whose tables are staged (H = 0: it has none).
static struct {
  int H = 0;
  IntGeom g{};
  std::vector<HostTw> k1, pair, k2, stages[4];
  std::vector<RowPair> rows;
  std::vector<uint8_t> flags, span, e;
} h_int;

struct DeviceSlot {
  unsigned char* base = nullptr;  // device address of g_noalloc_scratch on this device
  int p = 0, N = 0;               // test whose tables the scratch holds (0: none whole)
  bool int_known = false;         // whether the integer form's tables were asked for
  int64_t without_int = 0;        // iterations of this test run before that
  int H = 0;                      // integer form: column length, geometry (H = 0: none)
  IntGeom g{};
  int nrows = 0;
};
static DeviceSlot g_slots[kMaxDevices];
static std::mutex g_mutex;  // host-side state: staging buffers and the slots

// Fill the host staging tables for (p, N) with the entry helpers a GL_MODE_PLAIN plan's
// tables are built from (gl_tables.cpp), so the two cannot drift apart.
void build_tables(int p, int N) {
  const int M = N / 2;
  for (int k = 0; k < M; ++k) {
    const HostCplx w = twiddle(k, M);
    const HostCplx c = pair_coeff(k, M);
    h_twM[k] = {w.re, w.im};
    h_pair[k] = {c.re, c.im};
  }
  for (int j = 0; j < N; ++j) weight_entry(p, N, j, (double)M, &h_A[j], &h_Ainv[j]);
  for (int j = 0; j < N; ++j) h_flags[j] = word_flags(p, N, j);
}

// The same for the integer form, from the helpers a plan's tables are built from.
void build_int_tables(int p, int N, int n) {
  h_int.H = 0;
  int H = 0;
  if (!gl_int_layout(p, N, &H, &h_int.g)) return;
  const int M = N / 2, W = M / H, t = h_int.g.t, V = W / t;
  gf_pass_tables(W, H, t, h_int.k1, h_int.pair, h_int.k2);
  gf_row_pairs(V, H, h_int.rows);
  std::vector<uint8_t> e;
  gf_weights(p, N, e);
  int off[8];
  const LinePlan &pw = h_int.g.pw, &ph = h_int.g.ph;
  gf_stage_twiddles(pw.radix, pw.nst, false, h_int.stages[0], off);
  gf_stage_twiddles(pw.radix, pw.nst, true, h_int.stages[1], off);
  gf_stage_twiddles(ph.radix, ph.nst, false, h_int.stages[2], off);
  gf_stage_twiddles(ph.radix, ph.nst, true, h_int.stages[3], off);
  for (const auto& s : h_int.stages)
    if (s.size() > (size_t)kNoAllocMaxLine) return;
  if (h_int.rows.size() > (size_t)kNoAllocMaxLine) return;
  h_int.flags.resize((size_t)N);
  h_int.span.resize((size_t)N);
  h_int.e.resize((size_t)N);
  for (int j = 0; j < N; ++j) {  // column-major
    const int m = j >> 1, m2 = m / W, m1 = m - m2 * W;
    const int c = 2 * (m1 * H + m2) + (j & 1);
    int tot = 0;
    for (int i = 0; i <= n; ++i) tot += word_bits(p, N, (j + i) % N);
    h_int.flags[(size_t)c] = h_flags[j];
    h_int.span[(size_t)c] = (uint8_t)(tot > 255 ? 255 : tot);
    h_int.e[(size_t)c] = e[(size_t)j];
  }
  h_int.H = H;
}

// The integer form's tables are built once a test has asked for this many iterations since
// its tables were last loaded: they take about 0.05 us per word of host time and save 45 to
// 85 us an iteration (N = 1024 to 65536), so a program that takes a few iterations of one
// test after another would only pay for them.  N = 54432 after 49152, us a call of 2, 20 and
// 100 iterations: 82882, 84704 and 92781 without, 86152, 86561 and 89376 with them.
int64_t int_tables_after(int N) { return N / 1024 < 2 ? 2 : N / 1024; }

constexpr size_t stage_offset(int i) { return kOffStages + (size_t)i * align256(sizeof(HostTw) * kNoAllocMaxLine); }

// One FP64 iteration in this many, and the last of a call: the round-off a call reports
// is theirs.
constexpr int kNoAllocFp64Every = 64;

}  // namespace
}  // namespace gl

using namespace gl;

static int iterate_noalloc(int p, int N, const int64_t* ll_in, int64_t* ll_out, int64_t iters, double* max_roundoff,
                           void* stream) {
  if (!ll_in || !ll_out || iters < 0) return GL_ERR_ARG;
  if (p < 3 || N < 16 || (N & 1) || N > p) return GL_ERR_ARG;
  if (N > kNoAllocMaxN) return GL_ERR_TOO_LARGE;
  {
    // the same buffer is fine; buffers that share only part of their words are not
    const int64_t* out_c = ll_out;
    if (out_c != ll_in && out_c < ll_in + N && ll_in < out_c + N) return GL_ERR_ARG;
  }
  const int n = slice_depth(p, N);
  if (n < 0) return GL_ERR_RATIO;
  const int M = N / 2;
  PlainGeom pg{};
  // radices of the plain form (<= 4), by the helper a GL_MODE_PLAIN plan uses
  pg.nst = radix_plan_into(M, 4, pg.radix, 40);
  if (pg.nst <= 0) return GL_ERR_SIZE;
  pg.threads = 256;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  {
    // the call waits for its stream, which a stream being captured into a graph cannot do
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cs) != cudaSuccess) {
      cudaGetLastError();
      return GL_ERR_CUDA;
    }
    if (cs != cudaStreamCaptureStatusNone) return GL_ERR_ARG;
  }
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return GL_ERR_CUDA;
  if (dev < 0 || dev >= kMaxDevices) return GL_ERR_ARG;

  std::lock_guard<std::mutex> lock(g_mutex);
  DeviceSlot& slot = g_slots[dev];
  {
    // The array's device address, looked up with this device current on every call (the
    // lookup allocates nothing).  If it moved -- the context was reset and the module
    // loaded again -- the tables the slot remembers are gone too.
    void* ptr = nullptr;
    if (cudaGetSymbolAddress(&ptr, g_noalloc_scratch) != cudaSuccess || !ptr) return GL_ERR_CUDA;
    if (static_cast<unsigned char*>(ptr) != slot.base) {
      slot.base = static_cast<unsigned char*>(ptr);
      slot.p = slot.N = 0;
    }
  }
  unsigned char* base = slot.base;
  // The slot names no test while its tables are being replaced, so that a call that ends
  // half way (an error, an exception) leaves none that a later call would take for whole.
  const int held_p = slot.p, held_N = slot.N;
  slot.p = slot.N = 0;
  if (held_p != p || held_N != N) {
    build_tables(p, N);
    if (cudaMemcpyAsync(base + kOffTwM, h_twM, sizeof(DevCplx) * M, cudaMemcpyHostToDevice, s) ||
        cudaMemcpyAsync(base + kOffPair, h_pair, sizeof(DevCplx) * M, cudaMemcpyHostToDevice, s) ||
        cudaMemcpyAsync(base + kOffA, h_A, sizeof(double) * N, cudaMemcpyHostToDevice, s) ||
        cudaMemcpyAsync(base + kOffAinv, h_Ainv, sizeof(double) * N, cudaMemcpyHostToDevice, s) ||
        cudaMemcpyAsync(base + kOffFlags, h_flags, N, cudaMemcpyHostToDevice, s))
      return GL_ERR_CUDA;
    slot.int_known = false;
    slot.without_int = 0;
    slot.H = 0;
  }
  if (!slot.int_known) slot.without_int += iters;
  if (iters >= 2 && !slot.int_known && slot.without_int >= int_tables_after(N)) {
    build_int_tables(p, N, n);
    if (h_int.H) {
      auto up = [&](size_t off, const auto& v) {
        return cudaMemcpyAsync(base + off, v.data(), v.size() * sizeof(v[0]), cudaMemcpyHostToDevice, s) != cudaSuccess;
      };
      bool bad = up(kOffFlagsC, h_int.flags) || up(kOffSpan, h_int.span) || up(kOffExp, h_int.e) ||
                 up(kOffK1, h_int.k1) || up(kOffK2, h_int.k2) || up(kOffIntPair, h_int.pair) || up(kOffRows, h_int.rows);
      for (int i = 0; i < 4; ++i) bad = bad || up(stage_offset(i), h_int.stages[i]);
      if (bad || set_int_smem_limits(h_int.g, n, (int)h_int.rows.size(), false) != cudaSuccess) return GL_ERR_CUDA;
    }
    slot.H = h_int.H;
    slot.g = h_int.g;
    slot.nrows = (int)h_int.rows.size();
    slot.int_known = true;
  }
  slot.p = p;
  slot.N = N;

  IterArgs a{};
  a.N = N; a.M = M; a.LO = p / N; a.n = n;
  a.ll = reinterpret_cast<long long*>(ll_out);
  a.flags = base + kOffFlags;
  a.A = reinterpret_cast<const double*>(base + kOffA);
  a.Ainv = reinterpret_cast<const double*>(base + kOffAinv);
  a.Z = reinterpret_cast<DevCplx*>(base + kOffZ);
  a.Z2 = reinterpret_cast<DevCplx*>(base + kOffZ2);
  a.twM = reinterpret_cast<const DevCplx*>(base + kOffTwM);
  a.twPair = reinterpret_cast<const DevCplx*>(base + kOffPair);
  a.digit = reinterpret_cast<int*>(base + kOffDigit);
  a.hi = reinterpret_cast<signed char*>(base + kOffHi);
  a.status = reinterpret_cast<Status*>(base + kOffStatus);

  // the status word keeps the previous call's contents: clear it
  if (cudaMemsetAsync(a.status, 0, sizeof(Status), s) != cudaSuccess) return GL_ERR_CUDA;
  if (ll_out != ll_in &&
      cudaMemcpyAsync(ll_out, ll_in, sizeof(int64_t) * N, cudaMemcpyDeviceToDevice, s) != cudaSuccess)
    return GL_ERR_CUDA;
  if (!slot.H || iters < 2) {
    if (launch_dice(a, s) != cudaSuccess) return GL_ERR_CUDA;
    for (int64_t i = 0; i < iters; ++i)
      if (launch_plain_iteration(a, pg, s) != cudaSuccess) return GL_ERR_CUDA;
  } else {
    const int H = slot.H, W = M / H;
    IterArgs b = a;
    b.W = W; b.H = H; b.G = 1;
    b.ll = reinterpret_cast<long long*>(base + kOffLl);
    b.flags = base + kOffFlagsC;
    b.span = base + kOffSpan;
    auto tw = [&](size_t off) { return reinterpret_cast<const int4*>(base + off); };
    b.in.wf = tw(stage_offset(0)); b.in.wi = tw(stage_offset(1));
    b.in.hf = tw(stage_offset(2)); b.in.hi = tw(stage_offset(3));
    b.in.k1 = tw(kOffK1); b.in.pair = tw(kOffIntPair); b.in.k2 = tw(kOffK2); b.in.rows = tw(kOffRows);
    b.in.e = base + kOffExp;
    gl_int_args(H, W, slot.g, slot.nrows, &b.in);
    b.in.dependent = b.in.touch;  // no graph here: hides the passes' launches
    b.in.check_span = (n + 1) * (p / N) < 51;
    int64_t left = iters;
    while (left > 0) {
      const int64_t k = (left < kNoAllocFp64Every ? left : kNoAllocFp64Every) - 1;
      if (k > 0) {
        if (launch_permute_words(b, a.ll, b.ll, true, s) != cudaSuccess) return GL_ERR_CUDA;
        for (int64_t i = 0; i < k; ++i)
          if (launch_int_iteration(b, slot.g, s, false) != cudaSuccess) return GL_ERR_CUDA;
        if (launch_permute_words(b, b.ll, a.ll, false, s) != cudaSuccess) return GL_ERR_CUDA;
      }
      if (launch_dice(a, s) != cudaSuccess || launch_plain_iteration(a, pg, s) != cudaSuccess) return GL_ERR_CUDA;
      left -= k + 1;
    }
  }
  if (cudaMemcpyAsync(&h_status, a.status, sizeof(Status), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return GL_ERR_CUDA;
  const double e = (double)h_status.maxerr64 * 0x1p-64;
  if (max_roundoff) *max_roundoff = e;
  if (h_status.flags) return GL_ERR_OVERFLOW;
  if (e >= 0.4) return GL_ERR_ROUNDOFF;
  return GL_OK;
}

extern "C" int gl_iterate_noalloc(int p, int N, const int64_t* ll_in, int64_t* ll_out, int64_t iters,
                                  double* max_roundoff, void* stream) {
  try {
    return iterate_noalloc(p, N, ll_in, ll_out, iters, max_roundoff, stream);
  } catch (...) {  // host memory for the integer form's tables
    return GL_ERR_NOMEM;
  }
}
