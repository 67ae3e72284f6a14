// gl_int_kernels.cu -- one Lucas-Lehmer iteration in exact integer arithmetic.
//
// The same three passes as the fused FP64 form (gl_kernels.cu), over GF(q^2), q = 2^61 - 1
// (gl_gf61.cuh), instead of the complex numbers: weights are rotations by e bits, twiddles
// are field elements, and the inverse transform gives every product exactly (they are
// below 2^60 in magnitude), so nothing is rounded.  The layout (H x W, column-major
// per-word arrays), the dicing and the range checks are those of the FP64 form, and so are
// the products, bit for bit.  GB300's FP64 units bound the FP64 form; this one is bound by
// the integer pipes (a 32 x 32 -> 64-bit multiply-add holds one for 4 cycles per warp,
// other integer instructions 1 to 2).
//
// Two differences from the complex numbers:
//  * the row and position that a frequency pairs with (the real-signal split): conjugation
//    sends frequency k to q k mod M, which is -k only in the power-of-two part, so the row
//    pairs come from a table and the position in the partner row is q k1 + shift mod W;
//  * roots of odd order are scalars of GF(q), not of norm 1, so the inverse transform has
//    its own tables.
#include "gl_dice.cuh"
#include "gl_int_stage.cuh"
#include "gl_internal.h"

namespace gl {
namespace {

__device__ __forceinline__ g2 ldz(const DevCplx* p) {
  const longlong2 v = *reinterpret_cast<const longlong2*>(p);
  return g2{v.x, v.y};
}
__device__ __forceinline__ void stz(DevCplx* p, g2 v) {
  *reinterpret_cast<longlong2*>(p) = make_longlong2(v.re, v.im);
}

// Starts the load of n table entries into L1: one word of every 128-byte line, into a
// register nobody reads, so the pass does not wait for them here.  Where few CTAs run, a
// pass is a chain of latencies and every stage would wait on L2 for its twiddles.
__device__ __forceinline__ void touch(const int4* p, int n) {
  for (int i = threadIdx.x * 8; i < n; i += blockDim.x * 8) {
    asm volatile("{\n .reg .s32 d;\n ld.global.nc.s32 d, [%0];\n}" ::"l"(p + i));
  }
}
// With a.in.dependent every pass is launched as a programmatic dependent of the one before
// it: it becomes resident while that one runs, touches its tables, and waits here for that
// one's end.  Only then may the next pass become resident, so at most one waits at a time.
// What the pass before writes (products, work arrays) is read with ordinary loads: the wait
// makes it visible to them, not to the non-coherent path, which is for the tables alone.
// For iterations launched one by one (N = 65536 without allocation: 27.3 -> 20.6 us per
// iteration).  In a replayed graph it gains at some lengths and loses at others (65536: 18.3
// -> 17.2, 163840: 23.1 -> 24-26, 5120: 14.6 -> 15.5); plans do not use it.
__device__ __forceinline__ void after_previous_pass() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Starts bringing n table entries into L2 (one thread): with many CTAs the tables of the end
// of a pass come from DRAM, and every CTA of a wave asks for them at the same time.
__device__ __forceinline__ void prefetch_l2(const int4* p, int n) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(n * 16));
}
__device__ __forceinline__ int plan_slots(const LinePlan& lp) {  // entries of its stage table
  const int s = lp.nst - 1, R = lp.radix[s];
  return lp.off[s] + (s ? (R - 1) * (lp.L / R) : 0);
}

// In-place stage: every thread first reads the inputs of all its butterflies (at most P
// points) into registers, then, after a barrier, transforms and writes them.  One line
// buffer and 64 registers, so four CTAs of 256 threads are resident and the 576 columns of
// N = 2359296 run as one wave: 137.8 -> 132.3 us per iteration there (the integer passes
// alone) against two buffers and three CTAs.  Holding 16 points in 128 threads
// (122 registers) took 154.  Short columns are faster with two buffers, one barrier per
// stage (N = 49152: 20.4 against 21.1); the layout search times both.
template <int R, int P>
__host__ __device__ constexpr int ip_count() {
  return P / R > 0 ? P / R : 1;
}
template <int R, int S, int P>
__device__ __forceinline__ void int_stage_ip(g2* __restrict__ buf, int L, int Ns, const int4* __restrict__ tw) {
  constexpr int B = ip_count<R, P>();
  const int LR = L / R;
  const bool last = Ns == LR, pow2 = (Ns & (Ns - 1)) == 0;
  g2 held[B][R];
#pragma unroll
  for (int i = 0; i < B; ++i) {
    const int j = threadIdx.x + i * blockDim.x;
    const int jj = j < LR ? j : 0;  // a thread without this butterfly reads a valid slot
#pragma unroll
    for (int q = 0; q < R; ++q) held[i][q] = buf[ipad(jj + q * LR)];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < B; ++i) {
    const int j = threadIdx.x + i * blockDim.x;
    if (j < LR) {
      const int k = last ? j : pow2 ? (j & (Ns - 1)) : j % Ns;
      g2 v[R];
      gf::butterfly<R, S>(
          v, Ns > 1, [&](int q) { return held[i][q]; }, [&](int s) { return __ldg(tw + (k + s * Ns)); });
      const int base = (j - k) * R + k;
#pragma unroll
      for (int q = 0; q < R; ++q) buf[ipad(base + q * Ns)] = v[q];
    }
  }
  __syncthreads();
}

template <int S, bool B57, int P>
__device__ __forceinline__ void int_line_fft_ip(g2* a, const LinePlan& lp, const int4* tw) {
  int Ns = 1;
  for (int s = 0; s < lp.nst; ++s) {
    const int4* st = tw + lp.off[s];
    switch (lp.radix[s]) {
      case 8: int_stage_ip<8, S, P>(a, lp.L, Ns, st); break;
      case 4: int_stage_ip<4, S, P>(a, lp.L, Ns, st); break;
      case 2: int_stage_ip<2, S, P>(a, lp.L, Ns, st); break;
      case 3: int_stage_ip<3, S, P>(a, lp.L, Ns, st); break;
      default:
        if constexpr (B57) {
          if (lp.radix[s] == 5) int_stage_ip<5, S, P>(a, lp.L, Ns, st);
          else int_stage_ip<7, S, P>(a, lp.L, Ns, st);
        }
        break;
    }
    Ns *= lp.radix[s];
  }
}

// Forward column pass: dice, add carries, weight, length-H DFT, twiddle, store to row k2 of Z.
template <bool FROM_STATE, int NC, bool B57, int P>
__device__ __forceinline__ void int_col_fwd_body(const IterArgs& a, const int m1) {
  extern __shared__ g2 ism[];
  const int H = a.H, W = a.W, ls = a.in.ls_col;
  if (P == 0 && a.in.touch) {
    touch(a.in.hf, plan_slots(a.in.ph));
    touch(a.in.k1 + m1 * H, H);
  }
  if (P == 0 && a.in.dependent) after_previous_pass();
  if (P && threadIdx.x == 0) prefetch_l2(a.in.k1 + m1 * H, H);
  bool wide = false;
#pragma unroll (P == 0 ? 2 : 1)
  for (int m2 = threadIdx.x; m2 < H; m2 += blockDim.x) {
    int v0, v1;
    load_point<FROM_STATE, NC, P == 0>(a, m1, m2, &v0, &v1);
    if (FROM_STATE) wide |= v0 > a.in.vmax || v0 < -a.in.vmax || v1 > a.in.vmax || v1 < -a.in.vmax;
    const uchar2 e = __ldg(reinterpret_cast<const uchar2*>(a.in.e + 2 * (m1 * H + m2)));
    ism[ipad(m2)] = g2{gf::weighted(v0, e.x), gf::weighted(v1, e.y)};
  }
  if (FROM_STATE && wide) atomicOr(&a.status->flags, kStatusWide);
  __syncthreads();
  const g2* res = ism;
  if constexpr (P > 0) int_line_fft_ip<-1, B57, P>(ism, a.in.ph, a.in.hf);
  else res = int_line_fft<-1, B57>(ism, ism + ls, 1, ls, a.in.ph, a.in.hf);
#pragma unroll 2
  for (int k2 = threadIdx.x; k2 < H; k2 += blockDim.x)
    stz(a.Z + (k2 * W + m1), gf::cmul(res[ipad(k2)], __ldg(a.in.k1 + (m1 * H + k2))));
}

template <bool FROM_STATE, int NC, bool B57, int P>
__global__ void __launch_bounds__(kMaxThreads, B57 ? 2 : P ? 4 : 3) ki_col_fwd(IterArgs a) {
  int_col_fwd_body<FROM_STATE, NC, B57, P>(a, blockIdx.x);
}

// Row pair i of the table.  Loaded where it is used (volatile, so the compiler does not keep
// it in registers through the transforms, which need them all).
__device__ __forceinline__ int4 row_pair(const int4* rows, int i) {
  int4 r;
  asm volatile("ld.global.nc.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(rows + i));
  return r;
}

// Row pass over one row pair (a row paired with itself: one line).
template <bool B57>
__device__ __forceinline__ void int_row_body(const IterArgs& a, const int pair) {
  extern __shared__ g2 ism[];
  const int W = a.W, H = a.H, ls = a.in.ls_row;
  g2* other = ism + 2 * ls;
  int nl;
  {
    const int4 r = row_pair(a.in.rows, pair);
    nl = r.x == r.y ? 1 : 2;
    if (a.in.touch) {
      touch(a.in.wf, plan_slots(a.in.pw));
      touch(a.in.pair + r.x * W, W);
      touch(a.in.wi, plan_slots(a.in.pw));
      touch(a.in.k2 + r.x * W, W);
      touch(a.in.k2 + r.y * W, W);
      if (a.in.dependent) after_previous_pass();
    } else if (threadIdx.x < 3) {
      prefetch_l2(threadIdx.x == 0 ? a.in.pair + r.x * W : a.in.k2 + (threadIdx.x == 1 ? r.x : r.y) * W, W);
    }
    for (int idx = threadIdx.x; idx < nl * W; idx += blockDim.x) {
      const int l = idx >= W;
      const int k1 = idx - l * W;
      ism[l * ls + ipad(k1)] = ldz(a.Z + ((l ? r.y : r.x) * W + k1));
    }
  }
  __syncthreads();
  g2* sp = int_line_fft<-1, B57>(ism, other, nl, ls, a.in.pw, a.in.wf);
  g2* nx = sp == ism ? other : ism;
  {
    const int4 r = row_pair(a.in.rows, pair);
    const bool self = r.x == r.y;
    g2* lb = self ? sp : sp + ls;
    // partner position q t + shift mod W, stepped along with t
    const unsigned qW = (unsigned)a.in.qV, uW = (unsigned)W;
    int u = (int)((qW * threadIdx.x + (unsigned)r.z) % uW);
    const int du = (int)(qW * (blockDim.x % uW) % uW);
#pragma unroll 1
    for (int t = threadIdx.x; t < W; t += blockDim.x) {
      if (!self || t <= u) {
        g2 vk, vkp;
        gf::pair_square(sp[ipad(t)], lb[ipad(u)], __ldg(a.in.pair + (r.x * W + t)), &vk, &vkp);
        sp[ipad(t)] = vk;
        if (!self || t != u) lb[ipad(u)] = vkp;
      }
      u += du;
      u -= u >= W ? W : 0;
    }
  }
  __syncthreads();
  const g2* res = int_line_fft<+1, B57>(sp, nx, nl, ls, a.in.pw, a.in.wi);
  const int4 r = row_pair(a.in.rows, pair);
  for (int idx = threadIdx.x; idx < nl * W; idx += blockDim.x) {
    const int l = idx >= W;
    const int m1 = idx - l * W;
    const int row = l ? r.y : r.x;
    stz(a.Z2 + (m1 * H + row), gf::cmul(res[l * ls + ipad(m1)], __ldg(a.in.k2 + (row * W + m1))));
  }
}

// Row pass of a transform over polynomials (t > 1): a row is t interleaved lines of V
// points, line b holding coefficient b, and a frequency's t coefficients are squared mod
// y^t - z (poly_square).  With D = U - conj(U') as in pair_square,
// V = U^2 - (1 + y) D^2 / 4 and V' = U'^2 + conj(the same), coefficient by coefficient.
// U, U' and D are brought into limbs first (each is read t times), then one thread takes
// one coefficient of one frequency; D^2 goes through shared memory, since its product with
// y takes a coefficient from the neighbour.
__device__ __forceinline__ void int_row_poly_body(const IterArgs& a, const int pair) {
  extern __shared__ g2 ism[];
  const int W = a.W, H = a.H, ls = a.in.ls_row, t = a.in.t, V = a.in.V;
  const int4 r = __ldg(a.in.rows + pair);
  const bool self = r.x == r.y;
  const int rows = self ? 1 : 2, nl = rows * t;  // line mirror t + b
  if (a.in.touch) {
    touch(a.in.wf, plan_slots(a.in.pw));
    touch(a.in.pair + r.x * V, V);
    touch(a.in.wi, plan_slots(a.in.pw));
    touch(a.in.k2 + r.x * W, W);
    touch(a.in.k2 + r.y * W, W);
    if (a.in.dependent) after_previous_pass();
  }
  g2* other = ism + 2 * t * ls;
  int4* dif = reinterpret_cast<int4*>(ism + 4 * t * ls);  // line b: D in limbs
  g2* dsq = ism + 5 * t * ls;                             // line b: D^2
  for (int idx = threadIdx.x; idx < rows * W; idx += blockDim.x) {
    const int l = idx >= W;
    const int m1 = idx - l * W;
    const int v = m1 / t;
    ism[(l * t + m1 - v * t) * ls + ipad(v)] = ldz(a.Z + ((l ? r.y : r.x) * W + m1));
  }
  __syncthreads();
  g2* sp = int_line_fft<-1, true>(ism, other, nl, ls, a.in.pw, a.in.wf);
  g2* nx = sp == ism ? other : ism;
  int4* sl = reinterpret_cast<int4*>(sp);
#pragma unroll 1
  for (int step = 0; step < 3; ++step) {
#pragma unroll 1
    for (int x = threadIdx.x; x < W; x += blockDim.x) {
      const int b = x / V;
      const int v = x - b * V;  // frequency position
      const int u = (int)(((unsigned)a.in.qV * (unsigned)v + (unsigned)r.z) % (unsigned)V);
      if (self && u < v) continue;
      const int la = ipad(v), lb = (self ? 0 : t * ls) + ipad(u);
      const int4 z = __ldg(a.in.pair + (r.x * V + v));
      if (step == 0) {
        const g2 p = sp[la + b * ls], q = sp[lb + b * ls];
        dif[la + b * ls] = gf::as_limbs(gf::red(g2{p.re - q.re, p.im + q.im}));
        sl[la + b * ls] = gf::as_limbs(gf::red(p));
        if (la != lb) sl[lb + b * ls] = gf::as_limbs(gf::red(q));
      } else if (step == 1) {
        nx[la + b * ls] = gf::poly_square([&](int c) { return sl[la + c * ls]; }, t, b, z);
        if (la != lb) nx[lb + b * ls] = gf::poly_square([&](int c) { return sl[lb + c * ls]; }, t, b, gf::conj(z));
        dsq[la + b * ls] = gf::poly_square([&](int c) { return dif[la + c * ls]; }, t, b, z);
      } else {
        const g2 e = gf::add(dsq[la + b * ls], b ? dsq[la + (b - 1) * ls] : gf::cmul(dsq[la + (t - 1) * ls], z));
        const g2 pc = g2{gf::rmul(e.re, gf::kMinusQuarter), gf::rmul(e.im, gf::kMinusQuarter)};
        nx[la + b * ls] = gf::red(gf::add(nx[la + b * ls], pc));
        if (la != lb) {
          const g2 s = nx[lb + b * ls];
          nx[lb + b * ls] = gf::red(g2{s.re + pc.re, s.im - pc.im});
        }
      }
    }
    __syncthreads();
  }
  const g2* res = int_line_fft<+1, true>(nx, sp, nl, ls, a.in.pw, a.in.wi);
  for (int idx = threadIdx.x; idx < rows * W; idx += blockDim.x) {
    const int l = idx >= W;
    const int m1 = idx - l * W;
    const int v = m1 / t;
    const int row = l ? r.y : r.x;
    stz(a.Z2 + (m1 * H + row),
        gf::cmul(res[(l * t + m1 - v * t) * ls + ipad(v)], __ldg(a.in.k2 + (row * W + m1))));
  }
}

__global__ void __launch_bounds__(kRowThreads, 2) ki_row_poly(IterArgs a) { int_row_poly_body(a, blockIdx.x); }

// Two builds for radices 8, 4, 2, 3: five CTAs of 192 threads per SM (64 registers) where the
// row pairs are enough to fill them, else 80 registers, which shorten the dependent chains
// of a pass with few CTAs (N = 49152, 49 pairs: 14.1 us against 15.6).
constexpr int kRowsFor5 = 3 * kSms;
template <bool B57, int T, int MB>
__global__ void __launch_bounds__(T, MB) ki_row_sq(IterArgs a) {
  int_row_body<B57>(a, blockIdx.x);
}

// The two products of one point: unweight, check, -2 at word 0 (the LL step), store.
__device__ __forceinline__ void int_store_products(const IterArgs& a, g2 v, int s0, unsigned* fl) {
  const uchar2 e = __ldg(reinterpret_cast<const uchar2*>(a.in.e + s0));
  long long r0 = check_word(gf::unweighted(v.re, e.x), fl);
  const long long r1 = check_word(gf::unweighted(v.im, e.y), fl);
  if (a.in.check_span) {
    const uchar2 sp = __ldg(reinterpret_cast<const uchar2*>(a.span + s0));
    check_span(r0, sp.x, fl);
    check_span(r1, sp.y, fl);
  }
  if (s0 == 0) r0 -= 2;
  *reinterpret_cast<longlong2*>(a.ll + s0) = make_longlong2(r0, r1);
}

// Inverse column pass: inverse length-H DFT, unweight, -2 at word 0, range checks, products.
template <bool B57, int P>
__device__ __forceinline__ void int_col_inv_body(const IterArgs& a, const int m1) {
  extern __shared__ g2 ism[];
  const int H = a.H, ls = a.in.ls_col;
  if (P == 0 && a.in.touch) {
    touch(a.in.hi, plan_slots(a.in.ph));
    if (a.in.dependent) after_previous_pass();
  }
  for (int k2 = threadIdx.x; k2 < H; k2 += blockDim.x) ism[ipad(k2)] = ldz(a.Z2 + (size_t)m1 * H + k2);
  __syncthreads();
  const g2* res = ism;
  if constexpr (P > 0) int_line_fft_ip<+1, B57, P>(ism, a.in.ph, a.in.hi);
  else res = int_line_fft<+1, B57>(ism, ism + ls, 1, ls, a.in.ph, a.in.hi);
  unsigned fl = 0;
  for (int m2 = threadIdx.x; m2 < H; m2 += blockDim.x) int_store_products(a, res[ipad(m2)], 2 * (m1 * H + m2), &fl);
  fl = __reduce_or_sync(0xffffffffu, fl);
  if ((threadIdx.x & 31) == 0 && fl) atomicOr(&a.status->flags, fl);
}

template <bool B57, int P>
__global__ void __launch_bounds__(kMaxThreads, B57 ? 2 : P ? 4 : 3) ki_col_inv(IterArgs a) {
  int_col_inv_body<B57, P>(a, blockIdx.x);
}

// One pass; as a programmatic dependent of the launch before it where the kernel waits for
// that itself (after_previous_pass).
void run(void (*kernel)(IterArgs), int grid, int block, size_t smem, cudaStream_t s, const IterArgs& a, bool dependent) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = dependent ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, a);
}

using IntKernel = void (*)(IterArgs);

template <bool FS, bool B57, int P>
IntKernel col_fwd_nc(int n) {
  const IntKernel kernels[5] = {ki_col_fwd<FS, 2, B57, P>, ki_col_fwd<FS, 3, B57, P>, ki_col_fwd<FS, 4, B57, P>,
                                ki_col_fwd<FS, 5, B57, P>, ki_col_fwd<FS, 6, B57, P>};
  return kernels[n - 2];
}
bool cols_in_place(const IntGeom& g) { return g.col_p && !has57(g.ph); }

// The kernels of the three passes for a geometry.
IntKernel col_fwd_kernel(const IntGeom& g, int n, bool from_state) {
  if (cols_in_place(g)) return from_state ? col_fwd_nc<true, false, kIntHeld>(n) : col_fwd_nc<false, false, kIntHeld>(n);
  if (has57(g.ph)) return from_state ? col_fwd_nc<true, true, 0>(n) : col_fwd_nc<false, true, 0>(n);
  return from_state ? col_fwd_nc<true, false, 0>(n) : col_fwd_nc<false, false, 0>(n);
}
IntKernel row_kernel(const IntGeom& g, int nrows) {
  if (g.t > 1) return ki_row_poly;
  if (has57(g.pw)) return ki_row_sq<true, 256, 2>;
  if (g.t_row <= 192 && nrows > kRowsFor5) return ki_row_sq<false, 192, 5>;
  return ki_row_sq<false, 256, 3>;
}
IntKernel col_inv_kernel(const IntGeom& g) {
  if (cols_in_place(g)) return ki_col_inv<false, kIntHeld>;
  return has57(g.ph) ? ki_col_inv<true, 0> : ki_col_inv<false, 0>;
}

void launch_pass(const IterArgs& a, const IntGeom& g, cudaStream_t s, int which, bool from_state) {
  if (which == 1) run(row_kernel(g, a.in.nrows), a.in.nrows, g.t_row, g.sm_row, s, a, a.in.dependent);
  else
    run(which == 0 ? col_fwd_kernel(g, a.n, from_state) : col_inv_kernel(g), a.W, g.t_col, g.sm_col, s, a,
        !cols_in_place(g) && a.in.dependent);
}

// A kernel's limit is process-wide: it is raised to the layout chooser's bound, whoever asks
// first, and only where a launch needs more than every kernel may have.
cudaError_t raise(IntKernel kernel, size_t smem) {
  if (smem <= 48 * 1024) return cudaSuccess;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxIntSmem);
}

}  // namespace

cudaError_t set_int_smem_limits(const IntGeom& g, int n, int nrows, bool from_state) {
  cudaError_t e;
  if ((e = raise(col_fwd_kernel(g, n, false), g.sm_col))) return e;
  if (from_state && (e = raise(col_fwd_kernel(g, n, true), g.sm_col))) return e;
  if ((e = raise(row_kernel(g, nrows), g.sm_row))) return e;
  return raise(col_inv_kernel(g), g.sm_col);
}

cudaError_t launch_int_kernel(const IterArgs& a, const IntGeom& g, cudaStream_t s, int which) {
  launch_pass(a, g, s, which, false);
  return cudaGetLastError();
}

cudaError_t launch_int_iteration(const IterArgs& a, const IntGeom& g, cudaStream_t s, bool from_state) {
  for (int w = 0; w < 3; ++w) launch_pass(a, g, s, w, from_state);
  return cudaGetLastError();
}

}  // namespace gl
