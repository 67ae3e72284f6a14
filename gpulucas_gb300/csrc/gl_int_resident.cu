// gl_int_resident.cu -- the resident form of short tests in exact integer arithmetic.
//
// One thread-block cluster holds the test, as in the FP64 resident form (gl_kernels.cu):
// products, exponents, flags, the inter-pass tables and the stage tables in distributed
// shared memory, many iterations per launch, the passes separated by cluster barriers.
// Lines are short (tens of points), so an iteration is a chain of latencies: a radix-8
// butterfly of one warp takes some 4000 cycles in FP64, where every instruction holds the
// pipe for 64, and about 700 here.  N = 2048: 14.3 -> 10.2 us per iteration; what is left
// is one warp's latencies and instruction fetch between barriers (radix-4 or -2 stages,
// 128 threads, and line DFTs out of line measured the same or slower).
//
// Columns of a power-of-two length H only: then row k2 pairs with row H - k2, and pair c
// is row-table entry c.
#include <cooperative_groups.h>

#include "gl_dice.cuh"
#include "gl_int_stage.cuh"

namespace gl {
namespace cg = cooperative_groups;

namespace {

struct IntResidentArgs {
  IterArgs a;
  IntResidentGeom g;
  int iters;
};

template <int NC>
__global__ void __launch_bounds__(kIntResidentThreads, 1) ki_resident(const __grid_constant__ IntResidentArgs ra) {
  cg::cluster_group cl = cg::this_cluster();
  const IterArgs& a = ra.a;
  const IntResidentGeom& g = ra.g;
  extern __shared__ __align__(16) unsigned char rsm[];
  const int rank = (int)cl.block_rank();
  const int C = g.C, cw = g.cw, H = a.H, W = a.W;
  const int lsc = a.in.ls_col, lsr = a.in.ls_row;
  const int c0 = rank * cw;
  const int npl = (H / 2 - rank) / C + 1;  // my pairs c = rank + C lp <= H/2 (rank < C <= H/2 + 1)
  g2* zc = reinterpret_cast<g2*>(rsm + g.o_zc);
  g2* zc2 = reinterpret_cast<g2*>(rsm + g.o_zc2);
  g2* zr = reinterpret_cast<g2*>(rsm + g.o_zr);
  g2* zr2 = reinterpret_cast<g2*>(rsm + g.o_zr2);
  long long* ll = reinterpret_cast<long long*>(rsm + g.o_ll);
  unsigned char *ex = rsm + g.o_ex, *fl = rsm + g.o_fl, *sp = rsm + g.o_sp;
  int4* K1 = reinterpret_cast<int4*>(rsm + g.o_K1);
  int4* pr = reinterpret_cast<int4*>(rsm + g.o_pr);
  int4* K2 = reinterpret_cast<int4*>(rsm + g.o_K2);
  int4* hf = reinterpret_cast<int4*>(rsm + g.o_hf);
  int4* hi = reinterpret_cast<int4*>(rsm + g.o_hi);
  int4* wf = reinterpret_cast<int4*>(rsm + g.o_wf);
  int4* wi = reinterpret_cast<int4*>(rsm + g.o_wi);
  const int T = blockDim.x, tid = threadIdx.x;
  // H (int_resident_geom) and C (8 or 16) are powers of two, so divisions by them are
  // shifts: an iteration is a chain of latencies, and a division by a run-time value is
  // tens of instructions of it.  us per iteration: 12.67 -> 12.38 at N = 4096, 14.05 -> 13.46
  // at 3840, 10.44 -> 10.18 at 1536, 10.20 -> 10.18 at 2048.
  const int lh = 31 - __clz(H), lC = 31 - __clz(C);

  const int nw = cw * 2 * H;  // my words: one contiguous block of the column-major arrays
  const int wbase = c0 * 2 * H;
  for (int i = tid; i < nw; i += T) {
    ll[i] = a.ll[wbase + i];
    ex[i] = a.in.e[wbase + i];
    fl[i] = a.flags[wbase + i];
    sp[i] = a.span[wbase + i];
  }
  for (int i = tid; i < cw * H; i += T) K1[i] = __ldg(a.in.k1 + c0 * H + i);
  for (int i = tid; i < npl * W; i += T) {
    const int lp = i / W, t = i - lp * W;
    pr[i] = __ldg(a.in.pair + (rank + C * lp) * W + t);
  }
  for (int i = tid; i < 2 * npl * W; i += T) {
    const int s = i / W, m1 = i - s * W;
    const int c = rank + C * (s >> 1);
    const int row = (s & 1) ? (H - c) % H : c;
    K2[i] = __ldg(a.in.k2 + row * W + m1);
  }
  for (int i = tid; i < g.hn; i += T) {
    hf[i] = __ldg(a.in.hf + i);
    hi[i] = __ldg(a.in.hi + i);
  }
  for (int i = tid; i < g.wn; i += T) {
    wf[i] = __ldg(a.in.wf + i);
    wi[i] = __ldg(a.in.wi + i);
  }
  cl.sync();

  unsigned flg = 0;
  for (int it = 0; it < ra.iters; ++it) {
    // (A) dice, weight, column DFTs, twiddle, scatter to the row owners
    for (int idx = tid; idx < cw * H; idx += T) {
      const int lc = idx >> lh, m2 = idx - (lc << lh);
      const int m1 = c0 + lc, s0 = 2 * idx;
      long long P[NC + 3];
      P[0] = ll[s0 + 1];
      P[1] = ll[s0];
      uint32_t fm = 0;
#pragma unroll
      for (int d = 1; d <= (NC + 2) / 2; ++d) {  // the words of point m - d, column m1 - d
        int c = m1 - d, r = m2;
        if (c < 0) {
          c += W;
          r = r == 0 ? H - 1 : r - 1;
        }
        const int o = c / cw;
        const int li = 2 * ((c - o * cw) * H + r);
        if (d == 1) fm = *cl.map_shared_rank(fl + li + 1, o);
        const long long* q = cl.map_shared_rank(ll + li, o);
        P[2 * d] = q[1];
        if (2 * d + 1 < NC + 3) P[2 * d + 1] = q[0];
      }
      int v0, v1;
      dice_pair<NC>(P, a.LO, fm, fl[s0], fl[s0 + 1], &v0, &v1);
      zc[lc * lsc + ipad(m2)] = g2{gf::weighted(v0, ex[s0]), gf::weighted(v1, ex[s0 + 1])};
    }
    __syncthreads();
    {
      const g2* res = int_line_fft<-1, true, true>(zc, zc2, cw, lsc, a.in.ph, hf);
      for (int idx = tid; idx < cw * H; idx += T) {
        const int lc = idx >> lh, k2 = idx - (lc << lh);
        const g2 v = gf::cmul(res[lc * lsc + ipad(k2)], K1[idx]);
        const int c = k2 <= H / 2 ? k2 : H - k2;
        const int slot = 2 * (c >> lC) + (k2 == c ? 0 : 1);
        *cl.map_shared_rank(zr + slot * lsr + ipad(c0 + lc), c & (C - 1)) = v;
      }
    }
    cl.sync();

    // (B) row pairs
    {
      const int nl = 2 * npl;
      g2* s1 = int_line_fft<-1, true, true>(zr, zr2, nl, lsr, a.in.pw, wf);
      g2* other = s1 == zr ? zr2 : zr;
      for (int idx = tid; idx < npl * W; idx += T) {
        const int lp = idx / W, t = idx - lp * W;
        const int c = rank + C * lp;
        const bool self = c == 0 || 2 * c == H;
        g2* la = s1 + 2 * lp * lsr;
        g2* lb = self ? la : la + lsr;
        const unsigned uq = (unsigned)a.in.qV * (unsigned)t + (unsigned)__ldg(&a.in.rows[c].z);
        const int u = (int)((W & (W - 1)) == 0 ? uq & (unsigned)(W - 1) : uq % (unsigned)W);
        if (self && u < t) continue;
        g2 vk, vkp;
        gf::pair_square(la[ipad(t)], lb[ipad(u)], pr[idx], &vk, &vkp);
        la[ipad(t)] = vk;
        if (!self || t != u) lb[ipad(u)] = vkp;
      }
      __syncthreads();
      const g2* res = int_line_fft<+1, true, true>(s1, other, nl, lsr, a.in.pw, wi);
      for (int idx = tid; idx < nl * W; idx += T) {
        const int s = idx / W, m1 = idx - s * W;
        const int c = rank + C * (s >> 1);
        if ((s & 1) && (c == 0 || 2 * c == H)) continue;  // a self-paired row has one line
        const int row = (s & 1) ? H - c : c;
        const g2 v = gf::cmul(res[s * lsr + ipad(m1)], K2[idx]);
        const int o = m1 / cw;
        *cl.map_shared_rank(zc + (m1 - o * cw) * lsc + ipad(row), o) = v;
      }
    }
    cl.sync();

    // (C) inverse column DFTs, unweight, range checks, -2
    {
      const g2* res = int_line_fft<+1, true, true>(zc, zc2, cw, lsc, a.in.ph, hi);
      for (int idx = tid; idx < cw * H; idx += T) {
        const int lc = idx >> lh, m2 = idx - (lc << lh);
        const int s0 = 2 * idx;
        const g2 v = res[lc * lsc + ipad(m2)];
        long long r0 = check_word(gf::unweighted(v.re, ex[s0]), &flg);
        const long long r1 = check_word(gf::unweighted(v.im, ex[s0 + 1]), &flg);
        if (a.in.check_span) {
          check_span(r0, sp[s0], &flg);
          check_span(r1, sp[s0 + 1], &flg);
        }
        if (rank == 0 && idx == 0) r0 -= 2;  // word 0
        ll[s0] = r0;
        ll[s0 + 1] = r1;
      }
    }
    cl.sync();
  }
  if (flg) atomicOr(&a.status->flags, flg);
  for (int i = tid; i < nw; i += T) a.ll[wbase + i] = ll[i];
}

void cluster_config(int C, int smem, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at) {
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = C;
  at->val.clusterDim.y = 1;
  at->val.clusterDim.z = 1;
  cfg->gridDim = dim3(C);
  cfg->blockDim = dim3(kIntResidentThreads);
  cfg->dynamicSmemBytes = smem;
  cfg->attrs = at;
  cfg->numAttrs = 1;
}

template <int NC>
cudaError_t fits(int smem, int C, int* clusters) {
  cudaError_t e = cudaFuncSetAttribute(ki_resident<NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess && C > 8)
    e = cudaFuncSetAttribute(ki_resident<NC>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at;
  cluster_config(C, smem, &cfg, &at);
  return cudaOccupancyMaxActiveClusters(clusters, ki_resident<NC>, &cfg);
}

template <int NC>
cudaError_t launch(const IntResidentArgs& ra, cudaStream_t s) {
  // the attribute is the largest any plan asked for
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at;
  cluster_config(ra.g.C, ra.g.smem, &cfg, &at);
  cfg.stream = s;
  return cudaLaunchKernelEx(&cfg, ki_resident<NC>, ra);
}

}  // namespace

cudaError_t int_resident_geom(int H, int W, const IntGeom& ig, int hn, int wn, int n, IntResidentGeom* r) {
  if (ig.t != 1 || (H & (H - 1))) return cudaErrorInvalidConfiguration;
  for (int C : {8, 16}) {
    if (W % C || H / 2 + 1 < C) continue;
    IntResidentGeom g{};
    g.C = C;
    g.cw = W / C;
    g.hn = hn;
    g.wn = wn;
    const int npl = (H / 2) / C + 1;
    size_t o = 0;
    auto take = [&](size_t bytes) {
      const size_t at = o;
      o = (o + bytes + 15) & ~(size_t)15;
      return (int)at;
    };
    const size_t colb = (size_t)g.cw * int_stride(H) * 16, rowb = (size_t)2 * npl * int_stride(W) * 16;
    const size_t words = (size_t)g.cw * 2 * H;
    g.o_zc = take(colb);
    g.o_zc2 = take(colb);
    g.o_zr = take(rowb);
    g.o_zr2 = take(rowb);
    g.o_ll = take(words * 8);
    g.o_ex = take(words);
    g.o_fl = take(words);
    g.o_sp = take(words);
    g.o_K1 = take((size_t)g.cw * H * 16);
    g.o_pr = take((size_t)npl * W * 16);
    g.o_K2 = take((size_t)2 * npl * W * 16);
    g.o_hf = take((size_t)hn * 16);
    g.o_hi = take((size_t)hn * 16);
    g.o_wf = take((size_t)wn * 16);
    g.o_wi = take((size_t)wn * 16);
    if (o > (size_t)kIntResidentSmem) continue;
    g.smem = (int)o;
    int clusters = 0;
    cudaError_t e = cudaErrorInvalidValue;
    switch (n) {
      case 2: e = fits<2>(kIntResidentSmem, C, &clusters); break;
      case 3: e = fits<3>(kIntResidentSmem, C, &clusters); break;
      case 4: e = fits<4>(kIntResidentSmem, C, &clusters); break;
      case 5: e = fits<5>(kIntResidentSmem, C, &clusters); break;
      default: e = fits<6>(kIntResidentSmem, C, &clusters); break;
    }
    if (e != cudaSuccess || clusters < 1) {
      cudaGetLastError();  // clear a refused configuration
      continue;
    }
    *r = g;
    return cudaSuccess;
  }
  return cudaErrorInvalidConfiguration;
}

cudaError_t launch_int_resident(const IterArgs& a, const IntResidentGeom& g, int iters, cudaStream_t s) {
  const IntResidentArgs ra{a, g, iters};
  switch (a.n) {
    case 2: return launch<2>(ra, s);
    case 3: return launch<3>(ra, s);
    case 4: return launch<4>(ra, s);
    case 5: return launch<5>(ra, s);
    default: return launch<6>(ra, s);
  }
}

}  // namespace gl
