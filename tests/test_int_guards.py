"""Guards around the integer form: memory that an early-resident pass reads, what a failed call
leaves behind, which form a plan runs, and the calls of an integer plan that run in FP64."""
import ctypes
import os
import re
import subprocess
import sys

import numpy as np
import pytest

from gpulucas_gb300 import _build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "gpulucas_gb300", "csrc")


def _code(name):
    """A source file without its comments."""
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_early_resident_passes_read_written_memory_with_ordinary_loads():
    """A programmatic dependent is resident while the pass before it still writes the
    products and work arrays, so it may not read them through the non-coherent path."""
    nc = re.compile(r"__ldg\s*\((?:[^()]|\([^()]*\))*\ba\.(?:ll|Z|Z2|digit|hi)\b")
    for name in ("gl_dice.cuh", "gl_int_kernels.cu"):
        assert not nc.search(_code(name)), name
    k = _code("gl_int_kernels.cu")
    # every pass that may be launched as a dependent (P == 0) asks for the ordinary loads
    assert re.findall(r"load_point<([^>]*)>", k) == ["FROM_STATE, NC, P == 0"]
    assert "dependent) after_previous_pass()" in k


@pytest.mark.gpu
def test_batch_gives_row_units_room_for_the_stage_values(gl):
    """A plan with row_pass = 2 reads its stage values through L1; the batch's row kernel
    copies them behind the line buffers all the same."""
    p, N = 1257787, 65536
    o = {"fft_h": 128, "max_radix_row": 4}
    with gl.Plan(p, N, row_pass=2, **o) as a, gl.Plan(p, N, row_pass=1, **o) as b, gl.Plan(p, N) as want:
        assert a.info.row_variant == 2 and b.info.row_variant == 1
        assert a.info.smem_row < b.info.smem_row
        with gl.Batch(plans=[a]) as batch:
            assert batch.info.smem_row >= b.info.smem_row
            batch.iterate(70)
        want.iterate(70)
        assert (a.products() == want.products()).all()


# operator new that fails on request for blocks of a size or more
_NEW_SHIM = r"""
#include <cstdlib>
#include <new>
static std::size_t g_limit = 0;
extern "C" void fail_new_from(std::size_t n) { g_limit = n; }
void* operator new(std::size_t n) {
  if (g_limit && n >= g_limit) throw std::bad_alloc();
  void* p = std::malloc(n ? n : 1);
  if (!p) throw std::bad_alloc();
  return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
"""

_NOALLOC_CHILD = r"""
import ctypes, sys
import numpy as np
import torch
sys.path.insert(0, sys.argv[1])
import gpulucas_gb300 as gl
arm = ctypes.CDLL(None).fail_new_from
arm.argtypes = [ctypes.c_size_t]

def call(p, N, k, limit=0):
    d = torch.zeros(N, dtype=torch.int64, device="cuda")
    d[0] = 4
    err = ctypes.c_double()
    torch.cuda.synchronize()
    arm(limit)
    rc = gl.lib.gl_iterate_noalloc(p, N, ctypes.c_void_p(d.data_ptr()), ctypes.c_void_p(d.data_ptr()), k,
                                   ctypes.byref(err), None)
    arm(0)
    return rc, d.cpu().numpy()

def want(p, N, k):
    with gl.Plan(p, N, mode=gl.MODE_PLAIN) as pl:
        pl.iterate(k)
        return pl.products()

A, B, C = (21701, 1024), (44497, 2048), (86243, 4096)  # growing: staging is kept between calls
rc, a = call(*A, 5)
assert rc == 0 and (a == want(*A, 5)).all()
rc, _ = call(*B, 5, 4096)           # no memory for B's integer tables
assert rc == gl.GL_ERR_NOMEM, rc
rc, a = call(*A, 5)                 # B's FP64 tables had replaced A's
assert rc == 0 and (a == want(*A, 5)).all()
rc, b = call(*B, 5)
assert rc == 0 and (b == want(*B, 5)).all()
for k in (0, 1, 2):                 # N/1024 iterations pay for the integer form's tables
    rc, c = call(*C, k, 4096)
    assert rc == 0 and (k == 0 or (c == want(*C, k)).all()), (k, rc)
rc, c = call(*C, 2, 4096)
assert rc == gl.GL_ERR_NOMEM, rc
rc, c = call(*C, 5)
assert rc == 0 and (c == want(*C, 5)).all()
print("done")
"""


@pytest.mark.gpu
def test_noalloc_call_that_runs_out_of_host_memory_leaves_no_stale_tables(tmp_path):
    src, shim = tmp_path / "new.cpp", tmp_path / "new.so"
    src.write_text(_NEW_SHIM)
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", str(src), "-o", str(shim)], check=True)
    r = subprocess.run([sys.executable, "-c", _NOALLOC_CHILD, ROOT], env=dict(os.environ, LD_PRELOAD=str(shim)),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "done" in r.stdout, r.stderr[-2000:]


_FIRST_CALL_CHILD = r"""
import sys
import torch
sys.path.insert(0, sys.argv[1])
import gpulucas_gb300 as gl
p, N = 859433, 49152
d = torch.zeros(N, dtype=torch.int64, device="cuda")
d[0] = 4
torch.cuda.synchronize()
free = [torch.cuda.mem_get_info()[0]]
for _ in range(2):
    gl.iterate_noalloc(p, N, d.data_ptr(), d.data_ptr(), 70, 0)
    free.append(torch.cuda.mem_get_info()[0])
print(free[0] - free[1], free[1] - free[2])
"""


@pytest.mark.gpu
def test_noalloc_first_call_loads_only_the_kernels_it_launches():
    """The call allocates nothing, but the driver loads each kernel's code when it is first
    named, in granules of 2 MiB: two for the plain form's kernels, one for the integer form's
    three of this geometry.  All of the integer form's kernels would take two."""
    r = subprocess.run([sys.executable, "-c", _FIRST_CALL_CHILD, ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    first, second = map(int, r.stdout.split())
    assert first <= 6 << 20 and second == 0


@pytest.mark.gpu
def test_fp64_iterations_of_an_integer_plan_run_a_timed_variant(gl):
    """The integer search fixes the column length; the FP64 form's variants are timed for it.
    At 2048 x 2048 every timed variant beats the untimed default (two line buffers, radix-8
    rows in the kernel for any radix) by several per cent."""
    p, N = 74207281, 4194304
    with gl.Plan(p, N) as pl:
        assert pl.info.col_variant != -1 or pl.info.row_variant != -1
        assert pl.iterate(60).max_roundoff == 0.0  # integer iterations
    with gl.Plan(p, N, autotune=0) as pl:
        assert pl.info.col_variant == -1 and pl.info.row_variant == -1


# a device of a given size: cudaMalloc fails beyond it, as it would on a full one
_MALLOC_SHIM = r"""
#include <cuda_runtime.h>
#include <map>
#include <mutex>
static std::mutex g_lock;
static std::map<void*, size_t> g_held;
static size_t g_used = 0, g_limit = 0;
extern "C" {
cudaError_t __real_cudaMalloc(void**, size_t);
cudaError_t __real_cudaFree(void*);
void shim_limit(size_t n) { g_limit = n; }
size_t shim_used() { return g_used; }
cudaError_t __wrap_cudaMalloc(void** p, size_t n) {
  std::lock_guard<std::mutex> l(g_lock);
  if (g_limit && g_used + n > g_limit) return cudaErrorMemoryAllocation;
  const cudaError_t e = __real_cudaMalloc(p, n);
  if (e == cudaSuccess) g_used += g_held[*p] = n;
  return e;
}
cudaError_t __wrap_cudaFree(void* p) {
  std::lock_guard<std::mutex> l(g_lock);
  g_used -= g_held[p];
  g_held.erase(p);
  return __real_cudaFree(p);
}
}
"""


@pytest.fixture(scope="module")
def limited(tmp_path_factory):
    """The library linked with a cudaMalloc that a test can limit."""
    d = tmp_path_factory.mktemp("limited")
    (d / "shim.cu").write_text(_MALLOC_SHIM)
    objs = [os.path.join(_build.BUILD, os.path.splitext(s)[0] + ".o") for s in _build.SOURCES]
    if not all(map(os.path.exists, objs)):
        pytest.skip("the library's object files are not here")
    subprocess.run([_build.nvcc(), "-c", "-std=c++17", "-Xcompiler", "-fPIC", str(d / "shim.cu"), "-o", str(d / "shim.o")],
                   check=True)
    subprocess.run([_build.nvcc(), "-shared"] + _build.ARCH + ["-o", str(d / "limited.so")] + objs +
                   [str(d / "shim.o"), "-Xlinker", "--wrap=cudaMalloc", "-Xlinker", "--wrap=cudaFree"], check=True)
    lib = ctypes.CDLL(str(d / "limited.so"))
    lib.shim_limit.argtypes = [ctypes.c_size_t]
    lib.shim_used.restype = ctypes.c_size_t
    lib.gl_iterate.argtypes = [ctypes.c_void_p, ctypes.c_int64, ctypes.c_void_p]
    return lib


@pytest.mark.gpu
def test_plan_without_room_for_the_integer_tables_runs_fp64(gl, limited):
    """Device memory for the FP64 form's arrays but not for the integer form's 25 bytes per
    word beside them: the plan is made, and runs FP64 in every iteration."""
    p, N, k = 1257787, 65536, 66
    with gl.Plan(p, N, error_limit=0.39) as ref:
        need = ref.info.device_bytes
        ref.iterate(k)
        want = ref.products()
    h, info, rep = ctypes.c_void_p(), gl.PlanInfo(), gl.IterReport()
    out = np.empty(N, np.int64)
    for limit, fits in ((need + 65536, False), (need + 30 * N, True), (need // 2, None)):
        limited.shim_limit(limit)
        rc = limited.gl_plan_create(p, N, None, ctypes.byref(h))
        if fits is None:
            assert rc == gl.GL_ERR_NOMEM and limited.shim_used() == 0
            continue
        assert rc == 0, (limit, rc)
        assert limited.gl_plan_get_info(h, ctypes.byref(info)) == 0
        assert (info.device_bytes > need + 24 * N) == fits and limited.shim_used() == info.device_bytes
        assert limited.gl_iterate(h, 60, ctypes.byref(rep)) == 0
        assert (rep.max_roundoff == 0.0) == fits  # an FP64 iteration measures its round-off
        assert limited.gl_iterate(h, k - 60, ctypes.byref(rep)) == 0
        assert limited.gl_get_products(h, ctypes.c_void_p(out.ctypes.data)) == 0
        assert (out == want).all()
        assert limited.gl_plan_destroy(h) == 0 and limited.shim_used() == 0
    limited.shim_limit(0)


@pytest.mark.gpu
def test_find_signal_size_reports_the_time_of_the_plan_it_describes(gl):
    """The length is ranked and its time reported for the form that a plan of it runs.  Where
    that is the integer form, FP64 takes about twice as long at these lengths."""
    p = 9300017
    N, ms, err = gl.find_signal_size(p)
    with gl.Plan(p, N) as pl:
        integer = pl.iterate(60).max_roundoff == 0.0
        pl.iterate(64)
        plan_ms = min(pl.iterate(256).ms for _ in range(3)) / 256
    assert 0.8 < ms / plan_ms < 1.25 and 0.0 < err < 0.30
    with gl.Plan(p, N, error_limit=0.39) as pl:
        pl.iterate(64)
        fp64_ms = min(pl.iterate(256).ms for _ in range(3)) / 256
    assert integer and plan_ms < 0.75 * fp64_ms


Q = (1 << 61) - 1
R = (1 << 60) + (1 << 35)
MAX_PRODUCT = (1 << 60) - 6


@pytest.fixture(scope="module")
def hc():
    lib = ctypes.CDLL(_build.HOSTCHECK)
    i64 = np.ctypeslib.ndpointer(np.int64, flags="C_CONTIGUOUS")
    lib.hc_gf_as_limbs.argtypes = [i64, np.ctypeslib.ndpointer(np.int32, flags="C_CONTIGUOUS")]
    lib.hc_gf_poly_square.argtypes = [ctypes.c_int, i64, np.ctypeslib.ndpointer(np.uint64, flags="C_CONTIGUOUS"), i64]
    lib.hc_gf_unweighted.argtypes = [ctypes.c_longlong, ctypes.c_int]
    lib.hc_gf_unweighted.restype = ctypes.c_longlong
    return lib


# values whose limbs are at their bounds, and those within R at its ends
_EDGE = [s * v for s in (1, -1) for v in ((1 << 60) + (1 << 30), (1 << 60) - (1 << 30) - 1, (1 << 60) + (1 << 35), 1 << 60,
                                          1 << 30, (1 << 31) - 1, 0)]


def test_values_in_limbs_at_their_bounds(hc):
    out = np.zeros(4, np.int32)
    for a in _EDGE:
        for b in _EDGE:
            hc.hc_gf_as_limbs(np.array([a, b], np.int64), out)
            c = [int(v) for v in out]
            assert c[0] + (c[1] << 31) == a and c[2] + (c[3] << 31) == b
            assert abs(c[0]) <= 1 << 30 and abs(c[2]) <= 1 << 30
            assert abs(c[1]) <= (1 << 29) + 16 and abs(c[3]) <= (1 << 29) + 16


@pytest.mark.parametrize("t", [3, 5, 7, 9, 15, 21, 25, 27, 35, 45, 49])
def test_polynomial_squares_at_the_limbs_bounds(hc, t):
    """Every length of polynomial that the integer form takes, against Python integers: all
    coefficients at one bound (the sums of products at their largest), mixed, and random."""
    rng = np.random.default_rng(t)
    out = np.zeros(2 * t, np.int64)
    zs = [(0, Q - 1), (Q >> 1, (Q >> 1) + 1), ((1 << 60) - 1, 1 << 60), (1 << 30, Q - (1 << 30))]
    cases = [[e] * (2 * t) for e in _EDGE] + [[e, -e] * t for e in _EDGE[:4]]
    cases += [[_EDGE[i] for i in rng.integers(len(_EDGE), size=2 * t)] for _ in range(6)]
    cases += [[int(v) for v in rng.integers(-R, R + 1, size=2 * t)] for _ in range(6)]
    for i, u in enumerate(cases):
        zc, zd = zs[i % len(zs)] if i % 3 else [int(v) for v in rng.integers(0, Q, 2)]
        hc.hc_gf_poly_square(t, np.array(u, np.int64), np.array([zc, zd], np.uint64), out)
        for b in range(t):
            re = im = 0
            for half in (0, 1):
                hr = hi = 0
                for j in range(t):
                    k = b + half * t - j
                    if 0 <= k < t:
                        hr += u[2 * j] * u[2 * k] - u[2 * j + 1] * u[2 * k + 1]
                        hi += u[2 * j] * u[2 * k + 1] + u[2 * j + 1] * u[2 * k]
                if half:
                    hr, hi = hr * zc - hi * zd, hr * zd + hi * zc
                re, im = re + hr, im + hi
            x, y = int(out[2 * b]), int(out[2 * b + 1])
            assert (x - re) % Q == 0 and (y - im) % Q == 0, (i, b)
            assert abs(x) <= R and abs(y) <= R


def test_products_up_to_their_bound_come_back_themselves(hc):
    """Any representative that the inverse transform may give of a product within the bound
    that plans are held to."""
    rng = np.random.default_rng(60)
    ns = [s * (MAX_PRODUCT - d) for s in (1, -1) for d in (0, 1, 2, 3, 1 << 20)] + [
        s * (1 << 59) + d for s in (1, -1) for d in (-1, 0, 1)] + [
        int(v) for v in rng.integers(-MAX_PRODUCT, MAX_PRODUCT + 1, 200)]
    for n in ns:
        for e in range(61):
            for k in (-1, 0, 1):
                x = n * pow(2, e, Q) % Q + k * Q
                if abs(x) <= 3 * R:
                    assert hc.hc_gf_unweighted(x, e) == n


def test_int_info_layout_matches_header(tmp_path, gl):
    lines = ["#include <stdio.h>", "#include <stddef.h>", '#include "gpulucas.h"', "int main(void) {",
             'printf("%zu\\n", sizeof(gl_int_info));']
    names = [n for n, _ in gl.IntInfo._fields_]
    lines += [f'printf("%zu\\n", offsetof(gl_int_info, {n}));' for n in names] + ["return 0; }"]
    (tmp_path / "l.c").write_text("\n".join(lines))
    subprocess.run(["gcc", "-std=c11", "-I", os.path.join(ROOT, "include"), str(tmp_path / "l.c"), "-o",
                    str(tmp_path / "l")], check=True)
    got = [int(x) for x in subprocess.run([str(tmp_path / "l")], check=True, capture_output=True, text=True).stdout.split()]
    assert got == [ctypes.sizeof(gl.IntInfo)] + [getattr(gl.IntInfo, n).offset for n in names]


# every length that tests/test_int_form.py and the test below compare, with the polynomial length of its integer
# form and whether the resident form runs it
_INTEGER = [(100003, 5120, 1, 0), (100003, 6272, 7, 0), (90007, 5600, 1, 0), (1000003, 53760, 1, 0),
            (859433, 49152, 1, 0), (859433, 50400, 1, 0), (2976221, 163840, 1, 0), (2976221, 201600, 1, 0),
            (1398269, 86016, 1, 0), (9300017, 524288, 1, 0), (20996011, 1179648, 1, 0), (24000001, 1310720, 1, 0),
            (74207281, 4194304, 1, 0), (100003, 5184, 9, 0), (500009, 27648, 3, 0), (300007, 16000, 5, 0),
            (748003, 44100, 7, 0), (300007, 16200, 9, 0), (1000003, 52500, 25, 0), (1000003, 54432, 27, 0),
            (1500007, 78400, 7, 0), (800011, 43904, 49, 0),
            (1257787, 65536, 1, 0), (9689, 512, 1, 1), (21701, 1024, 1, 1),
            (33013, 1536, 1, 1), (44497, 2048, 1, 1), (60013, 3072, 1, 1), (86243, 4096, 1, 1), (76003, 3840, 1, 1)]


@pytest.mark.gpu
@pytest.mark.parametrize("p,N,t,resident", _INTEGER)
def test_the_lengths_compared_run_the_integer_form(gl, p, N, t, resident):
    """A silent fall back to FP64 would pass every comparison of products.  Both by what the
    plan says and by what it does: 60 iterations without a round-off, against some in FP64."""
    for opts in ({}, {"autotune": 0}) if N < 100000 else ({"autotune": 0},):
        with gl.Plan(p, N, **opts) as pl:
            f = pl.int_info
            assert f.integer == 1 and f.fp64_every == 64 and f.poly == t and bool(f.resident_ctas) == bool(resident)
            V, H = pl.info.fft_w // t, pl.info.fft_h
            assert np.prod([r for r in f.radix_w if r]) == V and np.prod([r for r in f.radix_h if r]) == H
            assert f.threads_col and f.threads_row and f.smem_col and f.smem_row
            assert pl.iterate(60).max_roundoff == 0.0 and pl.iterate(4).max_roundoff > 0.0
            row = "ki_row_poly" if t > 1 else "ki_row_sq"
            assert list(pl.profile_kernels(1)) == ["ki_col_fwd", row, "ki_col_inv"]


@pytest.mark.gpu
@pytest.mark.parametrize("opts", [{"error_limit": 0.39}, {"fft_h": 64}, {"batch_layout": 1}, {"col_inplace": -1}])
def test_options_that_keep_a_plan_in_fp64_say_so(gl, opts):
    with gl.Plan(100003, 5120, **opts) as pl:
        f = pl.int_info
        assert not f.integer and not f.fp64_every and not f.threads_col
        assert pl.iterate(60).max_roundoff > 0.0
        assert list(pl.profile_kernels(1)) == ["k_col_fwd", "k_row_sq", "k_col_inv"]


@pytest.mark.gpu
@pytest.mark.parametrize("p,N", [(800011, 43904), (45878401, 2592000)])
def test_longest_polynomials_equal_fp64_form(gl, orc, p, N):
    """t = 49 and 45 (odd parts 7^3 and 3^4 5^3), the longest that the integer form takes."""
    for k in (1, 66):
        with gl.Plan(p, N) as a, gl.Plan(p, N, error_limit=0.39) as b:
            assert a.int_info.poly in (45, 49) and not b.int_info.integer
            a.iterate(k)
            b.iterate(k)
            assert (a.products() == b.products()).all(), k
            assert k == 1 or p > 1000000 or a.res64() == orc.Exact(p).iterate(k).res64()


@pytest.mark.gpu
@pytest.mark.parametrize("N", [81000, 98784, 162000, 324000])
def test_plans_run_fp64_where_it_is_faster(gl, N):
    """Long polynomials (t = 45, 49) at lengths where the FP64 form takes 5 to 12 % less: the
    plan runs it, as a plan that may not run the other does."""
    p = int(18.3 * N) | 1
    ms = []
    for limit in (0.4, 0.39):
        with gl.Plan(p, N, error_limit=limit) as pl:
            pl.iterate(64, check=False)
            ms.append(min(pl.iterate(256, check=False).ms for _ in range(3)) / 256)
    assert ms[0] < 1.03 * ms[1]


@pytest.mark.gpu
@pytest.mark.parametrize("first,second", [((86243, 4096, 0.4), (9689, 512, 0.4)), ((76003, 3840, 0.4), (76003, 3840, 0.39)),
                                          ((44497, 2048, 0.39), (21701, 1024, 0.39))])
def test_a_resident_plan_runs_on_after_a_smaller_one_is_made(gl, orc, first, second):
    """The resident kernels' shared-memory limit is the process's, not a plan's."""
    p, N, limit = first
    with gl.Plan(p, N, error_limit=limit) as a, gl.Plan(second[0], second[1], error_limit=second[2]) as b:
        assert a.info.resident_ctas and b.info.resident_ctas
        a.iterate(70)
        assert (a.products() == orc.IBDWT(p, N).iterate(70).ll()).all()
