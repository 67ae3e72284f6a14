"""The integer form (GF(q^2), q = 2^61 - 1) against Python integers on the CPU and against the
FP64 form and the oracle on the GPU.  Everything is exact, so every comparison is equality."""
import ctypes

import numpy as np
import pytest

from gpulucas_gb300 import _build

Q = (1 << 61) - 1
R = (1 << 60) + (1 << 35)


@pytest.fixture(scope="module")
def hc():
    L = ctypes.CDLL(_build.HOSTCHECK)
    i64 = np.ctypeslib.ndpointer(np.int64, flags="C_CONTIGUOUS")
    L.hc_gf_square.argtypes = [ctypes.c_int] * 3 + [np.ctypeslib.ndpointer(np.int32, flags="C_CONTIGUOUS"), i64,
                                                    ctypes.POINTER(ctypes.c_longlong)]
    L.hc_gf_cmul.argtypes = [i64, np.ctypeslib.ndpointer(np.uint64, flags="C_CONTIGUOUS"), i64]
    for f, a in (("hc_gf_red", [ctypes.c_longlong]), ("hc_gf_weighted", [ctypes.c_int, ctypes.c_int]),
                 ("hc_gf_unweighted", [ctypes.c_longlong, ctypes.c_int])):
        getattr(L, f).argtypes = a
        getattr(L, f).restype = ctypes.c_longlong
    return L


def test_field_operations_at_their_bounds(hc):
    rng = np.random.default_rng(61)
    edge = [(1 << 62) - 1, -(1 << 62), 0, 1, -1, Q, -Q, 1 << 61, -(1 << 61), (1 << 31) - 1, -(1 << 31)]
    res = [0, 1, Q - 1, Q >> 1, (Q >> 1) + 1, 1 << 60, (1 << 60) - 1, (1 << 31) - 1, 1 << 30, Q - (1 << 30)]
    for _ in range(20000):
        x = [int(v) for v in rng.integers(-(1 << 62), 1 << 62, 2)]
        w = [int(v) for v in rng.integers(0, Q, 2)]
        for k in range(2):
            if rng.random() < 0.3:
                x[k] = edge[rng.integers(len(edge))]
            if rng.random() < 0.3:
                w[k] = res[rng.integers(len(res))]
        out = np.zeros(2, np.int64)
        hc.hc_gf_cmul(np.array(x, np.int64), np.array(w, np.uint64), out)
        re, im = int(out[0]), int(out[1])
        assert (re - (x[0] * w[0] - x[1] * w[1])) % Q == 0 and (im - (x[0] * w[1] + x[1] * w[0])) % Q == 0
        assert abs(re) <= R and abs(im) <= R
        y = int(rng.integers(-(1 << 63) + (1 << 60) + 1, (1 << 63) - (1 << 60) - 1))
        r = hc.hc_gf_red(y)
        assert (r - y) % Q == 0 and -(1 << 60) - 4 <= r <= (1 << 60) + 3
        e = int(rng.integers(61))
        v = int(rng.integers(-(1 << 28), 1 << 28))
        g = hc.hc_gf_weighted(v, e)
        assert (g - v * pow(2, e, Q)) % Q == 0 and abs(g) <= R
        u = hc.hc_gf_unweighted(x[0] - x[0] // 4, e)  # within 3 R
        assert (u * pow(2, e, Q) - (x[0] - x[0] // 4)) % Q == 0 and -(1 << 60) - 4 <= u <= (1 << 60) + 3
        n = int(rng.integers(-(1 << 59), 1 << 59))  # a product: any representative of it gives it back
        z = n * pow(2, e, Q) % Q + (int(rng.integers(3)) - 1) * Q
        assert hc.hc_gf_unweighted(z - Q if z > 3 * (1 << 60) else z, e) == n


# layouts with every radix first and later, columns or rows with an odd part (rows that pair
# with themselves in number), an odd number of points, and the smallest width
@pytest.mark.parametrize("W,H", [(4, 4), (9, 8), (8, 64), (18, 16), (20, 10), (21, 8), (25, 6), (72, 5), (7, 32),
                                 (36, 35), (15, 15), (63, 25), (128, 8), (5, 2)])
def test_square_of_weighted_words(hc, W, H):
    """out[k] = sum over i + j = k mod N of v_i v_j 2^(b_i + b_j - b_k (- p past the end)),
    b_j = ceil(jp/N): the products an iteration rounds to, without rounding."""
    N = 2 * W * H
    p = 17 * N + 5
    rng = np.random.default_rng(N)
    for amp in (1 << 17, 1):
        v = rng.integers(-amp, amp + 1, N).astype(np.int32)
        if amp > 1:
            v[:] = np.where(rng.random(N) < 0.5, amp, -amp)  # the largest words a state holds
        b = [-((-p * j) // N) for j in range(N + 1)]
        out = np.zeros(N, np.int64)
        peak = ctypes.c_longlong()
        assert hc.hc_gf_square(p, W, H, v, out, ctypes.byref(peak)) == 0
        assert peak.value <= 3 * R
        i = np.arange(N)
        for k in range(0, N, max(1, N // 61)):
            j = (k - i) % N
            s = sum(int(v[x]) * int(v[y]) << (b[x] + b[y] - b[k] - (p if x + y >= N else 0)) for x, y in zip(i, j))
            assert s == out[k]


def test_lengths_the_field_has_no_roots_for(hc):
    out, peak = np.zeros(54, np.int64), ctypes.c_longlong()
    assert hc.hc_gf_square(1000, 27, 1, np.zeros(54, np.int32), out, ctypes.byref(peak)) == -1


def _products(gl, p, N, k, **opts):
    with gl.Plan(p, N, **opts) as pl:
        rep = pl.iterate(k)
        return pl.products(), rep, (pl.info.fft_h, pl.info.fft_w)


# short and long lines, odd parts 1, 3, 5, 7, 9, 15, 25, 63 and carry depths 2..4; a limit
# below the default keeps a plan in FP64
@pytest.mark.gpu
@pytest.mark.parametrize("p,N", [(100003, 5120), (100003, 6272), (90007, 5600), (1000003, 53760), (859433, 49152),
                                 (859433, 50400), (2976221, 163840), (2976221, 201600), (1398269, 86016)])
def test_int_form_products_equal_fp64_form(gl, p, N):
    for k in (1, 2, 70):
        a, ra, _ = _products(gl, p, N, k)
        b, rb, _ = _products(gl, p, N, k, error_limit=0.39)
        assert ra.status == rb.status == 0
        assert (a == b).all(), k
    assert 0.0 < ra.max_roundoff <= rb.max_roundoff


# in-place columns (the layout search may pick either form): long power-of-two columns, and
# rows of more than one butterfly per thread
@pytest.mark.gpu
@pytest.mark.parametrize("p,N", [(9300017, 524288), (20996011, 1179648), (24000001, 1310720), (74207281, 4194304)])
def test_int_form_long_lines_equal_fp64_form(gl, p, N):
    a, ra, _ = _products(gl, p, N, 67)
    b, rb, _ = _products(gl, p, N, 67, error_limit=0.39)
    c, rc, _ = _products(gl, p, N, 67, autotune=0)
    assert ra.status == rb.status == rc.status == 0 and (a == b).all() and (c == b).all()


@pytest.mark.gpu
def test_int_form_follows_the_oracle_and_a_loaded_state(gl, orc):
    p, N = 100003, 5120
    o = orc.IBDWT(p, N).iterate(37)
    d, h = o.state()
    with gl.Plan(p, N) as pl:
        pl.set_carry_state(d, h, 37)
        pl.iterate(100)
        assert (pl.products() == o.iterate(100).ll()).all()
        assert pl.res64() == orc.Exact(p).iterate(137).res64()


@pytest.mark.gpu
@pytest.mark.parametrize("big", [0, 3000000, -(1 << 24)])
def test_captured_host_step_with_words_beyond_the_bound(gl, big):
    """The captured one-iteration step runs in the integer form; a loaded word beyond that
    form's bound sends the step through FP64, in place and into another buffer, with the
    same words as the pageable path (FP64) gives."""
    import torch
    p, N = 1000003, 53760
    rng = np.random.default_rng(3)
    w = rng.integers(-5, 6, N).astype(np.int32) if big else rng.integers(-(1 << 17), 1 << 17, N).astype(np.int32)
    if big:
        w[17] = big
    a = torch.from_numpy(w.copy()).pin_memory()
    b = torch.empty(N, dtype=torch.int32).pin_memory()
    ap, bp = ctypes.c_void_p(a.data_ptr()), ctypes.c_void_p(b.data_ptr())
    rep = gl.IterReport()
    with gl.Plan(p, N) as pl, gl.Plan(p, N) as ref:
        want, _ = ref.iterate_host_words(w, 1)
        assert gl.lib.gl_iterate_host_words(pl._h, ap, 1, bp, ctypes.byref(rep)) == 0
        assert rep.total_iterations == 1 and (b.numpy() == want).all() and (a.numpy() == w).all()
        assert gl.lib.gl_iterate_host_words(pl._h, ap, 1, ap, ctypes.byref(rep)) == 0
        assert rep.total_iterations == 2 and (a.numpy() == want).all()
        for _ in range(70):  # past the FP64 iteration of the schedule
            want, _ = ref.iterate_host_words(want, 1)
            assert gl.lib.gl_iterate_host_words(pl._h, ap, 1, ap, ctypes.byref(rep)) == 0
        assert (a.numpy() == want).all() and (pl.products() == ref.products()).all()


def test_balanced_split_in_32_bits_equals_64(hc):
    """The 32-bit split of the dicing against the general one, ties included."""
    hc.hc_balanced_split.argtypes = [ctypes.c_longlong, ctypes.c_int, ctypes.POINTER(ctypes.c_int),
                                     ctypes.POINTER(ctypes.c_int)]
    hc.hc_balanced_split32.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.POINTER(ctypes.c_int),
                                       ctypes.POINTER(ctypes.c_int)]
    d, h, d2, h2 = (ctypes.c_int() for _ in range(4))
    rng = np.random.default_rng(32)
    for bits in range(14, 24):
        half = 1 << (bits - 1)
        sums = [k * half + o for k in range(-9, 10) for o in (-1, 0, 1)] + [int(v) for v in rng.integers(-8 * half, 8 * half, 300)]
        for s in sums:
            hc.hc_balanced_split(s, bits, d, h)
            hc.hc_balanced_split32(s, bits, d2, h2)
            assert (d.value, h.value) == (d2.value, h2.value), (s, bits)


# lengths whose odd part the field's roots do not cover: transforms over polynomials mod
# y^t - z, t = 3, 5, 7, 9, 25, 27, 49, with and without radices 5 and 7 in the rows
@pytest.mark.gpu
@pytest.mark.parametrize("p,N", [(100003, 5184), (500009, 27648), (300007, 16000), (748003, 44100), (300007, 16200),
                                 (1000003, 52500), (1000003, 54432), (1500007, 78400)])
def test_polynomial_transforms_equal_fp64_form(gl, p, N):
    for k in (1, 66):
        a, ra, _ = _products(gl, p, N, k)
        b, rb, _ = _products(gl, p, N, k, error_limit=0.39)
        assert ra.status == rb.status == 0 and (a == b).all(), k


# layouts chosen without timing (radix-4 stages, a thread per two points) and the
# no-allocation entry on the same lengths: one block of integer iterations, several, none
@pytest.mark.gpu
@pytest.mark.parametrize("p,N", [(100003, 5120), (300007, 16200), (859433, 49152), (1000003, 54432), (1257787, 65536)])
def test_untimed_layouts_and_noalloc_equal_fp64_form(gl, p, N):
    import torch
    start = np.zeros(N, np.int64)
    start[0] = 4
    for k in (1, 2, 66, 130):
        want, _, _ = _products(gl, p, N, k, error_limit=0.39)
        got, _, _ = _products(gl, p, N, k, autotune=0)
        assert (got == want).all(), k
        d = torch.from_numpy(start).cuda()
        err = gl.iterate_noalloc(p, N, d.data_ptr(), d.data_ptr(), k, torch.cuda.current_stream().cuda_stream)
        assert (d.cpu().numpy() == want).all() and 0.0 <= err < 0.4, k


# the resident integer form: one and several launches between FP64 iterations, odd parts in
# the rows, the largest word size it runs at, and lengths whose layout leaves it to FP64
@pytest.mark.gpu
@pytest.mark.parametrize("p,N", [(9689, 512), (21701, 1024), (33013, 1536), (44497, 2048), (60013, 3072), (86243, 4096),
                                 (21023, 1120), (12379, 640), (76003, 3840)])
def test_resident_integer_form_follows_the_oracle(gl, orc, p, N):
    o = orc.IBDWT(p, N)
    with gl.Plan(p, N) as pl:
        assert pl.info.resident_ctas in (8, 16)
        for k in (1, 2, 60, 3, 130):
            rep = pl.iterate(k)
            o.iterate(k)
            assert rep.status == 0 and (pl.products() == o.ll()).all(), k
        d, h = pl.carry_state()
        pl.set_carry_state(d, h, 0)
        pl.iterate(5)
        assert (pl.products() == o.iterate(5).ll()).all()


# the smallest lengths and words of a few bits (where the slice check is not implied by the
# size check), up to the largest carry depth
@pytest.mark.gpu
@pytest.mark.parametrize("p,N", [(127, 16), (127, 64), (607, 40), (1279, 70), (3217, 180), (4423, 1000), (9941, 2250)])
def test_smallest_lengths_and_words_equal_fp64_form(gl, orc, p, N):
    for k in (1, 3, 66):
        want, ra, _ = _products(gl, p, N, k, error_limit=0.39)
        got, rb, _ = _products(gl, p, N, k)
        assert ra.status == rb.status == 0 and (got == want).all(), k
    assert (got == orc.IBDWT(p, N).iterate(66).ll()).all()
