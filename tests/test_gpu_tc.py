"""Split-precision tensor-core class (tcgen05, 3xTF32) vs the FP64 oracle.

GEMM-shaped pairs in PREC_3XTF32 contexts (M, N >= 64, K >= 16) run on the
tcgen05 kernels; tolerance 1e-5 relative to the largest result magnitude
(3xTF32 products with FP32 accumulation over K <= 1024).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-5
TC_LAUNCHES = 4  # result index table, pack A, pack B, persistent tcgen05 GEMM
OZ_LAUNCHES = 5  # exponents of A and B, slices of B, result index table, GEMM


def launches_for(be, k):
    return OZ_LAUNCHES if be.precision in (3, 5) and k <= 512 else TC_LAUNCHES


def rel_err(a, b):
    a = np.asarray(a).reshape(-1)
    b = np.asarray(b).reshape(-1)
    return float(np.max(np.abs(a - b)) / np.max(np.abs(b)))


def rand(rng, dims):
    return rng.standard_normal(dims) + 1j * rng.standard_normal(dims)


@pytest.fixture(params=[(2, None), (2, 0), (4, None), (5, None), (5, 0), (3, None)],
                ids=["3xtf32-mixed", "3xtf32-c64all", "6xtf32-mixed", "ozaki-mixed", "ozaki-c64all", "3xbf16-mixed"])
def be(request, pq):
    prec, small = request.param
    b = pq.GB300Backend(prec, small_elems=small)
    yield b
    b.close()


def run(be, A, ia, B, ib):
    be.save_tensor_data("A", A)
    be.save_tensor_data("B", B)
    n0 = be.launch_count()
    be.contract_tensors("A", ia, "B", ib, "C")
    launched = be.launch_count() - n0
    return be.load_tensor_data("C"), launched


def test_plain_matrix_product(be, O):
    rng = np.random.default_rng(0)
    A = rand(rng, (256, 64))
    B = rand(rng, (64, 128))
    got, nl = run(be, A, [-1, 1], B, [1, -2])
    assert nl == launches_for(be, 64)
    assert rel_err(got, A @ B) < TOL


@pytest.mark.parametrize("m,n,k", [(400, 72, 40), (128, 128, 64), (130, 260, 48), (1000, 96, 272), (200, 80, 600)])
def test_ragged_tiles(be, O, m, n, k):
    rng = np.random.default_rng(m + n + k)
    A = rand(rng, (k, m))
    B = rand(rng, (n, k))
    got, nl = run(be, A, [1, -1], B, [-2, 1])
    assert nl == launches_for(be, k)
    assert rel_err(got, A.T @ B.T) < TOL


def test_persistent_tiles_across_batch(pq, O, be):
    # more output tiles than SMs: each persistent CTA walks several tiles,
    # crossing batch (z) boundaries; ragged M, N and K
    rng = np.random.default_rng(5)
    m, n, k, z = 1000, 100, 40, 7
    A = rand(rng, (m, k, z))
    B = rand(rng, (k, n, z))
    be.save_tensor_data("a", A)
    be.save_tensor_data("b", B)
    import ctypes as C
    from pqgb300 import _lib as L

    h = C.c_void_p()
    rc = be.lib.pq_plan_create(be.ctx, 2, L.arr(C.c_int32, [3, 3]), L.arr(C.c_int32, [0, 1, 3, 1, 2, 3]), 4,
                               L.arr(C.c_int64, [m, k, n, z]), 1, L.arr(C.c_int32, [0, 1]), 3,
                               L.arr(C.c_int32, [3, 2, 0]), C.byref(h))
    L.check(rc, be.ctx, "plan_create")
    ids = L.arr(C.c_int64, [be.id_of("a"), be.id_of("b")])
    L.check(be.lib.pq_plan_execute(h, ids, be.id_of("r")), be.ctx, "execute")
    got = be.load_tensor_data("r")
    ref = np.einsum("mkz,knz->znm", A, B)
    assert rel_err(got, ref) < TOL
    be.lib.pq_plan_destroy(h)


def test_truncation_bias_is_corrected(pq):
    """The tensor core truncates accumulations; the kernel adds the expected
    shrinkage back.  The mean relative change of |C| over a large random
    product stays within 1e-8 (uncorrected it is about -9e-8), so it does not
    build up along a chain of contractions."""
    rng = np.random.default_rng(6)
    A = rand(rng, (512, 256)).astype(np.complex64)
    B = rand(rng, (256, 256)).astype(np.complex64)
    ref = A.astype(np.complex128) @ B.astype(np.complex128)
    for prec in (2, 4):
        be = pq.GB300Backend(prec, small_elems=0)
        got, nl = run(be, A, [-1, 1], B, [1, -2])
        be.close()
        assert nl == TC_LAUNCHES
        bias = float(np.mean(np.abs(got) / np.abs(ref)) - 1)
        assert abs(bias) < 1e-8, (prec, bias)


def test_permuted_bond2_modes(be, O):
    # interleaved free / contracted bond-2 modes in both operands
    rng = np.random.default_rng(3)
    ia = [-1, 1, -2, 2, -3, 3, -4, 4, -5, -6, 5, -7, 6, -8]
    ib = [3, -9, 1, -10, 5, 2, -11, 6, 4, -12, -13, -14, -15, -16]
    A = rand(rng, [2] * len(ia))
    B = rand(rng, [2] * len(ib))
    got, nl = run(be, A, ia, B, ib)
    assert nl == launches_for(be, 2 ** 6)
    assert rel_err(got, O.contract_tensors_arrays(A, ia, B, ib)) < TOL


def test_batched_hyper_mode_via_plan(pq, O, be):
    # a label shared by both operands and the result (batch) inside a plan
    rng = np.random.default_rng(4)
    A = rand(rng, (96, 32, 5))   # m, k, z
    B = rand(rng, (32, 80, 5))   # k, n, z
    be.save_tensor_data("a", A)
    be.save_tensor_data("b", B)
    import ctypes as C
    from pqgb300 import _lib as L

    h = C.c_void_p()
    rc = be.lib.pq_plan_create(be.ctx, 2, L.arr(C.c_int32, [3, 3]), L.arr(C.c_int32, [0, 1, 3, 1, 2, 3]), 4,
                               L.arr(C.c_int64, [96, 32, 80, 5]), 1, L.arr(C.c_int32, [0, 1]), 3,
                               L.arr(C.c_int32, [0, 2, 3]), C.byref(h))
    L.check(rc, be.ctx, "plan_create")
    ids = L.arr(C.c_int64, [be.id_of("a"), be.id_of("b")])
    L.check(be.lib.pq_plan_execute(h, ids, be.id_of("r")), be.ctx, "execute")
    got = be.load_tensor_data("r")
    ref = np.einsum("mkz,knz->mnz", A, B)
    assert rel_err(got, ref) < TOL
    be.lib.pq_plan_destroy(h)


@pytest.mark.parametrize("prec", [2, 4, 5, 3], ids=["3xtf32", "6xtf32", "ozaki", "3xbf16"])
def test_tc_plan_amplitude(pq, O, prec):
    """A sliced single amplitude on the tensor-core path vs the state vector."""
    be = pq.GB300Backend(prec)
    r, c, d = 4, 4, 10
    bits = "0110100111001010"
    g = pq.random_grid_gates(r, c, d, seed=3)
    net = pq.build_network(16, g, backend=be, decompose=True)
    pq.add_input(net, "0" * 16)
    pq.add_output(net, bits)
    steps, cm, mx, _ = pq.planning.best_flop_plan(net, out_edges=[], candidates=("sweep",))
    plan = pq.NetworkPlan(net, steps=steps, out_edges=[])
    sliced = plan.choose_slices(max_sliced=4, log2_target=28)
    amp = plan.run_sliced(sliced, batch=16)
    ref = O.statevector(16, g)[O.amplitude_index(bits)]
    # three bf16 slices keep about 21 bits: a looser bound for that mode
    assert abs(amp - ref) / 2.0 ** -8 < (2e-5 if prec == 3 else 1e-6)
    plan.close()
    be.close()


# ---- exact-accumulation (Ozaki scheme) kernels ------------------------------

def ozaki_backend(pq, small=0):
    return pq.GB300Backend(5, small_elems=small)


def ozaki_bound(A, B, ref):
    from oracle import ozaki_oracle as Z

    return Z.error_bound(np.asarray(A, dtype=np.complex128), np.asarray(B, dtype=np.complex128), ref)


def test_ozaki_matches_cpu_restatement(pq):
    """The device result equals the CPU restatement of the scheme (exact level
    0 and 1 sums, one final rounding): bit for bit on most elements (the
    device's FP32 level-2..4 sum, about 2^-30 of the scale, moves a few % of
    the final roundings), otherwise within one complex64 ulp plus 2^-28 of
    |row of A| |column of B|; and it is the FP64 product up to the scheme's
    error bound."""
    from oracle import ozaki_oracle as Z

    rng = np.random.default_rng(7)
    A = rand(rng, (512, 256)).astype(np.complex64)
    B = rand(rng, (256, 192))  # complex128 (a small tensor)
    be = ozaki_backend(pq, small=1 << 16)
    got, nl = run(be, A, [-1, 1], B, [1, -2])
    be.close()
    assert nl == OZ_LAUNCHES
    got = got.astype(np.complex64)
    orc, _ = Z.ozaki_matmul(A.astype(np.complex128), B)
    na = np.sqrt(np.sum(np.abs(A.astype(np.complex128)) ** 2, axis=1))
    nb = np.sqrt(np.sum(np.abs(B) ** 2, axis=0))
    for part in (np.real, np.imag):
        g, o = part(got).astype(np.float64), part(orc).astype(np.float64)
        ulp = np.spacing(np.abs(o).astype(np.float32)).astype(np.float64)
        assert np.all(np.abs(g - o) <= ulp + 2.0 ** -28 * np.outer(na, nb))
        assert np.mean(g == o) > 0.95
    ref = A.astype(np.complex128) @ B
    assert np.all(np.abs(got - ref) <= ozaki_bound(A, B, ref))


@pytest.mark.parametrize("order", ["mk", "km"])
def test_ozaki_row_scales_and_zero_rows(pq, order):
    """Rows and columns of wildly different magnitude (per-row scaling), an
    all-zero row of A and an all-zero column of B; A contiguous along M (row
    per thread exponent pass) or along K (row per warp)."""
    rng = np.random.default_rng(8)
    A = rand(rng, (300, 128)) * np.exp2(rng.integers(-60, 60, size=(300, 1)))
    B = rand(rng, (128, 100)) * np.exp2(rng.integers(-40, 40, size=(1, 100)))
    A[17] = 0
    B[:, 5] = 0
    A = A.astype(np.complex64)
    be = ozaki_backend(pq)
    if order == "km":
        got, nl = run(be, A.T, [1, -1], B.astype(np.complex64), [1, -2])
    else:
        got, nl = run(be, A, [-1, 1], B.astype(np.complex64), [1, -2])
    be.close()
    assert nl == OZ_LAUNCHES
    B = B.astype(np.complex64).astype(np.complex128)
    ref = A.astype(np.complex128) @ B
    assert np.all(got[17] == 0) and np.all(got[:, 5] == 0)
    assert np.all(np.abs(got - ref) <= ozaki_bound(A, B, ref))


@pytest.mark.parametrize("m,n,k", [(4096, 16, 64), (3000, 24, 48), (2000, 8, 256), (16, 5000, 32), (40, 900, 96)])
def test_ozaki_narrow_pairs(pq, m, n, k):
    """Narrow pairs: 16- and 32-wide tiles for small N, and A/B swapped when
    M is the narrow side (boundary tensors absorbing one qubit's tensor)."""
    rng = np.random.default_rng(m + n + k)
    A = rand(rng, (m, k)).astype(np.complex64)
    B = rand(rng, (k, n)).astype(np.complex64)
    be = ozaki_backend(pq)
    got, nl = run(be, A, [-1, 1], B, [1, -2])
    be.close()
    assert nl == OZ_LAUNCHES
    A, B = A.astype(np.complex128), B.astype(np.complex128)
    ref = A @ B
    assert np.all(np.abs(got - ref) <= ozaki_bound(A, B, ref))


def test_3xbf16_matches_cpu_restatement(pq):
    """Three bf16 slices: the device result is the CPU restatement with
    n_slices = 3 up to one final rounding, within the scheme's bound."""
    from oracle import ozaki_oracle as Z

    rng = np.random.default_rng(10)
    A = rand(rng, (384, 128)).astype(np.complex64)
    B = rand(rng, (128, 200)).astype(np.complex64)
    be = pq.GB300Backend(3, small_elems=0)
    got, nl = run(be, A, [-1, 1], B, [1, -2])
    be.close()
    assert nl == OZ_LAUNCHES
    A, B = A.astype(np.complex128), B.astype(np.complex128)
    orc, _ = Z.ozaki_matmul(A, B, n_slices=3)
    ref = A @ B
    assert np.all(np.abs(got - ref) <= Z.error_bound(A, B, ref, n_slices=3))
    assert np.max(np.abs(got - orc)) <= 2.0 ** -22 * np.max(np.abs(orc))


def test_ozaki_k512_exact_limit(pq):
    """K = 512 is the largest K whose level sums stay exact; K = 513 runs on
    the 6xTF32 kernels."""
    rng = np.random.default_rng(9)
    for k, launches in ((512, OZ_LAUNCHES), (513, TC_LAUNCHES)):
        A = rand(rng, (256, k)).astype(np.complex64)
        B = rand(rng, (k, 128)).astype(np.complex64)
        be = ozaki_backend(pq)
        got, nl = run(be, A, [-1, 1], B, [1, -2])
        be.close()
        assert nl == launches
        ref = A.astype(np.complex128) @ B.astype(np.complex128)
        if launches == OZ_LAUNCHES:
            assert np.all(np.abs(got - ref) <= ozaki_bound(A, B, ref))
        else:
            assert rel_err(got, ref) < TOL


def _restatement_match(got, A, B):
    """complex64 result vs the CPU restatement: within one ulp plus 2^-28 of
    |row of A| |column of B|, bit-identical on most elements."""
    from oracle import ozaki_oracle as Z

    orc, _ = Z.ozaki_matmul(A, B)
    na = np.sqrt(np.sum(np.abs(A) ** 2, axis=1))
    nb = np.sqrt(np.sum(np.abs(B) ** 2, axis=0))
    for part in (np.real, np.imag):
        g, o = part(got).astype(np.float64), part(orc).astype(np.float64)
        ulp = np.spacing(np.abs(o).astype(np.float32)).astype(np.float64)
        assert np.all(np.abs(g - o) <= ulp + 2.0 ** -28 * np.outer(na, nb))
        assert np.mean(g == o) > 0.95


@pytest.mark.parametrize("order", ["mk", "km"])
@pytest.mark.parametrize("n,k,small", [(16, 40, 0), (16, 256, 0), (32, 24, 0), (32, 72, 0), (48, 40, 0),
                                       (64, 256, 0), (16, 48, 1 << 30)],
                         ids=["n16-k40", "n16-k256", "n32-k24", "n32-k72", "n48-k40", "n64-k256", "n16-c128"])
def test_ozaki_narrow_many_tiles_per_cta(pq, order, n, k, small):
    """Narrow tiles (N <= 64: two accumulator sets in TMEM, alternate tiles)
    over many row tiles: 64 * 152 * 3 + 37 rows give every persistent CTA
    three or four tiles (the last one ragged), and with an odd number of K
    tiles the two converter groups (alternate K tiles) swap roles from one
    tile to the next; A contiguous along M or along K (the K-major exponent
    pass), complex64 or complex128, with an all-zero row; a ragged last K
    tile."""
    rng = np.random.default_rng(n + k)
    m = 64 * 152 * 3 + 37
    A = rand(rng, (m, k))
    A[1000] = 0
    B = rand(rng, (k, n))
    if not small:
        A, B = A.astype(np.complex64), B.astype(np.complex64)
    be = ozaki_backend(pq, small=small)
    if order == "km":
        got, nl = run(be, A.T, [1, -1], B, [1, -2])  # stored column-major: K contiguous
    else:
        got, nl = run(be, A, [-1, 1], B, [1, -2])
    be.close()
    assert nl == OZ_LAUNCHES
    A, B = A.astype(np.complex128), B.astype(np.complex128)
    ref = A @ B
    assert np.all(got[1000] == 0)
    assert np.all(np.abs(got - ref) <= ozaki_bound(A, B, ref))
    if not small:
        _restatement_match(got, A, B)


def test_ozaki_narrow_tiles_across_batch(pq, O):
    """A narrow batched pair (hyper mode z kept in the result): persistent
    CTAs cross z boundaries as well as row tiles, three K tiles per tile."""
    import ctypes as C
    from pqgb300 import _lib as L

    rng = np.random.default_rng(12)
    m, k, n, z = 3000, 40, 16, 9
    A = rand(rng, (m, k, z)).astype(np.complex64)
    B = rand(rng, (k, n, z)).astype(np.complex64)
    be = ozaki_backend(pq)
    be.save_tensor_data("a", A)
    be.save_tensor_data("b", B)
    h = C.c_void_p()
    rc = be.lib.pq_plan_create(be.ctx, 2, L.arr(C.c_int32, [3, 3]), L.arr(C.c_int32, [0, 1, 3, 1, 2, 3]), 4,
                               L.arr(C.c_int64, [m, k, n, z]), 1, L.arr(C.c_int32, [0, 1]), 3,
                               L.arr(C.c_int32, [3, 2, 0]), C.byref(h))
    L.check(rc, be.ctx, "plan_create")
    ids = L.arr(C.c_int64, [be.id_of("a"), be.id_of("b")])
    n0 = be.launch_count()
    L.check(be.lib.pq_plan_execute(h, ids, be.id_of("r")), be.ctx, "execute")
    assert be.launch_count() - n0 == OZ_LAUNCHES
    got = be.load_tensor_data("r")
    be.lib.pq_plan_destroy(h)
    be.close()
    A, B = A.astype(np.complex128), B.astype(np.complex128)
    for iz in range(z):
        ref = A[:, :, iz] @ B[:, :, iz]
        assert np.all(np.abs(got[iz].T - ref) <= ozaki_bound(A[:, :, iz], B[:, :, iz], ref))


def test_3xbf16_narrow_many_tiles_per_cta(pq):
    """Three bf16 slices on 16-wide tiles, two or three tiles per CTA."""
    from oracle import ozaki_oracle as Z

    rng = np.random.default_rng(13)
    A = rand(rng, (64 * 152 * 2 + 5, 64)).astype(np.complex64)
    B = rand(rng, (64, 16)).astype(np.complex64)
    be = pq.GB300Backend(3, small_elems=0)
    got, nl = run(be, A, [-1, 1], B, [1, -2])
    be.close()
    assert nl == OZ_LAUNCHES
    A, B = A.astype(np.complex128), B.astype(np.complex128)
    ref = A @ B
    assert np.all(np.abs(got - ref) <= Z.error_bound(A, B, ref, n_slices=3))


def test_ozaki_tall_narrow_pair(pq):
    """More than 65535 * 128 rows (a 2^23-row boundary tensor absorbing a
    16-column gate tensor over K = 32, stored contiguous along K): the exact
    path takes it, the exponent pass on grid x with no 65535 limit."""
    rng = np.random.default_rng(14)
    m, k, n = (1 << 23) + 4097, 32, 16
    A = rng.standard_normal((m, 2 * k), dtype=np.float32).view(np.complex64)
    B = rand(rng, (k, n)).astype(np.complex64)
    be = ozaki_backend(pq)
    got, nl = run(be, A.T, [1, -1], B, [1, -2])  # A.T is (K, M) column-major: no host copy
    be.close()
    assert nl == OZ_LAUNCHES
    rows = np.concatenate([np.arange(64), rng.choice(m, 4096, replace=False), np.arange(m - 64, m)])
    A, B = A[rows].astype(np.complex128), B.astype(np.complex128)
    ref = A @ B
    assert np.all(np.abs(got[rows] - ref) <= ozaki_bound(A, B, ref))


@pytest.mark.parametrize("ia", [[1, -1, -2, 2, -3, 3, -4, 4, -5, 5, -6, 6, -7, -8, -9, -10],
                                [1, 2, -1, -2, 3, -3, 4, -4, 5, -5, 6, -6, -7, -8, -9, -10],
                                [1, 2, 3, -1, -2, 4, -3, 5, -4, 6, -5, -6, -7, -8, -9, -10]],
                         ids=["k-run-2", "k-run-4", "k-run-8"])
def test_ozaki_stride1_mode_contracted(pq, O, ia):
    """A's unit-stride mode is contracted, in a run of 2, 4 or 8 elements
    before its first open mode (a boundary tensor whose fastest qubits meet
    the gate tensor): the exponent pass reads A K-major with 2, 4 or 8 lanes
    per row; all bond-2 modes, K = 64, M = 1024, N = 16."""
    rng = np.random.default_rng(15 + len(ia))
    ib = [1, 2, 3, 4, 5, 6, -11, -12, -13, -14]
    A = (rand(rng, [2] * len(ia)) * np.exp2(rng.integers(-30, 30, size=[2] * len(ia)) // 8)).astype(np.complex64)
    B = rand(rng, [2] * len(ib)).astype(np.complex64)
    be = ozaki_backend(pq)
    got, nl = run(be, A, ia, B, ib)
    be.close()
    assert nl == OZ_LAUNCHES
    ref = O.contract_tensors_arrays(A.astype(np.complex128), ia, B.astype(np.complex128), ib)
    assert rel_err(got, ref) < 3e-7


@pytest.mark.parametrize("small", [1 << 16, 1 << 62], ids=["c64-storage", "c128-storage"])
def test_ozaki4_matches_cpu_restatement(pq, small):
    """Four bf16 slices (PQ_PREC_OZAKI4, ten slice-pair products): the device
    result is the CPU restatement with n_slices = 4 up to the FP32 sum of the
    small levels and the output rounding, and the FP64 product within the
    scheme's bound; with every tensor stored as complex128 the result is not
    rounded to complex64 at all."""
    from oracle import ozaki_oracle as Z

    rng = np.random.default_rng(12)
    A = rand(rng, (384, 256))
    B = rand(rng, (256, 200))
    if small < (1 << 62):
        A = A.astype(np.complex64).astype(np.complex128)
    be = pq.GB300Backend(pq.PREC_OZAKI4, small_elems=small)
    got, nl = run(be, A, [-1, 1], B, [1, -2])
    be.close()
    assert nl == OZ_LAUNCHES
    c128 = small >= (1 << 62)
    orc, _ = Z.ozaki_matmul(A, B, out_dtype=np.complex128 if c128 else np.complex64, n_slices=4)
    ref = A @ B
    bound = Z.error_bound(A, B, ref, n_slices=4)
    assert np.all(np.abs(got - ref) <= bound)
    na = np.sqrt(np.sum(np.abs(A) ** 2, axis=1))
    nb = np.sqrt(np.sum(np.abs(B) ** 2, axis=0))
    tol = (2.0 ** -23 * np.abs(orc) if small < (1 << 62) else 0) + 2.0 ** -28 * np.outer(na, nb)
    assert np.all(np.abs(got - orc) <= tol)


def test_ozaki4_c128_plan_amplitude(pq, O):
    """A sliced amplitude with four slices and complex128 storage against
    the state vector: the error is far below the complex64-storage modes'."""
    be = pq.GB300Backend(pq.PREC_OZAKI4, small_elems=1 << 62)
    r, c, d = 4, 4, 10
    bits = "0110100111001010"
    g = pq.random_grid_gates(r, c, d, seed=3)
    net = pq.build_network(16, g, backend=be, decompose=True)
    pq.add_input(net, "0" * 16)
    pq.add_output(net, bits)
    steps, cm, mx, _ = pq.planning.best_flop_plan(net, out_edges=[], candidates=("sweep",))
    plan = pq.NetworkPlan(net, steps=steps, out_edges=[])
    sliced = plan.choose_slices(max_sliced=4, log2_target=28)
    amp = plan.run_sliced(sliced, batch=16)
    ref = O.statevector(16, g)[O.amplitude_index(bits)]
    assert abs(amp - ref) / 2.0 ** -8 < 1e-7
    plan.close()
    be.close()


@pytest.mark.parametrize("order", ["mk", "km", "k4", "k6"])
@pytest.mark.parametrize("k,n", [(24, 128), (96, 8), (144, 136), (264, 72), (504, 24)])
def test_ozaki_half_split(pq, O, order, k, n):
    """Complex64 results (three fp16 slices): the first slice's 8 or 7 bits on
    either side of K = 128 and 256, ragged K tiles, 16- to 128-wide tiles, A
    contiguous along M, along all of K, and in K runs of 4 (32-byte loads) and 6
    (value by value).  Random rows spanning 12 binades: the scheme's bound.
    Equal entries c (1 + i): every level-0 sum is at its largest, 2K c^2, and
    must be exact; level 1 is 2^-7 of it at most and is truncated at most
    4 ceil(K / 16) <= 128 times by 2^-24 of itself, 2^-24 in all, so with the
    final rounding (2^-24) the result is within 2^-23 of the product."""
    rng = np.random.default_rng(k + n)
    m = 1400  # at least 2^20 multiply-adds in every case
    for data in ("rows", "equal"):
        if data == "rows":
            A = (rand(rng, (m, k)) * np.exp2(-rng.integers(0, 13, size=(m, k)))).astype(np.complex64)
            B = rand(rng, (k, n)).astype(np.complex64)
        else:
            A = np.full((m, k), (1 + 1j) * (1 - 2.0 ** -13), dtype=np.complex64)
            B = np.full((k, n), (1 + 1j) * (1 - 2.0 ** -12), dtype=np.complex64)
        be = ozaki_backend(pq)
        if order == "mk":
            got, nl = run(be, A, [-1, 1], B, [1, -2])
        elif order == "km":
            got, nl = run(be, A.T, [1, -1], B, [1, -2])
        else:
            r = 4 if order == "k4" else 6
            T = A.reshape(m, k // r, r).transpose(2, 0, 1)  # fastest K run first, then M
            got, nl = run(be, T, [2, -1, 1], B.reshape(k // r, r, n), [1, 2, -2])
        be.close()
        assert nl == OZ_LAUNCHES
        A, B = A.astype(np.complex128), B.astype(np.complex128)
        ref = A @ B
        if data == "rows":
            assert np.all(np.abs(got - ref) <= ozaki_bound(A, B, ref))
        else:
            assert np.max(np.abs(got - ref)) <= 2.0 ** -23 * np.max(np.abs(ref))


@pytest.mark.parametrize("k", [16, 24, 48, 64, 136])
@pytest.mark.parametrize("order", ["mk", "km"])
def test_ozaki_wide_many_tiles_per_cta(pq, order, k):
    """128-wide tiles, three or four per persistent CTA with a ragged last one,
    from one K tile (fewer than the ring's three stages) to nine: the sums of a
    tile parked while the next tile's level-2 MMAs run in the other TMEM
    block.  Complex64, an all-zero row, columns past N (N = 200: a full and a
    ragged column tile)."""
    rng = np.random.default_rng(k)
    m, n = 64 * 152 + 64 * 70 + 37, 200
    A = rand(rng, (m, k)).astype(np.complex64)
    A[1000] = 0
    B = rand(rng, (k, n)).astype(np.complex64)
    be = ozaki_backend(pq)
    if order == "km":
        got, nl = run(be, A.T, [1, -1], B, [1, -2])
    else:
        got, nl = run(be, A, [-1, 1], B, [1, -2])
    be.close()
    assert nl == OZ_LAUNCHES
    A, B = A.astype(np.complex128), B.astype(np.complex128)
    ref = A @ B
    assert np.all(got[1000] == 0)
    assert np.all(np.abs(got - ref) <= ozaki_bound(A, B, ref))
    _restatement_match(got, A, B)


@pytest.mark.parametrize("prec", [2, 4], ids=["3xtf32", "6xtf32"])
@pytest.mark.parametrize("m,n,k,a_order,c_order", [
    (64, 64, 272, "mk", "mn"),       # one tile, half its rows padding
    (1281, 65, 17, "mk", "mn"),      # one row, column and K value past a tile; rows not 32-byte aligned
    (300, 127, 33, "mk", "nm"),      # transposed result: scattered stores
    (2500, 128, 68, "km", "mn"),     # A contiguous along M; K tiles grouped in a pack block
    (20000, 129, 36, "mk", "mn"),    # several output tiles per CTA, odd result rows
    (128, 4100, 132, "km", "nm"),    # B the wide side
])
def test_tf32_tile_edges(pq, prec, m, n, k, a_order, c_order):
    """The TF32 kernels at the edges of their 128 x 64 tiles and 16-deep K tiles
    and on both sides of the wide loads and stores (aligned adjacent values, or
    not).  TF32 terms of an operand are exact to 2^-22 and a chunk of 16 takes a
    few truncations of 2^-23, so that an element is within 2^-20 of
    |row of A| |column of B|."""
    rng = np.random.default_rng(m + n + k)
    A = rand(rng, (m, k)).astype(np.complex64)
    B = rand(rng, (k, n)).astype(np.complex64)
    be = pq.GB300Backend(prec, small_elems=0)
    got, nl = run(be, A if a_order == "mk" else A.T, [-1, 1] if a_order == "mk" else [1, -1], B,
                  [1, -2])
    if c_order == "nm":
        # the same product with the operands' roles exchanged: C is stored n by m
        got, nl = run(be, B, [1, -1], A if a_order == "mk" else A.T, [-2, 1] if a_order == "mk" else [1, -2])
        got = got.T
    be.close()
    assert nl == TC_LAUNCHES
    A, B = A.astype(np.complex128), B.astype(np.complex128)
    bound = np.outer(np.sqrt(np.sum(np.abs(A) ** 2, axis=1)), np.sqrt(np.sum(np.abs(B) ** 2, axis=0)))
    assert np.all(np.abs(got - A @ B) <= 2.0 ** -20 * bound)


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("k1,k2,k3", [(2, 2, 32), (2, 8, 16), (2, 3, 24), (4, 3, 8), (3, 2, 8), (2, 32, 4), (8, 64, 1)])
def test_ozaki_row_scales_over_split_k_runs(pq, dtype, k1, k2, k3):
    """Row exponents of an operand whose leading run along K is several modes
    that its partner stores apart (runs of 4 to 512, some no multiple of four
    or of the lanes), with rows of wildly different magnitude; error_bound is
    the scheme's own bound on each element."""
    rng = np.random.default_rng(k1 * 1000 + k2 * 10 + k3)
    m1, m2, n = 5, 301, 96
    A = rand(rng, (k1, k2, m1, k3, m2)) * np.exp2(rng.integers(-50, 50, size=(1, 1, m1, 1, m2)))
    B = rand(rng, (k2, n, k1, k3))
    A, B = A.astype(dtype), B.astype(dtype)
    be = ozaki_backend(pq, small=0 if dtype is np.complex64 else 1 << 30)
    got, nl = run(be, A, [1, 2, -1, 3, -2], B, [2, -3, 1, 3])
    be.close()
    assert nl == OZ_LAUNCHES
    A2 = A.astype(np.complex128).transpose(2, 4, 0, 1, 3).reshape(m1 * m2, -1)
    B2 = B.astype(np.complex128).transpose(2, 0, 3, 1).reshape(-1, n)
    ref = A2 @ B2
    assert np.all(np.abs(got.reshape(m1 * m2, n) - ref) <= ozaki_bound(A2, B2, ref))


@pytest.mark.parametrize("m,n,k,spread", [
    (2048, 128, 16, 0),     # every warp's columns whole and in range
    (2500, 200, 16, 10),    # a ragged last column range, rows past the end
    (1100, 256, 40, 62),    # products of the scales leave the normal floats: both loops in one tile
])
def test_ozaki_wide_store_loops(pq, m, n, k, spread):
    """128-wide tiles store a warp's columns without branches where all scales
    are normal floats, one by one elsewhere (ragged N, zero rows and columns,
    results below 2^-126); within the scheme's bound either way.  Results
    below the smallest normal float round to multiples of 2^-149."""
    rng = np.random.default_rng(m + n + k)
    A = rand(rng, (m, k)) * np.exp2(rng.integers(-spread, 1, size=(m, 1)))
    B = rand(rng, (k, n)) * np.exp2(rng.integers(-spread, 1, size=(1, n)))
    A[m // 2] = 0
    B[:, n - 3] = 0
    A[: m // 3] *= 2.0 ** -min(spread, 60)
    A, B = A.astype(np.complex64), B.astype(np.complex64)
    be = ozaki_backend(pq)
    got, nl = run(be, A, [-1, 1], B, [1, -2])
    be.close()
    assert nl == OZ_LAUNCHES
    A, B = A.astype(np.complex128), B.astype(np.complex128)
    ref = A @ B
    assert np.all(got[m // 2] == 0) and np.all(got[:, n - 3] == 0)
    assert np.all(np.abs(got - ref) <= ozaki_bound(A, B, ref) + 2.0 ** -148)


@pytest.mark.parametrize("k", [16, 32])
@pytest.mark.parametrize("n", [128, 40])
def test_ozaki_bf16_small_products_first(pq, k, n):
    """Five bf16 slices with complex128 results: within a K tile the rest's
    products go in by level, the smallest first, so that few of them meet the
    accumulator at its full size.  The rms error is that of the sums restated in
    this order, with 5 % for sampling; in the order of A's slices the device's
    is 11 to 12 % above it."""
    from oracle import ozaki_oracle as Z

    rng = np.random.default_rng(k + n)
    m = (1 << 21) // (k * n)
    A, B = rand(rng, (m, k)), rand(rng, (k, n))
    be = ozaki_backend(pq, small=1 << 62)
    got, nl = run(be, A, [-1, 1], B, [1, -2])
    be.close()
    assert nl == OZ_LAUNCHES
    A, got = A[:96], got[:96].astype(np.clongdouble)
    ref = A.astype(np.clongdouble) @ B.astype(np.clongdouble)
    scale = np.exp2((Z.row_exponents(A)[:, None] + Z.row_exponents(B.T)[None, :]).astype(np.float64))

    def rms(x):
        return np.sqrt(np.mean((np.abs(x - ref) / scale) ** 2))

    assert rms(got) <= 1.05 * rms(Z.accumulate(A, B, False))


@pytest.mark.parametrize("k", [64, 128, 144, 256, 272, 512])
@pytest.mark.parametrize("n", [128, 40, 16])
def test_ozaki_cancelling_leading_level(pq, k, n):
    """Rows whose leading slices cancel over K while the next ones add up
    (+-0.75 alternating plus 0.95 2^-8, columns equal in pairs): level 1 is then
    the result and has to be exact.  Either split, all tile widths, within the
    scheme's bound (a second slice of 12 bits, whose level 1 does not fit, is at
    ten times that for K = 512)."""
    rng = np.random.default_rng(k + n)
    m = max(1400, (1 << 21) // (k * n))
    a = np.where(np.arange(k) % 2 == 0, 0.75, -0.75) + 0.95 * 2.0 ** -8
    A = (np.tile(a, (m, 1)) * np.exp2(rng.integers(-20, 20, (m, 1)))).astype(np.complex64)
    A[m // 2:] *= 1j
    B = np.repeat(rng.uniform(0.9, 1.0, (k // 2, n)), 2, axis=0).astype(np.complex64)
    be = ozaki_backend(pq)
    got, nl = run(be, A, [-1, 1], B, [1, -2])
    be.close()
    assert nl == OZ_LAUNCHES
    A, B = A.astype(np.complex128), B.astype(np.complex128)
    ref = A @ B
    assert np.all(np.abs(got - ref) <= ozaki_bound(A, B, ref))


@pytest.mark.parametrize("k", [32, 128, 256])
@pytest.mark.parametrize("n", [128, 40, 16])
def test_ozaki_half_split_keeps_small_slices(pq, k, n):
    """Results near 2^-20 of the scales (columns equal in pairs, rows that
    nearly cancel over them), where the complex64 rounding hides nothing: the
    rms error is that of the restated sums, with a factor of 2 for the adder's
    own alignment.  Lost fp16 subnormals or a residual of 2^-33 (three slices)
    would be 8 times that and more."""
    from oracle import ozaki_oracle as Z

    rng = np.random.default_rng(k + n)
    m = max(1400, (1 << 21) // (k * n))
    B = np.repeat(rng.uniform(0.5, 1, (k // 2, n)) * np.exp(2j * np.pi * rng.random((k // 2, n))), 2, axis=0)
    a = rand(rng, (m, k // 2))
    A = np.empty((m, k), dtype=np.complex128)
    A[:, 0::2], A[:, 1::2] = a, -a + 1e-6 * rand(rng, a.shape)
    A, B = A.astype(np.complex64), B.astype(np.complex64)
    be = ozaki_backend(pq)
    got, nl = run(be, A, [-1, 1], B, [1, -2])
    be.close()
    assert nl == OZ_LAUNCHES
    A, B = A.astype(np.complex128)[:48], B.astype(np.complex128)
    ref = A.astype(np.clongdouble) @ B.astype(np.clongdouble)
    scale = np.exp2((Z.row_exponents(A)[:, None] + Z.row_exponents(B.T)[None, :]).astype(np.float64))

    def rms(x):
        return np.sqrt(np.mean((np.abs(x - ref) / scale) ** 2))

    assert rms(got[:48].astype(np.clongdouble)) <= 2 * rms(Z.accumulate(A, B, True).astype(np.complex64))


@pytest.mark.parametrize("prec", [2, 4], ids=["3xtf32", "6xtf32"])
@pytest.mark.parametrize("m,n,k,z", [
    (300, 128, 36, 1),   # two whole column tiles, every row of C on a 32-byte boundary
    (300, 127, 33, 1),   # rows of C on 8-byte boundaries only
    (400, 68, 20, 3),    # a ragged column tile of four, batched
    (400, 70, 20, 2),    # the last group of four half outside N; rows on 16-byte boundaries
    (500, 65, 48, 2),    # one column past the tile
])
def test_tf32_columns_adjacent_in_result(pq, prec, m, n, k, z):
    """The result stored with B's free index fastest (a plan's requested order),
    where four adjacent columns leave as one 32-byte store if aligned.  An
    element is within 2^-20 of |row of A| |column of B| (TF32 terms of an operand
    are exact to 2^-22, a chunk of 16 takes a few truncations of 2^-23)."""
    import ctypes as C
    from pqgb300 import _lib as L

    rng = np.random.default_rng(m + n + k + z)
    A = rand(rng, (m, k, z)).astype(np.complex64)
    B = rand(rng, (k, n, z)).astype(np.complex64)
    be = pq.GB300Backend(prec, small_elems=0)
    be.save_tensor_data("a", A)
    be.save_tensor_data("b", B)
    h = C.c_void_p()
    rc = be.lib.pq_plan_create(be.ctx, 2, L.arr(C.c_int32, [3, 3]), L.arr(C.c_int32, [0, 1, 3, 1, 2, 3]), 4,
                               L.arr(C.c_int64, [m, k, n, z]), 1, L.arr(C.c_int32, [0, 1]), 3,
                               L.arr(C.c_int32, [2, 0, 3]), C.byref(h))
    L.check(rc, be.ctx, "plan_create")
    ids = L.arr(C.c_int64, [be.id_of("a"), be.id_of("b")])
    n0 = be.launch_count()
    L.check(be.lib.pq_plan_execute(h, ids, be.id_of("r")), be.ctx, "execute")
    assert be.launch_count() - n0 == TC_LAUNCHES
    got = be.load_tensor_data("r")
    be.lib.pq_plan_destroy(h)
    be.close()
    A, B = A.astype(np.complex128), B.astype(np.complex128)
    for iz in range(z):
        bound = np.outer(np.linalg.norm(A[:, :, iz], axis=1), np.linalg.norm(B[:, :, iz], axis=0))
        assert np.all(np.abs(got[:, :, iz].T - A[:, :, iz] @ B[:, :, iz]) <= 2.0 ** -20 * bound)
