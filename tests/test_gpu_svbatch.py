"""Grouped state vectors of many circuits (pq_svbatch_*) against the FP64
oracle's state-vector simulator of the original, unfused gates.

Tolerance: complex64 states with FP32 block products, 2e-6 of the largest
amplitude magnitude of each circuit's state.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _circuits(pq, specs, n_bits=16):
    from pqgb300 import circuits as CI

    out, raw = [], []
    for i, (n, d) in enumerate(specs):
        r, c = CI.grid_shape(n)
        gates = pq.random_grid_gates(r, c, d, seed=500 + i)
        bits = pq.random_bitstrings(n, n_bits, seed=900 + i)
        out.append((n, CI.fuse_gates(gates, 4), bits))
        raw.append((n, r, c, d, 500 + i, bits))
    return out, raw


SPECS = [(6, 5), (9, 7), (12, 9), (14, 6), (10, 12), (7, 3), (13, 8)]


def _reference(O, raw):
    refs = []
    for n, r, c, d, seed, bits in raw:
        sv = O.statevector(n, O.random_grid_gates(r, c, d, seed=seed))
        refs.append((sv[[O.amplitude_index(b) for b in bits]], np.max(np.abs(sv))))
    return refs


def test_svbatch_matches_oracle(pq, O):
    from pqgb300.svbatch import StateVectorBatch

    circs, raw = _circuits(pq, SPECS)
    refs = _reference(O, raw)
    be = pq.GB300Backend(pq.PREC_C64)
    sb = StateVectorBatch(be, circs)
    info = sb.info()
    assert info["chunks"] == 1
    # one launch per block index of the deepest circuit, plus init and gather
    assert info["kernel_launches"] == 2 + max(len(b) for _, b, _ in circs)
    for _ in range(2):  # the first execution records the graph, the second replays it
        got = sb.execute()
        for g, (ref, scale) in zip(got, refs):
            assert np.max(np.abs(g - ref)) <= 2e-6 * scale
    sb.close()
    be.close()


def test_svbatch_chunks_give_the_same_amplitudes(pq, O):
    """A budget of one 2^14-amplitude state splits the batch: the 14-qubit
    circuit alone, then every smaller one (2^13 + 2^12 + ... fits); the
    amplitudes are bit-identical to one chunk's."""
    from pqgb300.svbatch import StateVectorBatch

    circs, raw = _circuits(pq, SPECS)
    be = pq.GB300Backend(pq.PREC_C64)
    one = StateVectorBatch(be, circs).execute()
    sb = StateVectorBatch(be, circs, state_budget_bytes=8 << 14)
    assert sb.info()["chunks"] == 2
    many = sb.execute()
    for a, b in zip(one, many):
        assert np.array_equal(a, b)
    sb.close()
    be.close()


def test_svbatch_rejects_bad_input(pq):
    from pqgb300 import _lib as L
    from pqgb300.svbatch import StateVectorBatch

    be = pq.GB300Backend(pq.PREC_C64)
    H = np.array([[1, 1], [1, -1]]) / np.sqrt(2)
    with pytest.raises(L.PQError):
        StateVectorBatch(be, [(3, [(H, [4])], ["000"])])  # qubit 4 of a 3-qubit circuit
    with pytest.raises(L.PQError):
        StateVectorBatch(be, [(3, [(np.eye(32), [1, 2, 3, 4, 5])], ["000"])])  # five-qubit block
    with pytest.raises(ValueError):
        StateVectorBatch(be, [(3, [(np.eye(4), [1])], ["000"])])  # matrix of the wrong size
    sb = StateVectorBatch(be, [(3, [(H, [2])], ["000", "010"])])
    got = sb.execute()[0]
    assert np.allclose(got, [1 / np.sqrt(2), 1 / np.sqrt(2)], atol=1e-7)
    sb.close()
    be.close()


@pytest.mark.parametrize("n,qs", [(1, [1]), (2, [2, 1]), (2, [2]), (5, [1]), (5, [2, 1]), (5, [1, 3]), (6, [4, 1, 2]),
                                  (6, [3, 2, 5]), (4, [4, 2, 1, 3]), (7, [1, 7, 2, 4]), (9, [6, 1, 9, 3]),
                                  (11, [5, 11, 2, 8])])
def test_svbatch_block_positions(pq, n, qs):
    """One dense block after a random product state, its qubits listed in any
    order: qubits 1 and 2 in the block (four adjacent amplitudes per access),
    qubit 1 alone (two), neither; the smallest states.  Every amplitude is two
    sums of 2^k FP32 products (2^k + 2 roundings each of unit-norm rows and
    fibers) after n one-qubit passes of the same kind with two products."""
    from pqgb300.svbatch import StateVectorBatch

    rng = np.random.default_rng(n * 100 + sum(qs))

    def haar(d):
        q, r = np.linalg.qr(rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d)))
        return q * (np.diag(r) / np.abs(np.diag(r)))

    blocks = [(haar(2), [q]) for q in range(1, n + 1)] + [(haar(1 << len(qs)), qs)]
    psi = np.zeros((2,) * n, dtype=np.complex128)
    psi[(0,) * n] = 1
    for U, b in blocks:  # axis a holds qubit n - a; the first listed qubit is U's low bit
        k = len(b)
        axes = [n - q for q in reversed(b)]
        psi = np.tensordot(U.reshape((2,) * (2 * k)), psi, axes=(list(range(k, 2 * k)), axes))
        psi = np.moveaxis(psi, list(range(k)), axes)
    bits = [format(i, f"0{n}b")[::-1] for i in range(1 << n)]
    be = pq.GB300Backend(pq.PREC_C64)
    sb = StateVectorBatch(be, [(n, blocks, bits)])
    got = sb.execute()[0]
    sb.close()
    be.close()
    tol = 2.0 ** -24 * (2 * (len(qs) ** 2 + 2 ** len(qs) + 2) + 8 * n)
    assert np.linalg.norm(got - psi.reshape(-1)) <= tol


@pytest.mark.parametrize("n,qs", [(3, [2]), (6, [1, 2]), (7, [1, 5]), (8, [3, 7]), (9, [2, 4, 9])])
def test_svbatch_sums_of_small_blocks(pq, n, qs):
    """One-qubit blocks add each output's real part up in one chain of fused
    multiply-adds, larger ones as the difference of two: whichever rounds less
    with that many terms.  Equal to those sums in FP32, bit for bit."""
    from pqgb300.svbatch import StateVectorBatch

    def fma(a, b, c):
        return (np.asarray(a, np.longdouble) * np.longdouble(b) + np.asarray(c, np.longdouble)).astype(np.float32)

    rng = np.random.default_rng(n + sum(qs))

    def haar(d):
        q, r = np.linalg.qr(rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d)))
        return q * (np.diag(r) / np.abs(np.diag(r)))

    blocks = [(haar(2), [q]) for q in range(1, n + 1)] + [(haar(1 << len(qs)), qs), (haar(2), [n])]
    re, im = np.zeros(1 << n, np.float32), np.zeros(1 << n, np.float32)
    re[0] = 1
    index = np.arange(1 << n)
    for U, b in blocks:
        mask = sum(1 << (q - 1) for q in b)
        base = index[(index & mask) == 0]
        at = [base + sum(((c >> i) & 1) << (q - 1) for i, q in enumerate(b)) for c in range(1 << len(b))]
        x, y = [re[a] for a in at], [im[a] for a in at]
        for o, a in enumerate(at):
            sr, sm, si = np.float32(0), np.float32(0), np.float32(0)
            for c in range(1 << len(b)):
                ux, uy = np.float32(U[o, c].real), np.float32(U[o, c].imag)
                sr = fma(x[c], ux, sr)
                if len(b) == 1:
                    sr = fma(-y[c], uy, sr)
                else:
                    sm = fma(y[c], uy, sm)
                si = fma(y[c], ux, fma(x[c], uy, si))
            re[a], im[a] = sr - sm, si
    be = pq.GB300Backend(pq.PREC_C64)
    sb = StateVectorBatch(be, [(n, blocks, [format(i, f"0{n}b")[::-1] for i in range(1 << n)])])
    got = sb.execute()[0]
    sb.close()
    be.close()
    assert np.array_equal(got.real, re) and np.array_equal(got.imag, im)


@pytest.mark.parametrize("count", [127, 128, 129, 16384, 16385, 20000])
def test_svbatch_many_small_circuits(pq, count):
    """Launch tables around 128 entries (one look by 128 threads) and 128^2 (two
    rounds of narrowing): circuits of one and two qubits, each with a rotation
    of its own, so that a block working on another's entry shows."""
    from pqgb300.svbatch import StateVectorBatch

    angle = np.random.default_rng(count).uniform(0, np.pi, count)
    circs = []
    for i, a in enumerate(angle):
        R = np.array([[np.cos(a), -np.sin(a)], [np.sin(a), np.cos(a)]])
        circs.append((1 + i % 2, [(R, [1 + i % 2])], ["01" if i % 2 else "1"]))
    be = pq.GB300Backend(pq.PREC_C64)
    sb = StateVectorBatch(be, circs)
    got = np.concatenate(sb.execute())
    sb.close()
    be.close()
    assert np.array_equal(got, np.sin(angle).astype(np.float32).astype(np.complex128))
