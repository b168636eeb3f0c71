"""The work that users of this framework have it do, as cases to time and compare.

Each case is a plain dict; ``prepare`` builds what a program has in hand before
the call (tensors, compiled plan, batch or model handle), ``run`` makes one
pass through the public entry points, ``exact`` gives the same outputs from
plain 64-bit torch / numpy code, and ``work`` counts the bytes and flops that
a pass cannot do without.

Kinds of case
  gate      one backend contraction: state and gate uploaded, contracted,
            result read back (the backend method table used directly)
  qft       a whole circuit contracted pair by pair: network built, wavefunction
            contracted, state vector read back
  state     a compiled plan over a circuit fused into blocks of up to four
            qubits, executed for 1024 amplitudes of random bitstrings
  svbatch   many uneven circuits as one grouped state-vector batch
  amp       amplitudes of a grid circuit for bitstrings that share all but their
            last bits (a sampler's group), one after the other through one
            compiled plan, every leaf uploaded anew for each, unsliced or sliced
  multi     64 amplitudes of a grid circuit in one contraction (a shared
            bitstring index on the output tensors)
  mlp       the cost model's forward and backward pass over a batch
"""
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]


def _package():
    """The framework's package directory, imported as ``pqgb300``."""
    if "pqgb300" in sys.modules:
        return sys.modules["pqgb300"]
    pkg = ROOT / "picoquant.jl_gb300"
    spec = importlib.util.spec_from_file_location("pqgb300", pkg / "__init__.py", submodule_search_locations=[str(pkg)])
    mod = importlib.util.module_from_spec(spec)
    sys.modules["pqgb300"] = mod
    spec.loader.exec_module(mod)
    return mod


# ---- the cases ---------------------------------------------------------------

def listed():
    return [
        # the smallest call: a two-qubit gate on a 10-qubit state, uploads and
        # download included (latency of the method table)
        {"name": "gate_n10_c128", "kind": "gate", "n": 10, "k": 2, "prec": "c128"},
        # a 10-qubit QFT contracted interactively to its state vector, in the
        # reference's element type: ~70 nodes, every pair one launch
        {"name": "qft_n10_c128", "kind": "qft", "n": 10, "prec": "c128"},
        # 1024 amplitudes of the 4x5 depth-12 circuit in complex128 and in the
        # mixed-precision mode (every block one pass over 2^20 amplitudes)
        {"name": "state_4x5_d12_c128", "kind": "state", "rows": 4, "cols": 5, "depth": 12, "prec": "c128"},
        {"name": "state_4x5_d12_ozaki", "kind": "state", "rows": 4, "cols": 5, "depth": 12, "prec": "ozaki"},
        # the same on 24 qubits: passes over a state larger than L2
        {"name": "state_4x6_d16_c64", "kind": "state", "rows": 4, "cols": 6, "depth": 16, "prec": "c64"},
        # an uneven batch: 32 circuits of 12 to 21 qubits, 64 amplitudes each
        {"name": "svbatch_32", "kind": "svbatch", "count": 32, "qmin": 12, "qmax": 21, "dmin": 8, "dmax": 24},
        # small sliced amplitudes: many small tensors, launches count
        {"name": "amp_4x4_d10_sliced", "kind": "amp", "rows": 4, "cols": 4, "depth": 10, "prec": "ozaki", "slices": 6,
         "amps": 8},
        # 64 amplitudes of one 25-qubit circuit in one contraction (batched pairs)
        {"name": "multi_5x5_d14", "kind": "multi", "rows": 5, "cols": 5, "depth": 14, "prec": "ozaki", "amps": 64},
        # 30-qubit amplitudes in the TF32 split mode and on the plain FP64 path
        {"name": "amp_5x6_d14_3xtf32", "kind": "amp", "rows": 5, "cols": 6, "depth": 14, "prec": "3xtf32", "slices": 0,
         "amps": 8},
        {"name": "amp_5x6_d14_c128", "kind": "amp", "rows": 5, "cols": 6, "depth": 14, "prec": "c128", "slices": 0,
         "amps": 4},
        # the headline: amplitudes of the 6x6 depth-16 circuit, ten sliced
        # bonds, exact-accumulation tensor cores
        {"name": "amp_6x6_d16_sliced", "kind": "amp", "rows": 6, "cols": 6, "depth": 16, "prec": "ozaki", "slices": 10,
         "amps": 8},
        # one training batch of the cost model, forward and backward
        {"name": "mlp_grad_1024", "kind": "mlp", "n": 1024},
    ]


def draw(rng):
    kind = rng.choice(["gate", "qft", "state", "svbatch", "amp", "amp", "multi", "mlp"])
    if kind == "gate":
        return {"kind": kind, "n": rng.randint(5, 18), "k": rng.randint(1, 4), "prec": rng.choice(["c128", "c64"])}
    if kind == "qft":
        return {"kind": kind, "n": rng.randint(3, 12), "prec": rng.choice(["c128", "c64"])}
    if kind == "state":
        r, c = rng.choice([(3, 4), (2, 7), (3, 5), (4, 4), (3, 6), (2, 9), (4, 5), (3, 7), (2, 11), (4, 6)])
        prec = rng.choice(["c128", "ozaki", "c64"] if r * c <= 20 else ["ozaki", "c64"])
        return {"kind": kind, "rows": r, "cols": c, "depth": rng.randint(8, 20), "prec": prec}
    if kind == "svbatch":
        lo = rng.randint(8, 15)
        return {"kind": kind, "count": rng.randint(5, 48), "qmin": lo, "qmax": rng.randint(lo + 1, 21),
                "dmin": 8, "dmax": rng.randint(10, 24)}
    if kind == "mlp":
        return {"kind": kind, "n": int(round(2 ** rng.uniform(7, 14)))}
    if kind == "multi":
        r, c = rng.choice([(3, 5), (4, 4), (4, 5), (3, 7), (5, 5)])
        return {"kind": kind, "rows": r, "cols": c, "depth": rng.randint(8, 14),
                "prec": rng.choice(["ozaki", "c64", "c128"]), "amps": rng.randint(9, 64)}
    prec = rng.choice(["ozaki", "ozaki", "c64", "3xtf32", "c128"])
    shapes = [(4, 4), (4, 5), (5, 5), (5, 6)] + ([(6, 6)] if prec == "ozaki" else [])
    r, c = rng.choice(shapes)
    return {"kind": "amp", "rows": r, "cols": c, "depth": rng.randint(8, 16 if prec == "ozaki" else 14), "prec": prec,
            "slices": rng.choice([0, 0, rng.randint(2, 10)]), "amps": rng.randint(2, 4)}


# ---- inputs from the seed ----------------------------------------------------

_CZ = np.diag([1, 1, 1, -1]).astype(np.complex128)


def _haar(rng, d, count):
    """``count`` Haar-random d x d unitaries."""
    z = rng.standard_normal((count, d, d)) + 1j * rng.standard_normal((count, d, d))
    q, r = np.linalg.qr(z)
    ph = np.diagonal(r, axis1=1, axis2=2)
    return q * (ph / np.abs(ph))[:, None, :]


def _grid_gates(rows, cols, depth, rng):
    """Per layer a Haar gate on every qubit, then CZ on one of four alternating
    nearest-neighbour edge patterns (qubits 1-based, row-major)."""
    pats = [[], [], [], []]
    for r in range(rows):
        for c in range(cols):
            q = r * cols + c + 1
            if c + 1 < cols:
                pats[c % 2].append((q, q + 1))
            if r + 1 < rows:
                pats[2 + r % 2].append((q, q + cols))
    n = rows * cols
    us = _haar(rng, 2, depth * n)
    gates = []
    for layer in range(depth):
        gates += [(us[layer * n + q], [q + 1]) for q in range(n)]
        gates += [(_CZ, list(e)) for e in pats[layer % 4]]
    return gates


def _grid_shape(n):
    r = max(x for x in range(1, int(math.isqrt(n)) + 1) if n % x == 0)
    return r, n // r


def _bits(rng, n, count):
    return ["".join("1" if b else "0" for b in row) for row in rng.integers(0, 2, size=(count, n))]


def _qft_gates(n, rng):
    """The QFT of a random product state: one Haar gate per qubit, then H and
    controlled phases, then the swaps that reverse the qubit order."""
    h = np.array([[1, 1], [1, -1]], dtype=np.complex128) / math.sqrt(2)
    swap = np.array([[1, 0, 0, 0], [0, 0, 1, 0], [0, 1, 0, 0], [0, 0, 0, 1]], dtype=np.complex128)
    g = [(u, [q + 1]) for q, u in enumerate(_haar(rng, 2, n))]
    for i in range(1, n + 1):
        g.append((h, [i]))
        g += [(np.diag([1, 1, 1, np.exp(1j * math.pi / 2 ** (j - i + 1))]), [j + 1, i]) for j in range(i, n)]
    return g + [(swap, [i, n - i + 1]) for i in range(1, n // 2 + 1)]


def _inputs(case, seed):
    """Everything a case's values depend on, from the seed alone."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "gate":
        n, k = case["n"], case["k"]
        psi = rng.standard_normal(2 ** n) + 1j * rng.standard_normal(2 ** n)
        qs = [int(q) for q in rng.choice(n, size=k, replace=False)]  # positions among the state's modes
        return psi / np.linalg.norm(psi), _haar(rng, 2 ** k, 1)[0], qs
    if kind == "qft":
        return _qft_gates(case["n"], rng)
    if kind == "svbatch":
        shapes = np.random.default_rng(case["count"] * 1000 + case["qmin"])  # sizes are the case's, values the seed's
        out = []
        for _ in range(case["count"]):
            n, d = int(shapes.integers(case["qmin"], case["qmax"] + 1)), int(shapes.integers(case["dmin"], case["dmax"] + 1))
            out.append((n, _grid_gates(*_grid_shape(n), d, rng), _bits(rng, n, 64)))
        return out
    if kind == "mlp":
        # step features (log2 sizes over 16) and log-microsecond targets
        x = (rng.random((case["n"], 5)) * 24 / 16).astype(np.float32)
        return x, (x.sum(1) + 0.3 * rng.standard_normal(case["n"])).astype(np.float32)
    gates = _grid_gates(case["rows"], case["cols"], case["depth"], rng)
    n = case["rows"] * case["cols"]
    if kind == "amp":
        head = _bits(rng, n - 4, 1)[0]
        return gates, [head + format(int(v), "04b") for v in rng.choice(16, size=case["amps"], replace=False)]
    return gates, _bits(rng, n, case.get("amps", 1024))


# ---- prepare and run -----------------------------------------------------------

def _prec(pq, name):
    return {"c128": pq.PREC_C128, "c64": pq.PREC_C64, "3xtf32": pq.PREC_3XTF32, "ozaki": pq.PREC_OZAKI}[name]


def _dtype(prec):
    return np.complex128 if prec == "c128" else np.complex64  # the context's element type


def _shared_outputs(pq, net, bitstrings):
    """Output tensors for all bitstrings at once: qubit q's output is a 2 x B
    matrix, and the B axis is one index shared by all of them."""
    from pqgb300 import network as nw

    for i in range(net.number_qubits):
        index = net.output_qubits[net.qubit_ordering[i] - 1]
        data = np.zeros((2, len(bitstrings)), dtype=np.complex128)
        for b, s in enumerate(bitstrings):
            data[int(s[i]), b] = 1.0
        label = pq.new_label(net, "node")
        net.nodes[label] = pq.Node([index, "amps"], [2, len(bitstrings)], label)
        net.node_layers[label] = -1
        nw.save_tensor_data(net, label, data)
        net.edges[index].dst = label


def _grid_network(pq, case, backend, gates, bits):
    n = case["rows"] * case["cols"]
    net = pq.build_network(n, gates, decompose=True, backend=backend)
    pq.add_input(net, "0" * n)
    if case["kind"] == "amp":
        pq.add_output(net, bits[0])
        return net, [], None
    from pqgb300 import planning as pl

    _shared_outputs(pq, net, bits)
    nodes, ranks, flat, dims, label_of = pl._leaf_arrays(net, ["amps"])
    steps, _, _ = pl.sweep_steps(net, nodes, [label_of["amps"]], label_of, ranks, flat, dims)
    return net, ["amps"], steps


def prepare(case, seed):
    pq = _package()
    kind, inp = case["kind"], _inputs(case, seed)
    st = {"case": case, "pq": pq, "inp": inp}
    be = pq.GB300Backend(_prec(pq, case["prec"]) if "prec" in case else pq.PREC_C64)
    st["be"] = be
    if kind == "gate":
        psi, u, qs = inp
        n, k = case["n"], case["k"]
        st["psi"] = np.asfortranarray(psi.reshape((2,) * n, order="F").astype(_dtype(case["prec"])))
        st["u"] = np.asfortranarray(pq.operator_to_tensor(u))
        ia = [-(i + 1) for i in range(n)]
        for j, q in enumerate(qs):
            ia[q] = j + 1
        st["labels"] = ia, list(range(1, k + 1)) + [-(n + j + 1) for j in range(k)]
    elif kind == "state":
        from pqgb300 import circuits as ci

        gates, st["bits"] = inp
        n = case["rows"] * case["cols"]
        net = pq.build_network(n, ci.fuse_gates(gates, 4), backend=be)
        pq.add_input(net, "0" * n)
        steps = pq.planning.best_flop_plan(net, candidates=("wavefunction", "statevector"))[0]
        st["plan"] = pq.NetworkPlan(net, steps=steps)
        st["plan"].capture()
    elif kind == "svbatch":
        from pqgb300 import circuits as ci
        from pqgb300.svbatch import StateVectorBatch

        st["batch"] = StateVectorBatch(be, [(n, ci.fuse_gates(g, 4), b) for n, g, b in inp])
    elif kind in ("amp", "multi"):
        gates, bits = inp
        net, out, steps = _grid_network(pq, case, be, gates, bits)
        if steps is None:
            steps = pq.planning.best_flop_plan(net, out_edges=[], candidates=("sweep",), sweep_random=64)[0]
        plan = st["plan"] = pq.NetworkPlan(net, steps=steps, out_edges=out)
        # host copies of every leaf, as a program that rewrites its gates keeps them
        labels = [net.nodes[x].data_label for x in plan.leaves]
        host = {x: np.asfortranarray(be.load_tensor_data(x)).astype(_dtype(case["prec"])) for x in labels}
        st["leaves"] = be.prepare_tensors(list(host.items()))
        if kind == "amp":
            outs = [net.edges[net.output_qubits[q - 1]].dst for q in net.qubit_ordering]
            st["outputs"] = [host[net.nodes[x].data_label] for x in outs]
        if case.get("slices"):
            st["sliced"] = plan.choose_slices(max_sliced=case["slices"], log2_target=28.0)
            st["slices_per_launch"] = plan.auto_batch(st["sliced"])
        else:
            plan.capture()
    elif kind == "mlp":
        from pqgb300.costmodel import CostModel

        st["model"] = CostModel(be, hidden=128, layers=3, seed=seed)
    return st


def _contract(st):
    """The plan's result for the leaves' current host values."""
    case, be, plan = st["case"], st["be"], st["plan"]
    be.save_prepared(st["leaves"])
    if "sliced" in st:
        return np.asarray(plan.run_sliced(st["sliced"], batch=st["slices_per_launch"])).astype(_dtype(case["prec"])).reshape(-1)
    return np.asarray(be.load_tensor_data(plan.execute(), dtype=_dtype(case["prec"]))).reshape(-1)


def run(st):
    case, pq, be = st["case"], st["pq"], st["be"]
    kind = case["kind"]
    if kind == "gate":
        be.save_tensor_data("psi", st["psi"])
        be.save_tensor_data("u", st["u"])
        be.contract_tensors("psi", st["labels"][0], "u", st["labels"][1], "out")
        return be.load_tensor_data("out", dtype=_dtype(case["prec"]))
    if kind == "qft":
        net = pq.build_network(case["n"], st["inp"], backend=be)
        pq.add_input(net, "0" * case["n"])
        pq.full_wavefunction_contraction(net, "vector")
        return be.load_tensor_data("result", dtype=_dtype(case["prec"]))
    if kind == "state":
        return st["plan"].amplitudes(st["bits"], dtype=_dtype(case["prec"]))
    if kind == "svbatch":
        # the batch keeps its states in complex64 and returns them widened
        return np.concatenate(st["batch"].execute()).astype(np.complex64)
    if kind == "amp":
        amps = []
        for bits in st["inp"][1]:
            for vec, b in zip(st["outputs"], bits):
                vec[:] = (0, 1) if b == "1" else (1, 0)
            amps.append(_contract(st))
        return np.concatenate(amps)
    if kind == "multi":
        return _contract(st)
    grads, loss = st["model"].gradients(*st["inp"])
    return {"gradients": grads, "loss": float(np.float32(loss))}


# ---- 64-bit values ---------------------------------------------------------------

def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _statevector(n, gates):
    """The state from |0...0> (qubit 1 the lowest bit of the index)."""
    psi = torch.zeros(2 ** n, dtype=torch.complex128, device=_dev())
    psi[0] = 1
    for u, qs in gates:
        if len(qs) == 1:
            v = psi.view(2 ** (n - qs[0]), 2, -1)
            a, b = v[:, 0].clone(), v[:, 1].clone()
            v[:, 0] = complex(u[0, 0]) * a + complex(u[0, 1]) * b
            v[:, 1] = complex(u[1, 0]) * a + complex(u[1, 1]) * b
            continue
        lo, hi = min(qs), max(qs)
        v = psi.view(2 ** (n - hi), 2, 2 ** (hi - lo - 1), 2, 2 ** (lo - 1))
        if u is _CZ:
            v[:, 1, :, 1] *= -1
            continue
        # the first listed qubit is the low bit of u's index
        at = (lambda b: (b & 1, b >> 1)) if qs[0] == lo else (lambda b: (b >> 1, b & 1))
        old = [v[:, at(b)[1], :, at(b)[0]].clone() for b in range(4)]
        for o in range(4):
            v[:, at(o)[1], :, at(o)[0]] = sum(complex(u[o, i]) * old[i] for i in range(4))
    return psi


def _pick(psi, bits):
    idx = torch.tensor([sum(1 << i for i, ch in enumerate(b) if ch == "1") for b in bits], device=psi.device)
    return psi[idx].cpu().numpy()


def _sweep_amplitudes(rows, cols, gates, bitstrings):
    """Amplitudes of a grid circuit too large for a state vector, for bitstrings
    that differ in their last four bits only: CZ as a bond (the value of its
    first qubit), each qubit's timeline one tensor over its bonds, the qubits
    absorbed row by row into a boundary, the last four for every bitstring."""
    n = rows * cols
    tens = [(torch.tensor([1, 0], dtype=torch.complex128, device=_dev()), []) for _ in range(n)]
    eye = torch.eye(2, dtype=torch.complex128, device=_dev())
    sign = torch.tensor([[1, 1], [1, -1]], dtype=torch.complex128, device=_dev())
    for k, (u, qs) in enumerate(gates):
        if len(qs) == 1:
            t, legs = tens[qs[0] - 1]
            tens[qs[0] - 1] = (t @ torch.tensor(u, device=_dev()).T, legs)
        else:
            for q, m in zip(qs, (eye, sign)):  # legs stay in front, the qubit's value last
                t, legs = tens[q - 1]
                tens[q - 1] = ((t.unsqueeze(-2) * m).contiguous(), legs + [k])

    def absorb(bnd, q, bit):
        t, legs = tens[q][0][..., int(bit)], tens[q][1]
        common = [x for x in legs if x in bnd[1]]
        ia, ib = [bnd[1].index(x) for x in common], [legs.index(x) for x in common]
        return (torch.tensordot(bnd[0], t, dims=(ia, ib)),
                [x for x in bnd[1] if x not in common] + [x for x in legs if x not in common])

    first = (torch.ones((), dtype=torch.complex128, device=_dev()), [])
    for q in range(n - 4):
        first = absorb(first, q, bitstrings[0][q])
    out = []
    for bits in bitstrings:
        bnd = first
        for q in range(n - 4, n):
            bnd = absorb(bnd, q, bits[q])
        out.append(bnd[0].item())
    return np.array(out)


def exact(case, seed):
    kind, inp = case["kind"], _inputs(case, seed)
    if kind == "gate":
        psi, u, qs = inp
        n, k = case["n"], case["k"]
        if case["prec"] != "c128":
            psi = psi.astype(np.complex64).astype(np.complex128)  # what prepare() hands over
        t = np.transpose(u.reshape((2,) * (2 * k)), range(2 * k)[::-1])  # in bits, then out bits, lowest first
        return np.tensordot(psi.reshape((2,) * n, order="F"), t, axes=(qs, list(range(k))))
    if kind == "qft":
        return _statevector(case["n"], inp).cpu().numpy()
    if kind == "svbatch":
        return np.concatenate([_pick(_statevector(n, g), b) for n, g, b in inp])
    if kind == "mlp":
        return _mlp_exact(case, seed, *inp)
    gates, bits = inp
    n = case["rows"] * case["cols"]
    if n <= 26:
        return _pick(_statevector(n, gates), bits)
    return _sweep_amplitudes(case["rows"], case["cols"], gates, bits)


def _mlp_exact(case, seed, x, y):
    pq = _package()
    from pqgb300.costmodel import CostModel

    be = pq.GB300Backend(pq.PREC_C64)
    w = torch.tensor(CostModel(be, hidden=128, layers=3, seed=seed).params, dtype=torch.float64, device=_dev())
    w.requires_grad_(True)
    h, p = torch.tensor(x, dtype=torch.float64, device=_dev()), 0
    for i, (a, b) in enumerate([(5, 128), (128, 128), (128, 128), (128, 1)]):
        h = h @ w[p:p + a * b].view(a, b) + w[p + a * b:p + a * b + b]
        p += a * b + b
        h = torch.relu(h) if i < 3 else h
    loss = ((h[:, 0] - torch.tensor(y, dtype=torch.float64, device=_dev())) ** 2).mean()
    loss.backward()
    return {"gradients": w.grad.cpu().numpy(), "loss": loss.item()}


# ---- work a pass cannot do without -------------------------------------------------

_counted = {}


def _step_work(pq, case):
    """(bytes, flops) of a sweep plan: every pair's operands read and result
    written once in the element type, eight flops per complex multiply-add."""
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _counted:
        from pqgb300 import planning as pl

        gates, bits = _inputs(case, 0)
        be = pq.GB300Backend(pq.PREC_C128)
        net, out, steps = _grid_network(pq, case, be, gates, bits)
        nodes, ranks, flat, dims, label_of = pl._leaf_arrays(net, out)
        if steps is None:
            steps = pq.planning.best_flop_plan(net, out_edges=[], candidates=("sweep",), sweep_random=64)[0]
        labs, pos = [], 0
        for r in ranks:
            labs.append(set(flat[pos:pos + r]))
            pos += r
        left = {}
        for ls in labs:
            for x in ls:
                left[x] = left.get(x, 0) + 1
        for e in out:
            left[label_of[e]] += 1
        size = lambda ls: math.prod(dims[x] for x in ls)
        elems = macs = 0
        for a, b in zip(steps[0::2], steps[1::2]):
            for x in list(labs[a]) + list(labs[b]):
                left[x] -= 1
            c = {x for x in labs[a] | labs[b] if left[x] > 0}
            for x in c:
                left[x] += 1
            labs.append(c)
            elems += size(labs[a]) + size(labs[b]) + size(c)
            macs += size(labs[a] | labs[b])
        be.close()
        _counted[key] = elems, macs
    elems, macs = _counted[key]
    reps = case["amps"] if case["kind"] == "amp" else 1
    return {"bytes": reps * elems * (16 if case["prec"] == "c128" else 8), "flops": reps * 8 * macs}


def work(case):
    pq = _package()
    from pqgb300 import circuits as ci

    kind = case["kind"]
    if kind == "gate":
        elem = 16 if case["prec"] == "c128" else 8
        return {"bytes": 2 * elem * 2 ** case["n"] + 16 * 4 ** case["k"], "flops": 8 * 2 ** (case["n"] + case["k"])}
    if kind == "qft":
        n, gates = case["n"], _inputs(case, 0)
        return {"bytes": 16 * 2 ** n + sum(16 * u.size for u, _ in gates),
                "flops": sum(8 * 2 ** (n + len(qs)) for _, qs in gates)}
    if kind in ("state", "svbatch"):
        # a state vector is read and written once for every block of the circuit
        circuits = _inputs(case, 0) if kind == "svbatch" else [(case["rows"] * case["cols"], _inputs(case, 0)[0], None)]
        elem = 16 if case.get("prec") == "c128" else 8
        blocks = [(n, len(qs)) for n, g, _ in circuits for _, qs in ci.fuse_gates(g, 4)]
        return {"bytes": sum(2 * elem * 2 ** n for n, _ in blocks), "flops": sum(8 * 2 ** (n + k) for n, k in blocks)}
    if kind == "mlp":
        params = 5 * 128 + 2 * 128 * 128 + 128
        return {"bytes": 4 * (case["n"] * 6 + 2 * params), "flops": 6 * case["n"] * params}
    return _step_work(pq, case)
