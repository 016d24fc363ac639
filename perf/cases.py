"""Work that users of this framework have it do, as cases that can be timed
and checked: whole amplitude evaluations (the drop-in ``simulate`` call, a
batch of output strings, an open output region) and the tensor operations
they consist of (products in each complex64 precision, reorders), each
through its public entry point.

  listed()            the cases that stand for the path
  draw(rng)           one more case of the same ranges
  prepare(case, seed) what a program holds before the call
  run(state)          one pass through the public entry points
  work(case)          bytes and flop a pass cannot do without
  exact(case, seed)   what run() returns, in 64 bits
"""
from __future__ import annotations

import math

import numpy as np
import torch

from qflex_gb300 import Context, rqc, simulate
from qflex_gb300._lib import PRECISIONS

LIMIT = float(1 << 40)  # memory limit of the evaluations, in the reference's formula


def listed():
    return [
        # One amplitude of a 20-qubit circuit through the drop-in call of a Cirq simulator: latency.
        {"name": "simulate_4x5", "kind": "simulate", "rows": 4, "cols": 5, "depth": 16},
        # The 36-qubit workload with its cut summed in full, default precision, a batch of strings.
        {"name": "amplitudes_6x6_fp32", "kind": "amplitudes", "rows": 6, "cols": 6, "depth": 24, "strings": 16,
         "cut_values": 0, "precision": "fp32"},
        # The headline workload: 49 qubits, depth (1+32+1), 16 slices, 8 strings on the tensor cores.
        {"name": "amplitudes_7x7_fp16x3", "kind": "amplitudes", "rows": 7, "cols": 7, "depth": 32, "strings": 8,
         "cut_values": 4, "precision": "fp16x3"},
        # 53-qubit fSim circuit, one prefix whose open region gives 64 amplitudes: large, batch of one.
        {"name": "region_6x9_fsim_fp16x3", "kind": "region", "cycles": 8, "prefixes": 1, "precision": "fp16x3"},
        # The merge of two 24-index patches: the largest product of the 7x7 contraction.
        {"name": "multiply_4096_fp16x3", "kind": "multiply", "m": 4096, "n": 4096, "k": 4096, "batch": 1,
         "precision": "fp16x3"},
        # The product of a 7x7 expansion step, four strings at a time.
        {"name": "multiply_tall_fp16x3", "kind": "multiply", "m": 65536, "n": 256, "k": 256, "batch": 4,
         "precision": "fp16x3"},
        # A merge in each of the other split precisions.
        {"name": "multiply_2048_tf32x3", "kind": "multiply", "m": 2048, "n": 2048, "k": 2048, "batch": 1,
         "precision": "tf32x3"},
        {"name": "multiply_wide_bf16x3", "kind": "multiply", "m": 4096, "n": 1024, "k": 2048, "batch": 1,
         "precision": "bf16x3"},
        # Sizes that fill no tile, as the tensor-level call takes them.
        {"name": "multiply_ragged_fp16x3", "kind": "multiply", "m": 3001, "n": 690, "k": 1100, "batch": 1,
         "precision": "fp16x3"},
        # An expansion by a tensor of small bonds: a long, narrow product on the default precision.
        {"name": "multiply_narrow_fp32", "kind": "multiply", "m": 1048576, "n": 16, "k": 16, "batch": 1,
         "precision": "fp32"},
        # The reorder before an expansion: six bonds of dimension 16.
        {"name": "permute_2p24", "kind": "permute", "dims": "16,16,16,16,16,16", "order": "0,2,4,5,1,3", "batch": 1},
        # Tensor::reorder of dimensions that are not powers of two.
        {"name": "reorder_odd_dims", "kind": "permute", "dims": "12,15,7,24,10,27", "order": "3,0,5,2,1,4",
         "batch": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_multiply(rng):
    precision = rng.choice(["fp16x3", "fp16x3", "tf32x3", "bf16x3", "fp32"])
    while True:
        m, n, k = _log(rng, 16, 1 << 20), _log(rng, 1, 4096), _log(rng, 2, 4096)
        if rng.random() < 0.6:  # the contraction's own sizes: powers of two
            m, n, k = (1 << int(round(math.log2(x))) for x in (m, n, k))
        batch = rng.choice([1, 1, 1, 2, 4, 7])
        elems, flop = (m * k + k * n + m * n) * batch, 8.0 * m * n * k * batch
        if elems <= 1 << 28 and flop <= 2e12 and k * n <= 1 << 24:
            return {"kind": "multiply", "m": m, "n": n, "k": k, "batch": batch, "precision": precision}


def _draw_permute(rng):
    two = rng.random() < 0.6
    size, dims, want = 1, [], 1 << rng.randint(8, 26)
    while size < want:
        d = 1 << rng.randint(1, 4) if two else rng.randint(2, 30)
        dims.append(d)
        size *= d
    order = list(range(len(dims)))
    rng.shuffle(order)
    batch = rng.choice([1, 1, 2, 5]) if size <= 1 << 22 else 1
    return {"kind": "permute", "dims": ",".join(map(str, dims)), "order": ",".join(map(str, order)), "batch": batch}


def draw(rng):
    kind = rng.choice(["simulate", "amplitudes", "amplitudes", "region", "multiply", "multiply", "multiply",
                       "permute", "permute"])
    if kind == "simulate":
        return {"kind": kind, "rows": rng.randint(3, 5), "cols": rng.randint(3, 5), "depth": rng.randint(8, 20)}
    if kind == "amplitudes":
        if rng.random() < 0.5:
            return {"kind": kind, "rows": 7, "cols": 7, "depth": 32, "strings": rng.randint(1, 4),
                    "cut_values": rng.randint(1, 2), "precision": rng.choice(["fp16x3", "tf32x3", "bf16x3"])}
        return {"kind": kind, "rows": 6, "cols": 6, "depth": rng.randint(16, 24), "strings": _log(rng, 1, 32),
                "cut_values": 0, "precision": rng.choice(["fp32", "fp16x3", "tf32x3", "bf16x3"])}
    if kind == "region":
        return {"kind": kind, "cycles": rng.randint(4, 8), "prefixes": rng.randint(1, 2), "precision": "fp16x3"}
    return _draw_multiply(rng) if kind == "multiply" else _draw_permute(rng)


# ---- inputs ---------------------------------------------------------------------

_contexts = {}


def _context(precision):
    """The process's engine context of a precision, on a stream of its own,
    as a serving program keeps one."""
    if precision not in _contexts:
        _contexts[precision] = Context(0, PRECISIONS[precision])
    return _contexts[precision]


def _network(case, seed):
    """(circuit, ordering, grid, initial, finals): a circuit of the case's
    size and output strings made from the seed."""
    if case["kind"] == "region":
        circuit, ordering, grid, initial, finals = rqc.workload_c4(cycles=case["cycles"], n_prefixes=1)
        open_at = [c == "x" for c in finals[0]]
        finals = ["".join("x" if x else b for x, b in zip(open_at, s))
                  for s in rqc.random_bitstrings(len(open_at), case["prefixes"], seed + 2)]
        return circuit, ordering, grid, initial, finals
    rows, cols = case["rows"], case["cols"]
    circuit, grid = rqc.random_circuit(rows, cols, case["depth"], seed=0), rqc.grid_text(rows, cols)
    values = tuple(range(case.get("cut_values", 0))) or None
    if case["kind"] == "simulate":
        ordering = rqc.row_sweep_ordering(rows, cols)
    elif rows == 6:
        ordering = rqc.ordering_6x6(values)
    elif values == (0, 1, 2, 3):
        ordering = rqc.ordering_7x7_learned()
    else:
        ordering = rqc.ordering_7x7(values, values)
    initial = rqc.random_bitstrings(rows * cols, 1, 1)[0]
    return circuit, ordering, grid, initial, rqc.random_bitstrings(rows * cols, case.get("strings", 1), seed + 2)


def _ints(text):
    return [int(x) for x in text.split(",")]


def _randn(shape, seed):
    """Tensor entries of a contraction in progress: complex Gaussian, small."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, dtype=torch.complex64, device="cuda", generator=g) * 2.0 ** -6


def _operands(case, seed):
    """One buffer per string holding A, B and C of its product, as in the
    engine's arena: entry b at b * stride. C starts as zeros."""
    m, n, k, batch = (case[x] for x in ("m", "n", "k", "batch"))
    stride = m * k + k * n + m * n
    buf = _randn((batch, stride), seed)
    buf[:, m * k + k * n:] = 0
    return buf


def prepare(case, seed):
    state = dict(case)
    kind = case["kind"]
    if kind == "simulate":
        circuit, ordering, grid, initial, finals = _network(case, seed)
        state["options"] = {"circuit": circuit.splitlines(), "ordering": ordering.splitlines(),
                            "grid": grid.splitlines(), "initial_state": initial, "final_state": finals[0]}
    elif kind in ("amplitudes", "region"):
        state["network"] = _network(case, seed)
        state["ctx"] = _context(case["precision"])
    elif kind == "multiply":
        state["buf"] = _operands(case, seed)
        state["ctx"] = _context(case["precision"])
    else:
        state["shape"], state["perm"] = _ints(case["dims"]), _ints(case["order"])
        state["src"] = _randn((case["batch"], math.prod(state["shape"])), seed)
        state["dst"] = torch.empty_like(state["src"])
        state["ctx"] = _context("fp32")
    return state


def run(state):
    kind = state["kind"]
    if kind == "simulate":
        out = simulate(state["options"])
    elif kind in ("amplitudes", "region"):
        circuit, ordering, grid, initial, finals = state["network"]
        out = state["ctx"].evaluate_many(circuit, ordering, grid, initial, finals, LIMIT)
    elif kind == "multiply":
        m, n, k, buf = state["m"], state["n"], state["k"], state["buf"]
        at, stride = buf.data_ptr(), buf.shape[1]
        state["ctx"].multiply(at, at + 8 * m * k, at + 8 * (m * k + k * n), m, n, k, state["batch"], stride)
        return buf[:, m * k + k * n:].view(state["batch"], m, n)
    else:
        src, dst = state["src"], state["dst"]
        state["ctx"].permute(src.data_ptr(), dst.data_ptr(), state["shape"], state["perm"], state["batch"],
                             src.shape[1])
        return dst
    # Sums of complex64 tensors: complex64 holds what they carry.
    return np.array([a for _, a in out], dtype=np.complex64)


def work(case):
    kind = case["kind"]
    if kind == "multiply":
        m, n, k, batch = (case[x] for x in ("m", "n", "k", "batch"))
        return {"bytes": 8.0 * (m * k + k * n + m * n) * batch, "flops": 8.0 * m * n * k * batch}
    if kind == "permute":
        return {"bytes": 16.0 * math.prod(_ints(case["dims"])) * case["batch"], "flops": 0.0}
    # The products of the ordering, 8 m n k each, for every string; strings in, amplitudes out.
    circuit, ordering, grid, initial, finals = _network(case, 0)
    plan = Context(-1, PRECISIONS["fp16x3"])
    amplitudes = len(plan.evaluate(circuit, ordering, grid, initial, finals[0], LIMIT))
    flop = plan.stats()["gemm_flop"]
    plan.close()
    return {"bytes": len(finals) * (len(initial) + 16.0 * amplitudes), "flops": flop * len(finals)}


# ---- results in 64 bits ------------------------------------------------------------

_HALF, _R = 0.5 + 0.5j, math.sqrt(0.5)
_GATES = {  # [input][output]
    "h": [[_R, _R], [_R, -_R]],
    "t": [[1, 0], [0, complex(_R, _R)]],
    "x_1_2": [[_HALF, _HALF.conjugate()], [_HALF.conjugate(), _HALF]],
    "y_1_2": [[_HALF, _HALF], [-_HALF, _HALF]],
}


def _amplitude(circuit, rows, cols, initial, final):
    """<final| circuit |initial> of an h, t, x_1_2, y_1_2, cz circuit on a
    grid: every cz is sum_v P_v x Z^v, every qubit's column of gates a tensor
    over the digits v of its bonds, contracted site by site in row order."""
    bonds, vec = {}, {}
    for q in range(rows * cols):
        vec[q] = torch.zeros(2, dtype=torch.complex128, device="cuda")
        vec[q][int(initial[q])] = 1
    for line in circuit.splitlines()[1:]:
        word = line.split()
        qubits = [int(x) for x in word[2:]]
        if word[1] != "cz":
            gate = torch.tensor(_GATES[word[1]], dtype=torch.complex128, device="cuda")
            vec[qubits[0]] = torch.tensordot(vec[qubits[0]], gate, dims=([0], [0])).movedim(-1, 0)
            continue
        label = (min(qubits), max(qubits), line)
        for q, project in zip(qubits, (True, False)):
            bonds.setdefault(q, []).append(label)
            v = vec[q]
            other = torch.stack([v[0], v[1] if project else -v[1]])
            zero = torch.zeros_like(v[0])
            # digit 0: P_0 or the identity; digit 1: P_1 or Z
            first = torch.stack([v[0], zero]) if project else v
            second = torch.stack([zero, v[1]]) if project else other
            vec[q] = torch.stack([first, second], dim=-1)
    state, legs = torch.ones((), dtype=torch.complex128, device="cuda"), []
    for q in range(rows * cols):
        site, mine = vec[q][int(final[q])], bonds.get(q, [])
        shared = [b for b in mine if b in legs]
        free = [b for b in mine if b not in legs]
        kept = [b for b in legs if b not in shared]
        left = state.permute([legs.index(b) for b in kept + shared]).reshape(-1, 2 ** len(shared))
        right = site.permute([mine.index(b) for b in shared + free]).reshape(2 ** len(shared), -1)
        legs = kept + free
        state = (left @ right).reshape([2] * len(legs))
    return complex(state)


def exact(case, seed):
    kind = case["kind"]
    if kind == "multiply":
        m, n, k = case["m"], case["n"], case["k"]
        buf = _operands(case, seed)
        return torch.stack([row[:m * k].view(m, k).to(torch.complex128) @
                            row[m * k:m * k + k * n].view(k, n).to(torch.complex128) for row in buf])
    if kind == "permute":
        dims, order = _ints(case["dims"]), _ints(case["order"])
        src = _randn((case["batch"], math.prod(dims)), seed).view([case["batch"]] + dims)
        return src.permute([0] + [1 + i for i in order]).reshape(case["batch"], -1).to(torch.complex128)
    if kind == "region" or case["rows"] == 7:
        return None  # minutes of 64-bit products
    circuit, _, _, initial, finals = _network(case, seed)
    return np.array([_amplitude(circuit, case["rows"], case["cols"], initial, f) for f in finals])
