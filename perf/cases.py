"""What the speed of this package is measured on: calls that its users make, over the sizes that they use.

A case names a seeded ring circuit (qubits, depth, T gates, open bits, parity slices: the circuits of
``workloads.py`` and others of the same family) and one public entry point with its options, or, for the
draw and the audit, the shape of the blocks.  ``prepare`` makes the inputs (prefixes, uniforms, blocks,
requests) from the seed; the engine of a circuit, with its plan and its tables, is kept from one state to
the next, as a program that samples one circuit keeps it.  ``exact`` contracts the graph state in plain torch
complex128 and draws with plain NumPy.
"""
import math

import numpy as np
import torch

from dcs245_classical_sampling_b200.audit import audit_vector_pair
from dcs245_classical_sampling_b200.circuits import build_ring_instance, ring_circuit
from dcs245_classical_sampling_b200.engine import HalfConditionalBlockGPU, InplaceConditionalBlockGPU
from dcs245_classical_sampling_b200.gather import ConditionalBlockGPU
from dcs245_classical_sampling_b200.plan import build_block_plan
from dcs245_classical_sampling_b200.sampling import draw_many, sample_checked
from dcs245_classical_sampling_b200.serve import CircuitRunner, Request, Server
from dcs245_classical_sampling_b200.workloads import choose_reference_slices, sweep_order


def _circuit(qubits, depth, t_gates, open_bits, slices, circuit_seed):
    return {"qubits": qubits, "depth": depth, "t_gates": t_gates, "open": open_bits, "slices": slices,
            "circuit_seed": circuit_seed}


RING16 = _circuit(16, 20, 24, 8, 1, 1016)
RING24 = _circuit(24, 24, 60, 10, 2, 1024)
RING32 = _circuit(32, 37, 79, 14, 0, 1032)
RING40 = _circuit(40, 45, 190, 16, 1, 1040)
RING48 = _circuit(48, 55, 177, 17, 0, 1048)
RING64 = _circuit(64, 73, 314, 20, 2, 1064)


def listed():
    return [
        # one amplitude block of the smallest workload: a first call, a notebook, a unit test of a user's own
        {"name": "block_16q", "what": "blocks", **RING16, "engine": "complex64", "batch": 1, "at_once": 0},
        # every prefix of that workload's sampling run in one call, its work items sharing launches
        {"name": "blocks_16q_256", "what": "blocks", **RING16, "engine": "complex64", "batch": 256, "at_once": 512},
        # the serving loop on a backlog of requests against two circuits
        {"name": "serve_24q_32q", "what": "serve", "requests": 12, "most": 16},
        # blocks of the 40-qubit workload with the engine's own choices
        {"name": "blocks_40q_8", "what": "blocks", **RING40, "engine": "complex64", "batch": 8, "at_once": 0},
        # the worker's loop on it as a sampling run drives it: generated kernels, host blocks, NumPy's CDF values
        {"name": "worker_40q_8", "what": "worker", **RING40, "batch": 8},
        # the recontraction in complex128 that an audit of a 48-qubit sample makes
        {"name": "block_48q_complex128", "what": "blocks", **RING48, "engine": "complex128", "batch": 1, "at_once": 0},
        # the half-storage engine, which users take where a table would not fit
        {"name": "block_48q_half", "what": "blocks", **RING48, "engine": "half", "batch": 1, "at_once": 0},
        # the second engine (gather form), in complex128 as the comparison with the first one wants it
        {"name": "gather_32q_complex128", "what": "blocks", **RING32, "engine": "gather128", "batch": 1, "at_once": 0},
        # the record's draw from the largest block, with the CDF values that NumPy's cumulative sum has
        {"name": "draw_2^20_numpy", "what": "draw", "bits": 20, "batch": 1, "numpy_cdf": True},
        # draws from a batch of middle-sized blocks (a user who wants indices only)
        {"name": "draw_2^14_x64", "what": "draw", "bits": 14, "batch": 64, "numpy_cdf": False},
        # the audit of a sample of the largest workload: the overlap of two full vectors
        {"name": "audit_2^20", "what": "audit", "bits": 20},
        # the headline workload: one block of 2^20 amplitudes of 64 qubits, tuned generated kernels
        {"name": "block_64q", "what": "blocks", **RING64, "engine": "fused", "batch": 1, "at_once": 0},
    ]


def _constrained(c):
    """Whether some parity of a circuit's closed bits is the same in every outcome, so that prefixes of the
    other parity have a zero block (which a sampling run never asks for): a product of their Z operators that
    stays one Pauli operator through the gates, back to one of Z operators alone on the first state."""
    group = [(0, 1 << q) for q in range(c["qubits"] - c["open"])]  # (x mask, z mask)

    def commuting(q):  # the part of the group without X on q
        pivot = next((g for g in group if g[0] >> q & 1), None)
        return [(x ^ pivot[0], z ^ pivot[1]) if x >> q & 1 else (x, z) for x, z in group
                if (x, z) != pivot] if pivot else group

    for name, qs in reversed(ring_circuit(c["qubits"], c["depth"], c["t_gates"], c["circuit_seed"])):
        a, b = qs[0], qs[-1]
        if name == "t":
            group = commuting(a)
        elif name == "h":
            group = [(x ^ (d := ((x ^ z) >> a & 1) << a), z ^ d) for x, z in group]
        elif name in ("s", "sdg"):
            group = [(x, z ^ ((x >> a & 1) << a)) for x, z in group]
        elif name == "cz":
            group = [(x, z ^ ((x >> a & 1) << b) ^ ((x >> b & 1) << a)) for x, z in group]
        else:  # cx: control a, target b
            group = [(x ^ ((x >> a & 1) << b), z ^ ((z >> b & 1) << a)) for x, z in group]
    for q in range(c["qubits"]):
        group = commuting(q)
    return bool(group)


def _draw_circuit(rng, least, most):
    while True:
        n = rng.randint(least, most)
        t = round(n * rng.uniform(1.5, 4.75 if n <= 40 else 3.7))
        k = max(3, round(n * rng.uniform(0.25, 0.5 if n < 30 else 0.4)))
        c = _circuit(n, round(n * rng.uniform(1.0, 1.2)) + 2, t, k, rng.randint(0, 2), rng.randrange(1, 10 ** 6))
        if _constrained(c):
            continue
        if n <= 24:  # T gates that combine can leave such a parity too, mostly in small circuits
            w, xs = _workload(c), _prefixes({**c, "batch": 4}, 0)
            if min(float(torch.linalg.norm(_block64(w, x, "cpu"))) for x in xs) < 1e-6:
                continue
        return c


def draw(rng):
    what = rng.choice(["blocks"] * 6 + ["worker", "serve", "draw", "draw", "draw", "audit"])
    if what == "blocks":
        engine = rng.choice(["complex64", "complex64", "complex128", "half", "gather64", "gather128", "fused128"])
        c = _draw_circuit(rng, 36 if engine == "fused128" else 12, 40 if engine.startswith("gather") else 48)
        batch, at_once = 1, 0
        if engine in ("complex64", "complex128"):
            batch = max(1, round(2 ** rng.uniform(0, min(8, (46 - c["qubits"]) / 2.5))))
            at_once = rng.choice([0, batch << c["slices"]])
        return {"what": "blocks", **c, "engine": engine, "batch": batch, "at_once": at_once}
    if what == "worker":
        return {"what": "worker", **_draw_circuit(rng, 32, 44), "batch": rng.randint(1, 12)}
    if what == "serve":
        return {"what": "serve", "requests": rng.randint(1, 20), "most": rng.randint(1, 32)}
    if what == "draw":
        k = rng.randint(1, 20)
        return {"what": "draw", "bits": k, "batch": max(1, round(2 ** rng.uniform(0, min(9, 21 - k)))),
                "numpy_cdf": rng.random() < 0.5}
    return {"what": "audit", "bits": rng.randint(4, 22)}


# ---------------------------------------------------------------- what a program has in hand

_last = {}  # the workload, plan and engine of the last case: one circuit's tables at a time


def _kept(key, make):
    if key not in _last:
        if len(_last) > 3 or any(k[0] == "engine" for k in _last):
            _last.clear()
        _last[key] = make()
    return _last[key]


def _workload(c):
    """The engine's arguments for a circuit."""
    def make():
        inst = build_ring_instance(c["qubits"], c["depth"], c["t_gates"], c["circuit_seed"])
        n = c["qubits"]
        opened = list(range(n - c["open"], n))
        order = sweep_order(inst, opened)
        ops = choose_reference_slices(inst["graph"], n, order, c["slices"], opened)
        return {"graph": inst["graph"], "unitaries": inst["unitaries"], "n": n, "order": order,
                "parity_operations": [list(op) for op in ops], "open_vertices": opened}
    return _kept(("workload",) + tuple(c[k] for k in sorted(RING16)), make)


def _args(w):
    return w["graph"], w["unitaries"], w["n"], w["order"], w["parity_operations"], w["open_vertices"]


def _engine(case):
    def make():
        args, kind = _args(w), case.get("engine", "fused")
        if kind == "half":
            engine = HalfConditionalBlockGPU(*args)
            engine.alloc()
        elif kind in ("gather64", "gather128"):
            engine = ConditionalBlockGPU(*args)
            engine.alloc(np.complex64 if kind == "gather64" else np.complex128)
        else:
            engine = InplaceConditionalBlockGPU(*args)
            dtype = np.complex64 if kind in ("complex64", "fused") else np.complex128
            mode = "fused" if kind in ("fused", "fused128") else None
            engine.alloc(dtype, mode=mode, items=case.get("at_once") or None)
            if case["what"] == "worker":  # the generated kernels, as the benchmark runs this workload
                engine.set_fused_config(variant=12, low=3, grouping="bytes", jit=True)
        return engine
    w = _workload(case)
    return _kept(("engine",) + tuple(str(case.get(k)) for k in ("what", "engine", "at_once", *sorted(RING16))), make)


def _runners():
    def make():
        got = {}
        for i, c in enumerate((RING24, RING32)):
            got["q%d" % c["qubits"]] = CircuitRunner("q%d" % c["qubits"], _workload(c), 77 + i, 32)
        return got
    return _kept(("engine", "serve"), make)


def _prefixes(case, seed):
    rng = np.random.default_rng([seed, 1])
    return [rng.integers(0, 2, case["qubits"]).astype(np.uint8) for _ in range(case["batch"])]


def _vectors(bits, batch, seed):
    """Blocks as random circuits give them: Gaussian amplitudes, squared norms near 1."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    v = torch.randn((batch, 1 << bits, 2), generator=g, dtype=torch.float64, device="cuda")
    return torch.view_as_complex(v) * math.sqrt(0.5 / (1 << bits))


def prepare(case, seed):
    what = case["what"]
    if what in ("blocks", "worker"):
        state = {"xs": _prefixes(case, seed), "engine": _engine(case)}
        if what == "worker":
            state["us"] = np.random.default_rng([seed, 2]).random(case["batch"]).tolist()
    elif what == "serve":
        rng = np.random.default_rng([seed, 3])
        first = int(rng.integers(0, 1 << 24)) * 64
        state = {"runners": _runners(), "asked": [(first + i, "q24" if rng.random() < 0.5 else "q32",
                                                   1 + (5 * i + 2) % case["most"])
                                                  for i in range(case["requests"])]}
    elif what == "draw":
        state = {"blocks": _vectors(case["bits"], case["batch"], seed),
                 "us": np.random.default_rng([seed, 4]).random(case["batch"])}
    else:
        a, b = _vectors(case["bits"], 2, seed)
        state = {"ref": a.clone(), "ap": a + 1e-6 * b}
    return {"case": case, **state}


# ---------------------------------------------------------------- the calls

def _numbers(record):
    return {k: v for k, v in record.items() if isinstance(v, (bool, int, float))}


def run(state):
    case = state["case"]
    what = case["what"]
    if what == "blocks":
        engine, xs = state["engine"], state["xs"]
        if len(xs) == 1:
            return engine.block(xs[0])[0]
        return engine.blocks(xs)
    if what == "worker":
        records, blocks = sample_checked(state["engine"], state["xs"], state["us"], exact_cdf=True,
                                         keep_host_blocks=True)
        rows = [_numbers(r) for r in records]
        return {"blocks": np.stack(blocks), "records": {k: np.array([r[k] for r in rows]) for k in rows[0]}}
    if what == "serve":
        done = Server(state["runners"]).run([Request(rid, c, m, 0.0) for rid, c, m in state["asked"]], realtime=False)
        rows = [r.records[i] for r in sorted(done, key=lambda r: r.rid) for i in range(r.nsamples)]
        records = np.stack([row[0] for row in rows])
        return {"prefixes": np.array([row[1] for row in rows]), **{k: records[k] for k in records.dtype.names}}
    if what == "draw":
        records = draw_many(state["blocks"], state["us"], exact_cdf=case["numpy_cdf"])
        return {k: records[k] for k in records.dtype.names}
    return _numbers(audit_vector_pair(state["ref"], state["ap"], 0))


# ---------------------------------------------------------------- what a pass cannot do without

def _block_work(c, batch):
    w = _workload(c)
    p = _kept(("plan",) + tuple(c[k] for k in sorted(RING16)), lambda: build_block_plan(*_args(w)))
    flops = 0.0
    for st in p.steps:  # an entry that a step writes: two complex products and a sum, or one product
        flops += (14.0 if st.free else 6.0) * (1 << len(st.active_out))
    k = len(p.open_full)
    out = 16 << k
    tail = (4 + 16) * k * (1 << k)
    return {"bytes": batch * (out + c["qubits"]), "flops": batch * (flops * (1 << len(p.slices)) + tail)}


def work(case):
    what = case["what"]
    if what in ("blocks", "worker"):
        return _block_work(case, case["batch"])
    if what == "serve":
        samples = sum(1 + (5 * i + 2) % case["most"] for i in range(case["requests"]))
        a, b = _block_work(RING24, 1), _block_work(RING32, 1)
        return {"bytes": samples * 104, "flops": samples * (a["flops"] + b["flops"]) / 2}
    n = 1 << case["bits"]
    if what == "draw":
        return {"bytes": case["batch"] * (16 * n + 112), "flops": case["batch"] * 10.0 * n}
    return {"bytes": 32 * n, "flops": 14.0 * n}


# ---------------------------------------------------------------- the same in 64 bits

def _parity(mask, size, device):
    """(size,) +-1 in float64: the sign (-1)^popcount(i & mask)."""
    sign = torch.ones(1, dtype=torch.float64, device=device)
    b = 0
    while (1 << b) < size:
        sign = torch.cat([sign, -sign if mask >> b & 1 else sign])
        b += 1
    return sign


def _dependency(vectors):
    """A set of positions whose vectors (bit masks) add up to zero over GF(2), or None."""
    rows = []
    for i, v in enumerate(vectors):
        comb = 1 << i
        for r, c in rows:
            if v ^ r < v:
                v, comb = v ^ r, comb ^ c
        if not v:
            return comb
        rows.append((v, comb))
        rows.sort(reverse=True)
    return None


def _block64(w, x, device):
    """The conditional block of one prefix by elimination of the graph's vertices in order: the sum over the
    closed vertices' values, as a function of the neighbour parities s that they leave on the later vertices.
    s is kept in coordinates of a GF(2) basis (entry c of `table`: s = XOR of basis[i] over the bits i of c)."""
    A, U, n, order, opened = np.asarray(w["graph"]), w["unitaries"], w["n"], w["order"], w["open_vertices"]
    N = len(A)
    bra = np.array([1.0, np.exp(0.25j * math.pi)])
    table, basis = torch.ones(1, dtype=torch.complex128, device=device), []
    later = [v for v in order if v not in set(opened)]
    bit = {v: 1 << i for i, v in enumerate(order)}
    left = sum(bit.values())
    for v in later:
        u = np.asarray(U[v], np.complex128)
        f = u[int(x[v])] if v < n else bra @ u
        sees = sum(1 << i for i, b in enumerate(basis) if b & bit[v])
        left &= ~bit[v]
        near = sum(bit[int(q)] for q in np.flatnonzero(A[v])) & left
        table = torch.cat([table * complex(f[0]), table * _parity(sees, table.numel(), device) * complex(f[1])])
        basis = [b & left for b in basis] + [near]
        while (comb := _dependency(basis)) is not None:
            j = comb.bit_length() - 1
            other = torch.arange(table.numel(), device=device) ^ comb
            table = (table + table[other]).view(-1, 2, 1 << j)[:, 0].reshape(-1)
            del basis[j], other
    k = len(opened)
    at = torch.zeros(1, dtype=torch.int64, device=device)
    for b in basis:
        m = sum(1 << j for j, q in enumerate(opened) if b & bit[q])
        at = torch.cat([at, at ^ m])
    block = torch.zeros(1 << k, dtype=torch.complex128, device=device)
    block[at] = table
    for j in range(k):
        v = block.view(-1, 2, 1 << j)
        block = torch.stack([v[:, 0] + v[:, 1], v[:, 0] - v[:, 1]], 1).reshape(-1)
    y = torch.arange(1 << k, device=device)
    odd = torch.zeros_like(y)
    for a in range(k):
        for b in range(a):
            if A[opened[a], opened[b]]:
                odd ^= (y >> a) & (y >> b) & 1
    block = torch.where(odd.bool(), -block, block)
    for j, q in enumerate(opened):
        u = np.asarray(U[q], np.complex128)
        v = block.view(-1, 2, 1 << j)
        block = torch.stack([v[:, 0] * complex(u[0, 0]) + v[:, 1] * complex(u[0, 1]),
                             v[:, 0] * complex(u[1, 0]) + v[:, 1] * complex(u[1, 1])], 1).reshape(-1)
    return block * 2.0 ** (-(N - n + k) / 2)


def _phase(w):
    """The global phase that the parity slices give a block: a local complementation at v is
    exp(-i pi/4 X) on v and exp(i pi/4 Z) on its d neighbours, which is e^(i pi (d - 1) / 4) times the
    complemented graph state."""
    A, eighths = np.array(w["graph"], np.uint8), 0

    def complement(v):
        near = np.flatnonzero(A[v])
        A[np.ix_(near, near)] ^= 1
        A[near, near] = 0
        return len(near) - 1

    for kind, v, u in w["parity_operations"]:
        for q in {"X": (u, v, u), "Y": (v,), "Z": ()}[kind]:
            eighths += complement(q)
    return complex(np.exp(0.25j * math.pi * (eighths % 8)))


def _draw64(v, u, numpy_cdf):
    weights = v.real * v.real + v.imag * v.imag
    sums = np.cumsum(weights)
    cdf = sums / sums[-1]
    cdf[-1] = 1.0
    i = int(np.searchsorted(cdf, u, side="right"))
    total = math.fsum(weights)
    before = math.fsum(weights[:i])
    low, high = before / total, math.fsum([before, weights[i]]) / total
    last = i == len(weights) - 1
    p = weights / total
    return {"index": i, "status": 0, "total_cdf": float(sums[-1]) if numpy_cdf else total, "total_exact": total,
            "selected_weight": float(weights[i]),
            "cdf_lower": (float(cdf[i - 1]) if i else 0.0) if numpy_cdf else low,
            "cdf_upper": float(cdf[i]) if numpy_cdf else 1.0 if last else high,
            "cdf_lower_exact": low, "cdf_upper_exact": high, "uniform": u, "weight_l2": math.fsum(p * p)}


def exact(case, seed):
    what = case["what"]
    if what in ("blocks", "worker"):
        w = _workload(case)
        if build_block_plan(*_args(w)).maxslots + case["slices"] > 27:  # too large, too long
            return None
        blocks = torch.stack([_block64(w, x, "cuda") for x in _prefixes(case, seed)]) * _phase(w)
        if what == "worker":
            return {"blocks": blocks.cpu().numpy(), "records": None}
        return blocks[0] if case["batch"] == 1 else blocks
    if what == "draw":
        vectors = _vectors(case["bits"], case["batch"], seed).cpu().numpy()
        us = np.random.default_rng([seed, 4]).random(case["batch"])
        rows = [_draw64(v, float(u), case["numpy_cdf"]) for v, u in zip(vectors, us)]
        return {k: np.array([r[k] for r in rows]) for k in rows[0]}
    if what == "audit":
        a, b = (t.cpu().numpy().astype(np.clongdouble) for t in _vectors(case["bits"], 2, seed))
        ap = (torch.from_numpy(a.astype(np.complex128)) + 1e-6 * torch.from_numpy(b.astype(np.complex128))).numpy()
        ap = ap.astype(np.clongdouble)
        rr, aa = float((np.abs(a) ** 2).sum()), float((np.abs(ap) ** 2).sum())
        score = float(abs((a.conj() * ap).sum())) / math.sqrt(aa)
        return {"reference_scaled_mass": rr, "approximate_input_mass": aa, "uncapped_overlap_witness": score}
    return None
