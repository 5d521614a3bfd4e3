"""The framework's performance cases: the work its users have it do, through its public calls.

Every case is a dict of plain values.  `kind` picks the path:

  circuit   random gates (uniform over the 18 calls) on one statevector or density matrix,
            then `mean` of a diagonal observable
  channels  one-qubit Kraus channels on every qubit of a density matrix, then `mean`
  noisy     exact energies of a noisy variational circuit on a tiled density matrix
  qaoa      a batch of diagonal-cost circuits evaluated from host angles to host means
  gradients forward and backward pass of the surrogate network on one minibatch
  forward   screening of candidates by the surrogate network

`listed` are the cases of the benchmark configurations, `draw` gives others of the same ranges,
`prepare` makes what a program holds before the call, `run` is one pass, `work` what the pass
cannot do without, and `exact` the result in 64 bits by plain torch and numpy.
"""
import ctypes
import math

import numpy as np
import torch

import orkan_b200
from orkan_b200 import surrogate
from orkan_b200.batch import QaoaBatch

PLAIN_1Q = ("x", "y", "z", "h", "s", "sdg", "t", "tdg", "hy")
ANGLE_1Q = ("rx", "ry", "rz", "p")
PAIRS = ("cx", "cy", "cz", "swap")
GATES = PLAIN_1Q + ANGLE_1Q + PAIRS + ("ccx",)
TILE = 32                                   # tile side of the library loaded here
NOISE = 0.01                                # depolarizing strength of the noisy circuits


def listed():
    return [
        # the parity configuration's 200-gate circuit on 12 qubits: a program that runs many
        # small circuits, bound by calls and launches
        {"name": "circuit_pure_12q", "kind": "circuit", "layout": "pure", "n": 12, "gates": 200},
        # an ordinary statevector simulation, an odd qubit count and a state within L2's reach
        {"name": "circuit_pure_21q", "kind": "circuit", "layout": "pure", "n": 21, "gates": 120},
        # the largest statevector of the benchmark, 16 GiB, with its 200-gate circuit
        {"name": "circuit_pure_30q", "kind": "circuit", "layout": "pure", "n": 30, "gates": 200},
        # the parity configuration's circuit on a small tiled density matrix
        {"name": "circuit_tiled_8q", "kind": "circuit", "layout": "tiled", "n": 8, "gates": 200},
        # the gate calls on the 14-qubit density matrices of the throughput sweep, both layouts
        {"name": "circuit_tiled_14q", "kind": "circuit", "layout": "tiled", "n": 14, "gates": 60},
        {"name": "circuit_packed_14q", "kind": "circuit", "layout": "packed", "n": 14, "gates": 60},
        # the Kraus-channel configuration: four channels on each of 13 qubits, packed storage
        {"name": "channels_packed_13q", "kind": "channels", "layout": "packed", "n": 13, "per_qubit": 4},
        # exact scores of the noisy surrogate search: 12 qubits, six layers, depolarizing noise
        {"name": "noisy_tiled_12q", "kind": "noisy", "n": 12, "p": 6, "evals": 2},
        # the batched configuration: 3-regular MaxCut of 16 to 24 qubits, four layers
        {"name": "qaoa_mixed_64", "kind": "qaoa", "count": 64, "n_min": 16, "n_max": 24, "p": 4, "weighted": False},
        # the surrogate's exact evaluator: one weighted graph of 24 qubits at many angle sets
        {"name": "qaoa_weighted_24q", "kind": "qaoa", "count": 8, "n_min": 24, "n_max": 24, "p": 6, "weighted": True},
        # one training step's gradients of the 12-256-256-1 network, and of its inputs
        {"name": "mlp_gradients_1024", "kind": "gradients", "rows": 1024, "n_in": 12, "hidden": 256},
        # one screening round of the surrogate search: 32 x 1024 candidates
        {"name": "mlp_forward_32768", "kind": "forward", "rows": 32768, "n_in": 12, "hidden": 256},
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("circuit", "circuit", "circuit", "channels", "noisy", "qaoa", "qaoa", "gradients", "forward"))
    if kind == "circuit":
        layout = rng.choice(("pure", "tiled", "packed"))
        if layout == "pure":
            return {"kind": kind, "layout": layout, "n": rng.randint(6, 29), "gates": spread(24, 200)}
        n = rng.randint(4, 14)
        return {"kind": kind, "layout": layout, "n": n, "gates": spread(24, 60 if n > 12 else 200)}
    if kind == "channels":
        return {"kind": kind, "layout": rng.choice(("tiled", "packed")), "n": rng.randint(5, 13),
                "per_qubit": rng.randint(1, 4)}
    if kind == "noisy":
        return {"kind": kind, "n": rng.randint(6, 12), "p": rng.randint(1, 6), "evals": rng.randint(1, 6)}
    if kind == "qaoa":
        if rng.random() < 0.4:                # many angle sets of one weighted graph
            n = rng.randint(10, 24)
            return {"kind": kind, "count": rng.randint(2, 8) * (1 if n > 22 else 4), "n_min": n, "n_max": n,
                    "p": rng.randint(1, 6), "weighted": True}
        lo = rng.randint(8, 20)
        return {"kind": kind, "count": spread(5, 64), "n_min": lo, "n_max": rng.randint(lo, 24), "p": rng.randint(1, 6),
                "weighted": False}
    n_in = 2 * rng.randint(1, 8)
    if kind == "gradients":
        return {"kind": kind, "rows": spread(64, 2048), "n_in": n_in, "hidden": 256}
    return {"kind": kind, "rows": spread(1000, 40000), "n_in": n_in, "hidden": 256}


# ---------------------------------------------------------------------------------------
# inputs, made from the case and the seed alone
# ---------------------------------------------------------------------------------------
def _arity(name):
    return 3 if name == "ccx" else 2 if name in PAIRS else 1


def _circuit(case, seed):
    """[(gate, qubits, angle or None)]: gates uniform over the 18 calls, distinct qubits."""
    rng = np.random.default_rng([seed, 1])
    out = []
    for _ in range(case["gates"]):
        name = GATES[int(rng.integers(len(GATES)))]
        qs = tuple(int(q) for q in rng.choice(case["n"], size=_arity(name), replace=False))
        out.append((name, qs, float(rng.uniform(0.0, 2.0 * math.pi)) if name in ANGLE_1Q else None))
    return out


def _gaussian(out, gen):
    """Fill the complex vector out with a Gaussian-random normalised state, in place."""
    r = torch.view_as_real(out)
    r.normal_(generator=gen)
    r.mul_(1.0 / float(torch.linalg.vector_norm(r)))
    return out


def _generator(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 16 + salt)
    return g


def _observable(n, seed):
    return torch.rand(1 << n, generator=_generator(seed, 2), device="cuda", dtype=torch.float64) * 2.0 - 1.0


def _density(n, seed):
    """A Dirichlet(1,1,1,1)-weighted mixture of four Gaussian-random pure states, d x d."""
    w = np.random.default_rng([seed, 3]).dirichlet(np.ones(4))
    gen = _generator(seed, 3)
    rho = torch.zeros((1 << n, 1 << n), dtype=torch.complex128, device="cuda")
    for wi in w:
        p = _gaussian(torch.empty(1 << n, dtype=torch.complex128, device="cuda"), gen)
        rho.addr_(p * float(wi), p.conj())
    return rho


def _store(layout, rho):
    """The stored elements of a density matrix: packed lower triangle by columns, or the
    lower-triangular grid of row-major tiles."""
    d = rho.shape[0]
    if layout == "packed":
        return rho.t()[torch.ones((d, d), dtype=torch.bool, device=rho.device).triu_()]
    if d < TILE:
        padded = torch.zeros((TILE, TILE), dtype=rho.dtype, device=rho.device)
        padded[:d, :d] = rho
        return padded.reshape(-1)
    nt = d // TILE
    tr, tc = torch.tril_indices(nt, nt, device=rho.device)
    return rho.view(nt, TILE, nt, TILE).permute(0, 2, 1, 3)[tr, tc].reshape(-1)


def _kraus(case, seed):
    """[(Kraus operators, qubit)]: depolarizing, amplitude damping, phase damping and a random
    four-operator channel (a Gaussian isometry) on every qubit, the first `per_qubit` of them."""
    rng = np.random.default_rng([seed, 4])
    x, y, z = np.array([[0, 1], [1, 0]]), np.array([[0, -1j], [1j, 0]]), np.array([[1, 0], [0, -1]])
    out = []
    for q in range(case["n"]):
        p, g, lam = rng.uniform(0.0, 0.1), rng.uniform(0.0, 0.2), rng.uniform(0.0, 0.2)
        iso, _ = np.linalg.qr(rng.standard_normal((8, 2)) + 1j * rng.standard_normal((8, 2)))
        a, b = math.sqrt(1 - 3 * p / 4), math.sqrt(p / 4)
        sets = [[iso[2 * i:2 * i + 2] for i in range(4)],
                [a * np.eye(2), b * x, b * y, b * z],
                [np.diag([1, math.sqrt(1 - g)]), np.array([[0, math.sqrt(g)], [0, 0]])],
                [np.diag([1, math.sqrt(1 - lam)]), np.diag([0, math.sqrt(lam)])]]
        out += [([np.asarray(k, dtype=np.complex128) for k in ks], q) for ks in sets[:case["per_qubit"]]]
    return out


def _regular(n, rng):
    """A random 3-regular graph (one vertex of degree 2 when n is odd): shuffled stubs, paired
    until no loop and no double edge is left."""
    deg = np.full(n, 3)
    if n % 2:
        deg[rng.integers(n)] = 2
    while True:
        ends = rng.permutation(np.repeat(np.arange(n), deg)).reshape(-1, 2)
        edges = {(int(min(e)), int(max(e))) for e in ends}
        if len(edges) == len(ends) and all(u != v for u, v in edges):
            return [(int(u), int(v)) for u, v in ends]


def _weighted(n, rng):
    """An Erdos-Renyi graph (edge probability 0.3) and weights uniform in [0, 1]."""
    edges = [(u, v) for u in range(n) for v in range(u + 1, n) if rng.random() < 0.3] or [(0, n - 1)]
    return edges, [float(w) for w in rng.uniform(0.0, 1.0, len(edges))]


def _batch(case, seed):
    """Qubit counts, edges, weights (or None) and the angles of a batch."""
    rng = np.random.default_rng([seed, 5])
    count, p = case["count"], case["p"]
    if case["weighted"]:
        edges, w = _weighted(case["n_min"], rng)
        ns, es, ws = [case["n_min"]] * count, [edges] * count, [w] * count
    else:
        ns = [int(n) for n in rng.integers(case["n_min"], case["n_max"] + 1, count)]
        es, ws = [_regular(n, rng) for n in ns], None
    return ns, es, ws, rng.uniform(0, math.pi, (count, p)), rng.uniform(0, math.pi / 2, (count, p))


def _noisy(case, seed):
    rng = np.random.default_rng([seed, 6])
    edges, w = _weighted(case["n"], rng)
    shape = (case["evals"], case["p"])
    return edges, w, rng.uniform(0, math.pi, shape), rng.uniform(0, math.pi / 2, shape)


def _network(case, seed):
    """Parameters in the network's layout (W1, b1, W2, b2, W3, b3), inputs in [-1, 1], targets."""
    rng = np.random.default_rng([seed, 7])
    i, h = case["n_in"], case["hidden"]

    def u(fan_in, *shape):
        return rng.uniform(-1.0, 1.0, shape) * math.sqrt(6.0 / fan_in)

    p = np.concatenate([u(i, i * h), 0.1 * u(1, h), u(h, h * h), 0.1 * u(1, h), u(h, h), 0.1 * u(1, 1)])
    x = rng.uniform(-1.0, 1.0, (case["rows"], i))
    return p.astype(np.float32), x.astype(np.float32), rng.standard_normal(case["rows"]).astype(np.float32)


class _State:
    """A device state and a tensor over its storage; the state is freed when neither this
    object nor the tensor, which holds the memory's owner, is in use any more."""

    class _Memory:
        def __init__(self, ork, st):
            self.ork, self.st = ork, st
            self.__cuda_array_interface__ = {"shape": (int(ork.lib.state_len(ctypes.byref(st))),), "typestr": "<c16",
                                             "data": (int(st.data), False), "version": 3, "strides": None}

        def __del__(self):
            self.ork.free(self.st)

    def __init__(self, ork, layout, n):
        self.st = ork.state(layout, n)
        self.tensor = torch.as_tensor(self._Memory(ork, self.st), device="cuda")


def prepare(case, seed):
    ork = orkan_b200.load(5)
    kind = case["kind"]
    if kind in ("circuit", "channels"):
        layout, n = case["layout"], case["n"]
        if n > 24:
            torch.cuda.empty_cache()          # room for the state itself
        own = _State(ork, layout, n)
        if layout == "pure":
            _gaussian(own.tensor, _generator(seed, 1))
        else:
            own.tensor.copy_(_store(layout, _density(n, seed)))
        s = {"kind": kind, "ork": ork, "own": own, "obs": _observable(n, seed)}
        if kind == "circuit":
            s["gates"] = _circuit(case, seed)
        else:
            s["channels"] = [(ork.superop(ks), q) for ks, q in _kraus(case, seed)]
        return s
    if kind == "noisy":
        edges, w, g, b = _noisy(case, seed)
        ev = surrogate.NoisyEvaluator(ork, case["n"], edges, w, case["p"], NOISE)
        return {"kind": kind, "evaluate": ev, "g": g, "b": b}
    if kind == "qaoa":
        ns, es, ws, g, b = _batch(case, seed)
        return {"kind": kind, "batch": QaoaBatch(ork, ns, es, ws, case["p"]), "g": g, "b": b}
    p, x, t = _network(case, seed)
    net = surrogate.Mlp(ork, n_in=case["n_in"], hidden=case["hidden"],
                        max_batch=max(1024, case["rows"]) if kind == "gradients" else 1024)
    net.set_params(p)
    return {"kind": kind, "net": net, "x": torch.from_numpy(x).cuda(), "t": torch.from_numpy(t).cuda()}


def run(s):
    kind = s["kind"]
    if kind in ("circuit", "channels"):
        ork, st = s["ork"], s["own"].st
        if kind == "circuit":
            for name, qubits, theta in s["gates"]:
                ork.gate(st, name, qubits, theta)
        else:
            for sop, q in s["channels"]:
                ork.channel_1q(st, sop, q)
        m = ork.mean(st, s["obs"].data_ptr())
        return {"mean": np.array([m]), "state": s["own"].tensor}     # mean launched every gate
    if kind == "noisy":
        return s["evaluate"](s["g"], s["b"])
    if kind == "qaoa":
        return s["batch"].run(s["g"], s["b"])
    if kind == "gradients":
        loss, g, gx = s["net"].gradients(s["x"], s["t"], want_x=True)
        return {"loss": loss, "params": g, "inputs": gx}
    return s["net"].forward(s["x"])


# ---------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------
# share of a density matrix's elements a gate call changes, and its flops per changed element
_SHARE = {"cx": 0.75, "cy": 0.75, "swap": 0.75, "ccx": 7 / 16, "cz": 3 / 8,
          "z": 0.5, "s": 0.5, "sdg": 0.5, "t": 0.5, "tdg": 0.5, "rz": 0.5, "p": 0.5}
_FLOPS = {"h": 4, "hy": 4, "rx": 6, "ry": 6, "rz": 6, "p": 3, "t": 2, "tdg": 2}


def _stored(layout, n):
    d = 1 << n
    if layout == "pure":
        return d
    if layout == "packed":
        return d * (d + 1) // 2
    nt = max(1, d // TILE)
    return nt * (nt + 1) // 2 * TILE * TILE


def work(case):
    kind = case["kind"]
    if kind == "circuit":
        n, size = case["n"], _stored(case["layout"], case["n"])
        gates = _circuit(case, 1)
        if case["layout"] == "pure":          # gate calls are queued: the state in and out once
            return {"bytes": 32 * size + 8 * (1 << n), "flops": size * sum(_FLOPS.get(g, 0) for g, _, _ in gates)}
        return {"bytes": 32 * size * sum(_SHARE.get(g, 1.0) for g, _, _ in gates),   # call by call
                "flops": 2 * size * sum(_FLOPS.get(g, 0) * _SHARE.get(g, 1.0) for g, _, _ in gates)}
    if kind == "channels":
        size, calls = _stored(case["layout"], case["n"]), case["n"] * case["per_qubit"]
        return {"bytes": 32 * size * calls, "flops": 32 * size * calls}
    if kind == "noisy":                       # in: costs and angles, out: energies; the rest is arithmetic
        size = _stored("tiled", case["n"])
        return {"bytes": case["evals"] * (8 << case["n"]), "flops": case["evals"] * case["p"] * size * (32 * case["n"] + 6)}
    if kind == "qaoa":                        # four-FMA pair updates, a phase per layer, the mean
        ns = _batch(case, 1)[0]
        return {"bytes": sum((8 if case["weighted"] else 1) << n for n in (ns[:1] if case["weighted"] else ns)),
                "flops": sum((1 << n) * (case["p"] * (4 * n + 6) + 4) for n in ns)}
    i, h, rows = case["n_in"], case["hidden"], case["rows"]
    params = i * h + h * h + 3 * h + 1
    if kind == "forward":
        return {"bytes": 4 * (rows * (i + 1) + params), "flops": 2 * rows * (i * h + h * h + h)}
    return {"bytes": 4 * (rows * (2 * i + 1) + 2 * params), "flops": 6 * rows * (i * h + h * h + h)}


# ---------------------------------------------------------------------------------------
# the same results in 64 bits by plain torch and numpy
# ---------------------------------------------------------------------------------------
def _matrix(name, theta):
    r = math.sqrt(0.5)
    i2 = np.eye(2, dtype=np.complex128)
    x, y = np.array([[0, 1], [1, 0]], dtype=np.complex128), np.array([[0, -1j], [1j, 0]])
    if theta is not None:
        c, s = math.cos(theta / 2), math.sin(theta / 2)
        return {"rx": np.array([[c, -1j * s], [-1j * s, c]]), "ry": np.array([[c, -s], [s, c]], dtype=np.complex128),
                "rz": np.diag([complex(c, -s), complex(c, s)]),
                "p": np.diag([1, complex(math.cos(theta), math.sin(theta))])}[name]
    one = {"x": x, "y": y, "z": np.diag([1, -1 + 0j]), "h": r * np.array([[1, 1], [1, -1]], dtype=np.complex128),
           "s": np.diag([1, 1j]), "sdg": np.diag([1, -1j]), "t": np.diag([1, complex(r, r)]),
           "tdg": np.diag([1, complex(r, -r)]), "hy": r * np.array([[1, -1], [1, 1]], dtype=np.complex128)}
    if name in one:
        return one[name]
    u = np.eye(8 if name == "ccx" else 4, dtype=np.complex128)
    if name == "swap":
        return u[[0, 2, 1, 3]]
    u[-2:, -2:] = {"cx": x, "cy": y, "cz": np.diag([1, -1]), "ccx": x}[name] @ i2
    return u


def _apply(v, bits, qubits, u):
    """v <- u v on the listed bits of a 2^bits vector (the first is the local index's highest)."""
    order = sorted(qubits, reverse=True)
    shape, top = [], bits
    for q in order:
        shape += [1 << (top - q - 1), 2]
        top = q
    t = v.view(shape + [1 << top])
    k = len(qubits)

    def part(l):
        at = [slice(None)] * t.dim()
        for j, q in enumerate(qubits):
            at[2 * order.index(q) + 1] = (l >> (k - 1 - j)) & 1
        return t[tuple(at)]

    rows = [l for l in range(1 << k) if not (u[l, l] == 1 and np.count_nonzero(u[l]) == 1)]
    new = []
    for l in rows:
        acc = None
        for m in np.nonzero(u[l])[0]:
            c = complex(u[l, m])
            acc = part(int(m)) * c if acc is None else acc.add_(part(int(m)), alpha=c)
        new.append(acc if acc is not None else torch.zeros_like(part(l)))
    for l, x in zip(rows, new):
        part(l).copy_(x)


def _superop(kraus):
    return sum(np.einsum("ik,jl->ijkl", k, k.conj()).reshape(4, 4) for k in kraus)


def _bits_cost(n, edges, w):
    x = torch.arange(1 << n, device="cuda")
    cost = torch.zeros(1 << n, dtype=torch.float64, device="cuda")
    for e, (a, b) in enumerate(edges):
        cost += (1.0 if w is None else w[e]) * (((x >> a) ^ (x >> b)) & 1).double()
    return cost


def _exact_noisy(case, seed):
    edges, w, g, b = _noisy(case, seed)
    n = case["n"]
    d = 1 << n
    cost = _bits_cost(n, edges, w)
    x, y, z = np.array([[0, 1], [1, 0]]), np.array([[0, -1j], [1j, 0]]), np.array([[1, 0], [0, -1]])
    noise = [math.sqrt(1 - 0.75 * NOISE) * np.eye(2)] + [math.sqrt(NOISE / 4) * m for m in (x, y, z)]
    out = []
    for e in range(case["evals"]):
        rho = torch.full((d, d), 1.0 / d, dtype=torch.complex128, device="cuda")
        for k in range(case["p"]):
            ph = torch.exp(-1j * float(g[e, k]) * cost)
            rho *= ph[:, None] * ph.conj()[None, :]
            sop = _superop([m @ _matrix("rx", 2.0 * float(b[e, k])) for m in noise])
            for q in range(n):
                _apply(rho.view(-1), 2 * n, (n + q, q), sop)
        out.append(float((rho.diagonal().real * cost).sum()))
    return np.array(out)


def _exact_qaoa(case, seed):
    ns, es, ws, g, b = _batch(case, seed)
    out = []
    for i, n in enumerate(ns):
        cost = _bits_cost(n, es[i], None if ws is None else ws[i])
        v = torch.full((1 << n,), 2.0 ** (-n / 2), dtype=torch.complex128, device="cuda")
        for k in range(case["p"]):
            v *= torch.exp(-1j * float(g[i, k]) * cost)
            u = _matrix("rx", 2.0 * float(b[i, k]))
            for q in range(n):
                _apply(v, n, (q,), u)
        out.append(float((v.real.square() * cost).sum() + (v.imag.square() * cost).sum()))
    return np.array(out)


def _exact_network(case, seed):
    p, x, t = (torch.from_numpy(a).cuda().double() for a in _network(case, seed))
    i, h = case["n_in"], case["hidden"]
    p.requires_grad_(True)
    x.requires_grad_(True)
    w1, b1, w2, b2, w3, b3 = torch.split(p, [i * h, h, h * h, h, h, 1])
    a1 = torch.nn.functional.gelu(x @ w1.view(i, h) + b1)
    a2 = torch.nn.functional.gelu(a1 @ w2.view(h, h) + b2)
    y = a2 @ w3 + b3
    if case["kind"] == "forward":
        return y.detach()
    loss = (y - t).square().mean()
    gp, gx = torch.autograd.grad(loss, (p, x))
    return {"loss": float(loss.detach()), "params": gp, "inputs": gx}


def exact(case, seed):
    kind = case["kind"]
    if kind == "noisy":
        return _exact_noisy(case, seed)
    if kind == "qaoa":
        return _exact_qaoa(case, seed)
    if kind in ("gradients", "forward"):
        return _exact_network(case, seed)
    n, layout = case["n"], case["layout"]
    obs = _observable(n, seed)
    if layout == "pure":
        v = _gaussian(torch.empty(1 << n, dtype=torch.complex128, device="cuda"), _generator(seed, 1))
        for name, qs, theta in _circuit(case, seed):
            _apply(v, n, qs, _matrix(name, theta))
        m = sum(float((torch.view_as_real(c).square().sum(1) * o).sum())
                for c, o in zip(v.split(1 << 26), obs.split(1 << 26)))
        return {"mean": np.array([m]), "state": v}
    rho = _density(n, seed)
    if kind == "circuit":
        for name, qs, theta in _circuit(case, seed):
            u = _matrix(name, theta)
            _apply(rho.view(-1), 2 * n, tuple(n + q for q in qs), u)
            _apply(rho.view(-1), 2 * n, qs, u.conj())
    else:
        for ks, q in _kraus(case, seed):
            _apply(rho.view(-1), 2 * n, (n + q, q), _superop(ks))
    m = float((rho.diagonal().real * obs).sum())
    return {"mean": np.array([m]), "state": _store(layout, rho)}
