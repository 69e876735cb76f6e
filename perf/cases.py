"""The work that users of this framework have it do, as cases to be timed.

Each case is a plain dict; prepare() builds what a program holds before the call (states in
HBM, circuits, engines, a server), run() makes one pass through the public Python API and
returns the results whole, work() counts the bytes and operations that the pass cannot do
without, and exact() gives the same results in 64 bits from plain torch.

Kinds:

  calls    one State method per gate on a small or medium ket: interactive use, where a
           call's latency and launch count (the tests' and config 1's gate mix: 70% Haar
           1-qudit, 30% Haar 2-qudit, some controlled gates)
  sequence the same mix as one Circuit (1000 gates + 100 controlled on 20 qubits is the
           benchmark's first configuration), plain or fused
  layered  a Circuit of layers (Haar 1-qubit gate on every qubit, then Haar 2-qubit gates on
           a random perfect matching): the benchmark's headline workload
  rho_ops  density-matrix steps on resident states: gates or a 16-operator pair channel, then
           ptrace, ptranspose and syspermute (the benchmark's second configuration and its
           mixed-dimension variant)
  rho_run  a layered Circuit with a pair channel after every 2-qubit gate on a density
           matrix: the circuits that noisy requests on density matrices bring
  batch    many independent kets and density matrices of uneven sizes, each with its own
           circuit, in one call (the benchmark's batched configuration, scaled down)
  qft      QFT / TFQ of a whole register or of part of it (the reference's QFT benchmark)
  engine   QEngine: reset, execute(shots) of a layered circuit that ends in measurements
  serve    QNoisyEngine requests (trajectories of kets, exact density matrices) through the
           batching server, all submitted at once, results read back
"""
from __future__ import annotations

import math

import numpy as np
import torch

import qpp_b200 as qb
from qpp_b200 import serving
from qpp_b200.workloads import haar_unitary

_PREC = {"c128": (qb.C128, 16, torch.complex128, "<c16"), "c64": (qb.C64, 8, torch.complex64, "<c8")}
_FORM = {"plain": qb.PLAIN, "fused": qb.FUSED}


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # 12 qubits, one Python call per gate: the smallest calls, bound by latency
        {"name": "calls_12q_c128", "kind": "calls", "d": 2, "n": 12, "prec": "c128", "gates": 24, "ctrl": 6},
        # the benchmark's first configuration: 1100 gates on 2^20 amplitudes (L2-resident)
        {"name": "sequence_20q_plain_c128", "kind": "sequence", "n": 20, "prec": "c128", "form": "plain", "gates": 1000, "ctrl": 100},
        {"name": "sequence_20q_fused_c128", "kind": "sequence", "n": 20, "prec": "c128", "form": "fused", "gates": 1000, "ctrl": 100},
        # the headline workload (30 qubits there) at a size that is still far above the L2
        {"name": "layered_28q_plain_c128", "kind": "layered", "n": 28, "prec": "c128", "form": "plain", "depth": 3},
        # its fused single-precision form
        {"name": "layered_28q_fused_c64", "kind": "layered", "n": 28, "prec": "c64", "form": "fused", "depth": 8},
        # one step of the second configuration: channel on a pair, ptrace, ptranspose, syspermute
        {"name": "rho_ops_12q_c128", "kind": "rho_ops", "dims": "2" * 12, "prec": "c128", "op": "channel"},
        # its mixed-dimension variant: odd sizes everywhere
        {"name": "rho_ops_mixed_c128", "kind": "rho_ops", "dims": "33223223", "prec": "c128", "op": "gates"},
        # a noisy density-matrix request's circuit in the fused form
        {"name": "rho_run_12q_fused_c64", "kind": "rho_run", "n": 12, "prec": "c64", "form": "fused", "depth": 6},
        # uneven instances: 96 kets of 10-22 qubits and 24 density matrices of 6-11 qubits
        {"name": "batch_c64", "kind": "batch", "kets": 96, "kmin": 10, "kmax": 22, "rhos": 24, "rmin": 6, "rmax": 11, "depth": 20},
        # QFT of every qubit of a large register
        {"name": "qft_28q_c128", "kind": "qft", "n": 28, "prec": "c128", "part": "all", "inverse": False, "swap": True},
        # a measured circuit, 1000 shots, through the engine
        {"name": "engine_20q_c128", "kind": "engine", "n": 20, "prec": "c128", "depth": 6, "shots": 1000},
        # a burst of noisy requests as the serving mix has them
        {"name": "serve_burst", "kind": "serve", "kets": 22, "nmin": 12, "nmax": 16, "rhos": 2, "rmin": 8, "rmax": 9, "depth": 24, "shots": 400},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["calls", "sequence", "layered", "layered", "rho_ops", "rho_ops", "rho_run", "batch", "qft",
                       "engine", "serve"])
    prec = rng.choice(["c128", "c64"])
    form = rng.choice(["plain", "fused"])
    if kind == "calls":
        d = rng.choice([2, 2, 3])
        return {"kind": kind, "d": d, "n": rng.randint(4, 22) if d == 2 else rng.randint(3, 13), "prec": prec,
                "gates": rng.randint(12, 48), "ctrl": rng.randint(2, 12)}
    if kind == "sequence":
        return {"kind": kind, "n": rng.randint(10, 24), "prec": prec, "form": form,
                "gates": _log_int(rng, 60, 700), "ctrl": rng.randint(0, 70)}
    if kind == "layered":
        n = rng.randint(13, 27)
        return {"kind": kind, "n": n, "prec": prec, "form": form, "depth": rng.randint(1, 3 if n > 25 else 8)}
    if kind == "rho_ops":
        if rng.random() < 0.5:
            dims = "2" * rng.randint(4, 12)
        else:  # mixed dimensions, two subsystems of each kind at least, 12 to 3000 levels
            while True:
                dims = "".join(rng.choice("223345") for _ in range(rng.randint(4, 9)))
                if 12 <= math.prod(int(x) for x in dims) <= 3000 and len(set(dims)) > 1:
                    break
        return {"kind": kind, "dims": dims, "prec": prec,
                "op": rng.choice(["channel", "gates"]) if set(dims) == {"2"} else "gates"}
    if kind == "rho_run":
        n = rng.randint(4, 12)
        if prec == "c128":  # the fused form of density matrices is a single-precision one
            form = "plain"
        return {"kind": kind, "n": n, "prec": prec, "form": form, "depth": rng.randint(2, 8)}
    if kind == "batch":
        lo, rlo = rng.randint(8, 16), rng.randint(4, 8)
        return {"kind": kind, "kets": _log_int(rng, 8, 80), "kmin": lo, "kmax": min(22, lo + rng.randint(2, 9)),
                "rhos": rng.randint(2, 20), "rmin": rlo, "rmax": min(11, rlo + rng.randint(1, 4)),
                "depth": rng.randint(5, 20)}
    if kind == "qft":
        return {"kind": kind, "n": rng.randint(8, 28), "prec": prec, "part": rng.choice(["all", "all", "some"]),
                "inverse": rng.random() < 0.5, "swap": rng.random() < 0.75}
    if kind == "engine":
        return {"kind": kind, "n": rng.randint(8, 23), "prec": "c128", "depth": rng.randint(2, 8),
                "shots": _log_int(rng, 1, 2000)}
    return {"kind": kind, "kets": rng.randint(4, 20), "nmin": 12, "nmax": rng.randint(12, 16), "rhos": rng.randint(1, 2),
            "rmin": 8, "rmax": rng.randint(8, 10), "depth": rng.randint(10, 24), "shots": _log_int(rng, 20, 400)}


# -------------------------------------------------------- inputs from the seed
def _gauss(size, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    v = torch.randn(size, dtype=dtype, device="cuda", generator=g)
    r = torch.view_as_real(v).reshape(-1)
    return v.div_(float(torch.linalg.vector_norm(r)))


def _rho(D, rank, dtype, seed):
    """A random density matrix (rank columns), column-major: entry [c, r] of the tensor."""
    W = _gauss(D * rank, torch.complex128, seed).view(rank, D)
    return (W.conj().t() @ W).to(dtype).contiguous()


def _gate_mix(rng, n, d, gates, ctrl):
    """[(U, controls, targets)]: 70% Haar 1-qudit, 30% Haar 2-qudit, then controlled 1-qudit
    gates with 1-3 controls (one control for d > 2)."""
    seq = []
    for _ in range(gates):
        k = 1 if rng.random() < 0.7 else 2
        t = [int(x) for x in rng.choice(n, size=k, replace=False)]
        seq.append((haar_unitary(rng, d ** k), [], t))
    for _ in range(ctrl):
        nc = int(rng.integers(1, min(4, n))) if d == 2 else 1
        sub = [int(x) for x in rng.choice(n, size=nc + 1, replace=False)]
        seq.append((haar_unitary(rng, d), sub[:nc], sub[nc:]))
    return seq


def _layers(rng, n, depth, bank=64):
    """[(U, [], targets)] of a layered circuit; gates from a bank of Haar matrices."""
    one = [haar_unitary(rng, 2) for _ in range(bank)]
    two = [haar_unitary(rng, 4) for _ in range(bank)]
    seq = []
    for _ in range(depth):
        seq += [(one[int(rng.integers(bank))], [], [q]) for q in range(n)]
        p = [int(x) for x in rng.permutation(n)]
        seq += [(two[int(rng.integers(bank))], [], [p[2 * i], p[2 * i + 1]]) for i in range(n // 2)]
    return seq


def _circuit(seq, n, d=2, nc=0):
    c = qb.Circuit(n, d, nc)
    for U, cs, t in seq:
        c.CTRL(U, cs, t) if cs else c.gate(U, t)
    return c


def _noisy_layers(rng, n, depth, chan, each):
    """A layered circuit with `chan` after every 2-qubit gate (each = False: on its pair) or on
    every qubit after every layer (each = True): [(matrix or Kraus list, targets)]."""
    steps = []
    one = [haar_unitary(rng, 2) for _ in range(32)]
    two = [haar_unitary(rng, 4) for _ in range(32)]
    for _ in range(depth):
        steps += [(one[int(rng.integers(32))], [q]) for q in range(n)]
        p = [int(x) for x in rng.permutation(n)]
        for i in range(n // 2):
            t = [p[2 * i], p[2 * i + 1]]
            steps.append((two[int(rng.integers(32))], t))
            if chan is not None and not each:
                steps.append((chan, t))
        if chan is not None and each:
            steps += [(chan, [q]) for q in range(n)]
    return steps


def _noisy_circuit(steps, n, nc=0):
    c = qb.Circuit(n, 2, nc)
    for A, t in steps:
        serving.c_channel(c, A, t) if isinstance(A, list) else c.gate(A, t)
    return c


def _depol(p):
    I2, X, Z = np.eye(2), np.array([[0, 1], [1, 0]]), np.diag([1, -1])
    Ks = [math.sqrt(1 - p) * I2] + [math.sqrt(p / 3) * P for P in (X, 1j * X @ Z, Z)]
    return [np.asarray(K, dtype=np.complex128) for K in Ks]


def _rho_step(case, rng):
    """The matrices and subsystems of one rho_ops step."""
    dims = [int(x) for x in case["dims"]]
    n = len(dims)
    half = n // 2
    if case["op"] == "channel":
        ops = [(serving.pair_channel(), [int(x) for x in rng.choice(n, 2, replace=False)])]
    else:
        a, b = (int(x) for x in rng.choice(n, 2, replace=False))
        ops = [(haar_unitary(rng, dims[a]), [a]), (haar_unitary(rng, dims[a] * dims[b]), [a, b])]
    return (dims, ops, sorted(int(x) for x in rng.choice(n, half, replace=False)),
            sorted(int(x) for x in rng.choice(n, half, replace=False)), [int(x) for x in rng.permutation(n)])


def _spread(lo, hi, count):
    return [lo + i % (hi - lo + 1) for i in range(count)]


def _batch_parts(case, seed):
    """[(kind, n, steps, seed of the state)] of a batch; sizes come from the case alone."""
    rng = np.random.default_rng(seed)
    chan = _depol(0.005)
    parts = []
    for i, n in enumerate(_spread(case["kmin"], case["kmax"], case["kets"])):
        parts.append((qb.KET, n, _noisy_layers(rng, n, case["depth"], None, True), seed + 100 + i))
    for i, n in enumerate(_spread(case["rmin"], case["rmax"], case["rhos"])):
        parts.append((qb.RHO, n, _noisy_layers(rng, n, case["depth"], chan, True), seed + 100000 + i))
    return parts


def _part_state(kind, n, seed):
    return _gauss(2 ** n, torch.complex64, seed) if kind == qb.KET else _rho(2 ** n, 8, torch.complex64, seed)


def _qft_targets(case, seed):
    n = case["n"]
    if case["part"] == "all":
        return None
    rng = np.random.default_rng(seed + 1)
    return [int(x) for x in rng.permutation(n)[: max(2, (2 * n) // 3)]]


# ---------------------------------------------------------------- device views
class _Buffer:
    """A State's memory as a CUDA array (the State lives as long as its tensor)."""

    def __init__(self, state):
        self.state = state
        n = state.D if state.kind == qb.KET else state.D * state.D
        typestr = "<c16" if state.prec == qb.C128 else "<c8"
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "version": 2,
                                         "data": (state.device_ptr(), False), "strides": None}


def _view(state):
    return torch.as_tensor(_Buffer(state), device="cuda")


def _state(ctx, kind, dims, prec, values):
    s = qb.State(ctx, kind, dims, _PREC[prec][0])
    ctx.synchronize()
    v = _view(s)
    v.copy_(values.reshape(-1))
    torch.cuda.current_stream().synchronize()
    return s, v


_server = None
_requests = []  # a server's requests keep their circuits: they live as long as it does


def _the_server():
    global _server
    if _server is None:
        _server = serving.Server(0)
    return _server


# --------------------------------------------------------------------- prepare
def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    ctx = qb.default_context()
    st = {"case": case, "kind": kind, "ctx": ctx}
    if kind in ("calls", "sequence", "layered"):
        n, d = case["n"], case.get("d", 2)
        st["s"], st["v"] = _state(ctx, qb.KET, [d] * n, case["prec"], _gauss(d ** n, _PREC[case["prec"]][2], seed))
        seq = _layers(rng, n, case["depth"]) if kind == "layered" else _gate_mix(rng, n, d, case["gates"], case["ctrl"])
        if kind == "calls":
            st["seq"] = seq
        else:
            st["c"], st["form"] = _circuit(seq, n), _FORM[case["form"]]
    elif kind == "rho_ops":
        st["dims"], st["ops"], st["tr"], st["tp"], st["perm"] = _rho_step(case, rng)
        D = math.prod(st["dims"])
        st["s"], st["v"] = _state(ctx, qb.RHO, st["dims"], case["prec"], _rho(D, min(64, D), _PREC[case["prec"]][2], seed))
    elif kind == "rho_run":
        n = case["n"]
        st["c"] = _noisy_circuit(_noisy_layers(rng, n, case["depth"], serving.pair_channel(), False), n)
        st["form"] = _FORM[case["form"]]
        st["s"], st["v"] = _state(ctx, qb.RHO, [2] * n, case["prec"], _rho(2 ** n, 8, _PREC[case["prec"]][2], seed))
    elif kind == "batch":
        st["c"], st["s"], st["v"] = [], [], {}
        for k, n, steps, sd in _batch_parts(case, seed):
            st["c"].append(_noisy_circuit(steps, n))
            s, v = _state(ctx, k, [2] * n, "c64", _part_state(k, n, sd))
            st["s"].append(s)
            st["v"].setdefault(("ket" if k == qb.KET else "rho") + str(n), []).append(v)
        st["stream"] = torch.cuda.ExternalStream(ctx.stream())
    elif kind == "qft":
        n = case["n"]
        st["targets"] = _qft_targets(case, seed)
        st["s"], st["v"] = _state(ctx, qb.KET, [2] * n, case["prec"], _gauss(2 ** n, _PREC[case["prec"]][2], seed))
    elif kind == "engine":
        n = case["n"]
        c = _circuit(_layers(rng, n, case["depth"]), n, 2, n)
        for q in range(n):
            c.measure([q], q, destructive=False)
        st["e"], st["seed"] = qb.Engine(ctx, c, qb.KET, _PREC[case["prec"]][0]), seed % (1 << 31)
    else:
        srv = _the_server()
        reqs = []
        # sizes as the serving mix has them: P(n) ~ 2^-(n - nmin); shots log-uniform
        for i in range(case["kets"]):
            n = case["nmin"]
            while n < case["nmax"] and (i + 1) % (2 << (n - case["nmin"])) == 0:
                n += 1
            shots = max(1, int(round(case["shots"] ** ((i * 7 % case["kets"] + 1) / case["kets"]))))
            c = _noisy_circuit(_noisy_layers(rng, n, case["depth"], None, True), n, 2 if i % 5 == 4 else 1)
            if i % 5 == 4:
                for j in range(2):
                    c.measure([int(rng.integers(n))], j, destructive=False)
            reqs.append((c, qb.KET, 1e-3, shots, seed % (1 << 31) + i))
        for i, n in enumerate(_spread(case["rmin"], case["rmax"], case["rhos"])):
            c = _noisy_circuit(_noisy_layers(rng, n, case["depth"], serving.pair_channel(), False), n, 1)
            reqs.append((c, qb.RHO, 0.0, 16, seed % (1 << 31) + 1000 + i))
        _requests.extend(reqs)
        st["srv"], st["reqs"] = srv, reqs
    return st


# ------------------------------------------------------------------------- run
def run(st):
    kind, s = st["kind"], st.get("s")
    if kind == "calls":
        for U, cs, t in st["seq"]:
            s.apply_ctrl(U, cs, t) if cs else s.apply(U, t)
        return st["v"]
    if kind in ("sequence", "layered", "rho_run"):
        st["c"].run(s, st["form"])
        return st["v"]
    if kind == "rho_ops":
        for A, t in st["ops"]:
            s.apply_kraus(A, t) if isinstance(A, list) else s.apply(A, t)
        return {"rho": st["v"], "ptrace": _view(s.ptrace(st["tr"])), "ptranspose": _view(s.ptranspose(st["tp"])),
                "syspermute": _view(s.syspermute(st["perm"]))}
    if kind == "batch":
        qb.run_batch(st["ctx"], st["c"], s, qb.FUSED)
        with torch.cuda.stream(st["stream"]):
            return {k: torch.cat(v) for k, v in st["v"].items()}
    if kind == "qft":
        inv, swap = st["case"]["inverse"], st["case"]["swap"]
        if st["targets"] is None:
            s.qft(2, swap, inv)
        elif inv:
            s.apply_tfq(st["targets"], 2, swap)
        else:
            s.apply_qft(st["targets"], 2, swap)
        return _view(s)  # a transform may leave the state in another buffer
    if kind == "engine":
        e = st["e"]
        e.set_seed(st["seed"]).reset().execute(st["case"]["shots"])
        stats = sorted(e.get_stats().items())
        dits, probs = e.get_dits()
        outcomes = np.zeros((st["case"]["shots"], len(dits) + 1), dtype=np.int64)  # a row each, its count last
        for i, (k, v) in enumerate(stats):
            outcomes[i, :-1], outcomes[i, -1] = k, v
        return {"outcomes": outcomes, "dits": np.array(dits, dtype=np.int64), "probs": np.array(probs)}
    srv = st["srv"]
    ids = [srv.submit(*r) for r in st["reqs"]]
    got = [srv.wait(i, shots=r[3], nc=r[0].nc) for i, r in zip(ids, st["reqs"])]
    return {"samples": np.concatenate([g[1] for g in got]).astype(np.int64),
            "dits": np.concatenate([g[2] for g in got]).astype(np.int64)}


# ------------------------------------------------------------------------ work
def _seq_flops(seq, D, d=2):
    """Real operations of the gates one by one: a complex multiply-add (8) per matrix entry
    and amplitude column; a controlled gate acts on the amplitudes its controls select."""
    return sum(8.0 * len(U) * D / d ** len(cs) for U, cs, _ in seq)


def work(case):
    kind = case["kind"]
    rng = np.random.default_rng(1)
    if kind in ("calls", "sequence", "layered"):
        d, n = case.get("d", 2), case["n"]
        D, eb = float(d ** n), _PREC[case["prec"]][1]
        if kind == "layered":
            flops = case["depth"] * (n * 16.0 + (n // 2) * 32.0) * D
        else:
            flops = _seq_flops(_gate_mix(rng, n, d, case["gates"], case["ctrl"]), D, d)
        if kind == "calls":  # every call reads and writes what its controls select
            byts = sum(2.0 * eb * D / d ** len(cs) for _, cs, _ in _gate_mix(rng, n, d, case["gates"], case["ctrl"]))
        else:
            byts = 2.0 * eb * D
        return {"bytes": byts, "flops": flops}
    if kind == "rho_ops":
        D, eb = float(math.prod(int(x) for x in case["dims"])), _PREC[case["prec"]][1]
        dims, ops, tr, _, _ = _rho_step(case, rng)
        Db = D / math.prod(dims[q] for q in tr)
        flops = sum(8.0 * D * D * (math.prod(dims[q] for q in t) ** 2 if isinstance(A, list) else 2 * len(A)) for A, t in ops)
        nops = len(ops)
        return {"bytes": eb * (2.0 * nops * D * D + 4.0 * D * D + D * Db + Db * Db), "flops": flops}
    if kind == "rho_run":
        D2 = 4.0 ** case["n"]
        pairs = case["n"] // 2
        return {"bytes": 2.0 * _PREC[case["prec"]][1] * D2,
                "flops": case["depth"] * 8.0 * D2 * (case["n"] * 4 + pairs * (8 + 16))}
    if kind == "batch":
        byts = flops = 0.0
        for n in _spread(case["kmin"], case["kmax"], case["kets"]):
            byts += 16.0 * 2 ** n
            flops += case["depth"] * (16.0 * n + 32.0 * (n // 2)) * 2 ** n
        for n in _spread(case["rmin"], case["rmax"], case["rhos"]):
            byts += 16.0 * 4 ** n
            flops += case["depth"] * 8.0 * (4 * n + 8 * (n // 2) + 4 * n) * 4 ** n
        return {"bytes": byts, "flops": flops}
    if kind == "qft":
        D, eb = 2.0 ** case["n"], _PREC[case["prec"]][1]
        k = case["n"] if case["part"] == "all" else max(2, (2 * case["n"]) // 3)
        return {"bytes": 2.0 * eb * D, "flops": 5.0 * k * D}
    if kind == "engine":
        D, n = 2.0 ** case["n"], case["n"]
        return {"bytes": _PREC[case["prec"]][1] * D, "flops": case["depth"] * (16.0 * n + 32.0 * (n // 2)) * D}
    flops = 0.0  # every trajectory runs its gates; states never need to leave the chip
    shots = 0
    for i in range(case["kets"]):
        n = case["nmin"]
        while n < case["nmax"] and (i + 1) % (2 << (n - case["nmin"])) == 0:
            n += 1
        sh = max(1, int(round(case["shots"] ** ((i * 7 % case["kets"] + 1) / case["kets"]))))
        shots += sh
        flops += sh * case["depth"] * (16.0 * n + 32.0 * (n // 2)) * 2 ** n
    for n in _spread(case["rmin"], case["rmax"], case["rhos"]):
        flops += case["depth"] * 8.0 * 4 ** n * (n * 4 + (n // 2) * 24)
        shots += 16
    return {"bytes": 12.0 * shots, "flops": flops}


# ----------------------------------------------------------------------- exact
def _apply(psi, U, targets, dims, ctrl=()):
    """U on the targets of the flat complex128 ket psi over dims (plain torch); controlled
    qubit gates act where every control reads 1, controlled qudit gates as U^r."""
    U = torch.as_tensor(np.ascontiguousarray(U), device=psi.device)
    if ctrl:
        d = dims[ctrl[0]]
        v = psi.view(dims).clone()
        for r in range(1, d):
            idx = tuple(r if q in ctrl else slice(None) for q in range(len(dims)))
            rest = [q for q in range(len(dims)) if q not in ctrl]
            sub = v[idx].contiguous()
            v[idx] = _apply(sub.view(-1), np.linalg.matrix_power(U.cpu().numpy(), r), [rest.index(t) for t in targets],
                            [dims[q] for q in rest]).view(sub.shape)
        return v.reshape(-1)
    # dims merged into runs around the (sorted) targets
    order = sorted(targets)
    k = len(targets)
    shape, at = [], 0
    for t in order:
        shape += [math.prod(dims[at:t]), dims[t]]
        at = t + 1
    shape.append(math.prod(dims[at:]))
    td = [dims[t] for t in targets]
    v = psi.view(shape)
    axis = [2 * order.index(t) + 1 for t in targets]
    rest = [x for x in range(len(shape)) if x not in axis]
    m = v.permute(*axis, *rest).reshape(math.prod(td), -1)
    out = (U @ m).view(td + [shape[x] for x in rest])
    back = [0] * len(shape)
    for i, x in enumerate(axis + rest):
        back[x] = i
    assert k == len(td)
    return out.permute(*back).reshape(-1)


def _rho_apply(rho, A, t, dims):
    """A gate, or the channel of a Kraus list, on the flat column-major matrix."""
    n, D2 = len(dims), list(dims) + list(dims)
    Ks = A if isinstance(A, list) else [A]
    S = sum(np.kron(K.conj(), K) for K in Ks)
    return _apply(rho, S, list(t) + [n + q for q in t], D2)


def _dft(x, sign):
    """sum_j exp(sign 2 pi i j k / N) x[:, j] / sqrt(N) for N = N1 N2 a power of two, as N1-point
    and N2-point transforms with the twiddles between them."""
    B, N = x.shape
    N1 = 1 << ((N.bit_length() - 1) // 2)
    N2 = N // N1
    f = torch.fft.ifft if sign > 0 else torch.fft.fft
    x = f(x.view(B, N1, N2), dim=1, norm="ortho")
    jk = torch.arange(N1, device=x.device)[:, None] * torch.arange(N2, device=x.device)[None, :]
    ang = jk.to(torch.float64).mul_(sign * 2 * math.pi / N)
    x = f(x * torch.polar(torch.ones_like(ang), ang), dim=2, norm="ortho")
    return x.transpose(1, 2).reshape(B, N)


def exact(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind in ("calls", "sequence", "layered"):
        n, d = case["n"], case.get("d", 2)
        seq = _layers(rng, n, case["depth"]) if kind == "layered" else _gate_mix(rng, n, d, case["gates"], case["ctrl"])
        v = _gauss(d ** n, _PREC[case["prec"]][2], seed).to(torch.complex128)
        if d ** n * len(seq) > 2 ** 37:  # over 20 seconds of plain torch
            return None
        for U, cs, t in seq:
            v = _apply(v, U, t, [d] * n, cs)
        return v
    if kind == "rho_ops":
        dims, ops, tr, tp, perm = _rho_step(case, rng)
        D, n = math.prod(dims), len(dims)
        v = _rho(D, min(64, D), _PREC[case["prec"]][2], seed).to(torch.complex128).view(-1)
        for A, t in ops:
            v = _rho_apply(v, A, t, dims)
        m = v.view(dims + dims)  # [column digits, row digits]
        keep = [q for q in range(n) if q not in tr]
        p = m.permute(keep + [n + q for q in keep] + tr + [n + q for q in tr])
        Db, DS = math.prod(dims[q] for q in keep), math.prod(dims[q] for q in tr)
        pt = p.reshape(Db, Db, DS, DS).diagonal(dim1=2, dim2=3).sum(-1)
        swap = [q + n if q in tp else q for q in range(n)] + [q if q in tp else q + n for q in range(n)]
        return {"rho": v, "ptrace": pt.reshape(-1), "ptranspose": m.permute(swap).reshape(-1),
                "syspermute": m.permute(perm + [n + q for q in perm]).reshape(-1)}
    if kind == "rho_run":
        n = case["n"]
        v = _rho(2 ** n, 8, _PREC[case["prec"]][2], seed).to(torch.complex128).view(-1)
        for A, t in _noisy_layers(rng, n, case["depth"], serving.pair_channel(), False):
            v = _rho_apply(v, A, t, [2] * n)
        return v
    if kind == "batch":
        out = {}
        for k, n, steps, sd in _batch_parts(case, seed):
            v = _part_state(k, n, sd).to(torch.complex128).view(-1)
            for A, t in steps:
                v = _apply(v, A, t, [2] * n) if k == qb.KET else _rho_apply(v, A, t, [2] * n)
            out.setdefault(("ket" if k == qb.KET else "rho") + str(n), []).append(v)
        return {k: torch.cat(v) for k, v in out.items()}
    if kind == "qft":
        n = case["n"]
        t = _qft_targets(case, seed) or list(range(n))
        k = len(t)
        v = _gauss(2 ** n, _PREC[case["prec"]][2], seed).to(torch.complex128).view([2] * n)
        rest = [q for q in range(n) if q not in t]
        rev = list(range(len(rest))) + [len(rest) + k - 1 - i for i in range(k)]
        v = v.permute(rest + t)
        if case["inverse"]:  # the target reversal comes first, the transform's adjoint after it
            if not case["swap"]:
                v = v.permute(rev)
            v = _dft(v.reshape(-1, 2 ** k), -1).view([2] * n)
        else:
            v = _dft(v.reshape(-1, 2 ** k), 1).view([2] * n)
            if not case["swap"]:
                v = v.permute(rev)
        back = [0] * n
        for i, q in enumerate(rest + t):
            back[q] = i
        return v.permute(back).reshape(-1)
    return None  # drawn outcomes: whole numbers
