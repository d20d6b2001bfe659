"""What is measured: the work a program has this engine do, through its public entry points.

Kinds of case (the key ``kind``) and what they stand for:

* ``vqe``     a variational loop on one circuit template: every pass takes a new parameter set into
              the planned program, replays it as one CUDA graph and reads a Pauli sum's terms;
* ``run``     ``ls.run`` of a whole circuit, as a drop-in caller has it: evolve, sample, count;
* ``expect``  one wide statevector evolved and measured on a Pauli sum;
* ``sweep``   parameter sets of one template as members of one register (the served sweeps);
* ``dm``      noise instances of one circuit as density matrices: probabilities and <Z>, <ZZ>;
* ``traj``    noisy shots with mid-circuit measurement, conditions and reset, all shots at once
              ("batched") or one after another in the drop-in draw order ("serial");
* ``stab``    a wide Clifford circuit with Pauli and readout noise, counts from Pauli frames.

Circuits are the layers the benchmark runs: u3 on every qubit with uniform angles, then cx on
alternating neighbours (small turns where expectations are read); templates are ry, rz layers with
a linear cx chain. Results of a
single-precision request are handed on in single precision: FP64 reductions of FP32 amplitudes
hold no more than that.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import lucivant_sim_gb300 as ls
from lucivant_sim_gb300 import _lib, engine, serve, stabilizer, workloads
from lucivant_sim_gb300.batch import DensityBatch
from lucivant_sim_gb300.trajectories import TrajectoryProgram

PRECISION = {"c128": _lib.C128, "c64": _lib.C64}
TERMS = 20  # Pauli terms of a measured observable (the served jobs' size)
# Circuits whose observables are read turn little per layer (a time step, an optimisation under
# way): their expectations are of order one. Uniform turns at these widths leave noise-sized ones.
STEP, WARM = 0.2, 0.5


def listed():
    return [
        # the smallest call: a few microseconds of device work, launches and copies count
        dict(name="vqe-8q-c128", kind="vqe", n=8, layers=4, precision="c128"),
        # a drop-in call at the size the configuration names: 20 qubits, 20 layers, 10,000 shots
        dict(name="run-20q-c128", kind="run", n=20, layers=20, shots=10000),
        # a wide double-precision statevector: bound by FP64 arithmetic
        dict(name="expect-22q-c128", kind="expect", n=22, layers=20, precision="c128"),
        # the widest register the engine takes, single precision, 512 MiB of amplitudes
        dict(name="expect-26q-c64", kind="expect", n=26, layers=40, precision="c64"),
        # a served parameter sweep: 8 members of one template
        dict(name="sweep-17q-c64", kind="sweep", n=17, layers=6, members=8, precision="c64"),
        # the headline batch in FP64, single and double-float (fewer instances: a pass under a second)
        dict(name="dm-12q-c128", kind="dm", n=12, layers=12, members=64, precision="c128"),
        dict(name="dm-12q-c64", kind="dm", n=12, layers=12, members=128, precision="c64"),
        dict(name="dm-12q-df64", kind="dm", n=12, layers=12, members=64, precision="df64"),
        # a small noisy register, where few tiles exist
        dict(name="dm-9q-c128", kind="dm", n=9, layers=20, members=8, precision="c128"),
        # noisy mid-circuit shots at the configuration's width, all at once
        dict(name="traj-18q-c64", kind="traj", n=18, rounds=16, shots=512, mode="batched", precision="c64"),
        # the default trajectory mode of the drop-in call: shots in sequence
        dict(name="traj-13q-c128", kind="traj", n=13, rounds=6, shots=40, mode="serial", precision="c128"),
        # the tableau and the Pauli frames at the configuration's width
        dict(name="stab-2048q", kind="stab", n=2048, layers=100, shots=1000),
    ]


def draw(rng):
    """One more case of the same ranges; each kind's cost stays below the largest listed case."""

    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["vqe", "run", "expect", "sweep", "dm", "dm", "traj", "stab"])
    if kind == "vqe":
        return dict(kind=kind, n=rng.randint(4, 14), layers=log(1, 6), precision=rng.choice(["c128", "c64"]))
    if kind == "run":
        return dict(kind=kind, n=rng.randint(5, 21), layers=log(2, 24), shots=log(100, 20000))
    if kind == "expect":
        precision = rng.choice(["c128", "c64"])
        return dict(kind=kind, n=rng.randint(11, 23 if precision == "c128" else 26), layers=log(3, 40), precision=precision)
    if kind == "sweep":
        return dict(kind=kind, n=rng.randint(6, 20), layers=log(1, 6), members=rng.randint(2, 16), precision=rng.choice(["c128", "c64"]))
    if kind == "dm":
        n = rng.randint(3, 11)
        return dict(kind=kind, n=n, layers=log(2, 24), members=log(1, min(64, 4 ** (13 - n))), precision=rng.choice(["c128", "c64", "df64"]))
    if kind == "traj":
        mode = rng.choice(["batched", "serial"])
        n = rng.randint(8, 18 if mode == "batched" else 16)
        return dict(kind=kind, n=n, rounds=log(1, 12), shots=log(32, 512) if mode == "batched" else log(8, 48), mode=mode,
                    precision=rng.choice(["c128", "c64"]) if mode == "serial" or n < 16 else "c64")
    return dict(kind=kind, n=log(40, 2048), layers=log(4, 120), shots=log(100, 1500))


# ------------------------------------------------------------------------------- inputs


def _brickwork(n, layers, seed, turn=2 * math.pi):
    """Gates of the brickwork circuit: ("u3", q, theta, phi, lambda) and ("cx", a, b). theta is
    uniform on [0, turn), the phases on [0, 2 pi)."""
    angles = np.random.default_rng(seed).uniform(0.0, 1.0, size=(layers, n, 3)) * [turn, 2 * math.pi, 2 * math.pi]
    gates = []
    for layer in range(layers):
        gates += [("u3", q, *map(float, angles[layer, q])) for q in range(n)]
        gates += [("cx", a, a + 1) for a in range(layer % 2, n - 1, 2)]
    return gates


def _ansatz(n, layers, seed):
    """Gates of the hardware-efficient template: ("ry", q, t), ("rz", q, t), a cx chain."""
    angles = np.random.default_rng(seed).uniform(0.0, 1.0, size=(layers, n, 2)) * [WARM, 2 * math.pi]
    gates = []
    for layer in range(layers):
        for q in range(n):
            gates += [("ry", q, float(angles[layer, q, 0])), ("rz", q, float(angles[layer, q, 1]))]
        gates += [("cx", a, a + 1) for a in range(n - 1)]
    return gates


def _circuit(n, gates, measure=False):
    lines = ["OPENQASM 3.0;", 'include "stdgates.inc";', f"qubit[{n}] q;"] + ([f"bit[{n}] c;"] if measure else [])
    for g in gates:
        if g[0] == "cx":
            lines.append(f"cx q[{g[1]}], q[{g[2]}];")
        else:
            lines.append(f"{g[0]}({', '.join(repr(v) for v in g[2:])}) q[{g[1]}];")
    return ls.parse("\n".join(lines + (["c = measure q;"] if measure else [])) + "\n")


def _labels(n, seed):
    """Pauli strings of a measured sum, qubit 0 rightmost: half of them neighbour couplings and
    fields of a spin chain, half drawn at random."""
    rng = np.random.default_rng([seed, 17])
    labels = []
    for k in range(TERMS):
        word = ["I"] * n
        if k % 2 == 0:
            q = int(rng.integers(0, n - 1))
            word[n - 1 - q], word[n - 2 - q] = [("Z", "Z"), ("X", "I"), ("X", "X")][int(rng.integers(0, 3))]
        else:
            word = ["IXYZ"[int(v)] for v in rng.integers(0, 4, size=n)]
        labels.append("".join(word))
    return labels


def _masks(labels):
    pairs = [engine.pauli_masks(lab) for lab in labels]
    return [p[0] for p in pairs], [p[1] for p in pairs]


def _errors(members, seed):
    """One- and two-qubit error rates of the noise instances."""
    rng = np.random.default_rng([seed, 23])
    return rng.uniform(1e-4, 5e-3, size=members), rng.uniform(1e-3, 3e-2, size=members)


def _noises(members, seed):
    return [ls.NoiseModel.uniform(two=float(t), readout=2e-2).add_gate_error(workloads.thermal_depolarizing(float(s)), gates="u3")
            for s, t in zip(*_errors(members, seed))]


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    if kind == "vqe":
        reg = _lib.Register(n, PRECISION[case["precision"]])
        lists = [engine.sv_oplist(_circuit(n, _ansatz(n, case["layers"], seed + 1000 * k))) for k in range(2)]
        return dict(case=case, reg=reg, prog=_lib.Program(reg, lists[1]), ops=lists[0], masks=_masks(_labels(n, seed)))
    if kind == "run":
        return dict(case=case, seed=seed, circuit=_circuit(n, _brickwork(n, case["layers"], seed), measure=True))
    if kind == "expect":
        reg = _lib.Register(n, PRECISION[case["precision"]])
        ops = engine.sv_oplist(_circuit(n, _brickwork(n, case["layers"], seed, STEP)))
        return dict(case=case, reg=reg, prog=_lib.Program(reg, ops), masks=_masks(_labels(n, seed)))
    if kind == "sweep":
        reg = _lib.Register(n, PRECISION[case["precision"]], case["members"])
        ops = serve.sweep_oplist([_circuit(n, _ansatz(n, case["layers"], seed + 1000 * k)) for k in range(case["members"])])
        return dict(case=case, reg=reg, prog=_lib.Program(reg, ops), masks=_masks(_labels(n, seed)))
    if kind == "dm":
        circuit = _circuit(n, _brickwork(n, case["layers"], seed))
        batch = DensityBatch(circuit, _noises(case["members"], seed), precision=case["precision"], autotune=False)
        return dict(case=case, batch=batch, labels=workloads.z_observables(n))
    if kind == "traj":
        circuit = ls.parse(workloads.midcircuit(n, case["rounds"], seed=seed))
        noise = ls.NoiseModel.uniform(single=1e-3, two=1e-2)
        serial = case["mode"] == "serial"
        prog = TrajectoryProgram(circuit, noise, PRECISION[case["precision"]], 1 if serial else case["shots"])
        uniforms = np.random.default_rng([seed, 29]).random((case["shots"], max(prog.max_draws, 1)))
        return dict(case=case, prog=prog, uniforms=uniforms.reshape(-1) if serial else uniforms)
    circuit = workloads.clifford_layers_circuit(n, case["layers"], seed=seed)
    return dict(case=case, circuit=circuit, noise=workloads.stabilizer_noise(), seed=seed)


# --------------------------------------------------------------------------------- one pass


def _handed_on(values, precision):
    """Results of a single-precision request in single precision."""
    return values.astype(np.float32) if precision == "c64" else values


def _each(outcomes, tally):
    """Every shot's outcome, a row each, from the distinct ones and how often they came."""
    return np.repeat(outcomes, np.fromiter(tally.values(), dtype=np.int64, count=len(tally)), axis=0)


def run(state):
    case = state["case"]
    kind, precision = case["kind"], case.get("precision")
    if kind == "vqe":
        state["prog"].set_data(state["reg"], state["ops"])
        state["prog"].graph_run(state["reg"])
        return _handed_on(state["reg"].expect(0, *state["masks"]), precision)
    if kind == "run":
        result = ls.run(state["circuit"], shots=case["shots"], seed=state["seed"], method="statevector")
        outcomes = np.frombuffer("".join(result.counts).encode(), dtype=np.uint8).reshape(-1, case["n"])
        return dict(statevector=result.statevector, outcomes=_each(outcomes, result.counts))
    if kind in ("expect", "sweep"):
        state["prog"].run_from_basis(state["reg"])
        return _handed_on(state["reg"].expect(0, *state["masks"]), precision)
    if kind == "dm":
        batch = state["batch"]
        batch.evolve()
        return dict(probabilities=_handed_on(batch.probabilities(), precision),
                    expectations=_handed_on(batch.expectations(state["labels"]), precision))
    if kind == "traj":
        if case["mode"] == "serial":
            bits, used, _ = state["prog"].run_serial(case["shots"], state["uniforms"])
            return dict(bits=bits.view(np.int64), used=used)
        bits, used, _ = state["prog"].run_batched(state["uniforms"])
        return dict(bits=bits.view(np.int64), used=used)
    tally = stabilizer.run_counts(state["circuit"], case["shots"], state["noise"], np.random.default_rng(state["seed"]))
    width = (case["n"] + 7) // 8
    outcomes = np.frombuffer(b"".join(k.to_bytes(width, "little") for k in tally), dtype=np.uint8).reshape(-1, width)
    return dict(outcomes=_each(outcomes, tally))


def work(case):
    kind, n, layers = case["kind"], case["n"], case.get("layers", case.get("rounds"))
    size = {"c128": 16, "c64": 8, "df64": 8, None: 16}[case.get("precision")]
    if kind == "stab":
        # per layer n one-qubit gates and n two-qubit ones on 2n tableau rows and on every shot's frame
        rows = 2.0 * n + case["shots"]
        return dict(bytes=n * 2.0 * rows / 8 + case["shots"] * n, flops=layers * 2.0 * n * 4.0 * rows / 32)
    # a one-qubit gate on a statevector: two complex products and a sum an amplitude (14 operations)
    gates = 14.0 * layers * n * 2.0**n
    if kind in ("vqe", "sweep", "expect"):
        members = case.get("members", 1)
        # the state written, and read once for the observable's terms
        return dict(bytes=members * 2.0 * size * 2.0**n, flops=members * (gates + 6.0 * TERMS * 2.0**n))
    if kind == "run":
        return dict(bytes=2.0 * size * 2.0**n + 8.0 * case["shots"], flops=gates + 4.0 * 2.0**n)
    if kind == "dm":
        # real coefficients: a noisy one-qubit gate is 10 products and 7 sums on 4 coefficients, a
        # noisy cx one product a coefficient; the register written and its diagonal read
        members, elem = case["members"], 4 if case["precision"] == "c64" else 8
        pairs = sum(len(range(k % 2, n - 1, 2)) for k in range(layers))
        return dict(bytes=members * (elem * 4.0**n + 2.0 * elem * 2.0**n), flops=members * 4.0**n * (4.25 * layers * n + pairs))
    # trajectories: gates, and per round the four measured and reset qubits (norms, a renormalisation)
    return dict(bytes=2.0 * size * case["shots"] * 2.0**n, flops=case["shots"] * (gates + layers * 8 * 4.0 * 2.0**n))


# ---------------------------------------------------------------- the same in 64 bits, plain torch


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _matrix(gate):
    name, angles = gate[0], gate[2:]
    c, s = math.cos(angles[0] / 2), math.sin(angles[0] / 2)
    if name == "ry":
        return [[c, -s], [s, c]]
    if name == "rz":
        return [[complex(c, -s), 0], [0, complex(c, s)]]
    phi, lam = angles[1], angles[2]
    return [[c, -complex(math.cos(lam), math.sin(lam)) * s],
            [complex(math.cos(phi), math.sin(phi)) * s, complex(math.cos(phi + lam), math.sin(phi + lam)) * c]]


def _statevector(n, gates):
    psi = torch.zeros(2**n, dtype=torch.complex128, device=_device())
    psi[0] = 1
    for gate in gates:
        if gate[0] == "cx":
            control, target = gate[1], gate[2]
            hi, lo = max(control, target), min(control, target)
            v = psi.view(2 ** (n - 1 - hi), 2, 2 ** (hi - lo - 1), 2, 2**lo)
            a, b = (v[:, 1, :, 0], v[:, 1, :, 1]) if control > target else (v[:, 0, :, 1], v[:, 1, :, 1])
            kept = a.clone()
            a.copy_(b)
            b.copy_(kept)
        else:
            m = _matrix(gate)
            v = psi.view(2 ** (n - 1 - gate[1]), 2, 2 ** gate[1])
            a, b = v[:, 0].clone(), v[:, 1].clone()
            v[:, 0] = m[0][0] * a + m[0][1] * b
            v[:, 1] = m[1][0] * a + m[1][1] * b
    return psi


def _parity(x):
    for shift in (16, 8, 4, 2, 1):
        x = x ^ (x >> shift)
    return x & 1


def _expectations(psi, n, labels):
    values = []
    for label in labels:
        letters = label[::-1]
        x = sum(1 << q for q in range(n) if letters[q] in "XY")
        z = sum(1 << q for q in range(n) if letters[q] in "ZY")
        total, step = 0.0, 1 << 22
        for at in range(0, 2**n, step):
            i = torch.arange(at, min(at + step, 2**n), device=psi.device)
            terms = psi[i ^ x].conj() * psi[i] * (1 - 2 * _parity(i & z))
            total = total + (terms.sum() * 1j ** bin(x & z).count("1")).real
        values.append(total)
    return torch.stack(values)


def _density(case, seed):
    """Pauli coefficients of every instance, digits I, X, Y, Z per qubit (qubit 0 fastest), evolved
    through gates and channels; the probabilities (members, 2^n)."""
    n, members, device = case["n"], case["members"], _device()
    single, two = (torch.tensor(v, device=device) for v in _errors(members, seed))
    t1, t2, time = 120.0, 90.0, 0.05
    gamma = 1 - math.exp(-time / t1)
    lam = max(0.0, 1 - math.exp(-2 * time / t2 + time / t1))
    paulis = [np.eye(2), np.array([[0, 1], [1, 0]]), np.array([[0, -1j], [1j, 0]]), np.diag([1, -1])]
    noise = torch.zeros(members, 4, 4, dtype=torch.float64, device=device)
    keep = 1 - 2 * single  # depolarising of average infidelity r: p = 2 r; then relaxation
    flat = math.sqrt((1 - gamma) * (1 - lam))
    noise[:, 0, 0], noise[:, 1, 1], noise[:, 2, 2] = 1, flat * keep, flat * keep
    noise[:, 3, 0], noise[:, 3, 3] = gamma, (1 - gamma) * keep
    cx = np.eye(4)[[0, 1, 3, 2]]  # control the most significant
    pairs = [np.kron(paulis[k // 4], paulis[k % 4]) for k in range(16)]  # control digit, target digit
    table = np.array([[np.trace(a @ cx @ b @ cx.T).real / 4 for b in pairs] for a in pairs])
    # the neighbour (a, a + 1): the control a is the fast digit of the pair in the register
    swap = [4 * (k % 4) + k // 4 for k in range(16)]
    table = table[np.ix_(swap, swap)]
    source = torch.tensor(np.abs(table).argmax(axis=1), device=device)
    sign = torch.tensor([round(table[k, int(s)]) for k, s in enumerate(source.tolist())], dtype=torch.float64, device=device)
    scale = (1 - two * 4 / 3)[:, None] * torch.ones(16, dtype=torch.float64, device=device)
    scale[:, 0] = 1
    scale = (scale * sign)[:, None, :, None]
    r = torch.zeros(members, 4**n, dtype=torch.float64, device=device)
    basis = torch.zeros(1, dtype=torch.int64, device=device)
    for q in range(n):
        basis = torch.cat([basis, basis + 3 * 4**q])
    r[:, basis] = 1  # |0...0>: every I/Z string has coefficient 1
    for gate in _brickwork(n, case["layers"], seed):
        if gate[0] == "cx":
            a = gate[1]
            v = r.view(members, 4 ** (n - 2 - a), 16, 4**a)
            r = (v[:, :, source] * scale).reshape(members, -1)
        else:
            m = np.array(_matrix(gate))
            ptm = np.array([[np.trace(p @ m @ s @ m.conj().T).real / 2 for s in paulis] for p in paulis])
            t = noise @ torch.tensor(ptm, device=device)
            v = r.view(members, 4 ** (n - 1 - gate[1]), 4, 4 ** gate[1])
            out = torch.empty_like(v)
            for i in range(4):
                out[:, :, i] = t[:, i, 0, None, None] * v[:, :, 0]
                for j in range(1, 4):
                    out[:, :, i].addcmul_(t[:, i, j, None, None], v[:, :, j])
            r = out.reshape(members, -1)
    for q in range(n):
        v = r.view(members, -1, 4, 2**q)
        r = torch.stack([(v[:, :, 0] + v[:, :, 3]) / 2, (v[:, :, 0] - v[:, :, 3]) / 2], dim=2).reshape(members, -1)
    return r.clamp_min(0)


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if kind in ("traj", "stab"):
        return None  # whole numbers only
    if kind == "run":
        psi = _statevector(n, _brickwork(n, case["layers"], seed))
        return dict(statevector=psi.cpu().numpy(), outcomes=None)
    labels = _labels(n, seed) if kind != "dm" else _z_labels(n)
    if kind == "dm":
        p = _density(case, seed)
        index = torch.arange(2**n, device=p.device)
        rows = []
        for label in labels:
            z = int(label.replace("I", "0").replace("Z", "1"), 2)
            rows.append((p * (1 - 2 * _parity(index & z))).sum(dim=1))
        return dict(probabilities=p.cpu().numpy(), expectations=torch.stack(rows).cpu().numpy())
    if kind == "sweep":
        return torch.stack([_expectations(_statevector(n, _ansatz(n, case["layers"], seed + 1000 * k)), n, labels)
                            for k in range(case["members"])], dim=1).cpu().numpy()
    gates = _ansatz(n, case["layers"], seed) if kind == "vqe" else _brickwork(n, case["layers"], seed, STEP)
    return _expectations(_statevector(n, gates), n, labels)[:, None].cpu().numpy()


def _z_labels(n):
    """<Z_i> of every qubit, then <Z_i Z_i+1> of the neighbours (qubit 0 rightmost)."""
    ones = [1 << i for i in range(n)] + [3 << i for i in range(n - 1)]
    return [format(v, f"0{n}b").replace("0", "I").replace("1", "Z") for v in ones]
