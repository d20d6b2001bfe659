"""support() in panels of 64 columns at the sizes where its threads, panels and rows per thread change,
against the path with a launch per column; noise masks drawn by a thread per gate and word, against the
oracle's frames, at shot counts around a word, with one- and two-qubit branches, all-or-nothing
probabilities and a first branch that is not the identity; frames of more qubits than one CTA's threads."""

from __future__ import annotations

import numpy as np
import pytest

import lucivant_sim_gb300 as ls
from lucivant_sim_gb300 import stabilizer as st
from lucivant_sim_gb300.clifford import all_gates
from lucivant_sim_gb300.noise import NoiseModel, ReadoutError, depolarizing, pauli_channel
from oracle import tableau

pytestmark = pytest.mark.gpu


def _clifford(n, layers, seed, frac=1.0, measure=False):
    rng = np.random.default_rng(seed)
    active = rng.permutation(n)[: max(1, int(frac * n))]
    lines = [f'OPENQASM 3.0; include "stdgates.inc"; qubit[{n}] q;' + (f" bit[{n}] c;" if measure else "")]
    for _ in range(layers):
        for q in active:
            lines.append(f"{['h', 's', 'x', 'sdg', 'sx'][rng.integers(5)]} q[{q}];")
        perm = rng.permutation(active)
        for i in range(0, len(perm) - 1, 2):
            lines.append(f"{['cx', 'cz', 'swap', 'cy'][rng.integers(4)]} q[{perm[i]}], q[{perm[i + 1]}];")
    return ls.parse("\n".join(lines + (["c = measure q;"] if measure else [])))


@pytest.mark.parametrize("n", [1, 31, 64, 65, 127, 255, 256, 257, 511, 512, 513, 577, 1024, 1985, 2048])
def test_support_panels_equal_launch_per_column(n, monkeypatch):
    circuit = _clifford(n, 3, n, frac=0.7)
    enc = st.Encoder(None)
    t = st.Tableau(n)
    try:
        t.apply(enc.encode(all_gates(circuit.operations), False), enc)
        qubits = [list(range(n)), list(range(n))[::-1], list(range(0, n, 2))]
        got = [t.support(q) for q in qubits]
        alone = [t.support(q, want_basis=False)[0] for q in qubits]
        monkeypatch.setenv("LSG_SUPPORT_STEPS", "1")
        for q, (x0, basis), x1 in zip(qubits, got, alone, strict=True):
            want, rows = t.support(q)
            assert np.array_equal(x0, want) and np.array_equal(x1, want) and np.array_equal(basis, rows)
    finally:
        t.free()


@pytest.mark.parametrize("n,shots", [(1, 1), (2, 31), (5, 32), (9, 33), (70, 97), (600, 65), (1100, 40)])
@pytest.mark.parametrize("kind", ["depolarizing", "pauli", "certain"])
def test_frames_equal_the_oracles(n, shots, kind):
    noise = NoiseModel()
    if kind == "depolarizing":
        noise.add_gate_error(depolarizing(0.1, 1)).add_gate_error(depolarizing(0.2, 2))
    elif kind == "pauli":
        noise.add_gate_error(pauli_channel({"X": 0.5, "Y": 0.2, "Z": 0.3}), gates=["h", "s"])
        noise.add_gate_error(pauli_channel({"XZ": 0.3, "IY": 0.1, "ZI": 0.05}))
    else:
        noise.add_gate_error(pauli_channel({"Y": 1.0}), gates=["h", "x"])
        noise.add_gate_error(pauli_channel({"ZX": 1.0}))
    noise.add_readout_error(ReadoutError(0.1, 0.3))
    circuit = _clifford(n, 4, n + shots, measure=True)
    a, b = np.random.default_rng(n), np.random.default_rng(n)
    assert st.run_counts(circuit, shots, noise, a) == tableau.frames(circuit, shots, noise, b)
    # the stream's position (without the buffered half of a draw, which is stale when it is not in use)
    x, y = a.bit_generator.state, b.bit_generator.state
    assert x["state"] == y["state"] and x["has_uint32"] == y["has_uint32"]
    assert not x["has_uint32"] or x["uinteger"] == y["uinteger"]
