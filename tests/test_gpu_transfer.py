"""Real64 density programs run their one-qubit transfer operators as shears with the scales in the
block's diagonals: equal to the dense products and to the vectorised complex form to 1e-13 (some hundred
operators of a few units of 1e-16 each, on coefficients of at most one), and a member of a batch
bit-identical to itself alone, over noise that factors well (thermal, depolarising), badly (full
dephasing, strong damping) or not at all (resets), with gates that let a rotation pass and that do not."""

from __future__ import annotations

import numpy as np
import pytest

import lucivant_sim_gb300 as ls
from lucivant_sim_gb300 import _lib, engine, noise as nm, workloads as wl

pytestmark = pytest.mark.gpu


def _source(n, layers, seed, resets):
    rng = np.random.default_rng(seed)
    lines = [f'OPENQASM 3.0; include "stdgates.inc"; qubit[{n}] q;']
    for k in range(layers):
        for q in range(n):
            a, b, c = rng.choice([0.0, np.pi / 2, np.pi, -1.3, 0.7, 2.9, 1e-9], 3)
            lines.append([f"u3({a}, {b}, {c}) q[{q}];", f"rz({a}) q[{q}];", f"ry({b}) q[{q}];", f"h q[{q}];",
                          f"u3({c}, {a}, {b}) q[{q}]; u3({a}, {b}, {c}) q[{q}];"][rng.integers(5)])
            if resets and rng.random() < 0.1:
                lines.append(f"reset q[{q}];")
        for q in range(k % 2, n - 1, 2):
            a, b = (q, q + 1) if rng.random() < 0.5 else (q + 1, q)
            lines.append(["cx", "cx", "cz", "cy", "swap", "crz(0.4)", "ch"][rng.integers(7)] + f" q[{a}], q[{b}];")
    return "\n".join(lines)


def _noises(kind):
    if kind == "thermal":
        return [ls.NoiseModel.uniform(two=t).add_gate_error(wl.thermal_depolarizing(s), gates="u3")
                for s, t in ((1e-3, 1e-2), (2e-2, 5e-2), (1e-4, 2e-3))]
    one = {"phase": [nm.phase_damping(p) for p in (0.1, 1.0, 0.999999)],
           "amplitude": [nm.amplitude_damping(p) for p in (0.3, 1.0, 1e-8)],
           "pauli": [nm.pauli_channel({"X": x, "Y": 0.02, "Z": 0.1}) for x in (0.1, 0.0, 0.3)]}[kind]
    return [ls.NoiseModel.uniform(two=0.02).add_gate_error(c, gates=["u3", "h"]) for c in one]


def _density(circuit, noises, member=0):
    with engine.evolve_density(circuit, noises, _lib.C128) as reg:
        return [engine.density_download(reg, m) for m in ([member] if member is not None else range(len(noises)))]


@pytest.mark.parametrize("kind", ["thermal", "phase", "amplitude", "pauli"])
@pytest.mark.parametrize("n,layers,seed,resets", [(1, 4, 1, False), (2, 6, 2, False), (3, 8, 3, True), (5, 9, 4, False),
                                                  (7, 6, 5, True)])
def test_shears_equal_products(n, layers, seed, resets, kind, monkeypatch):
    circuit = ls.parse(_source(n, layers, seed, resets))
    noises = _noises(kind)
    assert engine.dm_form(circuit, noises) == "ptm"
    got = _density(circuit, noises, None)
    kinds = [row[0] for row in engine.ptm_oplist(circuit, noises).rows]
    for m, noise in enumerate(noises):
        # (full dephasing beside a partial one: the batch's operators hold both patterns, another list)
        if [row[0] for row in engine.ptm_oplist(circuit, [noise]).rows] == kinds:
            assert np.array_equal(_density(circuit, [noise])[0], got[m])
    monkeypatch.setenv("LSG_JIT", "0")
    plain = _density(circuit, noises, None)
    monkeypatch.setenv("LSG_FUSE_BLOCKS", "0")
    products = _density(circuit, noises, None)
    monkeypatch.setenv("LSG_DM_FORM", "superop")
    general = _density(circuit, noises, None)
    for m in range(len(noises)):
        assert np.array_equal(got[m], plain[m])
        assert np.max(np.abs(got[m] - products[m])) < 1e-13
        assert np.max(np.abs(got[m] - general[m])) < 1e-13
