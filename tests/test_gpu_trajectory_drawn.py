"""Complex64 trajectory passes of rounds, renames and noise mixtures (branches resolved by the producer
warp) against the same segments without lowering, on swizzled and plain tiles: the same measured
bits for the same uniforms. A uniform decides the other way when it lies within the two forms'
difference of a probability, about 2e-6: 200 shots of some twenty draws expect 0.01 such shots, one is let
pass. Noise strong enough that tiles take one- and two-qubit branches other than the identity."""

from __future__ import annotations

import numpy as np
import pytest

import lucivant_sim_gb300 as ls
from lucivant_sim_gb300 import _lib
from lucivant_sim_gb300.noise import NoiseModel, depolarizing, pauli_channel
from lucivant_sim_gb300.trajectories import TrajectoryProgram

pytestmark = pytest.mark.gpu


def _source(n, rounds, seed, plain):
    rng = np.random.default_rng(seed)
    lines = [f'OPENQASM 3.0; include "stdgates.inc"; qubit[{n}] q; bit[{rounds}] c; bit[{n}] d;']
    for r in range(rounds):
        for q in range(n):
            a, b, c = rng.uniform(-3, 3, 3)
            lines.append([f"U({a}, {b}, {c}) q[{q}];", f"ry({a}) q[{q}]; rz({b}) q[{q}];", f"sx q[{q}]; t q[{q}];",
                          f"h q[{q}];"][rng.integers(4)])
        for q in range(r % 2, n - 1, 2):
            gate = ["cx", "cz", "swap", "rzz(0.3)"] if plain else ["cx", "cz", "cry(0.8)", "ch"]
            lines.append(gate[rng.integers(4)] + f" q[{q}], q[{q + 1}];")
        lines.append(f"c[{r}] = measure q[{r % n}];")
        lines.append(f"if (c[{r}] == 1) {{ ry(0.4) q[{(r + 1) % n}]; x q[{r % n}]; }}")
        lines.append(f"reset q[{(r + 1) % n}];")
    return "\n".join(lines + ["d = measure q;"])


@pytest.mark.parametrize("plain", [True, False], ids=["rounds", "controlled"])
@pytest.mark.parametrize("n", [2, 4, 7, 8, 9, 12, 13, 15])
def test_drawn_passes_measure_the_same_bits(n, plain, monkeypatch):
    circuit = ls.parse(_source(n, 4, n, plain))
    noise = NoiseModel().add_gate_error(depolarizing(0.1, 1), gates=["u", "ry", "h"])
    noise.add_gate_error(depolarizing(0.15, 2), gates=["cx", "cz", "swap"])
    noise.add_gate_error(pauli_channel({"X": 0.2, "Z": 0.1}), gates=["sx"])
    shots = 200
    got = []
    for fuse, swizzle in (("1", "1"), ("0", "1"), ("1", "0")):
        monkeypatch.setenv("LSG_FUSE_BLOCKS", fuse)
        monkeypatch.setenv("LSG_SWIZZLE", swizzle)
        prog = TrajectoryProgram(circuit, noise, _lib.C64, shots)
        uniforms = np.random.default_rng(n).random((shots, max(prog.max_draws, 1)))
        bits, used, _ = prog.run_batched(uniforms)
        serial = TrajectoryProgram(circuit, noise, _lib.C64, 1)
        one, ones, _ = serial.run_serial(20, uniforms[:20].reshape(-1))
        got.append((np.array(bits), np.array(used), np.array(one)))
    for bits, used, one in got[1:]:
        assert np.sum(np.any((bits != got[0][0]).reshape(shots, -1), axis=1)) <= 1
        assert np.sum(used != got[0][1]) <= 1
        assert np.sum(np.any((one != got[0][2]).reshape(len(one), -1), axis=1)) <= 1
