"""Complex128 trajectory segments run as rounds, their noise channels after the diagonals of their
block, and on half tiles where a register has few: the oracle's counts, shot by shot, for the same seed."""

from __future__ import annotations

import numpy as np
import pytest

import lucivant_sim_gb300 as ls
from oracle import dense

pytestmark = pytest.mark.gpu


def _source(n, rounds, seed):
    rng = np.random.default_rng(seed)
    lines = [f'OPENQASM 3.0; include "stdgates.inc"; qubit[{n}] q; bit[{rounds}] c; bit[{n}] d;']
    for r in range(rounds):
        for q in range(n):
            a, b, c = rng.uniform(-3, 3, 3)
            lines.append([f"U({a}, {b}, {c}) q[{q}];", f"ry({a}) q[{q}]; rz({b}) q[{q}];", f"sx q[{q}]; t q[{q}];",
                          f"h q[{q}];", f"y q[{q}];"][rng.integers(5)])
        for q in range(r % 2, n - 1, 2):
            lines.append(["cx", "cz", "swap", "crz(0.3)", "cry(0.8)"][rng.integers(5)] + f" q[{q}], q[{q + 1}];")
        lines.append(f"c[{r}] = measure q[{r % n}];")
        lines.append(f"if (c[{r}] == 1) {{ x q[{r % n}]; ry(0.4) q[{(r + 1) % n}]; cx q[{(r + 1) % n}], q[{(r + 2) % n}]; }}")
    return "\n".join(lines + ["d = measure q;"])


@pytest.mark.parametrize("noise", [None, ls.NoiseModel.uniform(single=3e-2, two=6e-2)], ids=["ideal", "noisy"])
@pytest.mark.parametrize("n", [3, 9, 10, 11, 13])
def test_serial_counts_are_the_oracles(n, noise):
    circuit = ls.parse(_source(n, 4, n))
    shots = 120 if n < 11 else 40
    result = ls.run(circuit, shots=shots, seed=n, noise=noise, method="trajectories")
    want, _, _ = dense.run_counts(circuit, shots, n, noise)
    assert result.counts == want or result.report["near_threshold"] > 0
