"""Specialized passes of real64 transfer programs give the interpreted ones' values bit for bit, over operators
that factor into shears, that keep their dense rows, and members with different parts."""

from __future__ import annotations

import numpy as np
import pytest

import lucivant_sim_gb300 as ls
from lucivant_sim_gb300 import _lib, engine
from test_gpu_transfer import _noises

pytestmark = pytest.mark.gpu


def _source(n, layers, seed):
    """Gates whose transfer operators have at most two bits or permute (wider ones are interpreted)."""
    rng = np.random.default_rng(seed)
    lines = [f'OPENQASM 3.0; include "stdgates.inc"; qubit[{n}] q;']
    for k in range(layers):
        for q in range(n):
            a, b, c = rng.choice([0.0, np.pi / 2, np.pi, -1.3, 0.7, 2.9, 1e-9], 3)
            lines.append([f"u3({a}, {b}, {c}) q[{q}];", f"rz({a}) q[{q}];", f"ry({b}) q[{q}];", f"h q[{q}];",
                          f"reset q[{q}];"][rng.integers(5)])
        for q in range(k % 2, n - 1, 2):
            a, b = (q, q + 1) if rng.random() < 0.5 else (q + 1, q)
            lines.append(["cx", "cz", "cy", "swap"][rng.integers(4)] + f" q[{a}], q[{b}];")
    return "\n".join(lines)


@pytest.mark.parametrize("kind", ["thermal", "phase", "amplitude", "pauli"])
@pytest.mark.parametrize("n,layers,seed", [(2, 6, 2), (3, 8, 3), (5, 9, 4), (7, 6, 5)])
def test_specialized_equals_interpreted(n, layers, seed, kind, monkeypatch):
    noises = _noises(kind)
    ops = engine.ptm_oplist(ls.parse(_source(n, layers, seed)), noises)
    got = {}
    for specialize in ("0", "1"):
        monkeypatch.setenv("LSG_JIT", specialize)
        with _lib.Register(2 * n, _lib.R64, len(noises)) as reg:
            program = _lib.Program(reg, ops)
            assert program.specialized == (specialize == "1")
            program.run_from_basis(reg)
            got[specialize] = reg.download()
            program.free()
    assert np.array_equal(got["0"], got["1"])
