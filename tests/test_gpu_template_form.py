"""New values of a program's operators change what it does, not its form, once it has met values of the
general kind: diagonals whose entries are one and parts of a transfer operator that are the identity are
multiplied all the same. Observed from the operations per element, which a form without them lacks; the
register is bit for bit that of a program made for the values."""

from __future__ import annotations

import numpy as np
import pytest

import lucivant_sim_gb300 as ls
from lucivant_sim_gb300 import _lib, engine, noise as nm, qasm, workloads as wl

pytestmark = pytest.mark.gpu


def _template(n, values):
    ops = _lib.OpList()
    circuit = qasm.parse(wl.hea_template(n, 2), {f"p{k}": float(v) for k, v in enumerate(values)})
    for op in engine.fuse_runs(circuit.operations):
        m = np.asarray(op.matrix, dtype=complex)
        ops.add(*((_lib.OP_MATRIX, list(op.qubits), m) if len(op.qubits) == 1 else
                  (engine.classify(m)[0], list(op.qubits), engine.classify(m)[1])))
    return ops


def _density(n, angles):
    """u3 gates with damping and dephasing, as transfer operators."""
    lines = [f'OPENQASM 3.0; include "stdgates.inc"; qubit[{n}] q;']
    for row in angles:
        lines += [f"u3({a}, {b}, {c}) q[{q}];" for q, (a, b, c) in enumerate(row.tolist())]
        lines += [f"cx q[{q}], q[{q + 1}];" for q in range(n - 1)]
    noise = [ls.NoiseModel.uniform(two=t).add_gate_error(nm.amplitude_damping(g), gates="u3") for t, g in ((0.01, 0.1), (0.02, 0.3))]
    circuit = ls.parse("\n".join(lines))
    assert engine.dm_form(circuit, noise) == "ptm"
    return engine.ptm_oplist(circuit, noise)


def _work(program):
    return float(np.sum(program.pass_info()["flops_per_element"]))


def _check(nbits, precision, members, lists, graph):
    """lists: general values, special ones (zeros), general ones again."""
    with _lib.Register(nbits, precision, members) as reg:
        made, grown = _lib.Program(reg, lists[0]), _lib.Program(reg, lists[1])
        full, small = _work(made), _work(grown)
        assert small < full
        for program in (made, grown):
            for ops in (lists[1], lists[2], lists[1], lists[0], lists[1]):
                program.set_data(reg, ops)
                if graph:
                    program.graph_run(reg)
                program.run_from_basis(reg)
                got = reg.download()
                alone = _lib.Program(reg, ops)
                alone.run_from_basis(reg)
                assert np.array_equal(got, reg.download())
                alone.free()
                if program is made or ops is not lists[1]:
                    assert _work(program) == full
            assert _work(program) == full
        specialized = made.specialized
        made.free()
        grown.free()
    return specialized


@pytest.mark.parametrize("specialize", ["0", "1"])
@pytest.mark.parametrize("precision", [_lib.C128, _lib.C64])
def test_statevector_templates(precision, specialize, monkeypatch):
    monkeypatch.setenv("LSG_JIT", specialize)
    n = 8
    rng = np.random.default_rng(3)
    # (angles of either sign of the half angle's cosine)
    lists = [_template(n, rng.uniform(0.1, 6, 4 * n)), _template(n, np.zeros(4 * n)), _template(n, rng.uniform(0.1, 6, 4 * n))]
    assert _check(n, precision, 1, lists, True) == (specialize == "1")


@pytest.mark.parametrize("specialize", ["0", "1"])
def test_density_templates(specialize, monkeypatch):
    monkeypatch.setenv("LSG_JIT", specialize)
    n = 4
    rng = np.random.default_rng(4)
    angles = rng.uniform(0.1, 3, size=(2, 3, n, 3))
    plain = angles[0].copy()
    plain[:, :, 1] = 0.0  # no outer rotation; its entries not exact zeros, which would be another structure
    lists = [_density(n, angles[0]), _density(n, plain), _density(n, angles[1])]
    lists[1].chunks = [np.where((z == 0) & (g != 0), 2e-16, z) for g, z in zip(lists[0].chunks, lists[1].chunks, strict=True)]
    assert _check(2 * n, _lib.R64, 2, lists, False) == (specialize == "1")
