"""The error of lowered complex128 blocks (rounds) beside that of dense products of the same gates, against
the gates' matrices applied in extended precision.

Bound: a dense 2x2 complex product rounds an amplitude eight times, about 0.66 units of 1.1e-16 (rms) in
all; a gate's share of a round is fewer operations, about 0.5 units, and one rounding of each of its
coefficients, which is common to all amplitudes and of the same size as the gate matrix's own, 0.66. Per
gate that is 1.25 of the dense product's; 1.6 leaves room for six seeds' spread. (Coefficients formed
in double precision, some twenty roundings each, give 2.4.)"""

from __future__ import annotations

import numpy as np
import pytest

from lucivant_sim_gb300 import _lib, engine, qasm, workloads as wl

pytestmark = pytest.mark.gpu


def _extended(circuit):
    n = circuit.num_qubits
    psi = np.zeros(1 << n, dtype=np.clongdouble)
    psi[0] = 1
    index = np.arange(1 << n)
    for op in circuit.operations:
        if op.name == "cx":
            control, target = op.qubits
            psi = psi[np.where((index >> control) & 1, index ^ (1 << target), index)]
            continue
        m = np.asarray(op.matrix).astype(np.clongdouble)
        v = psi.reshape(-1, 2, 1 << op.qubits[0])
        psi = np.stack([m[0, 0] * v[:, 0] + m[0, 1] * v[:, 1], m[1, 0] * v[:, 0] + m[1, 1] * v[:, 1]], axis=1).reshape(-1)
    return psi


def _rms(values):
    return float(np.sqrt(np.mean(np.square(values))))


@pytest.mark.parametrize("n,layers", [(9, 20), (11, 20), (13, 8)])
def test_rounds_are_as_accurate_as_dense_products(n, layers, monkeypatch):
    errors = {"0": [], "1": []}
    for seed in range(6):
        circuit = qasm.parse(wl.brickwork(n, layers, seed=seed, measure=False))
        want = _extended(circuit)
        for fuse, found in errors.items():
            monkeypatch.setenv("LSG_FUSE_BLOCKS", fuse)
            with _lib.Register(n, _lib.C128) as reg:
                reg.apply_from_basis(engine.sv_oplist(circuit))
                found.append(np.linalg.norm(np.abs(reg.download()[0] - want).astype(float)))
    assert _rms(errors["1"]) < 1.6 * _rms(errors["0"]), errors
