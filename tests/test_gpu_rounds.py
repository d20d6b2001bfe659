"""Lowered register blocks (rounds: one diagonal, then plane rotations; outer factors of one-bit
operators moved into later ones) on swizzled tiles, against a host interpreter of the operator list,
at the sizes where the tile and block shapes change: a register smaller than a tile, exactly one
tile, the first with several, and around the widths where blocks narrow.

Tolerances: every operator rounds an amplitude a few times at most (a dense 2-bit operator eight), so
N operators leave at most 8 N units of the last place of amplitudes of modulus at most 1: 90
operators give 8e-14 (complex128, unit 1.1e-16) and 4.3e-5 (complex64, unit 6e-8)."""

from __future__ import annotations

import numpy as np
import pytest

from lucivant_sim_gb300 import _lib, engine, qasm, workloads as wl
from test_host import run_oplist

pytestmark = pytest.mark.gpu

TOL = {_lib.C128: 8e-14, _lib.C64: 4.3e-5}


def _unitary(rng, d):
    return np.linalg.qr(rng.normal(size=(d, d)) + 1j * rng.normal(size=(d, d)))[0]


def _ops(rng, nbits, members, count=90):
    """One-bit unitaries (some a cosine or a sine away from a permutation), renames, permutations with
    phases, diagonals, wider matrices and matrices that are not unitary, some per member."""
    ops = _lib.OpList()
    for i in range(count):
        pick = rng.integers(0, 12)
        k = 1 if pick < 6 else 2 if pick < 11 else min(3, nbits)
        bits = [int(b) for b in rng.choice(nbits, size=min(k, nbits), replace=False)]
        d = 1 << len(bits)
        if pick == 0:  # next to a permutation: cosine of 1e-9 and 1e-17
            t = np.pi - 2 * (1e-9 if i % 2 else 1e-17)
            mats = [np.array([[np.cos(t / 2), -np.sin(t / 2)], [np.sin(t / 2), np.cos(t / 2)]]) * np.exp(1j * rng.uniform(0, 6))]
        elif pick == 1:  # not unitary: stays dense
            mats = [0.6 * _unitary(rng, d) + 0.3 * _unitary(rng, d)]
        elif pick in (7, 8):
            ops.add(_lib.OP_PERM, bits, np.array([1, 1, 1, 1, 0, 1, 3, 2], dtype=complex) if d == 4 else
                    np.array([1, 1, 1, 0], dtype=complex))
            continue
        elif pick == 9:
            ops.add(_lib.OP_PERM, bits, np.concatenate([np.exp(1j * rng.uniform(0, 6, size=d)), rng.permutation(d)]))
            continue
        elif pick == 10:
            ops.add(_lib.OP_DIAG, bits, np.exp(1j * rng.uniform(0, 6, size=d)))
            continue
        else:
            mats = [_unitary(rng, d) for _ in range(members if i % 3 == 0 else 1)]
        if len(mats) == 1:
            ops.add(_lib.OP_MATRIX, bits, mats[0])
        else:
            ops.add_batched(_lib.OP_MATRIX, bits, np.stack(mats))
    return ops


@pytest.mark.parametrize("precision", [_lib.C128, _lib.C64])
@pytest.mark.parametrize("nbits,members", [(1, 1), (3, 2), (5, 1), (6, 3), (9, 2), (10, 1), (11, 2), (12, 1), (13, 3), (15, 1)])
def test_random_programs_match_the_operator_list(precision, nbits, members):
    rng = np.random.default_rng(1000 * nbits + members)
    ops = _ops(rng, nbits, members)
    start = rng.normal(size=(members, 1 << nbits)) + 1j * rng.normal(size=(members, 1 << nbits))
    start /= np.linalg.norm(start, axis=1, keepdims=True)
    with _lib.Register(nbits, precision, members) as reg:
        reg.upload(start)
        reg.apply(ops)
        got = reg.download()
    for b in range(members):
        want = run_oplist(ops, nbits, start[b], member=b)
        assert np.max(np.abs(got[b] - want)) < TOL[precision], (b, np.max(np.abs(got[b] - want)))


@pytest.mark.parametrize("precision", [_lib.C128, _lib.C64])
def test_members_get_the_arithmetic_they_get_alone(precision):
    """Members whose rotations exchange rows or need no diagonal where others do: bit for bit the
    register each has by itself."""
    n, members = 9, 4
    rng = np.random.default_rng(5)
    template = wl.hea_template(n, 3)
    values = rng.uniform(0, 2 * np.pi, size=(members, 2 * n * 3))
    values[1, ::4] = 0.0  # identities
    values[2, ::6] = np.pi  # half turns
    circuits = [qasm.parse(template, {f"p{k}": float(v) for k, v in enumerate(row)}) for row in values]
    lists = [engine.fuse_runs(c.operations) for c in circuits]
    both = _lib.OpList()
    alone = [_lib.OpList() for _ in range(members)]
    for position in zip(*lists, strict=True):
        mats = [np.asarray(op.matrix, dtype=complex) for op in position]
        bits = list(position[0].qubits)
        if len(bits) == 2:
            for o in [both, *alone]:
                o.add(*engine.classify(mats[0])[:1], bits, engine.classify(mats[0])[1])
            continue
        both.add_batched(_lib.OP_MATRIX, bits, np.stack(mats))
        for o, m in zip(alone, mats, strict=True):
            o.add(_lib.OP_MATRIX, bits, m)
    with _lib.Register(n, precision, members) as reg:
        reg.apply_from_basis(both)
        got = reg.download()
    for b in range(members):
        with _lib.Register(n, precision) as reg:
            reg.apply_from_basis(alone[b])
            assert np.array_equal(got[b], reg.download()[0]), b


@pytest.mark.parametrize("precision", [_lib.C128, _lib.C64])
def test_template_data_that_lowers_to_other_blocks(precision):
    """New template data may need diagonals that the first set did not (and the other way): taken,
    with the register a program made for it leaves, plain and as a graph."""
    n = 7
    template = wl.hea_template(n, 2)
    sets = [np.zeros(28), np.random.default_rng(3).uniform(0.1, 6, 28), np.zeros(28)]
    sets[2][::2] = 0.7  # rotations about Y alone
    lists = []
    for values in sets:
        ops = _lib.OpList()
        for op in engine.fuse_runs(qasm.parse(template, {f"p{k}": float(v) for k, v in enumerate(values)}).operations):
            m = np.asarray(op.matrix, dtype=complex)
            ops.add(*((_lib.OP_MATRIX, list(op.qubits), m) if len(op.qubits) == 1 else
                      (engine.classify(m)[0], list(op.qubits), engine.classify(m)[1])))
        lists.append(ops)
    with _lib.Register(n, precision) as reg:
        prog = _lib.Program(reg, lists[0])
        got = []
        for ops in [*lists, lists[1]]:
            prog.set_data(reg, ops)
            for _ in range(2):
                prog.graph_run(reg)
            reg.sync()
            got.append(reg.download()[0])
        prog.free()
    for ops, g in zip([*lists, lists[1]], got, strict=True):
        with _lib.Register(n, precision) as reg:
            reg.apply_from_basis(ops)
            assert np.array_equal(g, reg.download()[0])
