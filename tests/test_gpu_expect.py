"""Pauli expectations of statevector registers against a host computation from the register's own
amplitudes: registers of one amplitude pair up to several blocks of partial sums, strings whose X part
ends at qubit 0 (its pair shares one 16-byte word) and elsewhere, more terms than travel with the
launch, members, and states whose norm is not one.

Tolerances: a sum of 2^n products of squared norm N, complex128 within 2^n * 2 units of 1.1e-16 of N
at the most (2^14: 4e-12, and far less for the tree), complex64 summands in FP32: 8 roundings of 6e-8
per summand, so 5e-7 of N, and 1e-6 of N for a state whose own norm is divided out."""

from __future__ import annotations

import numpy as np
import pytest

from lucivant_sim_gb300 import _lib, engine, qasm, workloads as wl

pytestmark = pytest.mark.gpu


def _want(v, x, z):
    idx = np.arange(v.size)
    sign = 1.0 - 2.0 * np.array([bin(i & z).count("1") & 1 for i in range(v.size)])
    return float(np.real(1j ** bin(x & z).count("1") * np.sum(np.conj(v[idx ^ x]) * v * sign)))


def _terms(rng, n, count):
    top = (1 << n) - 1
    xs = [0, 1 & top, top, 1 << (n - 1), 2 & top] + [int(v) for v in rng.integers(0, top + 1, size=count)]
    zs = [top, 1 & top, 0, top, 1 & top] + [int(v) for v in rng.integers(0, top + 1, size=count)]
    return xs[:count], zs[:count]


@pytest.mark.parametrize("precision,tol", [(_lib.C128, 4e-12), (_lib.C64, 5e-7)])
@pytest.mark.parametrize("n,members,count", [(1, 1, 4), (2, 3, 5), (3, 1, 70), (9, 2, 12), (12, 1, 64), (13, 3, 66), (14, 1, 5)])
def test_uploaded_states(precision, tol, n, members, count):
    rng = np.random.default_rng(100 * n + count)
    v = rng.normal(size=(members, 1 << n)) + 1j * rng.normal(size=(members, 1 << n))
    xs, zs = _terms(rng, n, count)
    with _lib.Register(n, precision, members) as reg:
        reg.upload(v)
        got = reg.expect(0, xs, zs)
        held = reg.download()
    for b in range(members):
        scale = float(np.sum(np.abs(held[b]) ** 2))  # far from one: not divided out
        for t, (x, z) in enumerate(zip(xs, zs, strict=True)):
            assert abs(got[t, b] - _want(held[b], x, z)) < tol * scale, (b, t)


@pytest.mark.parametrize("members", [1, 3])
def test_complex64_states_of_unitary_circuits_have_norm_one(members):
    """The identity's expectation is one; an operator that is not unitary, or an upload, gives the sum
    as it is again."""
    n = 10
    ops = engine.sv_oplist(qasm.parse(wl.brickwork(n, 6, seed=3, measure=False)))
    half = _lib.OpList()
    half.add(_lib.OP_MATRIX, [4], np.diag([0.5, 0.5]) + 0.1 * np.array([[0, 1], [1, 0]]))
    with _lib.Register(n, _lib.C64, members) as reg:
        reg.apply_from_basis(ops)
        assert np.array_equal(reg.expect(0, [0], [0]), np.ones((1, members)))
        held = reg.download()
        got = reg.expect(0, [3, 1], [5, 1 << 7])
        for b in range(members):
            for t, (x, z) in enumerate([(3, 5), (1, 1 << 7)]):
                assert abs(got[t, b] - _want(held[b], x, z) / np.sum(np.abs(held[b]) ** 2)) < 1e-6
        reg.apply(half)
        norm = np.sum(np.abs(reg.download()) ** 2, axis=1)
        assert np.all(np.abs(reg.expect(0, [0], [0])[0] - norm) < 5e-7)
        assert np.all(norm < 0.5)
