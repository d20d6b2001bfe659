"""Collapsed amplitudes of a complex128 trajectory are the quotients by the norm, bit for bit: amplitudes of
few bits, whose squares' sum is exact in any order, over many magnitudes down to subnormal numbers,
with zeros of either sign."""

from __future__ import annotations

from types import SimpleNamespace

import numpy as np
import pytest

from lucivant_sim_gb300 import _lib
from lucivant_sim_gb300.trajectories import TrajectoryProgram

pytestmark = pytest.mark.gpu

N = 6


def _state(ops, uniform):
    circuit = SimpleNamespace(num_qubits=N, num_clbits=1, operations=ops)
    program = TrajectoryProgram(circuit, None, _lib.C128, 1)
    try:
        rows, _, _ = program.run_serial(1, np.full(max(program.max_draws, 1), uniform))
        return program.reg.download()[0], int(rows[0, 0])
    finally:
        program.free()


@pytest.mark.parametrize("small", [-3, -40, -300, -510, -530, -1000, -1060])
@pytest.mark.parametrize("seed", range(4))
def test_quotients_are_exact(seed, small):
    rng = np.random.default_rng([seed, -small])
    ops = []
    for q in range(N):
        m = (rng.integers(-3, 4, size=(2, 2)) + 1j * rng.integers(-3, 4, size=(2, 2))) / 8.0
        m[:, 0] += np.where(m[:, 0] == 0, 0.25, 0.0)  # the column that acts on |0>
        if q == 1:  # half of the amplitudes far below the others, their squares below the sum's last bit
            m[1] *= 2.0**small
        if q == 2:
            m[1, 0] = -m[1, 0].real  # zeros of both signs among the products
        ops.append(SimpleNamespace(kind="gate", name="g", matrix=m, qubits=[q]))
    before, _ = _state(ops, 0.5)
    index = np.arange(1 << N)
    for uniform, want in ((0.0, 1), (1.0 - 2.0**-53, 0)):
        got, bit = _state([*ops, SimpleNamespace(kind="measure", qubit=0, clbit=0)], uniform)
        assert bit == want
        p1 = float(np.sum(np.abs(before[(index & 1) == 1].real) ** 2 + np.abs(before[(index & 1) == 1].imag) ** 2))
        kept = np.where((index & 1) == want, before, 0.0)
        expected = (kept.view(float) / np.sqrt(p1 if want else 1.0 - p1))
        assert np.array_equal(got.view(float), expected)
        chosen = np.repeat((index & 1) == want, 2)
        assert np.array_equal(np.signbit(got.view(float)[chosen]), np.signbit(expected[chosen]))
