"""Trajectories that measure and reset qubits whose value is known already (measured, and untouched
since), on the main line and under conditions, against the oracle: identical counts for the same seed
shot by shot, and batched counts against the exact outcome distribution."""

from __future__ import annotations

import numpy as np
import pytest
from scipy import stats

import lucivant_sim_gb300 as ls
from oracle import dense

pytestmark = pytest.mark.gpu

HEAD = 'OPENQASM 3.0; include "stdgates.inc"; qubit[{n}] q; bit[4] c; bit[4] d;\n'
# a reset and a second measurement of measured qubits; a diagonal between them; a qubit touched again;
# a branch that resets or flips a measured qubit; a qubit never touched
BODY = """
ry(0.7) q[0]; ry(1.1) q[1]; ry(2.0) q[2]; cx q[0], q[3]; cx q[1], q[4];
d[3] = measure q[{last}];
c[0] = measure q[0]; c[1] = measure q[1]; c[2] = measure q[2];
rz(0.4) q[1];
d[0] = measure q[1];
if (c[2] == 1) {{ reset q[2]; x q[3]; }}
d[1] = measure q[2];
reset q[0]; reset q[1];
ry(0.9) q[1];
d[2] = measure q[1];
if (c[0] == 1) x q[1];
reset q[1];
c[3] = measure q[3];
"""


def _source(n):
    return HEAD.format(n=n) + BODY.format(last=n - 1)


def _noise():
    return ls.NoiseModel.uniform(single=2e-2, two=5e-2, readout=3e-2)


@pytest.mark.parametrize("noise", [None, _noise()], ids=["ideal", "noisy"])
@pytest.mark.parametrize("n", [5, 6, 12, 13])
def test_serial_counts_are_the_oracles(n, noise):
    circuit = ls.parse(_source(n))
    shots = 300 if n < 10 else 60
    result = ls.run(circuit, shots=shots, seed=11, noise=noise, method="trajectories")
    want, _, _ = dense.run_counts(circuit, shots, 11, noise)
    assert result.counts == want or result.report["near_threshold"] > 0


@pytest.mark.parametrize("precision", ["c128", "c64"])
def test_batched_counts_follow_the_exact_distribution(precision):
    circuit = ls.parse(_source(6))
    noise = _noise()
    shots = 20000
    result = ls.run(circuit, shots=shots, seed=5, noise=noise, method="trajectories", trajectory_mode="batched",
                    precision=precision)
    exact = dense.exact_outcomes(circuit, noise)
    keys = [k for k, p in exact.items() if p * shots >= 5]
    from lucivant_sim_gb300.circuit import format_bits

    seen = np.array([result.counts.get(format_bits(circuit, k), 0) for k in keys], dtype=float)
    want = np.array([exact[k] for k in keys]) * shots
    rest_seen, rest_want = shots - seen.sum(), shots - want.sum()
    if rest_want > 5:
        seen, want = np.append(seen, rest_seen), np.append(want, rest_want)
    else:
        want *= seen.sum() / want.sum()
    assert stats.chisquare(seen, want).pvalue > 1e-6
