"""Members of a batch whose operators are products of many gates: lowered like single gates, bit for bit the
register each has by itself."""

from __future__ import annotations

import numpy as np
import pytest

from lucivant_sim_gb300 import _lib, engine, gates

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [_lib.C128, _lib.C64])
def test_members_of_long_gate_products_get_the_arithmetic_they_get_alone(precision):
    n, members = 8, 3
    rng = np.random.default_rng(11)
    both = _lib.OpList()
    alone = [_lib.OpList() for _ in range(members)]
    cx = np.array([[1, 0, 0, 0], [0, 1, 0, 0], [0, 0, 0, 1], [0, 0, 1, 0]], dtype=complex)
    for layer in range(6):
        for q in range(n):
            mats = []
            for length in (1, 2000, 50):
                m = np.eye(2, dtype=complex)
                for t, p, lam in rng.uniform(0, 2 * np.pi, size=(length, 3)):
                    m = gates.u3(t, p, lam) @ m
                mats.append(m)
            both.add_batched(_lib.OP_MATRIX, [q], np.stack(mats))
            for o, m in zip(alone, mats, strict=True):
                o.add(_lib.OP_MATRIX, [q], m)
        for a in range(layer % 2, n - 1, 2):
            for o in [both, *alone]:
                o.add(*engine.classify(cx)[:1], [a, a + 1], engine.classify(cx)[1])
    with _lib.Register(n, precision, members) as reg:
        reg.apply_from_basis(both)
        got = reg.download()
    for b in range(members):
        with _lib.Register(n, precision) as reg:
            reg.apply_from_basis(alone[b])
            assert np.array_equal(got[b], reg.download()[0]), b
