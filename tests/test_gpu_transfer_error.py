"""The error of real64 transfer operators run as shears beside that of their dense products, against the same
operators applied in extended precision.

Bound: a dense row rounds three times; the shears round twice per pair map and once in the diagonal, on
coefficients that are each rounded once, which adds about a tenth to the products' error. 1.5 leaves
room for six circuits' spread. (Coefficients formed in double precision give 1.9.)"""

from __future__ import annotations

import numpy as np
import pytest

import lucivant_sim_gb300 as ls
from lucivant_sim_gb300 import _lib, engine, workloads as wl

pytestmark = pytest.mark.gpu


def _extended(ops, nbits, member):
    pool = np.concatenate(ops.chunks).real.astype(np.longdouble)
    v = np.zeros(1 << nbits, dtype=np.longdouble)
    v[: 1 << (nbits // 2)] = 1  # |0...0>
    for kind, k, bits, at, stride in ops.rows:
        at += member * stride
        d = 1 << k
        axes = [nbits - 1 - b for b in bits]
        t = np.moveaxis(v.reshape((2,) * nbits), axes, range(k)).reshape(d, -1)
        if kind == _lib.OP_MATRIX:
            t = pool[at : at + d * d].reshape(d, d) @ t
        elif kind == _lib.OP_DIAG:
            t = pool[at : at + d, None] * t
        else:
            assert kind == _lib.OP_PERM
            t = pool[at : at + d, None] * t[pool[at + d : at + 2 * d].astype(int)]
        v = np.moveaxis(t.reshape((2,) * nbits), range(k), axes).reshape(-1)
    return v


def _rms(values):
    return float(np.sqrt(np.mean(np.square(values))))


@pytest.mark.parametrize("n,layers", [(4, 20), (5, 12)])
def test_shears_are_as_accurate_as_products(n, layers, monkeypatch):
    errors = {"0": [], "1": []}
    noises = [ls.NoiseModel.uniform(two=t).add_gate_error(wl.thermal_depolarizing(s), gates="u3") for s, t in ((1e-3, 1e-2), (4e-3, 2e-2))]
    for seed in range(6):
        ops = engine.ptm_oplist(ls.parse(wl.brickwork(n, layers, seed=seed, measure=False)), noises)
        want = [_extended(ops, 2 * n, m) for m in range(2)]
        for fuse, found in errors.items():
            monkeypatch.setenv("LSG_FUSE_BLOCKS", fuse)
            with _lib.Register(2 * n, _lib.R64, 2) as reg:
                reg.apply_from_basis(ops)
                got = reg.download()
            for m in range(2):
                found.append(float(np.linalg.norm((got[m].real - want[m]).astype(float)) / np.linalg.norm(want[m].astype(float))))
    assert _rms(errors["1"]) < 1.5 * _rms(errors["0"]), errors
