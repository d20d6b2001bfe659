"""Passes that start under the tail of the kernel before them: many runs enqueued back to back, with no
wait between, leave the state that one run with waits leaves, bit for bit, over registers of one tile,
of fewer tiles than SMs and of more than sixteen tiles a block; so do replays of a captured graph, and two
registers on streams of their own."""

from __future__ import annotations

import numpy as np
import pytest

from lucivant_sim_gb300 import _lib, engine, qasm, workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [_lib.C64, _lib.C128])
@pytest.mark.parametrize("n,batch", [(5, 1), (13, 1), (13, 40), (17, 3), (20, 1), (21, 16)])
def test_back_to_back_runs_equal_one(n, batch, precision, monkeypatch):
    monkeypatch.setenv("LSG_JIT", "0")
    ops = engine.sv_oplist(qasm.parse(wl.brickwork(n, 9, seed=n, measure=False)))
    with _lib.Register(n, precision, batch) as a, _lib.Register(n, precision, batch) as b:
        prog = _lib.Program(a, ops)
        other = _lib.Program(b, ops)
        try:
            prog.run_from_basis(a, 0)
            a.sync()
            want = a.download()[0]
            for _ in range(25):
                prog.run_from_basis(a, 0)
                other.run_from_basis(b, 0)
            a.sync()
            b.sync()
            for got in (a.download(), b.download()):
                assert all(np.array_equal(member, want) for member in got)
            for _ in range(6):
                prog.graph_run(a, 0)
            a.sync()
            assert all(np.array_equal(member, want) for member in a.download())
        finally:
            prog.free()
            other.free()
