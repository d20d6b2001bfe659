"""What a complex64 statevector's expectations are divided by depends on its amplitudes alone: the same
values for the state a circuit left, for the same amplitudes uploaded, for the entry point that takes
device pointers, and for a member beside one whose norm is its own.

Tolerance: the same FP32 summands in another order of FP64 sums (2^13 of them: below 1e-12); the norm of
the states here drifts by more than 1e-7, so a missing or a spare division shows."""

from __future__ import annotations

import numpy as np
import pytest

from lucivant_sim_gb300 import _lib, engine, qasm, workloads as wl
from test_zz_no_alloc import _noalloc, _terms

pytestmark = pytest.mark.gpu

N = 13


def _circuit():
    return engine.sv_oplist(qasm.parse(wl.brickwork(N, 60, seed=1, measure=False)))


def _evolved(reg, scale=()):
    reg.apply_from_basis(_circuit())
    if scale:
        ops = _lib.OpList()
        ops.add_batched(_lib.OP_MATRIX, [3], np.stack([np.eye(2) * s for s in scale]))
        reg.apply(ops)
    return reg.download()


def test_an_uploaded_state_gives_what_the_circuit_gave():
    xs, zs = _terms(N, 3, 9)
    with _lib.Register(N, _lib.C64) as made, _lib.Register(N, _lib.C64) as given:
        held = _evolved(made)
        assert abs(np.sum(np.abs(held) ** 2) - 1) > 1e-7
        given.upload(held)
        assert np.array_equal(given.download(), held)
        assert np.array_equal(made.expect(0, xs, zs), given.expect(0, xs, zs))


def test_the_pointer_entry_point_divides_alike():
    torch = pytest.importorskip("torch")
    xs, zs = _terms(N, 4, 11)
    scale = (1.0, 0.5, 1.0 + 1e-4)
    with _lib.Register(N, _lib.C64, 3) as reg:
        amps = torch.from_numpy(_evolved(reg, scale).reshape(-1).astype(np.complex64)).to("cuda")
        want = reg.expect(0, [0, *xs], [0, *zs])
        out = torch.zeros(12 * 3, dtype=torch.float64, device="cuda")
        stream = torch.cuda.current_stream().cuda_stream
        assert _noalloc(_lib.library(), amps.data_ptr(), _lib.C64, N, 3, 0, [0, *xs], [0, *zs], out.data_ptr(), stream) == 0
        assert np.max(np.abs(out.cpu().numpy().reshape(12, 3) - want)) < 1e-12
    assert want[0, 0] == 1.0
    assert abs(want[0, 1] - 0.25) < 1e-6 and abs(want[0, 2] - 1.0002) < 1e-5


def test_a_member_beside_one_of_another_norm():
    xs, zs = _terms(N, 5, 8)
    with _lib.Register(N, _lib.C64, 2) as both, _lib.Register(N, _lib.C64) as one:
        _evolved(both, (1.0, 0.5))
        _evolved(one)
        got, alone = both.expect(0, xs, zs), one.expect(0, xs, zs)
    assert np.max(np.abs(got[:, 0] - alone[:, 0])) < 1e-12
