"""Batched kets above shared-memory size with controlled gates (one to three controls, on
bits inside and outside a tile, controlled on 0 through the shift): within 2e-5 (max-norm,
complex64) of the oracle's gates one by one."""
import numpy as np
import pytest

from oracle import oracle as orc
from tests.qpp_helpers import gaussian_ket, haar_unitary

pytestmark = pytest.mark.gpu


def test_batched_controlled_gates(ctx):
    import qpp_b200 as qb
    rng = np.random.default_rng(77)
    circuits, states, want = [], [], []
    for n in (15, 15, 16, 17):
        x = gaussian_ket(rng, 2 ** n)
        c, ref = qb.Circuit(n), x
        for k in range(40):
            nc = int(rng.integers(0, 4))
            q = [int(v) for v in rng.choice(n, size=nc + 1, replace=False)]
            U = haar_unitary(rng, 2)
            shift = [int(v) for v in rng.integers(0, 2, nc)] if k % 3 == 0 else None
            if nc:
                c.CTRL(U, q[:nc], q[nc:], shift)
                ref = orc.applyCTRL(ref, U, q[:nc], q[nc:], [2] * n, shift)
            else:
                c.gate(U, q)
                ref = orc.apply(ref, U, q, [2] * n)
        circuits.append(c)
        states.append(qb.State.from_numpy(ctx, x, [2] * n, qb.C64))
        want.append(ref)
    qb.run_batch(ctx, circuits, states, qb.FUSED)
    for s, w in zip(states, want):
        assert np.max(np.abs(s.numpy() - w)) / np.max(np.abs(w)) < 2e-5
