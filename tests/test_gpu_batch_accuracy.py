"""Batched density matrices are as exact as one at a time: their mean distance from the
plain complex128 run stays within 1% of that of the fused complex64 form, which merges
the same blocks in 64 bits (other sums of the same products move it by a few parts in ten
thousand; products of narrower blocks left to 32 bits by 2 to 10%)."""
import numpy as np
import pytest

from tests.qpp_helpers import depolarizing_kraus, haar_unitary, random_rho

pytestmark = pytest.mark.gpu


def distance(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("n", [9, 10])
def test_batched_density_matrices_are_as_exact_as_single_ones(ctx, n):
    import qpp_b200 as qb
    from qpp_b200.serving import c_channel
    rng = np.random.default_rng(n)
    chan = depolarizing_kraus(0.005)
    circuits, states, single, want = [], [], [], []
    for _ in range(6):
        c = qb.Circuit(n)
        for _ in range(12):
            for q in range(n):
                c.gate(haar_unitary(rng, 2), [q])
            perm = [int(x) for x in rng.permutation(n)]
            for i in range(n // 2):
                c.gate(haar_unitary(rng, 4), [perm[2 * i], perm[2 * i + 1]])
            for q in range(n):
                c_channel(c, chan, [q])
        x = random_rho(rng, 2 ** n, 4)
        circuits.append(c)
        states.append(qb.State.from_numpy(ctx, x, [2] * n, qb.C64))
        one = states[-1].clone()
        exact = qb.State.from_numpy(ctx, states[-1].numpy(), [2] * n)
        c.run(one, qb.FUSED)
        c.run(exact, qb.PLAIN)
        single.append(distance(one.numpy(), exact.numpy()))
        want.append(exact.numpy())
    qb.run_batch(ctx, circuits, states, qb.FUSED)
    batched = [distance(s.numpy(), w) for s, w in zip(states, want)]
    assert np.mean(batched) <= 1.01 * np.mean(single)
