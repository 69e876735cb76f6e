"""Runs of an engine's steps on a ket: measurements drawn and collapsed on the
device one after the other, gates between them as register tile passes. The
reference is the same engine step by step: with the identity as noise and the
recorded outcomes replayed, every step takes the general path. The sizes have
fewer amplitudes than a block, several per chunk with a ragged last one (3^9,
2^19), dimensions that are no power of two, destructive steps in between, and
the 7-bit edge of the smallest tile."""
import numpy as np
import pytest

from tests.qpp_helpers import gaussian_ket, haar_unitary

pytestmark = pytest.mark.gpu


def circuit(qb, n, d, rng, destructive):
    c = qb.Circuit(n, d, n + 2)
    one = lambda: haar_unitary(rng, d)
    for q in range(n):
        c.gate(one(), [q])
    for q in range(0, n - 1, 2):
        c.gate(haar_unitary(rng, d * d), [q, q + 1])
    c.measure([n - 1, 0], 0, destructive=destructive)
    c.measure([n // 2], 2, destructive=False)
    left = [q for q in range(n) if not (destructive and q in (0, n - 1))]
    for q in left:
        c.gate(one(), [q])
    if len(left) > 1:
        c.CTRL(one(), [left[0]], [left[-1]])
        c.gate(haar_unitary(rng, d * d), [left[-1], left[0]])
    for i, q in enumerate(left):
        c.measure([q], 2 + i, destructive=destructive and i % 2 == 0)
    return c


@pytest.mark.parametrize("n,d,prec", [(3, 2, "c128"), (7, 2, "c128"), (8, 2, "c64"), (13, 2, "c128"),
                                      (19, 2, "c128"), (9, 3, "c128"), (3, 6, "c64")])
@pytest.mark.parametrize("destructive", [False, True])
def test_runs_match_single_steps(ctx, n, d, prec, destructive):
    import qpp_b200 as qb
    p = qb.C128 if prec == "c128" else qb.C64
    # rounding of ~60 gates and 20 renormalisations: sums of up to 2^19 terms in
    # 64 bits, amplitudes at the state's type
    tol = 1e-12 if prec == "c128" else 2e-5
    rng = np.random.default_rng([n, d, destructive])
    c = circuit(qb, n, d, rng, destructive)
    psi = qb.State.from_numpy(ctx, gaussian_ket(rng, d ** n), [d] * n, prec=p)
    for seed in range(3):
        a = qb.Engine(ctx, c, qb.KET, p).set_seed(seed).set_state(psi).execute()
        outs, _ = a.get_record()
        b = qb.Engine(ctx, c, qb.KET, p).set_noise([np.eye(d)], [1.0]).set_state(psi)
        b.set_replay(outs, [0] * (4 * n * n + 40)).execute()
        assert a.get_dits()[0] == b.get_dits()[0]
        np.testing.assert_allclose(a.get_dits()[1], b.get_dits()[1], rtol=0, atol=tol)
        np.testing.assert_allclose(a.get_state().numpy(), b.get_state().numpy(), rtol=0, atol=tol)


def test_draws_are_those_of_single_steps(ctx):
    """The same generator gives the same outcomes as one measurement at a time
    (an engine whose circuit ends after each of them), also from a state whose
    weight lies in its last chunk only."""
    import qpp_b200 as qb
    n = 17
    rng = np.random.default_rng(5)
    psi = gaussian_ket(rng, 2 ** n)
    tail = np.zeros_like(psi)
    tail[-40:] = psi[-40:]
    for x in (psi, tail):
        x = x / np.linalg.norm(x)
        for seed in range(4):
            c = qb.Circuit(n, 2, n)
            for q in range(n):
                c.measure([q], q, destructive=False)
            s = qb.State.from_numpy(ctx, x, [2] * n)
            e = qb.Engine(ctx, c).set_seed(seed).set_state(s).execute()
            # qpp: the first draw fixes the basis state, the later ones repeat it
            c1 = qb.Circuit(n, 2, n).measure(list(range(n)), 0, destructive=False)
            one = qb.Engine(ctx, c1).set_seed(seed).set_state(s)
            got = e.get_dits()[0]
            assert got[0] == one.execute().get_dits()[0][0]
            index = int("".join(map(str, got)), 2)
            assert abs(x[index]) > 0
            np.testing.assert_allclose(np.prod(e.get_dits()[1]), abs(x[index]) ** 2, rtol=1e-10)


