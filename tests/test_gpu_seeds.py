"""Seeded complex64 outcomes stay what they were: sampled indices depend on the last
bits of the amplitudes, so the paths behind them keep their arithmetic. The hashes are
of the outcomes since engines run QFT blocks as transforms, and since the server fuses
density matrices (other roundings move up to a few draws in a hundred)."""
import hashlib

import numpy as np
import pytest

from tests.qpp_helpers import haar_unitary

pytestmark = pytest.mark.gpu


def digest(a):
    return hashlib.sha256(np.ascontiguousarray(a, dtype=np.int64).tobytes()).hexdigest()[:16]


def engine_outcomes(ctx, n, shots):
    import qpp_b200 as qb
    rng = np.random.default_rng(n)
    c = qb.Circuit(n, 2, n)
    for q in range(n):
        c.gate(haar_unitary(rng, 2), [q])
    for q in range(n - 1):
        c.gate(haar_unitary(rng, 4), [q, q + 1])
    c.QFT()
    for q in range(n):
        c.gate(haar_unitary(rng, 2), [q])
    for q in range(n):
        c.measure([q], q, destructive=False)
    e = qb.Engine(ctx, c, qb.KET, qb.C64)
    e.set_seed(3).reset().execute(shots)
    return np.array([list(k) + [v] for k, v in sorted(e.get_stats().items())])


def server_samples(n, shots):
    import qpp_b200 as qb
    from qpp_b200 import serving
    rng = np.random.default_rng(n)
    c = qb.Circuit(n, 2, 1)
    for _ in range(4):
        for q in range(n):
            c.gate(haar_unitary(rng, 2), [q])
        perm = [int(x) for x in rng.permutation(n)]
        for i in range(n // 2):
            t = [perm[2 * i], perm[2 * i + 1]]
            c.gate(haar_unitary(rng, 4), t)
            serving.c_channel(c, serving.pair_channel(), t)
    srv = serving.Server(0)
    try:
        rid = srv.submit(c, qb.RHO, 0.0, shots, 5)
        return srv.wait(rid, shots=shots, nc=1)[1]
    finally:
        srv.close()


def test_engine_qft_outcomes(ctx):
    assert digest(engine_outcomes(ctx, 22, 5000)) == "4218b43186320eac"


def test_server_density_matrix_samples(ctx):
    assert digest(server_samples(12, 200000)) == "a2e074d1d8be8611"
