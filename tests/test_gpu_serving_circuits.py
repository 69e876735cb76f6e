"""The server runs the circuit it is given: steps added between two requests, and
circuits made and freed one after the other (whose addresses repeat)."""
import numpy as np
import pytest

from tests.qpp_helpers import X

pytestmark = pytest.mark.gpu


def final_index(srv, qb, c, kind):
    _, samples, _ = srv.wait(srv.submit(c, kind, 0.0, 3, 1), shots=3, nc=1)
    assert len(set(samples.tolist())) == 1
    return int(samples[0])


@pytest.mark.parametrize("kind,n", [(0, 3), (1, 3), (1, 8)])
def test_requests_run_the_circuit_as_it_is(ctx, kind, n):
    import qpp_b200 as qb
    from qpp_b200 import serving
    kind = (qb.KET, qb.RHO)[kind]
    srv = serving.Server(0)
    try:
        c = qb.Circuit(n, 2, 1)
        want = 0
        for q in range(n):
            c.gate(X, [q])
            want |= 1 << (n - 1 - q)
            assert final_index(srv, qb, c, kind) == want
        for q in range(4 * n):
            c = qb.Circuit(n, 2, 1)
            c.gate(X, [q % n])
            assert final_index(srv, qb, c, kind) == 1 << (n - 1 - q % n)
            del c
    finally:
        srv.close()
