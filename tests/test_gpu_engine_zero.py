"""A run of measurements that meets a ket without weight fails as single measurements do:
the same error, the generator where the failing step's draw left it, and the state and
its qudits as they were, so that the engine goes on with another state."""
import numpy as np
import pytest

from tests.qpp_helpers import gaussian_ket

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("destructive", [False, True])
@pytest.mark.parametrize("prec", ["C128", "C64"])
def test_zero_ket_in_a_run_of_measurements(ctx, destructive, prec):
    import qpp_b200 as qb
    n = 4
    prec = getattr(qb, prec)
    zero = qb.State.from_numpy(ctx, np.zeros(2 ** n, dtype=np.complex128), [2] * n, prec)
    good = qb.State.from_numpy(ctx, gaussian_ket(np.random.default_rng(1), 2 ** n), [2] * n, prec)
    outcomes = []
    for single in (False, True):
        c = qb.Circuit(n, 2, n)
        for t in ([2, 0], [1], [3]):
            c.measure(t, t[0], destructive=destructive)
            if single:  # a gate ends the run
                left = [q for q in range(n) if q not in (2, 0, *(() if t == [2, 0] else (1,)))]
                if not destructive or t != [3]:
                    c.gate(np.eye(2), [left[-1]])
        e = qb.Engine(ctx, c, qb.KET, prec).set_seed(9)
        e.set_state(zero)
        with pytest.raises(qb.QppError) as err:
            e.execute()
        assert err.value.what == "zero probability"
        assert e.get_state().dims == [2] * n
        got = []
        for _ in range(6):
            e.set_state(good)
            e.execute()
            got.append(e.get_dits()[0])
            e.reset()
        outcomes.append(got)
    assert outcomes[0] == outcomes[1]
