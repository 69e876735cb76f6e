"""Gate runs captured into a CUDA graph: the graph keeps its own copy of the tile
programs, so it gives the circuit's result at every launch, also after the circuit has
grown, been planned again and been freed."""
import numpy as np
import pytest

from tests.qpp_helpers import gaussian_ket, haar_unitary

pytestmark = pytest.mark.gpu


def circuit(qb, rng, n):
    c = qb.Circuit(n)
    for _ in range(200):
        k = 1 if rng.random() < 0.6 else 2
        c.gate(haar_unitary(rng, 2 ** k), [int(x) for x in rng.choice(n, size=k, replace=False)])
    return c


@pytest.mark.parametrize("prec,form", [("C128", "PLAIN"), ("C128", "FUSED"), ("C64", "PLAIN")])
@pytest.mark.parametrize("planned", [False, True])
def test_captured_gate_runs_keep_their_programs(ctx, prec, form, planned):
    import qpp_b200 as qb
    rt = pytest.importorskip("cuda.bindings.runtime")

    def ok(r):
        assert r[0] == rt.cudaError_t.cudaSuccess
        return r[1] if len(r) > 1 else None

    prec, form = getattr(qb, prec), getattr(qb, form)
    rng = np.random.default_rng(5)
    n = 14
    psi = gaussian_ket(rng, 2 ** n)
    c = circuit(qb, rng, n)
    s = qb.State.from_numpy(ctx, psi, [2] * n, prec)
    once, twice = s.clone(), s.clone()
    if planned:
        c.run(s.clone(), form)
    ctx.synchronize()
    stream = ctx.stream()
    ok(rt.cudaStreamBeginCapture(stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal))
    c.run(s, form)
    graph = ok(rt.cudaStreamEndCapture(stream))
    instance = ok(rt.cudaGraphInstantiate(graph, 0))
    ok(rt.cudaGraphDestroy(graph))
    c.run(once, form)
    c.run(twice, form)
    c.run(twice, form)
    c.gate(haar_unitary(rng, 2), [0])
    c.run(s.clone(), form)  # planned again
    del c
    others = [circuit(qb, rng, n) for _ in range(4)]
    for o in others:
        o.run(s.clone(), form)
    assert np.array_equal(s.numpy(), qb.State.from_numpy(ctx, psi, [2] * n, prec).numpy())
    for want in (once, twice):
        ok(rt.cudaGraphLaunch(instance, stream))
        ctx.synchronize()
        assert np.array_equal(s.numpy(), want.numpy())
    ok(rt.cudaGraphExecDestroy(instance))


@pytest.mark.parametrize("prec", ["C128", "C64"])
def test_passes_of_one_gate_are_a_launch_each(ctx, prec):
    """A circuit whose passes hold one uncontrolled gate each needs no tables: no buffer,
    no copy, one kernel node a gate in a captured run."""
    import qpp_b200 as qb
    rt = pytest.importorskip("cuda.bindings.runtime")
    rng = np.random.default_rng(3)
    n = 14
    s = qb.State.from_numpy(ctx, gaussian_ket(rng, 2 ** n), [2] * n, getattr(qb, prec))
    c = qb.Circuit(n)
    c.gate(haar_unitary(rng, 2), [4])
    for planned in (False, True):
        ctx.synchronize()
        rt.cudaStreamBeginCapture(ctx.stream(), rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal)
        c.run(s, qb.PLAIN)
        err, graph = rt.cudaStreamEndCapture(ctx.stream())
        assert err == rt.cudaError_t.cudaSuccess
        assert rt.cudaGraphGetNodes(graph, 0)[-1] == 1, planned
        rt.cudaGraphDestroy(graph)
