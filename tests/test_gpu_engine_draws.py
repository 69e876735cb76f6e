"""The outcomes that an engine's runs of measurements draw, against the same draws on
the host: std::generate_canonical on std::mt19937, the first index whose running weight
reaches the fraction, a collapse, the next draw. Sizes with hundreds of chunk sums, the
last ragged; steps whose later draws still have several outcomes; a state with its
weight in the last chunk; both precisions, dropped and kept qudits."""
import numpy as np
import pytest

from tests.qpp_helpers import gaussian_ket

pytestmark = pytest.mark.gpu


def canonical(gen):
    lo, hi = int(gen.random_raw()), int(gen.random_raw())
    return (float(lo) + float(hi) * 2.0 ** 32) / 2.0 ** 64


def draws(psi, n, d, targets, seed):
    """Outcomes of measuring the groups of qudits one group after the other."""
    gen = np.random.RandomState(seed)._bit_generator
    psi = psi.reshape([d] * n)
    out = []
    for group in targets:
        w = np.cumsum(np.abs(psi.reshape(-1)) ** 2)
        at = np.unravel_index(int(np.searchsorted(w, canonical(gen) * w[-1])), psi.shape)
        out += [int(at[q]) for q in group]
        keep = np.zeros_like(psi)
        sel = tuple(at[q] if q in group else slice(None) for q in range(n))
        keep[sel] = psi[sel]
        psi = keep / np.linalg.norm(keep)
    return out


@pytest.mark.parametrize("n,d,prec", [(17, 2, "C128"), (20, 2, "C128"), (18, 2, "C64"), (11, 3, "C128")])
@pytest.mark.parametrize("destructive", [False, True])
@pytest.mark.parametrize("tail", [False, True])
def test_runs_draw_what_the_generator_says(ctx, n, d, prec, destructive, tail):
    import qpp_b200 as qb
    prec = getattr(qb, prec)
    rng = np.random.default_rng([n, d, tail])
    psi = gaussian_ket(rng, d ** n)
    if tail:
        psi[:-40] = 0
    s = qb.State.from_numpy(ctx, psi / np.linalg.norm(psi), [d] * n, prec)
    x = s.numpy()
    targets = [[0, 1], [n - 1, 3], [2], [n // 2, 4, n - 2], [6]]
    c = qb.Circuit(n, d, n)
    at = 0
    for t in targets:
        c.measure(t, at, destructive=destructive)
        at += len(t)
    for seed in range(6):
        e = qb.Engine(ctx, c, qb.KET, prec).set_seed(seed).set_state(s).execute()
        assert e.get_dits()[0][:at] == draws(x, n, d, targets, seed)
