"""Register QFT passes (k_qft_reg): whole and partial transforms of kets against
numpy's DFT over the target digits and through the inverse; the smallest sizes that
take them (one tile), one, two and three passes, rounds of one to five steps,
scattered targets."""
import numpy as np
import pytest

from tests.qpp_helpers import gaussian_ket

pytestmark = pytest.mark.gpu


def dft(x, n, t, swap):
    k = len(t)
    rest = [q for q in range(n) if q not in t]
    v = x.reshape([2] * n).transpose(t + rest).reshape(2 ** k, -1)
    v = np.fft.ifft(v, axis=0, norm="ortho").reshape([2] * n)
    if not swap:  # the result's digits in reversed order
        v = v.transpose(list(range(k))[::-1] + list(range(k, n)))
    return v.transpose(np.argsort(t + rest)).reshape(-1)


# 24 steps in 64 bits (32 bits), a few ulp each, over amplitudes of similar size
@pytest.mark.parametrize("prec,tol", [("c128", 1e-12), ("c64", 2e-5)])
@pytest.mark.parametrize("n,k,order", [(24, 24, "all"), (24, 9, "first"), (24, 10, "last"), (24, 13, "any"),
                                       (24, 18, "any"), (12, 12, "all"), (13, 13, "all"), (13, 5, "any"),
                                       (14, 8, "last"), (17, 11, "first"), (20, 20, "all"), (21, 19, "any")])
def test_against_dft(ctx, prec, tol, n, k, order):
    import qpp_b200 as qb
    rng = np.random.default_rng([n, k, len(order)])
    t = [int(q) for q in rng.permutation(n)]
    t = {"all": list(range(n)), "first": list(range(k)), "last": list(range(n - k, n)), "any": t[:k]}[order]
    psi = gaussian_ket(rng, 2 ** n)
    p = qb.C128 if prec == "c128" else qb.C64
    for swap in (True, False):
        s = qb.State.from_numpy(ctx, psi, [2] * n, prec=p)
        want = dft(psi, n, t, swap)
        s.apply_qft(t, 2, swap)
        big = np.max(np.abs(want))
        assert np.max(np.abs(s.numpy() - want)) < tol * big
        s.apply_tfq(t, 2, swap)
        assert np.max(np.abs(s.numpy() - psi)) < tol * np.max(np.abs(psi))
