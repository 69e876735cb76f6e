"""Gates of many levels (k_smem): one subsystem's gate at the sizes around 48 KB of
shared memory, where a launch needs the larger limit, against numpy."""
import numpy as np
import pytest

import qpp_b200 as qb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("levels,prec", [(13, qb.C128), (2944, qb.C128), (2945, qb.C128), (3072, qb.C128),
                                         (3073, qb.C128), (4096, qb.C64)])
def test_gate_of_many_levels(levels, prec):
    rng = np.random.default_rng(levels)
    A = rng.normal(size=(levels, levels)) + 1j * rng.normal(size=(levels, levels))
    psi = rng.normal(size=2 * levels) + 1j * rng.normal(size=2 * levels)
    ctx = qb.default_context()
    s = qb.State.from_numpy(ctx, psi, [levels, 2], prec)
    s.apply(A, [0])
    want = (A @ psi.reshape(levels, 2)).reshape(-1)
    # sums of `levels` products, each of unit size, against sums of size
    # sqrt(levels): an error of levels * eps / sqrt(levels) at most in eps of the type
    eps = 2.0 ** -53 if prec == qb.C128 else 2.0 ** -24
    tol = 16 * levels * eps
    assert np.abs(s.numpy() - want).max() <= tol * np.abs(want).max()
