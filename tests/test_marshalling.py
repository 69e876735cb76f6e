"""Matrices on their way into the library: column-major complex128 values, copied as
bytes while small, by pointer (and not at all where they lie right) above."""
import ctypes as ct

import numpy as np
import pytest

import qpp_b200 as qb


@pytest.mark.parametrize("d", [1, 2, 24, 25, 64])
@pytest.mark.parametrize("order", ["C", "F", "strided"])
@pytest.mark.parametrize("dtype", [np.complex128, np.float64])
def test_gate_values(d, order, dtype):
    rng = np.random.default_rng(d)
    A = rng.normal(size=(d, d)).astype(dtype)
    if order == "strided":
        A = np.repeat(np.repeat(A, 2, 0), 3, 1)[::2, ::3]
    else:
        A = np.asarray(A, order=order)
    buf, rows = qb._gate(A)
    n = A.size * 16
    got = buf if isinstance(buf, bytes) else ct.string_at(buf, n)
    assert rows == d and len(got) == n
    np.testing.assert_array_equal(np.frombuffer(got, np.complex128).reshape(d, d, order="F"), A)


def test_large_gates_are_not_copied_to_bytes():
    A = np.asfortranarray(np.eye(144, dtype=np.complex128))
    buf, _ = qb._gate(A)
    assert buf.value == A.ctypes.data
    C = np.ascontiguousarray(A + 1j)
    assert not isinstance(qb._gate(C)[0], bytes)
