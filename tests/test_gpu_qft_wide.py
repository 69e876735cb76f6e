"""Register QFT passes on a state of 2^31 amplitudes (64-bit offsets in the kernel): a
basis state becomes the plane wave of its index, and TFQ gives it back. Complex64,
16 GB; with the reversal a second buffer of the same size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("swap", [False, True])
def test_basis_state_of_31_qubits(ctx, swap):
    import torch
    import qpp_b200 as qb

    class View:
        def __init__(self, state):
            self.__cuda_array_interface__ = {"shape": (state.D,), "typestr": "<c8", "version": 2,
                                             "data": (state.device_ptr(), False), "strides": None}

    n, at = 31, 0x5a3c19e7
    s = qb.State(ctx, qb.KET, [2] * n, qb.C64)
    ctx.synchronize()
    v = torch.as_tensor(View(s), device="cuda")
    v.zero_()
    v[at] = 1
    torch.cuda.synchronize()
    s.qft(2, swap, False)
    ctx.synchronize()
    v = torch.as_tensor(View(s), device="cuda")
    i = np.random.default_rng(2).integers(0, 2 ** n, 4096)
    k = i if swap else np.array([int(f"{x:031b}"[::-1], 2) for x in i])
    phase = (k.astype(object) * at % 2 ** n).astype(np.float64) / 2 ** n
    want = np.exp(2j * np.pi * phase)
    got = v[torch.as_tensor(i, device="cuda")].cpu().numpy() * np.sqrt(2.0 ** n)
    # 31 steps, each a rounded phase and sum: a few units of 2^-24 a step
    assert np.max(np.abs(got - want)) < 31 * 4 * 2.0 ** -24
    del v
    s.qft(2, swap, True)
    ctx.synchronize()
    v = torch.as_tensor(View(s), device="cuda")
    assert abs(complex(v[at].item()) - 1) < 62 * 4 * 2.0 ** -24
    v[at] = 0
    # chunked: abs() of the whole would be another 8 GB
    assert max(float(x.abs().max()) for x in v.split(1 << 26)) < 62 * 4 * 2.0 ** -24
    del v
    s.free()
