"""Both forms of the trajectory kernel on registers in shared memory (in sweeps, gate
by gate) at the sizes and noise levels on either side of the rule between them: every
shot replayed through the oracle within the complex64 tolerance (2e-5 relative,
max-norm)."""
import numpy as np
import pytest

from tests.test_gpu_traj import build, random_program, replay, run_traj

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,p", [(4, 0.03), (10, 0.003), (11, 0.0), (11, 0.003), (11, 0.01), (12, 0.002),
                                  (12, 0.03), (13, 0.005), (13, 0.02), (14, 0.015), (14, 0.05)])
def test_shots_of_both_forms_replay_through_oracle(ctx, nq, p):
    import qpp_b200 as qb
    rng = np.random.default_rng(1000 * nq + int(1e4 * p))
    steps, nc = random_program(rng, nq, 50)
    c = build(qb, steps, nq, nc)
    shots = 6
    samples, dits, states, events = run_traj(qb, ctx, c, nq, p, shots, seed=3, max_events=256)
    for s in range(shots):
        ref, _ = replay(steps, nq, dits[s], events[s])
        assert np.max(np.abs(states[s] - ref)) / np.max(np.abs(ref)) < 2e-5
        assert samples[s] < 2 ** nq and np.abs(states[s][samples[s]]) > 0
