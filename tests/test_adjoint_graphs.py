"""Repeated adjoint windows: the replay and reverse graphs, shared by every step, change from a
chain to the orders the data needs after 16 steps.  The gradient may differ by the order of
atomic adds only, and memory returns to the start state, word for word."""
import numpy as np
import pytest

from tests import helpers
from thunderengine_web_b200 import scenario, timestep


# 37x9x13: odd extents and a ragged last block of steps; 16x12x6: steps in one block
@pytest.mark.gpu
@pytest.mark.parametrize('dims,steps,every', [((37, 9, 13), 5, 2), ((16, 12, 6), 6, 6)])
def test_gradient_and_memory_of_repeated_windows(dims, steps, every):
    run = timestep.Run(scenario.tiny(*dims, dx=500.0, dz=250.0, dt=3.0, nsound=7, us=25.0), core=True)
    tape = run.tape(1)
    start = helpers.cpu_run(tape, run.initial_buffers(), nsteps=1, hashes=False)
    core = run.tape(1, core=True)
    r = helpers.gpu_replayer(core, {b['id']: start.buffer_words(b['id']).tobytes() for b in tape['buffers']}, hashes=False)
    before = r.read(r.buffers_end)
    g, base = run.grid, r.base[run.rec.ids['arena']]
    seed = np.random.default_rng(5).standard_normal(g.count).astype(np.float32)
    grads, ends = [], []
    for _ in range(6):   # 30 and 36 steps in each direction
        r.adjoint_forward(steps, every)
        ends.append(r.read(r.buffers_end))
        r.adjoint_write_words(base + run.fields['w'] // 4, seed)
        r.adjoint_backward()
        grads.append([r.adjoint_read(g.count, base + run.fields[n] // 4).astype(np.float64) for n in ('th', 'u_a', 'v_a')])
        assert np.array_equal(r.read(r.buffers_end), before)
    r.close()
    for e in ends[1:]:
        assert np.array_equal(e, ends[0])
    for q in grads[1:]:
        for a, b in zip(q, grads[0]):
            assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b)


# A new time step (use_step, the same structure) between windows: tables and graphs follow it
@pytest.mark.gpu
def test_gradient_after_a_change_of_parameters():
    run = timestep.Run(scenario.tiny(16, 12, 6, dx=500.0, dz=250.0, dt=3.0, nsound=7, us=25.0), core=True)
    tape = run.tape(1)
    start = helpers.cpu_run(tape, run.initial_buffers(), nsteps=1, hashes=False)
    init = {b['id']: start.buffer_words(b['id']).tobytes() for b in tape['buffers']}
    core = run.tape(1, core=True)
    run.set_time_step(2.0, 7)
    later = run.tape(1, core=True)
    seed = np.random.default_rng(5).standard_normal(run.grid.count).astype(np.float32)

    def gradient(r):
        base = r.base[run.rec.ids['arena']]
        r.adjoint_forward(4, 2)
        r.adjoint_write_words(base + run.fields['w'] // 4, seed)
        r.adjoint_backward()
        return [r.adjoint_read(run.grid.count, base + run.fields[n] // 4).astype(np.float64) for n in ('th', 'u_a', 'v_a')]

    fresh = helpers.gpu_replayer(later, init, hashes=False)
    want = gradient(fresh)
    fresh.close()
    r = helpers.gpu_replayer(core, init, hashes=False)
    other = gradient(r)
    r.use_step(later['steps'][0])
    got = [gradient(r) for _ in range(5)][-1]   # 20 steps: past the chain
    r.close()
    for a, b, c in zip(got, want, other):
        assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b)
        assert np.linalg.norm(c - b) > 1e-3 * np.linalg.norm(b)
