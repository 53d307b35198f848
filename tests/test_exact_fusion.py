"""Exact mode runs a phase fused where the step stores the phase's scratch again later.  Every
memory word after a step must be the one the ops in tape order leave."""
import numpy as np
import pytest

from tests import helpers
from thunderengine_web_b200 import scenario, timestep


def _step(tape, init, ops):
    r = helpers.gpu_replayer(tape, init, hashes=False)
    for _ in range(2):
        if ops:
            r.run_ops(0, r.num_ops - 1)
        else:
            r.encode_steps(1)
    mem = r.read(r.buffers_end)
    r.close()
    return mem


@pytest.mark.gpu
@pytest.mark.parametrize('dims,kw', [((12, 10, 8), {}), ((37, 29, 13), {}), ((34, 9, 5), dict(align=True)),
                                     ((48, 20, 10), dict(moist=False)), ((5, 3, 8), {}), ((33, 32, 24), dict(core=True)),
                                     ((20, 18, 12), dict(weno_momentum=False))])
def test_every_word_of_a_synthetic_step(dims, kw):
    kw = dict(kw)
    cfg = scenario.tiny(*dims, dx=500.0, dz=250.0, dt=3.0, nsound=7, us=25.0, align_rows=kw.pop('align', False))
    run = timestep.Run(cfg, **kw)
    tape = run.tape(1, core=kw.get('core', False))
    init = run.initial_buffers()
    assert np.array_equal(_step(tape, init, False), _step(tape, init, True))


@pytest.mark.gpu
@pytest.mark.parametrize('name', ['single_cell', 'squall_line', 'supercell_stretched'])
def test_every_word_of_a_recorded_step(name):
    tape, init, _, _ = helpers.load_golden_scenario(name)
    assert np.array_equal(_step(tape, init, False), _step(tape, init, True))


# Bindings that put two roles of a phase on one field, or half over one another, keep the
# ops' own order: (pipe whose binding moves, binding, field it moves to, words added).
@pytest.mark.gpu
@pytest.mark.parametrize('pipe,index,field,words', [('acoustic_w_solve', 10, 'cB', 0), ('acoustic_fpk', 6, 'w', 0),
                                                    ('adv_flux_x', 3, 'fy', 0), ('acoustic_uv', 4, 'vten', 64),
                                                    ('adv_assemble', 6, 'fz', 0), ('rk_update', 2, 'tend', 0)])
def test_aliased_phases(pipe, index, field, words):
    run = timestep.Run(scenario.tiny(20, 14, 10, dx=500.0, dz=250.0, dt=3.0, nsound=6, us=25.0))
    tape = run.tape(1)
    now = None
    for c in tape['steps'][0]:
        if c['op'] == 'pipe':
            now = c['name']
        elif c['op'] == 'buf' and now == pipe and c['index'] == index:
            c['offset'] = run.fields[field] + 4 * words
    init = run.initial_buffers()
    assert np.array_equal(_step(tape, init, False), _step(tape, init, True))
