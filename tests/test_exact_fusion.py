"""Exact mode runs a phase fused where the step stores the phase's scratch again later.  Every
memory word after a step must be the one the ops in tape order leave."""
import numpy as np
import pytest

from oracle.player import CpuPlayer
from tests import helpers
from thunderengine_web_b200 import scenario, timestep


def _step(tape, init, ops, mode=0):
    r = helpers.gpu_replayer(tape, init, hashes=False, mode=mode)
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


def _run():
    return timestep.Run(scenario.tiny(20, 14, 10, dx=500.0, dz=250.0, dt=3.0, nsound=6, us=25.0))


def _bind(tape, pipe, index, offset, only=None):
    """Moves binding `index` of `pipe` to `offset` (bytes) in its buffer; of every such dispatch or
    of the `only`-th."""
    now, seen = None, 0
    for c in tape['steps'][0]:
        if c['op'] == 'pipe':
            now = c['name']
        elif c['op'] in ('buf', 'bufoff') and now == pipe and c['index'] == index:
            if only is None or seen == only:
                c['offset'] = offset
            seen += 1
    assert seen


def _same_words(run, tape, init, mode):
    got, want = _step(tape, init, False, mode), _step(tape, init, True)
    if mode == 0:
        assert np.array_equal(got, want)
        return
    layout = CpuPlayer(tape, helpers.kernels_meta())
    layout.plan(False)
    base, aid = layout.base, run.rec.ids['arena']
    for name in run.fields:   # fused mode does not keep the step's scratch fields
        if name not in helpers.SCRATCH:
            a, b = (helpers.field_view(m, run, base[aid], name) for m in (got, want))
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), name
    for b in tape['buffers']:
        if b['id'] != aid:
            at = slice(base[b['id']], base[b['id']] + b['length'] // 4)
            assert np.array_equal(got[at], want[at]), b['label']


# The same in both modes, for the substep's bindings: one of its inputs on a field that a run of
# substeps moves to its workspace (u, v), whose halos it leaves unfilled (u, v, w, ppd) or that
# it adds to.
@pytest.mark.gpu
@pytest.mark.parametrize('mode', [0, 1])
@pytest.mark.parametrize('pipe,index,field,words', [('acoustic_uv', 4, 'u', 0), ('acoustic_uv', 5, 'v', 0),
                                                    ('acoustic_uv', 3, 'ppd', 0), ('acoustic_fpk', 7, 'u', 3),
                                                    ('acoustic_fpk', 5, 'ppd', 0), ('acoustic_fpk', 6, 'rrw', 0),
                                                    ('acoustic_accumulate', 7, 'rru', 0)])
def test_aliased_substeps(pipe, index, field, words, mode):
    run = _run()
    tape = run.tape(1)
    _bind(tape, pipe, index, run.fields[field] + 4 * words)
    _same_words(run, tape, run.initial_buffers(), mode)
