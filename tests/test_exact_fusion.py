"""Exact mode runs a phase fused where the step stores the phase's scratch again later.  Every
memory word after a step must be the one the ops in tape order leave."""
import base64
import copy
import struct

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


# One substep whose column solve reads the coefficients the substep before it left, and stores its
# own there or elsewhere.
@pytest.mark.gpu
@pytest.mark.parametrize('binds', [((7, 'cA'),), ((5, 'cB'),), ((7, 'cA'), (10, 'fx'))])
def test_a_later_op_that_reads_skipped_scratch(binds):
    run = _run()
    tape = run.tape(1)
    for index, field in binds:
        _bind(tape, 'acoustic_w_solve', index, run.fields[field], only=4)
    _same_words(run, tape, run.initial_buffers(), 0)


# qv's x faces of stage 1 but the last: its assembly reads that one as th's dispatch left it.
@pytest.mark.gpu
@pytest.mark.parametrize('mode', [0, 1])
def test_a_flux_dispatch_of_a_part_of_the_faces(mode):
    run = _run()
    tape = run.tape(1)
    at = [q for q, c in enumerate(tape['steps'][0]) if c['op'] == 'pipe' and c['name'] == 'adv_flux_x'][1]
    next(c for c in tape['steps'][0][at:] if c['op'] == 'dispatch')['grid'] = [run.grid.nx, run.grid.ny, run.grid.nz]
    _same_words(run, tape, run.initial_buffers(), mode)


def _probe(tape, run):
    """A further buffer of one field, outside the arena."""
    tape['buffers'].append(dict(id=len(tape['buffers']), label='probe', length=run.grid.count * 4))
    return tape['buffers'][-1]['id']


def _adv_u(tape, run, stage, opened, after):
    """u's assembly of RK stage `stage` stores its tendency in `tend` instead of adding it to uten,
    with open x edges (whose faces keep what tend held) or closed ones; `after` follows it."""
    now, seen, mine, out = None, -1, False, []
    for c in tape['steps'][0]:
        if c['op'] == 'pipe':
            now, mine = c['name'], False
        if now == 'adv_assemble' and c['op'] == 'bytes':
            if c['index'] == 1:
                u = struct.unpack('<i', base64.b64decode(c['data'])[:4])[0] == 2
                seen += u
                mine = u and seen == stage
            elif mine and c['index'] == 12:
                c['data'] = base64.b64encode(struct.pack('<i', 0)).decode()
            elif mine and c['index'] == 17:
                c['data'] = base64.b64encode(struct.pack('<ii', int(opened), 0)).decode()
        if mine and c['op'] in ('buf', 'bufoff') and c['index'] == 11:
            c['offset'] = run.fields['tend']
        out.append(c)
        if mine and c['op'] == 'dispatch':
            out += after
            mine = False
    tape['steps'][0] = out
    assert seen >= stage
    _bind(tape, 'adv_assemble', 19, run.fields['qzero'])   # a field it does not use; by default tend too


# An assembly of u on open edges leaves the tendency's edge faces alone, so a copy after it
# reads there what th's assembly stored before it.
@pytest.mark.gpu
@pytest.mark.parametrize('mode', [0, 1])
def test_open_edge_faces_of_a_shared_tendency(mode):
    run = _run()
    tape = run.tape(1)
    _adv_u(tape, run, 1, True, [dict(op='copy', src=run.rec.ids['arena'], srcOffset=run.fields['tend'],
                                     dst=_probe(tape, run), dstOffset=0, size=run.grid.count * 4)])
    for pipe, index, only in (('adv_assemble', 11, 4), ('rk_update', 3, 1)):   # qv's tendency of stage 1 elsewhere
        _bind(tape, pipe, index, run.fields['cA'], only)
    _same_words(run, tape, run.initial_buffers(), mode)


# Closed edges in stage 1, open ones in stage 2: the second assembly does not store the faces
# that the first one did.
@pytest.mark.gpu
def test_a_store_on_closed_edges_is_not_repeated_on_open_ones():
    run = _run()
    tape = run.tape(1)
    probe = _probe(tape, run)
    cmds = tape['steps'][0]
    first = next(q for q, c in enumerate(cmds) if c['op'] == 'pipe' and c['name'] == 'rk_update')
    rk = copy.deepcopy(cmds[first:first + 1 + next(q for q, c in enumerate(cmds[first:]) if c['op'] == 'dispatch')])
    for c in rk:   # rk_update of u's tendency into the probe
        if c['op'] == 'bytes' and c['index'] == 1:
            c['data'] = base64.b64encode(struct.pack('<i', 2)).decode()
        elif c['op'] == 'buf' and c['index'] in (2, 3):
            c['offset'] = run.fields[{2: 'u_a', 3: 'tend'}[c['index']]]
        elif c['op'] == 'buf' and c['index'] == 4:
            c['buf'], c['offset'] = probe, 0
        elif c['op'] == 'dispatch':
            c['grid'] = [run.grid.nx + 1, run.grid.ny, run.grid.nz]
    assert [c['index'] for c in rk if c['op'] == 'buf'] == [30, 2, 3, 4]
    for stage, opened in ((0, False), (1, True)):
        _adv_u(tape, run, stage, opened, copy.deepcopy(rk))
    _same_words(run, tape, run.initial_buffers(), 0)


# Fields in a buffer that is not marked as an arena; acoustic_pp's binding 9 left at an earlier
# kernel's field (w) in the substeps that store nothing there: all substeps fuse in fused mode
@pytest.mark.gpu
@pytest.mark.parametrize('form', ['no arena', 'no ppx'])
def test_forms_that_stay_fused(form):
    run = _run()
    tape = run.tape(1)
    if form == 'no arena':
        for b in tape['buffers']:
            b['arena'] = False
    else:
        cmds, held = [], []
        for c in tape['steps'][0]:   # binding 9 of acoustic_pp where it does not store there
            if c['op'] == 'pipe':
                held = [c] if c['name'] == 'acoustic_pp' else []
            if not held:
                cmds.append(c)
                continue
            if c is not held[0]:
                held.append(c)
            if c['op'] == 'dispatch':
                save = next(h for h in held if h['op'] == 'bytes' and h['index'] == 10)
                if struct.unpack('<i', base64.b64decode(save['data'])[:4])[0] == 0:
                    held = [h for h in held if not (h['op'] == 'buf' and h['index'] == 9)]
                cmds += held
                held = []
        tape['steps'][0] = cmds
    r = helpers.gpu_replayer(tape, {}, hashes=False, mode=1)
    assert sum(s[0] == 1 for s in r.fused_segments()) == 11
    r.close()
    for mode in (0, 1):
        _same_words(run, tape, run.initial_buffers(), mode)
