"""The linear scalar advection of large grids (warps of 31 cells walking up 16 levels) against the
per-dispatch kernels, word for word: a last strip of one cell, an odd last row, a last walk of
one level, few levels, open edges, fluxes dropped and stored."""
import base64
import struct

import numpy as np
import pytest

from tests import helpers
from thunderengine_web_b200 import scenario, timestep


def _open(tape):
    """adv_assemble's open-edge branches (the step's other kernels stay periodic)."""
    name = None
    for c in tape['steps'][0]:
        if c['op'] == 'pipe':
            name = c['name']
        elif c['op'] == 'bytes' and name == 'adv_assemble' and c['index'] == 17:
            c['data'] = base64.b64encode(struct.pack('<ii', 1, 1)).decode()


# each has at least 2368 = 148 x 16 warps of the walk: strips x row pairs x walks
@pytest.mark.gpu
@pytest.mark.parametrize('dims,opened', [((32, 1185, 17), False), ((311, 431, 5), False), ((311, 431, 6), True),
                                         ((156, 133, 98), False)])
def test_steps_equal_the_per_dispatch_kernels(dims, opened):
    nx, ny, nz = dims
    assert -(-nx // 31) * ((ny + 1) // 2) * -(-nz // 16) >= 148 * 16
    run = timestep.Run(scenario.tiny(*dims, dx=500.0, dz=150.0, dt=3.0, nsound=2, us=25.0))
    tape = run.tape(1)
    if opened:
        _open(tape)
    init = run.initial_buffers()
    mem = []
    for mode in (None, 0, 1):
        r = helpers.gpu_replayer(tape, init, hashes=False, mode=mode or 0)
        for _ in range(2):
            if mode is None:
                r.run_ops(0, r.num_ops - 1)
            else:
                r.encode_steps(1)
        mem.append(r.read(r.buffers_end))
        arena = r.base[run.rec.ids['arena']]
        r.close()
    assert np.array_equal(mem[1], mem[0])
    for name in run.fields:
        if name not in helpers.SCRATCH:
            a, b = (helpers.field_view(m, run, arena, name) for m in (mem[2], mem[0]))
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), name


# Copies of fx, fy, fz behind qv's linear phases, which then store every face (th's drop theirs)
@pytest.mark.gpu
@pytest.mark.parametrize('dims,opened', [((32, 1185, 17), False), ((311, 431, 5), False), ((311, 431, 6), True),
                                         ((310, 475, 7), False)])
def test_stored_fluxes_equal_the_per_dispatch_kernels(dims, opened):
    nx, ny, nz = dims
    assert -(-nx // 31) * ((ny + 1) // 2) * -(-nz // 16) >= 148 * 16
    run = timestep.Run(scenario.tiny(*dims, dx=500.0, dz=150.0, dt=3.0, nsound=2, us=25.0))
    tape = run.tape(1)
    if opened:
        _open(tape)
    probes, cmds, name, seen = [], [], None, 0
    for c in tape['steps'][0]:
        cmds.append(c)
        if c['op'] == 'pipe':
            name = c['name']
            seen += name == 'adv_flux_x'
        elif c['op'] == 'dispatch' and name == 'adv_assemble' and seen == 2 * (len(probes) // 3 + 1):
            for f in ('fx', 'fy', 'fz'):   # th and qv are the scalars of a stage
                tape['buffers'].append(dict(id=len(tape['buffers']), label='probe', length=run.grid.count * 4))
                probes.append(tape['buffers'][-1]['id'])
                cmds.append(dict(op='copy', src=run.rec.ids['arena'], srcOffset=run.fields[f], dst=probes[-1], dstOffset=0,
                                 size=run.grid.count * 4))
    assert len(probes) == 6   # RK stages 1 and 2
    tape['steps'][0] = cmds
    init = run.initial_buffers()
    arena = np.frombuffer(init[run.rec.ids['arena']], np.float32).copy()
    rng = np.random.default_rng(nx)
    for f in ('u', 'v', 'w', 'u_a', 'v_a', 'w_a'):   # winds of both signs in every direction
        at = run.fields[f] // 4
        arena[at:at + run.grid.count] += 4 * rng.random(run.grid.count, np.float32) - 2
    init[run.rec.ids['arena']] = arena.tobytes()
    mem = []
    for mode in (None, 0, 1):
        r = helpers.gpu_replayer(tape, init, hashes=False, mode=mode or 0)
        if mode is None:
            r.run_ops(0, r.num_ops - 1)
        else:
            r.encode_steps(1)
        mem.append(r.read(r.buffers_end))
        base = list(r.base)
        r.close()
    assert np.array_equal(mem[1], mem[0])
    sJ, sK = nx + 7, ny + 7
    for n, b in enumerate(probes):
        face = [m[base[b]:base[b] + run.grid.count].reshape(nz + 1, sK, sJ) for m in (mem[2], mem[0])]
        box = [slice(0, nz), slice(3, 3 + ny), slice(3, 3 + nx)]
        box[2 - n % 3] = slice(box[2 - n % 3].start, box[2 - n % 3].stop + 1)
        assert np.count_nonzero(face[1][tuple(box)]) > 0
        assert np.array_equal(face[0][tuple(box)], face[1][tuple(box)]), n
