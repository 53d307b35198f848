"""The linear scalar advection of large grids (warps of 31 cells walking up 16 levels) against the
per-dispatch kernels, word for word: a last strip of one cell, an odd last row, a last walk of
one level, few levels, open edges (fluxes stored and dropped alike in exact mode)."""
import numpy as np
import pytest

from tests import helpers
from thunderengine_web_b200 import scenario, timestep


# each has at least 2368 = 148 x 16 warps of the walk: strips x row pairs x walks
@pytest.mark.gpu
@pytest.mark.parametrize('dims,opened', [((32, 1185, 17), False), ((311, 431, 5), False), ((311, 431, 6), True),
                                         ((156, 133, 98), False)])
def test_steps_equal_the_per_dispatch_kernels(dims, opened):
    nx, ny, nz = dims
    assert -(-nx // 31) * ((ny + 1) // 2) * -(-nz // 16) >= 148 * 16
    run = timestep.Run(scenario.tiny(*dims, dx=500.0, dz=150.0, dt=3.0, nsound=2, us=25.0))
    tape = run.tape(1)
    if opened:   # adv_assemble's open-edge branches (the step's other kernels stay periodic)
        import base64
        import struct
        name = None
        for c in tape['steps'][0]:
            if c['op'] == 'pipe':
                name = c['name']
            elif c['op'] == 'bytes' and name == 'adv_assemble' and c['index'] == 17:
                c['data'] = base64.b64encode(struct.pack('<ii', 1, 1)).decode()
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
