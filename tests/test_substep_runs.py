"""Fused acoustic substeps: runs of them leave out the halo fills in between.  Substep counts
that are odd and even per stage, extents narrower than the halos, rows that are padded."""
import numpy as np
import pytest

from tests import helpers
from thunderengine_web_b200 import scenario, timestep


@pytest.mark.gpu
@pytest.mark.parametrize('dims,nsound,align', [((5, 3, 8), 7, False), ((2, 9, 6), 8, False), ((33, 8, 5), 6, False),
                                               ((64, 5, 13), 9, True), ((31, 40, 12), 2, False),
                                               # the column kernel's sizes: 64 levels, 65 with one
                                               # wave of tiles, 85
                                               ((20, 9, 64), 4, False), ((33, 10, 65), 4, False),
                                               ((16, 8, 85), 4, False)])
def test_fused_steps_equal_the_oracle(dims, nsound, align):
    run = timestep.Run(scenario.tiny(*dims, dx=500.0, dz=250.0, dt=3.0, nsound=nsound, us=25.0, align_rows=align))
    tape = run.tape(1)
    init = run.initial_buffers()
    cpu = helpers.cpu_run(tape, init, nsteps=2, hashes=False)
    r = helpers.gpu_replayer(tape, init, hashes=False, mode=1)
    r.encode_steps(2)
    mem = r.read(r.buffers_end)
    arena = r.base[run.rec.ids['arena']]
    r.close()
    for name in run.fields:
        if name not in helpers.SCRATCH:
            a, b = (helpers.field_view(m, run, arena, name) for m in (mem, cpu.M))
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), name


# te_run_segment on its own: whichever segment is played, its fields end as its ops leave them
@pytest.mark.gpu
@pytest.mark.parametrize('dims,nsound', [((20, 14, 10), 6), ((33, 8, 5), 7)])
def test_each_segment_equals_its_ops(dims, nsound):
    run = timestep.Run(scenario.tiny(*dims, dx=500.0, dz=250.0, dt=3.0, nsound=nsound, us=25.0))
    tape = run.tape(1)
    init = run.initial_buffers()
    seg = helpers.gpu_replayer(tape, init, hashes=False, mode=1)
    ops = helpers.gpu_replayer(tape, init, hashes=False)
    seg.run_ops(0, seg.num_ops - 1)   # a state in motion, scratch fields filled
    state = seg.read(seg.buffers_end)
    arena = seg.base[run.rec.ids['arena']]
    segments = seg.fused_segments()
    assert sum(s[0] == 1 for s in segments) >= 4
    for n, (kind, first, last, _) in enumerate(segments):
        if kind == 0:
            continue
        seg.write_words(0, state)
        ops.write_words(0, state)
        seg.run_segment(n)
        ops.run_ops(first, last)
        a, b = seg.read(seg.buffers_end), ops.read(ops.buffers_end)
        for name in run.fields:
            if name not in helpers.SCRATCH or (kind == 1 and name in ('rru', 'rrv', 'rrw')):
                x, y = (helpers.field_view(m, run, arena, name).view(np.uint32) for m in (a, b))
                assert np.array_equal(x, y), (n, kind, name)
    seg.close()
    ops.close()
