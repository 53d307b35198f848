"""The workspace of a run of substeps is two fields beyond the word memory.  A plan that leaves no
room for it is accepted all the same, and its fused steps are the same words."""
import numpy as np
import pytest

from tests import helpers
from thunderengine_web_b200 import scenario, timestep


@pytest.mark.gpu
def test_a_plan_that_leaves_no_room_for_the_workspace():
    import torch
    run = timestep.Run(scenario.tiny(320, 320, 80, dx=500.0, dz=250.0, dt=3.0, nsound=6, us=25.0))
    tape = run.tape(1)
    r = helpers.gpu_replayer(tape, {}, hashes=False)
    need = r.mem_words * 4
    r.close()
    torch.cuda.empty_cache()
    room = need + tape['fieldStride'] + tape['fieldStride'] // 4   # not the two fields more
    fill = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device='cuda')
    r = helpers.gpu_replayer(tape, {}, hashes=False)
    assert r.mem_words * 4 == need
    del fill
    torch.cuda.empty_cache()
    for b, data in run.initial_buffers().items():
        r.upload(b, data)
    state = r.read(r.buffers_end)
    r.run_ops(0, r.num_ops - 1)
    want = r.read(r.buffers_end)
    r.write_words(0, state)
    r.set_mode(1)
    r.encode_steps(1)
    got = r.read(r.buffers_end)
    arena = r.base[run.rec.ids['arena']]
    r.close()
    for name in run.fields:
        if name not in helpers.SCRATCH:
            a, b = (helpers.field_view(m, run, arena, name).view(np.uint32) for m in (got, want))
            assert np.array_equal(a, b), name


# A step structure that comes later brings the first runs of substeps
@pytest.mark.gpu
@pytest.mark.parametrize('mode', [0, 1])
def test_runs_of_substeps_in_a_later_step(mode):
    run = timestep.Run(scenario.tiny(20, 14, 10, dx=500.0, dz=250.0, dt=3.0, nsound=6, us=25.0))
    tape = run.tape(1)
    step = tape['steps'][0]
    tape['steps'][0] = [c for c in step if c['op'] == 'copy'][:1]
    r = helpers.gpu_replayer(tape, run.initial_buffers(), hashes=False, mode=mode)
    r.encode_steps(1)
    r.use_step(step)
    state = r.read(r.buffers_end)
    r.run_ops(0, r.num_ops - 1)
    want = r.read(r.buffers_end)
    r.write_words(0, state)
    r.encode_steps(1)
    got = r.read(r.buffers_end)
    arena = r.base[run.rec.ids['arena']]
    r.close()
    for name in run.fields:
        if mode == 0 or name not in helpers.SCRATCH:
            a, b = (helpers.field_view(m, run, arena, name).view(np.uint32) for m in (got, want))
            assert np.array_equal(a, b), name
