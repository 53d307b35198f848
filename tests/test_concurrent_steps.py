"""Repeated steps: from the 33rd launch on, a step runs as a graph that holds only the orders
its data needs.  Its memory must equal, word for word, that of the same steps played op by op
in tape order."""
import numpy as np
import pytest

from tests import helpers
from thunderengine_web_b200 import scenario, timestep

STEPS = 36   # four of them past the chain


def _both(tape, init, mode):
    out = []
    for graph in (True, False):
        r = helpers.gpu_replayer(tape, init, hashes=False, mode=mode if graph else 0)
        if graph:
            r.encode_steps(STEPS)
        else:
            for _ in range(STEPS):
                r.run_ops(0, r.num_ops - 1)
        out.append(r.read(r.buffers_end))
        base = list(r.base)
        r.close()
    return out, base


# 12x10x8: the smallest; 37x29x13: odd extents; 40x24x16 dry on aligned rows
@pytest.mark.gpu
@pytest.mark.parametrize('mode', [0, 1])
@pytest.mark.parametrize('dims,moist,align', [((12, 10, 8), True, False), ((37, 29, 13), True, False),
                                              ((40, 24, 16), False, True)])
def test_synthetic_steps_equal_the_ops_in_tape_order(dims, moist, align, mode):
    run = timestep.Run(scenario.tiny(*dims, dx=500.0, dz=250.0, dt=3.0, nsound=8, us=25.0, align_rows=align), moist=moist)
    tape = run.tape(1)
    (graph, ops), base = _both(tape, run.initial_buffers(), mode)
    if mode == 0:
        assert np.array_equal(graph, ops)
        return
    for name in run.fields:   # fused mode does not keep the step's scratch fields
        if name not in helpers.SCRATCH:
            a, b = (helpers.field_view(m, run, base[run.rec.ids['arena']], name) for m in (graph, ops))
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), name


# A refused change of parameters leaves the step as it was, also for the graph that is built later
@pytest.mark.gpu
@pytest.mark.parametrize('how', ['step', 'words'])
def test_a_refused_change_of_parameters(how):
    import base64
    import copy
    import struct
    run = timestep.Run(scenario.tiny(12, 10, 8, dx=500.0, dz=250.0, dt=3.0, nsound=8, us=25.0))
    tape = run.tape(1)
    init = run.initial_buffers()
    (want, _), _ = _both(tape, init, 0)
    r = helpers.gpu_replayer(tape, init, hashes=False)
    r.encode_steps(4)
    step = copy.deepcopy(tape['steps'][0])
    dims = [c for c in step if c['op'] == 'bytes' and c['index'] == 0][40]   # of a dispatch amid the step
    raw = base64.b64decode(dims['data'])
    with pytest.raises(RuntimeError, match='GridDims'):
        if how == 'step':
            dims['data'] = base64.b64encode(struct.pack('<i', 0) + raw[4:]).decode()
            r.use_step(step)
        else:
            r.write_words(_payload_offset(tape, step, dims), np.zeros(1, np.uint32))
    r.encode_steps(STEPS - 4)
    assert np.array_equal(r.read(r.buffers_end), want)
    r.close()


def _payload_offset(tape, step, cmd):
    """Word offset of the parameter words of a setBytes command (its place among them)."""
    from oracle.player import CpuPlayer
    p = CpuPlayer(tape, helpers.kernels_meta())
    p.plan(False)
    at = p.buffers_end
    for c in step:
        if c is cmd:
            return at
        if c['op'] == 'bytes':
            import base64
            at += -(-(-(-len(base64.b64decode(c['data'])) // 4)) // 4) * 4 + 4


# A tape may leave the field stride 0: the regions of its fields are then their grid's
@pytest.mark.gpu
@pytest.mark.parametrize('mode', [0, 1])
def test_steps_of_a_tape_without_a_field_stride(mode):
    run = timestep.Run(scenario.tiny(37, 29, 13, dx=500.0, dz=250.0, dt=3.0, nsound=8, us=25.0))
    tape = run.tape(1)
    tape['fieldStride'] = 0
    (graph, ops), base = _both(tape, run.initial_buffers(), mode)
    for name in run.fields:
        if mode == 0 or name not in helpers.SCRATCH:
            a, b = (helpers.field_view(m, run, base[run.rec.ids['arena']], name) for m in (graph, ops))
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), name


@pytest.mark.gpu
@pytest.mark.parametrize('mode', [0, 1])
@pytest.mark.parametrize('name', ['single_cell', 'squall_line'])
def test_recorded_physics_steps_equal_the_ops_in_tape_order(name, mode):
    tape, init, _, _ = helpers.load_golden_scenario(name)
    (graph, ops), base = _both(tape, init, mode)
    if mode == 0:
        assert np.array_equal(graph, ops)
        return
    arena = next(b['id'] for b in tape['buffers'] if b['arena'])
    scratch = set(helpers.SCRATCH)
    for field in tape['fields']:
        if field not in scratch:
            a, b = (helpers.field_view(m, tape, base[arena], field) for m in (graph, ops))
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), field
