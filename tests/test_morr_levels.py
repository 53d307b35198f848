"""The CUDA Morrison and reflectivity columns, levels in parallel, against the serial columns of the
same source built for the host, word for word."""
import numpy as np
import pytest

from tests import helpers
from tests.test_morr import host_kernels, morr_case, refl_case


# columns of the recording's 40 levels with seeded condensate; 33 x 5 columns (a ragged block) of
# fewer levels than warps, of one level, and of a level count that is no multiple of the warps
@pytest.mark.gpu
@pytest.mark.parametrize('variant,seed,nx,ny,nz', [('random', 1, 50, 9, 40), ('supersaturated', 3, 50, 9, 40),
                                                   ('random', 5, 33, 5, 7), ('supersaturated', 6, 33, 5, 1),
                                                   ('random', 7, 65, 3, 21)])
def test_gpu_column_equals_the_host_build(variant, seed, nx, ny, nz):
    from thunderengine_web_b200.replayer import Replayer
    cpu, op, M0 = morr_case(variant, seed)
    M0[op.bind[0]:op.bind[0] + 3] = np.array([nx, ny, nz], np.uint32)
    cpu.M = M0.copy()
    cpu.run(host_kernels().get, ops=[op])
    tape, _, _, _ = helpers.load_golden_scenario('single_cell')
    r = Replayer(tape, helpers.kernels_meta())
    r.plan(False)
    r.build()
    r.write_words(0, M0[:r.buffers_end])
    for w, n in ((op.bind[19], 1), (op.bind[0], 127)):   # dorad and the parameter struct
        r.write_words(w, M0[w:w + n])
    oi = [k for k, o in enumerate(cpu.ops) if o is op][0]
    r.run_ops(oi, oi)
    got = r.read(r.buffers_end)
    r.close()
    assert np.count_nonzero(cpu.M[:cpu.buffers_end] != M0[:cpu.buffers_end]) > nx * ny * nz
    bad = np.nonzero(got != cpu.M[:r.buffers_end])[0]
    assert bad.size == 0, 'first differing word %d of %d' % (bad[0], bad.size)


@pytest.mark.gpu
def test_more_levels_in_device_memory_than_planned():
    """nz of the device's parameter struct raised behind the host's copy (half a word written): the
    column keeps to the planned levels."""
    import ctypes
    from thunderengine_web_b200.replayer import Replayer
    cpu, op, M0 = morr_case('random', 1)
    nz = int(M0[op.bind[0] + 2])
    M0[op.bind[0]:op.bind[0] + 2] = np.array([50, 9], np.uint32)
    cpu.M = M0.copy()
    cpu.run(host_kernels().get, ops=[op])
    tape, _, _, _ = helpers.load_golden_scenario('single_cell')
    r = Replayer(tape, helpers.kernels_meta())
    r.plan(False)
    r.build()
    r.write_words(0, M0[:r.buffers_end])
    for w, n in ((op.bind[19], 1), (op.bind[0], 127)):   # dorad and the parameter struct
        r.write_words(w, M0[w:w + n])
    low = (ctypes.c_uint16 * 1)(nz + 24)
    r._check(r.lib.te_write_words(r.h, int(op.bind[0]) + 2, low, 2))
    oi = [k for k, o in enumerate(cpu.ops) if o is op][0]
    r.run_ops(oi, oi)
    got = r.read(r.buffers_end)
    r.close()
    assert np.array_equal(got, cpu.M[:r.buffers_end])


@pytest.mark.gpu
@pytest.mark.parametrize('nx,ny,nz', [(50, 9, 40), (33, 5, 9)])
def test_gpu_reflectivity_equals_the_host_build(nx, ny, nz):
    from thunderengine_web_b200.replayer import Replayer
    cpu, tape, op, M0 = refl_case(seed=nz)
    M0[op.bind[0]:op.bind[0] + 3] = np.array([nx, ny, nz], np.uint32)
    cpu.M = M0.copy()
    cpu.run(host_kernels().get, ops=[op])
    # the diagnostic's first op forms the temperature from th and pi' again, the same words
    r = Replayer(tape, helpers.kernels_meta())
    r.plan(False)
    r.build()
    r.write_words(0, M0[:r.buffers_end])
    r.write_words(op.bind[0], M0[op.bind[0]:op.bind[0] + 127])
    r.encode_diag()
    got = r.read(r.buffers_end)
    r.close()
    assert np.count_nonzero(cpu.M[:cpu.buffers_end] != M0[:cpu.buffers_end]) >= nx * ny * nz * 9 // 10
    bad = np.nonzero(got != cpu.M[:r.buffers_end])[0]
    assert bad.size == 0, 'first differing word %d of %d' % (bad[0], bad.size)
