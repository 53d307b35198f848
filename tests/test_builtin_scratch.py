"""The library's own kernel table plans the per-thread scratch that kernels.json does."""
import pytest

from tests import helpers


@pytest.mark.gpu
def test_memory_is_planned_alike_with_and_without_kernels_json():
    from thunderengine_web_b200.replayer import Replayer
    tape, _, _, _ = helpers.load_golden_scenario('single_cell')
    words = []
    for kernels in (helpers.kernels_meta(), None):
        r = Replayer(tape, kernels)
        r.plan(False)
        r.build()
        words.append(r.mem_words)
        r.close()
    assert words[0] == words[1]
