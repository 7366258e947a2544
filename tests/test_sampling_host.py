"""The uniform numbers of a step's draws, made for all rows by the host library."""
from array import array

import numpy as np
import pytest


@pytest.mark.parametrize("seeds,indices", [([0], [0]), ([1 << 64, -1, (1 << 64) - 1, 7, 7], [3, 0, 5, 8, 9]), (list(range(-40, 40)), [1 << 40] * 80)])
def test_uniforms_of_many_draws(seeds, indices):
    """The same numbers as `uniform_for`, draw by draw: functions of (seed, index) as 64-bit patterns."""
    from kestrel_llm_b200.cache.manager import host_library
    from kestrel_llm_b200.sampling import uniform_for
    mask = (1 << 64) - 1
    s, i = array("Q", [x & mask for x in seeds]), array("Q", [x & mask for x in indices])
    out = np.zeros(len(seeds), np.float32)
    host_library().kbatch_uniforms(len(seeds), s.buffer_info()[0], i.buffer_info()[0], out.ctypes.data)
    assert out.tolist() == [np.float32(uniform_for(a, b)) for a, b in zip(seeds, indices)]
    assert ((out > 0) & (out <= 1)).all()
