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


@pytest.fixture
def sampler(monkeypatch):
    """A Sampler whose options stay on the host: (sampler, the options of its calls)."""
    from types import SimpleNamespace

    import torch
    from kestrel_llm_b200.csrc import ops
    from kestrel_llm_b200.sampling.sampler import Sampler
    s, seen = Sampler("cpu"), []
    pinned = torch.full((5 * 64,), float("nan"))
    slot = SimpleNamespace(pinned=pinned, floats=pinned.numpy(), ints=pinned.numpy().view(np.int32), done=SimpleNamespace(record=lambda: None), pending=False)
    monkeypatch.setattr(s, "_slot", lambda rows: slot)
    monkeypatch.setattr(ops, "sample_options", lambda logits, options, out: seen.append(options.clone()))
    monkeypatch.setattr(ops, "argmax", lambda logits, out: seen.append("argmax"))
    return s, seen


@pytest.mark.parametrize("more", [(1, 0, 0), (0, 2, 0), (0, 0, 3), (2, 1, 0), (0, 1, 1)])
def test_longer_lists_are_cut_to_the_rows(sampler, more):
    import torch
    from kestrel_llm_b200.sampling import SamplingParams
    s, seen = sampler
    params = [SamplingParams(temperature=0.5 + 0.1 * i, top_k=3 + i, top_p=0.9, min_p=0.01 * i) for i in range(6)]
    seeds, indices = list(range(20, 26)), list(range(40, 46))
    for extra in ((0, 0, 0), more):
        s.sample(torch.zeros(3, 8), *(x[:3 + n] for x, n in zip((params, seeds, indices), extra)))
    assert torch.equal(seen[0].view(torch.int32), seen[1].view(torch.int32)) and seen[0].shape == (5, 3)


@pytest.mark.parametrize("lengths", [(2, 3, 3), (3, 2, 3), (3, 3, 1), (4, 4, 4), (2, 2, 2)])
def test_rows_without_options_are_refused(sampler, lengths):
    """Fewer options than rows, or more in every list; rows that all take the first maximum need none."""
    import torch
    from kestrel_llm_b200.sampling import SamplingParams
    s, seen = sampler
    n, m, k = lengths
    with pytest.raises(ValueError, match="3 rows of logits"):
        s.sample(torch.zeros(3, 8), [SamplingParams(temperature=0.5)] * n, [1] * m, [2] * k)
    assert not seen
    s.sample(torch.zeros(3, 8), [SamplingParams(temperature=0.0)] * n, [1] * m, [2] * k)
    assert seen == ["argmax"]


def test_options_of_another_shape_are_refused(monkeypatch):
    import torch
    from kestrel_llm_b200.csrc import ops
    monkeypatch.setattr(ops, "_need", lambda *a: None)
    for rows, results in ((2, 3), (4, 3), (3, 2)):
        with pytest.raises(ops.KernelError, match="for 3 rows"):
            ops.sample_options(torch.zeros(3, 8), torch.zeros(5, rows), torch.zeros(results, dtype=torch.int32))
