"""The row of parameters that a request's sampling options are packed into."""

from __future__ import annotations

import numpy as np
import pytest

from litinfer_b200.sampling.sampler import _ALONE, _DRAWS, _SMALL_TOP_K, Sampler, SamplingParams

OPTIONS = [(0.7, 50, 0.8, 123456789012345), (1.0, 0, 0.9, -5), (1.0, -7, 1.0, 2**70 + 3), (0.3, 2**40, 0.5, 0), (1.0, 1, 0.5, 1), (0.0, 9, 0.2, 2),
           (1.0, 257, 1.0, 3), (1.0, 256, 0.0, 4), (0.8, 2, 0.99999999999, 5), (0.8, 0, 0.99999999999, 6), (float("nan"), 0, 1e-50, 7)]


def test_rows_are_the_options_as_the_kernel_reads_them():
    params = [SamplingParams(*o) for o in OPTIONS]
    rows = Sampler("cpu")._upload(b"".join(p.packed[0] for p in params), list(range(3, 3 + len(params)))).numpy()
    want = np.empty((len(params), 6), dtype=np.int32)
    want.view(np.float32)[:, 0] = [0.0 if p.greedy else p.temperature for p in params]
    want[:, 1] = [min(max(p.top_k, -1), 2**31 - 1) for p in params]
    want.view(np.float32)[:, 2] = [p.top_p for p in params]
    seeds = np.array([p.seed & 0xFFFF_FFFF_FFFF_FFFF for p in params], dtype=np.uint64)
    want[:, 3:5] = seeds.view(np.uint32).reshape(-1, 2).view(np.int32)
    want[:, 5] = range(3, 3 + len(params))
    assert np.array_equal(rows, want)


@pytest.mark.parametrize("option", OPTIONS, ids=str)
def test_what_a_row_needs_of_the_kernels(option):
    p = SamplingParams(*option)
    temperature, top_p = np.frombuffer(p.packed[0], dtype=np.float32)[[0, 2]]
    assert bool(p.packed[1] & _DRAWS) == (not p.greedy)
    assert bool(p.packed[1] & _SMALL_TOP_K) == (1 < p.top_k <= 256)
    # a row that the kernel draws by temperature alone, for some vocabulary beyond 256, must have been announced
    if temperature > 0 and not 0 < p.top_k <= 256 and not 0 < top_p < 1:
        assert p.packed[1] & _ALONE


def test_greedy_rows_need_nothing_else():
    assert SamplingParams(0.0, None, None).packed == (None, 0)
    with pytest.raises(TypeError):
        SamplingParams(1.0, 5, None).packed
