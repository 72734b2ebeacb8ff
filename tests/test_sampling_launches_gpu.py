"""Sampling with a small top-k: what the one-pass kernel settles by itself, and what a call launches."""

from __future__ import annotations

import ctypes

import pytest
import torch

from test_fast_paths_gpu import K, params

pytestmark = pytest.mark.gpu


def kernels_of(fn):
    """How many kernels a call launches: the nodes of its capture."""
    fn()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        fn()
    n = ctypes.c_size_t()
    runtime = ctypes.CDLL("libcudart.so.12")
    assert runtime.cudaGraphGetNodes(ctypes.c_void_p(graph.raw_cuda_graph()), None, ctypes.byref(n)) == 0
    return n.value


@pytest.mark.parametrize("option", [(0.7, 50, 0.8), (1.0, 0, 1.0), (1.0, 0, 0.9), (0.0, 1, 1.0), (1.0, 257, 0.9)], ids=str)
def test_no_kernel_for_options_that_a_call_does_not_have(option):
    """Up to 64 rows of a large vocabulary: one kernel that looks at every row, and the draw of rows with temperature alone."""
    x = torch.randn((9, 20000), device="cuda")
    p, out = params([(*option, 3, i) for i in range(9)]), torch.empty(9, dtype=torch.int32, device="cuda")
    assert kernels_of(lambda: K().sample(x, p, out)) == 2
    if not 1 < option[1] <= 256:
        told = torch.empty_like(out)
        p.small_top_k = False
        assert kernels_of(lambda: K().sample(x, p, told)) == 2
        assert told.tolist() == out.tolist()


def test_the_sampler_says_which_options_its_rows_have(monkeypatch):
    from litinfer_b200.sampling import sampler as S

    said, sample = [], S.K.sample
    monkeypatch.setattr(S.K, "sample", lambda x, rows, out: (said.append(rows.small_top_k), sample(x, rows, out))[1])
    x = torch.randn((3, 20000), device="cuda")
    for ks in ((0, 257, 1), (0, 50, 1), (2, 0, 0), (0, 0, 0)):
        S.Sampler("cuda:0").sample(x, [S.SamplingParams(0.8, k, 0.9, 7) for k in ks], [0, 1, 2])
    assert said == [False, True, True, False]


def test_the_sampler_says_whether_a_row_is_drawn_by_temperature_alone(monkeypatch):
    from litinfer_b200.sampling import sampler as S

    x = torch.randn((2, 20000), device="cuda")
    said, sample = [], S.K.sample
    monkeypatch.setattr(S.K, "sample", lambda x, rows, out: (said.append(rows), sample(x, rows, out))[1])
    for k, p in ((0, 0.9), (50, 1.0), (0, 1.0), (19999, 1.0)):
        both = [S.SamplingParams(0.8, k, p, 7), S.SamplingParams(0.8, 30, 0.9, 8)]
        got = S.Sampler("cuda:0").sample(x, both, [0, 1])
        rows, all_kernels = said[-1].clone(), torch.empty_like(got)
        sample(x, rows, all_kernels)
        assert got.tolist() == all_kernels.tolist()
        rows.draws_alone = said[-1].draws_alone
        assert kernels_of(lambda: sample(x, rows, all_kernels)) == (2 if rows.draws_alone else 1)
    assert [r.draws_alone for r in said] == [False, False, True, True]


@pytest.mark.parametrize("V", [16384, 16387, 32000, 151936])
@pytest.mark.parametrize("R", [1, 15, 16, 32, 33, 64])
def test_ordinary_rows_are_settled_in_one_pass(R, V):
    """Where the candidates of a row are few: eight blocks a row up to 15 rows, four up to 32, then two."""
    g = torch.Generator(device="cuda").manual_seed(V + R)
    x = torch.randn((R, V), generator=g, device="cuda") * 2.5
    blocks = 8 if R <= 15 else 4 if R <= 32 else 2
    most = min(256, V // 160, min(V // 40, 1024) // blocks)                # the largest top_k that is taken
    ks = [50 if most >= 50 else 20, min(most, 800 // blocks), 20, 2, most + 1]
    p = params([(0.8, ks[i % 5], (0.8, 1.0)[i % 2], 100 + i, i) for i in range(R)])
    got, all_rows = torch.full((R,), -7, dtype=torch.int32, device="cuda"), torch.empty(R, dtype=torch.int32, device="cuda")
    K().sample(x, p, all_rows)
    K().library().li_sample_leave_rows(1)
    try:
        K().sample(x, p, got)
        torch.cuda.synchronize()
    finally:
        K().library().li_sample_leave_rows(0)
    assert min(all_rows.tolist()) >= 0
    assert got.tolist() == [-1 if i % 5 == 4 else t for i, t in enumerate(all_rows.tolist())]


def test_rows_that_the_pass_leaves():
    """Other options, rows with no number, and more equal values than there is room for."""
    x = torch.randn((6, 30000), device="cuda")
    x[1, 7] = float("nan")
    x[2] = float("-inf")
    x[3] = 1.5
    p = params([(0.7, 50, 0.8, 5, i) for i in range(4)] + [(1.0, 0, 0.9, 5, 4), (0.0, 50, 0.9, 5, 5)])
    got = torch.empty(6, dtype=torch.int32, device="cuda")
    K().library().li_sample_leave_rows(1)
    try:
        K().sample(x, p, got)
        torch.cuda.synchronize()
    finally:
        K().library().li_sample_leave_rows(0)
    assert got[0] >= 0 and got[1:].tolist() == [-1] * 5
