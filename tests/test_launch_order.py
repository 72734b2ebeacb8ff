"""Kernels with tensor memory let the kernel behind them start only once they hold their columns.

The streaming product takes its columns before it waits for the kernel before it.  If that kernel's CTAs had not allocated yet
and found the product's CTA beside them on a multiprocessor, each would wait for the other, and ``tcgen05.alloc`` waits without
a limit."""

from __future__ import annotations

import ctypes
import re
from pathlib import Path

import pytest
import torch

CSRC = Path(__file__).resolve().parent.parent / "litinfer_b200" / "csrc"


def kernels_with_tensor_memory():
    for f in sorted(CSRC.glob("*.cu")):
        parts = re.split(r"^__global__ ", re.sub(r"//[^\n]*", "", f.read_text()), flags=re.M)
        for body in parts[1:]:
            body = body[:body.find("\n}\n")]
            if "tcgen05.alloc" in body:
                yield f.name, body


def test_dependents_are_let_go_behind_the_allocation():
    found = list(kernels_with_tensor_memory())
    assert {name for name, _ in found} == {"attention_tcgen05.cu", "gemm_tcgen05.cu", "gemm_tcgen05_persistent.cu", "gemv_tcgen05.cu"}
    for name, body in found:
        allocated, released = body.rfind("tcgen05.alloc"), body.find("pdl_launch_dependents()")
        assert body.count("pdl_launch_dependents()") == 1, name
        assert released > allocated, f"{name}: the dependents are let go before tensor memory is taken"
        # in the same run of statements: an allocation inside a lambda that a warp calls later is not one that has happened
        assert "};" not in body[allocated:released], f"{name}: the dependents are let go apart from the allocation"


@pytest.mark.gpu
def test_streaming_product_behind_attention_with_heads_of_64():
    """One portion of 64 tokens, heads of 64, and an o product on the streaming tcgen05 kernel, launched one behind the other."""
    from test_f32_gpu import on_device
    from test_kernels_gpu import make_attention_case

    from litinfer_b200 import kernels as K

    nh, nkv, dh, n, ctx, width = 64, 8, 64, 64, 700, 3072
    c = on_device(make_attention_case([n], [ctx], nh, nkv, dh, 16, torch.float32, seed=4))
    for k in ("qkv", "k_cache", "v_cache"):
        c[k] = torch.nan_to_num(c[k]).to(torch.bfloat16)
    w = (torch.randn((width, nh * dh), generator=torch.Generator().manual_seed(1)) * 0.02).to(torch.bfloat16).cuda()

    def attention(out):
        K.paged_attention(c["qkv"], out, c["k_cache"], c["v_cache"], c["block_table"], c["q_start"], c["ctx_lens"], c["seq_of_token"], c["positions"], nh, nkv, dh,
                          dh ** -0.5, None, n, ctx, implementation="prefill_tcgen05")

    alone = torch.empty((n, nh * dh), dtype=torch.bfloat16, device="cuda")
    attention(alone)
    torch.cuda.synchronize()
    ref = alone.float() @ w.float().T
    outs = [(torch.empty_like(alone), torch.empty((n, width), dtype=torch.bfloat16, device="cuda")) for _ in range(50)]
    for att, y in outs:
        attention(att)
        K.linear(att, w, None, y)
    torch.cuda.synchronize()
    for att, y in outs:
        assert torch.equal(att, alone)
        # float32 sums of 4,096 terms and one rounding to bfloat16
        assert bool(((y.float() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4).all())


def dependent_launches(fn):
    """Of the launches of a call: (all that have one before them, those that may begin while it still runs)."""
    fn()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        fn()
    runtime, handle, n = ctypes.CDLL("libcudart.so.12"), ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t()
    assert runtime.cudaGraphGetEdges_v2(handle, None, None, None, ctypes.byref(n)) == 0
    ends, data = [(ctypes.c_void_p * n.value)() for _ in range(2)], (ctypes.c_ubyte * (8 * n.value))()
    assert runtime.cudaGraphGetEdges_v2(handle, ends[0], ends[1], data, ctypes.byref(n)) == 0
    return n.value, sum(data[8 * i + 2] == 1 for i in range(n.value))          # the third byte: programmatic


@pytest.mark.gpu
@pytest.mark.parametrize("heads,options,early", [((12, 2, 128), {}, False), ((16, 2, 64), {}, False), ((24, 2, 128), {}, True), ((14, 2, 80), {}, True),
                                                 ((12, 2, 128), {"softcap": 20.0}, True)], ids=str)
def test_whole_contexts_start_early_but_for_the_column_form(heads, options, early):
    """Many sequences, a CTA a whole context: only the form that was measured to lose by it waits for its launch."""
    from test_kernels_gpu import make_attention_case

    from litinfer_b200 import kernels as K

    nh, nkv, dh = heads
    S, ctx = 80, 300
    c = make_attention_case([1] * S, [ctx] * S, nh, nkv, dh, 16, torch.bfloat16, seed=2)
    caches = [torch.randn((c["pages"], nkv, *shape), device="cuda").to(torch.bfloat16) for shape in ((16, dh), (dh, 16))]
    ints = [torch.as_tensor(c[k], dtype=torch.int32).cuda() for k in ("bt", "q_start", "ctx_lens", "seq_of", "pos")]
    qkv, out = c["qkv"].cuda(), torch.empty((S, nh * dh), dtype=torch.bfloat16, device="cuda")

    def twice():
        for _ in range(2):
            K.paged_attention(qkv, out, *caches, *ints, nh, nkv, dh, dh ** -0.5, None, 1, ctx, **options)

    assert dependent_launches(twice) == (1, 1 if early else 0)

