"""The kernels of the 32-bit path where they can go wrong: remainders of chunks, segments and tiles, every cut of the rows,
operands that are not aligned, and attention against the general kernel with every option."""

from __future__ import annotations

import pytest
import torch

from test_kernels_gpu import make_attention_case

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24


def K():
    from litinfer_b200 import kernels
    return kernels


def on_device(c):
    """The case of make_attention_case on the GPU; pages that no request holds are full of NaN."""
    kc = torch.full((c["pages"], c["nkv"], c["page"], c["dh"]), float("nan"))
    vc = torch.full((c["pages"], c["nkv"], c["dh"], c["page"]), float("nan"))
    for s in range(c["S"]):
        t = torch.arange(c["ctx_lens"][s])
        pages, offs = c["bt"][s].long()[t // c["page"]], t % c["page"]
        kc[pages.unique()], vc[pages.unique()] = 0.0, 0.0
        kc[pages, :, offs], vc[pages, :, :, offs] = c["keys"][s], c["vals"][s]

    def ints(x):
        return torch.as_tensor(x, dtype=torch.int32).cuda()

    return dict(qkv=c["qkv"].cuda(), k_cache=kc.cuda(), v_cache=vc.cuda(), block_table=ints(c["bt"]), q_start=ints(c["q_start"]),
                ctx_lens=ints(c["ctx_lens"]), seq_of_token=ints(c["seq_of"]), positions=ints(c["pos"]))


def product(a, w, bias):
    out = torch.full((a.shape[0], w.shape[0]), float("nan"), dtype=torch.float32, device="cuda")
    K().linear(a, w, bias, out)
    return out


def unaligned(t):
    """The same values four bytes behind a 16-byte boundary."""
    buf = torch.empty(t.numel() + 4, dtype=t.dtype, device=t.device)
    view = buf[1:1 + t.numel()].view(t.shape)
    view.copy_(t)
    return view


@pytest.mark.parametrize("N", [1, 33, 160, 1536, 4800])
@pytest.mark.parametrize("Kd", [4, 7, 64, 68, 512, 1000, 1540, 4612, 8960])
def test_product_every_cut_and_its_error(N, Kd):
    g = torch.Generator(device="cuda").manual_seed(Kd * 7 + N)
    a = torch.randn((150, Kd), generator=g, device="cuda")
    w = torch.randn((N, Kd), generator=g, device="cuda")
    bias = torch.randn(N, generator=g, device="cuda")
    whole = product(a, w, bias)
    exact = a.double() @ w.double().T + bias.double()
    # a chain of 32 products, 16 chunks, the segments, the bias: each term is rounded at most that often
    depth = 32 + 16 + -(-Kd // 512) + 1
    bound = depth * EPS * (a.double().abs() @ w.double().abs().T + bias.double().abs())
    assert bool(((whole.double() - exact).abs() <= bound).all())
    for rows in (1, 3, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 70, 81, 145):
        assert torch.equal(product(a[:rows].contiguous(), w, bias), whole[:rows]), f"{rows} rows differ from 150"
    last = product(a[149:].contiguous(), w, bias)
    assert torch.equal(last, whole[149:])
    assert torch.equal(product(unaligned(a[:3]), unaligned(w), bias), whole[:3])
    assert torch.equal(product(a[:6].contiguous(), w, None) + bias, whole[:6])


OPTIONS = [
    {}, {"window": 70}, {"window": 33, "keep_first": 5}, {"window": 200, "keep_first": 150}, {"chunk": 48}, {"softcap": 20.0}, {"slopes": True},
    {"sinks": True, "window": 1}, {"gate": "heads"}, {"gate": "elements", "slopes": True, "window": 130, "keep_first": 70},
]


@pytest.mark.parametrize("heads", [(12, 2, 128, 16), (4, 4, 16, 32), (9, 1, 36, 16), (20, 2, 64, 64)])
@pytest.mark.parametrize("opt", OPTIONS, ids=str)
def test_attention_against_the_general_kernel(heads, opt):
    nh, nkv, dh, page = heads
    for q_lens, ctx_lens in (([1, 1, 1], [1, 700, 65]), ([40, 1, 70], [40, 333, 150])):
        c = on_device(make_attention_case(q_lens, ctx_lens, nh, nkv, dh, page, torch.float32, seed=3))
        T = c["qkv"].shape[0]
        g = torch.Generator(device="cuda").manual_seed(5)
        kw = {k: opt[k] for k in ("keep_first", "chunk", "softcap") if k in opt}
        if opt.get("slopes"):
            kw["slopes"] = torch.rand(nh, generator=g, device="cuda") * 0.1
        if opt.get("sinks"):
            kw["sinks"] = torch.randn(nh, generator=g, device="cuda")
        if opt.get("gate"):
            elements = opt["gate"] == "elements"
            kw.update(gate=torch.randn((T, nh * (dh if elements else 1)), generator=g, device="cuda"), gate_elements=elements)

        def run(which, rows=None):
            out = torch.full((T, nh * dh), float("nan"), device="cuda")
            K().paged_attention(c["qkv"], out, c["k_cache"], c["v_cache"], c["block_table"], c["q_start"], c["ctx_lens"], c["seq_of_token"],
                                c["positions"], nh, nkv, dh, dh ** -0.5, opt.get("window"), max(q_lens), max(ctx_lens), implementation=which, **kw)
            return out

        ref, got = run("general"), run("float32")
        # probabilities and weighted sums of up to 700 keys, each in float32 on both sides, values about 1
        assert torch.isfinite(got).all()
        assert float((got - ref).abs().max()) <= 2e-5
        assert torch.equal(run(None), got)


def test_attention_does_not_depend_on_the_batch():
    """A token alone (its units over a cluster of eight blocks) and among a hundred (one block): the same bits."""
    nh, nkv, dh, page = 12, 2, 128, 16
    c = on_device(make_attention_case([100], [2500], nh, nkv, dh, page, torch.float32, seed=8))

    def run(lo, hi):
        n = hi - lo
        out = torch.empty((n, nh * dh), device="cuda")
        K().paged_attention(c["qkv"][lo:hi].contiguous(), out, c["k_cache"], c["v_cache"], c["block_table"],
                            torch.tensor([0, n], dtype=torch.int32, device="cuda"), c["ctx_lens"], c["seq_of_token"][lo:hi].contiguous(),
                            c["positions"][lo:hi].contiguous(), nh, nkv, dh, dh ** -0.5, None, n, 2500, implementation="float32")
        return out

    whole = run(0, 100)
    for lo, hi in ((0, 1), (57, 60), (99, 100)):
        assert torch.equal(run(lo, hi), whole[lo:hi])


@pytest.mark.parametrize("longest", [700, 2500])
def test_attention_in_clusters_of_every_size(longest):
    """One block to eight a token, by how many tokens there are: the same bits."""
    nh, nkv, dh, page = 12, 2, 128, 16
    c = on_device(make_attention_case([100], [longest], nh, nkv, dh, page, torch.float32, seed=9))

    def run(n):
        out = torch.empty((n, nh * dh), device="cuda")
        K().paged_attention(c["qkv"][:n].contiguous(), out, c["k_cache"], c["v_cache"], c["block_table"], torch.tensor([0, n], dtype=torch.int32, device="cuda"),
                            c["ctx_lens"], c["seq_of_token"][:n].contiguous(), c["positions"][:n].contiguous(), nh, nkv, dh, dh ** -0.5, None, n, longest,
                            implementation="float32")
        return out

    whole, seen = run(100), set()
    for n in (1, 9, 18, 37, 70):
        seen.add(K().library().li_attention_f32_blocks(n, nh, nkv, dh))
        assert torch.equal(run(n), whole[:n])
    assert {2, 4, 8} <= seen


@pytest.mark.parametrize("rows", [3, 17, 70])
def test_more_columns_than_a_grid_has_rows_of_blocks(rows):
    """8.4 million columns, 65,537 tiles of 128, in products of small whole numbers."""
    N = 65536 * 128 + 5
    g = torch.Generator(device="cuda").manual_seed(rows)
    a = torch.randint(-3, 4, (rows, 4), generator=g, device="cuda").float()
    w = torch.randint(-3, 4, (N, 4), generator=g, device="cuda").float()
    out = torch.empty((rows, N), device="cuda")
    K().linear(a, w, None, out)
    for r in range(0, rows, 16):
        assert torch.equal(out[r], (w * a[r]).sum(1))
    assert torch.equal(out[rows - 1], (w * a[rows - 1]).sum(1))


@pytest.mark.parametrize("width", [12 * 64, 12 * 64 + 4, 12 * 64 + 33, 1500])
def test_attention_of_queries_in_rows_of_their_own(width):
    """Rows of another length than q|k|v: queries alone, or beside something else, not on 16-byte boundaries."""
    nh, nkv, dh, page = 12, 2, 64, 16
    for q_lens, ctx_lens in (([1, 1], [1, 300]), ([40, 1, 20], [40, 333, 150])):
        c = on_device(make_attention_case(q_lens, ctx_lens, nh, nkv, dh, page, torch.float32, seed=6))
        T = c["qkv"].shape[0]
        rows = torch.full((T, width), float("nan"), device="cuda")
        rows[:, :nh * dh] = c["qkv"][:, :nh * dh]

        def run(qkv, which):
            out = torch.full((T, nh * dh), float("nan"), device="cuda")
            K().paged_attention(qkv, out, c["k_cache"], c["v_cache"], c["block_table"], c["q_start"], c["ctx_lens"], c["seq_of_token"], c["positions"], nh, nkv, dh,
                                dh ** -0.5, None, max(q_lens), max(ctx_lens), implementation=which)
            return out

        got = run(rows, "float32")
        assert torch.equal(got, run(c["qkv"], "float32"))
        assert float((got - run(rows, "general")).abs().max()) <= 2e-5



@pytest.mark.parametrize("tokens", [1, 40])
@pytest.mark.parametrize("lost", [(64, 65), (32, 64), (0, 40), (0, 65)])
def test_scores_of_minus_infinity(lost, tokens):
    """Keys whose scores are minus infinity have no weight, also where a unit of 32 keys has no others; a token that sees nothing
    else has no softmax (the same tokens of one block and of a cluster of them)."""
    nh, nkv, dh, page, ctx = 6, 2, 64, 16, 65
    c = make_attention_case([tokens], [ctx], nh, nkv, dh, page, torch.float32, seed=14)
    c["qkv"].view(tokens, -1, dh)[:, :nh, 0].abs_().add_(0.1)
    keys, vals = c["keys"][0], c["vals"][0]
    keys[lost[0]:lost[1], :, 0] = float("-inf")
    q = c["qkv"][:, :nh * dh].view(tokens, nh, dh).double()
    scores = torch.einsum("thd,khd->thk", q, keys.double().repeat_interleave(nh // nkv, 1)) * dh ** -0.5
    unseen = torch.arange(ctx)[None, :] > torch.arange(ctx - tokens, ctx)[:, None]
    exact = torch.einsum("thk,khd->thd", scores.masked_fill(unseen[:, None], float("-inf")).softmax(-1), vals.double().repeat_interleave(nh // nkv, 1))
    d = on_device(c)
    out = torch.empty((tokens, nh * dh), device="cuda")
    K().paged_attention(d["qkv"], out, d["k_cache"], d["v_cache"], d["block_table"], d["q_start"], d["ctx_lens"], d["seq_of_token"], d["positions"], nh, nkv, dh,
                        dh ** -0.5, None, tokens, ctx, implementation="float32")
    got = out.double().cpu().view(tokens, nh, dh)
    assert torch.equal(got.isnan(), exact.isnan())
    assert float((got - exact).nan_to_num().abs().max()) <= 2e-5


@pytest.mark.parametrize("tile", [(4, 1, 1), (4, 2, 3), (6, 1, 4), (6, 2, 1), (8, 1, 2), (8, 1, 6), (8, 2, 5), (10, 1, 1), (10, 2, 8), (10, 1, 8)], ids=str)
@pytest.mark.parametrize("M,N,Kd", [(17, 130, 1540), (81, 300, 260), (150, 257, 4612), (97, 1536, 512), (33, 4, 36)])
def test_product_gives_the_same_bits_in_every_tile(tile, M, N, Kd):
    """Rows a thread, groups of threads and clusters that share a tile's halves of segments: a token alone, through the streaming kernel,
    has the bits of all of them."""
    g = torch.Generator(device="cuda").manual_seed(Kd + M)
    a, w = torch.randn((M, Kd), generator=g, device="cuda"), torch.randn((N, Kd), generator=g, device="cuda")
    bias = torch.randn(N, generator=g, device="cuda")
    lib = K().library()
    by_size = product(a, w, bias)
    assert lib.li_linear_f32_force_tile(*tile) == 0
    try:
        assert torch.equal(product(a, w, bias), by_size)
    finally:
        lib.li_linear_f32_force_tile(0, 0, 0)
    assert torch.equal(product(a[M - 1:].contiguous(), w, bias), by_size[M - 1:])
    assert lib.li_linear_f32_force_tile(8, 1, 3) != 0 and lib.li_linear_f32_force_tile(5, 1, 1) != 0       # segments' halves come in pairs
