"""Branches that a rule on sizes or options chooses, against the general way to the same result."""

from __future__ import annotations

import pytest
import torch

import test_kernels_gpu as T

pytestmark = pytest.mark.gpu


def K():
    from litinfer_b200 import kernels
    return kernels


def params(rows):
    """(temperature, top_k, top_p, seed, output index) per row, as the sampler packs them."""
    out = torch.zeros((len(rows), 6), dtype=torch.int32)
    f = out.view(torch.float32)
    for i, (temperature, top_k, top_p, seed, index) in enumerate(rows):
        f[i, 0], out[i, 1], f[i, 2], out[i, 3], out[i, 5] = temperature, top_k, top_p, seed, index
    return out.cuda()


@pytest.mark.parametrize("R", [64, 32, 7])
@pytest.mark.parametrize("V", [16384, 16387, 50001, 151936])
def test_top_k_by_a_cluster_is_the_general_kernels_token(V, R):
    """Up to 64 rows the rows with a small top-k go to the kernel with several blocks a row; 65 and more go to the general one."""
    g = torch.Generator(device="cuda").manual_seed(V + R)
    x = torch.randn((R, V), generator=g, device="cuda") * 2.5
    options = [(0.7, 50, 0.8), (1.0, 256, 1.0), (0.3, 2, 0.999), (1.3, 20, 0.1), (1.0, 257, 0.9), (0.0, 50, 0.8), (1.0, 1, 1.0), (0.9, 0, 0.9), (1.0, 0, 1.0),
               (1e-6, 50, 0.8), (1e30, 50, 0.8)]
    rows = [(*options[i % len(options)], 100 + i, i) for i in range(R)]
    # rows in which thresholds meet equal values, masks, infinities and no numbers (the options of those rows differ with R)
    x[1] = x[1].round()                                  # hundreds of equal values at the threshold
    x[2, V // 3:] = torch.finfo(torch.float32).min
    x[3, 100:] = float("-inf")
    x[4] = 1.5
    x[5, 17] = float("inf")
    x[6, V - 1] = float("nan")
    if R > 8:
        rows[8:14] = [(0.7, 50, 0.8, 5, 1)] * 6
        x[8] = x[8].round()
        x[9, 30:] = torch.finfo(torch.float32).min       # fewer than top_k that are not masked
        x[10] = 0.0
        x[11, 3] = float("nan")
        x[12, V - 1] = float("inf")
        x[13] = float("-inf")
    p = params(rows)
    got = torch.full((R,), -7, dtype=torch.int32, device="cuda")
    K().sample(x, p, got)
    more = -(-65 // R)
    ref = torch.full((R * more,), -7, dtype=torch.int32, device="cuda")
    K().sample(x.repeat(more, 1), p.repeat(more, 1), ref)
    assert got.tolist() == ref[:R].tolist()


@pytest.mark.parametrize("cfg", [(28, 4, 128, 264, 1800), (40, 8, 128, 136, 1300), (28, 4, 128, 264, 2049)])
def test_rotation_in_the_epilogue_of_wide_long_steps(cfg):
    """q|k|v of so many rows that the plain product would go to the persistent kernel."""
    T.test_linear_rope_kv_fused(torch.bfloat16, cfg)


# (tiles of 256 x 256: 180, 153 and 200, then 119, 120 with less than 8,192 columns of k and with more, 150)
@pytest.mark.parametrize("shape", [(640, 15360, 4224), (520, 13000, 4168), (769, 12800, 5120), (1792, 4352, 4168), (2048, 3840, 4168), (2048, 3840, 8200),
                                   (2560, 3840, 8200)])
@pytest.mark.parametrize("epilogue", [None, "swiglu"])
def test_product_with_a_long_k_on_either_side_of_the_persistent_rule(shape, epilogue):
    M, N, Kd = shape
    N -= N % 16
    g = torch.Generator(device="cuda").manual_seed(M)
    a = torch.randn((M, Kd), generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn((N, Kd), generator=g, device="cuda") * Kd ** -0.5).to(torch.bfloat16)
    ref = a.float() @ w.float().T
    if epilogue:
        r = ref.view(M, N // 16, 2, 8)
        ref = (torch.nn.functional.silu(r[:, :, 0]) * r[:, :, 1]).reshape(M, N // 2)
    out = torch.full(ref.shape, float("nan"), dtype=torch.bfloat16, device="cuda")
    K().linear(a, w, None, out, epilogue=epilogue)
    assert torch.isfinite(out).all()
    # one rounding to bfloat16 of a float32 sum; the sums themselves are within a few 1e-6 of each other
    assert bool(((out.float() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-3).all())


@pytest.mark.parametrize("tokens", [1, 9, 16, 17, 33, 64])
# (few heads: on the register-fed kernel but for more than 32 tokens with rows of 8,192)
@pytest.mark.parametrize("cfg", [(28, 4, 128, 3136), (40, 8, 128, 4104), (16, 2, 128, 4096), (4, 1, 128, 4104), (4, 1, 128, 8200)])
def test_rotation_in_the_epilogue_of_the_streaming_tcgen05_product(cfg, tokens):
    """q|k|v of few tokens with long rows: a tile a head, its splits of k merged within a cluster."""
    T.test_linear_rope_kv_fused(torch.bfloat16, (*cfg, tokens))


@pytest.mark.parametrize("shape", [(1536, 8960), (128, 8192), (200, 4096), (3584, 3584), (5120, 4160)])
def test_splits_of_k_in_clusters_do_not_depend_on_the_batch(shape):
    """Each number of tokens that shares a token tile (16, 32, 64) gives a token the same bits, whoever merges its splits."""
    N, Kd = shape
    g = torch.Generator(device="cuda").manual_seed(N)
    a = torch.randn((64, Kd), generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn((N, Kd), generator=g, device="cuda") * Kd ** -0.5).to(torch.bfloat16)
    bias = torch.randn(N, generator=g, device="cuda")
    ref = a.float() @ w.float().T + bias
    for tile, counts in ((16, (1, 2, 5, 16)), (32, (17, 31, 32)), (64, (33, 50, 64))):
        whole = None
        for m in reversed(counts):
            out = torch.full((m, N), float("nan"), device="cuda")
            K().linear_with("gemv_tcgen05", a[:m].contiguous(), w, bias, out)
            assert float((out - ref[:m]).abs().max()) <= 1e-4          # float32 sums of Kd terms of size Kd ** -0.5
            if whole is not None:
                assert torch.equal(out, whole[:m]), (tile, m)
            whole = out if whole is None else whole


@pytest.mark.parametrize("heads", [(12, 2, 128), (24, 2, 64), (4, 1, 80)])
@pytest.mark.parametrize("options", [{}, {"window": 40}, {"window": 40, "keep_first": 20}, {"window": 300, "sinks": True}, {"chunk": 128, "gate": True}], ids=str)
def test_a_unit_that_is_its_sequences_only_one(heads, options):
    """Contexts, or what a window or a chunk leaves of them, within 256 keys at an absolute place: nothing is merged over units; beside
    them sequences of two units and more, in the same launch."""
    from test_f32_gpu import on_device

    nh, nkv, dh = heads
    ctx_lens = [1, 255, 256, 257, 511, 513, 600, 700]        # alone without options: the first three; with a window of 40 all but 257, 513
    c = on_device(T.make_attention_case([1] * 8, ctx_lens, nh, nkv, dh, 16, torch.float32, seed=12))
    for k in ("qkv", "k_cache", "v_cache"):
        c[k] = torch.nan_to_num(c[k]).to(torch.bfloat16)
    kw = {k: v for k, v in options.items() if k in ("keep_first", "chunk")}
    if "sinks" in options:
        kw["sinks"] = torch.linspace(-1, 2, nh, device="cuda")
    if "gate" in options:
        kw["gate"] = torch.linspace(-3, 3, 8 * nh, device="cuda").view(8, nh).to(torch.bfloat16)

    def run(dtype, which):
        q, k, v = (c[x].to(dtype) for x in ("qkv", "k_cache", "v_cache"))
        out = torch.full((8, nh * dh), float("nan"), dtype=dtype, device="cuda")
        more = {n: x.to(dtype) if n == "gate" else x for n, x in kw.items()}
        K().paged_attention(q, out, k, v, c["block_table"], c["q_start"], c["ctx_lens"], c["seq_of_token"], c["positions"], nh, nkv, dh, dh ** -0.5,
                            options.get("window"), 1, max(ctx_lens), implementation=which, **more)
        return out.float()

    got, ref = run(torch.bfloat16, "decode"), run(torch.float32, "general")
    # probabilities rounded to bfloat16 (2^-9 of each, values about 1) and the result once more
    assert float((got - ref).abs().max()) <= 2.0 ** -8 * float(ref.abs().max()) + 2.0 ** -8



@pytest.mark.parametrize("splits", [2, 3, 4, 5, 8])
@pytest.mark.parametrize("M", [1, 2, 9, 16, 17, 31, 33, 50, 64])
def test_streaming_product_with_its_splits_in_a_cluster(splits, M):
    """Tokens and CTAs that do not come out in fours: the product and its sum into the residual stream."""
    N, Kd = 300, 1048
    a = T.rnd(M, Kd, dtype=torch.bfloat16, seed=100 + M)
    w = T.rnd(N, Kd, dtype=torch.bfloat16, seed=splits, scale=0.05)
    bias = T.rnd(N, seed=13)

    def bound(a, w):
        # exact products, added in float32 sixteen at a time: each of these sums may lose a last place of what has come together
        return a.shape[1] / 16 * 2.0 ** -23 * float((a.abs().float() @ w.abs().float().T).max()) + 1e-5

    exact = a.double() @ w.double().T + bias.double()
    K().library().li_gemv_tcgen05_force_ksplit(splits)
    try:
        out = torch.full((M, N), float("nan"), dtype=torch.float32, device="cuda")
        K().linear_with("gemv_tcgen05", a, w, bias, out)
        assert float((out - exact).abs().max()) <= bound(a, w)
        # a product that the rule sends there, into the residual stream
        Nr, Kr = 1152, 4160
        a, w = T.rnd(M, Kr, dtype=torch.bfloat16, seed=200 + M), T.rnd(Nr, Kr, dtype=torch.bfloat16, seed=splits + 20, scale=0.05)
        x, bias, norm = T.rnd(M, Nr, seed=5), T.rnd(Nr, seed=6), T.rnd(Nr, seed=7)
        want = x.double() + a.double() @ w.double().T + bias.double()
        h = torch.empty((M, Nr), dtype=torch.bfloat16, device="cuda")
        parts = K().linear_add_scaled_parts(a, w, x, h)
        assert parts == Nr // 128
        ssq = torch.full((M, parts), float("nan"), device="cuda")
        K().linear_add_scaled(a, w, bias, x, norm, h, ssq)
        assert float((x - want).abs().max()) <= bound(a, w)
        assert float((h - want * norm.double()).abs().max()) <= 2.0 ** -8 * float((want * norm.double()).abs().max()) + bound(a, w) * float(norm.abs().max())
        assert torch.allclose(ssq.double(), (want * want).view(M, parts, 128).sum(2), rtol=1e-3)
    finally:
        K().library().li_gemv_tcgen05_force_ksplit(0)
    assert K().library().li_tcgen05_status() == 0


@pytest.mark.parametrize("heads", [(20, 4), (28, 4), (40, 8), (60, 8), (90, 9)], ids=str)
@pytest.mark.parametrize("tokens", [1, 7, 16, 30, 45, 64])
def test_rotation_in_the_streaming_product_of_every_split(heads, tokens):
    """q|k|v with four, three, two CTAs a cluster or none: every CTA rotates the tokens it finishes."""
    nh, nkv = heads
    T.test_linear_rope_kv_fused(torch.bfloat16, (nh, nkv, 128, tokens, 4160))


def forced(tile, width=0):
    lib = K().library()
    lib.li_tcgen05_force_tile(tile)
    assert lib.li_tcgen05_tokens_force_width(width) == 0


@pytest.mark.parametrize("width", [0, 32, 96, 256, 288, 416, 512])
@pytest.mark.parametrize("M", [1, 33, 129, 300, 544, 1100])
@pytest.mark.parametrize("N,Kd", [(256, 64), (384, 520), (1000, 256), (1026, 72), (1333, 200), (2064, 1536)])
def test_product_with_tokens_as_columns(N, Kd, M, width):
    """Tiles of every kind of width, rows of w and tokens that fill no tile, odd row lengths: against the tiles of 128 x 128, whose sums
    are the same ones in the same order."""
    a = T.rnd(M, Kd, dtype=torch.bfloat16, seed=M)
    w = T.rnd(N, Kd, dtype=torch.bfloat16, seed=N, scale=0.1)
    bias = T.rnd(N, seed=5)
    try:
        for epilogue, dtype in ((None, torch.bfloat16), (None, torch.float32), ("swiglu", torch.bfloat16), ("geglu", torch.bfloat16)):
            if epilogue and N % 16:
                continue
            out = torch.full((M, N // 2 if epilogue else N), float("nan"), dtype=dtype, device="cuda")
            ref = torch.full_like(out, float("nan"))
            forced(10, width)
            K().linear_with("tcgen05", a, w, None if epilogue else bias, out, epilogue)
            forced(1)
            K().linear_with("tcgen05", a, w, None if epilogue else bias, ref, epilogue)
            T.close(out, ref, dtype, f"tokens as columns {epilogue} {dtype}")
    finally:
        forced(0)
    assert K().library().li_tcgen05_status() == 0


@pytest.mark.parametrize("first", [0, 5])
@pytest.mark.parametrize("heads", [(28, 4), (3, 2)], ids=str)
@pytest.mark.parametrize("tokens", [70, 200, 530])
def test_rotation_with_tokens_as_columns(heads, tokens, first):
    """A last tile with one head, places in the cache that follow one another (values leave eight at a time where they are aligned),
    that do not, and that are not there; the rest of the cache is left alone."""
    nh, nkv = heads
    N, width, page = (nh + 2 * nkv) * 128, 264, 16
    pages = (tokens + first) // page + 3
    a, w = T.rnd(tokens, width, dtype=torch.bfloat16, seed=1), T.rnd(N, width, dtype=torch.bfloat16, seed=2, scale=0.1)
    bias = T.rnd(N, seed=3)
    positions = (torch.arange(tokens, dtype=torch.int32) % 300).cuda()
    denom = torch.pow(torch.tensor(10000.0), torch.arange(64, dtype=torch.float32) / 64).cuda()
    slots = torch.arange(first, first + tokens, dtype=torch.int32)
    slots[40:48] = slots[40:48].flip(0)
    slots[63] = -1
    table = torch.empty(tokens, 64, 2, device="cuda")
    K().rope_table(positions, denom, table)
    results = []
    try:
        for tile in (10, 11):
            forced(tile)
            qkv = torch.zeros(tokens, N, dtype=torch.bfloat16, device="cuda")
            kc = torch.full((pages, nkv, page, 128), 3.0, dtype=torch.bfloat16, device="cuda")
            vc = torch.full((pages, nkv, 128, page), 3.0, dtype=torch.bfloat16, device="cuda")
            K().linear_rope_kv(a, w, bias, qkv, positions, denom, 128, slots.cuda(), kc, vc, nh, nkv, 128, True, cos_sin=table)
            results.append((qkv[:, :nh * 128], kc, vc))
    finally:
        forced(0)
    for got, ref in zip(*results):
        assert torch.equal(got == 3.0, ref == 3.0)
        T.close(got, ref, torch.bfloat16, "rotation with tokens as columns")
    assert K().library().li_tcgen05_status() == 0


@pytest.mark.parametrize("window", [None, 150])
@pytest.mark.parametrize("dh", [64, 128])
def test_portions_with_a_cap_and_slopes_on_tensor_memory_tiles(dh, window):
    """Both changes of a score at once, against the tiles that took them alone before: small scores and ones beyond the cap."""
    from test_f32_gpu import on_device

    nh, nkv = 6, 2
    c = on_device(T.make_attention_case([130, 64, 5], [700, 64, 333], nh, nkv, dh, 16, torch.float32, seed=dh))
    for k in ("qkv", "k_cache", "v_cache"):
        c[k] = torch.nan_to_num(c[k]).to(torch.bfloat16)
    slopes = torch.tensor([2.0 ** -(h + 1) for h in range(nh)], device="cuda")
    outs = []
    for scale in (dh ** -0.5, 3.0):
        for implementation in ("prefill_tcgen05", "prefill"):
            out = torch.full((199, nh * dh), float("nan"), dtype=torch.bfloat16, device="cuda")
            K().paged_attention(c["qkv"], out, c["k_cache"], c["v_cache"], c["block_table"], c["q_start"], c["ctx_lens"], c["seq_of_token"], c["positions"], nh,
                                nkv, dh, scale, window, 130, 700, softcap=5.0, slopes=slopes, implementation=implementation)
            outs.append(out)
        T.close(outs[-2], outs[-1], torch.bfloat16, f"cap and slopes, scale {scale}")
    assert K().library().li_tcgen05_status() == 0


@pytest.mark.parametrize("M", [1, 8, 9, 16])
@pytest.mark.parametrize("N,Kd", [(2384, 1536), (2369, 2048), (4800, 1544), (2400, 1992)])
def test_streaming_product_of_one_round_gives_the_bits_of_its_parts(M, N, Kd):
    """More CTAs than multiprocessors, whose warps hold all of their weights at once, against parts of the matrix that go in one wave."""
    g = torch.Generator(device="cuda").manual_seed(N + Kd + M)
    a, w = (torch.randn(n, Kd, generator=g, device="cuda").to(torch.bfloat16) for n in (M, N))
    bias = torch.randn(N, generator=g, device="cuda")
    outs = {}
    for dt in (torch.bfloat16, torch.float32):
        whole = torch.full((M, N), 7.0, device="cuda", dtype=dt)
        K().linear_with("gemv", a, w, bias, whole)
        for n0 in range(0, N, 1200):
            n1 = min(n0 + 1200, N)
            part = torch.full((M, n1 - n0), 7.0, device="cuda", dtype=dt)
            K().linear_with("gemv", a, w[n0:n1], bias[n0:n1].clone(), part)
            assert torch.equal(whole[:, n0:n1], part)
        outs[dt] = whole
    # products are exact in float; K + 32 roundings of partial sums that the sum of magnitudes bounds
    exact = a.double() @ w.double().T + bias.double()
    bound = (Kd + 32) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T + bias.double().abs())
    assert bool(((outs[torch.float32].double() - exact).abs() <= bound).all())
    if N % 16 == 0:
        whole = torch.full((M, N // 2), 7.0, device="cuda", dtype=torch.bfloat16)
        K().linear_with("gemv", a, w, None, whole, epilogue="swiglu")
        for n0 in range(0, N, 1200):
            n1 = min(n0 + 1200, N)
            part = torch.full((M, (n1 - n0) // 2), 7.0, device="cuda", dtype=torch.bfloat16)
            K().linear_with("gemv", a, w[n0:n1], None, part, epilogue="swiglu")
            assert torch.equal(whole[:, n0 // 2:n1 // 2], part)
