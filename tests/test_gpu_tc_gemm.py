"""The tcgen05 matrix product alone against a float32 product of the same bfloat16 inputs:
every epilogue, token counts on both sides of every tile size, widths that are no multiple of
the tile, with and without split-K."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rnd(*shape, seed=0, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(torch.bfloat16)


def rel(a, b):
    return float((a.float().cpu() - b.float().cpu()).abs().max()) / max(float(b.abs().max()), 1e-30)


SHAPES = [(1, 128, 64), (8, 384, 200), (16, 100, 72), (17, 3072, 2048), (64, 2048, 2048), (100, 640, 520),
          (128, 256, 8192), (65, 2048, 4096), (96, 200, 1024), (300, 1000, 264), (1, 128256, 256), (8, 2048, 8192), (600, 512, 1024),
          # gate/up with the tokens on the accumulator's rows: tiles of 128 weight rows (many tiles) and of 64 (few)
          (900, 1536, 192), (40, 1000, 264),
          # steps of at most 8 tokens with K a multiple of 32 and N of 16 run the weight-streaming kernel
          # (one to four chunks of K per warp held in registers, or more, fetched chunk by chunk)
          (1, 48, 96), (3, 2048, 2048), (8, 8192, 2048), (8, 2048, 3072), (5, 3072, 4096), (8, 4096, 14336),
          (7, 208, 160), (2, 16, 32), (9, 2048, 2048)]


@pytest.mark.parametrize("T,N,K", SHAPES)
@pytest.mark.parametrize("split", [True, False])
def test_tc_gemm_epilogues(T, N, K, split):
    from rllm_b200.kernels import ops, sm100
    x, w = rnd(T, K, seed=1), rnd(2 * N, K, seed=2, scale=K ** -0.5)
    xd, wd = x.to(DEV), w.to(DEV)
    w1 = wd[:N].contiguous()
    ref = x.float() @ w[:N].float().t()
    up = x.float() @ w[N:].float().t()
    assert rel(sm100.gemm(xd, w1, ops.EPI_STORE, split=split), ref) <= 6e-3
    out32 = sm100.gemm(xd, w1, ops.EPI_STORE_F32, split=split)
    assert out32.dtype == torch.float32 and rel(out32, ref) <= 2e-5
    res = torch.randn(T, N, generator=torch.Generator().manual_seed(3))
    got = sm100.gemm(xd, w1, ops.EPI_ACCUM_F32, out=res.to(DEV).clone(), split=split)
    assert rel(got, res + ref) <= 2e-5
    want = ref / (1 + torch.exp(-ref)) * up
    assert rel(sm100.gemm(xd, wd, ops.EPI_SWIGLU, split=split), want) <= 6e-3
    sm100.check_error(DEV)
    # the same call again gives the same bits (the ranges of K are summed in rank order)
    again = sm100.gemm(xd, w1, ops.EPI_STORE_F32, split=split)
    assert torch.equal(again, out32)


@pytest.mark.parametrize("seed", range(6))
def test_products_of_random_sizes(seed):
    """Portions of 65 to 900 tokens against weights of any height and depth the kernels take (steps of 8):
    token tiles of every width the launcher may choose, partial tiles on every edge, an output with a
    row stride of its own, with and without the kernel that puts the tokens on the accumulator's rows."""
    import random
    from rllm_b200.kernels import ops, sm100
    r = random.Random(seed)
    for i in range(4):
        # the first of each seed under 128 tokens: one partial tile of the kernel with the tokens on the rows
        T, N, K = r.randint(65, 127 if i == 0 else 900), 8 * r.randint(1, 90), 8 * r.randint(1, 80)
        x, w = rnd(T, K, seed=seed + 1), rnd(2 * N, K, seed=seed + 2, scale=K ** -0.5)
        xd, wd = x.to(DEV), w.to(DEV)
        w1 = wd[:N].contiguous()
        ref = x.float() @ w[:N].float().t()
        up = x.float() @ w[N:].float().t()
        tag = f"T={T} N={N} K={K} plan={sm100.plan(ops.EPI_STORE, T, N, K)}"
        assert rel(sm100.gemm(xd, w1, ops.EPI_STORE), ref) <= 6e-3, tag
        assert rel(sm100.gemm(xd, w1, ops.EPI_STORE_F32), ref) <= 2e-5, tag
        # the residual as a view into a wider buffer: the untouched columns stay as they were
        wide = torch.randn(T, N + 24, generator=torch.Generator().manual_seed(seed)).to(DEV)
        keep = wide.clone()
        res = wide[:, 8: 8 + N]
        got = sm100.gemm(xd, w1, ops.EPI_ACCUM_F32, out=res)
        assert rel(got, keep[:, 8: 8 + N].cpu() + ref) <= 2e-5, tag
        assert torch.equal(wide[:, :8], keep[:, :8]) and torch.equal(wide[:, 8 + N:], keep[:, 8 + N:]), tag
        want = ref / (1 + torch.exp(-ref)) * up
        for rows_on in (True, False):
            sm100.set_token_rows(rows_on)
            try:
                assert rel(sm100.gemm(xd, wd, ops.EPI_SWIGLU), want) <= 6e-3, tag + f" token rows {rows_on}"
            finally:
                sm100.set_token_rows(True)
        sm100.check_error(DEV)


@pytest.mark.parametrize("seed", range(4))
def test_rotary_epilogue_of_random_sizes(seed):
    """Long portions through the product with rotation and cache write, at random head counts, head sizes
    of 16 to 128, page sizes and depths, against the plain formulas; scattered slots, some tokens unwritten."""
    import random
    import plain_llama as P
    from rllm_b200.kernels import ops, sm100
    r = random.Random(100 + seed)
    for _ in range(3):
        hd = r.choice([16, 32, 64, 128])
        nkv = r.randint(1, 4)
        nh = nkv * r.randint(1, 4)
        T, K, page = r.randint(65, 700), 8 * r.randint(2, 60), r.choice([4, 8, 16, 32])
        N = (nh + 2 * nkv) * hd
        x, w = rnd(T, K, seed=seed + 1), rnd(N, K, seed=seed + 2, scale=K ** -0.5)
        g = torch.Generator().manual_seed(seed)
        positions = torch.randint(0, 9000, (T,), generator=g, dtype=torch.int32)
        inv_freq = P.rope_inv_freq(hd, 500000.0, None)
        pages = (T + page - 1) // page + 2
        slots = torch.randperm(pages * page, generator=g)[:T].to(torch.int32)
        slots[r.randrange(T)] = -1
        kc = torch.zeros(pages, nkv, page, hd, dtype=torch.bfloat16, device=DEV)
        vc = torch.zeros_like(kc)
        table = ops.rope_table(positions.to(DEV), inv_freq.to(DEV), T)
        out = sm100.gemm_qkv_rope(x.to(DEV), w.to(DEV), positions.to(DEV), inv_freq.to(DEV), slots.to(DEV), kc, vc,
                                  nh, nkv, hd, page, hd, table=table)
        sm100.check_error(DEV)
        ref = x.float() @ w.float().t()
        q = P.rope(ref[:, : nh * hd].view(T, nh, hd), positions, inv_freq)
        k = P.rope(ref[:, nh * hd: (nh + nkv) * hd].view(T, nkv, hd), positions, inv_freq)
        v = ref[:, (nh + nkv) * hd:].view(T, nkv, hd)
        scale = float(ref.abs().max())
        tag = f"T={T} K={K} heads {nh}/{nkv} of {hd}, pages of {page}"
        got = out.float().cpu()
        assert float((got[:, : nh * hd].view(T, nh, hd) - q).abs().max()) <= 6e-3 * scale, tag
        assert float((got[:, nh * hd: (nh + nkv) * hd].view(T, nkv, hd) - k).abs().max()) <= 6e-3 * scale, tag
        assert float((got[:, (nh + nkv) * hd:].view(T, nkv, hd) - v).abs().max()) <= 6e-3 * scale, tag
        kcc, vcc = kc.float().cpu(), vc.float().cpu()
        want_k, want_v = torch.zeros_like(kcc), torch.zeros_like(vcc)
        for t in range(T):
            if slots[t] >= 0:
                want_k[int(slots[t]) // page, :, int(slots[t]) % page] = k[t]
                want_v[int(slots[t]) // page, :, int(slots[t]) % page] = v[t]
        assert float((kcc - want_k).abs().max()) <= 6e-3 * scale and float((vcc - want_v).abs().max()) <= 6e-3 * scale, tag
        assert float(kcc[want_k == 0].abs().sum()) == 0.0, tag            # nothing beside the written slots


NORM_SHAPES = [(1, 128, 64), (8, 384, 200), (16, 100, 72), (17, 3072, 2048), (33, 640, 520), (64, 2048, 2048),
               (5, 128256, 256), (8, 2048, 8192), (64, 256, 1000),
               (3, 2048, 2048), (8, 8192, 2048), (8, 3072, 3072), (6, 256, 4096), (2, 48, 96), (4, 128256, 2048)]


@pytest.mark.parametrize("T,N,K", NORM_SHAPES)
@pytest.mark.parametrize("split,g_dtype", [(True, torch.float32), (False, torch.bfloat16)])
def test_tc_gemm_with_rmsnorm_in_front(T, N, K, split, g_dtype):
    """rmsnorm(h[rows]) W^T in one kernel, every epilogue it has, against (a) the same formula with
    the kernel's one rounding (bf16 of h * g) and float elsewhere, tightly, and (b) the plain float
    formula, within bfloat16 rounding. h has a few large columns, as a residual stream has; the rows
    are picked out of a larger h through an index list in half of the cases."""
    from rllm_b200.kernels import ops, sm100
    g0 = torch.Generator().manual_seed(11)
    R = T + 5
    h = torch.randn(R, K, generator=g0)
    h[:, :: max(1, K // 7)] *= 25.0
    gw = (1.0 + 0.3 * torch.randn(K, generator=g0)).to(g_dtype)
    eps = 1e-5 if split else 1e-6
    w = rnd(2 * N, K, seed=2, scale=K ** -0.5)
    rows = torch.randperm(R, generator=g0)[:T].to(torch.int32) if split else None
    hs = h[rows.long()] if rows is not None else h[:T]
    rstd = torch.rsqrt((hs.double() ** 2).mean(-1, keepdim=True) + eps).float()
    xb = (hs * gw.float()).to(torch.bfloat16).float()                  # the kernel's rounding point
    x_plain = hs * rstd * gw.float()
    hd_, wd = (h if rows is not None else h[:T].contiguous()).to(DEV), w.to(DEV)
    rd = rows.to(DEV) if rows is not None else None
    gd = gw.to(DEV)
    w1 = wd[:N].contiguous()
    same = (xb @ w[:N].float().t()) * rstd
    plain = x_plain @ w[:N].float().t()
    out32 = sm100.gemm_norm(hd_, gd, eps, w1, ops.EPI_STORE_F32, rows=rd, split=split)
    assert out32.dtype == torch.float32 and rel(out32, same) <= 3e-5
    assert rel(out32, plain) <= 6e-3
    assert rel(sm100.gemm_norm(hd_, gd, eps, w1, ops.EPI_STORE, rows=rd, split=split), plain) <= 8e-3
    up = (xb @ w[N:].float().t()) * rstd
    want = same / (1 + torch.exp(-same)) * up
    assert rel(sm100.gemm_norm(hd_, gd, eps, wd, ops.EPI_SWIGLU, rows=rd, split=split), want) <= 8e-3
    sm100.check_error(DEV)
    again = sm100.gemm_norm(hd_, gd, eps, w1, ops.EPI_STORE_F32, rows=rd, split=split)
    assert torch.equal(again, out32)


def test_tc_gemm_with_norm_refuses_misfits():
    from rllm_b200.kernels import ops, sm100
    h = torch.randn(sm100.norm_max_tokens() + 1, 128, device=DEV)
    g, w = torch.ones(128, device=DEV), rnd(64, 128).to(DEV)
    assert not sm100.norm_supported(h, g, w)                                   # too many tokens
    assert sm100.norm_supported(h[:4], g, w)
    assert not sm100.norm_supported(h[:4, :100], g[:100], w[:, :100].contiguous())   # K % 8
    with pytest.raises(ops.KernelError):
        sm100.gemm_norm(h, g, 1e-5, w, ops.EPI_STORE)
    with pytest.raises(ops.KernelError):
        sm100.gemm_norm(h[:4], g, 1e-5, w, ops.EPI_ACCUM_F32)


def test_tc_gemm_takes_a_strided_view_and_refuses_misfits():
    from rllm_b200.kernels import ops, sm100
    big = rnd(40, 3 * 128, seed=5).to(DEV)
    x = big[:, 128:256]                                   # row stride 384, offset 256 bytes
    w = rnd(96, 128, seed=6).to(DEV)
    assert rel(sm100.gemm(x, w, ops.EPI_STORE_F32), x.float().cpu() @ w.float().cpu().t()) <= 2e-5
    assert not sm100.gemm_supported(rnd(4, 100).to(DEV), rnd(8, 100).to(DEV))      # K % 8
    assert not sm100.gemm_supported(big[:, 1:129], w)                               # misaligned
    with pytest.raises(ops.KernelError):
        sm100.gemm(rnd(4, 100).to(DEV), rnd(8, 100).to(DEV), ops.EPI_STORE)


PAIR_SHAPES = [(2048, 3072, 2048), (2048, 2048, 8192), (1000, 2176, 520), (513, 384, 64), (4096, 8192, 2048), (1500, 200, 136)]


@pytest.mark.parametrize("T,N,K", PAIR_SHAPES)
def test_products_of_long_portions_on_cta_pairs(T, N, K):
    """Tiles of 256 weight rows on pairs of CTAs (tcgen05.mma.cta_group::2): every epilogue against the
    float product, widths and token counts that end inside a tile and inside a CTA's half of it, and
    the same bits as the single-CTA kernel gives (same products, same order of K)."""
    from rllm_b200.kernels import ops, sm100
    x, w = rnd(T, K, seed=1), rnd(2 * N, K, seed=2, scale=K ** -0.5)
    xd, wd = x.to(DEV), w.to(DEV)
    w1 = wd[:N].contiguous()
    ref = x.float() @ w[:N].float().t()
    up = x.float() @ w[N:].float().t()
    res = torch.randn(T, N, generator=torch.Generator().manual_seed(3))
    outs = {}
    for pairs in (True, -1):                 # all on pairs, none
        sm100.set_pairs(pairs)
        try:
            o = [sm100.gemm(xd, w1, ops.EPI_STORE), sm100.gemm(xd, w1, ops.EPI_STORE_F32),
                 sm100.gemm(xd, w1, ops.EPI_ACCUM_F32, out=res.to(DEV).clone()), sm100.gemm(xd, wd, ops.EPI_SWIGLU)]
            sm100.check_error(DEV)
        finally:
            sm100.set_pairs(False)
        outs[pairs] = o
    o = outs[True]
    assert rel(o[0], ref) <= 6e-3 and rel(o[1], ref) <= 2e-5 and rel(o[2], res + ref) <= 2e-5
    assert rel(o[3], ref / (1 + torch.exp(-ref)) * up) <= 6e-3
    for a, b in zip(outs[True], outs[-1]):
        assert torch.equal(a, b)


def test_the_streaming_kernel_takes_the_decode_products():
    """Which products of a decode step run the weight-streaming kernel: those of the three model
    shapes the benchmark runs, at 1 to 8 tokens; not 9 tokens, not a K that is no multiple of 32."""
    from rllm_b200.kernels import ops, sm100
    for hidden, inter, q, qkv, hd in ((2048, 8192, 2048, 3072, 64), (3072, 8192, 3072, 5120, 128), (4096, 14336, 4096, 6144, 128)):
        for T in (1, 8):
            assert sm100.stream_supported(sm100.EPI_QKV_ROPE, True, T, qkv, hidden, hd)
            assert sm100.stream_supported(ops.EPI_ACCUM_F32, False, T, hidden, q)
            assert sm100.stream_supported(ops.EPI_SWIGLU, True, T, inter, hidden)
            assert sm100.stream_supported(ops.EPI_ACCUM_F32, False, T, hidden, inter)
            assert sm100.stream_supported(ops.EPI_STORE_F32, True, T, 128256, hidden)
    assert not sm100.stream_supported(ops.EPI_STORE, False, 9, 2048, 2048)
    assert not sm100.stream_supported(ops.EPI_STORE, False, 8, 2048, 200)
    assert not sm100.stream_supported(ops.EPI_STORE, False, 8, 100, 2048)
    assert sm100.stream_supported(ops.EPI_STORE, True, 8, 2048, 8192)
    assert not sm100.stream_supported(ops.EPI_STORE, True, 8, 2048, 14336)      # norm in front: K up to 8,192
    assert not sm100.stream_supported(sm100.EPI_QKV_ROPE, False, 8, 96, 64, 48)


def test_plan_splits_small_batches_only():
    from rllm_b200.kernels import ops, sm100
    bn, splits = sm100.plan(ops.EPI_STORE, 8, 3072, 2048)
    assert bn == 16 and 2 <= splits <= 8                 # 24 tiles: a cluster of ranges of K per tile
    assert sm100.plan(ops.EPI_ACCUM_F32, 64, 2048, 8192) == (32, 8)      # two tiles of 32 tokens
    assert sm100.plan(ops.EPI_ACCUM_F32, 128, 2048, 8192) == (64, 4)     # a narrow weight keeps its ranges of K
    assert sm100.plan(ops.EPI_ACCUM_F32, 129, 2048, 8192) == (128, 4)
    assert sm100.plan(ops.EPI_ACCUM_F32, 257, 2048, 8192) == (64, 1)
    assert sm100.plan(ops.EPI_STORE, 128, 3072, 2048) == (64, 1)
    assert sm100.plan(ops.EPI_STORE, 8, 3072, 2048, split=False) == (16, 1)
    # long portions on single CTAs: the tile width that fills whole waves of 148 (288 tiles of 176 tokens; 144 of 240); on pairs a
    # gate/up tile has 256 tokens
    sm100.set_pairs(-1)
    try:
        assert sm100.plan(ops.EPI_STORE, 2048, 3072, 2048) == (176, 1)
        assert sm100.plan(ops.EPI_ACCUM_F32, 2048, 2048, 8192) == (240, 1)
        assert sm100.plan(ops.EPI_SWIGLU, 2048, 8192, 2048) == (128, 1)
    finally:
        sm100.set_pairs(False)
    assert sm100.plan(ops.EPI_SWIGLU, 2048, 8192, 2048) == (256, 1)
    assert sm100.plan(ops.EPI_SWIGLU, 96, 8192, 2048) == (128, 1)        # tokens on the accumulator's rows from 65 on
    assert sm100.plan(ops.EPI_SWIGLU, 64, 8192, 2048) == (128, 1)        # and from 33 on where no norm is in front
    assert sm100.plan(ops.EPI_SWIGLU, 32, 8192, 2048) == (32, 2)
    assert sm100.plan(ops.EPI_STORE_F32, 8, 128256, 2048) == (16, 1)


@pytest.mark.parametrize("split", [True, False])
@pytest.mark.parametrize("T,K,nh,nkv,hd,page,rot", [
    (1, 64, 4, 2, 16, 16, None), (9, 96, 3, 1, 32, 8, None), (8, 2048, 32, 8, 64, 16, None),
    (70, 256, 5, 5, 64, 4, 32), (300, 128, 2, 1, 128, 16, None), (17, 512, 6, 2, 128, 32, 64),
    (5, 3072, 24, 8, 128, 16, None), (8, 96, 3, 1, 32, 8, None), (3, 160, 2, 2, 96, 4, None), (1, 2048, 32, 8, 64, 16, None),
    (600, 192, 6, 2, 64, 16, None), (1100, 256, 4, 2, 32, 8, 16), (257, 64, 3, 3, 16, 4, None),
    # 33 to 128 tokens against wide weights
    (64, 256, 32, 8, 64, 16, None), (100, 128, 12, 4, 128, 16, None), (40, 192, 30, 10, 64, 8, None),
    (33, 72, 40, 20, 32, 4, None), (128, 64, 24, 8, 64, 16, None)])
def test_qkv_product_with_rotary_epilogue(T, K, nh, nkv, hd, page, rot, split):
    """q/k/v projection, rotation of q and k, and the cache write in one kernel, against the
    plain formulas: widths that are no multiple of the tile, head sizes 16 to 128, partial
    rotation, scattered slots, one token that must not be written."""
    import plain_llama as P
    from rllm_b200.kernels import ops, sm100
    if 128 % hd and not split:
        pytest.skip("a head size that does not divide 128 runs in the kernel for steps of at most 8 tokens only")
    rot_dim = rot or hd
    N = (nh + 2 * nkv) * hd
    x, w = rnd(T, K, seed=1), rnd(N, K, seed=2, scale=K ** -0.5)
    g = torch.Generator().manual_seed(7)
    positions = torch.randint(0, 5000, (T,), generator=g, dtype=torch.int32)
    positions[0] = 0
    inv_freq = P.rope_inv_freq(rot_dim, 500000.0, {"rope_type": "llama3", "factor": 8.0, "low_freq_factor": 1.0,
                               "high_freq_factor": 4.0, "original_max_position_embeddings": 32})
    pages = (T + page - 1) // page + 3
    slots = torch.randperm(pages * page, generator=g)[:T].to(torch.int32)
    if T > 2:
        slots[T // 2] = -1
    kc = torch.zeros(pages, nkv, page, hd, dtype=torch.bfloat16, device=DEV)
    vc = torch.zeros_like(kc)
    out = sm100.gemm_qkv_rope(x.to(DEV), w.to(DEV), positions.to(DEV), inv_freq.to(DEV), slots.to(DEV), kc, vc,
                              nh, nkv, hd, page, rot_dim, split=split)
    sm100.check_error(DEV)
    ref = x.float() @ w.float().t()
    q = ref[:, : nh * hd].view(T, nh, hd)
    k = ref[:, nh * hd: (nh + nkv) * hd].view(T, nkv, hd)
    v = ref[:, (nh + nkv) * hd:].view(T, nkv, hd)

    def rope(t):
        r = P.rope(t[..., :rot_dim], positions, inv_freq)
        return torch.cat([r, t[..., rot_dim:]], -1)

    qr, kr = rope(q), rope(k)
    scale = float(ref.abs().max())
    got = out.float().cpu()
    assert float((got[:, : nh * hd].view(T, nh, hd) - qr).abs().max()) <= 6e-3 * scale
    assert float((got[:, nh * hd: (nh + nkv) * hd].view(T, nkv, hd) - kr).abs().max()) <= 6e-3 * scale
    assert float((got[:, (nh + nkv) * hd:].view(T, nkv, hd) - v).abs().max()) <= 6e-3 * scale
    written = torch.zeros(pages, page, dtype=torch.bool)
    kcc, vcc = kc.float().cpu(), vc.float().cpu()
    for t in range(T):
        if slots[t] < 0:
            continue
        pg, off = int(slots[t]) // page, int(slots[t]) % page
        written[pg, off] = True
        assert float((kcc[pg, :, off] - kr[t]).abs().max()) <= 6e-3 * scale
        assert float((vcc[pg, :, off] - v[t]).abs().max()) <= 6e-3 * scale
    mask = ~written[:, None, :].expand(-1, nkv, -1)
    assert float(kcc[mask].abs().sum()) == 0.0 and float(vcc[mask].abs().sum()) == 0.0   # nothing else touched
    # no cache write at all when no slots are given (a layer that reads another layer's cache)
    out2 = sm100.gemm_qkv_rope(x.to(DEV), w.to(DEV), positions.to(DEV), inv_freq.to(DEV), None, None, None,
                               nh, nkv, hd, page, rot_dim, split=split)
    assert torch.equal(out2, out)
    # the angles from a table made once for the step, as the engine passes them
    table = ops.rope_table(positions.to(DEV), inv_freq.to(DEV), T)
    kc4, vc4 = torch.zeros_like(kc), torch.zeros_like(vc)
    out4 = sm100.gemm_qkv_rope(x.to(DEV), w.to(DEV), positions.to(DEV), inv_freq.to(DEV), slots.to(DEV), kc4, vc4,
                               nh, nkv, hd, page, rot_dim, split=split, table=table)
    sm100.check_error(DEV)
    assert float((out4.float() - out.float()).abs().max()) <= scale * 2 ** -7      # a last place at most
    assert float((kc4.float() - kc.float()).abs().max()) <= scale * 2 ** -7
    assert torch.equal(vc4, vc)
    if T <= sm100.norm_max_tokens():
        # the same with RMSNorm in front, in the same kernel: h = x scaled per row, norm weight 1
        hrows = x.float() * torch.linspace(0.5, 3.0, T)[:, None]
        rstd = torch.rsqrt((hrows.double() ** 2).mean(-1, keepdim=True) + 1e-6).float()
        refn = ((hrows.to(torch.bfloat16).float() @ w.float().t()) * rstd)
        kc2, vc2 = torch.zeros_like(kc), torch.zeros_like(vc)
        out3 = sm100.gemm_qkv_rope(None, w.to(DEV), positions.to(DEV), inv_freq.to(DEV), slots.to(DEV), kc2, vc2,
                                   nh, nkv, hd, page, rot_dim, split=split,
                                   norm=(hrows.to(DEV), torch.ones(K, device=DEV), 1e-6))
        sm100.check_error(DEV)
        qn = rope(refn[:, : nh * hd].view(T, nh, hd))
        kn = rope(refn[:, nh * hd: (nh + nkv) * hd].view(T, nkv, hd))
        vn = refn[:, (nh + nkv) * hd:].view(T, nkv, hd)
        sc = float(refn.abs().max())
        g3 = out3.float().cpu()
        assert float((g3[:, : nh * hd].view(T, nh, hd) - qn).abs().max()) <= 6e-3 * sc
        assert float((g3[:, nh * hd: (nh + nkv) * hd].view(T, nkv, hd) - kn).abs().max()) <= 6e-3 * sc
        assert float((g3[:, (nh + nkv) * hd:].view(T, nkv, hd) - vn).abs().max()) <= 6e-3 * sc
        k2, v2 = kc2.float().cpu(), vc2.float().cpu()
        for t in range(T):
            if slots[t] >= 0:
                pg, off = int(slots[t]) // page, int(slots[t]) % page
                assert float((k2[pg, :, off] - kn[t]).abs().max()) <= 6e-3 * sc
                assert float((v2[pg, :, off] - vn[t]).abs().max()) <= 6e-3 * sc
