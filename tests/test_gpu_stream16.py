"""Products of 9 to 16 tokens on the weight-streaming kernel, against float products of the same bfloat16 inputs: relative to the
largest value 2^-8 of rounding for bfloat16 results (with the norm in front also of the normalised rows, against a reference that
rounds them alike: 2^-7) and 2e-5 for float sums; at the edges of its rule, with partial chunks of K, one slab to several a CTA."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rnd(*shape, seed=0, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(torch.bfloat16).to(DEV)


def rel(a, b):
    return float((a.float() - b.float()).abs().max()) / max(float(b.abs().max()), 1e-30)


@pytest.mark.parametrize("T", [9, 13, 16])
@pytest.mark.parametrize("N,K", [(16, 32), (48, 2048), (2368, 2080), (2384, 4096), (2048, 8192), (2368, 5440), (8192, 2048), (304, 4064)])
def test_streamed_products_of_9_to_16_tokens(T, N, K):
    from rllm_b200.kernels import ops, sm100
    assert sm100.stream_supported(ops.EPI_ACCUM_F32, False, T, N, K)
    assert sm100.stream_supported(ops.EPI_SWIGLU, False, T, N, K) == (K <= 4096)
    assert sm100.stream_supported(ops.EPI_SWIGLU, True, T, N, K) == (K <= 2048)
    x, w = rnd(T, K, seed=1), rnd(2 * N, K, seed=2, scale=K ** -0.5)
    y = x.float() @ w.float().t()
    res = torch.randn(T, N + 8, generator=torch.Generator().manual_seed(3)).to(DEV)
    out = res.clone()
    sm100.gemm(x, w[:N].contiguous(), ops.EPI_ACCUM_F32, out=out[:, :N])       # rows further apart than their length
    assert rel(out[:, :N], res[:, :N] + y[:, :N]) <= 2e-5 and torch.equal(out[:, N:], res[:, N:])
    want = torch.nn.functional.silu(y[:, :N]) * y[:, N:]
    assert rel(sm100.gemm(x, w, ops.EPI_SWIGLU), want) <= 6e-3
    h = torch.randn(2 * T, K, generator=torch.Generator().manual_seed(4)).to(DEV)
    g = torch.rand(K, generator=torch.Generator().manual_seed(5)).to(DEV) + 0.5
    rows = torch.randperm(2 * T, generator=torch.Generator().manual_seed(6))[:T].int().to(DEV)
    hr = h[rows.long()]
    n = (hr * g).to(torch.bfloat16).float() * torch.rsqrt(hr.pow(2).mean(1, keepdim=True) + 1e-5)
    y = n @ w.float().t()
    got = sm100.gemm_norm(h, g, 1e-5, w, ops.EPI_SWIGLU, rows=rows)
    assert rel(got, torch.nn.functional.silu(y[:, :N]) * y[:, N:]) <= 8e-3
    sm100.check_error(DEV)


def test_what_stays_on_the_tensor_memory_kernels():
    from rllm_b200.kernels import ops, sm100
    assert not sm100.stream_supported(ops.EPI_ACCUM_F32, False, 17, 2048, 2048)
    assert not sm100.stream_supported(ops.EPI_ACCUM_F32, False, 9, 2384, 8192)        # more slabs than SMs and long K
    assert not sm100.stream_supported(ops.EPI_ACCUM_F32, False, 9, 2048, 8224)
    assert not sm100.stream_supported(ops.EPI_SWIGLU, True, 9, 9488, 2048)            # a tcgen05 tile for every SM
    assert not sm100.stream_supported(ops.EPI_STORE, True, 9, 2048, 2048)
    assert not sm100.stream_supported(ops.EPI_STORE_F32, False, 16, 128256, 2048)
    assert not sm100.stream_supported(sm100.EPI_QKV_ROPE, False, 9, 288, 2048, 96)    # heads that do not divide 128


@pytest.mark.parametrize("T,nh,nkv,hd,K,norm", [(9, 4, 1, 32, 2048, True), (16, 32, 8, 64, 2048, True), (12, 3, 2, 128, 4096, False), (15, 2, 2, 64, 96, True)])
def test_streamed_rotation_of_9_to_16_tokens(T, nh, nkv, hd, K, norm):
    import plain_llama as P
    from rllm_b200.kernels import sm100
    N = (nh + 2 * nkv) * hd
    assert sm100.stream_supported(sm100.EPI_QKV_ROPE, norm, T, N, K, hd)
    w = rnd(N, K, seed=2, scale=K ** -0.5)
    h = torch.randn(T, K, generator=torch.Generator().manual_seed(4)).to(DEV)
    g = torch.rand(K, generator=torch.Generator().manual_seed(5)).to(DEV) + 0.5
    x = h.to(torch.bfloat16)
    rows = (h * g).to(torch.bfloat16).float() * torch.rsqrt(h.pow(2).mean(1, keepdim=True) + 1e-5) if norm else x.float()
    pos = torch.randint(0, 9000, (T,), generator=torch.Generator().manual_seed(7), dtype=torch.int32)
    inv = P.rope_inv_freq(hd, 500000.0, None)
    slots = torch.randperm(64, generator=torch.Generator().manual_seed(8))[:T].int()
    slots[T - 1] = -1
    kc = torch.zeros(4, nkv, 16, hd, dtype=torch.bfloat16, device=DEV)
    vc = torch.zeros_like(kc)
    out = sm100.gemm_qkv_rope(None if norm else x, w, pos.to(DEV), inv.to(DEV), slots.to(DEV), kc, vc, nh, nkv, hd, 16, hd,
                              norm=(h, g, 1e-5) if norm else None)
    sm100.check_error(DEV)
    ref = (rows @ w.float().t()).cpu()
    q = P.rope(ref[:, : nh * hd].view(T, nh, hd), pos, inv).reshape(T, -1)
    k = P.rope(ref[:, nh * hd: (nh + nkv) * hd].view(T, nkv, hd), pos, inv)
    v = ref[:, (nh + nkv) * hd:].view(T, nkv, hd)
    want = torch.cat((q, k.reshape(T, -1), v.reshape(T, -1)), 1)
    assert rel(out.cpu(), want) <= 8e-3
    scale = float(want.abs().max())
    for cache, rows in ((kc, k), (vc, v)):
        c, seen = cache.float().cpu(), torch.zeros(4, 16, dtype=torch.bool)
        for t in range(T - 1):
            p, o = int(slots[t]) // 16, int(slots[t]) % 16
            seen[p, o] = True
            assert float((c[p, :, o] - rows[t]).abs().max()) <= 8e-3 * scale
        assert not c.transpose(1, 2)[~seen].any()                  # nothing beside the written slots
