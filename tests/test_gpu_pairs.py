"""Products on pairs of CTAs (tiles of 256 weight rows x 64 to 256 tokens): the same bits as the one-CTA kernel gives, for every
epilogue, at tile widths and sizes that end inside a tile, inside a CTA's half of it and inside a block of K; and near a float
product of the same bfloat16 inputs (relative to the largest value: 2^-8 of rounding for bfloat16 results, 2e-5 for float ones,
whose error is that of a float sum of K products)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rnd(*shape, seed=0, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(torch.bfloat16).to(DEV)


def rel(a, b):
    return float((a.float() - b.float()).abs().max()) / max(float(b.abs().max()), 1e-30)


def both(run, pairs):
    from rllm_b200.kernels import sm100
    out = []
    for on in (pairs, -1):
        sm100.set_pairs(on)
        try:
            out.append(run())
            sm100.check_error(DEV)
        finally:
            sm100.set_pairs(False)
    return out


@pytest.mark.parametrize("T,N,K,width", [(65, 256, 64, 64), (129, 2048, 136, 96), (257, 260, 1000, 128), (300, 520, 72, 160), (1905, 384, 520, 192),
                                         (2047, 1160, 264, 224), (700, 128, 2048, 256), (513, 8192, 128, 256), (161, 4, 64, 64),
                                         (2834, 2048, 192, 160), (4096, 3072, 128, 192)])
def test_widths_and_edges(T, N, K, width):
    from rllm_b200.kernels import ops, sm100
    x, w = rnd(T, K, seed=1), rnd(2 * N, K, seed=2, scale=K ** -0.5)
    w1 = w[:N].contiguous()
    ref, up = x.float() @ w[:N].float().t(), x.float() @ w[N:].float().t()
    res = torch.randn(T, N, generator=torch.Generator().manual_seed(3)).to(DEV)
    for run, want, tol in ((lambda: sm100.gemm(x, w1, ops.EPI_STORE), ref, 6e-3), (lambda: sm100.gemm(x, w1, ops.EPI_STORE_F32), ref, 2e-5),
                           (lambda: sm100.gemm(x, w1, ops.EPI_STORE, act="relu2"), ref.clamp(min=0) ** 2, 6e-3),
                           (lambda: sm100.gemm(x, w1, ops.EPI_ACCUM_F32, out=res.clone()), res + ref, 2e-5),
                           (lambda: sm100.gemm(x, w, ops.EPI_SWIGLU), ref / (1 + torch.exp(-ref)) * up, 6e-3)):
        a, b = both(run, width)
        assert torch.equal(a, b) and rel(a, want) <= tol
    wide = torch.zeros(T, N + 12, dtype=torch.float32, device=DEV)              # rows with a stride of their own; what lies between stays
    a, b = both(lambda: sm100.gemm(x, w1, ops.EPI_STORE_F32, out=wide[:, 4: 4 + N]).clone(), width)
    assert torch.equal(a, b) and not wide[:, :4].any() and not wide[:, 4 + N:].any()


@pytest.mark.parametrize("T,nh,nkv,hd,rot,width", [(65, 32, 8, 64, 64, 64), (300, 5, 3, 64, 32, 96), (643, 6, 2, 128, 128, 128), (1905, 4, 4, 32, 16, 160),
                                                   (2048, 12, 4, 128, 64, 192), (257, 3, 1, 16, 16, 256)])
@pytest.mark.parametrize("table", [True, False])
def test_rotary_epilogue(T, nh, nkv, hd, rot, width, table):
    from rllm_b200.kernels import ops, sm100
    K, page = 200, 16
    x, w = rnd(T, K, seed=4), rnd((nh + 2 * nkv) * hd, K, seed=5, scale=K ** -0.5)
    pos = (torch.arange(T, dtype=torch.int32) + 7).to(DEV)
    inv = (10000.0 ** (-torch.arange(rot // 2).float() / (rot // 2))).to(DEV)
    slots = torch.randperm((T // page + 2) * page, generator=torch.Generator().manual_seed(6))[:T].int()
    slots[T // 2] = -1
    slots = slots.to(DEV)
    tab = ops.rope_table(pos, inv, T, 1.0) if table else None

    def run():
        kc = torch.zeros(T // page + 2, nkv, page, hd, dtype=torch.bfloat16, device=DEV)
        vc = torch.zeros_like(kc)
        return (sm100.gemm_qkv_rope(x, w, pos, inv, slots, kc, vc, nh, nkv, hd, page, rot, table=tab), kc, vc)

    got, want = both(run, width)
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    assert float(got[1].abs().max()) > 0 and float(got[2].abs().max()) > 0


@pytest.mark.parametrize("T,N,K", [(128, 2048, 8192), (129, 2048, 8192), (129, 3072, 2048), (643, 3072, 2048), (2048, 2048, 8192)])
def test_the_rule_gives_the_same_bits(T, N, K):
    from rllm_b200.kernels import ops, sm100
    x, w = rnd(T, K, seed=7), rnd(N, K, seed=8, scale=K ** -0.5)
    a, b = both(lambda: sm100.gemm(x, w, ops.EPI_STORE_F32), False)
    assert torch.equal(a, b)
