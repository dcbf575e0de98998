"""Products of 33 to 256 tokens whose tiles of 64 or 128 tokens are shared by ranges of K: against a float product of the same bfloat16
inputs (relative to the largest value: 2^-8 of rounding for bfloat16 results, 2e-5 for float sums of K products), at sizes on both sides
of the rule's lines, with partial tiles, and the same bits again."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rnd(*shape, seed=0, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(torch.bfloat16).to(DEV)


def rel(a, b):
    return float((a.float() - b.float()).abs().max()) / max(float(b.abs().max()), 1e-30)


# the sizes below that wide tiles and ranges of K take; the others lie behind the rule's lines
RANGED = [(65, 2048, 2048), (100, 2048, 8192), (64, 4096, 4104), (129, 2048, 8192), (192, 2044, 8200), (256, 4096, 16384), (33, 4090, 4104),
          (127, 4096, 5000)]


@pytest.mark.parametrize("T,N,K", [(65, 2048, 2048), (100, 2048, 8192), (128, 2048, 1000), (127, 4096, 1096), (33, 4096, 2048), (64, 4096, 4104),
                                   (129, 2048, 8192), (192, 2044, 8200), (256, 4096, 16384), (255, 1924, 5440), (256, 2048, 4096), (257, 2048, 8192),
                                   (32, 4096, 2048), (33, 4090, 4104), (127, 4096, 5000), (100, 4740, 2048), (97, 1800, 520), (96, 2048, 448)])
def test_ranges_of_wide_tiles(T, N, K):
    from rllm_b200.kernels import ops, sm100
    assert (sm100.plan(ops.EPI_STORE, T, N, K) in ((64, 2), (64, 4), (128, 2), (128, 4))) == ((T, N, K) in RANGED)
    x, w = rnd(T, K, seed=1), rnd(N, K, seed=2, scale=K ** -0.5)
    ref = x.float() @ w.float().t()
    res = torch.randn(T, N, generator=torch.Generator().manual_seed(3)).to(DEV)
    wide = torch.zeros(T, N + 8, dtype=torch.float32, device=DEV)
    for run, want, tol in ((lambda: sm100.gemm(x, w, ops.EPI_STORE), ref, 6e-3), (lambda: sm100.gemm(x, w, ops.EPI_STORE_F32), ref, 2e-5),
                           (lambda: sm100.gemm(x, w, ops.EPI_STORE, act="relu2"), ref.clamp(min=0) ** 2, 6e-3),
                           (lambda: sm100.gemm(x, w, ops.EPI_ACCUM_F32, out=res.clone()), res + ref, 2e-5),
                           (lambda: sm100.gemm(x, w, ops.EPI_STORE_F32, out=wide[:, :N]).clone(), ref, 2e-5)):
        a = run()
        assert rel(a, want) <= tol and torch.equal(a, run())
    assert not wide[:, N:].any()
    sm100.check_error(DEV)
