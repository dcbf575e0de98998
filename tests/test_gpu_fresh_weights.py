"""A product whose second matrix was written by the launch just before it (an own kernel, which lets its successors start at once):
the same bits as after a synchronisation, on every kernel that copies that matrix ahead where it is fixed."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rnd(*shape, seed=0, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(torch.bfloat16).to(DEV)


# tokens: the streaming kernel (4, 12), small tiles (20), ranges of wide tiles (100, 192), pairs (600, 2048), the persistent kernel (300)
@pytest.mark.parametrize("T", [4, 12, 20, 100, 192, 300, 600, 2048])
def test_a_matrix_of_the_launch_before(T):
    from rllm_b200.kernels import ops, sm100
    N, K, L = 2048, 2048, 4096
    a, b = rnd(N, L, seed=1, scale=L ** -0.5), rnd(K, L, seed=2)          # w = a b^T takes longer than the next launch's start
    x, res = rnd(T, K, seed=3), torch.randn(T, N, generator=torch.Generator().manual_seed(4)).to(DEV)
    sums = [res.clone(), res.clone()]                    # made beforehand: a copy between the two launches would keep them apart
    h, g = x.float(), torch.ones(K, device=DEV)
    pos = torch.arange(T, dtype=torch.int32, device=DEV)
    inv = torch.rand(32, generator=torch.Generator().manual_seed(5)).to(DEV)
    runs = [lambda w: sm100.gemm(x, w, ops.EPI_STORE), lambda w: sm100.gemm(x, w, ops.EPI_ACCUM_F32, out=sums.pop()),
            lambda w: sm100.gemm(x, w, ops.EPI_SWIGLU), lambda w: sm100.gemm_qkv_rope(x, w, pos, inv, None, None, None, 16, 8, 64, 16, 64)]
    if T <= sm100.norm_max_tokens():
        runs += [lambda w: sm100.gemm_norm(h, g, 1e-5, w, ops.EPI_STORE), lambda w: sm100.gemm_norm(h, g, 1e-5, w, ops.EPI_SWIGLU)]
    for run in runs:
        w = sm100.gemm(a, b, ops.EPI_STORE)
        torch.cuda.synchronize()
        want = run(w)
        w2 = torch.zeros_like(w)
        torch.cuda.synchronize()
        sm100.gemm(a, b, ops.EPI_STORE, out=w2)
        assert torch.equal(run(w2), want)
    sm100.check_error(DEV)
