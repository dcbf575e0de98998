"""Sums over a layer's rows at the widths of models, on each of the kernels that a launch may take: few rows and many, rows of one, two and four
pieces a thread; against 64 bits (float sums of some thousand terms: 2e-6 of the largest value)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rnd(*shape, seed=0, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(DEV)


def rel(a, b):
    return float((a.double() - b.double()).abs().max()) / max(float(b.double().abs().max()), 1e-30)


def rms(x, w, eps):
    x = x.double()
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w.double()


@pytest.mark.parametrize("H", [1024, 1028, 2048, 4096, 4100])
@pytest.mark.parametrize("norms,gated", [(2, False), (1, False), (0, True), (2, True), (0, False)])
def test_sum_of_a_layer_is_the_same_for_few_rows_and_many(H, norms, gated):
    """300 rows and the first 9 of them alone (rows of up to 4,096 numbers: another kernel) have the same bits."""
    from rllm_b200.kernels import hybrid
    T = 300
    h, z = rnd(T, H, seed=1), rnd(T, 4, seed=2, scale=2.0)
    a, b, parts, extra = rnd(T, H, seed=3, scale=3.0), rnd(T, H, seed=4, scale=0.2), rnd(T, 3, H, seed=5), rnd(T, H, seed=6)
    wa, wb = rnd(H, seed=7) + 1, rnd(H, seed=8) + 1
    want = h.double() + parts.double().sum(1) + extra.double() * (torch.sigmoid(z[:, 1:2].double()) if gated else 1.0)
    for x, w in ((a, wa), (b, wb))[:norms]:
        want += 0.5 * rms(x, w, 1e-5)

    def run(n):
        out = h[:n].clone()
        hybrid.combine(out, [(a[:n], wa), (b[:n], wb)][:norms], 0.5, 1e-5, [parts[:n], extra[:n]], z[:n, 1:] if gated else None)
        return out

    many = run(T)
    assert rel(many, want) < 2e-6
    for n in (1, 9, 256, 257):
        assert torch.equal(run(n), many[:n])


@pytest.mark.parametrize("H", [1024, 1028, 2048, 2052, 3072, 4096, 4100])
@pytest.mark.parametrize("T", [1, 9, 300])
@pytest.mark.parametrize("output", [False, True])
def test_norm_of_a_sum_by_pieces_a_thread(H, T, output):
    from rllm_b200.kernels import sink
    h, y, y2, zg = rnd(T, H, seed=1), rnd(T, 2, H, seed=2), rnd(T, H, seed=3), rnd(T, 3, seed=4)
    w = rnd(H, seed=5) + 1
    s = y.double().sum(1) + y2.double() * torch.sigmoid(zg[:, :1].double())
    want = h.double() + 0.75 * rms(s, w, 1e-5) if output else rms(s + 0.75 * h.double(), w, 1e-5)
    rows = []
    for dtype in (torch.bfloat16, torch.float32):
        for shift in (0, 1):                          # a copy that starts between two 16-byte boundaries goes the general way
            out, copy = h.clone(), torch.empty(T * H + 1, dtype=dtype, device=DEV)[shift: shift + T * H].view(T, H)
            sink.postnorm(out, y, 0.75, w, 1e-5, y2, zg, copy, output=output)
            assert rel(out, want) < 2e-6 and torch.equal(copy, out.to(dtype))
            rows.append(out)
    assert torch.equal(rows[0], rows[2])
