"""Row-wise kernels by vectors (convolution of four taps, gated norm of parts, biases, decays) and the gate/up product with gelu,
against their formulas in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DT = {"float32": torch.float32, "bfloat16": torch.bfloat16}


def rel(a, b):
    return float((a.double() - b).norm() / b.norm())


def rnd(*shape, seed, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(DEV)


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("dtype", list(DT))
@pytest.mark.parametrize("C", [4, 516, 640])
@pytest.mark.parametrize("lens", [((0, 1), (0, 2), (7, 1)), ((0, 9), (5, 3), (2, 511)), ((3, 600),)])
def test_convolution_of_four_taps(dtype, C, lens):
    """(tokens before the portion, tokens) per sequence; the middle one of three has no slot: zeros come before its portion."""
    from rllm_b200.kernels import hybrid
    T, S, col0 = sum(n for _, n in lens), len(lens), 8
    x = rnd(T, col0 + C + 4, seed=1).to(DT[dtype])
    w, b, tail = rnd(C, 4, seed=2), rnd(C, seed=3), rnd(S + 1, 3, C, seed=4)
    slots = [-1 if s == 1 else S - s for s in range(S)]
    cu, pos, seq, want = [0], [], [], []
    for s, (before, n) in enumerate(lens):
        mine = x[cu[-1]: cu[-1] + n, col0: col0 + C].double()
        old = tail[slots[s]].double() if slots[s] >= 0 else torch.zeros(3, C, dtype=torch.float64, device=DEV)
        old = old * (torch.arange(3, device=DEV) >= 3 - before)[:, None]        # before position 0 there is nothing
        rows = torch.cat([old, mine])
        y = b.double() + sum(w[:, j].double() * rows[j: j + n] for j in range(4))
        want.append(y * torch.sigmoid(y))
        cu.append(cu[-1] + n)
        pos += list(range(before, before + n))
        seq += [s] * n
    kept = tail.clone()
    got = hybrid.short_conv(x, col0, C, w, b, i32(seq), i32(pos), i32(cu), S, i32(slots), kept)
    assert rel(got, torch.cat(want)) < 1e-6
    assert torch.equal(kept[0], tail[0])


@pytest.mark.parametrize("dtype", list(DT))
@pytest.mark.parametrize("gsize,groups", [(128, 3), (256, 1), (512, 2), (1024, 1)])
@pytest.mark.parametrize("first", [True, False])
def test_gated_norm_of_parts(dtype, gsize, groups, first):
    from rllm_b200.kernels import hybrid
    T, n = 13, gsize * groups
    y, gate = rnd(T, n, seed=1, scale=2.0), rnd(T, 8 + n, seed=2).to(DT[dtype])
    shared = groups > 1
    w = rnd(gsize if shared else n, seed=3)
    g = gate[:, 8:].double()
    for act, f in (("silu", g * torch.sigmoid(g)), ("sigmoid", torch.sigmoid(g))):
        z = (y.double() * f if first else y.double()).view(T, groups, gsize)
        z = (z / torch.sqrt((z * z).mean(-1, keepdim=True) + 1e-5)).reshape(T, n) * w.double().repeat(groups if shared else 1)
        got = hybrid.gated_norm(y, gate, 8, w, 1e-5, groups, DT[dtype], first, act)
        assert rel(got, z if first else z * f) < (1e-6 if dtype == "float32" else 4e-3)


@pytest.mark.parametrize("dtype", list(DT))
@pytest.mark.parametrize("T,N", [(1, 8), (5, 1032), (4100, 24), (3, 37)])
def test_bias_and_decays(dtype, T, N):
    from rllm_b200.kernels import hybrid, ops
    y = rnd(T, N, seed=1).to(DT[dtype])
    bias = rnd(N, seed=2).to(DT[dtype])
    want = (y.float() + bias.float()).to(DT[dtype])
    assert torch.equal(ops.add_bias(y.clone(), bias), want)
    z, b, a_log = rnd(T, N + 3, seed=3, scale=3.0).to(DT[dtype]), rnd(N, seed=4), rnd(1, seed=5)
    step, decay = hybrid.softplus_decay(z, 3, N, b, a_log, want_step=True)
    d = torch.nn.functional.softplus(z[:, 3:].double() + b.double(), threshold=60)
    assert rel(step, d) < 1e-6 and rel(decay, torch.exp(-torch.exp(a_log.double()) * d)) < 2e-6


@pytest.mark.parametrize("T", [1, 8, 20, 64, 129, 300])
@pytest.mark.parametrize("F,K", [(64, 128), (200, 256), (1024, 512)])
def test_gate_with_gelu_in_the_product(T, F, K):
    from rllm_b200.kernels import ops, sm100
    x, w = rnd(T, K, seed=1).bfloat16(), rnd(2 * F, K, seed=2, scale=K ** -0.5).bfloat16()
    g, u = (x.double() @ w.double().T).split(F, 1)
    want = torch.nn.functional.gelu(g, approximate="tanh") * u
    assert rel(sm100.gemm(x, w, ops.EPI_SWIGLU, gelu_gate=True), want) < 4e-3         # one rounding to bfloat16
    if T <= sm100.norm_max_tokens():
        h, wn = rnd(T, K, seed=3), torch.ones(K, device=DEV)
        n = h.double() / torch.sqrt((h.double() ** 2).mean(-1, keepdim=True) + 1e-6)
        g, u = (n @ w.double().T).split(F, 1)
        got = sm100.gemm_norm(h, wn, 1e-6, w, ops.EPI_SWIGLU, gelu_gate=True)
        assert rel(got, torch.nn.functional.gelu(g, approximate="tanh") * u) < 1e-2   # the normed operand is rounded too
    with pytest.raises(ops.KernelError):
        sm100.gemm(x, w, ops.EPI_STORE, gelu_gate=True)


@pytest.mark.parametrize("rows", [8, 16, 64, 256])
def test_gate_with_gelu_as_in_a_pass_of_its_own(rows):
    """Products that are exact (small whole numbers, 32nds), so that only the activation can differ: no further from the 64-bit
    values' roundings than the kernel that activates floats."""
    from rllm_b200.kernels import hybrid, ops, sm100
    T, K, F = 256, 64, 1024
    g = torch.Generator().manual_seed(0)
    x = torch.randint(-4, 5, (T, K), generator=g).to(DEV).bfloat16()
    w = (torch.randint(-4, 5, (2 * F, K), generator=g).float() / 32).to(DEV).bfloat16()
    p = x.double() @ w.double().T
    a, u = p[:, :F], p[:, F:]
    want = (0.5 * a * (1 + torch.tanh((2 / torch.pi) ** 0.5 * (a + 0.044715 * a ** 3))) * u).float().bfloat16()
    apart = hybrid.glu_act(p.float(), torch.bfloat16, "gelu_tanh", 0.0, 1.0)
    got = torch.cat([sm100.gemm(x[i: i + rows], w, ops.EPI_SWIGLU, gelu_gate=True) for i in range(0, T, rows)])
    assert float(a.abs().max()) > 6 and int((got != want).sum()) <= int((apart != want).sum())
