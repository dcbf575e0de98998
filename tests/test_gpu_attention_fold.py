"""Prefill attention where an item's two row tiles lie at both ends of a sequence's rows (few items, no window): sequences with odd and even
numbers of row tiles side by side, one and several heads a kv head, portions behind earlier keys, pages by tensor copies and not; and
with so many items, or a window, that neighbours are taken. Against a float softmax of the same bfloat16 inputs: weights and outputs are
rounded to 8 bits (2^-8 of the largest value each), scores' sums are float."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("nh,nkv,hd", [(8, 2, 64), (3, 3, 64), (8, 2, 128), (2, 2, 128)])
@pytest.mark.parametrize("lens,page,window", [
    ([(129, 129)], 16, None), ([(256, 256), (1, 700), (385, 640)], 16, None), ([(700, 1500), (128, 128), (33, 520)], 10, None),
    ([(513, 513)], 64, None), ([(513, 900)], 16, 200), ([(1100, 1100)] * 8, 16, None)])
def test_row_tiles_of_an_item(nh, nkv, hd, lens, page, window):
    from rllm_b200.kernels import sm100
    g = torch.Generator().manual_seed(sum(n for n, _ in lens) + hd)
    rnd = lambda *s: torch.randn(*s, generator=g).bfloat16()
    P = max(-(-kv // page) for _, kv in lens)
    n_pages = P * len(lens) + 1
    k, v = rnd(n_pages, nkv, page, hd), rnd(n_pages, nkv, page, hd)
    table = torch.randperm(n_pages - 1, generator=g)[: P * len(lens)].view(len(lens), P).int()
    T = sum(n for n, _ in lens)
    q = rnd(T, nh * hd)
    cu = torch.tensor([0] + [n for n, _ in lens]).cumsum(0).int()
    kl = torch.tensor([kv for _, kv in lens]).int()
    out = sm100.attention_prefill_tc(q.to(DEV), k.to(DEV), v.to(DEV), cu.to(DEV), kl.to(DEV), table.to(DEV), max(n for n, _ in lens), nh,
                                     hd ** -0.5, window)
    sm100.check_error(DEV)
    for s, (n, kv) in enumerate(lens):
        pages = table[s].long()
        keys = k[pages].permute(0, 2, 1, 3).reshape(P * page, nkv, hd)[:kv].float().to(DEV).repeat_interleave(nh // nkv, 1)
        vals = v[pages].permute(0, 2, 1, 3).reshape(P * page, nkv, hd)[:kv].float().to(DEV).repeat_interleave(nh // nkv, 1)
        qs = q[cu[s]: cu[s + 1]].float().to(DEV).view(n, nh, hd)
        scores = torch.einsum("ihd,jhd->hij", qs, keys) * hd ** -0.5
        i, j = torch.arange(kv - n, kv, device=DEV)[:, None], torch.arange(kv, device=DEV)[None]
        seen = (j <= i) & (j > i - window if window else j >= 0)
        want = torch.einsum("hij,jhd->ihd", torch.softmax(scores.masked_fill(~seen, -float("inf")), -1), vals).reshape(n, nh * hd)
        got = out[cu[s]: cu[s + 1]].float()
        assert float((got - want).abs().max()) <= 2 * 2 ** -8 * float(want.abs().max())
