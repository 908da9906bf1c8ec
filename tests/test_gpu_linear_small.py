"""Narrow layers joined in one launch against one call per layer: the same bits, cached or not."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("widths,k,n_pop,bm,T,rank", [
    ([16] * 12, 64, 602, 16, 1, 8),      # heads of a block: more pairs than CTAs
    ([64] * 3, 36, 30, 28, 4, 16),       # rows of a pair over several blocks
    ([16] * 12, 64, 50, 4, 2, 16),       # more columns than a launch takes
    ([7, 3, 64], 33, 10, 5, 2, 3),       # ragged widths, inputs and rank
    ([10], 64, 2000, 1, 1, 1),           # two rows per pair
    ([32] * 6, 64, 4, 64, 2, 5),
    ([100, 20], 64, 6, 8, 2, 4),         # not narrow: one call after the other
])
@pytest.mark.parametrize("mean", [False, True])
def test_group_matches_single_calls(hs, widths, k, n_pop, bm, T, rank, mean):
    from hyperscalees_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(k + rank)
    x = torch.randn(T, n_pop, bm, k, device="cuda", generator=g)
    ws = [torch.randn(a, k, device="cuda", generator=g) for a in widths]
    keys = [11 + i for i in range(len(ws))]
    kw = dict(n_pop=n_pop, bm=bm, t_steps=T, sigma=0.2, rank=rank, epoch=3, first_thread=4, noise_reuse=2)
    got = ops.perturbed_linear_group(x, ws, keys, mean_steps=mean, **kw)
    caches = [ops.FactorCache(key, 3, 2, rank, w.shape[0], k, n_pop // 2, first_pair=2) for key, w in zip(keys, ws)]
    cached = ops.perturbed_linear_group(x, ws, keys, mean_steps=mean, caches=caches, **kw)
    for y, c, w, key, fc in zip(got, cached, ws, keys, caches):
        want = ops.perturbed_linear(x, w, key=key, **kw)
        if mean:
            want = ops.time_mean(want.view(T, n_pop * bm, -1))
        assert torch.equal(y, want) and torch.equal(c, want)
        ref = torch.einsum("tnbk,ak->tnba", x.double(), w.double())
        B, A = fc.B.double().repeat_interleave(2, 0), fc.A.double().repeat_interleave(2, 0)
        sgn = torch.tensor([1.0, -1.0], device="cuda", dtype=torch.double).repeat(n_pop // 2).view(1, -1, 1, 1)
        ref = ref + sgn * torch.einsum("tnbr,nar->tnba", torch.einsum("tnbk,nkr->tnbr", x.double(), B), A) * (0.2 / rank ** 0.5)
        ref = ref.mean(0) if mean else ref
        assert (y.double().view(ref.shape) - ref).abs().max() <= 3e-6 * ref.abs().max()
