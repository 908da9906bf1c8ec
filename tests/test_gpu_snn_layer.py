"""The fused SNN forward pass (one kernel per hidden layer) against the layer-by-layer path, at the sizes where its tiles,
chunks and pair blocks end."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,n_pop,bm,T,rank,reset", [
    ([784, 128, 10], 32, 8, 4, 4, 1),              # several pairs would fit a tile, few pairs: one each
    ([100, 33, 17, 10], 602, 1, 7, 5, 0),          # odd widths, packed pairs, a last tile with fewer of them
    ([64, 300, 130, 26], 6, 43, 3, 17, 1),         # a pair over several tiles, the last one short; two rank blocks
    ([70, 129, 5], 2, 1, 128, 64, 0),              # one sample per tile, T at its limit
    ([784, 128, 64, 10], 400, 16, 8, 4, 1),        # tiles of 256 rows, several per CTA
    ([36, 16, 40, 24, 100], 10, 70, 5, 33, 1),     # three hidden layers, readout in slices
    ([784, 320, 10], 1, 500, 8, 0, 1),             # clean, one member
    ([31, 257, 64, 10], 7, 9, 9, 0, 0),            # clean, odd numbers of members and inputs
])
@pytest.mark.parametrize("exact", [True, False])
def test_fused_forward_matches_the_layers(hs, dims, n_pop, bm, T, rank, reset, exact):
    from hyperscalees_b200 import models, noiser, ops
    g = torch.Generator(device="cuda").manual_seed(sum(dims) + T)
    net = models.SnnMlp(dims, tau_m=2.0, v_th=0.3, reset_mode=reset, seed=4)
    keys = models.default_base_keys(len(dims))
    args = ()
    if rank:
        frozen, nz = noiser.init_noiser(net.params(), 0.1, 0.0, 0, False, 0, rank, noiser.Solver.sgd(0.1))
        args = (frozen, nz, keys)
    img = torch.rand(n_pop * bm, dims[0], device="cuda", generator=g)
    x = ops.poisson_encode(img, T, [1, 2, 3, 4]).reshape(T, n_pop, bm, dims[0])
    if not exact:
        x = x * (1.0 + torch.rand(x.shape, device="cuda", generator=g))
    got = net.forward_population(x, *args, epoch=2)
    assert torch.equal(got, net.forward_population(x, *args, epoch=2))
    want, _ = net.forward_population(x, *args, epoch=2, want_hidden=True)
    # currents agree to about 1e-6, so a neuron exactly at its threshold may decide otherwise in a rare sample
    off = (got - want).abs().amax(1) > 1e-4 * want.abs().max()
    assert off.float().mean().item() <= 0.02 and torch.isfinite(got).all()
    if rank and exact:
        labels = torch.randint(0, dims[-1], (n_pop * bm,), device="cuda", generator=g, dtype=torch.int32)
        step = models.PopulationStep(net, frozen, nz, keys, T, n_pop, bm)
        raw, logits = step.eval(img, labels, [1, 2, 3, 4], epoch=2, want_logits=True)
        assert torch.equal(logits, got)
        assert torch.equal(raw, ops.member_mean(ops.fitness(logits, labels), n_pop, bm))
        step.build_caches(2)
        assert torch.equal(step.eval(img, labels, [1, 2, 3, 4], epoch=2), raw)
