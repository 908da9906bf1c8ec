"""Layers with many rows per member (weights resident in shared memory) against an fp64 reference, at the edges of tiles,
blocks of k, widths and ranks."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,a,rank,n_pop,bm,T", [
    (64, 64, 8, 40, 2048, 1),       # the token models' projection
    (64, 256, 8, 20, 300, 3),       # one accumulator; a last tile of 88 rows, members change inside a tile
    (256, 64, 16, 10, 1000, 2),     # four blocks of k
    (72, 96, 5, 300, 64, 1),        # one tile per pair; a second block of k with 8 inputs
    (8, 16, 1, 26, 1500, 1),
    (136, 96, 3, 12, 129, 16),      # three blocks of k, two rows in the last tile
])
def test_rows_path_matches_fp64(hs, k, a, rank, n_pop, bm, T):
    from hyperscalees_b200 import ops
    from hyperscalees_b200.core import get_context
    g = torch.Generator(device="cuda").manual_seed(k * a + rank)
    x = torch.randn(T, n_pop, bm, k, device="cuda", generator=g)
    w = torch.randn(a, k, device="cuda", generator=g)
    kw = dict(n_pop=n_pop, bm=bm, t_steps=T, sigma=0.3, rank=rank, key=7, epoch=1, first_thread=6, noise_reuse=1)
    ctx = get_context(0)
    ctx.profile_enable(False)
    y = ops.perturbed_linear(x, w, **kw)
    assert ctx.profile_read().get("linear_rows", (0,))[0] == 1
    c = ops.FactorCache(7, 1, 1, rank, a, k, n_pop // 2, first_pair=3)
    assert torch.equal(y, ops.perturbed_linear(x, w, cache=c, **kw))
    wide = torch.empty(T * n_pop * bm, a + 3, device="cuda")[:, 1:a + 1]
    assert torch.equal(y, ops.perturbed_linear(x, w, out=wide, **kw))
    B, A = c.B.double().repeat_interleave(2, 0), c.A.double().repeat_interleave(2, 0)
    sgn = torch.tensor([1.0, -1.0], device="cuda", dtype=torch.double).repeat(n_pop // 2).view(1, -1, 1, 1)
    ref = torch.einsum("tnbk,ak->tnba", x.double(), w.double())
    ref += sgn * torch.einsum("tnbr,nar->tnba", torch.einsum("tnbk,nkr->tnbr", x.double(), B), A) * (0.3 / rank ** 0.5)
    assert (y.double().view(ref.shape) - ref).abs().max() <= 3e-6 * ref.abs().max()
    assert ctx.device_status() == 0


def test_grouped_heads_take_the_rows_path(hs):
    from hyperscalees_b200 import ops
    n_pop, bm, k, hd, rank = 40, 1024, 64, 16, 8
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(n_pop, bm, k, device="cuda", generator=g)
    ws = [torch.randn(hd, k, device="cuda", generator=g) for _ in range(4)]
    caches = [ops.FactorCache(20 + i, 0, 0, rank, hd, k, n_pop // 2) for i in range(4)]
    grouped = ops.GroupedFactorCache(caches)
    y = ops.perturbed_linear(x, torch.cat(ws, 0), n_pop=n_pop, bm=bm, sigma=0.2, rank=rank, key=grouped.key, cache=grouped,
                             n_groups=4)
    for i, (w, c) in enumerate(zip(ws, caches)):
        one = ops.perturbed_linear(x, w, n_pop=n_pop, bm=bm, sigma=0.2, rank=rank, key=20 + i, cache=c)
        assert torch.equal(y[:, i * hd:(i + 1) * hd], one)


@pytest.mark.parametrize("bm,a", [(1024, 64), (20, 48)])   # fused, and as two calls
@pytest.mark.parametrize("post", ["swish", "add", "lif_rate"])
def test_post_matches_the_separate_calls(hs, post, bm, a):
    from hyperscalees_b200 import ops
    n_pop, k = 40, 64
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(n_pop, bm, k, device="cuda", generator=g)
    w = torch.randn(a, k, device="cuda", generator=g) / 8
    kw = dict(n_pop=n_pop, bm=bm, sigma=0.2, rank=8, key=20, tau_m=2.0, v_th=0.3)
    y = ops.perturbed_linear(x, w, **kw)
    acc = torch.randn(n_pop * bm, a, device="cuda", generator=g)
    want = {"swish": lambda: ops.swish(y), "add": lambda: ops.add_inplace(acc.clone(), y),
            "lif_rate": lambda: ops.lif_rate(y, 5, 2.0, 0.3)}[post]()
    got = ops.perturbed_linear(x, w, post=post, post_steps=5, out=acc if post == "add" else None, **kw)
    assert torch.equal(got, want)
