"""The packed tensor-core path of the perturbed linear layer (shapes that fit no tile) against the CPU oracle."""
import numpy as np
import pytest
import torch

from test_gpu_linear import KEY, dev, oracle_mm

pytestmark = pytest.mark.gpu


def launched(ctx, fn):
    ctx.profile_enable(False)
    out = fn()
    return out, {k for k, v in ctx.profile_read().items() if v[0]}


@pytest.mark.parametrize("n_pop,bm,k,a,rank,t_steps,first", [
    (5, 3, 37, 19, 2, 1, 1),        # everything ragged, odd first member: single-member pairs at both ends
    (1, 16, 784, 128, 4, 1, 3),     # one member
    (3, 1, 16, 8, 1, 1, 4),         # one row per member
    (6, 17, 100, 130, 6, 1, 0),     # 34 rows per pair: padded to 64, two chunks of columns
    (4, 24, 72, 300, 16, 1, 2),     # 48 rows per pair, three chunks of 112 columns (the last one of 76)
    (6, 12, 500, 250, 8, 3, 0),     # 72 rows per pair: a pair spans tiles
    (2, 40, 200, 96, 33, 4, 0),     # 320 rows per pair, rank above 32
    (4, 3, 64, 70, 33, 1, 0),       # 6 rows per pair, rank above 32: padded to 64
    (2, 20, 100, 40, 100, 2, 0),    # rank above 64 (one pair per tile, no staged stores)
    (6, 2, 96, 65, 128, 1, 2),      # the largest rank, few rows
    (40, 5, 784, 100, 6, 6, 0),     # several tiles, pairs of 60 rows
    (2, 50, 1030, 33, 3, 1, 0),     # rows longer than a warp's registers, k not a multiple of 4
])
@pytest.mark.parametrize("cached", [False, True])
def test_packed_path_matches_oracle(hs, oracle, n_pop, bm, k, a, rank, t_steps, first, cached):
    from hyperscalees_b200 import core, ops
    ctx = core.get_context(0)
    g = np.random.default_rng(n_pop * 100 + k)
    x = g.standard_normal((t_steps, n_pop, bm, k)).astype(np.float32)
    w = (g.standard_normal((a, k)) / np.sqrt(k)).astype(np.float32)
    sigma = 0.5
    cache = ops.FactorCache(KEY, 3, 1, rank, a, k, (first + n_pop - 1) // 2 - first // 2 + 2, first // 2) if cached else None
    kw = dict(n_pop=n_pop, bm=bm, t_steps=t_steps, sigma=sigma, rank=rank, key=KEY, epoch=3, first_thread=first,
              noise_reuse=1, cache=cache)
    want = oracle_mm(oracle, x, w, sigma, rank, KEY, 3, first, 1, acc64=True)
    scale = max(np.abs(want).max(), 1.0)
    got, names = launched(ctx, lambda: ops.perturbed_linear(dev(x), dev(w), **kw))
    assert "linear_pack" in names
    assert np.abs(got.cpu().numpy() - want).max() <= 2e-5 * scale
    assert ctx.device_status() == 0
    spikes, pot = ops.perturbed_linear(dev(x), dev(w), lif=True, tau_m=2.0, v_th=0.1, want_potentials=True, **kw)
    assert np.abs(pot.cpu().numpy() - 0.5 * want).max() <= 1e-5 * scale
    assert torch.equal(spikes, (pot >= 0.1).float())
    assert ctx.device_status() == 0


@pytest.mark.parametrize("rows,k,a", [(1, 5, 3), (127, 64, 128), (129, 784, 10), (300, 100, 257), (1000, 1100, 33)])
def test_packed_path_clean_product(hs, rows, k, a):
    from hyperscalees_b200 import core, ops
    ctx = core.get_context(0)
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, k, device="cuda", generator=g)
    w = torch.randn(a, k, device="cuda", generator=g)
    want = x.double() @ w.double().t()
    for xx in (x, (x > 1).float()):     # the second input is exact in fp16: its lo half is dropped
        want = xx.double() @ w.double().t()
        got, names = launched(ctx, lambda: ops.perturbed_linear(xx, w, n_pop=1, bm=rows, perturb=False, out_scale=1.5))
        assert "linear_pack" in names and ctx.device_status() == 0
        assert (got.double() - 1.5 * want).abs().max().item() <= 3e-6 * k ** 0.5 * max(1.0, want.abs().max().item())


def test_packed_path_pitched_operands(hs, oracle):
    from hyperscalees_b200 import ops
    g = np.random.default_rng(0)
    n_pop, bm, k, a = 3, 4, 102, 60
    xb, wb = torch.zeros(n_pop * bm, 129, device="cuda"), torch.zeros(a, 104, device="cuda")
    ob = torch.full((n_pop * bm, 67), float("nan"), device="cuda")
    x = g.standard_normal((n_pop, bm, k)).astype(np.float32)
    w = g.standard_normal((a, k)).astype(np.float32)
    xb[:, 1:1 + k], wb[:, :k] = dev(x.reshape(-1, k)), dev(w)
    ops.perturbed_linear(xb[:, 1:1 + k], wb[:, :k], n_pop=n_pop, bm=bm, sigma=0.1, rank=5, key=KEY, out=ob[:, 3:3 + a])
    want = oracle_mm(oracle, x, w, 0.1, 5, KEY, 0, 0, 0, acc64=True)
    assert np.abs(ob[:, 3:3 + a].cpu().numpy() - want).max() <= 2e-5 * np.abs(want).max()
    assert torch.isnan(ob[:, 3 + a:]).all() and torch.isnan(ob[:, :3]).all()


@pytest.mark.parametrize("n_pop,bm,k,a,rank,packed", [
    (1300, 1, 70, 19, 3, False),    # two rows of 32, more tiles than SMs
    (1300, 2, 70, 19, 3, False),    # four rows of 32
    (1300, 6, 150, 300, 28, True),  # twelve rows of 32, a wider rank
    (40, 1, 70, 19, 3, True),       # one wave
    (400, 1, 51, 10, 96, True),     # two rows of 128, two waves
    (12000, 1, 51, 10, 96, False),  # many
])
def test_pairs_of_few_rows(hs, oracle, n_pop, bm, k, a, rank, packed):
    """Many pairs of a row or two per member would be mostly padding: they stay on fp32 multiply-adds."""
    from hyperscalees_b200 import core, ops
    ctx = core.get_context(0)
    g = np.random.default_rng(k + rank)
    x = g.standard_normal((1, n_pop, bm, k)).astype(np.float32)
    w = (g.standard_normal((a, k)) / np.sqrt(k)).astype(np.float32)
    got, names = launched(ctx, lambda: ops.perturbed_linear(dev(x), dev(w), n_pop=n_pop, bm=bm, t_steps=1, sigma=0.5,
                                                            rank=rank, key=KEY, epoch=3, first_thread=0, noise_reuse=1))
    assert ("linear_pack" in names) == packed
    rows = slice(n_pop - 6, n_pop)
    want = oracle_mm(oracle, x[:, rows], w, 0.5, rank, KEY, 3, n_pop - 6, 1, acc64=True)
    assert np.abs(got.cpu().numpy().reshape(x.shape[:3] + (a,))[:, rows] - want.reshape(1, 6, bm, a)).max() <= 2e-5 * max(np.abs(want).max(), 1.0)
    assert ctx.device_status() == 0
