"""What the speed of this framework is measured on: the calls a training or evaluation program makes through the
public entry points, from one member's matrix product to a population of 65 536 members and a 12-layer language model.

`listed()` is the fixed list, `draw()` gives more cases of the same ranges, `prepare()` makes what such a program holds
before the call (inputs from the seed, the model, the step object), `run()` is one pass.  Sizes are those of the
repository's own configurations and tests, or generic ones.
"""
from __future__ import annotations

import functools
import math

import torch

from hyperscalees_b200 import kernels, models, noiser, ops
from hyperscalees_b200.rwkv_lm import LmNoise as RwkvNoise
from hyperscalees_b200.rwkv_lm import RwkvLM
from hyperscalees_b200.snn_transformer import SnnTransformer, TrainNoise
from hyperscalees_b200.spiking_lm import LmNoise as SpikingNoise
from hyperscalees_b200.spiking_lm import SpikingLM

KEY = 0x3C6EF372FE94F82A     # base key of parameter index 1 (models.default_base_keys)
SIGMA = 0.02
HEAD = 64                    # head size of the RWKV model
LORA_DIMS = (64, 32, 64, 128)
# tau and reset of the first configuration, with the default threshold: an untrained network then fires in every layer
LIF = {"tau_m": 2.0, "v_th": 0.3, "reset_mode": ops.RESET_SUBTRACT}


def listed():
    return [
        # One member's product, the call the per-member closure of a noiser makes: latency and launches.
        {"name": "member_product", "kind": "member", "bm": 16, "k": 784, "a": 128, "rank": 4},
        # The smallest training run: 32 members, one hidden layer, new noise every step.
        {"name": "mlp_step_small", "kind": "mlp_step", "dims": "784-128-10", "n_pop": 32, "bm": 8, "T": 4, "rank": 4,
         "cache": "off", "noise_reuse": 1, "solver": "adam"},
        # The ordinary training step: 256 members, 64 samples each, rank 4.
        {"name": "mlp_step_256x64", "kind": "mlp_step", "dims": "784-128-128-128-10", "n_pop": 256, "bm": 64, "T": 8,
         "rank": 4, "cache": "off", "noise_reuse": 0, "solver": "adamw"},
        # A network whose sizes fit no tile: widths, members, samples and rank as a user may well choose them.
        {"name": "mlp_step_ragged", "kind": "mlp_step", "dims": "784-300-100-10", "n_pop": 1000, "bm": 5, "T": 6,
         "rank": 6, "cache": "off", "noise_reuse": 1, "solver": "sgd"},
        # The large population: one sample per member, rank 64, factors kept while the epoch bucket stays.
        {"name": "mlp_step_65536", "kind": "mlp_step", "dims": "784-128-128-128-10", "n_pop": 65536, "bm": 1, "T": 8,
         "rank": 64, "cache": "auto", "noise_reuse": 0, "solver": "adamw"},
        # Test accuracy of the trained network: the clean forward pass over 10 000 encoded images.
        {"name": "mlp_test_set", "kind": "mlp_test", "dims": "784-128-128-10", "images": 10000, "T": 8},
        # One wide perturbed layer with its LIF step, every factor regenerated (the benchmark's headline).
        {"name": "layer_8192x16", "kind": "layer", "n_pop": 8192, "bm": 16, "T": 1, "k": 1024, "a": 1024, "rank": 16,
         "lif": True, "cache": False},
        # A layer of odd sizes over several time steps, factors from a cache, currents out.
        {"name": "layer_ragged", "kind": "layer", "n_pop": 1022, "bm": 12, "T": 3, "k": 500, "a": 250, "rank": 8,
         "lif": False, "cache": True},
        # The update of a transformer's matrices after an evaluation of 4096 members.
        {"name": "matrix_updates", "kind": "updates", "shapes": "16x64*24,64x64*2,256x64*2,64x256*2,256x64*1",
         "n_pop": 4096, "rank": 8, "solver": "adamw"},
        # The token-level spiking transformer: fitness of 4096 members on 32 sequences of 64 tokens.
        {"name": "spiking_lm_4096x32", "kind": "spiking_lm", "n_pop": 4096, "seqs": 32, "L": 64, "d": 64, "heads": 4,
         "blocks": 2, "vocab": 256, "T": 4, "rank": 8},
        # The rate-coded transformer classifier on a chunk of members, factors of the chunk generated once.
        {"name": "snn_transformer_4096", "kind": "snn_transformer", "n_pop": 4096, "tokens": 16, "token_in": 49, "d": 64,
         "heads": 4, "blocks": 2, "classes": 10, "T": 4, "rank": 8, "cache": True},
        # The RWKV-7 language model (bf16 products): fitness of 1024 members on one sequence of 256 tokens.
        {"name": "rwkv_lm_1024", "kind": "rwkv_lm", "layers": 12, "C": 768, "vocab": 50277, "n_pop": 1024, "T": 256,
         "rank": 1},
    ]


# ---- drawn cases ---------------------------------------------------------------------------------------------
def _log(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], spread over the logarithm."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step
    return max(lo, min(hi, v))


def _rank(rng, hi):
    """The ranks in use are mostly powers of two; any other is allowed."""
    common = [r for r in (1, 2, 4, 8, 16, 32, 64, 96, 128) if r <= hi]
    return rng.choice(common) if rng.random() < 0.7 else _log(rng, 1, hi)


def _draw_mlp_step(rng):
    n_pop = _log(rng, 32, 32768, 2)
    T = rng.randint(3, 8)
    bm = _log(rng, 1, max(1, min(64, 524288 // (n_pop * T))))
    widths = [_log(rng, 32, 320) for _ in range(rng.randint(1, 3))]
    dims = [784 if rng.random() < 0.6 else _log(rng, 64, 784, 4)] + widths + [rng.choice([10, 10, 10, 26, 47, 100])]
    cache = rng.choice(["off", "off", "auto"])
    room = (3.3e9 if cache == "auto" else 8e8) / (n_pop / 2 * sum(a + b for a, b in zip(dims, dims[1:])))
    return {"kind": "mlp_step", "dims": "-".join(map(str, dims)), "n_pop": n_pop, "bm": bm, "T": T,
            "rank": _rank(rng, max(1, min(96, int(room)))), "cache": cache,
            "noise_reuse": 0 if cache == "auto" else rng.choice([0, 1]), "solver": rng.choice(["sgd", "adam", "adamw"])}


def _draw_layer(rng):
    n_pop, T = _log(rng, 2, 8192, 2), rng.choice([1, 1, 2, 4, 8])
    bm = _log(rng, 1, max(1, min(64, 131072 // (n_pop * T))))
    k, a = _log(rng, 64, 1024, rng.choice([4, 32])), _log(rng, 16, 1024, rng.choice([1, 32]))
    return {"kind": "layer", "n_pop": n_pop, "bm": bm, "T": T, "k": k, "a": max(a, 16), "rank": _rank(rng, 32),
            "lif": rng.random() < 0.5, "cache": rng.random() < 0.5}


def draw(rng):
    kind = rng.choice(["mlp_step"] * 5 + ["layer"] * 3 + ["member", "mlp_test", "updates", "spiking_lm", "snn_transformer",
                                                         "rwkv_lm"])
    if kind == "mlp_step":
        return _draw_mlp_step(rng)
    if kind == "layer":
        return _draw_layer(rng)
    if kind == "member":
        return {"kind": kind, "bm": _log(rng, 1, 512), "k": _log(rng, 32, 1024), "a": _log(rng, 10, 1024),
                "rank": _rank(rng, 32)}
    if kind == "mlp_test":
        dims = [784] + [_log(rng, 32, 512) for _ in range(rng.randint(1, 3))] + [10]
        return {"kind": kind, "dims": "-".join(map(str, dims)), "images": _log(rng, 500, 20000), "T": rng.randint(3, 8)}
    if kind == "updates":
        d = _log(rng, 48, 768, 8)
        shapes = "%dx%d*%d,%dx%d*%d" % (d, d, rng.randint(1, 8), rng.choice([2, 3, 4]) * d, d, rng.randint(1, 4))
        return {"kind": kind, "shapes": shapes, "n_pop": _log(rng, 64, 4096, 2), "rank": _rank(rng, 16),
                "solver": rng.choice(["sgd", "adam", "adamw"])}
    if kind == "spiking_lm":
        heads = rng.choice([2, 4])
        return {"kind": kind, "n_pop": _log(rng, 16, 1024, 4), "seqs": 4 * rng.randint(1, 8), "L": 8 * rng.randint(2, 12),
                "d": heads * rng.choice([16, 32]), "heads": heads, "blocks": rng.randint(1, 3),
                "vocab": _log(rng, 64, 1024, 32), "T": rng.choice([2, 4, 8]), "rank": rng.choice([8, 8, 16])}
    if kind == "snn_transformer":
        return {"kind": kind, "n_pop": _log(rng, 64, 8192, 2), "tokens": rng.choice([4, 8, 16, 16, 28]),
                "token_in": _log(rng, 16, 64, 1), "d": 64, "heads": rng.choice([2, 4]), "blocks": rng.randint(1, 3),
                "classes": rng.choice([2, 10, 26]), "T": rng.choice([2, 4, 8]), "rank": rng.choice([1, 4, 8, 16]),
                "cache": rng.random() < 0.5}
    return {"kind": kind, "layers": rng.randint(1, 3), "C": rng.choice([256, 512, 768]), "vocab": _log(rng, 512, 50277),
            "n_pop": _log(rng, 8, 256, 2), "T": 32 * rng.randint(1, 12), "rank": rng.choice([1, 1, 2, 4])}


# ---- what a program holds before the call --------------------------------------------------------------------
def _dims(case):
    return [int(v) for v in case["dims"].split("-")]


def _shapes(case):
    out = []
    for part in case["shapes"].split(","):
        shape, count = part.split("*")
        out += [tuple(int(v) for v in shape.split("x"))] * int(count)
    return out


def _images(n, width, g):
    """Synthetic 28x28-like images: a pixel is 0 with probability 0.8, otherwise uniform."""
    img = torch.rand(n, width, device="cuda", generator=g)
    return img * (torch.rand(n, width, device="cuda", generator=g) >= 0.8)


def _solver(name, lr=1e-3):
    return {"sgd": noiser.Solver.sgd, "adam": noiser.Solver.adam, "adamw": noiser.Solver.adamw}[name](lr)


@functools.lru_cache(maxsize=1)
def _rwkv(layers, C, vocab):
    """A program keeps one language model and evaluates it on new tokens: the weights are made once."""
    return RwkvLM(layers, C, vocab, head_size=HEAD, lora_dims=LORA_DIMS, device="cuda", seed=4)


@functools.lru_cache(maxsize=1)
def _spiking(vocab, L, d, heads, blocks, T):
    return SpikingLM(vocab, L, d, heads, blocks, mlp_ratio=4, T=T, device="cuda", seed=2)


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    s = {"case": case, "i": 0}
    kind = case["kind"]
    if kind == "member":
        frozen, nz = noiser.init_noiser([], SIGMA, 0.0, 0, False, 0, case["rank"], noiser.Solver.sgd(0.1))
        s.update(roll=noiser.EggRoll(), frozen=frozen, nz=nz, x=rnd(case["bm"], case["k"]),
                 w=rnd(case["a"], case["k"]) / math.sqrt(case["k"]), info=noiser.IterInfo(0, int(seed) % 1000))
    elif kind == "mlp_step":
        dims, n = _dims(case), case["n_pop"]
        net = models.SnnMlp(dims, device="cuda", seed=int(seed) % 1000, **LIF)
        frozen, nz = noiser.init_noiser(net.params(), SIGMA, 0.0, 0, False, case["noise_reuse"], case["rank"],
                                        _solver(case["solver"]))
        step = models.PopulationStep(net, frozen, nz, models.default_base_keys(len(dims)), case["T"], n, case["bm"],
                                     cache=case["cache"], n_total=n)
        s.update(step=step, img=_images(n * case["bm"], dims[0], g), seed=int(seed) % 65536,
                 labels=torch.randint(0, dims[-1], (n * case["bm"],), device="cuda", generator=g, dtype=torch.int32))
    elif kind == "mlp_test":
        dims = _dims(case)
        s.update(net=models.SnnMlp(dims, device="cuda", seed=int(seed) % 1000, **LIF),
                 img=_images(case["images"], dims[0], g), seed=int(seed) % 65536)
    elif kind == "layer":
        n, a, k = case["n_pop"], case["a"], case["k"]
        s.update(x=rnd(case["T"], n, case["bm"], k), w=rnd(a, k),
                 cache=ops.FactorCache(KEY, 0, 0, case["rank"], a, k, n // 2) if case["cache"] else None)
    elif kind == "updates":
        shapes = _shapes(case)
        params = [rnd(*sh) / math.sqrt(sh[1]) for sh in shapes]
        frozen, nz = noiser.init_noiser(params, SIGMA, 0.0, 0, False, 0, case["rank"], _solver(case["solver"]))
        raw = rnd(case["n_pop"]) * 0.05 - 5.5    # mean log-likelihoods of an untrained model
        s.update(roll=noiser.EggRoll(), frozen=frozen, nz=nz, params=params, raw=raw,
                 keys=models.default_base_keys(len(params)), classes=[noiser.MM_PARAM] * len(params),
                 infos=[noiser.IterInfo(0, i) for i in range(case["n_pop"])])
    elif kind == "spiking_lm":
        model = _spiking(case["vocab"], case["L"], case["d"], case["heads"], case["blocks"], case["T"])
        s.update(model=model, ids=torch.randint(0, case["vocab"], (case["n_pop"], case["seqs"], case["L"]), device="cuda",
                                                generator=g, dtype=torch.int32),
                 noise=SpikingNoise(SIGMA, case["rank"], models.default_base_keys(len(model.params()))))
    elif kind == "snn_transformer":
        n, nt, d = case["n_pop"], case["tokens"], case["d"]
        model = SnnTransformer(case["token_in"], nt, case["classes"], d, case["heads"], case["blocks"], device="cuda",
                               seed=int(seed) % 1000)
        noise = TrainNoise(sigma=SIGMA, rank=case["rank"], base_keys=models.default_base_keys(len(model.params())),
                           pos_emb=rnd(n, nt, d) * SIGMA, out_gain=rnd(n, 1) * SIGMA, beta=rnd(n, 1) * SIGMA)
        if case["cache"]:
            noise.caches = model.build_caches(noise, n)
        s.update(model=model, noise=noise,
                 x=(torch.rand(case["T"], n, nt * case["token_in"], device="cuda", generator=g) < 0.2).float())
    elif kind == "rwkv_lm":
        s.update(model=_rwkv(case["layers"], case["C"], case["vocab"]), noise=RwkvNoise(SIGMA, case["rank"]),
                 ids=torch.randint(0, case["vocab"], (case["n_pop"], case["T"]), device="cuda", generator=g,
                                   dtype=torch.int32))
    else:
        raise ValueError(kind)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "member":
        return s["roll"].do_mm(s["frozen"], s["nz"], s["w"], KEY, s["info"], s["x"])
    if kind == "mlp_step":
        i, s["i"] = s["i"], s["i"] + 1        # the epoch: new spikes every step, new noise when noise_reuse is 1
        step = s["step"]
        raw = step.eval(s["img"], s["labels"], (1, 2, 3 + i, s["seed"]), epoch=i)
        step.update(raw, epoch=i)
        # out_gain's moment is left out: a single number, the difference of two nearly equal sums
        moments = [] if step.moments is None else step.moments[0][:-1]
        return {"fitness": raw, "params": list(step.params), "moments": list(moments)}
    if kind == "mlp_test":
        return s["net"].forward_population(kernels.poisson_encode_fused(s["img"], case["T"], (1, 2, 3, s["seed"]))
                                           .view(case["T"], 1, case["images"], -1))
    if kind == "layer":
        out = ops.perturbed_linear(s["x"], s["w"], n_pop=case["n_pop"], bm=case["bm"], t_steps=case["T"], sigma=SIGMA,
                                   rank=case["rank"], key=KEY, lif=case["lif"], tau_m=20.0, v_th=0.3, cache=s["cache"])
        return out.view(torch.int32) if case["lif"] else out    # spikes are compared as what they are, 0 or 1
    if kind == "updates":
        fit = s["roll"].convert_fitnesses(s["frozen"], s["nz"], s["raw"])
        return s["roll"].do_updates(s["frozen"], s["nz"], s["params"], s["keys"], fit, s["infos"], s["classes"])
    if kind == "spiking_lm":
        return s["model"].fitness(s["ids"], s["noise"])
    if kind == "snn_transformer":
        return s["model"].forward_batched(s["x"], s["noise"])
    return s["model"].fitness(s["ids"], s["noise"], chunk_members=1024)


# ---- what a pass cannot do without ---------------------------------------------------------------------------
def _layer_work(rows, k, a, r):
    """(bytes, flops) of one perturbed layer: x and W in, y out; the product and its rank-r term."""
    return 4.0 * (rows * (k + a) + a * k), 2.0 * rows * (k * a + r * (k + a))


def work(case):
    kind = case["kind"]
    if kind == "member":
        b, f = _layer_work(case["bm"], case["k"], case["a"], case["rank"])
    elif kind == "layer":
        rows, r = case["T"] * case["n_pop"] * case["bm"], case["rank"]
        b, f = _layer_work(rows, case["k"], case["a"], r)
        b += 4.0 * case["n_pop"] / 2 * r * (case["k"] + case["a"]) if case["cache"] else 0.0
    elif kind in ("mlp_step", "mlp_test"):
        # images in; the factors in, once for the forward pass and the update; parameters and moments in and out
        dims = _dims(case)
        test = kind == "mlp_test"
        n, r = (1, 0) if test else (case["n_pop"], case["rank"])
        rows = case["images"] if test else n * case["bm"]
        b, f = 4.0 * rows * (dims[0] + dims[-1]), 0.0
        for l, (k, a) in enumerate(zip(dims, dims[1:])):
            steps = case["T"] if l < len(dims) - 2 else 1
            f += 2.0 * rows * steps * (k * a + r * (k + a)) + (0.0 if test else 1.0 * n * r * k * a)
            b += 4.0 * a * k * (1 if test else 6)
            b += 4.0 * n / 2 * r * (k + a) if not test and case["cache"] == "auto" else 0.0
    elif kind == "updates":
        n, r = case["n_pop"], case["rank"]
        b = sum(4.0 * 6 * a * k for a, k in _shapes(case)) + 4.0 * n
        f = sum(1.0 * n * r * a * k for a, k in _shapes(case))
    elif kind == "spiking_lm":
        n, d, r, v = case["n_pop"], case["d"], case["rank"], case["vocab"]
        rows = float(n) * case["seqs"] * case["L"]
        per_row = case["blocks"] * (2.0 * (12 * d * d + r * 18 * d) + 2.0 * case["L"] * d) + 2.0 * (d * v + r * (d + v))
        b, f = rows * 4 + n * 4 + 4.0 * (2 * v * d + case["blocks"] * 12 * d * d), rows * per_row
    elif kind == "snn_transformer":
        n, nt, d, r, tin = case["n_pop"], case["tokens"], case["d"], case["rank"], case["token_in"]
        rows = float(n) * nt
        widths = 3 * (tin + d) + case["blocks"] * (3 * (case["heads"] * d + d) + 6 * d) + d + case["classes"]
        f = rows * (case["T"] * 3 * 2.0 * (tin * d + r * (tin + d)) + case["blocks"] * (2.0 * (6 * d * d + r * 12 * d) +
                                                                                   4.0 * nt * d))
        b = 4.0 * (case["T"] * rows * tin + rows * d + n * case["classes"])
        b += 4.0 * n / 2 * r * widths if case["cache"] else 0.0
    else:
        C, T, V = case["C"], case["T"], case["vocab"]
        rows = float(case["n_pop"]) * T
        per_layer = 4.0 * C * C + 8.0 * C * C + 2.0 * C * sum(LORA_DIMS)
        f = 2.0 * rows * (case["layers"] * (per_layer + 4.0 * C * HEAD) + C * V)
        b = rows * 4 + 2.0 * (case["layers"] * per_layer + 2.0 * C * V)     # tokens and the bf16 weights
    return {"bytes": b, "flops": f}


def tolerance(case):
    kind = case["kind"]
    if kind in ("member", "layer"):
        # fp32 products; spikes: the mismatch rate the framework states for potentials at the threshold
        return {"rel": 1e-5, "differ": 1e-4}
    if kind == "mlp_step":
        # a potential at its threshold spikes or not: one spike moves a member's fitness by 1e-4 of itself, the z-score
        # divides by a spread of 1e-2 of it, and the gradient (the first moment) follows the z-score.  Two fp32
        # products that add in another order differ by 1e-2 there, and by 1e-5 in the fitness itself
        return {"rel": 2e-2, "max": 0.5}
    if kind == "mlp_test":
        return {"rel": 2e-3, "max": 0.5}
    if kind == "updates":
        # Adam's first step is the gradient's sign: entries near zero may take the other one
        return {"rel": 1e-4, "max": 0.05}
    if kind == "spiking_lm":
        return {"rel": 1e-4, "max": 1e-2}
    if kind == "snn_transformer":
        return {"rel": 1e-4, "max": 1e-2}
    return {"rel": 1e-3, "max": 1e-2}    # bf16 products, a mean over hundreds of tokens
