"""The calls that users of this library make, as timed cases: the neighbour path at inference
(``BinnedSelectKnn`` + ``AccumulateKnn``), GravNet layers, training steps (forward and backward),
object condensation, the sibling ops of the graph-condensation layers, and batches that live in
host memory.  Sizes are those of the benchmark configurations and of the test suite, and what lies
between them.

Inputs have the distributions of ``hgcalml_b200.synth`` (Gaussian showers of very different density
on uniform noise, N(0,1) features, Gaussian blobs with a Beta(0.5, 5) spectrum), drawn on the GPU.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from hgcalml_b200.accknn_op import AccumulateKnn, AccumulateKnnDifferentiable
from hgcalml_b200.assign_condensate_op import BuildAndAssignCondensatesBinned
from hgcalml_b200.binned_select_knn_op import BinnedSelectKnn, BinnedSelectKnnDifferentiable
from hgcalml_b200.GravNetLayersRagged import DistanceWeightedMessagePassing, RaggedGravNet
from hgcalml_b200.local_distance_op import LocalDistance
from hgcalml_b200.pipeline import KnnAccumulatePipeline
from hgcalml_b200.push_knn_op import PushKnn


# ------------------------------------------------------------------------------------------- cases
def _infer(events, lo, hi, dims, K, F, shape="showers", n_bins=0, argmax=True):
    """Neighbour search and accumulation over ``events`` events of ``lo`` to ``hi`` hits."""
    return dict(kind="infer", events=events, lo=lo, hi=hi, dims=dims, K=K, F=F, shape=shape, n_bins=n_bins,
                argmax=argmax)


def _gravnet(events, lo, hi, dims, K, F, blocks, passes):
    """``blocks`` GravNet layers on top of each other, then ``passes`` message-passing steps (0: none)."""
    return dict(kind="gravnet", events=events, lo=lo, hi=hi, dims=dims, K=K, F=F, blocks=blocks, passes=passes)


def _train(events, lo, hi, dims, K, F):
    """The neighbour path forward and backward, as in a training step."""
    return dict(kind="train", events=events, lo=lo, hi=hi, dims=dims, K=K, F=F)


def _push(events, lo, hi, dims, K, F):
    """LocalDistance and PushKnn on a given neighbour table, forward and backward."""
    return dict(kind="push", events=events, lo=lo, hi=hi, dims=dims, K=K, F=F)


def _condense(events, lo, hi, dims, max_beta, keep_noise, per_hit_radius):
    """Object condensation after the network: condensate finding and assignment of every hit."""
    return dict(kind="condense", events=events, lo=lo, hi=hi, dims=dims, max_beta=max_beta, keep_noise=keep_noise,
                per_hit_radius=per_hit_radius)


def _host(events, lo, hi, dims, K, F):
    """The inference path for a batch in pinned host memory, results back in host memory."""
    return dict(kind="host", events=events, lo=lo, hi=hi, dims=dims, K=K, F=F)


def listed():
    named = [
        # one small event at a time, as an online service would see it: launches and host time count
        ("infer_tiny", _infer(1, 700, 700, 3, 16, 32)),
        # configuration 1: one event of 20k uniform hits, bins given by the caller
        ("infer_20k_uniform", _infer(1, 20000, 20000, 3, 16, 32, shape="uniform", n_bins=10)),
        # small ragged events, odd neighbour count, a feature width that is no multiple of four
        ("infer_odd_ragged", _infer(7, 1500, 31000, 5, 41, 22)),
        # configuration 2: a ragged batch of four mid-size shower events
        ("infer_ragged_4", _infer(4, 50000, 150000, 4, 64, 64)),
        # configuration 5: the large batch the throughput metric is quoted on
        ("infer_batch_64", _infer(64, 200000, 200000, 4, 64, 64)),
        # configuration 3: four GravNet blocks on one full-size event (the predictor's batch size is 1)
        ("gravnet_stack_200k", _gravnet(1, 200000, 200000, 4, 64, 64, 4, 0)),
        # a training step on a few small events, and on one full-size event
        ("train_small", _train(3, 5000, 9000, 3, 24, 32)),
        ("train_200k", _train(1, 200000, 200000, 4, 64, 64)),
        # configuration 4: condensation of four full-size events
        ("condense_4x200k", _condense(4, 200000, 200000, 3, True, False, False)),
        # condensation of a small ragged batch with per-hit radii, noise kept
        ("condense_small", _condense(3, 2000, 9000, 3, False, True, True)),
        # graph condensation: distances and pushed features on given neighbour tables, with gradients
        ("push_60k", _push(2, 25000, 35000, 4, 16, 32)),
        # a batch in host memory through the chunked pipeline
        ("host_8x100k", _host(8, 100000, 100000, 4, 64, 64)),
    ]
    return [dict(c, name=n) for n, c in named]


def draw(rng):
    def log_int(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["infer"] * 6 + ["gravnet"] * 3 + ["train"] * 4 + ["condense"] * 3 + ["push"] * 2 + ["host"])
    K = log_int(8, 100)
    F = rng.choice([8, 16, 16, 32, 32, 64, 64, 64, 96, 128, rng.randint(6, 70)])
    dims = rng.choice([2, 3, 3, 4, 4, 4, 5, 6])
    # hits of the batch, then how many events they are spread over
    top = {"infer": 3000000, "gravnet": 250000, "train": 400000, "condense": 1000000, "push": 300000,
           "host": 800000}[kind]
    total = log_int(600, top)
    # keep the neighbour tables and feature rows of a drawn batch below those of the largest listed one
    total = max(600, min(total, int(12.8e6 * 64 * 64 / (4 * K * max(F, 16)))))
    # events of about 300 to 250k hits
    events = max(min(log_int(1, 40), max(1, total // 300)), -(-total // 250000))
    mean = total / events
    spread = rng.choice([0., 0.3, 0.8])
    lo, hi = int(mean * (1 - spread)), int(mean * (1 + spread)) + rng.randint(0, 3)
    if kind == "infer":
        shape = rng.choice(["showers", "showers", "showers", "uniform"])
        return _infer(events, lo, hi, dims, K, F, shape=shape, argmax=rng.random() < 0.6)
    if kind == "gravnet":
        return _gravnet(events, lo, hi, max(3, dims), K, F, rng.randint(1, 3), rng.choice([0, 1, 3]))
    if kind == "train":
        return _train(events, lo, hi, dims, K, F)
    if kind == "condense":
        return _condense(events, lo, hi, rng.choice([2, 3, 3, 3, 4]), rng.random() < 0.5, rng.random() < 0.3,
                         rng.random() < 0.5)
    if kind == "push":
        return _push(events, lo, hi, dims, K, F)
    return _host(events, lo, hi, dims, K, F)


# ------------------------------------------------------------------------------------------ inputs
def _sizes(case, seed=None):
    """Hits per event: spread evenly over lo .. hi, in an order that depends on the seed."""
    e, lo, hi = case["events"], case["lo"], case["hi"]
    sizes = [lo + (hi - lo) * i // max(1, e - 1) for i in range(e)] if e > 1 else [(lo + hi) // 2]
    if seed is not None:
        np.random.default_rng(seed).shuffle(sizes)
    return sizes


def _hits(case):
    return sum(_sizes(case))


def _showers(sizes, dims, seed, g, dev):
    """Per event 300 Gaussian showers (fewer in small events) with exponentially distributed hit counts
    and 10 % uniform noise, in random order."""
    out = []
    for k, n in enumerate(sizes):
        rng = np.random.default_rng([seed, k])
        n_showers = max(3, min(300, n // 100))
        centres = torch.as_tensor(rng.uniform(-1., 1., (n_showers, dims)), dtype=torch.float32, device=dev)
        sigma = torch.as_tensor(rng.uniform(0.01, 0.05, n_showers), dtype=torch.float32, device=dev)
        w = np.cumsum(rng.exponential(1., n_showers))
        edges = torch.as_tensor(w / w[-1], dtype=torch.float32, device=dev)
        u = torch.rand(n, generator=g, device=dev)
        noise = u < 0.1
        label = torch.searchsorted(edges, ((u - 0.1) / 0.9).clamp_min(0.)).clamp_max(n_showers - 1)
        x = centres[label] + sigma[label, None] * torch.randn((n, dims), generator=g, device=dev)
        y = torch.rand((n, dims), generator=g, device=dev) * 2. - 1.
        out.append(torch.where(noise[:, None], y, x))
    return torch.cat(out)


def _blobs(sizes, dims, seed, g, dev):
    """Cluster coordinates and betas: one blob per 400 hits, the hit closest to each centre has a high beta."""
    cc, bb = [], []
    for k, n in enumerate(sizes):
        n_blobs = max(3, n // 400)
        rng = np.random.default_rng([seed, k])
        centres = torch.as_tensor(rng.uniform(-3., 3., (n_blobs, dims)), dtype=torch.float32, device=dev)
        label = torch.randint(0, n_blobs, (n,), generator=g, device=dev)
        off = 0.1 * torch.randn((n, dims), generator=g, device=dev)
        # Beta(0.5, 5) = X / (X + Y) with X ~ Gamma(0.5) (half a squared normal), Y ~ Gamma(5) (five exponentials)
        x = torch.randn(n, generator=g, device=dev).square() * 0.5
        y = -torch.rand((n, 5), generator=g, device=dev).clamp_min(1e-12).log().sum(dim=1)
        beta = x / (x + y)
        d2 = off.square().sum(dim=1)
        nearest = torch.full((n_blobs,), float("inf"), device=dev).scatter_reduce(0, label, d2, "amin")
        top = 0.8 + 0.2 * torch.rand(n, generator=g, device=dev)
        cc.append(centres[label] + off)
        bb.append(torch.where(d2 == nearest[label], top, beta))
    return torch.cat(cc), torch.cat(bb)[:, None]


def _dense(layer, g):
    with torch.no_grad():
        fan_in = layer.kernel.shape[0]
        layer.kernel.copy_(torch.randn(layer.kernel.shape, generator=g, device=g.device) / math.sqrt(fan_in))
        if layer.bias is not None:
            layer.bias.copy_(0.1 * torch.randn(layer.bias.shape, generator=g, device=g.device))


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    sizes = _sizes(case, seed)
    n, dims, kind = sum(sizes), case["dims"], case["kind"]
    splits = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    s = dict(case=case, rs=torch.as_tensor(splits, device=dev))
    if kind == "condense":
        s["cc"], s["beta"] = _blobs(sizes, dims, seed, g, dev)
        s["dist"] = torch.full((n, 1), 0.5, device=dev)
        if case["per_hit_radius"]:
            s["dist"] = 0.3 + 0.4 * torch.rand((n, 1), generator=g, device=dev)
        return s
    K, F = case["K"], case["F"]
    s["feats"] = torch.randn((n, F), generator=g, device=dev)
    if kind == "gravnet":
        layers = [RaggedGravNet(K - 1, dims, F, F, n_in=F).to(dev) for _ in range(case["blocks"])]
        for layer in layers:
            for d in (layer.input_feature_transform, layer.input_spatial_transform, layer.output_feature_transform):
                _dense(d, g)
        s["layers"] = layers
        s["messages"] = None
        if case["passes"]:
            s["messages"] = DistanceWeightedMessagePassing(_pass_widths(case), n_in=F).to(dev)
            for d in s["messages"].feature_tranformation_dense:
                _dense(d, g)
        return s
    if case.get("shape") == "uniform":
        s["coords"] = torch.rand((n, dims), generator=g, device=dev)
    else:
        s["coords"] = _showers(sizes, dims, seed, g, dev)
    if kind == "host":
        for name in ("coords", "feats"):
            s[name] = s[name].cpu().pin_memory()
        s["rs"] = splits
        s["out"] = torch.empty((n, 2 * F), dtype=torch.float32).pin_memory()
        s["pipe"] = KnnAccumulatePipeline(K, dev, events_per_chunk=1)
    elif kind == "train":
        s["coords"].requires_grad_(True)
        s["feats"].requires_grad_(True)
        s["grad"] = torch.randn((n, 2 * F), generator=g, device=dev)
    elif kind == "push":
        s["idx"], _ = BinnedSelectKnn(K, s["coords"], s["rs"])
        s["coords"].requires_grad_(True)
        s["feats"].requires_grad_(True)
        s["grad"] = torch.randn((n, F), generator=g, device=dev)
    return s


def _pass_widths(case):
    """Widths of the message-passing steps: halved every other step, as the layers are used."""
    return [max(8, case["F"] >> (i // 2)) for i in range(case["passes"])]


# ------------------------------------------------------------------------------------------- calls
def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "infer":
        idx, d2, sorting = BinnedSelectKnn(c["K"], s["coords"], s["rs"], n_bins=c["n_bins"] or None,
                                           return_sorting=True)
        out, arg = AccumulateKnn(d2, s["feats"], idx, order=sorting, distance_scale=10., with_max_idxs=c["argmax"])
        return idx, d2, out, arg
    if kind == "gravnet":
        with torch.no_grad():
            x, res = s["feats"], []
            for layer in s["layers"]:
                x, coords, idx, d2 = layer([x, s["rs"]])
                res += [coords, idx, d2]
            if s["messages"] is not None:
                x = s["messages"]([x, idx, d2])
            return [x] + res
    if kind == "train":
        idx, d2 = BinnedSelectKnnDifferentiable(c["K"], s["coords"], s["rs"])
        out, arg = AccumulateKnnDifferentiable(10. * d2, s["feats"], idx)
        gc, gf = torch.autograd.grad(out, (s["coords"], s["feats"]), s["grad"])
        return idx, d2, out, arg, gc, gf
    if kind == "push":
        d2 = LocalDistance(s["coords"], s["idx"])
        out = PushKnn(torch.exp(-10. * d2), s["feats"], s["idx"])
        gc, gf = torch.autograd.grad(out, (s["coords"], s["feats"]), s["grad"])
        return d2, out, gc, gf
    if kind == "condense":
        asg, asso, alpha, is_cond, n_cond = BuildAndAssignCondensatesBinned(
            s["cc"], s["beta"], s["dist"], s["rs"], 0.1, assign_by_max_beta=c["max_beta"],
            keep_noise=c["keep_noise"])
        # the list of condensates has as many entries as there are condensates: kept in a row per hit
        alphas = torch.nn.functional.pad(alpha, (0, asg.shape[0] - alpha.shape[0]), value=-1)
        return asg, asso, alphas, is_cond, n_cond
    return s["pipe"].run(s["coords"], s["feats"], s["rs"], s["out"])


# -------------------------------------------------------------------------------------------- work
def work(case):
    """Inputs read once, outputs written once; operations of the neighbour rows only (distances of the
    K nearest, weighted mean and maximum over them), not of the search that finds them."""
    n, C, kind = _hits(case), case["dims"], case["kind"]
    if kind == "condense":
        # coordinates, beta, radius; assignment, association, flag per hit
        return {"bytes": n * (4 * C + 8 + 9), "flops": n * 3 * C}
    K, F = case["K"], case["F"]
    search = 4 * C + 8 * K
    if kind == "infer":
        return {"bytes": n * (search + 4 * F + 8 * F + (4 * F if case["argmax"] else 0)),
                "flops": n * K * 3 * (C + F)}
    if kind == "gravnet":
        b, f = n * 4 * F, 0
        for _ in range(case["blocks"]):
            b += n * (search + 4 * F) + 4 * (F * F + F * C + 3 * F * F)
            f += n * (2 * F * (F + C) + 2 * 3 * F * F + K * 3 * (C + F))
        w_in = F
        for w in _pass_widths(case) if case["passes"] else []:
            b += n * 8 * w + 4 * w_in * w
            f += n * (2 * w_in * w + K * 3 * w)
            w_in = 2 * w
        return {"bytes": b + (n * 4 * F if case["passes"] else 0), "flops": f}
    if kind == "train":
        # forward, then the gradient of the features and of the coordinates from that of the result
        return {"bytes": n * (search + 4 * F + 12 * F + 8 * F + 4 * F + 4 * C),
                "flops": n * K * (3 * (C + F) + 4 * F + 6 * C)}
    if kind == "push":
        return {"bytes": n * (4 * C + 8 * K + 4 * F + 4 * F + 4 * F + 4 * F + 4 * C),
                "flops": n * K * (3 * C + 2 * F + 4 * F + 6 * C)}
    return {"bytes": n * (4 * C + 4 * F + 8 * F), "flops": n * K * 3 * (C + F)}


def tolerance(case):
    kind = case["kind"]
    if kind == "condense":
        return "exact"
    if kind == "gravnet":
        # sums of float32 products in another order move the learned coordinates by an ulp, and with
        # them, rarely, two neighbours that are almost equally far
        return {"rel": 3e-5, "max": 0.05, "differ": 1e-4}
    # float32 sums; the arg-max of two products that agree to the last bits may go either way
    return {"rel": 1e-5, "differ": 1e-6}
