"""Workloads of the framework's public entry points: what a user has it do, over the sizes it is used at.

A case is one call of ``ARTabPFNPredictor.sample_sequence`` ("sample"), ``evaluate_joint_density``
("density"), ``ARTabPFN.forward`` ("forward": the loss of the training-style masked pass, without
gradients) or ``hybrid_attention`` ("hybrid": the decode attention as a functional operator), with

  model      which network (MODELS below)
  precision  "fp32" or "bf16"
  shared     True: one context for all streams; False: every batch element has its own context
  batch      sample streams, candidate label vectors or datasets
  ctx, targets, features, buffers   row counts and columns

The models keep their weights and a predictor for the life of the process, as a program that
serves requests does; the rows, labels and random numbers come new with every preparation.
"""
from __future__ import annotations

import functools
import math
import os
import sys

import torch

_PKG = os.path.join(os.getcwd(), "ar-nanotabpfn_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import ar_tabpfn  # noqa: E402
from ar_tabpfn.model import create_dense_mask, create_row_mask  # noqa: E402
from ar_tabpfn.model import triton_kernels as operators  # noqa: E402

MODELS = {
    # the network of the benchmark configurations
    "six_layer_192": dict(d_model=192, n_heads=6, n_layers=6, d_ff=768, buffer_size=8, num_components=5),
    # what ARTabPFN() gives without arguments
    "default": dict(d_model=128, n_heads=4, n_layers=6, d_ff=256, buffer_size=8, num_components=5),
    # the default of the training script: deep, narrow, twenty mixture components
    "training_default": dict(d_model=64, n_heads=4, n_layers=12, d_ff=128, buffer_size=32, num_components=20),
    # the smallest benchmark configuration
    "two_layer_64": dict(d_model=64, n_heads=4, n_layers=2, d_ff=128, buffer_size=8, num_components=5),
}


def _case(name, op, model, precision, shared, batch, ctx, targets, features=0, buffers=0):
    return dict(name=name, op=op, model=model, precision=precision, shared=shared, batch=batch, ctx=ctx,
                targets=targets, features=features, buffers=buffers)


def listed():
    return [
        # smallest call: a handful of sample paths on one small table, fp32, the generator's own draws
        _case("sample_small_fp32", "sample", "two_layer_64", "fp32", True, 8, 128, 16, 8),
        # one ordinary request: a few sample paths of one dataset with odd row counts
        _case("sample_few_bf16", "sample", "six_layer_192", "bf16", True, 32, 300, 40, 13),
        # the headline benchmark: 512 sample streams on one shared context
        _case("sample_512_bf16", "sample", "six_layer_192", "bf16", True, 512, 1024, 128, 20),
        # the largest job: thousands of streams on a long, wide context
        _case("sample_4096_bf16", "sample", "six_layer_192", "bf16", True, 4096, 16384, 64, 100),
        # a batch of different datasets, one sample path each (the predictor's default context semantics)
        _case("sample_datasets_bf16", "sample", "six_layer_192", "bf16", False, 64, 500, 50, 20),
        # the constructor's default model in the precision its parameters have
        _case("sample_default_fp32", "sample", "default", "fp32", True, 64, 512, 48, 10),
        # a network as the training script makes it, sampled in bf16
        _case("sample_training_default_bf16", "sample", "training_default", "bf16", True, 100, 1000, 32, 10),
        # log density of the labels of many datasets at once (the teacher-forced benchmark)
        _case("density_datasets_bf16", "density", "six_layer_192", "bf16", False, 64, 2048, 256, 20),
        # a few candidate label vectors scored on one dataset, odd sizes
        _case("density_few_bf16", "density", "six_layer_192", "bf16", True, 24, 700, 37, 20),
        # the same for a batch of datasets in fp32, where log densities are compared to 1e-5
        _case("density_default_fp32", "density", "default", "fp32", False, 16, 200, 64, 10),
        # validation loss of the training script's model on one of its batches
        _case("forward_training_default_fp32", "forward", "training_default", "fp32", False, 64, 256, 256, 10, 32),
        # decode attention as an operator: one query per stream, private buffers of ragged length
        _case("hybrid_1024_bf16", "hybrid", "", "bf16", True, 1024, 4096, 0, 0, 63),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cost(case):
    # fp32 arithmetic runs at a small fraction of the tensor cores' rate
    return work(case)["flops"] * (1 if case["precision"] == "bf16" else 20)


def draw(rng):
    most = _cost(next(c for c in listed() if c["name"] == "sample_4096_bf16"))
    while True:
        op = rng.choice(["sample"] * 5 + ["density"] * 3 + ["forward", "hybrid"])
        precision = rng.choice(["fp32", "bf16"])
        model = rng.choice(sorted(MODELS))
        if op == "hybrid":
            c = _case("", op, "", precision, True, _log_int(rng, 1, 2048), _log_int(rng, 64, 8192), 0, 0,
                      rng.randint(1, 64))
        elif op == "forward":
            c = _case("", op, model, precision, False, _log_int(rng, 1, 64), _log_int(rng, 16, 1024),
                      _log_int(rng, 8, 512), rng.randint(1, 40),
                      rng.randint(1, MODELS[model]["buffer_size"]))
        else:
            shared = rng.random() < 0.6
            c = _case("", op, model, precision, shared, _log_int(rng, 1, 4096 if shared else 96),
                      _log_int(rng, 16, 16384 if shared else 2048),
                      _log_int(rng, 4, 128 if op == "sample" else 256), _log_int(rng, 1, 100))
        rows = c["batch"] * max(c["targets"], 1)
        if _cost(c) <= 0.5 * most and rows <= 65536:
            del c["name"]
            return c


# ------------------------------------------------------------------ what a program keeps
@functools.lru_cache(maxsize=None)
def _model(name, features, precision):
    torch.manual_seed(7)
    m = ar_tabpfn.ARTabPFN(num_features=features, **MODELS[name]).eval()
    with torch.no_grad():
        for mod in m.modules():
            if isinstance(mod, torch.nn.Linear):
                torch.nn.init.xavier_uniform_(mod.weight)
        for p in m.parameters():
            if precision == "bf16":  # bf16 serving: weights as a bf16 checkpoint holds them
                p.copy_(p.to(torch.bfloat16).float())
            p.requires_grad_(False)
    return m.cuda()


@functools.lru_cache(maxsize=None)
def _predictor(name, features, precision, shared):
    return ar_tabpfn.ARTabPFNPredictor.from_trained_model(
        _model(name, features, precision), backend="triton_shared_context" if shared else "flex_attention",
        precision=precision)


def _tables(g, n, rows, features):
    """n tables: x ~ N(0, 1), standardised; y = tanh-MLP of x plus N(0, 0.1^2) noise."""
    r = functools.partial(torch.randn, generator=g, device="cuda")
    x = r(n, rows, features)
    x = (x - x.mean(1, keepdim=True)) / (x.std(1, keepdim=True) + 1e-6)
    h = torch.tanh(x @ (r(n, features, 32) / features ** 0.5))
    h = torch.tanh(h @ (r(n, 32, 32) / 32 ** 0.5))
    y = (h @ (r(n, 32, 1) / 32 ** 0.5))[..., 0] + 0.1 * r(n, rows)
    return x, y


def _variates(g, steps, batch, components):
    """Random numbers handed to the sampler.  The mixture component of every draw is picked here,
    evenly over the components, and its Exp(1) variate made small enough that the pick stands
    whatever the weights: a near tie would otherwise go either way with the rounding of bf16."""
    expo = torch.empty(steps, batch, components, device="cuda").exponential_(1.0, generator=g).clamp_(min=0.02)
    pick = torch.randint(components, (steps, batch, 1), device="cuda", generator=g)
    expo.scatter_(2, pick, 1e-6)
    return expo, torch.randn(steps, batch, device="cuda", generator=g)


def _own_draws(case):
    """Small fp32 jobs draw from torch's generator inside the call; the others are given their numbers."""
    return case["precision"] == "fp32" and case["batch"] * case["targets"] <= 4096


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    B, Nc, Nt, Nb, F = (case[k] for k in ("batch", "ctx", "targets", "buffers", "features"))
    op = case["op"]
    if op == "hybrid":
        H, Dh = 4, 32
        dt = torch.bfloat16 if case["precision"] == "bf16" else torch.float32
        r = lambda *s: torch.randn(*s, generator=g, device="cuda").to(dt)
        lens = torch.randint(0, Nb + 1, (B,), device="cuda", generator=g)
        mask = (torch.arange(Nb, device="cuda")[None] < lens[:, None]).view(B, 1, 1, Nb)
        return dict(op=op, args=(r(B, H, 1, Dh), r(H, Nc, Dh), r(H, Nc, Dh), r(B, H, Nb, Dh), r(B, H, Nb, Dh), mask))
    n = 1 if case["shared"] else B
    x, y = _tables(g, n, Nc + Nb + Nt, F)
    if case["precision"] == "bf16":
        x, y = x.to(torch.bfloat16).float(), y.to(torch.bfloat16).float()
    parts = [x[:, :Nc], y[:, :Nc], x[:, Nc:Nc + Nb], y[:, Nc:Nc + Nb], x[:, Nc + Nb:], y[:, Nc + Nb:]]
    # a shared context is one table seen by every stream; different datasets are stacked
    xc, yc, xb, yb, xt, yt = [p.expand(B, *p.shape[1:]) if case["shared"] else p.contiguous() for p in parts]
    if op == "forward":
        dt = torch.bfloat16 if case["precision"] == "bf16" else torch.float32
        return dict(op=op, model=_model(case["model"], F, case["precision"]),
                    args=dict(x_context=xc.to(dt), y_context=yc.to(dt), x_buffer=xb.to(dt), y_buffer=yb.to(dt),
                              x_target=xt.to(dt), y_target=yt.to(dt),
                              mask_features=create_dense_mask(1, device="cuda"),
                              mask_rows=create_row_mask(Nc + Nb + Nt, Nc, Nb, device="cuda")))
    pred = _predictor(case["model"], F, case["precision"], case["shared"])
    if op == "density":
        if case["shared"]:  # candidate label vectors for the same rows
            yt = yt + 0.3 * torch.randn(B, Nt, generator=g, device="cuda")
        return dict(op=op, pred=pred, args=(xc, yc, xt, yt))
    K = MODELS[case["model"]]["num_components"]
    return dict(op=op, pred=pred, args=(xc, yc, xt), seed=seed,
                variates=None if _own_draws(case) else _variates(g, Nt, B, K))


def run(state):
    op = state["op"]
    if op == "hybrid":
        return operators.hybrid_attention(*state["args"])
    if op == "forward":
        loss = state["model"](**state["args"])
        return loss, state["model"].last_logdens
    pred = state["pred"]
    if op == "density":
        return pred.evaluate_joint_density(*state["args"])
    if state["variates"] is None:
        torch.cuda.manual_seed(state["seed"])
    samples = pred.sample_sequence(*state["args"], variates=state["variates"])
    return samples, pred.last_logdens, pred.last_components


# ------------------------------------------------------------------ the least a pass can do
def work(case):
    """Flops: products of every token with the weights (the feature attention over one token folds
    into one matrix) and attention of every query over its keys, 2 per multiply-add.  Bytes: inputs
    and weights once, results once."""
    B, Nc, Nt, Nb, F = (case[k] for k in ("batch", "ctx", "targets", "buffers", "features"))
    op = case["op"]
    size = 2 if case["precision"] == "bf16" else 4
    if op == "hybrid":
        H, Dh = 4, 32
        keys = Nc + Nb / 2  # lengths are uniform from 0 to Nb
        return {"bytes": size * H * Dh * (2 * B + 2 * Nc + B * Nb), "flops": 4.0 * B * H * Dh * keys}
    m = MODELS[case["model"]]
    D, Dff, L, K = m["d_model"], m["d_ff"], m["n_layers"], m["num_components"]
    G = 1 if case["shared"] else B
    token = 10 * D * D + 4 * D * Dff  # fold, Q | K | V, out-projection, MLP
    head = 2 * D * Dff + 6 * Dff * K
    # context rows: the last layer only has to give its keys and values
    flops = G * Nc * ((L - 1) * token + 6.0 * D * D) + (L - 1) * 4.0 * D * G * Nc * Nc
    weights = L * (5 * D * D + 2 * D * Dff) + D * Dff + 3 * K * Dff
    values = G * Nc * (F + 1) + G * Nt * F
    if op == "forward":
        queries, buffers, seen = B * Nt, B * Nb, Nb / 2
        values += G * Nb * (F + 1) + 2 * B * Nt
    else:
        queries, buffers, seen = B * Nt, B * (Nt - 1), Nt / 2
        values += 2 * B * Nt + (B * Nt * (K + 2) if op == "sample" else 0)
    # target tokens go through every layer; of a buffer token the last layer takes the keys and values
    flops += queries * (L * token + head) + buffers * ((L - 1) * token + 6.0 * D * D)
    flops += 4.0 * D * (Nc + seen) * (L * queries + (L - 1) * buffers)
    return {"bytes": 4 * values + size * weights, "flops": flops}


def tolerance(case):
    """bf16: rounding of stored queries, keys and values.  fp32: sums over up to 16384 keys and 12
    layers in another order."""
    return {"rel": 1e-2} if case["precision"] == "bf16" else {"rel": 3e-5}
