"""Workloads by which the speed of the compiled circuits is judged.

A case is one circuit, one batch size and one task, run through the package's public entry points:

    train   ``pc(x)``, ``lls.mean().backward()``, ``MiniBatchEM.step()``: one mini-batch EM step
    epoch   several batches of ``pc(x)`` and ``lls.mean().backward()``, then one ``FullBatchEM.step()``
    query   ``pc(x)`` under ``torch.no_grad()``: log-likelihoods only, as a density model is served

over the four circuit families of the structure generators: hidden trees over an image grid (``hclt``), Poon-Domingos
circuits (``pd``), random tensorised networks (``rat``) and homogeneous hidden Markov models (``hmm``).
"""
import functools
import math
import random

import numpy as np
import torch

import pyjuice_b200 as pj

DEVICE = "cuda:0"
STEP_SIZE, PSEUDOCOUNT = 0.1, 0.1
DTYPES = {"uint8": torch.uint8, "int32": torch.int32, "int64": torch.int64}


def _hclt(task, height, width, latents, cats, batch, dtype, **more):
    return dict(family="hclt", task=task, height=height, width=width, latents=latents, cats=cats, batch=batch,
                dtype=dtype, **more)


def _pd(task, height, width, latents, cats, interval, batch, dtype, **more):
    return dict(family="pd", task=task, height=height, width=width, latents=latents, cats=cats, interval=interval,
                batch=batch, dtype=dtype, **more)


def _rat(task, num_vars, latents, cats, depth, repetitions, batch, dtype, **more):
    return dict(family="rat", task=task, num_vars=num_vars, latents=latents, cats=cats, depth=depth,
                repetitions=repetitions, batch=batch, dtype=dtype, **more)


def _hmm(task, length, latents, cats, batch, dtype, **more):
    return dict(family="hmm", task=task, length=length, latents=latents, cats=cats, batch=batch, dtype=dtype, **more)


def listed():
    return [
        # a tabular data set of 32 small variables: the step is launches and host work
        _hclt("train", 4, 8, 8, 4, 256, "int64", name="train-hclt-32v-k8-b256"),
        # grey-scale images of 28 x 28 pixels, the usual hidden-tree size
        _hclt("train", 28, 28, 128, 256, 512, "uint8", name="train-hclt-784v-k128-b512"),
        # a wider circuit on small images; 100 = the ragged last batch of an epoch
        _hclt("train", 14, 14, 256, 256, 100, "int64", name="train-hclt-196v-k256-b100"),
        # Poon-Domingos circuit over 28 x 28 pixels: shared regions, block-sparse sums, memory-bound products
        _pd("train", 28, 28, 64, 256, 4, 512, "uint8", name="train-pd-784v-k64-b512"),
        # random tensorised network over 784 variables: shallow and wide, many small blocks
        _rat("train", 784, 32, 256, 5, 16, 1024, "uint8", name="train-rat-784v-k32-b1024"),
        # language-model HMM with tied transitions and a large vocabulary: the largest dense work
        _hmm("train", 128, 4096, 32768, 256, "int32", name="train-hmm-128t-k4096-b256"),
        # a mid-size HMM with an odd batch and a small vocabulary
        _hmm("train", 64, 512, 1000, 77, "int64", name="train-hmm-64t-k512-b77"),
        # full-batch EM over four batches: flows accumulate, one update at the end
        _pd("epoch", 16, 16, 32, 256, 4, 200, "uint8", name="epoch-pd-256v-k32-b200", batches=4),
        _hmm("epoch", 32, 1024, 10000, 128, "int64", name="epoch-hmm-32t-k1024-b128", batches=4),
        # one image scored at a time: latency
        _hclt("query", 28, 28, 32, 256, 1, "uint8", name="query-hclt-784v-k32-b1"),
        # scoring a test set in large batches; 1000 = a test set of 10000 in ten batches
        _rat("query", 784, 32, 256, 5, 16, 1000, "int64", name="query-rat-784v-k32-b1000"),
        # scoring sentences with a large-vocabulary HMM
        _hmm("query", 128, 1024, 50257, 64, "int64", name="query-hmm-128t-k1024-b64"),
    ]


def _spread(rng, lo, hi):
    """An integer of [lo, hi], even over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    task = rng.choice(["train", "train", "epoch", "query"])
    more = {"batches": rng.randint(2, 4)} if task == "epoch" else {}
    family = rng.choice(["hclt", "pd", "rat", "hmm"])
    batch = _spread(rng, 1, 1024) if task == "query" else _spread(rng, 16, 768)
    dtype = rng.choice(["uint8", "int32", "int64"])
    if family == "hmm":
        length, latents = _spread(rng, 8, 128), rng.choice([64, 128, 256, 320, 512, 768, 1024, 2048])
        cats = _spread(rng, 64, 50257 if latents <= 512 else 20000)
        return _hmm(task, length, latents, cats, min(batch, 256), rng.choice(["int32", "int64"]), **more)
    cats = _spread(rng, 2, 256)
    if family == "hclt":
        height, width = rng.randint(4, 20), rng.randint(4, 20)
        return _hclt(task, height, width, rng.choice([8, 16, 24, 32, 64, 96, 128, 256]), cats, batch, dtype, **more)
    if family == "pd":
        height, width = rng.randint(8, 20), rng.randint(8, 20)
        return _pd(task, height, width, rng.choice([16, 32, 64]), cats, rng.randint(3, 6), batch, dtype, **more)
    return _rat(task, rng.randint(64, 784), rng.choice([8, 16, 32, 64]), cats, rng.randint(3, 5), rng.randint(4, 12),
                batch, dtype, **more)


# ---- circuits ------------------------------------------------------------------------------------------------------

def _structure(case):
    """The circuit's node DAG.  What is random in a structure (tree, scope splits) is the same for every seed."""
    S, K, C = pj.structures, case["latents"], case["cats"]
    torch.manual_seed(11)
    random.seed(11)
    if case["family"] == "hclt":
        tree = S.random_grid_spanning_tree(case["height"], case["width"], np.random.default_rng(11))
        return S.tree_to_hidden_circuit(tree, tree.center(), num_latents=K, num_cats=C)
    if case["family"] == "pd":
        # cut positions are interior: a cut next to the border is not a split point of the generator
        cuts = [[p for p in range(case["interval"], n, case["interval"]) if p < n - 1] for n in (case["height"], case["width"])]
        return S.PD((case["height"], case["width"]), num_latents=K, split_points=cuts, num_cats=C)
    if case["family"] == "rat":
        return S.RAT_SPN(num_vars=case["num_vars"], num_latents=K, depth=case["depth"],
                         num_repetitions=case["repetitions"], num_cats=C)
    return S.HMM(seq_length=case["length"], num_latents=K, num_emits=C, homogeneous=True)


def _num_vars(case):
    return case.get("num_vars") or case.get("length") or case["height"] * case["width"]


def _pixels(g, batch, height, width, cats):
    """Smooth random images with ``cats`` levels: low-resolution noise, enlarged, plus pixel noise."""
    low = torch.randn(batch, 1, max(2, height // 4), max(2, width // 4), device=DEVICE, generator=g)
    img = torch.nn.functional.interpolate(low, size=(height, width), mode="bilinear", align_corners=False)[:, 0]
    img = img + 0.25 * torch.randn(batch, height, width, device=DEVICE, generator=g)
    return (torch.special.ndtr(img) * cats).long().clamp(0, cats - 1).reshape(batch, -1)


def _tokens(g, batch, length, cats):
    """Token sequences whose word frequencies follow Zipf's law."""
    u = torch.rand(batch, length, device=DEVICE, generator=g, dtype=torch.float64)
    return ((cats + 1.0) ** u - 1.0).long().clamp(0, cats - 1)


def _inputs(case, g):
    if case["family"] == "hmm":
        x = _tokens(g, case["batch"], case["length"], case["cats"])
    elif case["family"] == "rat":
        side = math.ceil(math.sqrt(case["num_vars"]))
        x = _pixels(g, case["batch"], side, side, case["cats"])[:, :case["num_vars"]].contiguous()
    else:
        x = _pixels(g, case["batch"], case["height"], case["width"], case["cats"])
    return x.to(DTYPES[case["dtype"]])


def prepare(case, seed):
    ns = _structure(case)
    torch.manual_seed(seed)                      # `compile` draws and normalises the parameters
    pc = pj.compile(ns, verbose=False).to(DEVICE)
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    opt = None
    if case["task"] == "train":
        opt = pj.optim.MiniBatchEM(pc, step_size=STEP_SIZE, pseudocount=PSEUDOCOUNT)
    elif case["task"] == "epoch":
        opt = pj.optim.FullBatchEM(pc, pseudocount=PSEUDOCOUNT)
    return dict(task=case["task"], pc=pc, opt=opt, xs=[_inputs(case, g) for _ in range(case.get("batches", 1))])


def run(state):
    pc, opt = state["pc"], state["opt"]
    if state["task"] == "query":
        with torch.no_grad():
            return pc(state["xs"][0])
    scores = []
    for x in state["xs"]:
        lls = pc(x)
        lls.mean().backward()
        scores.append(lls)
    opt.step()
    return dict(lls=scores, params=pc.params.data, leaf_params=[layer.params.data for layer in pc.input_layer_group])


# ---- what a pass cannot do without -----------------------------------------------------------------------------------

@functools.lru_cache(maxsize=64)
def _counts(key):
    """(sum edges, sum parameters, leaf parameters, leaf nodes) of a circuit."""
    edges = sum_params = leaf_params = leaves = 0
    for ns in _structure(dict(key)):
        if ns.is_sum():
            edges += ns.num_edges
            sum_params += 0 if ns.is_tied() else ns.num_edges
        elif ns.is_input():
            leaves += ns.num_nodes
            leaf_params += 0 if ns.is_tied() else ns.num_nodes * ns.dist.num_parameters()
    return edges, sum_params, leaf_params, leaves


def work(case):
    """Parameters and inputs read once, results written once; two operations per sum edge and sample, three times in
    training (values, flows of the children, flows of the edges).  A query looks up one leaf parameter per leaf node and
    sample, and no more than all of them."""
    shape = {k: v for k, v in case.items() if k not in ("name", "task", "batch", "batches", "dtype")}
    edges, sum_params, leaf_params, leaves = _counts(tuple(sorted(shape.items())))
    samples = case["batch"] * case.get("batches", 1)
    io = samples * (_num_vars(case) * torch.empty(0, dtype=DTYPES[case["dtype"]]).element_size() + 4)
    if case["task"] == "query":
        return {"bytes": io + 4.0 * (sum_params + min(leaf_params, leaves * samples)), "flops": 2.0 * edges * samples}
    return {"bytes": io + 8.0 * (sum_params + leaf_params), "flops": 6.0 * edges * samples}


def tolerance(case):
    """fp32 values and flows, carried as logarithms of magnitude up to some thousands (one rounding step of the stored
    value is 2.4e-4 there) through up to a hundred layers, with sums in any order."""
    return {"rel": 1e-5} if case["task"] == "query" else {"rel": 1e-4, "max": 1e-2}
