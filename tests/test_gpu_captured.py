"""Steps that are replayed from captured graphs, against the CPU oracle: what may change between two passes of a circuit has
to reach the replay."""
import numpy as np
import pytest
import torch

import pyjuice_b200 as pj
from helpers import OracleTrainer, folded_input_flows, rel_close
from pyjuice_b200.column import ColumnProgram

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _compiled(kind, latents=8, cats=7):
    torch.manual_seed(3)
    S = pj.structures
    if kind == "hclt":
        tree = S.random_grid_spanning_tree(4, 5, np.random.default_rng(3))
        ns = S.tree_to_hidden_circuit(tree, tree.center(), num_latents=latents, num_cats=cats)
    else:
        ns = S.HMM(seq_length=6, num_latents=latents, num_emits=cats, homogeneous=True)
    return pj.compile(ns, verbose=False).to(DEV)


def _batch(pc, B, seed=0):
    cats = min(layer.max_cats for layer in pc.input_layer_group)
    return torch.randint(0, cats, (B, pc.num_vars), generator=torch.Generator().manual_seed(seed)).to(DEV)


def _step(pc, opt, x):
    lls = pc(x)
    lls.mean().backward()
    opt.step()
    return lls


# (32 states, 600 categories: leaf flows through the transposed shadow)
@pytest.mark.parametrize("kind,latents,cats", [("hclt", 8, 7), ("hmm", 8, 7), ("hmm", 32, 600)])
def test_leaf_flow_buffer_handed_over_between_steps(kind, latents, cats):
    pc = _compiled(kind, latents, cats)
    opt = pj.optim.MiniBatchEM(pc, step_size=0.3, pseudocount=0.1)
    x = _batch(pc, 40)
    for _ in range(4):
        _step(pc, opt, x)
    layer, ref = pc.input_layer_group[0], OracleTrainer(pc)
    arena_part = layer.param_flows
    layer.param_flows = buf = torch.zeros_like(arena_part)
    for i in range(5):
        pc(x).mean().backward()
        ref.accumulate(x)
        if i == 0:
            assert layer.param_flows is buf
            ok, err = rel_close(folded_input_flows(layer, buf), folded_input_flows(layer, ref.ipf[0]))
            assert ok, err
            assert arena_part.abs().max().item() == 0.0
        opt.step()
        ref.update(0.3, 0.1)
        ref.check_params(pc)
        assert buf.abs().max().item() == 0.0                 # cleared with the others
    pc(x).mean().backward()
    before = layer.param_flows.clone()
    pc.init_param_flows(flows_memory=0.5)
    assert torch.equal(layer.param_flows, before * 0.5)


def test_leaf_flow_buffer_that_does_not_fit_is_refused():
    pc = _compiled("hclt")
    pc.init_param_flows(flows_memory=0.0)
    layer = pc.input_layer_group[0]
    n = layer.num_param_flows
    for bad in (torch.zeros(n - 1, device=DEV), torch.zeros(n, device=DEV, dtype=torch.float64),
                torch.zeros(2 * n, device=DEV)[::2]):
        with pytest.raises(ValueError, match="param_flows"):
            layer.param_flows = bad


def test_leaf_flow_buffer_taken_away_between_steps():
    pc = _compiled("hclt")
    opt = pj.optim.MiniBatchEM(pc, step_size=0.3, pseudocount=0.1)
    x = _batch(pc, 40)
    for _ in range(4):
        _step(pc, opt, x)
    ref = OracleTrainer(pc)
    pc.input_layer_group[0].param_flows = None
    with pytest.raises(RuntimeError, match="backward pass"):
        pc.mini_batch_em(step_size=0.3)
    for _ in range(4):
        _step(pc, opt, x)
        ref.accumulate(x)
        ref.update(0.3, 0.1)
        ref.check_params(pc)


def test_limit_of_the_dense_operands_changed_between_steps(monkeypatch):
    monkeypatch.setattr(ColumnProgram, "DENSE_PAR_WORK", 0)
    pc = _compiled("hmm", 256, 11)
    opt = pj.optim.MiniBatchEM(pc, step_size=0.3, pseudocount=0.1)
    x = _batch(pc, 77)
    for _ in range(3):
        _step(pc, opt, x)
    group, = pc._column_program.par(pc._nm.size(1))["dense"]
    assert list(group["tiles"]) == [group["n"]]               # all layers in one product
    ref = OracleTrainer(pc)
    pc.dense_par_max_bytes = 1 << 19
    for _ in range(4):
        _step(pc, opt, x)
        ref.accumulate(x)
        ref.update(0.3, 0.1)
        ref.check_params(pc)
    assert max(group["tiles"]) < group["n"]


@pytest.mark.parametrize("kind,latents,cats", [("hclt", 32, 7), ("hmm", 32, 600)])
def test_parameters_replaced_in_the_module_tables(kind, latents, cats):
    """`torch.func.functional_call` puts other tensors in the place of the parameters for one call."""
    pc, other = _compiled(kind, latents, cats), _compiled(kind, latents, cats)
    with torch.no_grad():
        other.params.copy_(pc.params)
        leaf = other.input_layer_group[0].params
        leaf.copy_(leaf[torch.randperm(leaf.numel(), device=DEV)])
    other.params.data = other.params.data ** 1.5
    x = _batch(pc, 24)
    with torch.no_grad():
        want = other(x)
        own = [pc(x) for _ in range(4)][-1]
        tensors = {n: p.detach().clone() for n, p in other.named_parameters()}
        got = [torch.func.functional_call(pc, tensors, (x,)) for _ in range(4)]
        assert torch.equal(pc(x), own)
    assert (want - own).abs().min().item() > 1e-2
    for g in got:
        assert torch.equal(g, want)


@pytest.mark.parametrize("kind,latents,cats", [("hclt", 32, 7), ("hclt", 128, 7), ("hmm", 32, 600)])
def test_parameters_at_the_address_of_freed_ones(kind, latents, cats):
    """Tables derived from parameters that are gone do not serve others that came to lie where they were."""
    pc, other = _compiled(kind, latents, cats), _compiled(kind, latents, cats)
    x = _batch(pc, 24)
    host = [{n: p.detach().cpu() ** (1.0 + 0.5 * i) for n, p in pc.named_parameters()} for i in range(5)]
    lls, at = [], []
    with torch.no_grad():
        for h in host:
            tensors = {n: p.to(DEV) for n, p in h.items()}
            at.append([t.data_ptr() for t in tensors.values()])
            lls.append(torch.func.functional_call(pc, tensors, (x,)).cpu())
            del tensors
        for h, got in zip(host, lls):
            for n, p in other.named_parameters():
                p.copy_(h[n])
            assert torch.equal(got, other(x).cpu()), at


@pytest.mark.parametrize("kind,latents,cats", [("hclt", 8, 7), ("hclt", 32, 7), ("hclt", 128, 7), ("hmm", 32, 600)])
def test_empty_batches_add_nothing(kind, latents, cats):
    pc = _compiled(kind, latents, cats)
    x = _batch(pc, 24)
    pc.init_param_flows(flows_memory=0.0)
    pc(x).mean().backward()
    flows, total = [pc.param_flows.clone(), pc.input_layer_group[0].param_flows.clone()], pc._cum_flow
    for _ in range(3):
        lls = pc(x[:0])
        assert lls.shape == (0, 1)
        lls.sum().backward()
        pc.backward(x[:0])
        assert pc.node_flows.shape == (pc.num_nodes, 0)
    assert torch.equal(pc.param_flows, flows[0]) and torch.equal(pc.input_layer_group[0].param_flows, flows[1])
    assert pc._cum_flow == total
    pc(x).mean().backward()
    assert (pc.param_flows - 2 * flows[0]).norm() <= 1e-5 * flows[0].norm() and pc._cum_flow == 2 * total


@pytest.mark.parametrize("B", [24, 21])
def test_public_buffers_can_be_given_back_and_written(B):
    pc = _compiled("hclt", 32, 7)
    x = _batch(pc, B)
    want = [pc(x).clone() for _ in range(3)][-1]
    pc.backward(x)
    own = slice(pc.num_dummy_nodes, None)                    # (nobody writes the flows of dummy rows)
    flows = pc.node_flows.clone()
    for name in ("node_mars", "element_mars", "node_flows", "element_flows"):
        setattr(pc, name, None)
        assert getattr(pc, name) is None
        assert torch.equal(pc(x), want)
        pc.backward(x)
        assert torch.equal(pc.node_flows[own], flows[own])
    pc.node_flows = torch.full_like(flows, 0.5)
    assert torch.equal(pc.node_flows, torch.full_like(flows, 0.5))
    with pytest.raises(ValueError, match="does not fit"):
        pc.node_flows = flows[:, :-1]
    pc.node_mars = None
    with pytest.raises(AssertionError, match="forward"):
        pc.backward(x)


@pytest.mark.parametrize("kind,latents,cats", [("hclt", 32, 7), ("hclt", 256, 7), ("hmm", 640, 11), ("hmm", 1280, 11)])
def test_memory_does_not_grow_with_the_number_of_batch_sizes(kind, latents, cats):
    """What a circuit holds after steps of ten sizes: at most what two circuits that saw the largest only would hold."""
    def held(sizes):
        pc = _compiled(kind, latents, cats)
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        opt = pj.optim.MiniBatchEM(pc, step_size=0.3, pseudocount=0.1)
        for B in sizes:
            for _ in range(3):
                _step(pc, opt, _batch(pc, B))
        torch.cuda.synchronize()
        return torch.cuda.memory_allocated() - before
    one, many = held([72]), held([72, 8, 16, 24, 32, 40, 48, 56, 64, 72])
    # (a MB for what graphs own)
    assert many <= 2 * one + (1 << 20), (many, one)


@pytest.mark.parametrize("kind,latents,cats", [("hclt", 64, 7), ("hclt", 256, 7), ("hmm", 640, 11)])
def test_parameter_tiles_have_memory_once_a_pass_needs_them(kind, latents, cats):
    pc = _compiled(kind, latents, cats)
    opt = pj.optim.MiniBatchEM(pc, step_size=0.3, pseudocount=0.1)
    x = _batch(pc, 40)
    for _ in range(3):
        _step(pc, opt, x)
    tiles = [e["buf"] for e in (*pc._packer.entries.values(), *pc._packer.sm_entries.values())]
    assert tiles and all(t.numel() == 0 for t in tiles)       # the column program ran
    ref = OracleTrainer(pc)
    pc.use_column_program = False
    for _ in range(3):
        _step(pc, opt, x)
        ref.accumulate(x)
        ref.update(0.3, 0.1)
    ref.check_params(pc)
    assert all(t.numel() > 0 for t in tiles)


@pytest.mark.parametrize("kind,latents,cats", [("hclt", 8, 7), ("hclt", 64, 7), ("hclt", 128, 7), ("hmm", 32, 600), ("hmm", 640, 11)])
def test_batch_sizes_change_between_steps(kind, latents, cats):
    """An epoch's ragged last batch and the full batches around it, other padded columns of one row width, and (600
    categories) both sides of the line up to which leaf flows go through the transposed shadow."""
    pc = _compiled(kind, latents, cats)
    opt, ref = pj.optim.MiniBatchEM(pc, step_size=0.3, pseudocount=0.1), OracleTrainer(pc)
    sizes = [72] * 4 + [37] + [72] * 4 + [37, 72, 69, 66, 72] + ([608] * 3 + [72] if cats == 600 else [])
    updates = set()
    for i, B in enumerate(sizes):
        x = _batch(pc, B, seed=i)
        lls = _step(pc, opt, x)
        want = ref.accumulate(x)
        assert (lls.detach().double().cpu() - want).abs().max().item() <= 1e-3
        ref.update(0.3, 0.1)
        ref.check_params(pc)
        updates.add(tuple(id(g) for k, g in pc._graphs.items() if k[0] == "em" and g != "warm"))
    if cats == 7:                                             # captured once, and kept when the width changed
        assert len(updates - {()}) == 1


def _structured(kind, latents):
    import random
    torch.manual_seed(3)
    random.seed(3)
    S = pj.structures
    ns = (S.PD((9, 7), latents, split_points=[[3, 6], [3]], num_cats=5) if kind == "pd" else
          S.RAT_SPN(num_vars=40, num_latents=latents, depth=2, num_repetitions=5, num_cats=6))
    return pj.compile(ns, verbose=False).to(DEV)


@pytest.mark.parametrize("kind,latents", [("pd", 64), ("pd", 16), ("rat", 32), ("rat", 8)])
@pytest.mark.parametrize("attr,value", [("WIDE_ITEMS", 1), ("PROD_READS", 0)])
@pytest.mark.parametrize("B", [40, 203])
def test_replayed_launches_of_single_levels(kind, latents, attr, value, B, monkeypatch):
    """Wide levels, products ahead of a level, and parameter flows on two streams, in their captured form."""
    monkeypatch.setattr(ColumnProgram, attr, value)
    pc = _structured(kind, latents)
    opt, ref = pj.optim.MiniBatchEM(pc, step_size=0.3, pseudocount=0.1), OracleTrainer(pc)
    for i in range(4):
        x = _batch(pc, B, seed=i)
        lls = _step(pc, opt, x)
        assert (lls.detach().double().cpu() - ref.accumulate(x)).abs().max().item() <= 1e-3
        ref.update(0.3, 0.1)
        ref.check_params(pc)
    assert all(g != "warm" for k, g in pc._graphs.items() if k[0] == "bk")


@pytest.mark.parametrize("homogeneous", [True, False])
def test_flows_accumulate_across_the_line_of_the_transposed_shadow(homogeneous):
    """Batches of at most as many samples as categories go through the shadow of tied tables, larger ones do not."""
    torch.manual_seed(3)
    pc = pj.compile(pj.structures.HMM(seq_length=5, num_latents=32, num_emits=600, homogeneous=homogeneous), verbose=False).to(DEV)
    opt, ref = pj.optim.FullBatchEM(pc, pseudocount=0.1), OracleTrainer(pc)
    layer = pc.input_layer_group[0]
    for sizes in ([40, 608, 600, 616, 40], [608, 40], [40, 40, 40], [608, 608]):
        for i, B in enumerate(sizes):
            x = _batch(pc, B, seed=i)
            pc(x).mean().backward()
            ref.accumulate(x)
            assert layer._shadow_ok(pc._nm.size(1)) == (homogeneous and B <= 600)
        ok, err = rel_close(folded_input_flows(layer, layer.param_flows), folded_input_flows(layer, ref.ipf[0]))
        assert ok, err
        opt.step()
        ref.update(1.0, 0.1)
        ref.check_params(pc)


@pytest.mark.parametrize("logspace", [True, False])
@pytest.mark.parametrize("kind,latents,cats", [("hclt", 8, 7), ("hclt", 64, 7), ("hclt", 128, 7), ("hclt", 256, 7), ("hmm", 32, 600),
                                               ("hmm", 640, 11), ("hmm", 1280, 11), ("pd", 32, 5), ("rat", 8, 6)])
def test_padding_columns_of_probability_zero(kind, latents, cats, logspace):
    """Rows are padded with samples of category 0; where that category has probability zero they are worth nothing."""
    pc = _structured(kind, latents) if kind in ("pd", "rat") else _compiled(kind, latents, cats)
    layer = pc.input_layer_group[0]
    with torch.no_grad():
        table = layer.params.view(-1, layer.max_cats)
        table[:, 0] = 0.0
        table /= table.sum(dim=1, keepdim=True)
    x = _batch(pc, 21).clamp(min=1)
    ref = OracleTrainer(pc)
    ref.accumulate(x)
    for i in range(3):
        pc.init_param_flows(flows_memory=0.0)
        lls = pc(x)
        pc.backward(x if i else None, logspace_flows=logspace)
        assert torch.isfinite(lls).all()
        ok, err = rel_close(pc.param_flows, ref.pf)
        assert ok, err
        ok, err = rel_close(folded_input_flows(layer, layer.param_flows), folded_input_flows(layer, ref.ipf[0]))
        assert ok, err


@pytest.mark.parametrize("dtype", [torch.uint8, torch.int64])
@pytest.mark.parametrize("B,V", [(3, 1), (1, 33), (70, 31), (5, 2_100_000), (2_100_000, 5)])
def test_inputs_of_any_number_of_variables_and_samples(B, V, dtype):
    from pyjuice_b200 import _lib
    x = torch.randint(0, 200, (B, V), generator=torch.Generator().manual_seed(B), dtype=dtype).to(DEV)
    W = -(-B // 8) * 8
    for src in (x, x.t().contiguous().t()):
        out = torch.full((V, W), -1, dtype=torch.int32, device=DEV)
        _lib.call("pcx_load_inputs", out, src, src.element_size(), B, V, src.stride(0), src.stride(1), W)
        assert torch.equal(out[:, :B], x.t().to(torch.int32)) and not out[:, B:].any()
