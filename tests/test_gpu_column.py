"""The column program (all levels of a circuit of small node blocks in one launch, wide levels on their own) against the CPU
oracle and against the per-layer kernels, at the sizes where its pieces meet: batches around the 8-, 16- and 32-column
tiles, node blocks on both sides of the fp32 / tensor-core line, levels wide enough for a launch of their own, products of
one, two and many children, stored element values, block-sparse tables and shared leaves."""
import pytest
import torch

import pyjuice_b200 as pj
from helpers import check_against_oracle
from pyjuice_b200.column import ColumnProgram

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _circuit(kind, latents):
    torch.manual_seed(3)
    import random
    random.seed(3)
    import numpy as np
    S = pj.structures
    if kind == "hclt":
        tree = S.random_grid_spanning_tree(4, 5, np.random.default_rng(3))
        return S.tree_to_hidden_circuit(tree, tree.center(), num_latents=latents, num_cats=7)
    if kind == "pd":
        return S.PD((9, 7), latents, split_points=[[3, 6], [3]], num_cats=5)
    if kind == "rat":
        return S.RAT_SPN(num_vars=40, num_latents=latents, depth=2, num_repetitions=5, num_cats=6)
    return S.HMM(seq_length=9, num_latents=latents, num_emits=11, homogeneous=True)


def _program(pc):
    assert pc._column_plan() is not None
    return pc._column_program


@pytest.mark.parametrize("B", [1, 8, 31, 200, 257])
@pytest.mark.parametrize("kind,latents", [("hclt", 8), ("hclt", 24), ("hclt", 64), ("hclt", 96), ("pd", 16), ("pd", 64),
                                          ("rat", 32), ("rat", 8), ("hmm", 64), ("hmm", 320), ("hmm", 4),
                                          ("hmm", 128), ("hmm", 512), ("hmm", 1024), ("hclt", 128), ("hclt", 256), ("rat", 128)])
def test_against_oracle(kind, latents, B):
    pc = pj.compile(_circuit(kind, latents)).to(DEV)
    cats = min(l.max_cats for l in pc.input_layer_group)
    x = torch.randint(0, cats, (B, pc.num_vars), generator=torch.Generator().manual_seed(B))
    errs = check_against_oracle(pc, x, step=0.2, pseudo=0.1)
    assert latents >= 128 or pc._column_plan() is not None
    pc.validate_tables()
    print(errs)


@pytest.mark.parametrize("kind,latents", [("hclt", 64), ("hclt", 8), ("pd", 32), ("pd", 64), ("rat", 32), ("rat", 16)])
@pytest.mark.parametrize("logspace", [True, False])
@pytest.mark.parametrize("B", [40, 264])
def test_wide_levels(kind, latents, logspace, B, monkeypatch):
    """Every level on its own (as in circuits that fill the machine), against the oracle."""
    monkeypatch.setattr(ColumnProgram, "WIDE_ITEMS", 1)
    pc = pj.compile(_circuit(kind, latents)).to(DEV)
    cats = min(l.max_cats for l in pc.input_layer_group)
    x = torch.randint(0, cats, (B, pc.num_vars), generator=torch.Generator().manual_seed(B))
    check_against_oracle(pc, x, step=0.2, pseudo=0.1, logspace_flows=logspace)
    launches = [l for m in (0, 1) for l in _program(pc).plan(pc._nm.size(1))[m]["launches"] if not isinstance(l, list)]
    assert any(l[2][3] > 0 for l in launches)
    pc.validate_tables()


@pytest.mark.parametrize("latents", [256, 384, 640])
@pytest.mark.parametrize("logspace", [True, False])
@pytest.mark.parametrize("B,most", [(1, 1 << 30), (77, 1 << 30), (256, 1 << 30), (77, 1 << 19)])
def test_tied_parameter_flows_as_one_product(latents, logspace, B, most, monkeypatch):
    """Tied transitions contracted over all their layers' samples: one part and several, a last chunk that is partly empty,
    output tiles that are partly empty, and (`most`) operand buffers that hold a few layers at a time."""
    monkeypatch.setattr(ColumnProgram, "DENSE_PAR_WORK", 0)
    pc = pj.compile(_circuit("hmm", latents)).to(DEV)
    pc.dense_par_max_bytes = most
    x = torch.randint(0, 11, (B, pc.num_vars), generator=torch.Generator().manual_seed(B))
    check_against_oracle(pc, x, step=0.2, pseudo=0.1, logspace_flows=logspace)
    assert _program(pc).par(pc._nm.size(1))["dense"]
    pc.validate_tables()


@pytest.mark.parametrize("kind,latents", [("hclt", 32), ("pd", 64), ("rat", 8), ("hmm", 64), ("hmm", 256), ("hmm", 1024),
                                          ("hclt", 256)])
def test_equals_the_per_layer_kernels(kind, latents):
    pc = pj.compile(_circuit(kind, latents)).to(DEV)
    cats = min(l.max_cats for l in pc.input_layer_group)
    x = torch.randint(0, cats, (72, pc.num_vars), generator=torch.Generator().manual_seed(5)).to(DEV)
    out = {}
    for on in (False, True):
        pc.use_column_program = on
        pc.init_param_flows(flows_memory=0.0)
        lls = pc(x)
        pc.backward(x)
        out[on] = (lls, pc.node_flows[pc.num_dummy_nodes:].exp().clone(), pc.param_flows.clone())
    assert (out[True][0] - out[False][0]).abs().max().item() <= 1e-3
    for a, b in zip(out[True][1:], out[False][1:]):
        assert (a - b).norm() <= 1e-4 * b.norm()


@pytest.mark.parametrize("latents,depth", [(32, 2), (8, 1), (16, 2)])
@pytest.mark.parametrize("B", [3, 40])
def test_products_of_many_children_ahead_of_a_fused_level(latents, depth, B, monkeypatch):
    """Stored elements from the product kernel in the middle of the fused levels: odd numbers of children, ragged batches."""
    monkeypatch.setattr(ColumnProgram, "PROD_READS", 0)
    pc = pj.compile(pj.structures.RAT_SPN(num_vars=45, num_latents=latents, depth=depth, num_repetitions=3, num_cats=6)).to(DEV)
    x = torch.randint(0, 6, (B, pc.num_vars), generator=torch.Generator().manual_seed(B))
    check_against_oracle(pc, x, step=0.2, pseudo=0.1)
    assert any(isinstance(launch, list) for launch in pc._column_plan()[0]["launches"])


@pytest.mark.parametrize("cats", [511, 512, 1100, 5000])
@pytest.mark.parametrize("homogeneous", [True, False])
@pytest.mark.parametrize("B", [5, 530])
def test_leaves_of_mid_size_vocabularies(cats, homogeneous, B):
    """Staged tables of several and of few long rows, and tied tables on both sides of the transposed shadow's line."""
    torch.manual_seed(5)
    pc = pj.compile(pj.structures.HMM(seq_length=3, num_latents=32, num_emits=cats, homogeneous=homogeneous)).to(DEV)
    x = torch.randint(0, cats, (B, 3), generator=torch.Generator().manual_seed(B))
    check_against_oracle(pc, x, step=0.2, pseudo=0.1)
    layer = pc.input_layer_group[0]
    assert layer._shadow_ok(pc._nm.size(1)) == (homogeneous and cats >= 512 and pc._nm.size(1) <= cats)


@pytest.mark.parametrize("tokens", [512, 513, 600])
def test_more_levels_than_one_launch_takes(tokens):
    """(Two categories: the log-likelihood of 600 tokens stays near 400, one fp32 rounding there is 3e-5.)"""
    torch.manual_seed(5)
    pc = pj.compile(pj.structures.HMM(seq_length=tokens, num_latents=128, num_emits=2, homogeneous=True)).to(DEV)
    x = torch.randint(0, 2, (5, tokens), generator=torch.Generator().manual_seed(1))
    check_against_oracle(pc, x, step=0.2, pseudo=0.1)
    plan = pc._column_plan()
    assert plan is not None and pc._column_program.big_steps > 0
    assert len(plan[0]["launches"]) == (1 if tokens <= 512 else 2) and sum(n for _, n, _ in plan[0]["launches"]) == tokens
