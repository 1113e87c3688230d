"""Chains of the column program (runs of tied levels in one launch): their tables, walked in float64 on the host, and the kernel
against the same levels by their tasks, at the sizes where its shapes meet: strips per CTA that do not divide the rows, one to
three column tiles per cluster, parameters beyond tensor memory, chains of odd and even length; then every shape of the kernel
against float64."""
import ctypes

import numpy as np
import pytest
import torch

import pyjuice_b200 as pj
from helpers import check_against_oracle, oracle_step
from pyjuice_b200.column import ColumnProgram, _Chain

DEV = "cuda:0"


def _hmm(latents, tokens, banded=False, homogeneous=True):
    torch.manual_seed(3)
    alpha = None
    if banded:                                             # most transitions are impossible
        i = torch.arange(latents)
        alpha = torch.rand(latents, latents) * ((i[:, None] - i[None, :]).abs() < 5)
        alpha = alpha / alpha.sum(dim=1, keepdim=True)
    return pj.compile(pj.structures.HMM(seq_length=tokens, num_latents=latents, num_emits=7, homogeneous=homogeneous, alpha=alpha),
                      verbose=False)


def _lse(x, axis):
    m = x.max(axis=axis, keepdims=True)
    m = np.where(np.isinf(m), 0.0, m)
    return np.log(np.exp(x - m).sum(axis=axis)) + m.squeeze(axis)


def _chains(plan, mode):
    return [c for c in plan[mode]["chained"] if isinstance(c, _Chain)]


def _value_first(latents, tokens):
    """The same chain, with the value of the level before as the first child of every product."""
    torch.manual_seed(3)
    with pj.set_block_size(32):
        leaf = lambda v: pj.inputs(v, num_nodes=latents, dist=pj.nodes.Categorical(num_cats=7))
        ns, tied = leaf(0), None
        for v in range(1, tokens):
            ns = pj.summate(ns, num_nodes=latents) if tied is None else tied.duplicate(ns, tie_params=True)
            tied = tied or ns
            ns = pj.multiply(ns, leaf(v))
        ns = pj.summate(ns, num_nodes=1, block_size=1)
    ns.init_parameters()
    return pj.compile(ns, verbose=False)


@pytest.mark.parametrize("latents,tokens,make", [(64, 5, _hmm), (96, 6, _hmm), (320, 4, _hmm), (96, 5, _value_first)])
def test_tables(latents, tokens, make):
    pc = make(latents, tokens)
    program = ColumnProgram(pc)
    plan = program.plan(16)
    bases, params = plan["bases"].numpy().reshape(-1, 4), pc.params.data.double().numpy()
    rng = np.random.default_rng(1)
    nm, nf = rng.normal(size=(pc.num_nodes, 2)), rng.normal(size=(pc.num_nodes, 2))
    nm[:pc.num_dummy_nodes] = 0.0
    want_nm, want_nf = nm.copy(), nf.copy()
    for mode, want in ((0, want_nm), (1, want_nf)):        # the same levels by their tasks
        from test_column_plan import _Walk
        walk = _Walk(pc, program, plan, want_nm)
        walk.nf = want_nf
        chain, = _chains(plan, mode)
        assert chain.n == tokens - 1 and chain.S == latents // 16
        tasks = list(walk.levels(mode))
        for t in (tasks[:-1] if mode == 0 else tasks[1:]):
            if t["n_rows"] == 1 and t["kind"] not in (0, 4):
                continue                                   # the root's level
            v, walk.first = walk.operand(t, mode)
            for st, n, theta in walk.outputs(t, mode):
                o = _lse(np.log(theta)[:, :, None] + v[None], 1)
                if mode == 0:
                    want_nm[st[0]:st[0] + n] = o
                else:
                    kids = [k for k in st[1:3].tolist() if k]
                    for k in kids:
                        want_nf[k:k + n] = o + sum(want_nm[j:j + n] for j in kids)
    for mode in (0, 1):
        chain, = _chains(plan, mode)
        rows, strips = chain.rows.numpy(), chain.strips.numpy()
        at = np.arange(16)
        of = lambda r: (r[:, None] + at).reshape(-1)
        theta = np.empty((16 * chain.S, 16 * chain.S))
        for s, (first, step) in enumerate(strips):
            for k in range(chain.S):
                b, sr, sk, _ = bases[first + k * step]
                theta[16 * s:16 * s + 16, 16 * k:16 * k + 16] = params[b + at[:, None] * sr + at[None, :] * sk]
        x, y = of(rows[0, :, 0]), of(np.where(rows[0, :, 1] > 0, rows[0, :, 1], 0))
        if mode == 0:
            v = nm[x] + np.where(np.repeat(rows[0, :, 1] > 0, 16)[:, None], nm[y], 0.0)
        else:
            v = want_nf[x] - want_nm[x]
        for l in range(chain.n):
            o = _lse(np.log(theta)[:, :, None] + v[None], 1)
            x, has = of(rows[l + 1, :, 0]), np.repeat(rows[l + 1, :, 1] > 0, 16)[:, None]
            y = of(rows[l + 1, :, 1])
            other = np.where(has, want_nm[y], 0.0)
            if mode == 0:
                np.testing.assert_allclose(o, want_nm[x], rtol=1e-12)
                v = o + other
            else:
                o = o + want_nm[x] + other
                np.testing.assert_allclose(o, want_nf[x], rtol=1e-9, atol=1e-9)
                assert not has.any() or np.allclose(o[has[:, 0]], want_nf[y][has[:, 0]])
                v = o - want_nm[x]


def test_what_is_no_chain():
    assert not _chains(ColumnProgram(_hmm(64, 3)).plan(8), 0)                       # two levels
    assert not _chains(ColumnProgram(_hmm(64, 6, homogeneous=False)).plan(8), 0)    # every level its own parameters
    assert not _chains(ColumnProgram(_hmm(32, 6)).plan(8), 0)                       # two strips


def _chain_below_wide_levels(length):
    """``length`` tied levels of 64 states under three levels of 1024 with parameters of their own."""
    torch.manual_seed(3)
    dist = pj.nodes.Categorical(num_cats=3)
    with pj.set_block_size(64):
        leaf = lambda v, n: pj.inputs(v, num_nodes=n, dist=dist)
        ns, tied = leaf(0, 64), None
        for v in range(1, length + 1):
            p = pj.multiply(ns, leaf(v, 64))
            ns = tied = pj.summate(p, num_nodes=64) if tied is None else tied.duplicate(p, tie_params=True)
        below = 64
        for v, n in enumerate((256, 1024, 1024, 1024), length + 1):
            ns, below = pj.summate(pj.multiply(ns, leaf(v, below)), num_nodes=n), n
        ns = pj.summate(pj.multiply(ns, leaf(length + 5, below)), num_nodes=1, block_size=1)
    ns.init_parameters()
    return pj.compile(ns, verbose=False)


def test_a_chain_elsewhere_does_not_excuse_large_levels():
    """Large levels outside a chain are judged as without one, however long the chain below them is."""
    alone, below = ColumnProgram(_chain_below_wide_levels(2)), ColumnProgram(_chain_below_wide_levels(9))
    assert alone.n_chains == 0 and below.n_chains == 1
    assert alone.suits(64) and below.suits(64)
    assert not alone.suits(1024) and not below.suits(1024)
    assert ColumnProgram(_hmm(256, 5)).suits(64)           # the large levels are the chain


@pytest.mark.gpu
@pytest.mark.parametrize("B", [1, 50, 130, 256])
@pytest.mark.parametrize("latents,tokens,banded", [(64, 4, False), (96, 5, False), (128, 9, True), (320, 6, False), (512, 7, False),
                                                   (768, 4, False), (1024, 5, False), (1024, 6, True)])
def test_against_the_tasks(latents, tokens, banded, B, monkeypatch):
    """Two bf16 parts per factor leave a relative error of about 3 * 2^-16 a level in either form, hence in a logarithm: 1e-4 for the
    two together; the float32 rounding of values near -20 is far below."""
    x = torch.randint(0, 7, (B, tokens), generator=torch.Generator().manual_seed(B)).to(DEV)
    got = []
    for tasks in (False, True):
        pc = _hmm(latents, tokens, banded).to(DEV)
        if tasks:
            cut = ColumnProgram._cut
            def without(self, W):
                plan = cut(self, W)
                for mode in (0, 1):
                    plan[mode]["chained"] = plan[mode]["launches"]
                return plan
            monkeypatch.setattr(ColumnProgram, "_cut", without)
        lls = pc(x)
        lls.mean().backward()
        plan = pc._column_plan()
        assert plan is not None and len(_chains(plan, 0)) == len(_chains(plan, 1))
        assert len(_chains(plan, 0)) == (0 if tasks or (latents == 1024 and B == 256) else 1)
        d = pc.num_dummy_nodes
        got.append((lls.detach(), pc.node_mars[d:].clone(), pc.node_flows[d:].exp(), pc.param_flows.clone()))
    for a, b in zip(got[0][:2], got[1][:2]):
        assert not torch.isnan(a).any() and (a - b).abs().nan_to_num().max() <= 1e-4 * tokens
        assert torch.equal(torch.isinf(a), torch.isinf(b))
    for a, b in zip(got[0][2:], got[1][2:]):
        assert (a - b).abs().max() <= 1e-4 * tokens * b.abs().max()
    assert pj._lib.get_status(DEV) == 0


# States, column tiles a cluster, strips a CTA: every kernel of the launcher (column tiles x strips a warp, see `_kernel`), each with
# warps that share a part of the contraction and that do not where both exist, and a last CTA of fewer strips.
SHAPES = ([(192, nt, per) for nt in (1, 2, 3) for per in (1, 2, 3)] + [(224, 3, 5), (224, 1, 6), (192, 2, 8), (224, 1, 8)]
          + [(320, nt, 2) for nt in (1, 2, 3)] + [(640, nt, 4) for nt in (1, 2, 3)] + [(640, 3, 3), (1024, 1, 8), (1024, 2, 4)])


def _kernel(states, nt, per):
    """(column tiles, strips a warp) of the kernel that the launcher takes for a chain."""
    strips = states // 16
    at_once = -(-per // (2 if per > 1 and -(-strips // per) <= 8 else 1))
    return nt, (1 if at_once == 1 else 2 if at_once == 2 else 4)


def test_the_shapes_are_all_there_are():
    assert {_kernel(*shape) for shape in SHAPES} == {(nt, ps) for nt in (1, 2, 3) for ps in (1, 2, 4)}


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("B", [5, 136, 520])
@pytest.mark.parametrize("states,nt,per", SHAPES)
def test_shapes_against_float64(states, nt, per, B, mode, monkeypatch):
    """Relative error of a level, hence absolute of a logarithm.  Two bf16 parts a factor (mode 1): 2^-18 for each factor's third
    part and 2^-18 for the product of the second parts, the exponential and the logarithm 2^-22 each, and the additions: three per
    16 children in the tensor core, 2^-23 each, some 2^-16 at 1024 states: 3 * 2^-16 with room for what they meet in.  One part
    (mode 2): 2^-9 for each factor.  A flow has gone up and down the chain; a parameter flow has one more product in it."""
    tokens, level = 6, (3 * 2.0 ** -16 if mode == 1 else 2.0 ** -8 + 3 * 2.0 ** -16)
    pc = _hmm(states, tokens).to(DEV)
    x = torch.randint(0, 7, (B, tokens), generator=torch.Generator().manual_seed(B))
    cut = ColumnProgram._cut

    def shaped(self, W):
        plan = cut(self, W)
        for m in (0, 1):
            assert len(_chains(plan, m)) == 1
            plan[m]["chained"] = [_Chain(c.rows, c.strips, c.n, c.S, W, nt, per) if isinstance(c, _Chain) else c
                                  for c in plan[m]["chained"]]
        return plan
    rooms = np.full(21, 1 << 20, dtype=np.int32)           # (clusters wait for one another's place, not for one another)
    monkeypatch.setattr(ColumnProgram, "_room", lambda self: rooms.ctypes.data_as(ctypes.c_void_p))
    monkeypatch.setattr(ColumnProgram, "_cut", shaped)
    ref, st, _ = oracle_step(pc, x)
    pc.sum_mode = mode
    pc.init_param_flows(flows_memory=0.0)
    lls = pc(x.to(DEV))
    pc.backward(x.to(DEV))
    assert pj._lib.get_status(DEV) == 0
    assert [(c.nt, c.per) for m in (0, 1) for c in _chains(pc._column_program.plan(pc._nm.size(1)), m)] == [(nt, per)] * 2
    d = pc.num_dummy_nodes
    rounding = lambda t: 2.0 ** -22 * t.abs()
    for got, want in ((lls, ref), (pc.node_mars[d:], st.node_mars[d:])):
        got = got.detach().double().cpu()
        assert bool(((got - want).abs() <= level * tokens + rounding(want)).all())
    flows, want = pc.node_flows[d:].double().cpu().exp(), st.node_flows[d:].exp()
    assert bool(((flows - want).abs() <= 2.1 * level * tokens * want + 1e-30).all())
    flows, want = pc.param_flows.double().cpu(), st.param_flows
    assert bool(((flows - want).abs() <= 2.1 * level * (tokens + 1) * want + 1e-30).all())


@pytest.mark.gpu
def test_linear_flows_go_by_the_tasks():
    pc = _hmm(128, 6).to(DEV)
    x = torch.randint(0, 7, (40, 6), generator=torch.Generator().manual_seed(1))
    check_against_oracle(pc, x, step=0.2, pseudo=0.1, logspace_flows=False)
