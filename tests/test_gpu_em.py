"""Update kernels against the update in float64, at the edges of their rounds and tiles: fan-ins and category counts on both
sides of what a thread keeps in registers, few blocks (narrow tiles of nodes) and many, narrow and wide tiles of categories."""
import pytest
import torch

from pyjuice_b200 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _update(old, flows, dim, step, pseudo, keep_zero):
    """The update of float64 tables whose normalised dimension is `dim`."""
    n = old.size(dim)
    dead = (old < 1e-12) if keep_zero else torch.zeros_like(old, dtype=torch.bool)
    total = torch.where(dead, 0.0, flows + pseudo / n).sum(dim, keepdim=True) if keep_zero else flows.sum(dim, keepdim=True) + pseudo
    return torch.where(dead, 0.0, (1 - step) * old + step * (flows + pseudo / n) / total)


def _bound(want, n):
    return 2.0 ** -24 * (n + 12) * want.abs() + 1e-12      # n additions of positive terms and a dozen roundings


@pytest.mark.parametrize("keep_zero", [0, 1])
@pytest.mark.parametrize("blocks,bs", [(1, 512), (3, 40), (300, 32), (297, 48), (5, 8), (400, 12), (7, 1), (2, 4)])
@pytest.mark.parametrize("fan", [1, 63, 65, 256, 257, 2100])
def test_sum_parameters(blocks, bs, fan, keep_zero):
    if blocks * bs * fan > 1 << 23:
        fan = 130
    g = torch.Generator(device=DEV).manual_seed(fan)
    old = torch.rand(blocks, fan, bs, device=DEV, generator=g)
    old[:, ::7] = 0.0
    old = (old + (0.0 if keep_zero else 1e-3)).contiguous()
    flows = torch.rand(blocks, fan, bs, device=DEV, generator=g) * 10 + (1e-3 if keep_zero else 0.0)
    at = torch.arange(blocks, device=DEV) * fan * bs
    full = lambda v: torch.full((blocks,), v, dtype=torch.int32, device=DEV)
    new = old.clone()
    _lib.call("pcx_em_sum", new, flows, at, at, full(fan), full(bs), blocks, bs, 0.3, 0.1, keep_zero)
    want = _update(old.double(), flows.double(), 1, 0.3, 0.1, keep_zero)
    assert bool(((new.double() - want).abs() <= _bound(want, fan)).all())


@pytest.mark.parametrize("keep_zero", [0, 1])
@pytest.mark.parametrize("cats", [2, 31, 256, 257, 1024, 1025, 2100])
@pytest.mark.parametrize("nodes", [1, 9])
def test_leaf_parameters(nodes, cats, keep_zero):
    g = torch.Generator(device=DEV).manual_seed(cats)
    old = torch.rand(nodes, cats, device=DEV, generator=g)
    old[:, 1::5] = 0.0
    flows = torch.rand(nodes, cats, device=DEV, generator=g)
    new, ids = old.clone(), torch.arange(nodes, dtype=torch.int32, device=DEV)
    at, n = (ids * cats).int(), torch.full((nodes,), cats, dtype=torch.int32, device=DEV)
    _lib.call("pcx_em_input_cat", new, flows, ids, at, at, n, nodes, cats, 0.3, 0.1, keep_zero)
    want = _update(old.double(), flows.double(), 1, 0.3, 0.1, keep_zero)
    assert bool(((new.double() - want).abs() <= _bound(want, cats)).all())


@pytest.mark.parametrize("rows,cats", [(1, 33), (130, 1000), (512, 1000), (512, 4700), (300, 6500)])
def test_leaf_parameters_from_the_transposed_flows(rows, cats):
    g = torch.Generator(device=DEV).manual_seed(rows)
    old = torch.rand(rows, cats, device=DEV, generator=g) + 1e-3
    flows = torch.rand(cats, rows, device=DEV, generator=g)
    new, logp = old.clone(), torch.empty(cats, rows, device=DEV)
    _lib.call("pcx_em_input_cat_t", new, logp, flows, torch.empty(16 * rows, device=DEV), rows, cats, 0.3, 0.1)
    want = _update(old.double(), flows.double().t(), 1, 0.3, 0.1, False)
    assert bool(((new.double() - want).abs() <= _bound(want, cats)).all())
    assert bool(((logp.t().double() - new.double().log()).abs() <= 2.0 ** -22 * (1 + new.double().log().abs())).all())
