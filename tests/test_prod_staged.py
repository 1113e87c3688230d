"""Products through shared memory: the planner's tables name the same rows as those of the general kernels (host), and the
kernel gives the sums and log-sum-exps of its tables in float64, at the edges of its lists, column tiles and number range."""
import random

import numpy as np
import pytest
import torch

import pyjuice_b200 as pj
from pyjuice_b200.column import K_PROD, TASK, ColumnProgram, _Staged


def _rat(num_vars, latents, depth, repetitions):
    torch.manual_seed(3)
    random.seed(3)
    return pj.compile(pj.structures.RAT_SPN(num_vars=num_vars, num_latents=latents, depth=depth, num_repetitions=repetitions,
                                            num_cats=3), verbose=False)


def _readers(staged):
    """{output row: (source rows, add)} of the tables."""
    rows, lists = staged.sources.cpu().tolist(), staged.lists.cpu().numpy().view(np.uint16).reshape(-1)
    return {row: ([rows[p] for p in lists[8 * at:8 * at + k].tolist()], add) for row, at, k, add in staged.items.cpu().tolist()}


@pytest.mark.parametrize("num_vars,latents,depth,repetitions", [(20, 32, 2, 5), (61, 16, 3, 9)])
def test_tables_name_the_rows_of_the_general_kernels(num_vars, latents, depth, repetitions, monkeypatch):
    monkeypatch.setattr(ColumnProgram, "WIDE_ITEMS", 1)
    pc = _rat(num_vars, latents, depth, repetitions)
    program = ColumnProgram(pc)
    plan = program.plan(1024)
    program.check(plan, 1024, pc, lambda what, at, extent, limit: None if 0 <= at <= at + extent <= limit else pytest.fail(what))
    found = 0
    for (form, i, q), staged in plan[0]["staged"].items():
        rows, cids, size = plan[0][form][i][q]
        assert size == staged.size
        want = {r: ([k for k in ks if k], 0) for r, ks in zip(rows.tolist(), cids.tolist())}
        assert _readers(staged) == want
        found += 1
    tasks, kids = plan[1]["tasks"].numpy().view(TASK), plan["kids"].numpy()
    for (form, i, q), staged in plan[1]["staged"].items():
        levels, n, how = plan[1][form][i]
        assert n == 1 and how[3] == 3
        first, count, _, _ = levels[0].tolist()
        got = _readers(staged)
        seen = set()
        for t in tasks[first:first + count]:
            assert t["kind"] == K_PROD
            row = int(t["strip_off"])
            block = max(r for r in got if r <= row)
            seen.add(block)
            sources = [int(k) - (row - block) for k in kids[t["kid_off"]:t["kid_off"] + t["n_k"]]]
            assert row - block < staged.size and got[block] == (sources, int(t["sk"]))
        assert seen == set(got)
        found += 1
    assert found >= 2
    assert not program.plan(24)[0]["staged"]               # narrower than a column tile


def test_tables_are_made_once(monkeypatch):
    """Without a chain both kinds of flows have one list of launches, and every table is in the blob once."""
    monkeypatch.setattr(ColumnProgram, "WIDE_ITEMS", 1)
    plan = ColumnProgram(_rat(61, 16, 3, 9)).plan(1024)
    for mode in (0, 1):
        assert plan[mode]["launches"] is plan[mode]["chained"]
        held = list(plan[mode]["staged"].values())
        assert held and len({s.items.data_ptr() for s in held}) == len({i for _, i, _ in plan[mode]["staged"]}) == len(held)


def _tables(rng, size, n_sources, counts, device):
    sources, items, lists = rng.sample(range(n_sources + 7), n_sources), [], []
    for i, n in enumerate(counts):
        items.append([i * size, len(lists) // 8, n, rng.randrange(2)])
        lists += [rng.randrange(n_sources) for _ in range(n)] + [n_sources] * (-n % 8)
    as_int = lambda a: torch.tensor(a, dtype=torch.int32, device=device)
    words = torch.from_numpy(np.asarray(lists, dtype=np.uint16).view(np.int32).copy()).to(device)
    return _Staged(as_int([s * size for s in sources]), as_int(items), words.view(-1, 4), size), len(counts) * size


@pytest.mark.gpu
@pytest.mark.parametrize("mode,logspace", [(0, True), (1, True), (1, False)])
@pytest.mark.parametrize("W", [32, 40, 264])
@pytest.mark.parametrize("size,n_sources", [(1, 3), (8, 65), (32, 130), (2, 880), (300, 4)])
def test_kernel(mode, logspace, W, size, n_sources):
    rng = random.Random(W + size)
    staged, n_out = _tables(rng, size, n_sources, [0, 1, 2, 7, 8, 9, 17, 64] * 17, "cuda:0")
    g = torch.Generator(device="cuda:0").manual_seed(5)
    n_src = size * (n_sources + 7)
    if mode == 1 and logspace:                             # spans past the fp32 range of one column, rows of -inf, a column of -inf
        src = -torch.rand(n_src, W, device="cuda:0", generator=g) ** 2 * 400.0 - 3.0
        src[torch.rand(n_src, W, device="cuda:0", generator=g) < 0.1] = -float("inf")
        src[:, W // 2] = -float("inf")
    else:
        src = torch.randn(n_src, W, device="cuda:0", generator=g) * (1.0 if mode == 0 else 0.0) + torch.rand(n_src, W, device="cuda:0", generator=g)
    before = -torch.rand(n_out, W, device="cuda:0", generator=g) * 50.0 if logspace else torch.rand(n_out, W, device="cuda:0", generator=g)
    out = before.clone()
    staged.run(mode, out, src, logspace)
    torch.cuda.synchronize()
    x, was, got = src.double().cpu(), before.double().cpu(), out.double().cpu()
    for row, (sources, add) in _readers(staged).items():
        at = torch.tensor(sources, dtype=torch.long)[:, None] + torch.arange(size)
        terms = x[at]                                                        # [sources, size, W]
        old = was[row:row + size]
        if mode == 1 and logspace:
            if add:
                terms = torch.cat([terms, old[None]])
            want = torch.logsumexp(terms, 0) if len(terms) else torch.full((size, W), -float("inf"), dtype=torch.float64)
            # the result's rounding (2^-24 of it, twice); the sum, in steps of eight: each step scales it by one exponential,
            # each term is one (ex2.approx: 2^-22), and n additions round; the logarithm of at most 65: 4 * 2^-22
            n = len(sources)
            bound = 2.0 ** -23 * want.abs().clamp(max=500) + 2.0 ** -22 * (n / 8 + 2 + 4) + n * 2.0 ** -24
        else:
            want = terms.sum(0) + (old if mode == 1 and add else 0)
            bound = 2.0 ** -24 * (len(sources) + 8) * (terms.abs().sum(0) + 1)
        mine = got[row:row + size]
        assert torch.equal(torch.isinf(mine), torch.isinf(want))
        close = (mine - want).abs() <= bound
        assert bool((close | torch.isinf(want)).all()), float((mine - want)[~torch.isinf(want)].abs().max())


@pytest.mark.gpu
@pytest.mark.parametrize("mode,logspace", [(0, True), (1, True), (1, False)])
def test_nan_comes_through(mode, logspace):
    """A NaN source reaches every row that reads it (also the only one of a row, whose value is passed on as it is), and no other."""
    staged, n_out = _tables(random.Random(1), 4, 40, [0, 1, 1, 2, 9] * 13, "cuda:0")
    g = torch.Generator(device="cuda:0").manual_seed(5)
    src = -torch.rand(4 * 47, 40, device="cuda:0", generator=g) - 1.0
    src[torch.rand(4 * 47, 40, device="cuda:0", generator=g) < 0.2] = float("nan")
    out = -torch.rand(n_out, 40, device="cuda:0", generator=g)
    out[torch.rand(n_out, 40, device="cuda:0", generator=g) < 0.2] = float("nan")
    was = out.isnan().cpu()
    staged.run(mode, out, src, logspace)
    x = src.isnan().cpu()
    for row, (sources, add) in _readers(staged).items():
        want = was[row:row + 4].clone() if mode == 1 and add else torch.zeros(4, 40, dtype=torch.bool)
        for s in sources:
            want |= x[s:s + 4]
        assert torch.equal(out[row:row + 4].isnan().cpu(), want)


@pytest.mark.gpu
@pytest.mark.parametrize("W", [33, 256])
@pytest.mark.parametrize("logspace", [True, False])
def test_circuit_against_oracle(W, logspace, monkeypatch):
    from helpers import check_against_oracle
    monkeypatch.setattr(ColumnProgram, "WIDE_ITEMS", 1)
    pc = _rat(61, 64, 3, 9).to("cuda:0")
    x = torch.randint(0, 3, (W, 61), generator=torch.Generator().manual_seed(W))
    check_against_oracle(pc, x, step=0.2, pseudo=0.1, logspace_flows=logspace)
    plan = pc._column_plan()
    assert (bool(plan[0]["staged"]) and bool(plan[1]["staged"])) or W == 33
    pc.validate_tables()
