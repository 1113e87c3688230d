"""The column program's planner on the host: its tables, walked task by task in float64, give the values, flows and parameter
flows of the CPU oracle, whatever the structure, the node-block size and the row width, for every launch shape it can choose."""
import random

import numpy as np
import pytest
import torch

import pyjuice_b200 as pj
from oracle import pc_oracle as orc
from pyjuice_b200.column import K_CTA, K_MMA, K_PROD, PAR, TASK, ColumnProgram, Unsupported

B = 3


def _circuit(kind, latents):
    torch.manual_seed(3)
    random.seed(3)
    S = pj.structures
    if kind == "hclt":
        tree = S.random_grid_spanning_tree(4, 4, np.random.default_rng(3))
        ns = S.tree_to_hidden_circuit(tree, tree.center(), num_latents=latents, num_cats=3)
    elif kind == "pd":
        ns = S.PD((9, 7), latents, split_points=[[3, 6], [3]], num_cats=3)
    elif kind == "pd-sparse":                              # block-sparse sums, products without parents
        ns = S.PD((8, 8), latents, split_intervals=(2, 2), max_prod_block_conns=2, num_cats=3)
    elif kind == "rat":
        ns = S.RAT_SPN(num_vars=20, num_latents=latents, depth=2, num_repetitions=5, num_cats=3)
    else:
        ns = S.HMM(seq_length=5, num_latents=latents, num_emits=4, homogeneous=True)
    return pj.compile(ns, verbose=False)


def _lse(x, axis):
    m = x.max(axis=axis, keepdims=True)
    m = np.where(np.isinf(m), 0.0, m)
    with np.errstate(divide="ignore"):
        return np.log(np.exp(x - m).sum(axis=axis)) + m.squeeze(axis)


class _Walk:
    """Runs a plan on the host."""

    def __init__(self, pc, program, plan, nm):
        self.pc, self.plan, self.nm = pc, plan, nm
        self.kids, self.bases = plan["kids"].numpy(), plan["bases"].numpy().reshape(-1, 4)
        self.params = pc.params.data.double().numpy()
        self.em = np.full((max(program.em_rows, 1), nm.shape[1]), np.nan)
        self.nf = np.full_like(nm, np.nan)
        self.ef = np.full((pc.num_elements, nm.shape[1]), np.nan)

    def levels(self, mode):
        p = self.plan[mode]
        tasks, self.strips = p["tasks"].numpy().view(TASK), p["strips"].numpy().reshape(-1, 4)
        for launch in p["launches"]:
            if isinstance(launch, list):
                for rows, cids, size in launch:
                    for r, ks in zip(rows.tolist(), cids.tolist()):
                        self.em[r:r + size] = sum(self.nm[k:k + size] for k in ks if k)
                continue
            levels, n, shape = launch
            assert levels.shape == (n, 4) and shape[0] in (1, 2, 4) and (shape[3] == 0 or n == 1)
            for t0, m, s0, k in levels.tolist():
                for t in tasks[t0:t0 + m].tolist() + tasks[s0:s0 + k].tolist():
                    yield dict(zip(TASK.names, t))

    def operand(self, t, mode):
        """Log-operand [depth, B] of a task (stored element values are written) and the entries' first words."""
        mma = t["kind"] in (K_MMA, K_CTA)
        span = 16 if mma else 1 << t["lg_entry"]
        n = t["n_k"] if mma else t["n_k"] >> t["lg_entry"]
        ent = self.kids[t["kid_off"]:t["kid_off"] + n * t["width"]].reshape(n, t["width"])
        first, ent = (None, ent) if mma else (ent[:, 0], ent[:, 1:])
        rows = lambda c: (ent[:, c, None] + np.arange(span)[None, :]).reshape(-1)
        if mode == 1:
            return self.nf[rows(0)] - self.nm[rows(0)], first
        if t["n_kids"] < 0:
            return self.em[rows(0)], first
        v = sum(self.nm[rows(c)] for c in range(t["n_kids"]))       # (an absent child is a dummy row: zeros)
        if ent.shape[1] > t["n_kids"]:
            self.em[rows(t["n_kids"])] = v
        return v, first

    def outputs(self, t, mode):
        """Per output strip: its record, rows, and parameters [rows, depth]."""
        if t["kind"] in (K_MMA, K_CTA):
            f = self.bases[t["par_off"]:t["par_off"] + t["n_k"] * t["n_rows"]].reshape(t["n_k"], t["n_rows"], 4)
            for s in range(t["n_rows"]):
                at = [b + np.arange(16)[:, None] * sr + np.arange(16)[None, :] * sk for b, sr, sk, _ in f[:, s].tolist()]
                yield self.strips[t["strip_off"] + s], 16, self.params[np.concatenate(at, axis=1)]
            return
        span = 1 << t["lg_entry"]
        k = (self.first[:, None] + np.arange(span)[None, :] * t["sk"]).reshape(-1)
        yield self.strips[t["strip_off"]], t["n_rows"], self.params[k[None, :] + np.arange(t["n_rows"])[:, None] * t["sr"]]

    def forward(self):
        for t in self.levels(0):
            v, self.first = self.operand(t, 0)
            for st, n, theta in self.outputs(t, 0):
                with np.errstate(divide="ignore"):
                    self.nm[st[0]:st[0] + n] = _lse(np.log(theta)[:, :, None] + v[None], 1)

    def backward(self):
        for t in self.levels(1):
            if t["kind"] == K_PROD:
                row, n = t["strip_off"], t["n_rows"]
                parts = [self.ef[p:p + n] for p in self.kids[t["kid_off"]:t["kid_off"] + t["n_k"]].tolist()]
                parts += [self.nf[row:row + n]] if t["sk"] else []
                self.nf[row:row + n] = _lse(np.stack(parts), 0) if parts else -np.inf
                continue
            v, self.first = self.operand(t, 1)
            for st, n, theta in self.outputs(t, 1):
                e, x, y, flag = st.tolist()
                if flag < 0:
                    value, kids = self.em[x:x + n], []
                else:
                    kids = [k for k in (x, y) if k] if flag < 2 else self.kids[x:x + y].tolist()
                    value = sum(self.nm[k:k + n] for k in kids)
                with np.errstate(divide="ignore"):
                    flow = _lse(np.log(theta)[:, :, None] + v[None], 1) + value
                for dst, at in [(self.nf, k) for k in kids] if flag in (1, 3) else [(self.ef, e)]:
                    dst[at:at + n] = flow

    def par_flows(self, par):
        out = np.zeros(self.pc.num_param_flows)
        kids, pp = par["kids"].numpy(), par["pp"].numpy().reshape(-1, 2)
        for kind, (jobs, n) in par["jobs"].items():
            for t in jobs.numpy().view(PAR).tolist():
                t = dict(zip(PAR.names, t))
                mma = kind != 1
                span = 16 if mma else 1 << t["lg_entry"]
                n_ent = t["n_k"] if mma else t["n_k"] >> t["lg_entry"]
                n_rows, row = (16, [t[f"row{i}"] for i in range(4)]) if mma else (t["n_strips"], [t["row0"]])
                ent = kids[t["kid_off"]:t["kid_off"] + n_ent * t["width"]].reshape(n_ent, t["width"])
                strips = t["n_strips"] if mma else 1
                for i in range(n_ent):
                    rows = [r + np.arange(span) for r in ent[i].tolist()]
                    y = self.em[rows[0]] if t["n_kids"] < 0 else sum(self.nm[r] for r in rows)
                    for s in range(strips):
                        a, f = pp[t["pp_off"] + i * strips + s]
                        r = row[s] + np.arange(n_rows)
                        x = np.exp((self.nf[r] - self.nm[r])[:, None] + y[None]).sum(axis=2)
                        o = np.arange(n_rows)[:, None] + np.arange(span)[None, :] * t["bs"]
                        np.add.at(out, f + o, self.params[a + o] * x)
        for g in par["dense"]:
            for m in range(g["n"]):
                y = self.nm[g["fk"][m].numpy()].sum(axis=1)
                for b, row in enumerate(g["nids"][m].tolist()):
                    r, o = row + np.arange(g["bs"]), np.arange(g["bs"])[:, None]
                    x = np.exp((self.nf[r] - self.nm[r])[:, None] + y[None]).sum(axis=2)
                    np.add.at(out, g["pfids"][b].numpy()[None, :] + o, self.params[g["pids"][b].numpy()[None, :] + o] * x)
        return out


def _check(pc, W):
    program = ColumnProgram(pc)
    x = torch.randint(0, 3, (B, pc.num_vars), generator=torch.Generator().manual_seed(1))
    leaf = [layer.params.data for layer in pc.input_layer_group]
    lls, st = orc.forward(pc, x, pc.params.data, leaf)
    orc.backward(pc, x, pc.params.data, leaf, st)
    nm = st.node_mars.numpy().copy()
    for group in pc.inner_layer_groups:
        if group.is_sum():
            for layer in group:
                nm[layer._layer_nid_range[0]:layer._layer_nid_range[1]] = np.nan
    plan = program.plan(W)
    walk = _Walk(pc, program, plan, nm)
    walk.forward()
    r0, r1 = pc._root_node_range
    # float64 against float64: what differs is the order of sums of some hundred terms
    close = lambda a, b: np.testing.assert_allclose(a, b, rtol=1e-9, atol=1e-9)
    close(walk.nm[r0:r1].T, lls.numpy())
    walk.nf[r0:r1] = 0.0
    walk.backward()
    d = pc.num_dummy_nodes
    close(np.exp(walk.nf[d:]), st.node_flows.exp().numpy()[d:])
    close(walk.par_flows(program.par(W)), st.param_flows.numpy())
    counts = []
    program.check(plan, W, pc, lambda what, at, extent, limit: counts.append(at >= 0 and at + extent <= limit))
    assert counts and all(counts)
    return program, plan


@pytest.mark.parametrize("W", [8, 40, 264])
@pytest.mark.parametrize("kind,latents", [("hclt", 4), ("hclt", 24), ("hclt", 64), ("hclt", 128), ("pd", 16), ("pd", 32),
                                          ("pd-sparse", 16), ("rat", 8), ("rat", 32), ("hmm", 8), ("hmm", 96), ("hmm", 256)])
def test_walk_gives_the_values_of_the_oracle(kind, latents, W):
    _check(_circuit(kind, latents), W)


@pytest.mark.parametrize("kind,latents", [("hclt", 64), ("pd", 32), ("rat", 32), ("rat", 8)])
@pytest.mark.parametrize("attr,value", [("WIDE_ITEMS", 1), ("PROD_READS", 0)])
def test_walk_with_launches_of_single_levels(kind, latents, attr, value, monkeypatch):
    monkeypatch.setattr(ColumnProgram, attr, value)
    _, plan = _check(_circuit(kind, latents), 40)
    shapes = {launch[2][3] for m in (0, 1) for launch in plan[m]["launches"] if not isinstance(launch, list)}
    if attr == "WIDE_ITEMS":
        assert 0 not in shapes
    elif kind == "rat":                                    # leaf products of many children
        assert any(isinstance(launch, list) for launch in plan[0]["launches"])


@pytest.mark.parametrize("work", [0, 1 << 60])
def test_walk_with_tied_tables_in_one_product(work, monkeypatch):
    monkeypatch.setattr(ColumnProgram, "DENSE_PAR_WORK", work)
    program, _ = _check(_circuit("hmm", 256), 8)
    assert bool(program.par(8)["dense"]) == (work == 0)


@pytest.mark.parametrize("latents", [4, 128])
def test_walk_of_more_levels_than_one_launch_takes(latents):
    torch.manual_seed(3)
    ns = pj.structures.HMM(seq_length=600, num_latents=latents, num_emits=3, homogeneous=True)
    _, plan = _check(pj.compile(ns, verbose=False), 8)
    assert all(n <= 512 for m in (0, 1) for _, n, _ in plan[m]["launches"]) and len(plan[0]["launches"]) == 2


def test_deep_tables_are_refused():
    S = pj.structures
    with pytest.raises(Unsupported):
        ColumnProgram(pj.compile(S.HMM(seq_length=3, num_latents=2048, num_emits=4, homogeneous=True), verbose=False))


def test_description_is_checked():
    """A description that points outside its tables raises on the host."""
    import ctypes
    from pyjuice_b200 import column
    desc, tables = column._describe(_circuit("hclt", 4))
    handle = ctypes.c_void_p()
    make = lambda d, n: column._native("pcx_colplan_new", column._pointer(d), d.size, column._pointer(tables), n, ctypes.byref(handle))
    with pytest.raises(pj._lib.PcxError, match="outside"):
        make(desc, tables.size - 1)
    with pytest.raises(pj._lib.PcxError, match="too short"):
        make(desc[:-1].copy(), tables.size)
    assert not handle.value


@pytest.mark.parametrize("kind,latents,chains", [("hclt", 4, 0), ("hmm", 96, 1)])
def test_a_device_is_asked_once(kind, latents, chains, monkeypatch):
    """What a device holds at a time is asked for by the first circuit, not by every one, and about chains only where there is one."""
    from contextlib import nullcontext
    from types import SimpleNamespace
    from pyjuice_b200 import _lib, column
    programs = [ColumnProgram(_circuit(kind, latents)) for _ in range(2)]
    asked, lib = [], _lib.load()

    class Device:
        def __getattr__(self, name):
            if not name.endswith("_clusters"):
                return getattr(lib, name)
            return lambda c, *args: asked.append((name, c, *args)) or 1
    monkeypatch.setattr(column, "_ROOMS", {}, raising=False)
    monkeypatch.setattr(_lib, "load", Device)
    monkeypatch.setattr(torch.cuda, "device", lambda d: nullcontext())
    for program in programs:
        program.device = SimpleNamespace(type="cuda", index=3)
        program._room()
    assert len(asked) == len(set(asked)) == 5 + 16 * chains
