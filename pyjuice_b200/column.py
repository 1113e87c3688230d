"""Host side of the column program (``csrc/pcx_column.cu``): the task lists of a circuit of small node blocks.

``ColumnProgram`` is made once per circuit, and ``ColumnProgram.plan(W)`` cuts the circuit into tasks for a row width of
``W`` samples; both walk the index tables natively (``csrc/pcx_column_plan.cpp``), because both happen inside a first pass.
"""
from __future__ import annotations

import ctypes
import weakref

import numpy as np
import torch

from . import _lib

K_MMA, K_SIMT, K_SPLIT, K_PROD, K_CTA = 0, 1, 2, 3, 4
WARPS = 16                   # per CTA of the column kernel
TASK = np.dtype([(n, "<i4") for n in ("kid_off", "n_k", "n_kids", "width", "strip_off", "n_rows", "par_off", "kind", "sk",
                                      "sr", "lg_entry", "pad")])
PAR = np.dtype([(n, "<i4") for n in ("row0", "row1", "n_strips", "kid_off", "n_k", "n_kids", "width", "pp_off", "bs",
                                     "lg_entry", "row2", "row3")])


class Unsupported(Exception):
    """The circuit has a table the column program does not cover; the per-layer kernels run instead."""


def _native(name, *args):
    """Calls a function of the planner that may refuse."""
    why = ctypes.create_string_buffer(256)
    rc = getattr(_lib.load(), name)(*args, why, len(why))
    if rc == 1:
        raise Unsupported(why.value.decode())
    if rc != 0:
        raise _lib.PcxError(f"{name}: {why.value.decode()}")


class _Blob:
    """Tables made by the planner: ``meta`` describes them, ``take`` gives sections of their device copy (one transfer)."""

    def __init__(self, device, name, *args):
        handle = ctypes.c_void_p()
        _native(name, *args, ctypes.byref(handle))
        try:
            data, n, meta, m = ctypes.c_void_p(), ctypes.c_int64(), ctypes.c_void_p(), ctypes.c_int64()
            _lib.load().pcx_colplan_blob(handle, ctypes.byref(data), ctypes.byref(n), ctypes.byref(meta), ctypes.byref(m))
            self.meta = np.ctypeslib.as_array(ctypes.cast(meta, ctypes.POINTER(ctypes.c_int64)), (m.value,)).tolist() if m.value else []
            host = (np.ctypeslib.as_array(ctypes.cast(data, ctypes.POINTER(ctypes.c_int32)), (n.value,)) if n.value
                    else np.zeros(0, dtype=np.int32))
            # (a copy of its own, also on the host: the planner's memory goes with the handle)
            self.tables = torch.empty(max(n.value, 16), dtype=torch.int32, device=device)
            if n.value:
                self.tables[:n.value].copy_(torch.from_numpy(host))
        finally:
            _lib.load().pcx_colplan_blob_free(handle)
        self._at = 0

    def next(self, n: int = 1):
        got = self.meta[self._at:self._at + n]
        self._at += n
        return got[0] if n == 1 else got

    def take(self, at: int, *shape):
        return self.tables[at:at + int(np.prod(shape))].view(*shape)


def _describe(pc):
    """The circuit's index tables as one int32 array on the host and the description `pcx_colplan_new` reads."""
    parts, at = [], 0
    r0, r1 = pc._root_node_range
    groups = pc.inner_layer_groups
    desc = [pc.num_nodes, pc.num_elements, pc.num_dummy_nodes, r0, r1, len(groups) // 2]

    def add(tables, cbs=0):
        nonlocal at
        desc.extend((tables[1].size(0), tables[1].size(1), cbs))
        for t in tables:
            desc.append(at)
            at += t.numel()
            parts.append(t.reshape(-1).to(torch.int32))

    for gi in range(0, len(groups), 2):
        desc.append(int(gi in pc._parentless))
        desc.append(len(groups[gi]))
        for layer in groups[gi]:
            desc.extend((layer.block_size, layer.num_fw_partitions))
            for tables in (layer._dev["fw"] if layer._dev else zip(layer.partitioned_nids, layer.partitioned_cids)):
                add(tables)
            desc.append(layer.num_bk_partitions)
            for u, par in (layer._dev["bk"] if layer._dev else zip(layer.partitioned_u_cids, layer.partitioned_parids)):
                add((u, par if layer._dev else pc._without_parentless(gi, par)))
        desc.append(len(groups[gi + 1]))
        for layer in groups[gi + 1]:
            desc.extend((layer.block_size, layer.num_fw_partitions))
            for tables in (layer._dev["fw"] if layer._dev else zip(layer.partitioned_nids, layer.partitioned_cids,
                                                                  layer.partitioned_pids, layer.partitioned_pfids)):
                add(tables)
            desc.append(layer.num_bk_partitions)
            for tables, cbs in zip(layer._dev["bk"] if layer._dev else zip(layer.partitioned_chids, layer.partitioned_parids,
                                                                          layer.partitioned_parpids), layer.cs_block_sizes):
                add(tables, cbs)
    return np.asarray(desc, dtype=np.int64), torch.cat(parts).cpu().numpy()


def _refuse_deep_tables(pc):
    """Tables that the planner would refuse for their depth alone, told from a row count on the device: the tables of a
    circuit of large dense blocks (several hundred MB) then need not come to the host."""
    groups = pc.inner_layer_groups
    for gi in range(0, len(groups), 2):
        if min(layer.block_size for layer in groups[gi]) < 32:
            continue
        for layer in groups[gi + 1]:
            if layer.block_size >= 128:
                for cids in layer.partitioned_cids:
                    if cids.size(1) > 1024 and int((cids != 0).sum(dim=1).max()) >= 1040:
                        raise Unsupported("a dense table deeper than a CTA task gathers")


class _Chain:
    """A launch of ``n`` levels of one tied group of ``S`` strips (see `pcx_column_chain`), and its exchange buffer."""

    def __init__(self, rows, strips, n, S, W, nt, per):
        self.rows, self.strips, self.n, self.S, self.nt, self.per = rows, strips, n, S, nt, per
        self.work = torch.empty(_lib.load().pcx_column_chain_bytes(S, W, nt, per), dtype=torch.uint8, device=rows.device)


class _Staged:
    """Tables of `pcx_prod_staged`: products of one block size, their sources through shared memory."""

    def __init__(self, sources, items, lists, size):
        self.sources, self.items, self.lists, self.size = sources, items, lists, size

    def run(self, mode, out, src, logspace):
        _lib.call("pcx_prod_staged", mode, out, src, self.sources, self.items, self.lists, self.sources.numel(), self.items.size(0),
                  self.size, src.size(1), int(logspace))

    def check(self, report, mode, pc, em_rows):
        """Bounds of every index the kernel forms (see `ColumnProgram.check`)."""
        lists, n = self.lists.cpu().numpy().view(np.uint16).reshape(-1, 8), self.sources.numel()
        limits = (em_rows, pc.num_nodes) if mode == 0 else (pc.num_nodes, pc.num_elements)
        for row, at, k, _ in self.items.cpu().tolist():
            report("column product rows", row, self.size, limits[0])
            places = lists[at:at + -(-k // 8)].reshape(-1)
            assert 0 <= at and places.size >= k and (places[:k] < n).all() and (places[k:] == n).all()
        for r in self.sources.cpu().tolist():
            report("column product sources", r, self.size, limits[1])


def _pointer(a):
    return a.ctypes.data_as(ctypes.c_void_p)


# {(question, device, its other arguments): answers}: what a device holds at a time does not change, and one answer costs the driver
# some microseconds of a first pass
_ROOMS = {}


def _clusters(device, name, sizes, *args):
    """How many clusters of each of ``sizes`` CTAs of a kernel the device holds at a time."""
    found = [-1] * len(sizes)
    if device.type == "cuda":
        with torch.cuda.device(device):
            key = (name, torch.cuda.current_device() if device.index is None else device.index, *args)
            found = _ROOMS.get(key) or [int(getattr(_lib.load(), name)(c, *args)) for c in sizes]
            if min(found) > 0:
                _ROOMS[key] = found
    return [n if n > 0 else max(1, (128 if c < 16 else 112) // c) for c, n in zip(sizes, found)]


class ColumnProgram:
    PROD_READS = 3000            # child rows a CTA may gather for the stored elements of a fused level

    # A level with this many (16-row strip, 32-column) pieces gives every warp of the machine one: a launch of its own.
    WIDE_ITEMS = 148 * WARPS

    # Tied tables contract one product over all their layers' samples.  A 64 x 64 tile of a job of its own forms the
    # exponentials of its rows and of its elements again for every tile they belong to; the product of the dense layers forms
    # them once (`pcx_sum_par_dense2_stage`) and multiplies on the fifth-generation tensor cores, but takes two launches and
    # two more passes over the operands.  Rows x children x samples where the two meet, from HMMs of 128 to 1024 states
    # (microseconds, jobs / product): 256 states, 31 layers, 128 samples 64 / 59; 512, 7, 64: 47 / 51; 512, 63, 16: 82 / 52;
    # 1024, 31, 128: 329 / 116.  Tables of 128 rows fill half a product tile and never gain.
    DENSE_PAR_WORK = 200_000_000

    def __init__(self, pc):
        self.device = pc.device
        _refuse_deep_tables(pc)
        desc, tables = _describe(pc)
        self._planner = ctypes.c_void_p()
        _native("pcx_colplan_new", _pointer(desc), desc.size, _pointer(tables), tables.size, ctypes.byref(self._planner))
        weakref.finalize(self, _lib.load().pcx_colplan_free, self._planner)
        info = [ctypes.c_int() for _ in range(3)]
        _lib.load().pcx_colplan_info(self._planner, *map(ctypes.byref, info))
        self.em_rows, self.big_steps, self.n_chains = (v.value for v in info)
        self._by_width, self._par, self._tied, self._rooms = {}, {}, None, None

    # ---- cutting into tasks ------------------------------------------------------------------------------------------
    def _room(self):
        """Clusters of 1, 2, 4, 8 and 16 CTAs the device holds at a time, then clusters of 1 ... 16 CTAs of a chain where the
        circuit has one."""
        if self._rooms is None:
            rooms = _clusters(self.device, "pcx_column_clusters", (1, 2, 4, 8, 16), bool(self.big_steps))
            if self.n_chains:
                rooms += _clusters(self.device, "pcx_column_chain_clusters", range(1, 17))
            self._rooms = np.asarray(rooms, dtype=np.int32)
        return _pointer(self._rooms)

    def suits(self, W: int) -> bool:
        """Whether the program is the better choice at this row width (see the planner's `suits`)."""
        return bool(_lib.load().pcx_colplan_suits(self._planner, W, self._room()))

    def plan(self, W: int):
        found = self._by_width.get(W)
        if found is None:
            found = self._by_width[W] = self._cut(W)
        return found

    def choose(self, W: int):
        """The plan for rows of W samples, or None where the per-layer kernels are the better choice."""
        if W not in self._by_width:
            self._by_width[W] = self._cut(W) if self.suits(W) else None
        return self._by_width[W]

    def keep(self, widths):
        """Drops what belongs to other row widths."""
        self._by_width = {W: plan for W, plan in self._by_width.items() if W in widths}
        if self._tied is not None:
            picks = [self._pick(W) for W in widths if W is not None]
            self._par = {pick: par for pick, par in self._par.items() if pick in picks}

    def _cut(self, W: int):
        blob = _Blob(self.device, "pcx_colplan_cut", self._planner, W, self._room(), self.WIDE_ITEMS, self.PROD_READS)
        n_frag, at_bases, at_kids, n_kids = blob.next(4)
        out = dict(frags=torch.empty(max(n_frag, 1) * 1024, dtype=torch.uint8, device=self.device), n_frag=n_frag,
                   bases=blob.take(at_bases, 4 * n_frag), kids=blob.take(at_kids, n_kids))
        for mode in (0, 1):
            tasks, n_tasks, strips, n_strips, levels, n_levels = blob.next(6)
            out[mode] = dict(tasks=blob.take(tasks, 12 * n_tasks), strips=blob.take(strips, n_strips),
                             levels=blob.take(levels, n_levels, 4), launches=[], chained=[], staged={})
        for mode, form in ((0, "chained"), (0, "launches"), (1, "chained"), (1, "launches")):
            n_launches = blob.next()
            if n_launches < 0:                               # (no chain: the same list)
                out[mode]["launches"] = out[mode]["chained"]
                continue
            launches, staged = out[mode][form], out[mode]["staged"]
            for _ in range(n_launches):
                kind, *words = blob.next(7)
                if kind == 4:                                # the launch before this one, staged
                    sources, n_sources, items, n_items, n_chunks, size = words
                    at = launches[-1]
                    staged[form, len(launches) - 1, len(at) - 1 if isinstance(at, list) else 0] = _Staged(
                        blob.take(sources, n_sources), blob.take(items, n_items, 4), blob.take(items + 4 * n_items, n_chunks, 4), size)
                    continue
                if kind == 0:                                # (levels, how many, (column groups, tiles, CTAs, wide))
                    first, n, *how = words
                    launches.append((out[mode]["levels"][first:first + n], n, tuple(how)))
                    continue
                if kind == 3:
                    rows, strips, n, S, nt, per = words
                    launches.append(_Chain(blob.take(rows, n + 1, S, 2), blob.take(strips, S, 2), n, S, W, nt, per))
                    continue
                rows, cids, n, width, size, _ = words        # products ahead of the next level, one set per block size
                if kind == 1:
                    launches.append([])
                launches[-1].append((blob.take(rows, n), blob.take(cids, n, width), size))
        return out

    # ---- parameter flows ---------------------------------------------------------------------------------------------
    def par(self, W: int):
        """Tables of the parameter flows for rows of W samples, made when the first pass needs them: the groups of tied
        tables that go through one dense product, and the jobs of all others."""
        if self._tied is None:
            self._tied = self._tied_groups()
        pick = self._pick(W)
        if pick not in self._par:
            self._par[pick] = self._par_jobs(pick)
        return self._par[pick]

    def _pick(self, W: int):
        """Which groups of tied tables go through the dense product."""
        return tuple(g["n"] * W * g["n_blocks"] * g["bs"] * g["K"] >= self.DENSE_PAR_WORK for g in self._tied)

    def _tied_groups(self):
        blob = _Blob(self.device, "pcx_colplan_tied", self._planner)
        out = []
        for _ in range(len(blob.meta) // 10):
            n, fc, K, bs, n_blocks, fk, nids, cids, pids, pfids = blob.next(10)
            out.append(dict(n=n, fc=fc, K=K, bs=bs, n_blocks=n_blocks, fk=blob.take(fk, n, K, fc), nids=blob.take(nids, n, n_blocks),
                            cids=blob.take(cids, n_blocks, K), pids=blob.take(pids, n_blocks, K), pfids=blob.take(pfids, n_blocks, K)))
        return out

    def _par_jobs(self, pick):
        flags = np.asarray(pick + (False,), dtype=np.uint8)
        blob = _Blob(self.device, "pcx_colplan_jobs", self._planner, _pointer(flags))
        pp, n_pp, kids, n_kids = blob.next(4)
        jobs = {}
        for kind in range(4):
            at, n = blob.next(2)
            if n:
                jobs[kind] = (blob.take(at, 12 * n), n)
        return dict(pp=blob.take(pp, n_pp), kids=blob.take(kids, n_kids), jobs=jobs,
                    dense=[g for g, p in zip(self._tied, pick) if p])

    # ---- launches ----------------------------------------------------------------------------------------------------
    def buffers(self, W: int):
        """Stored element values ``[em_rows, W]``."""
        em = getattr(self, "_em_buf", None)
        if em is None or em.size(1) != W:
            self._em_buf = em = torch.empty(max(self.em_rows, 1), W, device=self.device)
        return em

    def run(self, plan, mode: int, nm, nf, ef, params, logspace: bool = True):
        p = plan[mode]
        W = nm.size(1)
        em, terms = self.buffers(W), 1 if _lib.sum_mode() == 2 else 3
        form = "chained" if logspace or p["launches"] is p["chained"] else "launches"    # (a chain keeps its flows as logarithms)
        for i, launch in enumerate(p[form]):
            if isinstance(launch, list):
                for q, (nids, cids, size) in enumerate(launch):
                    if (form, i, q) in p["staged"]:
                        p["staged"][form, i, q].run(mode, em, nm, logspace)
                        continue
                    _lib.call("pcx_prod_fwd", em, nm, nids, cids, nids.numel(), cids.size(1), size, W)
                continue
            if isinstance(launch, _Chain):
                c = launch
                _lib.call("pcx_column_chain", mode, nm, nf, plan["frags"], c.work, c.rows, c.strips, c.n, c.S, W, c.nt, c.per, terms)
                continue
            levels, n, (nt, tiles, cluster, wide) = launch
            if (form, i, 0) in p["staged"]:
                p["staged"][form, i, 0].run(mode, nf, ef, logspace)
                continue
            if self.big_steps:
                _lib.call("pcx_column_run_big", mode, nm, nf, ef, em, params, plan["frags"], p["tasks"], plan["kids"],
                          p["strips"], levels, n, W, nt, cluster, self.big_steps, int(logspace), terms)
                continue
            _lib.call("pcx_column_run", mode, nm, nf, ef, em, params, plan["frags"], p["tasks"], plan["kids"], p["strips"],
                      levels, n, W, nt, tiles, cluster, wide, int(logspace), terms)

    def _dense_operands(self, g, n: int, W: int):
        """Operand tiles of n layers of a group of tied tables, W samples each (zero beyond the last sample)."""
        chunks = -(-n * W // 64)
        if g.get("W") != W:
            g["W"], g["tiles"] = W, {}
        if n not in g["tiles"]:
            make = lambda k: torch.zeros(k, dtype=torch.uint8, device=self.device)
            g["tiles"][n] = (make(g["n_blocks"] * (g["bs"] // 128) * chunks * 32768), make(-(-g["K"] // 256) * chunks * 65536))
        return (*g["tiles"][n], chunks)

    def drop_operands(self):
        """Gives back the operand buffers of the dense products."""
        for g in self._tied or ():
            g.pop("W", None)
            g.pop("tiles", None)

    def param_flows(self, pf, nf, nm, params, max_bytes: int, logspace: bool = True, beside=None):
        """``max_bytes``: limit of a dense product's operands.  ``beside``: None: all parameter flows; True: those that go
        beside the others on a second stream, False: the others.
        The jobs of kinds 0 and 1 (roots, products of many children) are few and long and leave most of an SM free, which
        the staged tiles, persistent and bound by shared memory, cannot use: 62 of 560 us of a Poon-Domingos circuit over 784
        variables.  Without other jobs they are not split off: they then run beside the leaves' flows."""
        W = nm.size(1)
        par = self.par(W)
        split = bool(par["dense"]) or any(k > 1 for k in par["jobs"])
        kinds = [k for k in par["jobs"] if beside is None or (split and k <= 1) == beside]
        for g in par["dense"] if beside is not True else ():
            # (as many layers at a time as the operand buffers may take)
            layer = 4 * W * (g["n_blocks"] * g["bs"] + -(-g["K"] // 256) * 256)
            step = max(1, min(g["n"], max_bytes // layer))
            for m in range(0, g["n"], step):
                n = min(step, g["n"] - m)
                x, y, chunks = self._dense_operands(g, n, W)
                _lib.call("pcx_sum_par_dense2_stage", x, y, nf, nm, None, g["nids"][m], None, g["fk"][m], g["fc"],
                          g["n_blocks"], g["K"], g["bs"], W, chunks, 0, n, int(logspace))
                _lib.call("pcx_sum_par_dense2_gemm", pf, params, x, y, g["cids"], g["pids"], g["pfids"], g["n_blocks"], g["K"],
                          g["bs"], chunks)
        for kind in kinds:
            jobs, n = par["jobs"][kind]
            _lib.call("pcx_column_par", kind, pf, nf, nm, self.buffers(W), params, jobs, par["kids"], par["pp"], n, W,
                      int(logspace), 1 if _lib.sum_mode() == 2 else 3)

    def check(self, plan, W: int, pc, report):
        """Bounds of every index the kernels form from the plan's tables; ``report(what, index, extent, limit)``."""
        par = self.par(W)
        kids, pp = plan["kids"].cpu().numpy(), par["pp"].cpu().numpy().reshape(-1, 2)
        n_par, n_flow = int(pc.params.numel()), int(pc.num_param_flows)
        bases = plan["bases"].cpu().numpy().reshape(-1, 4)[:plan["n_frag"]]
        for b in bases:
            report("column fragments", int(b[0]), 15 * int(b[1]) + 15 * int(b[2]) + 1, n_par)
        for mode in (0, 1):
            p = plan[mode]
            strips = p["strips"].cpu().numpy().reshape(-1, 4)
            tasks = p["tasks"].cpu().numpy().view(TASK)
            seen = 0
            for t0, n, s0, ns in p["levels"].cpu().tolist():
                assert t0 == seen and s0 == t0 + n, "column levels do not follow one another"
                seen = s0 + ns
            assert seen == tasks.size
            for c in p["chained"]:
                if isinstance(c, _Chain):
                    for r in c.rows.cpu().reshape(-1).tolist():
                        report("column chain rows", int(r), 16, pc.num_nodes)
                    for first, step in c.strips.cpu().tolist():
                        assert 0 <= first and first + (c.S - 1) * step < plan["n_frag"]
            for staged in p["staged"].values():
                staged.check(report, mode, pc, self.em_rows)
            for t in tasks:
                k, w, off = int(t["n_k"]), int(t["width"]), int(t["kid_off"])
                if t["kind"] == K_PROD:
                    report("column flow rows", int(t["strip_off"]), int(t["n_rows"]), pc.num_nodes)
                    for r in kids[off:off + k]:
                        report("column parent rows", int(r), int(t["n_rows"]), pc.num_elements)
                    continue
                n_ent = k if t["kind"] in (K_MMA, K_CTA) else (k >> int(t["lg_entry"]))
                span = 16 if t["kind"] in (K_MMA, K_CTA) else (1 << int(t["lg_entry"]))
                assert off + n_ent * w <= kids.size
                ent = kids[off:off + n_ent * w].reshape(n_ent, w)
                if t["kind"] in (K_MMA, K_CTA):
                    assert int(t["par_off"]) + k * int(t["n_rows"]) <= plan["n_frag"]
                else:
                    ext = (span - 1) * int(t["sk"]) + (int(t["n_rows"]) - 1) * int(t["sr"]) + 1
                    for q in ent[:, 0]:
                        report("column parameters", int(q), ext, n_par)
                    ent = ent[:, 1:]
                nk = abs(int(t["n_kids"]))
                limit = self.em_rows if t["n_kids"] < 0 else pc.num_nodes
                for r in ent[:, :nk].reshape(-1):
                    report("column operand rows", int(r), span, limit)
                for r in ent[:, nk:].reshape(-1):
                    report("column stored rows", int(r), span, self.em_rows)
                n_st = int(t["n_rows"]) if t["kind"] in (K_MMA, K_CTA) else 1
                rows = 16 if t["kind"] in (K_MMA, K_CTA) else int(t["n_rows"])
                for st in strips[int(t["strip_off"]):int(t["strip_off"]) + n_st]:
                    if mode == 0:
                        report("column output rows", int(st[0]), rows, pc.num_nodes)
                        continue
                    report("column element rows", int(st[0]), rows, pc.num_elements)
                    if st[3] < 0:
                        report("column stored rows", int(st[1]), rows, self.em_rows)
                    elif st[3] < 2:
                        for r in st[1:3]:
                            report("column child rows", int(r), rows, pc.num_nodes)
                    else:
                        for r in kids[int(st[1]):int(st[1]) + int(st[2])]:
                            report("column child rows", int(r), rows, pc.num_nodes)
        for g in par["dense"]:
            for r in g["nids"].cpu().reshape(-1).tolist():
                report("column flow rows", int(r), g["bs"], pc.num_nodes)
            report("column child rows", int(g["fk"].max()), 1, pc.num_nodes)
            report("column parameters", int(g["pids"].max()), g["bs"], n_par)
            report("column parameter flows", int(g["pfids"].max()), g["bs"], n_flow)
        kids = par["kids"].cpu().numpy()
        for kind, (jobs, n) in par["jobs"].items():
            for t in jobs.cpu().numpy().view(PAR):
                mma = kind != 1
                span = 16 if mma else (1 << int(t["lg_entry"]))
                n_ent = int(t["n_k"]) if mma else int(t["n_k"]) >> int(t["lg_entry"])
                rows = 16 if mma else int(t["n_strips"])
                for r in (t["row0"], t["row1"], t["row2"], t["row3"]) if mma else (t["row0"],):
                    report("column flow-tile rows", int(r), rows, pc.num_nodes)
                w = int(t["width"])
                limit = self.em_rows if t["n_kids"] < 0 else pc.num_nodes
                for r in kids[int(t["kid_off"]):int(t["kid_off"]) + n_ent * w]:
                    report("column flow-tile operand rows", int(r), span, limit)
                n_at = n_ent * (int(t["n_strips"]) if mma else 1)
                assert int(t["pp_off"]) + n_at <= pp.shape[0]
                ext = (span - 1) * int(t["bs"]) + rows
                for a, b in pp[int(t["pp_off"]):int(t["pp_off"]) + n_at]:
                    report("column parameters", int(a), ext, n_par)
                    report("column flows", int(b), ext, n_flow)
