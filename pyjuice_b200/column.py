"""Host side of the column program (``csrc/pcx_column.cu``): the task lists of a circuit of small node blocks.

``ColumnProgram`` is compiled once per circuit from the layers' index tables: for every depth the row groups (rows that
share one list of children), the child rows of every folded product, the parameter fragments, and for the backward pass
which level first touches a flow row.  ``ColumnProgram.plan(W)`` cuts the groups into warp tasks for a row width of ``W``
samples and puts the tables on the device.
"""
from __future__ import annotations

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


class _Pool:
    """Append-only int32 table; equal pieces (tied parameters, shared children) are stored once."""

    def __init__(self, width: int = 1):
        self.width, self.parts, self.n, self.seen, self.rows = width, [], 0, {}, []

    def add(self, arr) -> int:
        arr = np.ascontiguousarray(arr, dtype=np.int32)
        key = arr.tobytes()
        at = self.seen.get(key)
        if at is None:
            at = self.seen[key] = self.n
            self.parts.append(arr.reshape(-1))
            self.n += arr.size // self.width
            if self.width == 4 and arr.ndim == 2:
                self.rows.extend(arr[:, 3].tolist())
        return at

    def flag(self, at: int, n: int) -> int:
        """Largest last word of n records."""
        return max(int(self.rows[i]) for i in range(at, at + n))

    def tensor(self, device) -> torch.Tensor:
        flat = np.concatenate(self.parts) if self.parts else np.zeros(4 * self.width, dtype=np.int32)
        return torch.from_numpy(flat).to(device)


class _Group:
    """Rows with one operand list.  ``blocks``: (first row, rows) of every node block; ``ops``: per operand block its first
    row(s) and size; ``par[b][o]``: parameter of (block b, operand block o), ``flow`` likewise (forward groups)."""
    __slots__ = ("blocks", "ops", "par", "flow", "bs", "mma", "direct", "big", "depth")


def _np(t):
    return t.detach().cpu().numpy().astype(np.int64)


def _prefix(row):
    n = int((row != 0).sum())
    if n and not (row[:n] != 0).all():
        raise Unsupported("padding inside a table row")
    return n


class ColumnProgram:
    MAX_KIDS_FOLDED = 4          # elements of more children (shared leaves) keep their value for the backward pass
    MAX_FOLD_READS = 16          # child-row reads per element that folding may cost
    BIG_STRIPS, BIG_STEPS, BIG_MAX_STEPS = 8, 8, 64      # a group for CTA tasks: rows and depth (in 16) it has at least

    def __init__(self, pc):
        self.device = pc.device
        self.num_dummy = pc.num_dummy_nodes
        self._by_width, self._choice, self._rooms, self._par = {}, {}, {}, {}
        groups = pc.inner_layer_groups
        self.depths = []
        parents = np.zeros(pc.num_nodes + 1, dtype=np.int32)
        for gi in range(0, len(groups), 2):
            for layer in groups[gi]:
                j = np.arange(layer.block_size)
                for cids in layer.partitioned_cids:
                    c = _np(cids)
                    c = c[c != 0]
                    np.add.at(parents, (c[:, None] + j[None, :]).reshape(-1), 1)
        self.em_rows = self.big_steps = 0
        for gi in range(0, len(groups), 2):
            self.depths.append(self._depth(pc, gi, parents))
        written = np.zeros(pc.num_nodes, dtype=bool)
        r0, r1 = pc._root_node_range
        written[r0:r1] = True
        written[:pc.num_dummy_nodes] = True
        for d in reversed(self.depths):                       # which level first writes a flow row
            if d["direct"]:
                for kids in d["elems"].values():
                    for k in kids[1]:
                        written[k:k + kids[0]] = True
                continue
            for p in d["prod_bk"]:
                seen = written[p["row"]:p["row"] + p["size"]]
                if seen.any() and not seen.all():
                    raise Unsupported("a flow block is written in pieces")
                p["add"] = int(bool(seen.any()))
                written[p["row"]:p["row"] + p["size"]] = True
        if not written.all():
            raise Unsupported("a node without parents")
        if self.big_steps and len(self.depths) * 2 > 512:
            raise Unsupported("more levels than the CTA-task kernel lists")
        self._build_pack()

    # ---- tables of one depth ---------------------------------------------------------------------------------------
    def _depth(self, pc, gi, parents):
        pgroup, sgroup = pc.inner_layer_groups[gi], pc.inner_layer_groups[gi + 1]
        elems, order = {}, []                                 # element block start -> (size, child rows)
        for layer in pgroup:
            for nids, cids in zip(layer.partitioned_nids, layer.partitioned_cids):
                nids, cids = _np(nids), _np(cids)
                for e, row in zip(nids.tolist(), cids.tolist()):
                    elems[e] = (layer.block_size, [c for c in row if c != 0])
                    order.append(e)
        fmax = max(len(k) for _, k in elems.values())
        rows = [r for size, ks in elems.values() for k in ks for r in (k, k + size - 1)]
        direct = gi not in pc._parentless and bool((parents[np.asarray(rows)] == 1).all())
        if direct:
            direct = all(bool((parents[k:k + size] == 1).all()) for size, ks in elems.values() for k in ks)
        fw, reads = [], 0
        for layer in sgroup:
            merged = {}
            for nids, cids, pids, pfids in zip(layer.partitioned_nids, layer.partitioned_cids, layer.partitioned_pids,
                                               layer.partitioned_pfids):
                nids, cids, pids, pfids = _np(nids), _np(cids), _np(pids), _np(pfids)
                for i in range(nids.size):
                    n = _prefix(cids[i])
                    starts, at = [], 0
                    while at < n:
                        e = int(cids[i, at])
                        if e not in elems:
                            raise Unsupported("a child list that does not start at an element block")
                        starts.append((at, e))
                        at += elems[e][0]
                    pos = np.asarray([s for s, _ in starts], dtype=np.int64)
                    ids = [e for _, e in starts]
                    want = np.concatenate([np.arange(e, e + elems[e][0]) for e in ids]) if ids else np.zeros(0)
                    if at != n or not np.array_equal(cids[i, :n], want):
                        raise Unsupported("a child list that is not made of element blocks")
                    for tab in (pids, pfids):
                        for p, e in starts:
                            if tab[i, p + elems[e][0] - 1] != tab[i, p] + (elems[e][0] - 1) * layer.block_size:
                                raise Unsupported("parameters of an element block are not contiguous")
                    merged.setdefault(tuple(ids), []).append((int(nids[i]), pids[i, pos], pfids[i, pos]))
            for ids, blocks in merged.items():
                if not ids:
                    raise Unsupported("a sum node without children")
                g = _Group()
                g.bs, g.ops = layer.block_size, list(ids)
                g.blocks = [b[0] for b in blocks]
                g.par = np.stack([b[1] for b in blocks])
                g.flow = np.stack([b[2] for b in blocks])
                ebs = min(elems[e][0] for e in ids)
                g.mma = layer.block_size >= 32 and ebs >= 32
                g.depth = sum(elems[e][0] for e in ids)
                self._classify(g)
                if not g.big:
                    reads = max(reads, len(blocks) * max(1, layer.block_size // 64 if g.mma else layer.block_size // 16))
                fw.append(g)
        if reads * fmax > self.MAX_FOLD_READS and reads > 1:
            raise Unsupported("products shared by too many rows to be folded")
        store = {}
        if fmax > self.MAX_KIDS_FOLDED and not direct:
            for e in order:
                store[e] = self.em_rows
                self.em_rows += elems[e][0]
        bk, seen = [], set()
        for layer in sgroup:
            merged = {}
            for chids, parids, parpids, cbs in zip(layer.partitioned_chids, layer.partitioned_parids,
                                                   layer.partitioned_parpids, layer.cs_block_sizes):
                chids, parids, parpids = _np(chids), _np(parids), _np(parpids)
                for i in range(chids.size):
                    c = int(chids[i])
                    n = _prefix(parids[i])
                    if c in seen or c not in elems or elems[c][0] != cbs or n == 0:
                        raise Unsupported("element block split over layers")
                    seen.add(c)
                    merged.setdefault((cbs, tuple(parids[i, :n].tolist())), []).append((c, parpids[i, :n]))
            for (cbs, pars), blocks in merged.items():
                g = _Group()
                g.bs, g.ops = cbs, list(pars)
                g.blocks = [b[0] for b in blocks]
                g.par = np.stack([b[1] for b in blocks])
                g.flow = None
                g.mma = cbs >= 32 and layer.block_size >= 32
                g.direct = layer.block_size              # (parent block size)
                g.depth = len(pars) * layer.block_size
                self._classify(g)
                bk.append(g)
        if direct and len(seen) != len(elems):
            raise Unsupported("a product without a sum parent")
        prod_bk = []
        if not direct:
            for layer in pgroup:
                tabs = layer._dev["bk"]
                for u, par in tabs:
                    u, par = _np(u), _np(par)
                    for i in range(u.size):
                        prod_bk.append(dict(row=int(u[i]), size=layer.block_size, par=par[i][par[i] != 0], add=0))
        return dict(elems=elems, fw=fw, bk=bk, direct=direct, store=store, prod_bk=prod_bk)

    def _classify(self, g):
        steps, strips = g.depth // 16, len(g.blocks) * g.bs // 16
        g.big = g.mma and strips >= self.BIG_STRIPS and steps >= self.BIG_STEPS
        if g.mma and strips >= self.BIG_STRIPS and steps > self.BIG_MAX_STEPS:
            raise Unsupported("a dense table deeper than a CTA task gathers")
        if g.big:
            self.big_steps = max(self.big_steps, steps)

    # ---- parameter fragments ---------------------------------------------------------------------------------------
    def _build_pack(self):
        """Fragment bases of every MMA group, [strip][step] as arrays; ``frag_of`` hands out positions per task."""
        for d in self.depths:
            for g in d["fw"]:
                if g.mma:
                    sizes = [d["elems"][e][0] for e in g.ops]
                    g.par = (self._bases(g, sizes, g.bs, 1, g.bs), g.par)
            for g in d["bk"]:
                if g.mma:
                    g.par = (self._bases(g, [g.direct] * len(g.ops), g.direct, g.direct, 1), g.par)

    @staticmethod
    def _bases(g, sizes, bs, sr, sk):
        """[strips, steps, 4]: parameter of (row 0, child 0) of every 16 x 16 fragment, row and child strides."""
        off = np.concatenate([np.arange(0, s, 16) for s in sizes])
        blk = np.repeat(np.arange(len(sizes)), [s // 16 for s in sizes])
        r0 = np.arange(0, g.bs, 16)
        base = g.par[:, None, blk] + (off * sk)[None, None, :] + (r0 * sr)[None, :, None]       # [blocks, strips, steps]
        out = np.zeros((base.shape[0] * base.shape[1], base.shape[2], 4), dtype=np.int32)
        out[..., 0] = base.reshape(-1, base.shape[2])
        out[..., 1], out[..., 2] = sr, sk
        return out

    # ---- cutting into tasks ------------------------------------------------------------------------------------------
    def _room(self, c: int) -> int:
        """Clusters of ``c`` CTAs the device holds at a time."""
        key = (c, bool(self.big_steps))
        if key not in self._rooms:
            n = -1
            if self.device.type == "cuda":
                with torch.cuda.device(self.device):
                    n = int(_lib.load().pcx_column_clusters(*key))
            self._rooms[key] = n if n > 0 else max(1, (128 if c < 16 else 112) // c)
        return self._rooms[key]

    PROD_READS = 3000            # child rows a CTA may gather for the stored elements of a fused level (see `_cut`)

    # A level with this many (16-row strip, 32-column) pieces gives every warp of the machine one: a launch of its own.
    WIDE_ITEMS = 148 * WARPS

    def geometry(self, W: int, items: float):
        """(8-column groups per warp, warp tiles per cluster, CTAs per cluster) of the fused levels, for rows of W samples
        and ``items`` 16-row strips per level.

        As many CTAs as the machine holds at a time, but no larger a cluster than a level has strips for its warps; among
        equals the widest column group, which reads longer pieces of a value row.  (A device with 148 SMs holds 74, 33
        and 15 clusters of 2, 4 and 8 CTAs.)"""
        if self.big_steps:
            return self._big_geometry(W)
        best = None
        for cols in (8, 16):
            n = -(-W // cols)
            c = 1
            while c < 8 and self._room(c * 2) >= n and items > WARPS * c:
                c *= 2
            if best is None or (cols <= W and n * c >= best[0]):
                best = (n * c, cols // 8, 1, c)
        return best[1:]

    def _piece(self, groups, nt: int, c: int):
        """(strips per task, time) of a level's large groups on a cluster of c CTAs: rounds of tasks times what a task
        takes in microseconds: a fixed latency, the gather and exponentials of its operand, its multiplications, and parameters
        that neither stay in shared memory nor arrive during the gather.  (Measured per level, mean of the two
        directions, CTAs x columns: 512 x 512 on 4 x 8 / 8 x 16 8.5 / 9.6 us; 1024 x 1024 on 8 x 8 / 16 x 16 / 8 x 16 / 4 x 8
        12.4 / 13.2 / 16.2 / 16.9: sixteen columns cost the element flows two more microseconds than eight.)"""
        big = [(g.depth // 16, len(g.blocks) * g.bs // 16) for g in groups if g.big]
        if not big:
            return 1, 0.0
        steps = max(s for s, _ in big)
        best = None
        for size in (16, 8, 4, 2, 1):
            n = sum(-(-strips // size) for _, strips in big)
            stream = max(0.0, size * steps - max(0, 150 - steps * nt // 2)) * 0.01
            cost = -(-n // c) * (1.2 + 1.8 * nt + 0.025 * steps * nt + 0.003 * size * steps * nt + stream)
            if best is None or cost < best[1] - 1e-9:
                best = (size, cost)
        return best

    def _big_cost(self, nt: int, c: int, n: int) -> float:
        """Estimated time of a pass: all levels with their barriers, times the waves of clusters."""
        level = 0.5 + 0.03 * c
        return sum(level + self._piece(d["fw"], nt, c)[1] for d in self.depths) * -(-n // max(1, self._room(c)))

    def suits(self, W: int) -> bool:
        """Whether the program is the better choice at this row width.  With large groups it is while a level's CTA tasks go
        around the cluster about once: it is then bound by the latency of a level, which is lower than that of the
        per-layer kernels and of the tiles that wait on counters.  With several rounds per level a CTA works through its tasks
        one latency after the other, where those keep two tiles per SM under way (784-variable tree, 128 latents, 512
        samples: 745 us forward against 556)."""
        if not self.big_steps:
            return True
        nt, _, c, _ = self.plan(W)["fused"]
        size = [self._piece(d["fw"], nt, c)[0] for d in self.depths]
        tasks = [sum(-(-(len(g.blocks) * g.bs // 16) // p) for g in d["fw"] if g.big) for d, p in zip(self.depths, size)]
        waves = -(-(-(-W // (8 * nt))) // max(1, self._room(c)))
        return waves == 1 and sum(-(-n // c) for n in tasks) <= 1.5 * sum(1 for n in tasks if n)

    def _big_geometry(self, W: int):
        best = None
        for nt in (1, 2):
            n = -(-W // (8 * nt))
            for c in (1, 2, 4, 8, 16):
                cost = self._big_cost(nt, c, n)
                if best is None or cost < best[0] - 1e-9:
                    best = (cost, nt, 1, c)
        return best[1:]

    def plan(self, W: int):
        found = self._by_width.get(W)
        if found is None:
            found = self._by_width[W] = self._cut(W)
        return found

    def choose(self, W: int):
        """The plan for rows of W samples, or None where the per-layer kernels are the better choice."""
        if W not in self._choice:
            self._choice[W] = self.suits(W)
        return self.plan(W) if self._choice[W] else None

    @staticmethod
    def _count(groups):
        return sum(len(g.blocks) * max(1, g.bs // 16) for g in groups)

    def _cut(self, W: int):
        kids, frag = _Pool(), _Pool(4)
        strips = {0: _Pool(4), 1: _Pool(4)}
        tasks = {0: [], 1: []}
        levels = {0: [], 1: []}
        wide_tiles = -(-W // 32)
        is_wide = lambda strips: not self.big_steps and W >= 32 and strips * wide_tiles >= self.WIDE_ITEMS
        counts = [self._count(d["fw"]) for d in self.depths]
        small = [n for n in counts if not is_wide(n)]
        nt, tiles, c = self.geometry(W, float(np.mean(small)) if small else 1.0)
        fused = (nt, tiles, c, 0)
        wide = (4, wide_tiles, 1, 1)

        def shape(n):
            """(launch geometry, warps per column tile) of a level with n strips."""
            if is_wide(n):
                return wide, self.WIDE_ITEMS // wide_tiles
            return fused, (WARPS // tiles) * c

        before = {}                                           # product launches ahead of a level
        for i, (d, n) in enumerate(zip(self.depths, counts)):
            first = len(tasks[0])
            how, workers = shape(n)
            split = []
            # Elements of many children in a level that has the machine to itself: their values come from the product
            # kernel, whose 2048 threads per SM hide the latency of the gather better than the warp tasks (16384 elements
            # of 24 children, 1024 samples: 155 + 25 us instead of 320).  A CTA of a fused level gathers some 500 child rows
            # in a microsecond: from several microseconds' worth of rows the kernel's launch is the smaller cost.
            reads = sum(d["elems"][e][0] * len(d["elems"][e][1]) for e in d["store"])
            stored = bool(d["store"]) and (is_wide(n) or reads > self.PROD_READS * c)
            if stored:
                before[i] = self._prod_tables(d)
            for g in d["fw"]:
                if g.big:
                    self._cta_tasks(d, g, 0, self._piece(d["fw"], nt, c)[0], kids, frag, strips[0], split)
                    continue
                self._fw_tasks(d, g, stored, self._strips_per_task(n, workers), kids, frag, strips[0], tasks[0], split)
            self._level(tasks[0], levels[0], strips[0], first, split, how)
        for d in reversed(self.depths):
            first = len(tasks[1])
            n = self._count(d["bk"])
            how, workers = shape(n)
            split = []
            for g in d["bk"]:
                if g.big:
                    self._cta_tasks(d, g, 1, self._piece(d["bk"], nt, c)[0], kids, frag, strips[1], split)
                    continue
                self._bk_tasks(d, g, self._strips_per_task(n, workers), kids, frag, strips[1], tasks[1])
            self._level(tasks[1], levels[1], strips[1], first, split, how)
            if d["direct"]:
                continue
            first = len(tasks[1])
            for p in d["prod_bk"]:
                for r in range(0, p["size"], 16):
                    off = kids.add(p["par"] + r) if p["par"].size else 0
                    tasks[1].append((off, p["par"].size, 0, 1, p["row"] + r, min(16, p["size"] - r), 0, K_PROD, p["add"], 0, 0, 0))
            self._level(tasks[1], levels[1], strips[1], first, [], shape(len(tasks[1]) - first)[0])
        dev = self.device
        out = dict(fused=fused, kids=None, frags=torch.empty(max(frag.n, 1) * 1024, dtype=torch.uint8, device=dev),
                   bases=frag.tensor(dev), n_frag=frag.n)
        for m in (0, 1):
            rec = np.array(tasks[m], dtype=TASK)
            tab = torch.tensor([lv for lv, _ in levels[m]], dtype=torch.int32, device=dev)
            launches, at = [], 0
            while at < len(levels[m]):                        # consecutive fused levels are one launch
                how, end = levels[m][at][1], at + 1
                while (how is fused and end < len(levels[m]) and levels[m][end][1] is fused
                       and not (m == 0 and end in before)):
                    end += 1
                if m == 0 and at in before:
                    launches.append(before[at])
                launches.append((tab[at:end], end - at, how))
                at = end
            out[m] = dict(tasks=torch.from_numpy(rec.view(np.uint8)).to(dev), strips=strips[m].tensor(dev), levels=tab,
                          launches=launches)
        out["kids"] = kids.tensor(dev)
        return out

    def par(self, W: int):
        """Tables of the parameter flows for rows of W samples, built when the first pass needs them: the groups of tied
        tables that go through one dense product, and the jobs of all others."""
        if "tied" not in self._par:
            self._par["tied"] = self._tied_groups()
        pick = tuple(g["n"] * W * g["n_blocks"] * g["bs"] * g["K"] >= self.DENSE_PAR_WORK for g in self._par["tied"])
        if pick not in self._par:
            self._par[pick] = self._par_jobs([g for g, p in zip(self._par["tied"], pick) if p])
        return self._par[pick]

    @staticmethod
    def _level(tasks, levels, strips, first, split, how):
        n = len(tasks) - first
        if how[3]:                                            # a wide level: which of the three kernels can take it
            new = tasks[first:]
            if not split and all(t[7] == K_PROD for t in new):
                how = how[:3] + (3,)
            elif not split and all(t[7] == K_MMA and t[1] * t[3] <= 32 and t[2] <= 2 and strips.flag(t[4], t[5]) < 2 for t in new):
                how = how[:3] + (2,)
        tasks.extend(split)
        levels.append(((first, n, first + n, len(split)), how))

    @staticmethod
    def _strips_per_task(total: int, workers: int) -> int:
        """Few strips in a level: one per task, so that every warp has one (its rows share an operand with its neighbours',
        which each of them gathers for itself).  Many: two share the gather."""
        return max(1, min(2, total // max(1, workers)))

    def _prod_tables(self, d):
        """Arguments of the product kernel that fills the stored values of a depth, one set per block size."""
        by_size = {}
        for e, row in d["store"].items():
            size, ks = d["elems"][e]
            by_size.setdefault(size, []).append((row, ks))
        out = []
        for size, items in by_size.items():
            n = max(len(ks) for _, ks in items)
            cids = np.zeros((len(items), n), dtype=np.int32)
            for i, (_, ks) in enumerate(items):
                cids[i, :len(ks)] = ks
            out.append((torch.tensor([r for r, _ in items], dtype=torch.int32, device=self.device),
                        torch.from_numpy(cids).to(self.device), size))
        return out

    def _operand(self, d, g, mode):
        """Operand rows of an MMA group, one line per 16-deep step."""
        if mode == 1:
            return np.concatenate([np.arange(p, p + g.direct, 16) for p in g.ops])[:, None]
        elems, store = d["elems"], d["store"]
        nk = max(len(elems[e][1]) for e in g.ops)
        rows = []
        for e in g.ops:
            size, ks = elems[e]
            ks = ks + [0] * (nk - len(ks))
            for o in range(0, size, 16):
                # (an absent child is a dummy row: zeros, whatever the offset)
                rows.append([k + o if k else 0 for k in ks] + ([store[e] + o] if store else []))
        return np.asarray(rows)

    def _outputs(self, d, g, mode, kids):
        """Output records of an MMA group, one per strip."""
        if mode == 0:
            out = np.zeros((len(g.blocks) * (g.bs // 16), 4), dtype=np.int32)
            out[:, 0] = np.concatenate([np.arange(b, b + g.bs, 16) for b in g.blocks])
            return out
        return np.asarray([self._record(d, e, o, kids) for e in g.blocks for o in range(0, g.bs, 16)], dtype=np.int32)

    def _record(self, d, e, o, kids):
        """Output record of element block e from row o on (backward)."""
        size, ks = d["elems"][e]
        if d["store"]:
            return [e + o, d["store"][e] + o, 0, -1]
        if len(ks) <= 2:
            return [e + o, ks[0] + o, ks[1] + o if len(ks) == 2 else 0, int(d["direct"])]
        return [e + o, kids.add([k + o for k in ks]), len(ks), 2 + int(d["direct"])]

    def _cta_tasks(self, d, g, mode, per, kids, frag, strips, tasks):
        rows = self._operand(d, g, mode)
        out, bases = self._outputs(d, g, mode, kids), g.par[0]
        nk = rows.shape[1] - (1 if mode == 0 and d["store"] else 0)
        off = kids.add(rows)
        s = 0
        while s < len(out):
            n = min(per, len(out) - s)
            while n & (n - 1):                                 # powers of two divide the warps evenly
                n &= n - 1
            fo = frag.add(bases[s:s + n].transpose(1, 0, 2))
            tasks.append((off, rows.shape[0], nk, rows.shape[1], strips.add(out[s:s + n]), n, fo, K_CTA, 0, 0, 0, 0))
            s += n

    def _fw_tasks(self, d, g, stored, per, kids, frag, strips, tasks, split):
        elems, store = d["elems"], d["store"]
        nk = max(len(elems[e][1]) for e in g.ops)
        n_kids = -1 if stored else nk
        if g.mma:
            rows = self._operand(d, g, 0)
            if stored:
                rows = rows[:, -1:]
            off, out, bases = kids.add(rows), self._outputs(d, g, 0, kids), g.par[0]
            for s in range(0, len(out), per):
                n = min(per, len(out) - s)
                fo = frag.add(bases[s:s + n].transpose(1, 0, 2))
                tasks.append((off, rows.shape[0], n_kids, rows.shape[1], strips.add(out[s:s + n]), n, fo, K_MMA, 0, 0, 0, 0))
            return
        depth = sum(elems[e][0] for e in g.ops)
        lg = 3 if all(elems[e][0] % 8 == 0 for e in g.ops) else 0
        step = 1 << lg
        for b, pids in zip(g.blocks, g.par):
            for r in range(0, g.bs, 16):
                n = min(16, g.bs - r)
                rows = []
                for e, pid in zip(g.ops, pids.tolist()):
                    size, ks = elems[e]
                    ks = ks + [0] * (nk - len(ks))
                    for o in range(0, size, step):
                        rows.append([pid + o * g.bs + r] + ([store[e] + o] if stored else
                                    [k + o if k else 0 for k in ks] + ([store[e] + o] if store else [])))
                rows = np.asarray(rows)
                st = np.asarray([[b + r, 0, 0, 0]])
                kind = K_SPLIT if (n == 1 and depth >= 256) else K_SIMT
                (split if kind == K_SPLIT else tasks).append(
                    (kids.add(rows), depth, n_kids, rows.shape[1], strips.add(st), n, 0, kind, g.bs, 1, lg, 0))

    def _bk_tasks(self, d, g, per, kids, frag, strips, tasks):
        pbs = g.direct
        if g.mma:
            rows = self._operand(d, g, 1)
            off, out, bases = kids.add(rows), self._outputs(d, g, 1, kids), g.par[0]
            for s in range(0, len(out), per):
                n = min(per, len(out) - s)
                fo = frag.add(bases[s:s + n].transpose(1, 0, 2))
                tasks.append((off, rows.shape[0], 1, 1, strips.add(out[s:s + n]), n, fo, K_MMA, 0, 0, 0, 0))
            return
        lg = 3 if pbs % 8 == 0 else 0
        step = 1 << lg
        for e, pids in zip(g.blocks, g.par if not isinstance(g.par, tuple) else g.par[1]):
            for r in range(0, g.bs, 16):
                n = min(16, g.bs - r)
                rows = np.asarray([[pid + r * pbs + o, p + o] for p, pid in zip(g.ops, pids.tolist())
                                   for o in range(0, pbs, step)])
                st = np.asarray([self._record(d, e, r, kids)])
                tasks.append((kids.add(rows), len(g.ops) * pbs, 1, 2, strips.add(st), n, 0, K_SIMT, 1, pbs, lg, 0))

    # ---- parameter flows ---------------------------------------------------------------------------------------------
    # Tied tables contract one product over all their layers' samples.  A 64 x 64 tile of a job of its own forms the
    # exponentials of its rows and of its elements again for every tile they belong to; the product of the dense layers forms
    # them once (`pcx_sum_par_dense2_stage`) and multiplies on the fifth-generation tensor cores, but takes two launches and
    # two more passes over the operands.  Rows x children x samples where the two meet, from HMMs of 128 to 1024 states
    # (microseconds, jobs / product): 256 states, 31 layers, 128 samples 64 / 59; 512, 7, 64: 47 / 51; 512, 63, 16: 82 / 52;
    # 1024, 31, 128: 329 / 116.  Tables of 128 rows fill half a product tile and never gain.
    DENSE_PAR_ROWS, DENSE_PAR_DEPTH, DENSE_PAR_WORK = 256, 256, 200_000_000

    def _tied_groups(self):
        """Groups of tied tables whose parameter flows may be one dense product."""
        found = {}
        for d in self.depths:
            for g in d["fw"]:
                rows = len(g.blocks) * g.bs
                if (not g.mma or d["store"] or g.bs % 128 != 0 or not self.DENSE_PAR_ROWS <= rows <= 6144
                        or g.depth < self.DENSE_PAR_DEPTH or max(len(d["elems"][e][1]) for e in g.ops) > 8):
                    continue
                sizes = tuple(d["elems"][e][0] for e in g.ops)
                found.setdefault((g.par[1].tobytes(), g.bs, sizes), []).append((d["elems"], g))
        tied = []
        put = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).to(self.device)
        for (_, bs, sizes), members in found.items():
            if len(members) < 2:
                continue
            fc = max(len(elems[e][1]) for elems, g in members for e in g.ops)
            fc = 2 if fc <= 2 else (4 if fc <= 4 else 8)
            off = np.concatenate([np.arange(s) for s in sizes])
            fk = np.zeros((len(members), off.size, fc), dtype=np.int32)
            for m, (elems, g) in enumerate(members):
                for j in range(fc):
                    row = np.repeat([elems[e][1][j] if j < len(elems[e][1]) else 0 for e in g.ops], sizes)
                    fk[m, :, j] = np.where(row != 0, row + off, 0)
            g = members[0][1]
            each = lambda t: np.repeat(t, sizes, axis=1) + off[None, :] * bs
            tied.append(dict(members={id(g) for _, g in members}, n=len(members), fc=fc, K=off.size, bs=bs,
                             n_blocks=len(g.blocks), fk=put(fk), nids=put([g.blocks for _, g in members]),
                             cids=put(np.ones((len(g.blocks), off.size))), pids=put(each(g.par[1])), pfids=put(each(g.flow))))
        return tied

    def _par_jobs(self, dense):
        pp, kids = _Pool(2), _Pool()
        jobs = {0: [], 1: [], 2: [], 3: []}
        covered = set().union(*[g["members"] for g in dense])
        for d in self.depths:
            elems, store = d["elems"], d["store"]
            for g in d["fw"]:
                if id(g) in covered:
                    continue
                nk = max(len(elems[e][1]) for e in g.ops)
                par = g.par[1] if isinstance(g.par, tuple) else g.par

                def entry(e, o):
                    if store:
                        return [store[e] + o]
                    ks = elems[e][1]
                    return [k + o for k in ks] + [0] * (nk - len(ks))

                width = 1 if store else nk
                n_kids = -1 if store else nk
                if g.mma:
                    steps = [(e, o, i) for i, e in enumerate(g.ops) for o in range(0, elems[e][0], 16)]
                    strips = [(b, r) for b in range(len(g.blocks)) for r in range(0, g.bs, 16)]
                    # tiles of 64 x 64 where the group has them, of 32 x 32 otherwise
                    kind = 0 if n_kids > 2 else (3 if len(steps) > 2 and len(strips) > 2 else 2)
                    most = 4 if kind == 3 else 2
                    for k0 in range(0, len(steps), most):
                        ks = steps[k0:k0 + most]
                        off = kids.add([entry(e, o) for e, o, _ in ks])
                        for s0 in range(0, len(strips), most):
                            ss = strips[s0:s0 + most]
                            tab = [[par[b, i] + o * g.bs + r, g.flow[b, i] + o * g.bs + r] for _, o, i in ks for b, r in ss]
                            row = [g.blocks[b] + r for b, r in ss]
                            row += [row[-1]] * (4 - len(row))
                            jobs[kind].append((row[0], row[1], len(ss), off, len(ks), n_kids, width, pp.add(tab), g.bs, 0,
                                               row[2], row[3]))
                    continue
                lg = 3 if all(elems[e][0] % 8 == 0 for e in g.ops) else 0
                step = 1 << lg
                ents = [(e, o, i) for i, e in enumerate(g.ops) for o in range(0, elems[e][0], step)]
                per = 64 // step
                for k0 in range(0, len(ents), per):
                    ks = ents[k0:k0 + per]
                    off = kids.add([entry(e, o) for e, o, _ in ks])
                    for b, first in enumerate(g.blocks):
                        for r in range(0, g.bs, 16):
                            tab = [[par[b, i] + o * g.bs + r, g.flow[b, i] + o * g.bs + r] for _, o, i in ks]
                            jobs[1].append((first + r, 0, min(16, g.bs - r), off, len(ks) * step, n_kids, width, pp.add(tab),
                                            g.bs, lg, 0, 0))
        return dict(pp=pp.tensor(self.device), kids=kids.tensor(self.device), dense=dense,
                    jobs={k: (torch.from_numpy(np.array(v, dtype=PAR).view(np.uint8)).to(self.device), len(v))
                          for k, v in jobs.items() if v})

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
        for launch in p["launches"]:
            if isinstance(launch, list):
                for nids, cids, size in launch:
                    _lib.call("pcx_prod_fwd", em, nm, nids, cids, nids.numel(), cids.size(1), size, W)
                continue
            levels, n, (nt, tiles, cluster, wide) = launch
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
        for par in self._par.values():
            for g in par["dense"] if isinstance(par, dict) else ():
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
