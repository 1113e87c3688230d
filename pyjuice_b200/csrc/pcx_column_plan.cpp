// Host side of the column program (pcx_column.cu): cuts a circuit's levels into tasks.
//
// A planner is made once per circuit from its index tables: for every depth the row groups (rows that share one list of
// children), the child rows of every folded product, and for the backward pass which level first touches a flow row.  A cut
// is made per row width: the tasks, operand tables and launches of both directions.  Both run inside the first pass of a
// circuit or of a width, which is why they are native: the same walks over the tables in Python took 0.5 s for a
// Poon-Domingos circuit over 784 variables with 64 latents (1.3 M table entries, 94 k parameter fragments) and 0.25 s for each
// width, where the pass itself takes 2.5 ms.
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <memory>
#include <stdexcept>
#include <string>
#include <unordered_map>
#include <utility>
#include <vector>
#include "../../include/pcx_b200.h"

namespace {

// The circuit has a table the column program does not cover.
struct Unsupported : std::runtime_error {
    using std::runtime_error::runtime_error;
};

enum Kind { K_MMA = 0, K_SIMT = 1, K_SPLIT = 2, K_PROD = 3, K_CTA = 4 };
constexpr int WARPS = 16;                       // per CTA of the fused levels
constexpr int BIG_STRIPS = 8, BIG_STEPS = 8, BIG_MAX_STEPS = 64;   // a group for CTA tasks: rows and depth (in 16) it has at least, and at most
constexpr int MAX_KIDS_FOLDED = 4;              // elements of more children (shared leaves) keep their value for the backward pass
constexpr int MAX_FOLD_READS = 16;              // child-row reads per element that folding may cost

using Ints = std::vector<int32_t>;

uint64_t hash_words(const int32_t* p, size_t n) {
    uint64_t h = 0x9e3779b97f4a7c15ull ^ n;
    auto mix = [&h](uint64_t x) {
        h = (h ^ x) * 0xff51afd7ed558ccdull;
        h ^= h >> 29;
    };
    size_t i = 0;
    for (; i + 2 <= n; i += 2) {
        uint64_t x;
        std::memcpy(&x, p + i, 8);
        mix(x);
    }
    if (i < n) mix((uint32_t)p[i]);
    return h ^ (h >> 32);
}
struct HashInts {
    size_t operator()(const Ints& v) const { return hash_words(v.data(), v.size()); }
};

// Append-only table of records of `width` words; equal pieces (shared children, tied layers) are stored once.
struct Pool {
    explicit Pool(int w) : width(w), slots(1024) {}
    int add(const int32_t* p, size_t n) {
        if (2 * (used + 1) > slots.size()) grow();
        const uint64_t h = hash_words(p, n);
        size_t i = h & (slots.size() - 1);
        for (; slots[i].n != 0; i = (i + 1) & (slots.size() - 1))
            if (slots[i].hash == h && slots[i].n == n && std::memcmp(data.data() + slots[i].at, p, n * 4) == 0) return (int)(slots[i].at / width);
        const size_t at = data.size();
        if (at / width > INT32_MAX) throw Unsupported("tables beyond the 32-bit range");
        slots[i] = Slot{h, at, n};
        ++used;
        data.insert(data.end(), p, p + n);
        return (int)(at / width);
    }
    int add(const Ints& v) { return add(v.data(), v.size()); }
    int width;
    Ints data;

private:
    struct Slot { uint64_t hash = 0; size_t at = 0, n = 0; };               // n = 0: free (no empty piece is ever added)
    std::vector<Slot> slots;
    size_t used = 0;
    void grow() {
        std::vector<Slot> old(slots.size() * 2);
        old.swap(slots);
        for (const Slot& s : old)
            if (s.n != 0) {
                size_t i = s.hash & (slots.size() - 1);
                while (slots[i].n != 0) i = (i + 1) & (slots.size() - 1);
                slots[i] = s;
            }
    }
};

struct Elem { int id, size, first, n, store; };            // element block: children kids[first .. first + n), stored row or -1

// Rows with one operand list: the node blocks (`blocks`: first rows), per operand block its first row (`ops`), and for every
// (block, operand) its parameter and flow.
struct Group {
    int bs = 0, pbs = 0, depth = 0, tied = -1;
    int cls = -1;                               // groups of one class have the same parameters in the same order
    bool mma = false, big = false;
    Ints blocks, ops, par, flow;
    int strips() const { return (int)blocks.size() * bs / 16; }
    int steps() const { return depth / 16; }
};

struct ProdRow { int row, size, first, n, add; };           // node block (backward): its parent products

struct Depth {
    std::vector<Elem> elems;
    Ints kids, parents;                                     // children of `elems`, parents of `prod_bk`
    int lo = 0;
    Ints index;                                             // element id - lo -> place in `elems`
    std::vector<Group> fw, bk;
    std::vector<ProdRow> prod_bk;
    bool direct = false, stored = false;
    int max_kids = 0;
    const Elem* find(int e) const {
        const int64_t i = (int64_t)e - lo;
        return i >= 0 && i < (int64_t)index.size() && index[i] >= 0 ? &elems[index[i]] : nullptr;
    }
};

// Reads the description of a circuit's tables (see pcx_colplan_new).
struct Reader {
    const int64_t* p;
    const int64_t* end;
    const int32_t* tables;
    int64_t n_tables;
    int64_t num() {
        if (p >= end) throw std::runtime_error("column planner: the description is too short");
        return *p++;
    }
    const int32_t* table(int64_t n) {
        const int64_t at = num();
        if (at < 0 || n < 0 || at + n > n_tables) throw std::runtime_error("column planner: a table lies outside the array");
        return tables + at;
    }
};

int prefix(const int32_t* row, int n) {
    int m = 0;
    for (int i = 0; i < n; ++i) m += row[i] != 0;
    for (int i = 0; i < m; ++i)
        if (row[i] == 0) throw Unsupported("padding inside a table row");
    return m;
}

// Tables on their way to the device: one array with sections on 64-byte boundaries, and a description of the sections.
struct Blob {
    Ints data;
    std::vector<int64_t> meta;
    int64_t section(const int32_t* p, size_t n) {
        data.resize((data.size() + 15) & ~size_t(15));
        const int64_t at = (int64_t)data.size();
        data.insert(data.end(), p, p + n);
        return at;
    }
    int64_t section(const Ints& v) { return section(v.data(), v.size()); }
};

int cdiv(int64_t a, int64_t b) { return (int)((a + b - 1) / b); }

struct Shape { int nt, tiles, cluster, wide; };             // of a launch: see pcx_column_run

}  // namespace

struct PcxColPlanner {
    int64_t num_nodes = 0, num_elements = 0;
    std::vector<Depth> depths;
    int em_rows = 0, big_steps = 0, n_classes = 0;

    // One partition of a layer's tables: n rows; a [n], the others [n, width].  Products: (element, children), (node, parent
    // elements).  Sums: (node, children, parameters, flows), (element, parents, parameters) with child blocks of `cbs`.
    struct Part { int n, width, cbs; const int32_t *a, *b, *c, *d; };
    struct Layer { int bs; std::vector<Part> fw, bk; };

    void classify(Group& g) {
        g.big = g.mma && g.strips() >= BIG_STRIPS && g.steps() >= BIG_STEPS;
        if (g.mma && g.strips() >= BIG_STRIPS && g.steps() > BIG_MAX_STEPS) throw Unsupported("a dense table deeper than a CTA task gathers");
        if (g.big) big_steps = std::max(big_steps, g.steps());
    }

    void build(Reader& in) {
        num_nodes = in.num();
        num_elements = in.num();
        const int64_t num_dummy = in.num(), root0 = in.num(), root1 = in.num(), n_depths = in.num();
        std::vector<std::vector<Layer>> prods(n_depths), sums(n_depths);
        std::vector<char> parentless(n_depths);
        for (int64_t d = 0; d < n_depths; ++d) {
            parentless[d] = (char)in.num();
            for (int kind = 0; kind < 2; ++kind) {
                const int64_t n_layers = in.num();
                for (int64_t l = 0; l < n_layers; ++l) {
                    Layer layer;
                    layer.bs = (int)in.num();
                    for (int side = 0; side < 2; ++side) {
                        const int64_t parts = in.num();
                        for (int64_t q = 0; q < parts; ++q) {
                            Part t{};
                            t.n = (int)in.num();
                            t.width = (int)in.num();
                            t.cbs = (int)in.num();
                            const int64_t cells = (int64_t)t.n * t.width;
                            t.a = in.table(t.n);
                            t.b = in.table(cells);
                            if (kind == 1) t.c = in.table(cells);
                            if (kind == 1 && side == 0) t.d = in.table(cells);
                            (side == 0 ? layer.fw : layer.bk).push_back(t);
                        }
                    }
                    (kind == 0 ? prods : sums)[d].push_back(std::move(layer));
                }
            }
        }
        // parent products of every node in the whole circuit
        Ints parents(num_nodes + 1, 0);
        for (auto& layers : prods)
            for (auto& layer : layers)
                for (auto& t : layer.fw)
                    for (int64_t i = 0; i < (int64_t)t.n * t.width; ++i)
                        if (t.b[i] != 0) {
                            if (t.b[i] < 0 || t.b[i] + (int64_t)layer.bs > num_nodes) throw std::runtime_error("column planner: a child row outside the circuit");
                            for (int j = 0; j < layer.bs; ++j) ++parents[t.b[i] + j];
                        }
        depths.resize(n_depths);
        for (int64_t d = 0; d < n_depths; ++d) depth(depths[d], prods[d], sums[d], parentless[d] != 0, parents);
        std::unordered_map<Ints, int, HashInts> classes;
        Ints key;
        for (Depth& d : depths)
            for (int side = 0; side < 2; ++side)
                for (Group& g : side == 0 ? d.fw : d.bk) {
                    if (!g.mma) continue;
                    key = g.par;
                    for (int e : g.ops) key.push_back(side == 0 ? d.find(e)->size : g.pbs);
                    key.insert(key.end(), {side, g.bs, (int)g.ops.size()});
                    g.cls = classes.emplace(key, n_classes).first->second;
                    n_classes = (int)classes.size();
                }
        // which level first writes a flow row
        std::vector<char> written(num_nodes, 0);
        std::fill(written.begin() + root0, written.begin() + root1, 1);
        std::fill(written.begin(), written.begin() + num_dummy, 1);
        for (int64_t d = n_depths - 1; d >= 0; --d) {
            Depth& q = depths[d];
            if (q.direct) {
                for (const Elem& e : q.elems)
                    for (int c = 0; c < e.n; ++c) std::fill_n(written.begin() + q.kids[e.first + c], e.size, 1);
                continue;
            }
            for (ProdRow& p : q.prod_bk) {
                if (p.row < 0 || p.row + (int64_t)p.size > num_nodes) throw std::runtime_error("column planner: a flow row outside the circuit");
                int seen = 0;
                for (int j = 0; j < p.size; ++j) seen += written[p.row + j];
                if (seen != 0 && seen != p.size) throw Unsupported("a flow block is written in pieces");
                p.add = seen != 0;
                std::fill_n(written.begin() + p.row, p.size, 1);
            }
        }
        if (std::find(written.begin(), written.end(), 0) != written.end()) throw Unsupported("a node without parents");
    }

    void depth(Depth& d, const std::vector<Layer>& prods, const std::vector<Layer>& sums, bool parentless, const Ints& parents) {
        int lo = INT32_MAX, hi = -1;
        for (auto& layer : prods)
            for (auto& t : layer.fw)
                for (int i = 0; i < t.n; ++i) {
                    lo = std::min(lo, t.a[i]);
                    hi = std::max(hi, t.a[i]);
                }
        if (hi < lo) throw Unsupported("a depth without products");
        if (lo < 0 || hi >= num_elements) throw std::runtime_error("column planner: an element outside the circuit");
        d.lo = lo;
        d.index.assign((size_t)(hi - lo) + 1, -1);
        d.direct = !parentless;
        for (auto& layer : prods)
            for (auto& t : layer.fw)
                for (int i = 0; i < t.n; ++i) {
                    Elem e{t.a[i], layer.bs, (int)d.kids.size(), 0, -1};
                    for (int c = 0; c < t.width; ++c) {
                        const int k = t.b[(int64_t)i * t.width + c];
                        if (k == 0) continue;
                        d.kids.push_back(k);
                        ++e.n;
                        for (int j = 0; j < e.size; ++j) d.direct = d.direct && parents[k + j] == 1;
                    }
                    d.max_kids = std::max(d.max_kids, e.n);
                    d.index[e.id - lo] = (int)d.elems.size();
                    d.elems.push_back(e);
                }
        int64_t reads = 0;
        Ints ids, at;
        for (auto& layer : sums) {
            std::unordered_map<Ints, int, HashInts> merged;
            const size_t base = d.fw.size();
            for (auto& t : layer.fw)
                for (int i = 0; i < t.n; ++i) {
                    const int32_t *c = t.b + (int64_t)i * t.width, *p = t.c + (int64_t)i * t.width, *f = t.d + (int64_t)i * t.width;
                    const int n = prefix(c, t.width);
                    ids.clear();
                    at.clear();
                    for (int k = 0; k < n;) {
                        const Elem* e = d.find(c[k]);
                        if (!e) throw Unsupported("a child list that does not start at an element block");
                        if (k + e->size > n) throw Unsupported("a child list that is not made of element blocks");
                        for (int j = 1; j < e->size; ++j)
                            if (c[k + j] != c[k] + j) throw Unsupported("a child list that is not made of element blocks");
                        for (const int32_t* tab : {p, f})
                            if (tab[k + e->size - 1] != tab[k] + (e->size - 1) * layer.bs)
                                throw Unsupported("parameters of an element block are not contiguous");
                        ids.push_back(e->id);
                        at.push_back(k);
                        k += e->size;
                    }
                    auto found = merged.emplace(ids, (int)(d.fw.size() - base));
                    if (found.second) {
                        d.fw.emplace_back();
                        d.fw.back().ops = ids;
                        d.fw.back().bs = layer.bs;
                    }
                    Group& g = d.fw[base + found.first->second];
                    g.blocks.push_back(t.a[i]);
                    for (int k : at) {
                        g.par.push_back(p[k]);
                        g.flow.push_back(f[k]);
                    }
                }
            for (size_t q = base; q < d.fw.size(); ++q) {
                Group& g = d.fw[q];
                if (g.ops.empty()) throw Unsupported("a sum node without children");
                int smallest = INT32_MAX;
                for (int e : g.ops) {
                    smallest = std::min(smallest, d.find(e)->size);
                    g.depth += d.find(e)->size;
                }
                g.mma = g.bs >= 32 && smallest >= 32;
                classify(g);
                if (!g.big) reads = std::max<int64_t>(reads, (int64_t)g.blocks.size() * std::max(1, g.mma ? g.bs / 64 : g.bs / 16));
            }
        }
        if (reads * d.max_kids > MAX_FOLD_READS && reads > 1) throw Unsupported("products shared by too many rows to be folded");
        d.stored = d.max_kids > MAX_KIDS_FOLDED && !d.direct;
        if (d.stored)
            for (Elem& e : d.elems) {
                e.store = em_rows;
                em_rows += e.size;
            }
        std::vector<char> seen(d.elems.size(), 0);
        size_t n_seen = 0;
        for (auto& layer : sums) {
            std::unordered_map<Ints, int, HashInts> merged;
            const size_t base = d.bk.size();
            for (auto& t : layer.bk)
                for (int i = 0; i < t.n; ++i) {
                    const int32_t *p = t.b + (int64_t)i * t.width, *q = t.c + (int64_t)i * t.width;
                    const int n = prefix(p, t.width);
                    const Elem* e = d.find(t.a[i]);
                    if (!e || e->size != t.cbs || n == 0 || seen[e - d.elems.data()]) throw Unsupported("element block split over layers");
                    seen[e - d.elems.data()] = 1;
                    ++n_seen;
                    ids.assign(p, p + n);
                    ids.push_back(t.cbs);
                    auto found = merged.emplace(ids, (int)(d.bk.size() - base));
                    if (found.second) {
                        d.bk.emplace_back();
                        d.bk.back().ops.assign(p, p + n);
                        d.bk.back().bs = t.cbs;
                        d.bk.back().pbs = layer.bs;
                    }
                    Group& g = d.bk[base + found.first->second];
                    g.blocks.push_back(t.a[i]);
                    g.par.insert(g.par.end(), q, q + n);
                }
            for (size_t q = base; q < d.bk.size(); ++q) {
                Group& g = d.bk[q];
                g.mma = g.bs >= 32 && g.pbs >= 32;
                g.depth = (int)g.ops.size() * g.pbs;
                classify(g);
            }
        }
        if (d.direct && n_seen != d.elems.size()) throw Unsupported("a product without a sum parent");
        if (!d.direct)
            for (auto& layer : prods)
                for (auto& t : layer.bk)
                    for (int i = 0; i < t.n; ++i) {
                        ProdRow r{t.a[i], layer.bs, (int)d.parents.size(), 0, 0};
                        for (int c = 0; c < t.width; ++c)
                            if (t.b[(int64_t)i * t.width + c] != 0) {
                                d.parents.push_back(t.b[(int64_t)i * t.width + c]);
                                ++r.n;
                            }
                        d.prod_bk.push_back(r);
                    }
    }

    // ---- parameter flows of tied tables through one dense product: see column.py ------------------------------------
    static constexpr int DENSE_PAR_ROWS = 256, DENSE_PAR_MAX_ROWS = 6144, DENSE_PAR_DEPTH = 256;
    struct Tied { std::vector<std::pair<int, int>> members; };               // (depth, place in its `fw`)
    std::vector<Tied> tied;

    void find_tied() {
        std::vector<int> found(n_classes, -1);
        std::vector<Tied> all;
        for (int i = 0; i < (int)depths.size(); ++i)
            for (int q = 0; q < (int)depths[i].fw.size(); ++q) {
                const Depth& d = depths[i];
                const Group& g = d.fw[q];
                const int64_t rows = (int64_t)g.blocks.size() * g.bs;
                if (!g.mma || d.stored || g.bs % 128 != 0 || rows < DENSE_PAR_ROWS || rows > DENSE_PAR_MAX_ROWS || g.depth < DENSE_PAR_DEPTH) continue;
                int kids = 0;
                for (int e : g.ops) kids = std::max(kids, d.find(e)->n);
                if (kids > 8) continue;
                if (found[g.cls] < 0) {
                    found[g.cls] = (int)all.size();
                    all.emplace_back();
                }
                all[found[g.cls]].members.emplace_back(i, q);
            }
        for (Tied& t : all)
            if (t.members.size() >= 2) {
                for (auto& m : t.members) depths[m.first].fw[m.second].tied = (int)tied.size();
                tied.push_back(std::move(t));
            }
    }

    // ---- chains: see pcx_column_chain.cu -------------------------------------------------------------------------------
    // Runs of depths of one group each, with the same parameters, where the operand of a depth is the output of the one below
    // and at most one other row per element.  From three levels on: the launch costs about what two levels gain.
    static constexpr int CHAIN_LEVELS = 3, CHAIN_MIN_STRIPS = 4, CHAIN_MAX_STRIPS = 64;
    struct Chain {
        int first, n, strips;                   // depths first .. first + n - 1
        Ints rows[2];                           // tables of the two directions: see pcx_column_chain
    };
    std::vector<Chain> chains;

    // Child rows of 16-row pieces of the elements `ids`, two words each.
    static Ints pieces(const Depth& d, const Ints& ids, int strips) {
        Ints out;
        out.reserve(2 * (size_t)strips);
        for (int id : ids) {
            const Elem& e = *d.find(id);
            const int x = e.n > 0 ? d.kids[e.first] : 0, y = e.n > 1 ? d.kids[e.first + 1] : 0;
            for (int o = 0; o < e.size; o += 16) {
                out.push_back(x != 0 ? x + o : 0);
                out.push_back(y != 0 ? y + o : 0);
            }
        }
        return out;
    }
    // Puts the child first that is the row of the blocks' piece; false where there is none.
    static bool order(Ints& p, const Ints& blocks, int size) {
        size_t at = 0;
        for (int b : blocks)
            for (int r = b; r < b + size; r += 16, at += 2) {
                if (at + 2 > p.size()) return false;
                if (p[at + 1] == r) std::swap(p[at], p[at + 1]);
                if (p[at] != r || p[at + 1] == r) return false;
            }
        return at == p.size();
    }
    static bool chain_depth(const Depth& d) {
        if (d.fw.size() != 1 || d.bk.size() != 1 || !d.direct || d.stored || !d.fw[0].mma || !d.bk[0].mma || d.max_kids > 2) return false;
        const Group &f = d.fw[0], &b = d.bk[0];
        const int S = f.strips();
        if (S < CHAIN_MIN_STRIPS || S > CHAIN_MAX_STRIPS || f.depth != 16 * S || b.depth != 16 * S || b.strips() != S) return false;
        for (auto& e : d.elems)
            if (e.n < 1) return false;
        return true;
    }
    // Extends the pieces of a run of depths (operands forward, outputs backward) by those of `d`, if it follows.
    static bool follows(const Depth& d, const Depth& below, std::vector<Ints> (&sides)[2]) {
        if (d.fw[0].cls != below.fw[0].cls || d.bk[0].cls != below.bk[0].cls) return false;
        Ints f = pieces(d, d.fw[0].ops, d.fw[0].strips()), b = pieces(d, d.bk[0].blocks, d.fw[0].strips());
        if (!order(f, below.fw[0].blocks, below.fw[0].bs) || !order(b, below.bk[0].ops, below.bk[0].pbs)) return false;
        sides[0].push_back(std::move(f));
        sides[1].push_back(std::move(b));
        return true;
    }
    void find_chains() {
        const int n = (int)depths.size();
        for (int i = 0, end; i < n; i = end) {
            end = i + 1;
            const Depth& low = depths[i];
            if (!chain_depth(low)) continue;
            const int strips = low.fw[0].strips();
            std::vector<Ints> sides[2] = {{pieces(low, low.fw[0].ops, strips)}, {pieces(low, low.bk[0].blocks, strips)}};
            while (end < n && end - i < PCX_COLUMN_MAX_LEVELS && chain_depth(depths[end]) && follows(depths[end], depths[end - 1], sides)) ++end;
            if (end - i < CHAIN_LEVELS) continue;
            const Depth& top = depths[end - 1];
            Chain c{i, end - i, strips, {}};
            for (Ints& t : c.rows) t.reserve(2 * (size_t)strips * (size_t)(c.n + 1));
            auto add = [](Ints& to, const Ints& p) { to.insert(to.end(), p.begin(), p.end()); };
            auto rows_of = [](Ints& to, const Ints& blocks, int size) {
                for (int b : blocks)
                    for (int r = b; r < b + size; r += 16) to.insert(to.end(), {r, 0});
            };
            for (const Ints& p : sides[0]) add(c.rows[0], p);       // a level's outputs are the first children of the next one's operand
            rows_of(c.rows[0], top.fw[0].blocks, top.fw[0].bs);
            rows_of(c.rows[1], top.bk[0].ops, top.bk[0].pbs);
            for (size_t k = sides[1].size(); k-- > 0;) add(c.rows[1], sides[1][k]);
            chains.push_back(std::move(c));
        }
    }

    // Per group: members, children per element, depth, block size, blocks, then where child rows [members, depth, children],
    // node rows [members, blocks], ones, parameters and flows [blocks, depth] lie.
    void tied_tables(Blob& out) const {
        for (const Tied& t : tied) {
            const Depth& d0 = depths[t.members[0].first];
            const Group& g0 = d0.fw[t.members[0].second];
            int fc = 0;
            for (auto& m : t.members)
                for (int e : depths[m.first].fw[m.second].ops) fc = std::max(fc, depths[m.first].find(e)->n);
            fc = fc <= 2 ? 2 : (fc <= 4 ? 4 : 8);
            const int K = g0.depth, n_ops = (int)g0.ops.size();
            Ints fk, nids;
            for (auto& m : t.members) {
                const Depth& d = depths[m.first];
                const Group& g = d.fw[m.second];
                nids.insert(nids.end(), g.blocks.begin(), g.blocks.end());
                for (int id : g.ops) {
                    const Elem* e = d.find(id);
                    for (int o = 0; o < e->size; ++o)
                        for (int j = 0; j < fc; ++j) fk.push_back(j < e->n ? d.kids[e->first + j] + o : 0);
                }
            }
            Ints ones(g0.blocks.size() * (size_t)K, 1), each[2];
            for (int side = 0; side < 2; ++side)
                for (size_t b = 0; b < g0.blocks.size(); ++b)
                    for (int q = 0; q < n_ops; ++q)
                        for (int o = 0; o < d0.find(g0.ops[q])->size; ++o)
                            each[side].push_back((side == 0 ? g0.par : g0.flow)[b * n_ops + q] + o * g0.bs);
            for (int64_t v : {(int64_t)t.members.size(), (int64_t)fc, (int64_t)K, (int64_t)g0.bs, (int64_t)g0.blocks.size(),
                              out.section(fk), out.section(nids), out.section(ones), out.section(each[0]), out.section(each[1])})
                out.meta.push_back(v);
        }
    }

    // ---- launch geometry ---------------------------------------------------------------------------------------------
    struct Room {                               // clusters of 1, 2, 4, 8 and 16 CTAs that the device holds at a time, then, for a
        const int32_t* n;                       // circuit with chains, clusters of 1 ... 16 CTAs of a chain
        int operator()(int c) const { return std::max(1, (int)n[c == 1 ? 0 : c == 2 ? 1 : c == 4 ? 2 : c == 8 ? 3 : 4]); }
        int chain(int c) const { return std::max(1, (int)n[4 + c]); }
    };

    // Strips per CTA and columns per cluster of a chain of groups of S strips: the cheapest estimate of a level, in cycles, times
    // the waves of clusters.  `mma`: the products of a CTA's busiest scheduler, 8 cycles each (four warps share one); what else
    // grows with the rows and columns of a CTA (partial products, epilogue) grows with it.  `stream`: fragments that neither
    // tensor memory nor shared memory hold.  Cycles a level, measured forward / flows and estimated, states / columns a cluster x
    // strips a CTA, four clusters on the machine: 128 / 8 x 1 3140 / 3210, 3040; 256 / 8 x 2 3640 / 3770, 3470; 8 x 4 4020 / 4050, 4050;
    // 512 / 8 x 4 4460 / 4460, 5190; 8 x 8 5910 / 6110, 7490; 1024 / 8 x 4 5600 / 5720, 7490; 16 x 4 8770 / 9740, 12 080; 8 x 8 12 530 /
    // 12 550, 12 730; 24 x 4 15 970 / 17 200, 16 660; 16 x 8 22 010 / 22 920, 22 230.  Between the ends the estimate is up to 40 % high
    // (it was fitted when four strips of a warp cost more); the order of the shapes of one size, which is all it is for, is right.
    struct ChainShape { int nt, per, waves; double cost; };
    static ChainShape chain_shape(int64_t W, int S, const Room& room) {
        ChainShape best{0, 0, 0, 0.0};
        for (int nt : {1, 2, 3})
            for (int per : {1, 2, 3, 4, 6, 8}) {
                const int C = cdiv(S, per), halves = per > 1 && C <= 8 ? 2 : 1, kparts = 16 / halves;
                if (per > S || per * nt > 16 || C > kparts || cdiv(per, halves) > 4) continue;
                const int steps = cdiv(per, std::min(per, kparts / C)), q = cdiv(per, steps), strips = cdiv(per, halves);
                const int left = 231424 - 8960 - 2 * C * q * per * nt * 512;       // shared memory for fragments, as the launcher has it
                if (left < 0) continue;
                const int waves = cdiv(cdiv(W, 8 * nt), room.chain(C));
                const int slots = strips <= 1 ? 1 : strips <= 2 ? 2 : 4;
                const int held = 16 / slots + left / (16 * 1024 * slots);
                const double mma = 8.1 * 3 * nt * steps * strips * cdiv(C * q * halves, 4);
                const double stream = 1024.0 * C * q * halves * strips * std::max(0, steps - held) / 50.0;
                const double cost = waves * (2900.0 + 2.95 * mma + 0.25 * stream);
                if (best.nt == 0 || cost < best.cost - 1e-9) best = ChainShape{nt, per, waves, cost};
            }
        return best;
    }

    // (strips per task, time) of a level's large groups on a cluster of c CTAs: rounds of tasks times what a task takes in
    // microseconds: a fixed latency, the gather and exponentials of its operand, its multiplications, and parameters that
    // neither stay in shared memory nor arrive during the gather.  (Measured per level, mean of the two directions, CTAs x
    // columns: 512 x 512 on 4 x 8 / 8 x 16 8.5 / 9.6 us; 1024 x 1024 on 8 x 8 / 16 x 16 / 8 x 16 / 4 x 8 12.4 / 13.2 / 16.2 /
    // 16.9: sixteen columns cost the element flows two more microseconds than eight.)
    static std::pair<int, double> piece(const std::vector<Group>& groups, int nt, int c) {
        int steps = 0;
        for (auto& g : groups)
            if (g.big) steps = std::max(steps, g.steps());
        if (steps == 0) return {1, 0.0};
        std::pair<int, double> best{0, 0.0};
        for (int size : {16, 8, 4, 2, 1}) {
            int n = 0;
            for (auto& g : groups)
                if (g.big) n += cdiv(g.strips(), size);
            const double stream = std::max(0.0, (double)(size * steps - std::max(0, 150 - steps * nt / 2))) * 0.01;
            const double cost = cdiv(n, c) * (1.2 + 1.8 * nt + 0.025 * steps * nt + 0.003 * size * steps * nt + stream);
            if (best.first == 0 || cost < best.second - 1e-9) best = {size, cost};
        }
        return best;
    }

    // With large groups: the cheapest estimate of a pass, all levels with their barriers, times the waves of clusters.
    Shape big_shape(int64_t W, const Room& room) const {
        Shape best{};
        double least = 0.0;
        for (int nt : {1, 2}) {
            const int n = cdiv(W, 8 * nt);
            for (int c : {1, 2, 4, 8, 16}) {
                double cost = 0.0;
                for (auto& d : depths) cost += 0.5 + 0.03 * c + piece(d.fw, nt, c).second;
                cost *= cdiv(n, room(c));
                if (best.nt == 0 || cost < least - 1e-9) { best = Shape{nt, 1, c, 0}; least = cost; }
            }
        }
        return best;
    }

    // Without: as many CTAs as the machine holds at a time, but no larger a cluster than a level has strips for its warps
    // (`items` 16-row strips per level); among equals the widest column group, which reads longer pieces of a value row.  (A
    // device with 148 SMs holds 74, 33 and 15 clusters of 2, 4 and 8 CTAs.)
    static Shape small_shape(int64_t W, double items, const Room& room) {
        Shape best{};
        int64_t most = 0;
        for (int cols : {8, 16}) {
            const int n = cdiv(W, cols);
            int c = 1;
            while (c < 8 && room(c * 2) >= n && items > WARPS * c) c *= 2;
            if (best.nt == 0 || (cols <= W && (int64_t)n * c >= most)) {
                best = Shape{cols / 8, 1, c, 0};
                most = (int64_t)n * c;
            }
        }
        return best;
    }

    // Whether the program is the better choice at this row width.  With large groups it is while a level's CTA tasks go
    // around the cluster about once: it is then bound by the latency of a level, which is lower than that of the per-layer
    // kernels and of the tiles that wait on counters.  With several rounds per level a CTA works through its tasks one latency
    // after the other, where those keep two tiles per SM under way (784-variable tree, 128 latents, 512 samples: 745 us
    // forward against 556).
    bool suits(int64_t W, const Room& room) const {
        if (big_steps == 0) return true;
        // (or where every level of large groups lies inside a chain whose clusters fit at once)
        std::vector<char> chained(depths.size(), 0);
        for (auto& c : chains)
            if (chain_shape(W, c.strips, room).waves == 1) std::fill_n(chained.begin() + c.first, c.n, 1);
        bool all = true;
        for (size_t i = 0; i < depths.size(); ++i)
            for (auto& g : depths[i].fw) all = all && (!g.big || chained[i]);
        if (all) return true;
        const Shape s = big_shape(W, room);
        int64_t rounds = 0, levels = 0;
        for (auto& d : depths) {
            const int size = piece(d.fw, s.nt, s.cluster).first;
            int tasks = 0;
            for (auto& g : d.fw)
                if (g.big) tasks += cdiv(g.strips(), size);
            rounds += cdiv(tasks, s.cluster);
            levels += tasks > 0;
        }
        return cdiv(cdiv(W, 8 * s.nt), room(s.cluster)) == 1 && (double)rounds <= 1.5 * (double)levels;
    }
};

namespace {

// ---- cutting into tasks for one row width ------------------------------------------------------------------------------
struct Cutter {
    const PcxColPlanner& pc;
    const PcxColPlanner::Room room;
    const int64_t W;
    const int64_t wide_items;                   // (16-row strip, 32-column) pieces that give a level a launch of its own
    const int64_t prod_reads;                   // child rows a CTA may gather for the stored elements of a fused level
    Pool kids{1}, strips[2] = {Pool(4), Pool(4)};
    std::vector<PcxColTask> tasks[2], split;
    struct Level { int first, n, split_first, n_split; Shape how; int depth; };
    std::vector<Level> levels[2];
    Shape fused{};
    int wide_tiles;
    Ints rows, out;                             // scratch: operand entries, output records
    Ints frag;                                  // fragments, four words each
    std::vector<std::vector<std::pair<int64_t, int>>> made;                 // per class: (strip, strips) -> first fragment

    Cutter(const PcxColPlanner& p, int64_t W_, const int32_t* rooms, int64_t wide, int64_t reads)
        : pc(p), room{rooms}, W(W_), wide_items(wide), prod_reads(reads), wide_tiles(cdiv(W_, 32)), made(p.n_classes) {}

    bool is_wide(int64_t n) const { return pc.big_steps == 0 && W >= 32 && n * wide_tiles >= wide_items; }
    static int64_t count(const std::vector<Group>& groups) {
        int64_t n = 0;
        for (auto& g : groups) n += (int64_t)g.blocks.size() * std::max(1, g.bs / 16);
        return n;
    }
    Shape shape(int64_t n) const { return is_wide(n) ? Shape{4, wide_tiles, 1, 1} : fused; }
    // Few strips in a level: one per task, so that every warp has one (its rows share an operand with its neighbours', which
    // each of them gathers for itself).  Many: two share the gather.
    int strips_per_task(int64_t n) const {
        const int64_t workers = is_wide(n) ? wide_items / wide_tiles : (int64_t)WARPS * fused.cluster;
        return (int)std::max<int64_t>(1, std::min<int64_t>(2, n / std::max<int64_t>(1, workers)));
    }

    // Operand rows of an MMA group into `rows`, one entry per 16-deep step; returns the entries' width.
    int operand(const Depth& d, const Group& g, int mode, bool only_stored) {
        rows.clear();
        if (mode == 1) {
            for (int p : g.ops)
                for (int o = 0; o < g.pbs; o += 16) rows.push_back(p + o);
            return 1;
        }
        const int nk = children(d, g);
        for (int id : g.ops) {
            const Elem* e = d.find(id);
            for (int o = 0; o < e->size; o += 16) entry(d, *e, o, nk, only_stored);
        }
        return only_stored ? 1 : nk + d.stored;
    }
    static int children(const Depth& d, const Group& g) {
        int nk = 0;
        for (int e : g.ops) nk = std::max(nk, d.find(e)->n);
        return nk;
    }
    // (an absent child is a dummy row: zeros, whatever the offset)
    void entry(const Depth& d, const Elem& e, int o, int nk, bool only_stored) {
        if (!only_stored)
            for (int c = 0; c < nk; ++c) rows.push_back(c < e.n ? d.kids[e.first + c] + o : 0);
        if (d.stored) rows.push_back(e.store + o);
    }
    // Output record of element block e from row o on (backward).
    void record(const Depth& d, const Elem& e, int o) {
        const int32_t* k = d.kids.data() + e.first;
        if (d.stored) {
            out.insert(out.end(), {e.id + o, e.store + o, 0, -1});
        } else if (e.n <= 2) {
            out.insert(out.end(), {e.id + o, e.n > 0 ? k[0] + o : 0, e.n == 2 ? k[1] + o : 0, (int)d.direct});
        } else {
            Ints list(k, k + e.n);
            for (int& r : list) r += o;
            out.insert(out.end(), {e.id + o, kids.add(list), e.n, 2 + (int)d.direct});
        }
    }
    // Output records of an MMA group, one per strip.
    void outputs(const Depth& d, const Group& g, int mode) {
        out.clear();
        for (int b : g.blocks)
            for (int o = 0; o < g.bs; o += 16) {
                if (mode == 0) out.insert(out.end(), {b + o, 0, 0, 0});
                else record(d, *d.find(b), o);
            }
    }
    // Fragments [step][strip] of n strips of an MMA group from strip s on: parameter of (row 0, child 0), row and child strides.
    // Tied tables share theirs.
    int fragments(const Depth& d, const Group& g, int mode, int s, int n) {
        const int64_t key = (int64_t)s << 8 | n;
        auto& list = made[g.cls];
        if (!list.empty()) {
            auto it = std::lower_bound(list.begin(), list.end(), std::make_pair(key, 0));
            if (it != list.end() && it->first == key) return it->second;
        }
        const int sr = mode == 0 ? 1 : g.pbs, sk = mode == 0 ? g.bs : 1, per_block = g.bs / 16, n_ops = (int)g.ops.size();
        const int64_t at = (int64_t)frag.size() / 4;
        if (at + (int64_t)g.steps() * n > INT32_MAX) throw Unsupported("tables beyond the 32-bit range");
        frag.resize(frag.size() + (size_t)g.steps() * n * 4);
        int32_t* f = frag.data() + at * 4;
        for (int q = 0; q < n_ops; ++q) {
            const int size = mode == 0 ? d.find(g.ops[q])->size : g.pbs;
            for (int o = 0; o < size; o += 16)
                for (int i = s; i < s + n; ++i, f += 4) {
                    f[0] = g.par[(size_t)(i / per_block) * n_ops + q] + o * sk + (i % per_block) * 16 * sr;
                    f[1] = sr;
                    f[2] = sk;
                }
        }
        list.insert(std::lower_bound(list.begin(), list.end(), std::make_pair(key, 0)), {key, (int)at});
        return (int)at;
    }

    static PcxColTask task(int kid_off, int n_k, int n_kids, int width, int strip_off, int n_rows, int par_off, int kind, int sk = 0,
                           int sr = 0, int lg = 0) {
        PcxColTask t{};
        t.kid_off = kid_off; t.n_k = n_k; t.n_kids = n_kids; t.width = width; t.strip_off = strip_off; t.n_rows = n_rows;
        t.par_off = par_off; t.kind = kind; t.sk = sk; t.sr = sr; t.lg_entry = lg;
        return t;
    }

    void cta_tasks(const Depth& d, const Group& g, int mode, int per) {
        outputs(d, g, mode);
        const int width = operand(d, g, mode, false), nk = mode == 1 ? 1 : width - d.stored;
        const int off = kids.add(rows), n_out = (int)out.size() / 4;
        for (int s = 0; s < n_out;) {
            int n = std::min(per, n_out - s);
            while (n & (n - 1)) n &= n - 1;                 // powers of two divide the warps evenly
            const int fo = fragments(d, g, mode, s, n);
            split.push_back(task(off, g.steps(), nk, width, strips[mode].add(out.data() + 4 * s, 4 * (size_t)n), n, fo, K_CTA));
            s += n;
        }
    }
    void mma_tasks(const Depth& d, const Group& g, int mode, bool stored, int per) {
        const int width = operand(d, g, mode, stored), nk = mode == 1 ? 1 : (stored ? -1 : width - d.stored);
        const int off = kids.add(rows);
        outputs(d, g, mode);
        const int n_out = (int)out.size() / 4;
        for (int s = 0; s < n_out; s += per) {
            const int n = std::min(per, n_out - s), fo = fragments(d, g, mode, s, n);
            tasks[mode].push_back(task(off, g.steps(), nk, width, strips[mode].add(out.data() + 4 * s, 4 * (size_t)n), n, fo, K_MMA));
        }
    }
    void simt_forward(const Depth& d, const Group& g, bool stored) {
        const int nk = children(d, g), n_ops = (int)g.ops.size();
        int lg = 3;
        for (int e : g.ops)
            if (d.find(e)->size % 8 != 0) lg = 0;
        const int width = 1 + (stored ? 1 : nk + d.stored);
        for (size_t b = 0; b < g.blocks.size(); ++b)
            for (int r = 0; r < g.bs; r += 16) {
                const int n = std::min(16, g.bs - r);
                rows.clear();
                for (int q = 0; q < n_ops; ++q) {
                    const Elem* e = d.find(g.ops[q]);
                    for (int o = 0; o < e->size; o += 1 << lg) {
                        rows.push_back(g.par[b * n_ops + q] + o * g.bs + r);
                        entry(d, *e, o, nk, stored);
                    }
                }
                const int32_t st[4] = {g.blocks[b] + r, 0, 0, 0};
                const int kind = n == 1 && g.depth >= 256 ? K_SPLIT : K_SIMT;
                (kind == K_SPLIT ? split : tasks[0])
                    .push_back(task(kids.add(rows), g.depth, stored ? -1 : nk, width, strips[0].add(st, 4), n, 0, kind, g.bs, 1, lg));
            }
    }
    void simt_backward(const Depth& d, const Group& g) {
        const int lg = g.pbs % 8 == 0 ? 3 : 0, n_ops = (int)g.ops.size();
        for (size_t b = 0; b < g.blocks.size(); ++b)
            for (int r = 0; r < g.bs; r += 16) {
                rows.clear();
                for (int q = 0; q < n_ops; ++q)
                    for (int o = 0; o < g.pbs; o += 1 << lg) {
                        rows.push_back(g.par[b * n_ops + q] + r * g.pbs + o);
                        rows.push_back(g.ops[q] + o);
                    }
                out.clear();
                record(d, *d.find(g.blocks[b]), r);
                tasks[1].push_back(task(kids.add(rows), g.depth, 1, 2, strips[1].add(out), std::min(16, g.bs - r), 0, K_SIMT, 1, g.pbs, lg));
            }
    }

    // Closes a level; a wide one: which of the three kernels can take it.
    void level(int mode, size_t first, Shape how, int depth) {
        auto& list = tasks[mode];
        const int n = (int)(list.size() - first);
        if (how.wide != 0 && split.empty()) {
            bool products = true, plain = true;
            for (size_t i = first; i < list.size(); ++i) {
                const PcxColTask& t = list[i];
                products = products && t.kind == K_PROD;
                plain = plain && t.kind == K_MMA && t.n_k * t.width <= 32 && t.n_kids <= 2;
                for (int q = 0; plain && q < t.n_rows; ++q) plain = strips[mode].data[4 * ((size_t)t.strip_off + q) + 3] < 2;
            }
            how.wide = products ? 3 : (plain ? 2 : 1);
        }
        list.insert(list.end(), split.begin(), split.end());
        levels[mode].push_back(Level{(int)first, n, (int)first + n, (int)split.size(), how, depth});
        split.clear();
    }

    // Sections: fragments, then per direction tasks, strips, levels; then per direction two lists of launches, the second (by tasks
    // alone) only where it differs (-1: it does not).  A launch: (0, first level, levels, shape) or, a product launch, (1, node
    // rows, child rows, how many, children, block size) or, a chain, (3, rows, strips, levels, strips per level, nt, strips per CTA).
    void run(Blob& blob) {
        int64_t total = 0, n_small = 0;
        for (auto& d : pc.depths)
            if (!is_wide(count(d.fw))) { total += count(d.fw); ++n_small; }
        const double items = n_small ? (double)total / (double)n_small : 1.0;
        fused = pc.big_steps ? pc.big_shape(W, room) : PcxColPlanner::small_shape(W, items, room);
        std::vector<char> before(pc.depths.size(), 0);      // levels with product launches ahead of them
        for (size_t i = 0; i < pc.depths.size(); ++i) {
            const Depth& d = pc.depths[i];
            const size_t first = tasks[0].size();
            const int64_t n = count(d.fw);
            // Elements of many children in a level that has the machine to itself: their values come from the product
            // kernel, whose 2048 threads per SM hide the latency of the gather better than the warp tasks (16384 elements
            // of 24 children, 1024 samples: 155 + 25 us instead of 320).  A CTA of a fused level gathers some 500 child rows
            // in a microsecond: from several microseconds' worth of rows the kernel's launch is the smaller cost.
            int64_t reads = 0;
            for (auto& e : d.elems) reads += (int64_t)e.size * e.n;
            const bool stored = d.stored && (is_wide(n) || reads > prod_reads * fused.cluster);
            before[i] = stored;
            const int per = strips_per_task(n);
            for (auto& g : d.fw) {
                if (g.big) cta_tasks(d, g, 0, PcxColPlanner::piece(d.fw, fused.nt, fused.cluster).first);
                else if (g.mma) mma_tasks(d, g, 0, stored, per);
                else simt_forward(d, g, stored);
            }
            level(0, first, shape(n), (int)i);
        }
        for (size_t i = pc.depths.size(); i-- > 0;) {
            const Depth& d = pc.depths[i];
            size_t first = tasks[1].size();
            const int64_t n = count(d.bk);
            const int per = strips_per_task(n);
            for (auto& g : d.bk) {
                if (g.big) cta_tasks(d, g, 1, PcxColPlanner::piece(d.bk, fused.nt, fused.cluster).first);
                else if (g.mma) mma_tasks(d, g, 1, false, per);
                else simt_backward(d, g);
            }
            level(1, first, shape(n), (int)i);
            if (d.direct) continue;
            first = tasks[1].size();
            for (auto& p : d.prod_bk)
                for (int r = 0; r < p.size; r += 16) {
                    rows.assign(d.parents.begin() + p.first, d.parents.begin() + p.first + p.n);
                    for (int& x : rows) x += r;
                    tasks[1].push_back(task(p.n ? kids.add(rows) : 0, p.n, 0, 1, p.row + r, std::min(16, p.size - r), 0, K_PROD, p.add));
                }
            level(1, first, shape((int64_t)(tasks[1].size() - first)), -1);
        }
        auto& m = blob.meta;
        size_t chain_words = 0;
        for (auto& c : pc.chains) chain_words += c.rows[0].size() + c.rows[1].size();
        blob.data.reserve(frag.size() + kids.data.size() + 12 * (tasks[0].size() + tasks[1].size()) + strips[0].data.size() +
                          strips[1].data.size() + chain_words + 8192);
        m = {(int64_t)frag.size() / 4, blob.section(frag), blob.section(kids.data), (int64_t)kids.data.size()};
        for (int mode = 0; mode < 2; ++mode) {
            static_assert(sizeof(PcxColTask) == 48, "task records are twelve words");
            m.push_back(blob.section(reinterpret_cast<const int32_t*>(tasks[mode].data()), tasks[mode].size() * 12));
            m.push_back((int64_t)tasks[mode].size());
            m.push_back(blob.section(strips[mode].data));
            m.push_back((int64_t)strips[mode].data.size());
            Ints lv;
            for (auto& l : levels[mode]) lv.insert(lv.end(), {l.first, l.n, l.split_first, l.n_split});
            m.push_back(blob.section(lv));
            m.push_back((int64_t)levels[mode].size());
        }
        // With chains in the places of their levels; then, where there is a chain, by tasks alone.  What goes with a level is made
        // once for both.
        for (int mode = 0; mode < 2; ++mode) {
            const size_t n_levels = levels[mode].size();
            std::vector<const PcxColPlanner::Chain*> chain(n_levels);
            bool any = false;
            for (size_t at = 0; at < n_levels; ++at) any = (chain[at] = starts(mode, at)) != nullptr || any;
            std::vector<std::pair<int64_t, std::vector<int64_t>>> ahead(n_levels), staged(n_levels);    // launch records, how many
            for (int chained = 1; chained >= 0; --chained) {
                if (!chained && !any) {
                    m.push_back(-1);
                    break;
                }
                std::vector<int64_t> launches;
                int64_t n = 0;
                auto add = [&](const std::pair<int64_t, std::vector<int64_t>>& records) {
                    n += records.first;
                    launches.insert(launches.end(), records.second.begin(), records.second.end());
                };
                for (size_t at = 0, end; at < n_levels; at = end, ++n) {            // consecutive fused levels are one launch
                    const Shape how = levels[mode][at].how;
                    const size_t last = std::min(n_levels, at + PCX_COLUMN_MAX_LEVELS);
                    if (const auto* c = chained ? chain[at] : nullptr) {
                        const auto shape = PcxColPlanner::chain_shape(W, c->strips, room);
                        launches.insert(launches.end(), {3, blob.section(c->rows[mode]), blob.section(chain_strips(mode, at)),
                                                         c->n, c->strips, shape.nt, shape.per});
                        end = at + c->n;
                        continue;
                    }
                    for (end = at + 1; how.wide == 0 && end < last && levels[mode][end].how.wide == 0 && !(mode == 0 && before[end]) &&
                                       !(chained && chain[end]); ++end) {}
                    if (mode == 0 && before[at]) {
                        if (ahead[at].first == 0) ahead[at].first = products(pc.depths[at], blob, ahead[at].second);
                        add(ahead[at]);
                    }
                    launches.insert(launches.end(), {0, (int64_t)at, (int64_t)(end - at), how.nt, how.tiles, how.cluster, how.wide});
                    if (how.wide == 3) {
                        if (staged[at].first == 0)
                            staged[at].first = product_flows(pc.depths[levels[mode][at - 1].depth], blob, staged[at].second);
                        add(staged[at]);
                    }
                }
                m.push_back(n);
                m.insert(m.end(), launches.begin(), launches.end());
            }
        }
    }
    // The chain whose first level is `at`, if its clusters fit at once.  Where they do not, the tasks, which take more columns in
    // fewer CTAs, are about as fast (1024 states, 256 columns, 31 levels forward and back: 445 + 576 us by tasks, 512 + 556 in
    // two waves of 24 columns x 4 strips, which the estimate prefers; three of 16 x 4 take 453 + 488).  Where they do, the chain
    // is faster throughout (1024 states, 192 columns: 385 + 570 by tasks, 365 + 391; 512, 512: 268 + 370, 177 + 201).
    const PcxColPlanner::Chain* starts(int mode, size_t at) const {
        for (auto& c : pc.chains)
            if (levels[mode][at].depth == (mode == 0 ? c.first : c.first + c.n - 1)) {
                for (size_t l = at; l < at + c.n; ++l)
                    if (levels[mode][l].how.wide != 0) return nullptr;
                return PcxColPlanner::chain_shape(W, c.strips, room).waves == 1 ? &c : nullptr;
            }
        return nullptr;
    }
    // First fragment and fragments per step of every strip of a level's group.
    Ints chain_strips(int mode, size_t at) const {
        const Level& l = levels[mode][at];
        Ints t;
        for (int i = l.first; i < l.split_first + l.n_split; ++i) {
            const PcxColTask& k = tasks[mode][i];
            for (int r = 0; r < k.n_rows; ++r) t.insert(t.end(), {k.par_off + r, k.n_rows});
        }
        return t;
    }
    // Arguments of the product kernel that fills the stored values of a depth, one set per block size.
    int64_t products(const Depth& d, Blob& blob, std::vector<int64_t>& launches) const {
        int64_t made = 0;
        Ints sizes;
        for (auto& e : d.elems)
            if (std::find(sizes.begin(), sizes.end(), e.size) == sizes.end()) sizes.push_back(e.size);
        for (size_t q = 0; q < sizes.size(); ++q) {
            int n = 0;
            for (auto& e : d.elems)
                if (e.size == sizes[q]) n = std::max(n, e.n);
            Ints rows, cids;
            for (auto& e : d.elems)
                if (e.size == sizes[q]) {
                    rows.push_back(e.store);
                    for (int c = 0; c < n; ++c) cids.push_back(c < e.n ? d.kids[e.first + c] : 0);
                }
            launches.insert(launches.end(), {q == 0 ? 1 : 2, blob.section(rows), blob.section(cids), (int64_t)rows.size(), n, sizes[q], 0});
            std::vector<Item> readers;
            for (auto& e : d.elems)
                if (e.size == sizes[q]) readers.push_back({e.store, 0, d.kids.data() + e.first, e.n});
            made += 1 + staged(readers, sizes[q], blob, launches);
        }
        return made;
    }
    // The flows of a product level, if all of it can be staged.
    int64_t product_flows(const Depth& d, Blob& blob, std::vector<int64_t>& launches) const {
        std::vector<Item> readers;
        for (auto& p : d.prod_bk) {
            if (p.size != d.prod_bk[0].size) return 0;
            readers.push_back({p.row, p.add, d.parents.data() + p.first, p.n});
        }
        return readers.empty() ? 0 : staged(readers, d.prod_bk[0].size, blob, launches);
    }

    // Tables of `pcx_prod_staged` for the rows of one block size, as a launch record that replaces the one before it: (4, sources,
    // how many, items, how many, chunks of their lists behind them, block size).
    struct Item { int row, add; const int32_t* from; int n; };
    int64_t staged(std::vector<Item>& readers, int size, Blob& blob, std::vector<int64_t>& launches) const {
        if (W < PCX_STAGED_COLUMNS || (int64_t)size * cdiv(W, PCX_STAGED_COLUMNS) < STAGED_CTAS) return 0;
        int lo = INT32_MAX, hi = -1;
        for (auto& r : readers)
            for (int k = 0; k < r.n; ++k) { lo = std::min(lo, r.from[k]); hi = std::max(hi, r.from[k]); }
        if (hi < lo) return 0;
        Ints sources, items, place((size_t)(hi - lo) + 1, -1);
        int64_t reads = 0;
        for (auto& r : readers) {
            reads += r.n;
            for (int k = 0; k < r.n; ++k)
                if (place[r.from[k] - lo] < 0) {
                    place[r.from[k] - lo] = (int)sources.size();
                    sources.push_back(r.from[k]);
                }
            if (sources.size() > PCX_STAGED_SOURCES) return 0;
        }
        if (reads < STAGED_READS * (int64_t)sources.size()) return 0;
        std::stable_sort(readers.begin(), readers.end(), [](const Item& x, const Item& y) { return x.n > y.n; });
        std::vector<uint16_t> words;
        for (auto& r : readers) {
            items.insert(items.end(), {r.row, (int)(words.size() / 8), r.n, r.add});
            for (int k = 0; k < r.n; ++k) words.push_back((uint16_t)place[r.from[k] - lo]);
            while (words.size() % 8 != 0) words.push_back((uint16_t)sources.size());
        }
        items.resize(items.size() + words.size() / 2);       // (the lists, behind the items)
        std::memcpy(items.data() + items.size() - words.size() / 2, words.data(), words.size() * 2);
        launches.insert(launches.end(), {4, blob.section(sources), (int64_t)sources.size(), blob.section(items), (int64_t)readers.size(),
                                         (int64_t)words.size() / 8, size});
        return 1;
    }
    // A staged source is copied once and read from shared memory: below STAGED_READS readers a source, or with fewer CTAs than
    // SMs, the general kernels stay.
    static constexpr int64_t STAGED_READS = 4, STAGED_CTAS = 148;
};

// ---- parameter-flow jobs (no row width in them) --------------------------------------------------------------------------
struct Jobs {
    const PcxColPlanner& pc;
    Pool pp{2}, kids{1};
    std::vector<PcxColPar> jobs[4];
    Ints ent, tab;                              // scratch

    explicit Jobs(const PcxColPlanner& p) : pc(p) {}

    struct Step { int op, o; };
    int entries(const Depth& d, const Group& g, const std::vector<Step>& steps, size_t k0, size_t k1, int nk) {
        ent.clear();
        for (size_t k = k0; k < k1; ++k) {
            const Elem* e = d.find(g.ops[steps[k].op]);
            if (d.stored) ent.push_back(e->store + steps[k].o);
            else
                for (int c = 0; c < nk; ++c) ent.push_back(c < e->n ? d.kids[e->first + c] + steps[k].o : 0);
        }
        return kids.add(ent);
    }
    static PcxColPar job(const int32_t* row, int n_strips, int kid_off, int n_k, int n_kids, int width, int pp_off, int bs, int lg) {
        PcxColPar j{};
        j.row0 = row[0]; j.row1 = row[1]; j.row2 = row[2]; j.row3 = row[3];
        j.n_strips = n_strips; j.kid_off = kid_off; j.n_k = n_k; j.n_kids = n_kids; j.width = width; j.pp_off = pp_off;
        j.bs = bs; j.lg_entry = lg;
        return j;
    }
    void group(const Depth& d, const Group& g) {
        const int nk = Cutter::children(d, g), width = d.stored ? 1 : nk, n_kids = d.stored ? -1 : nk, n_ops = (int)g.ops.size();
        int lg = 3;
        for (int e : g.ops)
            if (d.find(e)->size % 8 != 0) lg = 0;
        std::vector<Step> steps;
        for (int q = 0; q < n_ops; ++q)
            for (int o = 0; o < d.find(g.ops[q])->size; o += g.mma ? 16 : 1 << lg) steps.push_back({q, o});
        if (g.mma) {
            // tiles of 64 x 64 where the group has them, of 32 x 32 otherwise
            const size_t per_block = g.bs / 16, n_strips = g.blocks.size() * per_block;
            const int kind = n_kids > 2 ? 0 : (steps.size() > 2 && n_strips > 2 ? 3 : 2);
            const size_t most = kind == 3 ? 4 : 2;
            for (size_t k0 = 0; k0 < steps.size(); k0 += most) {
                const size_t k1 = std::min(steps.size(), k0 + most);
                const int off = entries(d, g, steps, k0, k1, nk);
                for (size_t s0 = 0; s0 < n_strips; s0 += most) {
                    const size_t s1 = std::min(n_strips, s0 + most);
                    tab.clear();
                    for (size_t k = k0; k < k1; ++k)
                        for (size_t s = s0; s < s1; ++s)
                            for (const Ints* src : {&g.par, &g.flow})
                                tab.push_back((*src)[s / per_block * n_ops + steps[k].op] + steps[k].o * g.bs + (int)(s % per_block) * 16);
                    int32_t row[4];
                    for (size_t s = 0; s < 4; ++s) {
                        const size_t t = std::min(s0 + s, s1 - 1);
                        row[s] = g.blocks[t / per_block] + (int)(t % per_block) * 16;
                    }
                    jobs[kind].push_back(job(row, (int)(s1 - s0), off, (int)(k1 - k0), n_kids, width, pp.add(tab), g.bs, 0));
                }
            }
            return;
        }
        const size_t per = 64 >> lg;
        for (size_t k0 = 0; k0 < steps.size(); k0 += per) {
            const size_t k1 = std::min(steps.size(), k0 + per);
            const int off = entries(d, g, steps, k0, k1, nk);
            for (size_t b = 0; b < g.blocks.size(); ++b)
                for (int r = 0; r < g.bs; r += 16) {
                    tab.clear();
                    for (size_t k = k0; k < k1; ++k)
                        for (const Ints* src : {&g.par, &g.flow}) tab.push_back((*src)[b * n_ops + steps[k].op] + steps[k].o * g.bs + r);
                    const int32_t row[4] = {g.blocks[b] + r, 0, 0, 0};
                    jobs[1].push_back(job(row, std::min(16, g.bs - r), off, (int)(k1 - k0) << lg, n_kids, width, pp.add(tab), g.bs, lg));
                }
        }
    }
    // `dense`: which groups of tied tables go through a dense product instead.  Sections: offsets, operands, jobs per kind.
    void run(const uint8_t* dense, Blob& blob) {
        for (auto& d : pc.depths)
            for (auto& g : d.fw)
                if (g.tied < 0 || !dense[g.tied]) group(d, g);
        blob.meta = {blob.section(pp.data), (int64_t)pp.data.size(), blob.section(kids.data), (int64_t)kids.data.size()};
        for (auto& list : jobs) {
            static_assert(sizeof(PcxColPar) == 48, "job records are twelve words");
            blob.meta.push_back(blob.section(reinterpret_cast<const int32_t*>(list.data()), list.size() * 12));
            blob.meta.push_back((int64_t)list.size());
        }
    }
};

// Runs `fn`; no exception crosses the C boundary.  1: the circuit has a table the program does not cover; -1: an error.
template <typename F>
int guarded(char* why, int why_len, F fn) {
    std::string text;
    int rc = 0;
    try {
        fn();
    } catch (const Unsupported& e) {
        text = e.what();
        rc = 1;
    } catch (const std::exception& e) {
        text = e.what();
        rc = -1;
    } catch (...) {
        text = "unknown exception";
        rc = -1;
    }
    if (why && why_len > 0) {
        std::strncpy(why, text.c_str(), (size_t)why_len - 1);
        why[why_len - 1] = 0;
    }
    return rc;
}

}  // namespace

extern "C" {

int pcx_colplan_new(const int64_t* desc, int64_t n_desc, const int32_t* tables, int64_t n_tables, void** out, char* why, int why_len) {
    *out = nullptr;
    return guarded(why, why_len, [&] {
        auto p = std::make_unique<PcxColPlanner>();
        Reader in{desc, desc + n_desc, tables, n_tables};
        p->build(in);
        p->find_tied();
        p->find_chains();
        *out = p.release();
    });
}
int pcx_colplan_free(void* planner) {
    delete static_cast<PcxColPlanner*>(planner);
    return 0;
}
int pcx_colplan_info(const void* planner, int* em_rows, int* big_steps, int* n_chains) {
    const auto* p = static_cast<const PcxColPlanner*>(planner);
    *em_rows = p->em_rows;
    *big_steps = p->big_steps;
    *n_chains = (int)p->chains.size();
    return 0;
}
int pcx_colplan_suits(const void* planner, int64_t W, const int32_t* rooms) {
    return static_cast<const PcxColPlanner*>(planner)->suits(W, PcxColPlanner::Room{rooms});
}
int pcx_colplan_cut(const void* planner, int64_t W, const int32_t* rooms, int64_t wide_items, int64_t prod_reads, void** blob, char* why,
                    int why_len) {
    *blob = nullptr;
    return guarded(why, why_len, [&] {
        auto b = std::make_unique<Blob>();
        Cutter(*static_cast<const PcxColPlanner*>(planner), W, rooms, wide_items, prod_reads).run(*b);
        *blob = b.release();
    });
}
int pcx_colplan_tied(const void* planner, void** blob, char* why, int why_len) {
    *blob = nullptr;
    return guarded(why, why_len, [&] {
        auto b = std::make_unique<Blob>();
        static_cast<const PcxColPlanner*>(planner)->tied_tables(*b);
        *blob = b.release();
    });
}
int pcx_colplan_jobs(const void* planner, const uint8_t* dense, void** blob, char* why, int why_len) {
    *blob = nullptr;
    return guarded(why, why_len, [&] {
        auto b = std::make_unique<Blob>();
        Jobs(*static_cast<const PcxColPlanner*>(planner)).run(dense, *b);
        *blob = b.release();
    });
}
int pcx_colplan_blob(const void* blob, const int32_t** data, int64_t* n_data, const int64_t** meta, int64_t* n_meta) {
    const auto* b = static_cast<const Blob*>(blob);
    *data = b->data.data();
    *n_data = (int64_t)b->data.size();
    *meta = b->meta.data();
    *n_meta = (int64_t)b->meta.size();
    return 0;
}
int pcx_colplan_blob_free(void* blob) {
    delete static_cast<Blob*>(blob);
    return 0;
}

}  // extern "C"
