// The column program: all levels of a circuit in one launch, one thread-block cluster per group of batch columns.
//
// Samples are independent of one another, so the columns of the value buffers never exchange data.  A circuit of small
// node blocks (up to 64 nodes) is a hundred dependent levels of little work each; with a launch per level the step is
// launch boundaries and half-empty grids (a 784-variable tree with 32 latents and one sample: 114 kernels of 2 - 7 us).
// Here a cluster of C CTAs owns 8 * NT columns and walks ALL levels; what separates two levels is a cluster barrier (a
// __syncthreads when C = 1) instead of a kernel boundary, and clusters never wait for one another.
//
// The unit of work is a warp task: the rows that share one list of children, for the cluster's columns.  Nothing is
// staged in shared memory and warps never wait for each other inside a level.
//
//   MMA task   node blocks of 32 and more.  mma.sync m16n8k16: the parameters (16 rows x 16 children, bf16 hi / lo,
//              packed once per parameter update in the order of the instruction's A fragment, so a lane reads two 16-byte
//              words) times the exponentials.  The B fragment of a lane is the children 2t, 2t+1, 2t+8, 2t+9 of ONE
//              column, so the lane gathers exactly those values from the children's rows (32-byte sectors), takes the
//              column maximum with two shuffles, exponentiates and splits them in registers.  tcgen05 would want 128-row
//              tiles in shared memory and a round trip through tensor memory per 32-row block; these tasks are bound by
//              the gather and the exponentials around the multiplication, not by the multiplication.
//   SIMT task  blocks under 32 nodes (fp32 FMA throughout, as accurate as the tiled fp32 kernels): a lane owns a column
//              and some rows; every exponential is formed once per lane group.
//
// Tables longer than a chunk (64 children MMA, 8 SIMT) carry a running maximum.  Products are folded in: an element's
// value is the sum of its children's rows; where an element has many children its value is also stored for the backward
// pass.  Row 0 .. of node_mars (dummy rows) are zero, so absent children need no branch.
//
// Backward: element flows by the same tasks on the transposed tables (operand flow - value of the parents), stored
// straight into the children's flow rows where every child has one parent product, else into element_flows, followed
// by a level of product tasks (log-sum-exp over a node's parent products).  The first level that touches a row writes
// it, so the flow buffer needs no reset.
//
// Parameter flows of all levels are one more launch over all (row group, children) tiles; contraction over the batch.
#include <algorithm>
#include "pcx_common.cuh"
#include "pcx_column_ops.cuh"
#include "../../include/pcx_b200.h"

namespace {

constexpr int CT = 512;                     // threads per CTA (16 warps, 128 registers each)
constexpr int CW = CT / 32;
constexpr int MAX_LEVELS = PCX_COLUMN_MAX_LEVELS;          // of one launch: the level table sits in shared memory
constexpr int WT = 384;                     // of the wide launches: 12 warps, 168 registers each
constexpr int MAX_STRIPS = 2;               // 16-row strips an MMA task may hold (accumulators and element values)
enum ColKind { K_MMA = 0, K_SIMT = 1, K_SPLIT = 2, K_PROD = 3, K_CTA = 4 };

struct ColArgs {
    float* nm;                  // node_mars  [rows, W]
    float* nf;                  // node_flows (ELE)
    float* ef;                  // element_flows (ELE, products with several users)
    float* em;                  // stored element values (elements of many children)
    const float* params;
    const uint4* frags;         // packed parameter fragments
    const PcxColTask* tasks;
    const int32_t* kids;        // operand table
    const int4* strips;         // output table
    const int4* levels;         // [n_levels] (first warp task, how many, first split task, how many)
    int n_levels;
    int W;
    int logspace;
    int terms;
    int cluster;                // CTAs per cluster
    int tiles;                  // column tiles of 32 (wide launches)
    int wide;                   // one level, spread over the whole grid
};

// ---- task records and operand tables -------------------------------------------------------------------------------
// A record is held one word per lane, and so are the first 32 entries of the task's operand table, so that the records
// of the next two tasks and the entries of the next one cost a warp three registers while they are under way: with
// them, a task begins with its first operand loads.
__device__ __forceinline__ int fetch_record(const PcxColTask* tasks, int i) {
    const int lane = threadIdx.x & 31;
    return lane < (int)(sizeof(PcxColTask) / 4) ? __ldg(reinterpret_cast<const int*>(tasks + i) + lane) : 0;
}
__device__ __forceinline__ int fetch_kids(const ColArgs& a, int rec) {
    const int off = __shfl_sync(0xffffffffu, rec, 0);
    const int n = __shfl_sync(0xffffffffu, rec, 1) * __shfl_sync(0xffffffffu, rec, 3);
    const int lane = threadIdx.x & 31;
    return lane < n ? __ldg(a.kids + off + lane) : 0;
}
// The kernels that keep their operands in registers read records and tables through L1 where they need them (a word per
// lane and a shuffle per use costs them more than the L1's latency: 224 against 173 us for 53 levels of 16 tasks), after
// touching the lines a task ahead.
__device__ __forceinline__ PcxColTask load_record(const PcxColTask* tasks, int i) {
    PcxColTask t;
    const int4* src = reinterpret_cast<const int4*>(tasks + i);
    const int4 x = __ldg(src), y = __ldg(src + 1), z = __ldg(src + 2);
    t.kid_off = x.x; t.n_k = x.y; t.n_kids = x.z; t.width = x.w;
    t.strip_off = y.x; t.n_rows = y.y; t.par_off = y.z; t.kind = y.w;
    t.sk = z.x; t.sr = z.y; t.lg_entry = z.z; t.pad = 0;
    return t;
}
__device__ __forceinline__ void touch(const void* p) {
    int x;
    asm volatile("ld.global.nc.b32 %0, [%1];" : "=r"(x) : "l"(p));
}

// ---- MMA task ------------------------------------------------------------------------------------------------------
// Column of lane (g, t) and tile j: NT * g + j, so that a lane's values of all tiles are one vector load; accumulator
// register c of tile j is then column NT * (2t + (c & 1)) + j, and a lane's 2 * NT columns of a row are contiguous.
//
// A warp's time is memory latency, so every phase requests all it needs before it uses any of it: the child rows of a
// chunk (two children together, four where a chunk is two steps), and in the backward pass the element values of the
// next strip while one is finished.
template <int NT>
struct ElementValue { float x[2][2 * NT]; };               // two children

template <int NT>
__device__ __forceinline__ void load_element(const ColArgs& a, const int4& st, int row, int co, ElementValue<NT>& e) {
    if (st.w < 2) {                                         // stored value, or up to two child rows
        const float* src = st.w < 0 ? a.em : a.nm;
        ldvec<2 * NT>(src + (int64_t)(st.y + row) * a.W + co, e.x[0]);
        if (st.w >= 0) ldvec<2 * NT>(a.nm + (int64_t)(st.z + row) * a.W + co, e.x[1]);
        else
#pragma unroll
            for (int j = 0; j < 2 * NT; ++j) e.x[1][j] = 0.0f;
        return;
    }
#pragma unroll
    for (int j = 0; j < 2 * NT; ++j) { e.x[0][j] = 0.0f; e.x[1][j] = 0.0f; }
    for (int c = 0; c < st.z; c += 2) {
        const bool two = c + 1 < st.z;
        float x[2 * NT], y[2 * NT];
        ldvec<2 * NT>(a.nm + (int64_t)(__ldg(a.kids + st.y + c) + row) * a.W + co, x);
        ldvec<2 * NT>(a.nm + (int64_t)(two ? __ldg(a.kids + st.y + c + 1) + row : 0) * a.W + co, y);
#pragma unroll
        for (int j = 0; j < 2 * NT; ++j) { e.x[0][j] += x[j]; e.x[1][j] += two ? y[j] : 0.0f; }
    }
}

// Flow of an element row: into element_flows, or into its children's rows when it is their only user.
template <int N>
__device__ __forceinline__ void store_flow(const ColArgs& a, const int4& st, int row, int co, const float* o) {
    if (st.w == 1) {
        stvec<N>(a.nf + (int64_t)(st.y + row) * a.W + co, o);
        if (st.z != 0) stvec<N>(a.nf + (int64_t)(st.z + row) * a.W + co, o);
    } else if (st.w == 3) {
        for (int c = 0; c < st.z; ++c) stvec<N>(a.nf + (int64_t)(__ldg(a.kids + st.y + c) + row) * a.W + co, o);
    } else {
        stvec<N>(a.ef + (int64_t)(st.x + row) * a.W + co, o);
    }
}

template <int MODE, int NT, int KC>
__device__ void mma_task(const ColArgs& a, const PcxColTask& t, int col0) {
    const int lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
    const int W = a.W;
    const int cl = (col0 + NT * g < W) ? col0 + NT * g : 0;
    const int co = col0 + 2 * NT * tq;
    const bool co_ok = co < W;
    float m[NT];
    float acc[MAX_STRIPS][NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j) m[j] = PCX_NEG_INF;
#pragma unroll
    for (int s = 0; s < MAX_STRIPS; ++s)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[s][j][c] = 0.0f;

    const int width = t.width;                      // operand table entries per 16-deep step
    const int32_t* kid = a.kids + t.kid_off;
    ElementValue<NT> ev[2 * MAX_STRIPS];            // element values of eight rows each: strip, half
    int4 st[MAX_STRIPS];
#pragma unroll
    for (int s = 0; s < MAX_STRIPS; ++s) st[s] = __ldg(a.strips + t.strip_off + (s < t.n_rows ? s : 0));
    for (int k0 = 0; k0 < t.n_k; k0 += KC) {
        float v[KC][4][NT];
        const int live = min(KC, t.n_k - k0);
        if (MODE == C_FWD) {
            if (t.n_kids < 0) {                     // values stored by a product kernel
#pragma unroll
                for (int q = 0; q < KC; ++q) {
                    const int r = q < live ? __ldg(kid + k0 + q) : 0;
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        ldvec<NT>(a.em + (int64_t)(r + 2 * tq + (i & 1) + (i >> 1) * 8) * W + cl, v[q][i]);
                }
            } else if (width == 2) {                // two children (the second may be absent: zeros)
#pragma unroll
                for (int q = 0; q < KC; ++q) {
                    const int rx = q < live ? __ldg(kid + 2 * (k0 + q)) : 0;
                    const int ry = q < live ? __ldg(kid + 2 * (k0 + q) + 1) : 0;
                    float y[4][NT];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int o = 2 * tq + (i & 1) + (i >> 1) * 8;
                        ldvec<NT>(a.nm + (int64_t)(rx + o) * W + cl, v[q][i]);
                        ldvec<NT>(a.nm + (int64_t)(ry + o) * W + cl, y[i]);
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int j = 0; j < NT; ++j) v[q][i][j] += y[i][j];
                }
            } else {
                constexpr int KU = (NT == 4 || KC == 4) ? 2 : 4;
#pragma unroll
                for (int q = 0; q < KC; ++q)
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int j = 0; j < NT; ++j) v[q][i][j] = 0.0f;
                for (int c = 0; c < t.n_kids; c += KU) {
                    float x[KU][KC][4][NT];
#pragma unroll
                    for (int u = 0; u < KU; ++u)
#pragma unroll
                        for (int q = 0; q < KC; ++q) {
                            const int r = (q < live && c + u < t.n_kids) ? __ldg(kid + (k0 + q) * width + c + u) : 0;
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                ldvec<NT>(a.nm + (int64_t)(r + 2 * tq + (i & 1) + (i >> 1) * 8) * W + cl, x[u][q][i]);
                        }
#pragma unroll
                    for (int u = 0; u < KU; ++u)
#pragma unroll
                        for (int q = 0; q < KC; ++q)
#pragma unroll
                            for (int i = 0; i < 4; ++i)
#pragma unroll
                                for (int j = 0; j < NT; ++j) v[q][i][j] += c + u < t.n_kids ? x[u][q][i][j] : 0.0f;
                }
                if (width > t.n_kids) {             // elements of many children: keep their values for the backward pass
#pragma unroll
                    for (int q = 0; q < KC; ++q) {
                        if (q < live) {
                            const int r = __ldg(kid + (k0 + q) * width + t.n_kids);
                            if (col0 + NT * g < W)
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                stvec<NT>(a.em + (int64_t)(r + 2 * tq + (i & 1) + (i >> 1) * 8) * W + cl, v[q][i]);
                        }
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < KC; ++q)
                if (q >= live)
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int j = 0; j < NT; ++j) v[q][i][j] = PCX_NEG_INF;
        } else {
            float y[KC][4][NT];
#pragma unroll
            for (int q = 0; q < KC; ++q) {
                const int r = q < live ? __ldg(kid + k0 + q) : 0;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int64_t at = (int64_t)(r + 2 * tq + (i & 1) + (i >> 1) * 8) * W + cl;
                    ldvec<NT>(a.nf + at, v[q][i]);
                    ldvec<NT>(a.nm + at, y[q][i]);
                }
            }
            if (k0 + KC >= t.n_k) {                 // the element values are on their way by the time the flows are formed
                if (co_ok) load_element<NT>(a, st[0], g, co, ev[0]);
            }
#pragma unroll
            for (int q = 0; q < KC; ++q)
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < NT; ++j)
                        v[q][i][j] = q < live ? flow_over_value(v[q][i][j], y[q][i][j], a.logspace) : PCX_NEG_INF;
        }
        float sc[NT];
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            float mx = m[j];
#pragma unroll
            for (int q = 0; q < KC; ++q)
#pragma unroll
                for (int i = 0; i < 4; ++i) mx = fmaxf(mx, v[q][i][j]);
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            sc[j] = (m[j] == PCX_NEG_INF) ? 0.0f : fast_exp(m[j] - mx);
            m[j] = mx;
        }
        if (k0 > 0) {                               // accumulators follow the new maximum of their columns
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                const float s0 = __shfl_sync(0xffffffffu, sc[j], 8 * tq), s1 = __shfl_sync(0xffffffffu, sc[j], 8 * tq + 4);
#pragma unroll
                for (int s = 0; s < MAX_STRIPS; ++s) {
                    acc[s][j][0] *= s0; acc[s][j][1] *= s1; acc[s][j][2] *= s0; acc[s][j][3] *= s1;
                }
            }
        }
        uint32_t bh[KC][NT][2], bl[KC][NT][2];
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            const float sh = (m[j] == PCX_NEG_INF) ? 0.0f : m[j];
#pragma unroll
            for (int q = 0; q < KC; ++q) {
                float e[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) e[i] = fast_exp(v[q][i][j] - sh);     // exp(-inf) = 0
                split2(e[0], e[1], bh[q][j][0], bl[q][j][0]);
                split2(e[2], e[3], bh[q][j][1], bl[q][j][1]);
            }
        }
        if (MODE == C_ELE && k0 + KC >= t.n_k && co_ok) {
#pragma unroll
            for (int i = 1; i < 2 * MAX_STRIPS; ++i)
                if ((i >> 1) < t.n_rows) load_element<NT>(a, st[i >> 1], g + 8 * (i & 1), co, ev[i]);
        }
        const uint4* fr = a.frags + ((int64_t)t.par_off + (int64_t)k0 * t.n_rows) * 64 + lane;
#pragma unroll
        for (int q = 0; q < KC; ++q) {
            if (q < live) {
#pragma unroll
                for (int s = 0; s < MAX_STRIPS; ++s) {
                    if (s < t.n_rows) {
                        const uint4 ah = __ldg(fr + (q * t.n_rows + s) * 64), al = __ldg(fr + (q * t.n_rows + s) * 64 + 32);
#pragma unroll
                        for (int j = 0; j < NT; ++j) {
                            mma16816(acc[s][j], ah, bh[q][j][0], bh[q][j][1]);
                            if (a.terms == 3) {
                                mma16816(acc[s][j], ah, bl[q][j][0], bl[q][j][1]);
                                mma16816(acc[s][j], al, bh[q][j][0], bh[q][j][1]);
                            }
                        }
                    }
                }
            }
        }
    }
    float m0[NT], m1[NT];
#pragma unroll
    for (int j = 0; j < NT; ++j) {
        m0[j] = __shfl_sync(0xffffffffu, m[j], 8 * tq);
        m1[j] = __shfl_sync(0xffffffffu, m[j], 8 * tq + 4);
    }
    if (!co_ok) return;
#pragma unroll
    for (int s = 0; s < MAX_STRIPS; ++s) {
        if (s >= t.n_rows) break;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int row = g + 8 * h;
            float o[2 * NT];
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                const float x0 = acc[s][j][2 * h], x1 = acc[s][j][2 * h + 1];
                // (an empty sum has the shift -inf, which stands for the result; no term is ever +inf)
                o[j] = fast_log_plus(MODE == C_FWD ? fmaxf(x0, 1e-24f) : x0, m0[j]);
                o[NT + j] = fast_log_plus(MODE == C_FWD ? fmaxf(x1, 1e-24f) : x1, m1[j]);
            }
            if (MODE == C_FWD) {
                stvec<2 * NT>(a.nm + (int64_t)(st[s].x + row) * W + co, o);
                continue;
            }
#pragma unroll
            for (int j = 0; j < 2 * NT; ++j) {
                o[j] += ev[2 * s + h].x[0][j] + ev[2 * s + h].x[1][j];
                if (!a.logspace) o[j] = __expf(o[j]);
            }
            store_flow<2 * NT>(a, st[s], row, co, o);
        }
    }
}

// ---- SIMT task -----------------------------------------------------------------------------------------------------
// A warp is 8 * NT columns x G = 4 / NT lane groups; the groups share the rows, and where there are fewer rows than
// groups, the contraction.  OCT: eight consecutive children are one entry of the operand table (parameter offset, child
// rows, place of the stored element value); otherwise every child has its own.
template <int MODE, int NT, int RL, bool OCT>
__device__ __forceinline__ void simt_partial(const ColArgs& a, const PcxColTask& t, int cl, bool col_ok, int row0, int ck0,
                                             int ck_step, float& m, float* acc) {
    m = PCX_NEG_INF;
#pragma unroll
    for (int r = 0; r < RL; ++r) acc[r] = 0.0f;
    const int n_chunks = (t.n_k + 7) >> 3;
    for (int ck = ck0; ck < n_chunks; ck += ck_step) {
        float v[8];
        int pid[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int k = ck * 8 + i;
            const bool in = OCT || k < t.n_k;
            const int32_t* ent = a.kids + t.kid_off + (OCT ? ck : (in ? k : 0)) * t.width;
            const int off = OCT ? i : 0;
            pid[i] = __ldg(ent) + off * t.sk;
            if (MODE == C_ELE) {
                const int64_t at = (int64_t)(__ldg(ent + 1) + off) * a.W + cl;
                v[i] = in ? flow_over_value(ldv(a.nf + at), ldv(a.nm + at), a.logspace) : PCX_NEG_INF;
            } else {
                v[i] = in ? 0.0f : PCX_NEG_INF;
            }
        }
        if (MODE == C_FWD) {
            const float* src = t.n_kids < 0 ? a.em : a.nm;
            const int n_kids = t.n_kids < 0 ? 1 : t.n_kids;
            for (int c = 0; c < n_kids; c += 2) {
                float x[8], y[8];
                const bool two = c + 1 < n_kids;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int k = ck * 8 + i;
                    const bool in = OCT || k < t.n_k;
                    const int32_t* ent = a.kids + t.kid_off + (OCT ? ck : (in ? k : 0)) * t.width;
                    x[i] = ldv(src + (int64_t)(__ldg(ent + 1 + c) + (OCT ? i : 0)) * a.W + cl);
                    y[i] = two ? ldv(src + (int64_t)(__ldg(ent + 2 + c) + (OCT ? i : 0)) * a.W + cl) : 0.0f;
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] += x[i] + y[i];
            }
            if (t.width > n_kids + 1 && row0 == 0 && col_ok) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int k = ck * 8 + i;
                    if (OCT || k < t.n_k) {
                        const int32_t* ent = a.kids + t.kid_off + (OCT ? ck : k) * t.width;
                        a.em[(int64_t)(__ldg(ent + 1 + n_kids) + (OCT ? i : 0)) * a.W + cl] = v[i];
                    }
                }
            }
        }
        float mx = m;
#pragma unroll
        for (int i = 0; i < 8; ++i) mx = fmaxf(mx, v[i]);
        const float sh = (mx == PCX_NEG_INF) ? 0.0f : mx;
        const float sc = (m == PCX_NEG_INF) ? 0.0f : expf(m - sh);
        m = mx;
#pragma unroll
        for (int r = 0; r < RL; ++r) acc[r] *= sc;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float e = expf(v[i] - sh);
            const float* th = a.params + pid[i] + row0 * t.sr;
#pragma unroll
            for (int r = 0; r < RL; ++r) acc[r] += __ldg(th + r * t.sr) * e;
        }
    }
}

template <int RL>
__device__ __forceinline__ void simt_elements(const ColArgs& a, const int4& st, int cl, int row0, float* e) {
#pragma unroll
    for (int r = 0; r < RL; ++r) e[r] = 0.0f;
    if (st.w < 2) {
        const float* src = st.w < 0 ? a.em : a.nm;
        float y[RL];
#pragma unroll
        for (int r = 0; r < RL; ++r) {
            e[r] = ldv(src + (int64_t)(st.y + row0 + r) * a.W + cl);
            y[r] = st.w < 0 ? 0.0f : ldv(a.nm + (int64_t)(st.z + row0 + r) * a.W + cl);
        }
#pragma unroll
        for (int r = 0; r < RL; ++r) e[r] += y[r];
        return;
    }
    for (int c = 0; c < st.z; ++c) {
        const int k = __ldg(a.kids + st.y + c) + row0;
#pragma unroll
        for (int r = 0; r < RL; ++r) e[r] += ldv(a.nm + (int64_t)(k + r) * a.W + cl);
    }
}

template <int MODE, int RL>
__device__ __forceinline__ void simt_finish(const ColArgs& a, const int4& st, int cl, int row0, float m, const float* acc,
                                            const float* e) {
#pragma unroll
    for (int r = 0; r < RL; ++r) {
        const int row = row0 + r;
        float o;
        if (MODE == C_FWD) {
            o = (m == PCX_NEG_INF) ? PCX_NEG_INF : logf(fmaxf(acc[r], 1e-24f)) + m;
            a.nm[(int64_t)(st.x + row) * a.W + cl] = o;
            continue;
        }
        o = (m == PCX_NEG_INF || acc[r] <= 0.0f) ? PCX_NEG_INF : logf(acc[r]) + m;
        o = (o == PCX_NEG_INF || e[r] == PCX_NEG_INF) ? PCX_NEG_INF : o + e[r];
        if (!a.logspace) o = expf(o);
        store_flow<1>(a, st, row, cl, &o);
    }
}

template <int MODE, int NT, int RL, bool OCT>
__device__ void simt_run(const ColArgs& a, const PcxColTask& t, int col0) {
    constexpr int NC = 8 * NT, G = 32 / NC;
    const int lane = threadIdx.x & 31, c = lane % NC, grp = lane / NC;
    const bool col_ok = col0 + c < a.W;
    const int cl = col_ok ? col0 + c : 0;
    const int GR = min(G, t.n_rows / RL), GK = G / GR;
    const int gr = grp % GR, gk = grp / GR;
    float m, acc[RL], e[RL];
    const int4 st = __ldg(a.strips + t.strip_off);
    if (MODE == C_ELE) simt_elements<RL>(a, st, cl, gr * RL, e);
    simt_partial<MODE, NT, RL, OCT>(a, t, cl, col_ok, gr * RL, gk, GK, m, acc);
    for (int o = NC * GR; o < 32; o <<= 1) {               // the groups that shared the contraction
        const float mo = __shfl_xor_sync(0xffffffffu, m, o);
        const float mx = fmaxf(m, mo), sh = (mx == PCX_NEG_INF) ? 0.0f : mx;
        const float s0 = expf(m - sh), s1 = expf(mo - sh);
#pragma unroll
        for (int r = 0; r < RL; ++r) acc[r] = acc[r] * s0 + __shfl_xor_sync(0xffffffffu, acc[r], o) * s1;
        m = mx;
    }
    if (gk == 0 && col_ok) simt_finish<MODE, RL>(a, st, cl, gr * RL, m, acc, e);
}

template <int MODE, int NT>
__device__ __forceinline__ void simt_task(const ColArgs& a, const PcxColTask& t, int col0) {
    constexpr int G = 4 / NT;
    const int rl = t.n_rows >= G ? t.n_rows / G : 1;       // (16 only where a lane group is the whole warp)
    if (t.lg_entry == 3) {
        if (rl == 1) simt_run<MODE, NT, 1, true>(a, t, col0);
        else if (rl == 2) simt_run<MODE, NT, 2, true>(a, t, col0);
        else if (rl == 4) simt_run<MODE, NT, 4, true>(a, t, col0);
        else if (rl == 8) simt_run<MODE, NT, 8, true>(a, t, col0);
        else if (NT == 4) simt_run<MODE, NT, NT == 4 ? 16 : 8, true>(a, t, col0);
    } else {
        if (rl == 1) simt_run<MODE, NT, 1, false>(a, t, col0);
        else if (rl == 2) simt_run<MODE, NT, 2, false>(a, t, col0);
        else if (rl == 4) simt_run<MODE, NT, 4, false>(a, t, col0);
        else if (rl == 8) simt_run<MODE, NT, 8, false>(a, t, col0);
        else if (NT == 4) simt_run<MODE, NT, NT == 4 ? 16 : 8, false>(a, t, col0);
    }
}

// One row with a long table (roots): its contraction is split over the CTA's warps, their partial sums meet in shared
// memory.  Called by all threads of a CTA.
template <int NT, int NW>
__device__ void split_task(const ColArgs& a, const PcxColTask& t, int col0, float* s_part) {
    constexpr int NC = 8 * NT, G = 32 / NC;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = lane % NC, gk = lane / NC;
    const bool col_ok = col0 + c < a.W;
    const int cl = col_ok ? col0 + c : 0;
    float m, acc[1];
    if (t.lg_entry == 3) simt_partial<C_FWD, NT, 1, true>(a, t, cl, col_ok, 0, warp * G + gk, NW * G, m, acc);
    else simt_partial<C_FWD, NT, 1, false>(a, t, cl, col_ok, 0, warp * G + gk, NW * G, m, acc);
    s_part[(warp * 32 + lane) * 2] = m;
    s_part[(warp * 32 + lane) * 2 + 1] = acc[0];
    __syncthreads();
    if (warp == 0 && lane < NC) {
        float mx = PCX_NEG_INF, sum = 0.0f;
        for (int i = 0; i < NW * G; ++i) mx = fmaxf(mx, s_part[(i * NC + c) * 2]);
        const float sh = (mx == PCX_NEG_INF) ? 0.0f : mx;
        for (int i = 0; i < NW * G; ++i) sum += s_part[(i * NC + c) * 2 + 1] * expf(s_part[(i * NC + c) * 2] - sh);
        if (col_ok) simt_finish<C_FWD, 1>(a, __ldg(a.strips + t.strip_off), cl, 0, mx, &sum, nullptr);
    }
    __syncthreads();
}

// ---- product task (backward): flow of a node = log-sum-exp over its parent products ---------------------------------
template <int NT, int NQ>
__device__ __forceinline__ void prod_parents(const ColArgs& a, const int32_t* par, int p, int row, int n_rows, int co,
                                             float (*mx)[4], float (*sum)[4]) {
    constexpr int RP = 16 / NT, P = NT;                    // rows per pass, passes over 16 rows
    float x[P][NQ][4];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const int r = __ldg(par + p + q);
#pragma unroll
        for (int u = 0; u < P; ++u)
            ldvec<4>(a.ef + (int64_t)(r + (row + u * RP < n_rows ? row + u * RP : 0)) * a.W + co, x[u][q]);
    }
#pragma unroll
    for (int u = 0; u < P; ++u)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (!a.logspace) {
#pragma unroll
                for (int q = 0; q < NQ; ++q) sum[u][j] += x[u][q][j];
                continue;
            }
            float mn = mx[u][j];
#pragma unroll
            for (int q = 0; q < NQ; ++q) mn = fmaxf(mn, x[u][q][j]);
            const float sh = (mn == PCX_NEG_INF) ? 0.0f : mn;
            float t = sum[u][j] * fast_exp(mx[u][j] - sh);
#pragma unroll
            for (int q = 0; q < NQ; ++q) t += fast_exp(x[u][q][j] - sh);
            sum[u][j] = t;
            mx[u][j] = mn;
        }
}

template <int NT>
__device__ void prod_task(const ColArgs& a, const PcxColTask& t, int col0) {
    constexpr int LR = 2 * NT, RP = 32 / LR, P = 16 / RP;  // lanes per row (four columns each), rows per pass, passes
    const int lane = threadIdx.x & 31, row = lane / LR;
    const bool co_ok = col0 + (lane % LR) * 4 < a.W;
    const int co = co_ok ? col0 + (lane % LR) * 4 : 0;
    float mx[P][4], sum[P][4];
    const int32_t* par = a.kids + t.kid_off;
    if (t.n_k == 1 && !t.sk) {                             // one parent product: its flow
        const int r = __ldg(par);
#pragma unroll
        for (int u = 0; u < P; ++u)
            ldvec<4>(a.ef + (int64_t)(r + (row + u * RP < t.n_rows ? row + u * RP : 0)) * a.W + co, sum[u]);
    } else {
#pragma unroll
        for (int u = 0; u < P; ++u) {
#pragma unroll
            for (int j = 0; j < 4; ++j) { mx[u][j] = a.logspace ? PCX_NEG_INF : 0.0f; sum[u][j] = a.logspace ? 1.0f : 0.0f; }
            // flow from products of a level above (rows past the block: the first row, not used)
            if (t.sk) ldvec<4>(a.nf + (int64_t)(t.strip_off + (row + u * RP < t.n_rows ? row + u * RP : 0)) * a.W + co, mx[u]);
            if (t.sk && !a.logspace)
#pragma unroll
                for (int j = 0; j < 4; ++j) sum[u][j] = mx[u][j];
        }
        int p = 0;
        for (; p + 4 <= t.n_k; p += 4) prod_parents<NT, 4>(a, par, p, row, t.n_rows, co, mx, sum);
        if (t.n_k - p >= 2) { prod_parents<NT, 2>(a, par, p, row, t.n_rows, co, mx, sum); p += 2; }
        if (t.n_k - p == 1) prod_parents<NT, 1>(a, par, p, row, t.n_rows, co, mx, sum);
        if (a.logspace)
#pragma unroll
            for (int u = 0; u < P; ++u)
#pragma unroll
                for (int j = 0; j < 4; ++j) sum[u][j] = fast_log_plus(sum[u][j], mx[u][j]);
    }
#pragma unroll
    for (int u = 0; u < P; ++u)
        if (co_ok && row + u * RP < t.n_rows) stvec<4>(a.nf + (int64_t)(t.strip_off + row + u * RP) * a.W + co, sum[u]);
}

// ---- the level walk ---------------------------------------------------------------------------------------------------
template <int MODE, int NT>
__device__ __forceinline__ void run_task(const ColArgs& a, const PcxColTask& t, int col0) {
    if (t.kind == K_MMA) {
        if constexpr (NT < 4) {
            if (t.n_k > 2 && !(MODE == C_FWD && t.n_kids > 2)) {
                mma_task<MODE, NT, 4>(a, t, col0);
                return;
            }
        }
        mma_task<MODE, NT, 2>(a, t, col0);
    } else if (MODE == C_ELE && NT < 4 && t.kind == K_PROD) {              // (wide product levels: column_prod_kernel)
        prod_task<NT < 4 ? NT : 2>(a, t, col0);
    } else {
        simt_task<MODE, NT>(a, t, col0);
    }
}

// A level with work for every warp of the machine gains nothing from sharing a launch, and loses the SMs that the
// clusters leave idle: it is a launch of its own (`wide`), all warps of the grid over (task, tile of 32 columns) with the
// tiles of a task next to one another: a parameter fragment is then fetched once per SM, and the pieces of a value row that
// are requested at about the same time are neighbours (256 bytes of a DRAM page instead of 64: with 16 columns per
// cluster, the levels of a 784-variable Poon-Domingos circuit that outgrow the L2 ran at 0.8 TB/s).
template <int MODE>
__global__ void __launch_bounds__(WT, 1) column_wide_kernel(const ColArgs a) {
    constexpr int NT = 4, NW = WT / 32;
    __shared__ float s_part[NW * 64];
    const int4 lv = __ldg(a.levels);
    const int items = lv.y * a.tiles;
    for (int i = blockIdx.x * NW + (threadIdx.x >> 5); i < items; i += gridDim.x * NW)
        run_task<MODE, NT>(a, load_record(a.tasks, lv.x + i / a.tiles), (i % a.tiles) * 8 * NT);
    if (MODE == C_FWD)
        for (int i = blockIdx.x; i < lv.w * a.tiles; i += gridDim.x)
            split_task<NT, NW>(a, a.tasks[lv.z + i / a.tiles], (i % a.tiles) * 8 * NT, s_part);
}


// ---- wide levels of plain MMA tasks: operands through shared memory ---------------------------------------------------
// With the operands in registers a warp task is a chain of six to ten memory latencies, and registers bound how much a
// warp can have under way (a level of 1246 element-flow tasks at 512 samples: 149 us, 26 % of the issue slots, 1.5 TB/s of
// DRAM).  Here each warp owns two 8 KB stages and copies the next stage (cp.async) while it works on the current one,
// across task boundaries, so that its time is its instructions.  A stage is four groups of 16 rows x 32 columns: two
// 16-deep steps with two operand rows each (two children; flow and value), or the two children of two strips' elements.
// A row's eight 16-byte pieces are permuted by (row & 7): the B-fragment reads (eight pieces of rows 2t) and the epilogue's
// (two pieces of rows g) both touch every bank once.
constexpr int PIPE_STAGE = 4 * 16 * 128;
constexpr int PIPE_SMEM = (WT / 32) * 2 * PIPE_STAGE;

__device__ __forceinline__ void pipe_copy16(uint32_t smem_group, const float* rows, int64_t W, int col, int col_limit) {
    const int lane = threadIdx.x & 31, piece = lane & 7;
    const int c = col + piece * 4;
    const float* src = rows + (c < col_limit ? c : 0);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int row = j * 4 + (lane >> 3);
        const uint32_t dst = smem_group + row * 128 + ((piece ^ (row & 7)) << 4);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src + row * W) : "memory");
    }
}
__device__ __forceinline__ void pipe_read16(uint32_t smem_group, int row, int piece, float* v) {
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
                 : "r"(smem_group + row * 128 + ((piece ^ (row & 7)) << 4)));
}

// Requests stage `s` of a task (record, operand entries and strip records one word per lane).
template <int MODE>
__device__ __forceinline__ void pipe_request(const ColArgs& a, int rec, int kv, int sv, int s, int col, uint32_t buf) {
    const int n_k = __shfl_sync(0xffffffffu, rec, 1), n_kids = __shfl_sync(0xffffffffu, rec, 2);
    const int n_chunks = (n_k + 1) >> 1;
    if (MODE == C_ELE && s == n_chunks) {
        const int n_rows = __shfl_sync(0xffffffffu, rec, 5);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int y = __shfl_sync(0xffffffffu, sv, 4 * q + 1), z = __shfl_sync(0xffffffffu, sv, 4 * q + 2);
            const int w = __shfl_sync(0xffffffffu, sv, 4 * q + 3);
            if (q < n_rows) {
                pipe_copy16(buf + (2 * q) * 2048, (w < 0 ? a.em : a.nm) + (int64_t)y * a.W, a.W, col, a.W);
                if (w >= 0) pipe_copy16(buf + (2 * q + 1) * 2048, a.nm + (int64_t)z * a.W, a.W, col, a.W);
            }
        }
        return;
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int k = 2 * s + q;
        if (MODE == C_ELE || n_kids != 2) {
            const int r = __shfl_sync(0xffffffffu, kv, k & 31);
            if (k < n_k) {
                const float* src = MODE == C_ELE ? a.nf : (n_kids < 0 ? a.em : a.nm);
                pipe_copy16(buf + (2 * q) * 2048, src + (int64_t)r * a.W, a.W, col, a.W);
                if (MODE == C_ELE) pipe_copy16(buf + (2 * q + 1) * 2048, a.nm + (int64_t)r * a.W, a.W, col, a.W);
            }
        } else {
            const int r0 = __shfl_sync(0xffffffffu, kv, (2 * k) & 31), r1 = __shfl_sync(0xffffffffu, kv, (2 * k + 1) & 31);
            if (k < n_k) {
                pipe_copy16(buf + (2 * q) * 2048, a.nm + (int64_t)r0 * a.W, a.W, col, a.W);
                pipe_copy16(buf + (2 * q + 1) * 2048, a.nm + (int64_t)r1 * a.W, a.W, col, a.W);
            }
        }
    }
}
__device__ __forceinline__ int fetch_strips(const ColArgs& a, int rec) {
    const int off = __shfl_sync(0xffffffffu, rec, 4), n = __shfl_sync(0xffffffffu, rec, 5);
    const int lane = threadIdx.x & 31;
    return lane < 4 * n ? __ldg(reinterpret_cast<const int*>(a.strips + off) + lane) : 0;
}

template <int MODE>
__global__ void __launch_bounds__(WT, 1) column_pipe_kernel(const ColArgs a) {
    constexpr int NT = 4, NW = WT / 32;
    extern __shared__ __align__(128) uint8_t s_pipe[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(s_pipe) + warp * 2 * PIPE_STAGE;
    const int W = a.W;
    const int4 lv = __ldg(a.levels);
    const int items = lv.y * a.tiles, first = blockIdx.x * NW + warp, stride = gridDim.x * NW, last = items - 1;
    if (first >= items) return;
    int rec = fetch_record(a.tasks, lv.x + first / a.tiles);
    int rec1 = fetch_record(a.tasks, lv.x + min(first + stride, last) / a.tiles);
    int kv = fetch_kids(a, rec), sv = fetch_strips(a, rec);
    int p = 0;
    pipe_request<MODE>(a, rec, kv, sv, 0, (first % a.tiles) * 32, base);
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int i = first; i < items; i += stride) {
        const int kv1 = fetch_kids(a, rec1), sv1 = fetch_strips(a, rec1);
        const int rec2 = fetch_record(a.tasks, lv.x + min(i + 2 * stride, last) / a.tiles);
        const int n_k = __shfl_sync(0xffffffffu, rec, 1), n_rows = __shfl_sync(0xffffffffu, rec, 5);
        const int n_kids = __shfl_sync(0xffffffffu, rec, 2), par_off = __shfl_sync(0xffffffffu, rec, 6);
        const int col0 = (i % a.tiles) * 32;
        const int n_chunks = (n_k + 1) >> 1, n_stages = n_chunks + (MODE == C_ELE ? 1 : 0);
        float m[NT], acc[2][NT][4];
#pragma unroll
        for (int j = 0; j < NT; ++j) m[j] = PCX_NEG_INF;
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[q][j][c] = 0.0f;
        for (int st = 0; st < n_stages; ++st) {
            const uint32_t buf = base + p * PIPE_STAGE, other = base + (p ^ 1) * PIPE_STAGE;
            if (st + 1 < n_stages) pipe_request<MODE>(a, rec, kv, sv, st + 1, col0, other);
            else if (i + stride < items) pipe_request<MODE>(a, rec1, kv1, sv1, 0, ((i + stride) % a.tiles) * 32, other);
            asm volatile("cp.async.commit_group;" ::: "memory");
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncwarp();
            if (st < n_chunks) {
                const int k0 = 2 * st, live = min(2, n_k - k0);
                float v[2][4][NT];
#pragma unroll
                for (int q = 0; q < 2; ++q)
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const int row = 2 * tq + (r & 1) + (r >> 1) * 8;
                        if (q < live) {
                            pipe_read16(buf + (2 * q) * 2048, row, g, v[q][r]);
                            if (MODE == C_ELE || n_kids == 2) {
                                float y[NT];
                                pipe_read16(buf + (2 * q + 1) * 2048, row, g, y);
#pragma unroll
                                for (int j = 0; j < NT; ++j)
                                    v[q][r][j] = MODE == C_ELE ? flow_over_value(v[q][r][j], y[j], a.logspace) : v[q][r][j] + y[j];
                            }
                        } else {
#pragma unroll
                            for (int j = 0; j < NT; ++j) v[q][r][j] = PCX_NEG_INF;
                        }
                    }
                float sc[NT];
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    float mx = m[j];
#pragma unroll
                    for (int q = 0; q < 2; ++q)
#pragma unroll
                        for (int r = 0; r < 4; ++r) mx = fmaxf(mx, v[q][r][j]);
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
                    sc[j] = (m[j] == PCX_NEG_INF) ? 0.0f : fast_exp(m[j] - mx);
                    m[j] = mx;
                }
                if (st > 0) {
#pragma unroll
                    for (int j = 0; j < NT; ++j) {
                        const float s0 = __shfl_sync(0xffffffffu, sc[j], 8 * tq), s1 = __shfl_sync(0xffffffffu, sc[j], 8 * tq + 4);
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            acc[q][j][0] *= s0; acc[q][j][1] *= s1; acc[q][j][2] *= s0; acc[q][j][3] *= s1;
                        }
                    }
                }
                const uint4* fr = a.frags + ((int64_t)par_off + (int64_t)k0 * n_rows) * 64 + lane;
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    if (q < live) {
                        uint4 ah[2], al[2];
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const uint4* f = fr + (q * n_rows + (h < n_rows ? h : 0)) * 64;
                            ah[h] = __ldg(f); al[h] = __ldg(f + 32);
                        }
#pragma unroll
                        for (int j = 0; j < NT; ++j) {
                            const float sh = (m[j] == PCX_NEG_INF) ? 0.0f : m[j];
                            uint32_t bh0, bl0, bh1, bl1;
                            split2(fast_exp(v[q][0][j] - sh), fast_exp(v[q][1][j] - sh), bh0, bl0);
                            split2(fast_exp(v[q][2][j] - sh), fast_exp(v[q][3][j] - sh), bh1, bl1);
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                mma16816(acc[h][j], ah[h], bh0, bh1);
                                if (a.terms == 3) {
                                    mma16816(acc[h][j], ah[h], bl0, bl1);
                                    mma16816(acc[h][j], al[h], bh0, bh1);
                                }
                            }
                        }
                    }
                }
            }
            if (st + 1 == n_stages) {                       // the task's last stage: results
                const int co = col0 + 8 * tq;
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    int4 sr;
                    sr.x = __shfl_sync(0xffffffffu, sv, 4 * q); sr.y = __shfl_sync(0xffffffffu, sv, 4 * q + 1);
                    sr.z = __shfl_sync(0xffffffffu, sv, 4 * q + 2); sr.w = __shfl_sync(0xffffffffu, sv, 4 * q + 3);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        float o[2 * NT];
#pragma unroll
                        for (int j = 0; j < NT; ++j) {
                            const float m0 = __shfl_sync(0xffffffffu, m[j], 8 * tq), m1 = __shfl_sync(0xffffffffu, m[j], 8 * tq + 4);
                            const float x0 = acc[q][j][2 * h], x1 = acc[q][j][2 * h + 1];
                            o[j] = fast_log_plus(MODE == C_FWD ? fmaxf(x0, 1e-24f) : x0, m0);
                            o[NT + j] = fast_log_plus(MODE == C_FWD ? fmaxf(x1, 1e-24f) : x1, m1);
                        }
                        if (q >= n_rows || co >= W) continue;
                        const int row = g + 8 * h;
                        if (MODE == C_FWD) {
                            stvec<2 * NT>(a.nm + (int64_t)(sr.x + row) * W + co, o);
                            continue;
                        }
                        float e[2 * NT];
                        pipe_read16(buf + (2 * q) * 2048, row, 2 * tq, e);
                        pipe_read16(buf + (2 * q) * 2048, row, 2 * tq + 1, e + 4);
                        if (sr.w >= 0) {
                            float y[2 * NT];
                            pipe_read16(buf + (2 * q + 1) * 2048, row, 2 * tq, y);
                            pipe_read16(buf + (2 * q + 1) * 2048, row, 2 * tq + 1, y + 4);
#pragma unroll
                            for (int j = 0; j < 2 * NT; ++j) e[j] += y[j];
                        }
#pragma unroll
                        for (int j = 0; j < 2 * NT; ++j) {
                            o[j] += e[j];
                            if (!a.logspace) o[j] = __expf(o[j]);
                        }
                        store_flow<2 * NT>(a, sr, row, co, o);
                    }
                }
            }
            __syncwarp();                                   // the stage may be overwritten
            p ^= 1;
        }
        rec = rec1; rec1 = rec2; kv = kv1; sv = sv1;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// Wide product levels: a thread owns four columns of one row, so that an SM has 2048 rows' loads under way (a level of 2712
// tasks of 16 rows at 512 samples, 1.5 parents each: 78 us as warp tasks).  Long parent lists are taken four at a time: 25088
// rows of 16 parents, 1024 samples: 234 us two at a time, 185 now (1.6 GB of reads, from L2).
__global__ void __launch_bounds__(256) column_prod_kernel(const ColArgs a) {
    const int4 lv = __ldg(a.levels);
    const int W4 = a.W >> 2;
    const int64_t total = (int64_t)lv.y * 16 * W4;
    const float none = a.logspace ? PCX_NEG_INF : 0.0f;
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < total; i += (int64_t)gridDim.x * 256) {
        const uint32_t r = (uint32_t)(i / W4);
        const int co = (int)(i - (int64_t)r * W4) * 4;
        const PcxColTask* t = a.tasks + lv.x + (r >> 4);
        const int row = r & 15;
        if (row >= __ldg(&t->n_rows)) continue;
        const int n = __ldg(&t->n_k), add = __ldg(&t->sk);
        const int32_t* par = a.kids + __ldg(&t->kid_off);
        float* dst = a.nf + (int64_t)(__ldg(&t->strip_off) + row) * a.W + co;
        float mx[4], sum[4];
        if (n == 1 && !add) {
            ldvec<4>(a.ef + (int64_t)(__ldg(par) + row) * a.W + co, sum);
            stvec<4>(dst, sum);
            continue;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) { mx[j] = none; sum[j] = a.logspace ? 1.0f : 0.0f; }
        if (add) ldvec<4>(dst, mx);
        if (add && !a.logspace)
#pragma unroll
            for (int j = 0; j < 4; ++j) sum[j] = mx[j];
        int p = 0;
        for (; p + 4 <= n; p += 4) {
            float x[4][4];
#pragma unroll
            for (int q = 0; q < 4; ++q) ldvec<4>(a.ef + (int64_t)(__ldg(par + p + q) + row) * a.W + co, x[q]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (!a.logspace) { sum[j] += (x[0][j] + x[1][j]) + (x[2][j] + x[3][j]); continue; }
                const float mn = fmaxf(mx[j], fmaxf(fmaxf(x[0][j], x[1][j]), fmaxf(x[2][j], x[3][j])));
                const float sh = (mn == PCX_NEG_INF) ? 0.0f : mn;
                sum[j] = sum[j] * fast_exp(mx[j] - sh) + (fast_exp(x[0][j] - sh) + fast_exp(x[1][j] - sh))
                         + (fast_exp(x[2][j] - sh) + fast_exp(x[3][j] - sh));
                mx[j] = mn;
            }
        }
        for (; p < n; p += 2) {
            float x[2][4];
            ldvec<4>(a.ef + (int64_t)(__ldg(par + p) + row) * a.W + co, x[0]);
            if (p + 1 < n) ldvec<4>(a.ef + (int64_t)(__ldg(par + p + 1) + row) * a.W + co, x[1]);
            else
#pragma unroll
                for (int j = 0; j < 4; ++j) x[1][j] = none;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (!a.logspace) { sum[j] += x[0][j] + x[1][j]; continue; }
                const float mn = fmaxf(mx[j], fmaxf(x[0][j], x[1][j])), sh = (mn == PCX_NEG_INF) ? 0.0f : mn;
                sum[j] = sum[j] * fast_exp(mx[j] - sh) + fast_exp(x[0][j] - sh) + fast_exp(x[1][j] - sh);
                mx[j] = mn;
            }
        }
        if (a.logspace)
#pragma unroll
            for (int j = 0; j < 4; ++j) sum[j] = fast_log_plus(sum[j], mx[j]);
        stvec<4>(dst, sum);
    }
}

template <int MODE, int NT>
__global__ void __launch_bounds__(CT, 1) column_kernel(const ColArgs a) {
    __shared__ float s_part[CW * 64];
    __shared__ int4 levels[MAX_LEVELS];
    const int warp = threadIdx.x >> 5;
    const int rank = blockIdx.x % a.cluster;
    const int col0 = (blockIdx.x / a.cluster) * 8 * NT;
    const int worker = warp * a.cluster + rank, workers = CW * a.cluster;
    // The level table sits in shared memory; the record of the warp's next task is in registers and the lines of its tables
    // are on their way to L1, across levels: a level opens with the loads of its values.
    for (int i = threadIdx.x; i < a.n_levels; i += CT) levels[i] = __ldg(a.levels + i);
    __syncthreads();
    int next_l = 0, next_i = worker;                       // the task after the fetched ones
    auto advance = [&](int& task, int& at) {
        while (next_l < a.n_levels && next_i >= levels[next_l].y) { ++next_l; next_i = worker; }
        at = next_l;
        task = next_l < a.n_levels ? levels[next_l].x + next_i : 0;
        next_i += workers;
        touch(a.tasks + task);
    };
    int task, at, task1, at1;
    advance(task, at);
    advance(task1, at1);
    PcxColTask t = load_record(a.tasks, task);
    for (int l = 0; l < a.n_levels; ++l) {
        while (at == l) {
            const PcxColTask t1 = load_record(a.tasks, task1);
            touch(a.kids + t1.kid_off);
            if (t1.kind != K_PROD) touch(a.strips + t1.strip_off);
            if (t1.kind == K_MMA && (int)(threadIdx.x & 31) < 8 * t1.n_k * t1.n_rows)       // the first four fragments
                touch(a.frags + (int64_t)t1.par_off * 64 + (threadIdx.x & 31) * 8);
            int task2, at2;
            advance(task2, at2);
            run_task<MODE, NT>(a, t, col0);
            t = t1; at = at1;
            task1 = task2; at1 = at2;
        }
        const int4 lv = levels[l];
        if (MODE == C_FWD)
            for (int i = rank; i < lv.w; i += a.cluster) split_task<NT, CW>(a, a.tasks[lv.z + i], col0, s_part);
        if (a.cluster == 1) {
            __syncthreads();
        } else {
            __syncwarp();
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        }
    }
}

// ---- large groups: CTA tasks ---------------------------------------------------------------------------------------------
// Where many rows share a long child list (node blocks of 128 and more: hidden trees with 128 latents and up, the dense
// transitions of an HMM) warp tasks would each gather the list again.  A CTA task gathers, exponentiates and splits it once
// into shared memory in the order of the B fragments, and the 16 warps multiply strips (and, where a task has fewer than 16
// strips, parts of the contraction) from there.  What the task does not wait for is there before it starts: the parameter
// fragments of a CTA's next task are copied to shared memory while the current one finishes, and tied layers (every
// transition of a homogeneous HMM) find them there already -- 512 x 512 parameters over a cluster of 8 CTAs are 128 KB each.
// tcgen05 would need 128-row tiles and a trip through tensor memory per level; with 8 or 16 columns per cluster the
// multiplication is a tenth of a level, which is gather, two CTA barriers and the cluster barrier.
constexpr int BIG_MAX_STEPS = 64;

template <int NT>
struct BigSmem {
    static constexpr int MAX = CW * 8 * NT * 4;                        // column maxima per warp
    static constexpr int RED = CW * 32 * NT * 16;                      // partial accumulators
    static constexpr int LEVELS = MAX_LEVELS * 16;
    static constexpr int PART = CW * 64 * 4;                           // split tasks
    static constexpr int FIXED = MAX + RED + LEVELS + PART;
};

struct BigState {
    uint8_t* a_frag;            // shared: the parameter fragments of one task (its first `held` steps)
    uint4* b_frag;              // shared: [step][tile][lane]
    float* s_max;
    float4* s_red;
    int a_bytes;
    int a_off, a_held;          // fragments now in (or on their way to) a_frag: first fragment, steps
};

struct BigParams { int par_off, n_k, n_rows; };             // whose fragments: n_k = 0: nobody's

__device__ __forceinline__ void big_load_params(const ColArgs& a, const BigParams& t, BigState& b) {
    if (t.par_off == b.a_off) return;
    b.a_off = t.par_off;
    b.a_held = min(t.n_k, b.a_bytes / (t.n_rows * 1024));
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(b.a_frag);
    const uint8_t* src = reinterpret_cast<const uint8_t*>(a.frags) + (int64_t)t.par_off * 1024;
    const int bytes = b.a_held * t.n_rows * 1024;
    for (int i = threadIdx.x * 16; i < bytes; i += CT * 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i), "l"(src + i) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// What a warp needs of a CTA task before its first load of a value: fetched while the level before it closes.
struct BigAhead {
    int kid[4][2];              // operand rows of its first four half steps (children 0 and 1)
    int4 st;                    // its output record
};

template <int MODE>
__device__ __forceinline__ void big_look_ahead(const ColArgs& a, const PcxColTask& t, BigAhead& f) {
    const int warp = threadIdx.x >> 5, halves = 2 * t.n_k;
    const int32_t* kid = a.kids + t.kid_off;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int u = warp + CW * j, q = u < halves ? u >> 1 : 0;
        f.kid[j][0] = __ldg(kid + q * t.width);
        f.kid[j][1] = (MODE == C_FWD && t.n_kids > 1) ? __ldg(kid + q * t.width + 1) : 0;
    }
    f.st = __ldg(a.strips + t.strip_off + warp % t.n_rows);
}

// PER: half steps per warp (depth / 128, rounded up to 1, 2, 4 or 8).
template <int MODE, int NT, int PER, typename Next>
__device__ __forceinline__ void cta_task(const ColArgs& a, const PcxColTask& t, const BigAhead& f, int col0, BigState& b, Next next) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, tq = lane & 3;
    const int W = a.W;
    const int cl = (col0 + NT * g < W) ? col0 + NT * g : 0;
    const int co = col0 + 2 * NT * tq;
    const bool co_ok = co < W;
    const int32_t* kid = a.kids + t.kid_off;
    const int halves = 2 * t.n_k;

    // operand: half step u = rows 2t, 2t+1 (+ 8) of a 16-deep step; up to four at a time, with two operand rows each
    float v[PER][2][NT];
#pragma unroll
    for (int j0 = 0; j0 < PER; j0 += 4) {
        constexpr int N = PER < 4 ? PER : 4;
        float y[N][2][NT];
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const int u = warp + CW * (j0 + j), o = 2 * tq + 8 * (u & 1);
            int r0, r1;
            if (j0 == 0) {
                r0 = f.kid[j][0];
                r1 = f.kid[j][1];
            } else {
                const int32_t* e = kid + (u < halves ? u >> 1 : 0) * t.width;
                r0 = __ldg(e);
                r1 = (MODE == C_FWD && t.n_kids > 1) ? __ldg(e + 1) : 0;
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                ldvec<NT>((MODE == C_ELE ? a.nf : a.nm) + (int64_t)(r0 + o + i) * W + cl, v[j0 + j][i]);
                ldvec<NT>(a.nm + (int64_t)((MODE == C_ELE ? r0 : r1) + o + i) * W + cl, y[j][i]);
            }
        }
#pragma unroll
        for (int j = 0; j < N; ++j)
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int n = 0; n < NT; ++n)
                    v[j0 + j][i][n] = MODE == C_ELE ? flow_over_value(v[j0 + j][i][n], y[j][i][n], a.logspace) : v[j0 + j][i][n] + y[j][i][n];
        if (MODE == C_FWD) {
            for (int c = 2; c < t.n_kids; c += 2) {        // elements of more than two children
                float x[N][2][NT];
                const bool two = c + 1 < t.n_kids;
#pragma unroll
                for (int j = 0; j < N; ++j) {
                    const int u = warp + CW * (j0 + j), o = 2 * tq + 8 * (u & 1);
                    const int32_t* e = kid + (u < halves ? u >> 1 : 0) * t.width + c;
                    const int r0 = __ldg(e) + o, r1 = two ? __ldg(e + 1) + o : o;
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        ldvec<NT>(a.nm + (int64_t)(r0 + i) * W + cl, x[j][i]);
                        ldvec<NT>(a.nm + (int64_t)(r1 + i) * W + cl, y[j][i]);
                    }
                }
#pragma unroll
                for (int j = 0; j < N; ++j)
#pragma unroll
                    for (int i = 0; i < 2; ++i)
#pragma unroll
                        for (int n = 0; n < NT; ++n) v[j0 + j][i][n] += x[j][i][n] + (two ? y[j][i][n] : 0.0f);
            }
            if (t.width > t.n_kids && col0 + NT * g < W) { // keep the elements' values
#pragma unroll
                for (int j = 0; j < N; ++j) {
                    const int u = warp + CW * (j0 + j);
                    if (u < halves) {
                        const int r = __ldg(kid + (u >> 1) * t.width + t.n_kids) + 2 * tq + 8 * (u & 1);
#pragma unroll
                        for (int i = 0; i < 2; ++i) stvec<NT>(a.em + (int64_t)(r + i) * W + cl, v[j0 + j][i]);
                    }
                }
            }
        }
    }
    // strips and parts of the contraction (strips per task: a power of two up to 16)
    const int parts = CW / t.n_rows, strip = warp % t.n_rows, part = warp / t.n_rows;
    ElementValue<NT> ev[2];
    if (MODE == C_ELE && part == 0 && co_ok) {             // (in flight until the epilogue)
        load_element<NT>(a, f.st, g, co, ev[0]);
        load_element<NT>(a, f.st, g + 8, co, ev[1]);
    }
    float m[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        m[n] = PCX_NEG_INF;
#pragma unroll
        for (int j = 0; j < PER; ++j)
            if (warp + CW * j < halves) m[n] = fmaxf(m[n], fmaxf(v[j][0][n], v[j][1][n]));
        m[n] = fmaxf(m[n], __shfl_xor_sync(0xffffffffu, m[n], 1));
        m[n] = fmaxf(m[n], __shfl_xor_sync(0xffffffffu, m[n], 2));
        if (tq == 0) b.s_max[(NT * g + n) * CW + warp] = m[n];
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        // four lanes share a column: each takes the maxima of four warps
        const float4 q = *reinterpret_cast<const float4*>(b.s_max + (NT * g + n) * CW + tq * 4);
        m[n] = fmaxf(fmaxf(q.x, q.y), fmaxf(q.z, q.w));
        m[n] = fmaxf(m[n], __shfl_xor_sync(0xffffffffu, m[n], 1));
        m[n] = fmaxf(m[n], __shfl_xor_sync(0xffffffffu, m[n], 2));
        const float sh = (m[n] == PCX_NEG_INF) ? 0.0f : m[n];
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const int u = warp + CW * j;
            if (u < halves) {
                uint32_t hi, lo;
                split2(fast_exp(v[j][0][n] - sh), fast_exp(v[j][1][n] - sh), hi, lo);
                // (the two halves of a step interleave their words: see the reader)
                *reinterpret_cast<uint2*>(reinterpret_cast<uint32_t*>(b.b_frag + ((u >> 1) * NT + n) * 32 + lane) + 2 * (u & 1)) = make_uint2(hi, lo);
            }
        }
    }
    const int k_begin = part * t.n_k / parts, k_end = (part + 1) * t.n_k / parts;
    float acc[3][NT][4];                                    // the three products have accumulators of their own: no chain
#pragma unroll
    for (int x = 0; x < 3; ++x)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[x][n][c] = 0.0f;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    {
        const uint4* as = reinterpret_cast<const uint4*>(b.a_frag) + strip * 64 + lane;
        const uint4* ag = a.frags + ((int64_t)t.par_off + strip) * 64 + lane;
        const int stride = t.n_rows * 64, held = b.a_held;
        auto step = [&](int k, const uint4& ah, const uint4& al) {
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const uint4 w = b.b_frag[(k * NT + n) * 32 + lane];        // hi, lo of rows 2t; hi, lo of rows 2t + 8
                mma16816(acc[0][n], ah, w.x, w.z);
                if (a.terms == 3) {
                    mma16816(acc[1][n], ah, w.y, w.w);
                    mma16816(acc[2][n], al, w.x, w.z);
                }
            }
        };
        int k = k_begin;
#pragma unroll 4
        for (; k < min(k_end, held); ++k) step(k, as[k * stride], as[k * stride + 32]);
#pragma unroll 4
        for (; k < k_end; ++k) step(k, __ldg(ag + (int64_t)k * stride), __ldg(ag + (int64_t)k * stride + 32));
    }
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[0][n][c] += acc[1][n][c] + acc[2][n][c];
    if (part > 0) {
#pragma unroll
        for (int n = 0; n < NT; ++n)
            b.s_red[(warp * NT + n) * 32 + lane] = make_float4(acc[0][n][0], acc[0][n][1], acc[0][n][2], acc[0][n][3]);
    }
    __syncthreads();
    next();
    if (part > 0) return;
    for (int q = 1; q < parts; ++q)
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            const float4 x = b.s_red[((strip + q * t.n_rows) * NT + n) * 32 + lane];
            acc[0][n][0] += x.x; acc[0][n][1] += x.y; acc[0][n][2] += x.z; acc[0][n][3] += x.w;
        }
    float m0[NT], m1[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        m0[n] = __shfl_sync(0xffffffffu, m[n], 8 * tq);
        m1[n] = __shfl_sync(0xffffffffu, m[n], 8 * tq + 4);
    }
    if (!co_ok) return;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int row = g + 8 * h;
        float o[2 * NT];
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            const float x0 = acc[0][n][2 * h], x1 = acc[0][n][2 * h + 1];
            o[n] = fast_log_plus(MODE == C_FWD ? fmaxf(x0, 1e-24f) : x0, m0[n]);
            o[NT + n] = fast_log_plus(MODE == C_FWD ? fmaxf(x1, 1e-24f) : x1, m1[n]);
        }
        if (MODE == C_FWD) {
            stvec<2 * NT>(a.nm + (int64_t)(f.st.x + row) * W + co, o);
            continue;
        }
#pragma unroll
        for (int n = 0; n < 2 * NT; ++n) {
            o[n] += ev[h].x[0][n] + ev[h].x[1][n];
            if (!a.logspace) o[n] = __expf(o[n]);
        }
        store_flow<2 * NT>(a, f.st, row, co, o);
    }
}

template <int MODE, int NT>
__global__ void __launch_bounds__(CT, 1) column_big_kernel(const ColArgs a, int a_bytes, int b_bytes) {
    using C = BigSmem<NT>;
    extern __shared__ __align__(128) uint8_t s_pipe[];
    BigState b;
    b.a_frag = s_pipe;
    b.b_frag = reinterpret_cast<uint4*>(s_pipe + a_bytes);
    uint8_t* fixed = s_pipe + a_bytes + b_bytes;
    b.s_max = reinterpret_cast<float*>(fixed);
    b.s_red = reinterpret_cast<float4*>(fixed + C::MAX);
    int4* levels = reinterpret_cast<int4*>(fixed + C::MAX + C::RED);
    float* s_part = reinterpret_cast<float*>(fixed + C::MAX + C::RED + C::LEVELS);
    b.a_bytes = a_bytes;
    b.a_off = -1;
    b.a_held = 0;
    const int rank = blockIdx.x % a.cluster, warp = threadIdx.x >> 5;
    const int col0 = (blockIdx.x / a.cluster) * 8 * NT;
    const int worker = warp * a.cluster + rank, workers = CW * a.cluster;
    for (int i = threadIdx.x; i < a.n_levels; i += CT) levels[i] = __ldg(a.levels + i);
    __syncthreads();
    // this CTA's CTA tasks, across levels: the record of the next one is fetched when the products of the current one are
    // done, its parameters follow, and the rows it will read are known before the barrier opens
    int next_l = 0, next_i = rank;
    auto advance = [&](int& at) {
        while (next_l < a.n_levels && next_i >= levels[next_l].w) { ++next_l; next_i = rank; }
        at = next_l;
        const int task = next_l < a.n_levels ? levels[next_l].z + next_i : 0;
        next_i += a.cluster;
        return load_record(a.tasks, task);
    };
    int at;
    PcxColTask t = advance(at);
    BigAhead f;
    if (t.kind == K_CTA) {
        big_load_params(a, BigParams{t.par_off, t.n_k, t.n_rows}, b);
        big_look_ahead<MODE>(a, t, f);
    }
    for (int l = 0; l < a.n_levels; ++l) {
        const int4 lv = levels[l];
        for (int i = worker; i < lv.y; i += workers) run_task<MODE, NT>(a, load_record(a.tasks, lv.x + i), col0);
        while (at == l) {
            PcxColTask t1;
            int at1;
            auto next = [&]() {
                t1 = advance(at1);
                if (at1 < a.n_levels && t1.kind == K_CTA) big_load_params(a, BigParams{t1.par_off, t1.n_k, t1.n_rows}, b);
            };
            if (t.kind == K_CTA) {
                if (t.n_k <= 8) cta_task<MODE, NT, 1>(a, t, f, col0, b, next);
                else if (t.n_k <= 16) cta_task<MODE, NT, 2>(a, t, f, col0, b, next);
                else if (t.n_k <= 32) cta_task<MODE, NT, 4>(a, t, f, col0, b, next);
                else cta_task<MODE, NT, 8>(a, t, f, col0, b, next);
            } else {
                if (MODE == C_FWD) split_task<NT, CW>(a, t, col0, s_part);
                next();
            }
            t = t1; at = at1;
            if (at < a.n_levels && t.kind == K_CTA) big_look_ahead<MODE>(a, t, f);
        }
        if (a.cluster == 1) {
            __syncthreads();
        } else {
            __syncwarp();
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// ---- parameter fragments -----------------------------------------------------------------------------------------------
// Fragment f covers 16 rows x 16 children: element (row r, child k) is params[base + r * sr + k * sk].  64 words of 16
// bytes: the high parts of the 32 lanes' A registers, then the low parts.
__global__ void __launch_bounds__(256)
column_pack_kernel(uint4* __restrict__ frags, const int4* __restrict__ bases, int64_t n, const float* __restrict__ params) {
    const int64_t f = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (f >= n) return;
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int4 b = bases[f];                               // base, sr, sk
    const float* p = params + b.x;
    float x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int row = g + ((i >> 1) & 1) * 8, col = 2 * t + (i & 1) + (i >> 2) * 8;
        x[i] = __ldg(p + row * b.y + col * b.z);
    }
    uint4 h, l;
    split2(x[0], x[1], h.x, l.x);
    split2(x[2], x[3], h.y, l.y);
    split2(x[4], x[5], h.z, l.z);
    split2(x[6], x[7], h.w, l.w);
    frags[f * 64 + lane] = h;
    frags[f * 64 + 32 + lane] = l;
}

// ---- parameter flows -----------------------------------------------------------------------------------------------------
// flow[p, c] += theta[p, c] * sum_b exp(nf[p,b] - nm[p,b] - s_b) * exp(em[c,b] + s_b), s_b the maximum of the first exponent
// over the tile's rows.
struct ColParArgs {
    float* pf;
    const float* nf;
    const float* nm;
    const float* em;
    const float* params;
    const PcxColPar* jobs;
    const int32_t* kids;
    const int2* pp;             // (parameter, flow) offsets
    int n_jobs;
    int splits;                 // the batch is cut into this many pieces
    int per_split;              // samples per piece (a multiple of 16 / 32)
    int W;
    int logspace;
    int terms;
};

// Tensor-core tiles of elements of more than two children (up to two, and stored values: column_par_pipe_kernel): a warp owns
// 32 nodes (two strips) x 32 edges, the batch in steps of 16.  Flow and value of 32 rows are requested together, then the rows
// of 32 edges child by child.  The eight warps of a CTA take neighbouring tiles, which share one side's rows.
__device__ __forceinline__ void par_mma_tile(const ColParArgs& a, const PcxColPar& t, int b_begin, int b_end) {
    const int lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
    const int64_t W = a.W;
    float acc[2][4][4];
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[s][e][c] = 0.0f;
    const int64_t r0 = (int64_t)(t.row0 + g) * W, r1 = (int64_t)(t.row1 + g) * W;
    for (int b0 = b_begin; b0 < b_end; b0 += 16) {
        // lane t holds samples 4t .. 4t+3 where the fragments have 2t, 2t+1, 2t+8, 2t+9: the order of a sum's terms is free,
        // and this way a row is one 16-byte load
        const bool in = b0 + 4 * tq < b_end;
        const int64_t c0 = in ? b0 + 4 * tq : b0;
        float f[2][2][4], v[2][2][4];                      // strip, row half, sample
#pragma unroll
        for (int s = 0; s < 2; ++s)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int64_t at = (s == 0 ? r0 : r1) + 8 * h * W;
                ldvec<4>(a.nf + at + c0, f[s][h]);
                ldvec<4>(a.nm + at + c0, v[s][h]);
            }
        float y[4][4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int i = 0; i < 4; ++i) y[e][i] = 0.0f;
        for (int c = 0; c < t.n_kids; ++c) {
            float z[4][4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int k = __ldg(a.kids + t.kid_off + ((e >> 1) < t.n_k ? (e >> 1) : 0) * t.width + c) + g + 8 * (e & 1);
                ldvec<4>(a.nm + k * W + c0, z[e]);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int i = 0; i < 4; ++i) y[e][i] += z[e][i];
        }
        float sh[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float m = PCX_NEG_INF;
#pragma unroll
            for (int s = 0; s < 2; ++s)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const bool ok = s < t.n_strips && in;
                    f[s][h][i] = ok ? flow_over_value(f[s][h][i], v[s][h][i], a.logspace) : PCX_NEG_INF;
                    m = fmaxf(m, f[s][h][i]);
                }
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 4));
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 8));
            sh[i] = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 16));
        }
        uint4 ah[2], al[2];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            float q[2][4];
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int i = 0; i < 4; ++i) q[h][i] = fast_exp(f[s][h][i] - (sh[i] == PCX_NEG_INF ? 0.0f : sh[i]));
            split2(q[0][0], q[0][1], ah[s].x, al[s].x);
            split2(q[1][0], q[1][1], ah[s].y, al[s].y);
            split2(q[0][2], q[0][3], ah[s].z, al[s].z);
            split2(q[1][2], q[1][3], ah[s].w, al[s].w);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
#pragma unroll
            for (int i = 0; i < 4; ++i) y[e][i] = fminf(fast_exp(y[e][i] + sh[i]), 3.0e38f);
            uint32_t bh0, bl0, bh1, bl1;
            split2(y[e][0], y[e][1], bh0, bl0);
            split2(y[e][2], y[e][3], bh1, bl1);
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                mma16816(acc[s][e], ah[s], bh0, bh1);
                if (a.terms == 3) {
                    mma16816(acc[s][e], ah[s], bl0, bl1);
                    mma16816(acc[s][e], al[s], bh0, bh1);
                }
            }
        }
    }
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        if (s >= t.n_strips) break;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if ((e >> 1) < t.n_k) {
                const int2 at = __ldg(a.pp + t.pp_off + (e >> 1) * t.n_strips + s);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int o = ((e & 1) * 8 + 2 * tq + (c & 1)) * t.bs + g + (c >> 1) * 8;
                    const float x = __ldg(a.params + at.x + o) * acc[s][e][c];
                    if (x != 0.0f) atomicAdd(a.pf + at.y + o, x);
                }
            }
        }
    }
}

__global__ void __launch_bounds__(256, 2) column_par_mma_kernel(const ColParArgs a) {
    const int item = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (item >= a.n_jobs * a.splits) return;
    const int split = item / a.n_jobs, job = item - split * a.n_jobs;
    const PcxColPar t = a.jobs[job];
    const int b_begin = split * a.per_split, b_end = min(a.W, b_begin + a.per_split);
    par_mma_tile(a, t, b_begin, b_end);
}

// The same tiles with their operands copied ahead through shared memory (see column_pipe_kernel): MS strips of 16 nodes x NE
// steps of 16 edges per warp, 16 samples per stage, two stages.  What bounds a tile is what it reads: 64 x 64 tiles read half
// of what 32 x 32 tiles do (12 M edges, 512 samples: 773 us with 32 x 32 tiles in registers).
template <int MS, int NE>
struct ParPipe {
    static constexpr int STAGE = (2 * MS + 2 * NE) * 1024;
    static constexpr int WARPS = (MS == 4) ? 6 : 12;
    static constexpr int SMEM = WARPS * 2 * STAGE;
};

__device__ __forceinline__ void par_copy(uint32_t dst, const float* rows, int64_t W, int b0, int b_end) {
    const int lane = threadIdx.x & 31, b = b0 + (lane & 3) * 4;
    const float* src = rows + (b < b_end ? b : b0);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int row = j * 8 + (lane >> 2);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + row * 64 + (lane & 3) * 16), "l"(src + row * W) : "memory");
    }
}

// Lane words of a job: 0 - 3 node rows of its strips, 4 - 11 rows of its edges (per step: child 0, child 1).
template <int MS, int NE>
__device__ __forceinline__ void par_request(const ColParArgs& a, int words, int n_strips, int n_k, int n_kids, int b0, int b_end,
                                            uint32_t buf) {
#pragma unroll
    for (int s = 0; s < MS; ++s) {
        const int64_t at = (int64_t)__shfl_sync(0xffffffffu, words, s) * a.W;
        if (s < n_strips) {
            par_copy(buf + (2 * s) * 1024, a.nf + at, a.W, b0, b_end);
            par_copy(buf + (2 * s + 1) * 1024, a.nm + at, a.W, b0, b_end);
        }
    }
    const float* ysrc = n_kids < 0 ? a.em : a.nm;
#pragma unroll
    for (int k = 0; k < NE; ++k) {
        const int64_t r0 = (int64_t)__shfl_sync(0xffffffffu, words, 4 + 2 * k) * a.W;
        const int64_t r1 = (int64_t)__shfl_sync(0xffffffffu, words, 5 + 2 * k) * a.W;
        if (k < n_k) {
            par_copy(buf + (2 * MS + 2 * k) * 1024, ysrc + r0, a.W, b0, b_end);
            if (n_kids == 2) par_copy(buf + (2 * MS + 2 * k + 1) * 1024, a.nm + r1, a.W, b0, b_end);
        }
    }
}
__device__ __forceinline__ void par_read(uint32_t group, int row, int tq, float* v) {
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(group + row * 64 + tq * 16));
}

template <int MS, int NE>
__global__ void __launch_bounds__(ParPipe<MS, NE>::WARPS * 32, 1) column_par_pipe_kernel(const ColParArgs a) {
    using C = ParPipe<MS, NE>;
    extern __shared__ __align__(128) uint8_t s_pipe[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(s_pipe) + warp * 2 * C::STAGE;
    const int items = a.n_jobs * a.splits;
    for (int item = blockIdx.x * C::WARPS + warp; item < items; item += gridDim.x * C::WARPS) {
        const int split = item / a.n_jobs, job = item - split * a.n_jobs;
        const PcxColPar* t = a.jobs + job;
        const int n_strips = __ldg(&t->n_strips), n_k = __ldg(&t->n_k), n_kids = __ldg(&t->n_kids), bs = __ldg(&t->bs);
        const int width = __ldg(&t->width);
        int words = 0;
        if (lane < 4) words = __ldg(&t->row0 + (lane < 2 ? lane : 8 + lane));          // row0, row1, row2, row3
        else if (lane < 4 + 2 * NE) {
            const int k = (lane - 4) >> 1, c = (lane - 4) & 1;
            words = __ldg(a.kids + __ldg(&t->kid_off) + (k < n_k ? k : 0) * width + (c < width ? c : 0));
        }
        const int b_begin = split * a.per_split, b_end = min(a.W, b_begin + a.per_split);
        float acc[MS][2 * NE][4];
#pragma unroll
        for (int s = 0; s < MS; ++s)
#pragma unroll
            for (int e = 0; e < 2 * NE; ++e)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[s][e][c] = 0.0f;
        int p = 0;
        par_request<MS, NE>(a, words, n_strips, n_k, n_kids, b_begin, b_end, base);
        asm volatile("cp.async.commit_group;" ::: "memory");
        for (int b0 = b_begin; b0 < b_end; b0 += 16) {
            const uint32_t buf = base + p * C::STAGE;
            if (b0 + 16 < b_end)
                par_request<MS, NE>(a, words, n_strips, n_k, n_kids, b0 + 16, b_end, base + (p ^ 1) * C::STAGE);
            asm volatile("cp.async.commit_group;" ::: "memory");
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncwarp();
            const bool in = b0 + 4 * tq < b_end;            // (lane t: samples 4t .. 4t+3, see par_mma_tile)
            float x[MS][2][4], sh[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) sh[i] = PCX_NEG_INF;
#pragma unroll
            for (int s = 0; s < MS; ++s)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (s < n_strips) {
                        float v[4];
                        par_read(buf + (2 * s) * 1024, g + 8 * h, tq, x[s][h]);
                        par_read(buf + (2 * s + 1) * 1024, g + 8 * h, tq, v);
#pragma unroll
                        for (int i = 0; i < 4; ++i) x[s][h][i] = in ? flow_over_value(x[s][h][i], v[i], a.logspace) : PCX_NEG_INF;
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; ++i) x[s][h][i] = PCX_NEG_INF;
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) sh[i] = fmaxf(sh[i], x[s][h][i]);
                }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                sh[i] = fmaxf(sh[i], __shfl_xor_sync(0xffffffffu, sh[i], 4));
                sh[i] = fmaxf(sh[i], __shfl_xor_sync(0xffffffffu, sh[i], 8));
                sh[i] = fmaxf(sh[i], __shfl_xor_sync(0xffffffffu, sh[i], 16));
            }
            uint4 ah[MS], al[MS];
#pragma unroll
            for (int s = 0; s < MS; ++s) {
                float q[2][4];
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int i = 0; i < 4; ++i) q[h][i] = fast_exp(x[s][h][i] - (sh[i] == PCX_NEG_INF ? 0.0f : sh[i]));
                split2(q[0][0], q[0][1], ah[s].x, al[s].x);
                split2(q[1][0], q[1][1], ah[s].y, al[s].y);
                split2(q[0][2], q[0][3], ah[s].z, al[s].z);
                split2(q[1][2], q[1][3], ah[s].w, al[s].w);
            }
#pragma unroll
            for (int e = 0; e < 2 * NE; ++e) {
                if ((e >> 1) < n_k) {
                    float y[4];
                    const int row = g + 8 * (e & 1);
                    par_read(buf + (2 * MS + (e & ~1)) * 1024, row, tq, y);
                    if (n_kids == 2) {
                        float z[4];
                        par_read(buf + (2 * MS + (e & ~1) + 1) * 1024, row, tq, z);
#pragma unroll
                        for (int i = 0; i < 4; ++i) y[i] += z[i];
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) y[i] = fminf(fast_exp(y[i] + sh[i]), 3.0e38f);
                    uint32_t bh0, bl0, bh1, bl1;
                    split2(y[0], y[1], bh0, bl0);
                    split2(y[2], y[3], bh1, bl1);
#pragma unroll
                    for (int s = 0; s < MS; ++s) {
                        mma16816(acc[s][e], ah[s], bh0, bh1);
                        if (a.terms == 3) {
                            mma16816(acc[s][e], ah[s], bl0, bl1);
                            mma16816(acc[s][e], al[s], bh0, bh1);
                        }
                    }
                }
            }
            __syncwarp();
            p ^= 1;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        const int pp_off = __ldg(&t->pp_off);
#pragma unroll
        for (int s = 0; s < MS; ++s) {
            if (s < n_strips) {
#pragma unroll
                for (int e = 0; e < 2 * NE; ++e) {
                    if ((e >> 1) < n_k) {
                        const int2 at = __ldg(a.pp + pp_off + (e >> 1) * n_strips + s);
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            const int o = ((e & 1) * 8 + 2 * tq + (c & 1)) * bs + g + (c >> 1) * 8;
                            const float f = __ldg(a.params + at.x + o) * acc[s][e][c];
                            if (f != 0.0f) atomicAdd(a.pf + at.y + o, f);
                        }
                    }
                }
            }
        }
    }
}

// fp32 tiles for blocks under 32 nodes: a warp owns up to 16 nodes x 64 edges; 32 samples at a time go through the
// warp's shared memory (lane = sample), then a lane multiplies RLN rows x ELN edges.
constexpr int PS_LD = 36;                                  // row pitch: 16-byte aligned, rows 4 banks apart
constexpr int PS_ROWS = 16 + 64;
constexpr int PS_WARPS = 4;

template <int RG, int RLN>
__device__ void par_simt_tile(const ColParArgs& a, const PcxColPar& t, int b_begin, int b_end, float* sx, float* sy) {
    constexpr int EG = 32 / RG, ELN = 64 / EG;
    const int lane = threadIdx.x & 31, rg = lane % RG, eg = lane / RG;
    float acc[RLN][ELN];
#pragma unroll
    for (int r = 0; r < RLN; ++r)
#pragma unroll
        for (int e = 0; e < ELN; ++e) acc[r][e] = 0.0f;
    const int n_used = (t.n_k + EG - 1) / EG;              // edges per lane that exist
    const int oct = t.lg_entry == 3 ? 7 : 0;
    const int nk = t.n_kids < 0 ? 1 : t.n_kids;
    const float* ysrc = t.n_kids < 0 ? a.em : a.nm;
    for (int b0 = b_begin; b0 < b_end; b0 += 32) {
        const bool in = b0 + lane < b_end;
        const int64_t b = in ? b0 + lane : b_begin;
        float x[RG * RLN], v[RG * RLN], m = PCX_NEG_INF;
#pragma unroll
        for (int r = 0; r < RG * RLN; ++r) {
            const int64_t at = (int64_t)(t.row0 + r) * a.W + b;
            x[r] = ldv(a.nf + at);
            v[r] = ldv(a.nm + at);
        }
#pragma unroll
        for (int r = 0; r < RG * RLN; ++r) {
            x[r] = in ? flow_over_value(x[r], v[r], a.logspace) : PCX_NEG_INF;
            m = fmaxf(m, x[r]);
        }
#pragma unroll
        for (int r = 0; r < RG * RLN; ++r) sx[r * PS_LD + lane] = (m == PCX_NEG_INF) ? 0.0f : expf(x[r] - m);
        for (int k0 = 0; k0 < t.n_k; k0 += 8) {
            float y[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) y[i] = 0.0f;
            for (int c = 0; c < nk; c += 2) {              // two children of eight edges: sixteen rows requested together
                float u[8], w[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int k = min(k0 + i, t.n_k - 1);
                    const int32_t* ent = a.kids + t.kid_off + (k >> t.lg_entry) * t.width + c;
                    const int off = k & oct;
                    u[i] = ldv(ysrc + (int64_t)(__ldg(ent) + off) * a.W + b);
                    w[i] = c + 1 < nk ? ldv(ysrc + (int64_t)(__ldg(ent + 1) + off) * a.W + b) : 0.0f;
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) y[i] += u[i] + w[i];
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (k0 + i < t.n_k)
                    sy[(k0 + i) * PS_LD + lane] = (m == PCX_NEG_INF) ? 0.0f : fminf(expf(y[i] + m), 3.0e38f);
        }
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            float4 xr[RLN];
#pragma unroll
            for (int r = 0; r < RLN; ++r) xr[r] = *reinterpret_cast<const float4*>(sx + (r * RG + rg) * PS_LD + 4 * q);
#pragma unroll
            for (int e = 0; e < ELN; ++e) {
                if (e < n_used) {
                    const float4 ye = *reinterpret_cast<const float4*>(sy + (e * EG + eg) * PS_LD + 4 * q);
#pragma unroll
                    for (int r = 0; r < RLN; ++r)
                        acc[r][e] += xr[r].x * ye.x + xr[r].y * ye.y + xr[r].z * ye.z + xr[r].w * ye.w;
                }
            }
        }
        __syncwarp();
    }
#pragma unroll
    for (int e = 0; e < ELN; ++e) {
        const int k = e * EG + eg;
        if (k < t.n_k) {
            const int2 at = __ldg(a.pp + t.pp_off + (k >> t.lg_entry));
#pragma unroll
            for (int r = 0; r < RLN; ++r) {
                const int o = (k & oct) * t.bs + r * RG + rg;
                const float f = __ldg(a.params + at.x + o) * acc[r][e];
                if (f != 0.0f) atomicAdd(a.pf + at.y + o, f);
            }
        }
    }
}

__global__ void __launch_bounds__(PS_WARPS * 32) column_par_simt_kernel(const ColParArgs a) {
    __shared__ __align__(16) float s_tile[PS_WARPS][PS_ROWS * PS_LD];
    const int warp = threadIdx.x >> 5;
    const int item = blockIdx.x * PS_WARPS + warp;
    if (item >= a.n_jobs * a.splits) return;
    const int split = item / a.n_jobs, job = item - split * a.n_jobs;
    const PcxColPar t = a.jobs[job];
    const int b_begin = split * a.per_split, b_end = min(a.W, b_begin + a.per_split);
    float* sx = s_tile[warp];
    float* sy = sx + 16 * PS_LD;
    if (t.n_strips == 1) par_simt_tile<1, 1>(a, t, b_begin, b_end, sx, sy);
    else if (t.n_strips == 2) par_simt_tile<2, 1>(a, t, b_begin, b_end, sx, sy);
    else if (t.n_strips == 4) par_simt_tile<4, 1>(a, t, b_begin, b_end, sx, sy);
    else if (t.n_strips == 8) par_simt_tile<4, 2>(a, t, b_begin, b_end, sx, sy);
    else par_simt_tile<4, 4>(a, t, b_begin, b_end, sx, sy);
}

template <int MS, int NE>
int launch_par_pipe(const ColParArgs& a, cudaStream_t st) {
    using C = ParPipe<MS, NE>;
    static PcxOnce done;
    if (!done) {
        cudaError_t e = cudaFuncSetAttribute(column_par_pipe_kernel<MS, NE>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
        if (e != cudaSuccess) return (int)e;
        done = true;
    }
    const int64_t ctas = pcx_cdiv((int64_t)a.n_jobs * a.splits, C::WARPS);
    column_par_pipe_kernel<MS, NE><<<(unsigned)std::min<int64_t>(148, ctas), C::WARPS * 32, C::SMEM, st>>>(a);
    PCX_LAUNCH_CHECK();
    return 0;
}

template <int MODE, int NT>
cudaLaunchConfig_t column_config(int n_clusters, int cluster, cudaLaunchAttribute* attr, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(n_clusters * cluster));
    cfg.blockDim = dim3(CT);
    cfg.stream = st;
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = cluster;
    attr->val.clusterDim.y = 1;
    attr->val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 1 : 0;
    return cfg;
}

template <int MODE, int NT>
int launch_column(const ColArgs& a, cudaStream_t st) {
    cudaLaunchAttribute attr;
    cudaLaunchConfig_t cfg = column_config<MODE, NT>((int)pcx_cdiv(a.W, 8 * NT), a.cluster, &attr, st);
    cudaError_t e = cudaLaunchKernelEx(&cfg, column_kernel<MODE, NT>, a);
    if (e != cudaSuccess) return (int)e;
    PCX_LAUNCH_CHECK();
    return 0;
}

// Shared memory of the CTA-task kernel: operand fragments of the deepest task, the rest for parameter fragments.
constexpr int BIG_TOTAL = 227 * 1024;

template <int MODE, int NT>
int big_setup() {
    static PcxOnce done;
    if (!done) {
        cudaError_t e = cudaFuncSetAttribute(column_big_kernel<MODE, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, BIG_TOTAL);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(column_big_kernel<MODE, NT>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return (int)e;
        done = true;
    }
    return 0;
}

template <int MODE, int NT>
int launch_big(const ColArgs& a, int max_steps, cudaStream_t st) {
    int rc = big_setup<MODE, NT>();
    if (rc != 0) return rc;
    cudaLaunchAttribute attr;
    cudaLaunchConfig_t cfg = column_config<MODE, NT>((int)pcx_cdiv(a.W, 8 * NT), a.cluster, &attr, st);
    cfg.dynamicSmemBytes = BIG_TOTAL;
    const int b_bytes = max_steps * NT * 512;
    const int a_bytes = (BIG_TOTAL - BigSmem<NT>::FIXED - b_bytes) & ~1023;
    cudaError_t e = cudaLaunchKernelEx(&cfg, column_big_kernel<MODE, NT>, a, a_bytes, b_bytes);
    if (e != cudaSuccess) return (int)e;
    PCX_LAUNCH_CHECK();
    return 0;
}

template <int MODE>
int launch_column_nt(const ColArgs& a, int nt, cudaStream_t st) {
    if (a.wide == 1) {
        column_wide_kernel<MODE><<<148, WT, 0, st>>>(a);
        PCX_LAUNCH_CHECK();
        return 0;
    }
    if (a.wide == 2) {
        static PcxOnce done;
        if (!done) {
            cudaError_t e = cudaFuncSetAttribute(column_pipe_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, PIPE_SMEM);
            if (e != cudaSuccess) return (int)e;
            done = true;
        }
        column_pipe_kernel<MODE><<<148, WT, PIPE_SMEM, st>>>(a);
        PCX_LAUNCH_CHECK();
        return 0;
    }
    if (a.wide == 3) {
        column_prod_kernel<<<148 * 8, 256, 0, st>>>(a);
        PCX_LAUNCH_CHECK();
        return 0;
    }
    if (nt == 1) return launch_column<MODE, 1>(a, st);
    return launch_column<MODE, 2>(a, st);
}

}  // namespace

extern "C" {

int pcx_column_clusters(int cluster, int big) {
    if (cluster < 1 || cluster > (big ? 16 : 8)) return -1;
    cudaLaunchAttribute attr;
    cudaLaunchConfig_t cfg = column_config<C_ELE, 2>(1, cluster, &attr, nullptr);
    int n = 0;
    if (cluster == 1) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -1;
        return n;
    }
    cudaError_t e;
    if (big) {
        if (big_setup<C_ELE, 2>() != 0) return -1;
        cfg.dynamicSmemBytes = BIG_TOTAL;
        e = cudaOccupancyMaxActiveClusters(&n, column_big_kernel<C_ELE, 2>, &cfg);
    } else {
        e = cudaOccupancyMaxActiveClusters(&n, column_kernel<C_ELE, 2>, &cfg);
    }
    if (e != cudaSuccess) { cudaGetLastError(); return -1; }
    return n;
}

int pcx_column_run_big(int mode, float* node_mars, float* node_flows, float* element_flows, float* element_values,
                       const float* params, const void* frags, const PcxColTask* tasks, const int32_t* kids,
                       const int32_t* strips, const int32_t* levels, int n_levels, int W, int nt, int cluster, int max_steps,
                       int logspace, int terms, void* stream) {
    if (n_levels <= 0 || W <= 0) return 0;
    if (W % 8 != 0 || (nt != 1 && nt != 2) || cluster < 1 || cluster > 16 || (mode != 0 && mode != 1)) return -1;
    if (n_levels > MAX_LEVELS || max_steps < 1 || max_steps > BIG_MAX_STEPS) return -1;
    if (((reinterpret_cast<uintptr_t>(node_mars) | reinterpret_cast<uintptr_t>(node_flows) |
          reinterpret_cast<uintptr_t>(element_flows) | reinterpret_cast<uintptr_t>(element_values)) & 15) != 0) return -1;
    ColArgs a{};
    a.nm = node_mars; a.nf = node_flows; a.ef = element_flows; a.em = element_values; a.params = params;
    a.frags = reinterpret_cast<const uint4*>(frags); a.tasks = tasks; a.kids = kids;
    a.strips = reinterpret_cast<const int4*>(strips); a.levels = reinterpret_cast<const int4*>(levels);
    a.n_levels = n_levels; a.W = W; a.logspace = logspace; a.terms = terms; a.cluster = cluster; a.tiles = 1;
    cudaStream_t st = (cudaStream_t)stream;
    if (mode == 0) return nt == 1 ? launch_big<C_FWD, 1>(a, max_steps, st) : launch_big<C_FWD, 2>(a, max_steps, st);
    return nt == 1 ? launch_big<C_ELE, 1>(a, max_steps, st) : launch_big<C_ELE, 2>(a, max_steps, st);
}

int pcx_column_run(int mode, float* node_mars, float* node_flows, float* element_flows, float* element_values,
                   const float* params, const void* frags, const PcxColTask* tasks, const int32_t* kids,
                   const int32_t* strips, const int32_t* levels, int n_levels, int W, int nt, int tiles, int cluster,
                   int wide, int logspace, int terms, void* stream) {
    if (n_levels <= 0 || W <= 0) return 0;
    if (n_levels > MAX_LEVELS) return -1;
    if (wide < 0 || wide > 3 || (wide == 3 && mode == 0) || (wide > 0 && (n_levels != 1 || nt != 4 || tiles != (int)pcx_cdiv(W, 8 * nt)))) return -1;
    if (W % 8 != 0 || (nt != 1 && nt != 2 && !(nt == 4 && wide > 0)) || cluster < 1 || cluster > 8 || (mode != 0 && mode != 1)) return -1;
    if (wide == 0 && tiles != 1) return -1;
    if (((reinterpret_cast<uintptr_t>(node_mars) | reinterpret_cast<uintptr_t>(node_flows) |
          reinterpret_cast<uintptr_t>(element_flows) | reinterpret_cast<uintptr_t>(element_values)) & 15) != 0) return -1;
    ColArgs a{};
    a.nm = node_mars; a.nf = node_flows; a.ef = element_flows; a.em = element_values; a.params = params;
    a.frags = reinterpret_cast<const uint4*>(frags); a.tasks = tasks; a.kids = kids;
    a.strips = reinterpret_cast<const int4*>(strips); a.levels = reinterpret_cast<const int4*>(levels);
    a.n_levels = n_levels; a.W = W; a.logspace = logspace; a.terms = terms; a.cluster = cluster; a.tiles = tiles; a.wide = wide;
    return mode == 0 ? launch_column_nt<C_FWD>(a, nt, (cudaStream_t)stream) : launch_column_nt<C_ELE>(a, nt, (cudaStream_t)stream);
}

int pcx_column_pack(void* frags, const int32_t* bases, int64_t n, const float* params, void* stream) {
    if (n <= 0) return 0;
    column_pack_kernel<<<(unsigned)pcx_cdiv(n, 8), 256, 0, (cudaStream_t)stream>>>(
        reinterpret_cast<uint4*>(frags), reinterpret_cast<const int4*>(bases), n, params);
    PCX_LAUNCH_CHECK();
    return 0;
}

int pcx_column_par(int kind, float* param_flows, const float* node_flows, const float* node_mars,
                   const float* element_values, const float* params, const PcxColPar* jobs, const int32_t* kids,
                   const int32_t* offsets, int n_jobs, int W, int logspace, int terms, void* stream) {
    if (n_jobs <= 0 || W <= 0) return 0;
    if (W % 8 != 0 || kind < 0 || kind > 3) return -1;
    ColParArgs a{};
    a.pf = param_flows; a.nf = node_flows; a.nm = node_mars; a.em = element_values; a.params = params; a.jobs = jobs;
    a.kids = kids; a.pp = reinterpret_cast<const int2*>(offsets); a.n_jobs = n_jobs; a.W = W; a.logspace = logspace;
    a.terms = terms;
    // The batch is cut until every warp slot of the machine has two rounds, but not into pieces under 32 samples: each piece
    // pays an atomic per parameter.
    const int step = 32, warps[4] = {16, 20, 12, 6};
    const int pieces = (int)pcx_cdiv(W, step);
    const int want = (int)std::max<int64_t>(1, pcx_cdiv((int64_t)148 * warps[kind] * 2, n_jobs));
    a.per_split = (int)pcx_cdiv(pieces, std::min(pieces, want)) * step;
    a.splits = (int)pcx_cdiv(W, a.per_split);
    const int64_t items = (int64_t)n_jobs * a.splits;
    if (items > INT32_MAX) return -1;
    if (kind == 2) return launch_par_pipe<2, 2>(a, (cudaStream_t)stream);
    if (kind == 3) return launch_par_pipe<4, 4>(a, (cudaStream_t)stream);
    if (kind == 0) column_par_mma_kernel<<<(unsigned)pcx_cdiv(items, 8), 256, 0, (cudaStream_t)stream>>>(a);
    else column_par_simt_kernel<<<(unsigned)pcx_cdiv(items, PS_WARPS), PS_WARPS * 32, 0, (cudaStream_t)stream>>>(a);
    PCX_LAUNCH_CHECK();
    return 0;
}

}  // extern "C"
