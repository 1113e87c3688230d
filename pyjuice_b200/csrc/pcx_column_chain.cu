// Chains of the column program: consecutive levels of ONE dense group each, all with the same (tied) parameters and each
// reading the level before it -- the transitions of a homogeneous hidden Markov model -- in one launch.
//
// A cluster of C CTAs owns 8 * NT columns, as in pcx_column.cu, and every CTA the same `per` strips of 16 rows of every level,
// so that a CTA needs the same parameter fragments at every level: they are read once per launch and stay on the SM.  A
// quarter megabyte of tensor memory holds the first 256 fragments of a CTA (a warp reads its own lanes and columns with
// tcgen05.ld: 256 KB take 350 cycles, where shared memory takes 2000), shared memory the next ones, and only what is left
// comes from L2 at every level (1024 x 1024 on eight CTAs: 128 of 512).
//
// What a level costs is a chain of latencies, and the CTA tasks of pcx_column.cu, which this replaces, had these in it, of
// 9700 cycles for 512 x 512 and eight columns: gather of two operand rows per child and their maximum 3100, exponentials and
// split 900 (every CTA of the cluster formed those of all children), multiplications 1970 (bound by the shared memory that
// the fragments were read from), epilogue 1170 and the next task's look-ahead 850, and the cluster barrier 1620.  Here the CTA
// that owns a row adds the value of the element's other child to it, forms the exponential, splits it and stores it in the
// order of the B fragment; a warp of the next level reads 16-byte words that ARE its operand.  Exponentials are relative to
// the maximum of the CTA's own rows (nobody waits for a maximum over all CTAs), and the partial products of a CTA's rows are
// scaled where the parts of the contraction are added up.  4450 cycles a level now (512 x 512, eight columns, eight CTAs of four
// strips): from a CTA's stores to the operands in the others' registers 1600, scales of the parts 300, multiplications 1200, parts
// through shared memory and their sum 650, maximum over the CTA's strips, exponential, split and store 700.  With more columns
// and rows a CTA the multiplications take over: 1024 x 1024, 24 columns, 16 CTAs of four strips 7000 of 15 400.
// Microseconds a level, before / now (forward passes over 64 tokens, leaves and launches included): 128 states, 64 columns 3.5 /
// 2.0; 256, 64 4.3 / 2.3; 512, 77 5.6 / 2.8; 512, 256 6.9 / 3.9; 1024, 64 10.0 / 5.2; 1024, 128 12.9 / 8.8.
//
//   warp (kp, ws)   strips ws * strips_w .. of the CTA, children of part kp of the contraction (parts never cross the rows of
//                   two CTAs, so each has one scale).  Two warps share a part where the CTAs are few: half the partial products.
//   epilogue        a warp per (strip, tile of eight columns): adds the parts in order, logarithm, the element's other child,
//                   maximum over the CTA's strips (named barrier), exponential, split, store; only then the stores of the
//                   level's values or flows, which nobody in this launch reads.
#include <algorithm>
#include "pcx_column_ops.cuh"
#include "pcx_tc.cuh"
#include "../../include/pcx_b200.h"

namespace {

using namespace pcx_tc;

constexpr int CHAIN_THREADS = 512;
constexpr int CHAIN_WARPS = CHAIN_THREADS / 32;
constexpr int CHAIN_SMEM = 227 * 1024 - 1024;             // dynamic shared memory
constexpr int CHAIN_TMEM = 16;                            // fragments per warp in tensor memory

struct ChainArgs {
    float* nm;                  // node_mars  [rows, W]
    float* nf;                  // node_flows [rows, W] (element flows)
    const uint4* frags;
    uint4* operand;             // [2][clusters][S][NT][32]: B fragments of one level and the next
    uint4* shifts;              // [2][clusters][C][NT][4]: maxima of each CTA's rows, two columns a word, each with its own mark
    const int2* rows;           // [levels + 1][S]: see pcx_column_chain
    const int2* strips;         // [S]: first fragment of a strip, fragments per step
    int* status;                // the library's status word
    int n_levels;
    int S;                      // strips of 16 rows, steps of 16 children
    int per;                    // strips per CTA
    int C;                      // CTAs per cluster
    int q;                      // parts of the contraction per CTA whose rows it multiplies
    int steps;                  // steps per part
    int W;
    int terms;
    int strips_w;               // strips per warp
    int halves;                 // warps that share a part of the contraction (each has its strips)
    int smem_steps;             // steps per warp with fragments in shared memory
};

// Shared memory: scales [warp][part][8], maxima [tile][column][strip], partial products [2][part][strip][tile], fragments.
constexpr int CHAIN_SCALE = CHAIN_WARPS * 16 * 8 * 4;
constexpr int CHAIN_MAX = 3 * 8 * 8 * 4;
constexpr int CHAIN_FIXED = CHAIN_SCALE + CHAIN_MAX;

// Four registers per lane (the high or low part of a fragment) to tensor memory, and N such parts back.
__device__ __forceinline__ void tmem_store(uint32_t addr, const uint4& v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
template <int N>
__device__ __forceinline__ void tmem_load(uint32_t addr, uint4* v) {
    static_assert(N == 2 || N == 4 || N == 8, "parts of fragments");
    if constexpr (N == 8)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                     "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                     : "=r"(v[0].x), "=r"(v[0].y), "=r"(v[0].z), "=r"(v[0].w), "=r"(v[1].x), "=r"(v[1].y), "=r"(v[1].z), "=r"(v[1].w),
                       "=r"(v[2].x), "=r"(v[2].y), "=r"(v[2].z), "=r"(v[2].w), "=r"(v[3].x), "=r"(v[3].y), "=r"(v[3].z), "=r"(v[3].w),
                       "=r"(v[4].x), "=r"(v[4].y), "=r"(v[4].z), "=r"(v[4].w), "=r"(v[5].x), "=r"(v[5].y), "=r"(v[5].z), "=r"(v[5].w),
                       "=r"(v[6].x), "=r"(v[6].y), "=r"(v[6].z), "=r"(v[6].w), "=r"(v[7].x), "=r"(v[7].y), "=r"(v[7].z), "=r"(v[7].w) : "r"(addr));
    else if constexpr (N == 2)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(v[0].x), "=r"(v[0].y), "=r"(v[0].z), "=r"(v[0].w), "=r"(v[1].x), "=r"(v[1].y), "=r"(v[1].z), "=r"(v[1].w) : "r"(addr));
    else
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                     : "=r"(v[0].x), "=r"(v[0].y), "=r"(v[0].z), "=r"(v[0].w), "=r"(v[1].x), "=r"(v[1].y), "=r"(v[1].z), "=r"(v[1].w),
                       "=r"(v[2].x), "=r"(v[2].y), "=r"(v[2].z), "=r"(v[2].w), "=r"(v[3].x), "=r"(v[3].y), "=r"(v[3].z), "=r"(v[3].w) : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < N; ++i) asm volatile("" : "+r"(v[i].x), "+r"(v[i].y), "+r"(v[i].z), "+r"(v[i].w));
}

// ---- words that say whether they are there -------------------------------------------------------------------------------
// A level's operand goes to the other CTAs of the cluster through L2, in 16-byte words that are written and read as one
// (128-bit relaxed accesses).  The first 32 bits of a word hold the high parts of two exponentials (or a zero), which are not
// negative: their sign bits say in which round the word was written.  A buffer is written every second level, and nobody writes
// it again before all have read it (a CTA sends the next level only after it has read this one), so that one bit is enough.
// A reader asks for the words themselves and asks again for those that are not there.  The other ways, cycles from a CTA's last
// store to the operands in the others' registers, 512 rows of eight columns: store, cluster barrier (which waits for the
// store to reach L2), load: 2150; stores into every CTA's shared memory with a transaction barrier: these go at 16 bytes a
// cycle, 1000 cycles for 512 rows and 2000 for 1024, before the last one can start; this: 1500, and 64 bytes a cycle.
__device__ __forceinline__ uint4 load_word(const uint4* p) {
    uint64_t x, y;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}" : "=l"(x), "=l"(y) : "l"(p) : "memory");
    return make_uint4((uint32_t)x, (uint32_t)(x >> 32), (uint32_t)y, (uint32_t)(y >> 32));
}
__device__ __forceinline__ uint2 load_half(const uint4* p, int half) {
    uint2 v;
    asm volatile("{\n\t.reg .b64 t;\n\tld.relaxed.gpu.global.b64 t, [%2];\n\tmov.b64 {%0, %1}, t;\n\t}" : "=r"(v.x), "=r"(v.y) : "l"(reinterpret_cast<const uint2*>(p) + half) : "memory");
    return v;
}
__device__ __forceinline__ void store_word(uint4* p, const uint4& v) {
    const uint64_t x = (uint64_t)v.y << 32 | v.x, y = (uint64_t)v.w << 32 | v.z;
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%0, %1};\n\tst.relaxed.gpu.global.b128 [%2], t;\n\t}" ::"l"(x), "l"(y), "l"(p) : "memory");
}
constexpr uint32_t CHAIN_ROUND = 0x80008000u;             // the bits of an odd round
__device__ __forceinline__ bool here(uint32_t word, uint32_t round) { return (int)(word ^ round) >= 0; }
constexpr int CHAIN_POLLS = 1 << 20;

template <int MODE, int NT, int PS>
__global__ void __launch_bounds__(CHAIN_THREADS, 1) column_chain_kernel(const ChainArgs a) {
    constexpr int KT = CHAIN_TMEM / PS;                   // steps with fragments in tensor memory
    constexpr int AC = PS * NT <= 2 ? 3 : 1;              // accumulators of a strip and tile: short tables wait for the latency of a product
    constexpr bool SPLIT = PS * NT >= 8;                  // low parts fetched once the high ones are done with: registers
    constexpr int KB = NT == 1 ? (PS == 4 ? 2 : 4) : (NT == 2 && PS < 4 ? 2 : 1);   // steps whose operands are requested together
    extern __shared__ __align__(128) uint8_t s_chain[];
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_fail;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
    const int rank = blockIdx.x % a.C, group = blockIdx.x / a.C, groups = gridDim.x / a.C;
    const int col0 = group * 8 * NT, S = a.S, W = a.W;
    const int s0 = rank * a.per, n_s = min(a.per, S - s0);
    const int ws = warp % a.halves, kp = warp / a.halves;
    // this warp's part of the contraction and its strips
    const int from = min(kp / a.q, a.C - 1), parts = a.C * a.q, k_begin = min(S, from * a.per + (kp % a.q) * a.steps);
    const int n_k = kp < parts ? max(0, min(min(S, (from + 1) * a.per), k_begin + a.steps) - k_begin) : 0;
    const int first = ws * a.strips_w, n_p = max(0, min(a.strips_w, n_s - first));

    float* s_scale = reinterpret_cast<float*>(s_chain) + warp * 128;
    float* s_max = reinterpret_cast<float*>(s_chain + CHAIN_SCALE);
    float4* s_part = reinterpret_cast<float4*>(s_chain + CHAIN_FIXED);
    uint4* s_frag = reinterpret_cast<uint4*>(s_chain + CHAIN_FIXED + 2 * parts * a.per * NT * 512) + warp * a.smem_steps * PS * 64;

    // ---- once per launch: parameters; what the exchange buffers hold of the launch before is marked as not there ------------
    const int operand_buf = groups * S * NT * 32, shift_buf = groups * a.C * NT * 4;        // words of one level
    if (warp == 0) tmem_alloc(&s_tmem, 512);
    if (threadIdx.x < CHAIN_MAX / 4) s_max[threadIdx.x] = PCX_NEG_INF;        // (strips that the CTA lacks)
    if (threadIdx.x == 0) s_fail = 0;
    const uint4 none = make_uint4(CHAIN_ROUND, 0u, CHAIN_ROUND, 0u);
    for (int i = threadIdx.x; i < 2 * n_s * NT * 32; i += CHAIN_THREADS) {
        const int buf = i / (n_s * NT * 32), at = i - buf * (n_s * NT * 32);
        store_word(a.operand + buf * operand_buf + (group * S + s0) * NT * 32 + at, none);
    }
    if (threadIdx.x < 2 * NT * 4)
        store_word(a.shifts + (threadIdx.x / (NT * 4)) * shift_buf + (group * a.C + rank) * NT * 4 + threadIdx.x % (NT * 4), none);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    const uint32_t tmem = s_tmem + ((uint32_t)(warp & 3) << 21) + (warp >> 2) * (CHAIN_TMEM * 8);
    auto fragment = [&](int k, int p) {                   // of this warp's step k and strip p (strips that it lacks: the last)
        const int2 f = __ldg(a.strips + s0 + min(first + p, n_s - 1));
        return a.frags + ((int64_t)f.x + (int64_t)(k_begin + k) * f.y) * 64 + lane;
    };
    for (int k = 0; k < min(n_k, KT + a.smem_steps); ++k) {
#pragma unroll
        for (int p = 0; p < PS; ++p) {
            const uint4* f = fragment(k, p);
            const uint4 h = __ldg(f), l = __ldg(f + 32);
            if (k < KT) {
                tmem_store(tmem + (2 * k * PS + p) * 4, h);       // [step][part][strip]
                tmem_store(tmem + ((2 * k + 1) * PS + p) * 4, l);
            } else {
                s_frag[((k - KT) * PS + p) * 64 + lane] = h;
                s_frag[((k - KT) * PS + p) * 64 + 32 + lane] = l;
            }
        }
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");

    // ---- results of a strip and tile ---------------------------------------------------------------------------------------
    const bool fin = warp < n_s * NT;
    const int strip = warp / NT, tile = warp % NT;
    const int col = col0 + 8 * tile + 2 * tq;
    const bool live = fin && col0 + 8 * tile < W;         // (W is a multiple of 8)
    const int2* rows = a.rows + s0 + (fin ? strip : 0);
    auto load2 = [&](const float* buf, int row, float (*v)[2]) {
#pragma unroll
        for (int h = 0; h < 2; ++h) ldvec<2>(buf + (int64_t)(row + g + 8 * h) * W + col, v[h]);
    };
    auto store2 = [&](float* buf, int row, const float (*v)[2]) {
#pragma unroll
        for (int h = 0; h < 2; ++h) stvec<2>(buf + (int64_t)(row + g + 8 * h) * W + col, v[h]);
    };
    const int out = ((group * S + s0 + strip) * NT + tile) * 32 + (2 * tq + (g & 1)) * 4 + (g >> 1);
    const int shift_out = ((group * a.C + rank) * NT + tile) * 4 + tq;
    // Operand values v (rows g, g + 8; columns 2 tq, 2 tq + 1) of a level go to all CTAs as exponentials.
    auto publish = [&](const float (*v)[2], int level) {
        float m[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            m[j] = fmaxf(v[0][j], v[1][j]);
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) m[j] = fmaxf(m[j], __shfl_xor_sync(0xffffffffu, m[j], o));
        }
        if (n_s > 1) {
            if (g < 2) s_max[(tile * 8 + 2 * tq + g) * 8 + strip] = g == 0 ? m[0] : m[1];
            asm volatile("bar.sync %0, %1;" ::"r"(1 + tile), "r"(32 * n_s) : "memory");
            const float4* all = reinterpret_cast<const float4*>(s_max + (tile * 8 + 2 * tq) * 8);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float4 x = all[2 * j];
                m[j] = fmaxf(fmaxf(x.x, x.y), fmaxf(x.z, x.w));
                if (n_s > 4) {
                    const float4 z = all[2 * j + 1];
                    m[j] = fmaxf(m[j], fmaxf(fmaxf(z.x, z.y), fmaxf(z.z, z.w)));
                }
            }
        }
        float e[2][2], got[2];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int j = 0; j < 2; ++j) e[h][j] = fast_exp(v[h][j] - (m[j] == PCX_NEG_INF ? 0.0f : m[j]));
        // rows 2t, 2t + 1 of a column belong in one word: lanes of neighbouring rows trade columns
#pragma unroll
        for (int h = 0; h < 2; ++h) got[h] = __shfl_xor_sync(0xffffffffu, (g & 1) ? e[h][0] : e[h][1], 4);
        uint4 w;
        split2((g & 1) ? got[0] : e[0][0], (g & 1) ? e[0][1] : got[0], w.x, w.y);
        split2((g & 1) ? got[1] : e[1][0], (g & 1) ? e[1][1] : got[1], w.z, w.w);
        const uint32_t round = (level >> 1) & 1 ? CHAIN_ROUND : 0u;
        w.x = (w.x & ~CHAIN_ROUND) | round;
        store_word(a.operand + out + (level & 1) * operand_buf, w);
        if (strip == 0 && g == 0)
            store_word(a.shifts + shift_out + (level & 1) * shift_buf, make_uint4(round, __float_as_uint(m[0]), round, __float_as_uint(m[1])));
    };

    int shift_in[4];                                      // shifts of the parts lane / 8 + 4 i, column lane % 8 of the tile
#pragma unroll
    for (int i = 0; i < 4; ++i)
        shift_in[i] = ((group * a.C + min(((lane >> 3) + 4 * i) / a.q, a.C - 1)) * NT + (fin ? tile : 0)) * 4 + ((lane & 7) >> 1);
    int2 row{}, row1{};
    float v0[2][2] = {}, y0[2][2] = {};
    if (fin) {
        row = __ldg(rows);
        row1 = __ldg(rows + S);
    }
    if (live) {
        load2(MODE == C_FWD ? a.nm : a.nf, row.x, v0);
        load2(a.nm, MODE == C_FWD ? row.y : row.x, y0);
    }
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (fin) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int j = 0; j < 2; ++j) v0[h][j] = MODE == C_FWD ? v0[h][j] + y0[h][j] : flow_over_value(v0[h][j], y0[h][j], 1);
        publish(v0, 0);
    }
    for (int l = 0; l < a.n_levels; ++l) {
        const uint32_t round = (l >> 1) & 1 ? CHAIN_ROUND : 0u;
        const bool more = l + 1 < a.n_levels;
        const uint4* op = a.operand + (l & 1) * operand_buf + (group * S + k_begin) * NT * 32 + lane;
        uint4 b[KB][NT], next[KB][NT];
        uint2 sh[4];
        auto request = [&](int k0, uint4 (*to)[NT]) {
#pragma unroll
            for (int k = 0; k < KB; ++k)
#pragma unroll
                for (int n = 0; n < NT; ++n)
                    if (k0 + k < n_k) to[k][n] = load_word(op + ((k0 + k) * NT + n) * 32);
        };
        auto settle = [&](int k0, uint4 (*to)[NT], bool shifts) {     // asks again for what is not there yet
            for (int polls = 0;; ++polls) {
                bool all = true;
                if (shifts)
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (!here(sh[i].x, round)) {
                            all = false;
                            sh[i] = load_half(a.shifts + shift_in[i] + (l & 1) * shift_buf, lane & 1);
                        }
#pragma unroll
                for (int k = 0; k < KB; ++k)
#pragma unroll
                    for (int n = 0; n < NT; ++n)
                        if (k0 + k < n_k && !here(to[k][n].x, round)) {
                            all = false;
                            to[k][n] = load_word(op + ((k0 + k) * NT + n) * 32);
                        }
                if (__all_sync(0xffffffffu, all)) break;
                if (__any_sync(0xffffffffu, polls >= CHAIN_POLLS || s_fail != 0)) { s_fail = 1; break; }
            }
        };
        request(0, b);
        if (fin)
#pragma unroll
            for (int i = 0; i < 4; ++i) sh[i] = load_half(a.shifts + shift_in[i] + (l & 1) * shift_buf, lane & 1);
        row = row1;
        if (fin && more) row1 = __ldg(rows + (l + 2) * S);
        float x[2][2] = {}, y[2][2] = {};                 // what the results are combined with
        if (live) {
            if (MODE == C_ELE) load2(a.nm, row.x, x);
            load2(a.nm, row.y, y);
        }
        float acc[AC][PS][NT][4];
#pragma unroll
        for (int i = 0; i < AC; ++i)
#pragma unroll
            for (int p = 0; p < PS; ++p)
#pragma unroll
                for (int n = 0; n < NT; ++n)
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[i][p][n][c] = 0.0f;
        settle(0, b, fin);
        float t0 = 0.0f, t1 = 0.0f;
        if (fin) {                                        // scales of the parts, while others multiply
            float m[4], top = PCX_NEG_INF;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                m[i] = (lane >> 3) + 4 * i < parts ? __uint_as_float(sh[i].y) : PCX_NEG_INF;
                top = fmaxf(top, m[i]);
            }
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 8));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 16));
#pragma unroll
            for (int i = 0; i < 4; ++i) s_scale[lane + 32 * i] = m[i] == PCX_NEG_INF ? 0.0f : fast_exp(m[i] - top);
            t0 = __shfl_sync(0xffffffffu, top, 2 * tq);
            t1 = __shfl_sync(0xffffffffu, top, 2 * tq + 1);
        }
        for (int k0 = 0; k0 < n_k; k0 += KB) {
            if (k0 + KB < n_k) request(k0 + KB, next);
#pragma unroll
            for (int kk = 0; kk < KB; ++kk) {
                const int k = k0 + kk;
                if (k < n_k) {
                    uint4 f[SPLIT ? 1 : 2][PS];            // high and low parts
                    auto fetch = [&](int lo) {
                        if (k < KT) {
                            tmem_load<SPLIT ? PS : 2 * PS>(tmem + (2 * k + lo) * PS * 4, f[0]);
                            return;
                        }
#pragma unroll
                        for (int i = 0; i < (SPLIT ? 1 : 2); ++i)
#pragma unroll
                            for (int p = 0; p < PS; ++p)
                                f[i][p] = k < KT + a.smem_steps ? s_frag[((k - KT) * PS + p) * 64 + 32 * (lo + i) + lane]
                                                                : __ldg(fragment(k, p) + 32 * (lo + i));
                    };
                    fetch(0);
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
                        const uint4 w = b[kk][n];          // hi, lo of rows 2t; hi, lo of rows 2t + 8
#pragma unroll
                        for (int p = 0; p < PS; ++p) mma16816(acc[0][p][n], f[0][p], w.x ^ round, w.z);
                        if (a.terms == 3)
#pragma unroll
                            for (int p = 0; p < PS; ++p) mma16816(acc[AC == 3 ? 1 : 0][p][n], f[0][p], w.y, w.w);
                    }
                    if (a.terms == 3) {
                        if (SPLIT) fetch(1);
#pragma unroll
                        for (int n = 0; n < NT; ++n)
#pragma unroll
                            for (int p = 0; p < PS; ++p) mma16816(acc[AC == 3 ? 2 : 0][p][n], f[SPLIT ? 0 : 1][p], b[kk][n].x ^ round, b[kk][n].z);
                    }
                }
            }
            if (k0 + KB < n_k) {
                settle(k0 + KB, next, false);
#pragma unroll
                for (int k = 0; k < KB; ++k)
#pragma unroll
                    for (int n = 0; n < NT; ++n) b[k][n] = next[k][n];
            }
        }
        // (two buffers: the level before may still be read)
        float4* parts_here = s_part + (l & 1) * parts * a.per * NT * 32;
        if (kp < parts) {
#pragma unroll
            for (int p = 0; p < PS; ++p)
                if (p < n_p)
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
                        if constexpr (AC == 3)
#pragma unroll
                            for (int c = 0; c < 4; ++c) acc[0][p][n][c] += acc[1][p][n][c] + acc[2][p][n][c];
                        parts_here[((kp * n_s + first + p) * NT + n) * 32 + lane] = 
                            make_float4(acc[0][p][n][0], acc[0][p][n][1], acc[0][p][n][2], acc[0][p][n][3]);
                    }
        }
        __syncthreads();
        if (fin) {
            float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            const float4* part = parts_here + (strip * NT + tile) * 32 + lane;
            const int step = n_s * NT * 32;
            for (int p0 = 0; p0 < parts; p0 += 8) {       // eight parts requested together; parts that do not exist have the scale 0
                float4 v[8];
                float2 sc[8];
#pragma unroll
                for (int p = 0; p < 8; ++p) {
                    v[p] = part[(p0 + p < parts ? p0 + p : 0) * step];
                    sc[p] = *reinterpret_cast<const float2*>(s_scale + (p0 + p) * 8 + 2 * tq);
                }
#pragma unroll
                for (int p = 0; p < 8; ++p) {
                    sum[0] = fmaf(v[p].x, sc[p].x, sum[0]);
                    sum[1] = fmaf(v[p].y, sc[p].y, sum[1]);
                    sum[2] = fmaf(v[p].z, sc[p].x, sum[2]);
                    sum[3] = fmaf(v[p].w, sc[p].y, sum[3]);
                }
            }
            float o[2][2], v[2][2];
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const float z = sum[2 * h + j];
                    // (an empty sum has the shift -inf, which stands for the result)
                    o[h][j] = fast_log_plus(MODE == C_FWD ? fmaxf(z, 1e-24f) : z, j == 0 ? t0 : t1);
                    if (MODE == C_FWD) {
                        v[h][j] = o[h][j] + y[h][j];
                    } else {
                        o[h][j] += x[h][j] + y[h][j];
                        v[h][j] = flow_over_value(o[h][j], x[h][j], 1);
                    }
                }
            if (more) publish(v, l + 1);
            if (more) asm volatile("bar.arrive 4, %0;" ::"n"(CHAIN_THREADS) : "memory");
            if (live) {
                store2(MODE == C_FWD ? a.nm : a.nf, row.x, o);
                if (MODE == C_ELE && row.y != 0) store2(a.nf, row.y, o);
            }
        } else if (more) {                                // (asks for the next level once this CTA has sent its part)
            asm volatile("bar.sync 4, %0;" ::"n"(CHAIN_THREADS) : "memory");
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    if (threadIdx.x == 0 && s_fail != 0) atomicCAS(a.status, 0, 700 + s_fail);
    if (warp == 0) tmem_dealloc(s_tmem, 512);
}

template <int MODE, int NT, int PS>
int chain_setup() {
    static PcxOnce done;
    if (!done) {
        cudaError_t e = cudaFuncSetAttribute(column_chain_kernel<MODE, NT, PS>, cudaFuncAttributeMaxDynamicSharedMemorySize, CHAIN_SMEM);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(column_chain_kernel<MODE, NT, PS>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return (int)e;
        done = true;
    }
    return 0;
}

cudaLaunchConfig_t chain_config(int clusters, int cluster, size_t smem, cudaLaunchAttribute* attr, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(clusters * cluster));
    cfg.blockDim = dim3(CHAIN_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = cluster;
    attr->val.clusterDim.y = 1;
    attr->val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

template <int MODE, int NT, int PS>
int launch_chain(ChainArgs a, cudaStream_t st) {
    int rc = chain_setup<MODE, NT, PS>();
    if (rc != 0) return rc;
    const int fixed = CHAIN_FIXED + 2 * a.C * a.q * a.per * NT * 512;
    const int room = (CHAIN_SMEM - fixed) / (CHAIN_WARPS * PS * 1024);
    a.smem_steps = std::max(0, std::min(a.steps - CHAIN_TMEM / PS, room));
    cudaLaunchAttribute attr;
    // (all of the shared memory, whatever the size: tensor memory is claimed as a whole, so CTAs never share an SM)
    cudaLaunchConfig_t cfg = chain_config((int)pcx_cdiv(a.W, 8 * NT), a.C, CHAIN_SMEM, &attr, st);
    cudaError_t e = cudaLaunchKernelEx(&cfg, column_chain_kernel<MODE, NT, PS>, a);
    if (e != cudaSuccess) return (int)e;
    PCX_LAUNCH_CHECK();
    return 0;
}

template <int MODE, int NT>
int launch_chain_ps(const ChainArgs& a, cudaStream_t st) {
    const int strips = (int)pcx_cdiv(a.per, a.halves);
    if (strips == 1) return launch_chain<MODE, NT, 1>(a, st);
    if (strips == 2) return launch_chain<MODE, NT, 2>(a, st);
    return launch_chain<MODE, NT, 4>(a, st);
}

template <int MODE>
int launch_chain_nt(const ChainArgs& a, int nt, cudaStream_t st) {
    if (nt == 1) return launch_chain_ps<MODE, 1>(a, st);
    if (nt == 2) return launch_chain_ps<MODE, 2>(a, st);
    return launch_chain_ps<MODE, 3>(a, st);
}

}  // namespace

extern "C" {

int pcx_column_chain_clusters(int cluster) {
    if (cluster < 1 || cluster > 16) return -1;
    if (chain_setup<C_ELE, 2, 4>() != 0) return -1;
    cudaLaunchAttribute attr;
    cudaLaunchConfig_t cfg = chain_config(1, cluster, CHAIN_SMEM, &attr, nullptr);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, column_chain_kernel<C_ELE, 2, 4>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return -1;
    }
    return n;
}

int64_t pcx_column_chain_bytes(int n_strips, int W, int nt, int per) {
    if (n_strips < 1 || W < 1 || nt < 1 || per < 1) return -1;
    return 2 * pcx_cdiv(W, 8 * nt) * ((int64_t)n_strips * nt * 512 + pcx_cdiv(n_strips, per) * nt * 64);
}

int pcx_column_chain(int mode, float* node_mars, float* node_flows, const void* frags, void* work, const int32_t* rows,
                     const int32_t* strips, int n_levels, int n_strips, int W, int nt, int per, int terms, void* stream) {
    if (n_levels <= 0 || W <= 0) return 0;
    if (W % 8 != 0 || nt < 1 || nt > 3 || per < 1 || per > 8 || per * nt > CHAIN_WARPS || (mode != 0 && mode != 1)) return -1;
    const int C = (int)pcx_cdiv(n_strips, per), halves = per > 1 && C <= 8 ? 2 : 1, kparts = CHAIN_WARPS / halves;
    if (n_strips < 1 || n_strips > 64 || C > kparts || (per + halves - 1) / halves > 4) return -1;
    if (((reinterpret_cast<uintptr_t>(node_mars) | reinterpret_cast<uintptr_t>(node_flows) | reinterpret_cast<uintptr_t>(work) |
          reinterpret_cast<uintptr_t>(frags)) & 15) != 0) return -1;
    ChainArgs a{};
    a.nm = node_mars; a.nf = node_flows; a.frags = reinterpret_cast<const uint4*>(frags);
    a.status = pcx_status_word();
    if (a.status == nullptr) return -1;
    a.operand = reinterpret_cast<uint4*>(work);
    a.shifts = a.operand + 2 * pcx_cdiv(W, 8 * nt) * n_strips * nt * 32;
    a.rows = reinterpret_cast<const int2*>(rows); a.strips = reinterpret_cast<const int2*>(strips);
    a.n_levels = n_levels; a.S = n_strips; a.per = per; a.halves = halves;
    a.strips_w = (per + halves - 1) / halves; a.C = C; a.W = W; a.terms = terms;
    a.steps = (int)pcx_cdiv(per, std::min(per, kparts / C));
    a.q = (int)pcx_cdiv(per, a.steps);
    return mode == 0 ? launch_chain_nt<C_FWD>(a, nt, (cudaStream_t)stream) : launch_chain_nt<C_ELE>(a, nt, (cudaStream_t)stream);
}

}  // extern "C"
