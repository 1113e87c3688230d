// Product layers whose rows are read many times over (leaf products of random tensorised networks): rows through shared memory.
//
// Row j of a product block reads row j of its children's blocks only.  A tile is one j and 32 columns: row j of every source block
// (128 bytes each) is copied to shared memory once, and all output rows are formed from there.  What bounds it is the shared
// memory's 128 bytes a cycle, so one persistent CTA per SM copies the next tile while it works on the present one (two CTAs with
// one tile each ran in step, both copying, then both reading: forward 130 us), and the output rows are taken longest list first,
// so that the four rows of a warp end together.  The general kernels (`prod_fwd_kernel`, `column_prod_kernel`) fetch every row
// from L1 / L2 again for every reader.  784 variables x 32 nodes, 16384 elements of 24 children, 1024 samples (1.6 GB of reads
// of 103 MB of rows): forward 131 -> 95 us, flows (16 parents a row, 67 MB) 185 -> 152 us.
#include <algorithm>
#include "pcx_column_ops.cuh"
#include "../../include/pcx_b200.h"

namespace {

constexpr int ST = 768;                     // threads: 24 warps, four items each at a time (1024 spill)
constexpr int SC = PCX_STAGED_COLUMNS;      // columns of a CTA: a row is eight 16-byte pieces, one bank each
static_assert(SC == 32, "eight lanes of four columns take a row");

struct StagedArgs {
    float* out;                 // stored element values, or node_flows
    const float* src;           // node_mars, or element_flows
    const int32_t* rows;        // first row of every source block
    const int4* items;          // (first output row, first chunk of its list, sources in the list, flow to add to)
    const uint4* lists;         // chunks of eight 16-bit places in `rows`, filled up with n_sources
    int n_sources, n_items, W, tiles, n_tiles;          // tiles: of a row; n_tiles: in all
};

__device__ __forceinline__ void copy_tile(const StagedArgs& a, const int32_t* s_from, int t, uint32_t to) {
    const int c = (t % a.tiles) * SC + (threadIdx.x & 7) * 4;
    const float* src = a.src + (int64_t)(t / a.tiles) * a.W + (c < a.W ? c : 0);
#pragma unroll 4
    for (int i = threadIdx.x >> 3; i < a.n_sources; i += ST / 8)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + i * SC * 4), "l"(src + (int64_t)s_from[i] * a.W) : "memory");
}

// N rows of a list: sums, or log-sum-exps as (maximum `m`, sum of the exponentials around it).  (The exponentials are formed for
// every reader again.  Formed once per source, around the column's maximum, they leave the fp32 range: the flows of a trained
// circuit span hundreds of nats, and a row far under the maximum still has its logarithm.)
template <bool LOGS, int N>
__device__ __forceinline__ void take_rows(uint32_t mine, const uint32_t* words, float* m, float* acc) {
    float x[N][4];
#pragma unroll
    for (int u = 0; u < N; ++u)
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x[u][0]), "=f"(x[u][1]), "=f"(x[u][2]), "=f"(x[u][3])
                     : "r"(mine + ((words[u >> 1] >> (16 * (u & 1))) & 0xffffu) * (SC * 4)));
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        if (LOGS) {
            float hi = m[v];
#pragma unroll
            for (int u = 0; u < N; ++u) hi = fmaxf(hi, x[u][v]);
            const float sh = hi == PCX_NEG_INF ? 0.0f : hi;
            float t = acc[v] * fast_exp(m[v] - sh);
#pragma unroll
            for (int u = 0; u < N; ++u) t += fast_exp(x[u][v] - sh);
            acc[v] = t;
            m[v] = hi;
        } else {
#pragma unroll
            for (int u = 0; u < N; ++u) acc[v] += x[u][v];
        }
    }
}

__device__ __forceinline__ int4 record(const StagedArgs& a, int i) {
    return i < a.n_items ? __ldg(a.items + i) : make_int4(0, 0, 0, 0);
}

template <int MODE, bool LOGS>
__global__ void __launch_bounds__(ST, 1) prod_staged_kernel(const StagedArgs a) {
    extern __shared__ __align__(16) float s_rows[];          // two tiles of [sources + 1][SC], the last row of each empty
    __shared__ int32_t s_from[PCX_STAGED_SOURCES];
    const int piece = threadIdx.x & 7, first = threadIdx.x >> 3, words = (a.n_sources + 1) * SC;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(s_rows) + piece * 16;
    for (int i = threadIdx.x; i < a.n_sources; i += ST) s_from[i] = __ldg(a.rows + i);
    if (threadIdx.x < SC) s_rows[words - SC + threadIdx.x] = s_rows[2 * words - SC + threadIdx.x] = LOGS ? PCX_NEG_INF : 0.0f;
    __syncthreads();
    copy_tile(a, s_from, blockIdx.x, base);
    asm volatile("cp.async.commit_group;" ::: "memory");
    int p = 0;
    for (int t = blockIdx.x; t < a.n_tiles; t += gridDim.x, p ^= 1) {
        const int j = t / a.tiles, c = (t % a.tiles) * SC + piece * 4;
        // (the tile that the next one takes the place of was done with at the barrier that ended the round before)
        if (t + (int)gridDim.x < a.n_tiles) copy_tile(a, s_from, t + gridDim.x, base + (p ^ 1) * words * 4);
        asm volatile("cp.async.commit_group;" ::: "memory");
        // records two rounds ahead and lists one: an item begins with its shared-memory reads
        int4 item = record(a, first), next = record(a, first + ST / 8);
        uint4 list = item.z > 0 ? __ldg(a.lists + item.y) : make_uint4(0, 0, 0, 0);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const uint32_t mine = base + p * words * 4;
        for (int i = first; i < a.n_items; i += ST / 8) {
            const int4 now = item;
            uint4 l = list;
            item = next;
            next = record(a, i + 2 * (ST / 8));
            if (item.z > 0) list = __ldg(a.lists + item.y);
            const bool ok = c < a.W, add = MODE == C_ELE && now.w != 0;
            float* dst = a.out + (int64_t)(now.x + j) * a.W + (ok ? c : 0);
            float m[4], acc[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) { m[v] = PCX_NEG_INF; acc[v] = 0.0f; }
            if (add) ldvec<4>(dst, LOGS ? m : acc);
            if (LOGS && add)
#pragma unroll
                for (int v = 0; v < 4; ++v) acc[v] = 1.0f;
            for (int k = 0; k < now.z; k += 8) {
                const uint32_t q[4] = {l.x, l.y, l.z, l.w};
                if (k + 8 < now.z) l = __ldg(a.lists + now.y + k / 8 + 1);
                if (k + 4 < now.z) take_rows<LOGS, 8>(mine, q, m, acc);
                else take_rows<LOGS, 4>(mine, q, m, acc);
            }
            if (LOGS)                                        // (one parent: its flow as it is; a maximum passes over NaN, the sum does not)
#pragma unroll
                for (int v = 0; v < 4; ++v)
                    if (now.z != 1 || add || acc[v] != acc[v]) m[v] = fast_log_plus(acc[v], m[v] == PCX_NEG_INF ? 0.0f : m[v]);
            if (ok) stvec<4>(dst, LOGS ? m : acc);
        }
        __syncthreads();
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

template <int MODE, bool LOGS>
int launch_staged(const StagedArgs& a, cudaStream_t st) {
    static PcxOnce done;
    if (!done) {
        cudaError_t e = cudaFuncSetAttribute(prod_staged_kernel<MODE, LOGS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             2 * (PCX_STAGED_SOURCES + 1) * SC * 4);
        if (e != cudaSuccess) return (int)e;
        done = true;
    }
    prod_staged_kernel<MODE, LOGS><<<std::min(a.n_tiles, 148), ST, (size_t)2 * (a.n_sources + 1) * SC * 4, st>>>(a);
    PCX_LAUNCH_CHECK();
    return 0;
}

}  // namespace

extern "C" {

int pcx_prod_staged(int mode, float* out, const float* src, const int32_t* sources, const int32_t* items, const int32_t* lists,
                    int n_sources, int n_items, int block_size, int W, int logspace, void* stream) {
    if (n_items <= 0 || block_size <= 0 || W <= 0) return 0;
    if ((mode != 0 && mode != 1) || W % 4 != 0 || n_sources < 0 || n_sources > PCX_STAGED_SOURCES) return -1;
    if (((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(items) |
          reinterpret_cast<uintptr_t>(lists)) & 15) != 0) return -1;
    StagedArgs a{};
    a.out = out; a.src = src; a.rows = sources; a.items = reinterpret_cast<const int4*>(items);
    a.lists = reinterpret_cast<const uint4*>(lists);
    a.n_sources = n_sources; a.n_items = n_items; a.W = W; a.tiles = (int)pcx_cdiv(W, SC);
    if ((int64_t)block_size * a.tiles > INT32_MAX / 2) return -1;
    a.n_tiles = block_size * a.tiles;
    if (mode == 0) return launch_staged<C_FWD, false>(a, (cudaStream_t)stream);
    return logspace ? launch_staged<C_ELE, true>(a, (cudaStream_t)stream) : launch_staged<C_ELE, false>(a, (cudaStream_t)stream);
}

}  // extern "C"
