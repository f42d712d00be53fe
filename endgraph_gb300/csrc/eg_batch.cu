// eg_batch.cu — batched operators over one built graph (no reference counterpart; they batch the
// toolkits of toolkits/{bfs,sssp}.cpp and a personalised PageRank built on pagerank.cpp):
//
//  * eg_msbfs: bit-parallel BFS from up to 64 roots.  Every vertex keeps a u64 of the roots that
//    reached it and a u64 of the roots whose frontier it is in; a level either pushes the queued
//    frontier's words along the CSR or is one sweep over the CSC that ORs the in-neighbours'
//    frontier words (exact integer work, levels identical to 64 separate BFS runs).
//  * row engine: a destination's 64 values (one per seed / source) sit in one 256-byte row, up to 32
//    in one of 128; a warp walks the edges of a batch of lists and reads a whole row per edge, each
//    lane owning its columns.  Lists longer than a task (kTaskEdges) are split and their partial
//    rows combined in a small per-heavy-vertex buffer.  Used by
//      - eg_ppr: personalised PageRank x_{k+1} = a*e_seed + (1-a) * A^T x_k, A = row-normalised
//        edge weights, FP32;
//      - eg_ppr_backward: the adjoint of K unrolled iterations.  lambda_k = (1-a) A lambda_{k+1} is
//        a pull over the CSR (the transpose of the forward CSC); the same sweep accumulates
//        dL/dA_uv = (1-a) sum_k <x_k[u], lambda_{k+1}[v]>; the iterates x_k are kept while they fit
//        EG_OPT_PPR_KEEP_MIB, else recomputed from checkpoints;
//      - eg_sssp_batch: Bellman-Ford from up to 64 sources, in place, skipping sources whose
//        distance did not change in the previous sweep (bit-exact least fixpoint).
#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "eg_pull.cuh"

namespace eg {

constexpr uint32_t kTaskEdges = 512;
constexpr uint32_t kNoSlot = 0xFFFFFFFFu;

// ---------------------------------------------------------------------------------------------
// MS-BFS.  A level is a pull sweep over the CSC when the frontier's out-edges reach E / divisor
// (the switch of core/graph.hpp:1484-1491) and a push over the frontier queue otherwise.  Roots
// whose traversal has ended can add nothing, so a destination whose visited word already holds
// every root still running (`alive`) is skipped, and while the frontier is small a source outside
// the frontier bitmap is not gathered at all.  The traversal kernels only set bits; the next
// frontier is then listed once (k_bm_compact) and its level bytes written from that list
// (k_queue_levels), so no traversal thread loops over the bits of a word.
// L2-coherent (.cg): the persistent traversal reads bitmaps that the same launch wrote
__device__ __forceinline__ bool bm_has(const unsigned long long* bm, uint32_t v) {
    return (__ldcg(bm + (v >> 6)) >> (v & 63)) & 1ull;
}

struct MsBfsPullOp {  // k_pull_direct operator (several partitions, and the persistent traversal)
    using Acc = unsigned long long;
    const unsigned long long* front;
    const unsigned long long* front_bm;  // 1 bit per vertex: front[v] != 0
    int screen;                          // consult front_bm before gathering
    unsigned long long* visit;
    unsigned long long* next;
    unsigned long long* next_bm;
    const unsigned long long* alive;
    const int* stop;  // captured level loops: set once a level found nothing new
    __device__ bool stopped() const { return stop && *(volatile const int*)stop; }
    __device__ bool item_active(uint32_t v) const {
        const unsigned long long al = __ldg(alive);
        return (__ldcg(visit + v) & al) != al;
    }
    __device__ Acc identity() const { return 0ull; }
    __device__ Acc combine(Acc a, Acc b) const { return a | b; }
    __device__ Acc gather(uint32_t u) const {
        if (screen && !bm_has(front_bm, u)) return 0ull;
        return ld_keep(front + u);
    }
    __device__ __forceinline__ void finish_direct(uint32_t v, Acc m) const {
        const unsigned long long fresh = m & ~__ldcg(visit + v);
        if (!fresh) return;
        const unsigned long long nb = fresh & ~atomicOr(visit + v, fresh);
        if (nb && atomicOr(next + v, nb) == 0ull) atomicOr(next_bm + (v >> 6), 1ull << (v & 63));
    }
};

// A dense level as a full sweep: the walk of the PageRank sweep (eg_pagerank.cu: list starts as one bit
// per edge, 8 consecutive ids per lane, a segmented warp scan, lists finished one per lane) with OR in
// the place of the sum.  A list that lies in one run is this warp's alone: its vertex's words are
// stored plainly; pieces of longer lists are ORed in with atomics, each on its own.  As there, one CTA
// of 32 warps per SM takes runs by ticket, and with renumbered sources the frontier words of the
// hottest are kept in shared memory.  64 roots, 2^23 / 2^27 and 2^25 / 2^29: dense levels 1.47 / 5.8 ms with
// CTAs of 8 warps at 5 per SM, 1.45 / 5.6 so without the table, 1.37 / 5.4 with 4,096 words, 1.34 / 5.5 with
// 8,192, 1.34 / 5.7 with 12,288.  (At 2^23 a level had taken 1.05 ms with a CTA per 4,096 edges, entry
// bounds in shared memory and atomics for every list, 0.59 with the walk.)
constexpr uint32_t kMsBlock = 256;

struct MsSweepArgs {
    const uint32_t* adj;
    const uint32_t* heads;    // bit e: edge e is the first of its list
    const uint32_t* item_of;  // per kPrBlock edges: compressed entry that holds the first one
    const uint32_t* cvert;
    uint64_t E;
    uint64_t nruns;           // runs of kPrBlock << shift edges
    int shift;
    uint32_t nitems;
    const unsigned long long* alive;     // roots still running: a vertex that has them all gains nothing (null: not
                                         // looked at; in a graph batch no vertex has the roots of all graphs)
    const unsigned long long* front;
    const unsigned long long* front_bm;  // 1 bit per vertex: front[v] != 0
    int screen;                          // consult front_bm before gathering
    unsigned long long* visit;
    unsigned long long* next;
    unsigned long long* next_bm;
    const int* stop;  // captured level loops: set once a level found nothing new
    uint32_t hot;     // ranks of the renumbering (rank r is id 32 r) whose words are kept in shared memory
    uint32_t* ticket; // the sweep's next run, zero before it
};

__device__ __forceinline__ void ms_piece(const MsSweepArgs& a, uint32_t v, unsigned long long m) {
    const unsigned long long fresh = m & ~__ldcg(a.visit + v);
    if (!fresh) return;
    const unsigned long long nb = fresh & ~atomicOr(a.visit + v, fresh);
    if (nb && atomicOr(a.next + v, nb) == 0ull) atomicOr(a.next_bm + (v >> 6), 1ull << (v & 63));
}
__device__ __forceinline__ void ms_list(const MsSweepArgs& a, uint32_t v, unsigned long long m) {
    const unsigned long long vis = __ldcg(a.visit + v), nb = m & ~vis;
    if (!nb) return;
    a.visit[v] = vis | nb;
    a.next[v] = nb;
    atomicOr(a.next_bm + (v >> 6), 1ull << (v & 63));
}

constexpr uint32_t kMsHot = 8192, kMsThreads = 1024;
constexpr size_t kMsSmem = 8ull * (kMsHot + kMsThreads / 32 * kMsBlock);

__global__ void __launch_bounds__(kMsThreads, 1) k_ms_sweep(MsSweepArgs a) {
    extern __shared__ unsigned long long s_or[];
    if (a.stop && *(volatile const int*)a.stop) return;
    constexpr int G = 8;
    unsigned long long* s_list = s_or + (threadIdx.x >> 5) * kMsBlock;
    unsigned long long* s_hot = s_or + kMsThreads / 32 * kMsBlock;
    const uint32_t lane = threadIdx.x & 31, below = (1u << lane) - 1u;
    for (uint32_t r = threadIdx.x; r < a.hot; r += kMsThreads) s_hot[r] = __ldcg(a.front + 32ull * r);
    const uint32_t hot_addr = (uint32_t)__cvta_generic_to_shared(s_hot), hot = a.hot;
    unsigned long long keep;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 0.5;" : "=l"(keep));
    auto gather = [&](uint32_t id) {
        const uint32_t rank = __funnelshift_r(id, id, 5);  // ids that are no multiple of 32 come out large
        unsigned long long v;
        asm volatile(
            "{\n.reg .pred p;\nsetp.lt.u32 p, %1, %2;\n@p ld.shared.u64 %0, [%3];\n"
            "@!p ld.global.cg.L2::cache_hint.u64 %0, [%4], %5;\n}"
            : "=l"(v)
            : "r"(rank), "r"(hot), "r"(hot_addr + 8 * rank), "l"(a.front + id), "l"(keep));
        return v;
    };
    const uint64_t run_edges = (uint64_t)kPrBlock << a.shift;
    const unsigned long long al = a.alive ? __ldg(a.alive) : 0ull;
    uint32_t ticket = 0;
    if (lane == 0) ticket = atomicAdd(a.ticket, 1u);
    __syncthreads();
    while (true) {
        const uint64_t run = __shfl_sync(0xffffffffu, ticket, 0);
        if (run >= a.nruns) break;
        if (lane == 0) ticket = atomicAdd(a.ticket, 1u);
        const uint64_t e_begin = run * run_edges, e_end = min(a.E, e_begin + run_edges);
        uint32_t item = __ldg(a.item_of + (run << a.shift));
        // Few lists, all of whose vertices have every running root: nothing to read.  With few roots the first dense
        // level of a dense graph finds most vertices so (1,000 vertices, 2^26 edges, 3 roots: 1.42 -> 0.03 ms).
        if (al) {
            const uint32_t last_item = run + 1 < a.nruns ? __ldg(a.item_of + ((run + 1) << a.shift)) : a.nitems - 1;
            if (last_item - item < 32) {
                const bool idle = lane > last_item - item || !(al & ~__ldcg(a.visit + __ldg(a.cvert + item + lane)));
                if (__all_sync(0xffffffffu, idle)) continue;
            }
        }
        bool open_first = !(__ldg(a.heads + (e_begin >> 5)) & 1u);  // the first list began in an earlier run
        unsigned long long carry = 0;                                // OR of the open list so far
        for (uint64_t e0 = e_begin; e0 < e_end; e0 += kMsBlock) {
            const uint64_t e = e0 + lane * G;
            unsigned long long val[G];
            uint32_t id[G];
            uint32_t f = 0;
            if (e + G <= a.E) {
                const uint4 x = __ldcs(reinterpret_cast<const uint4*>(a.adj + e));
                const uint4 y = __ldcs(reinterpret_cast<const uint4*>(a.adj + e) + 1);
                id[0] = x.x; id[1] = x.y; id[2] = x.z; id[3] = x.w;
                id[4] = y.x; id[5] = y.y; id[6] = y.z; id[7] = y.w;
                if (a.screen) {
#pragma unroll
                    for (int j = 0; j < G; ++j) val[j] = bm_has(a.front_bm, id[j]) ? gather(id[j]) : 0ull;
                } else {
#pragma unroll
                    for (int j = 0; j < G; ++j) val[j] = gather(id[j]);
                }
            } else {
#pragma unroll
                for (int j = 0; j < G; ++j) val[j] = e + j < a.E ? gather(a.adj[e + j]) : 0ull;
            }
            if (e < a.E) f = __ldcs(reinterpret_cast<const uint8_t*>(a.heads) + e / 8);
            if (e == e_begin) f &= ~1u;  // the run's first edge opens nothing new
            uint32_t rank = 0, closed = 0;  // lists that end in earlier lanes, and in the block
#pragma unroll
            for (int j = 0; j < G; ++j) {
                const uint32_t b = __ballot_sync(0xffffffffu, (f >> j) & 1u);
                rank += __popc(b & below);
                closed += __popc(b);
            }
            const uint32_t v32 = lane < closed ? __ldg(a.cvert + item + lane) : 0u;
            unsigned long long t = 0, first = 0;
            uint32_t k = rank;
            bool seen = false;
#pragma unroll
            for (int j = 0; j < G; ++j) {
                if ((f >> j) & 1u) {
                    if (seen) s_list[k] = t;
                    else first = t;
                    ++k;
                    seen = true;
                    t = 0;
                }
                t |= val[j];
            }
            // the open list along the lanes: t becomes its OR up to and including this lane
            const uint32_t m = __ballot_sync(0xffffffffu, seen);
            const int begin = 31 - __clz(m & (below | (1u << lane)));  // last lane that opened one, or -1
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long y = __shfl_up_sync(0xffffffffu, t, o);
                if ((int)lane - o >= max(begin, 0)) t |= y;
            }
            if (begin < 0) t |= carry;
            unsigned long long before = __shfl_up_sync(0xffffffffu, t, 1);
            if (lane == 0) before = carry;
            if (seen) s_list[rank] = before | first;
            carry = __shfl_sync(0xffffffffu, t, 31);
            __syncwarp();
            for (uint32_t i = lane; i < closed; i += 32) {
                const unsigned long long x = s_list[i];
                if (!x) continue;
                const uint32_t v = i < 32 ? v32 : __ldg(a.cvert + item + i);
                if (i == 0 && open_first) ms_piece(a, v, x);
                else ms_list(a, v, x);
            }
            __syncwarp();
            if (closed) open_first = false;
            item += closed;
        }
        if (lane == 0 && carry) ms_piece(a, __ldg(a.cvert + item), carry);
    }
}

// Early-exit dense level: a destination stops reading in-edges as soon as its visited word holds
// every root still running (nothing more can reach it in this level).  One thread per compressed
// entry reads the first kMsHead in-edges; longer lists continue as kMsSeg-edge segments, one warp
// each, that apply their partial OR every 128 edges so that other segments of the same
// destination see the coverage.  Partial ORs are applied like finish_direct (idempotent).
constexpr uint32_t kMsHead = 8;
constexpr uint32_t kMsSeg = 1024;

struct MsBuArgs {
    const uint32_t* adj;
    const uint64_t* cidx;
    const uint32_t* cvert;
    uint64_t nitems;
    uint32_t V;
    const unsigned long long* front;
    unsigned long long* visit;
    unsigned long long* next;
    unsigned long long* next_bm;
    const unsigned long long* alive;
    unsigned long long* seg;  // (segment << 32) | compressed entry
    uint32_t* nseg;
    const int* stop;  // captured level loops: set once a level found nothing new
};

__device__ __forceinline__ void ms_apply(const MsBuArgs& a, uint32_t v, unsigned long long m) {
    const unsigned long long fresh = m & ~__ldcg(a.visit + v);
    if (!fresh) return;
    const unsigned long long nb = fresh & ~atomicOr(a.visit + v, fresh);
    if (nb && atomicOr(a.next + v, nb) == 0ull) atomicOr(a.next_bm + (v >> 6), 1ull << (v & 63));
}

__device__ __forceinline__ void ms_head_work(const MsBuArgs& a) {
    const int lane = threadIdx.x & 31;
    const unsigned long long al = __ldg(a.alive);
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < a.nitems; base += stride) {
        const uint64_t i = base + threadIdx.x;
        uint32_t nsg = 0;
        if (i < a.nitems) {
            const uint32_t v = a.cvert[i];
            const unsigned long long need = v < a.V ? al & ~__ldcg(a.visit + v) : 0ull;
            if (need) {
                const uint64_t s = a.cidx[i], e = a.cidx[i + 1];
                const uint64_t h = e - s > kMsHead ? s + kMsHead : e;
                unsigned long long acc = 0;
                for (uint64_t p = s; p < h && (acc & need) != need; p += 4) {
                    uint32_t u[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) u[q] = p + q < h ? __ldg(a.adj + p + q) : a.V;
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (u[q] < a.V) acc |= ld_keep(a.front + u[q]);
                }
                if (acc & need) ms_apply(a, v, acc);
                if ((acc & need) != need && e > h) nsg = (uint32_t)((e - h + kMsSeg - 1) / kMsSeg);
            }
        }
        uint32_t incl = nsg;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        const uint32_t tot = __shfl_sync(0xffffffffu, incl, 31);
        if (tot) {
            uint32_t at = 0;
            if (lane == 31) at = atomicAdd(a.nseg, tot);
            at = __shfl_sync(0xffffffffu, at, 31) + incl - nsg;
            for (uint32_t k = 0; k < nsg; ++k) a.seg[at + k] = ((unsigned long long)k << 32) | (uint32_t)i;
        }
    }
}

__global__ void __launch_bounds__(256) k_ms_head(MsBuArgs a) {
    if (a.stop && *(volatile const int*)a.stop) return;
    ms_head_work(a);
}

__device__ __forceinline__ void ms_tail_work(const MsBuArgs& a) {
    const uint32_t n = __ldcg(a.nseg);
    const int lane = threadIdx.x & 31;
    const unsigned long long al = __ldg(a.alive);
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t t = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < n; t += nwarps) {
        const unsigned long long ent = a.seg[t];
        const uint32_t i = (uint32_t)ent;
        const uint32_t v = a.cvert[i];
        const uint64_t e = a.cidx[i + 1];
        uint64_t p = a.cidx[i] + kMsHead + (ent >> 32) * kMsSeg;
        const uint64_t pe = p + kMsSeg < e ? p + kMsSeg : e;
        for (; p < pe; p += 128) {
            const unsigned long long vis = __shfl_sync(0xffffffffu, __ldcg(a.visit + v), 0);
            if ((vis & al) == al) break;  // every running root already reached v
            unsigned long long acc = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint64_t x = p + 32 * q + lane;
                if (x < pe) acc |= ld_keep(a.front + __ldg(a.adj + x));
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc |= __shfl_xor_sync(0xffffffffu, acc, o);
            if (lane == 0 && (acc & ~vis)) ms_apply(a, v, acc);
        }
    }
}

__global__ void __launch_bounds__(256) k_ms_tail(MsBuArgs a) {
    if (a.stop && *(volatile const int*)a.stop) return;
    ms_tail_work(a);
}

struct MsBfsPushOp {
    const unsigned long long* front;
    unsigned long long* visit;
    unsigned long long* next;
    unsigned long long* next_bm;
    __device__ unsigned long long payload(uint32_t u) const { return __ldcg(front + u); }
    __device__ bool relax(uint32_t, unsigned long long pay, uint32_t w, uint64_t) const {
        const unsigned long long m = pay & ~__ldcg(visit + w);
        if (!m) return false;
        const unsigned long long nb = m & ~atomicOr(visit + w, m);
        if (!nb || atomicOr(next + w, nb) != 0ull) return false;
        atomicOr(next_bm + (w >> 6), 1ull << (w & 63));
        return true;  // w joins the next frontier's queue
    }
};

// A traversal keeps its levels as bit planes, [V][4] words for bits 0..3 of the level of each root and
// [V][4] more for bits 4..7 (zeroed before the first level past 15: kHighPlanes): a vertex that new roots reach at
// level l gets their bits ORed into the planes of l, or, when they are its first, its four words
// written without a read (which is what clears them).  A level touches a sector per vertex where rows
// of 64 level bytes took a read and a write of up to two; the bytes are made once, at the end.  64
// roots at 2^23 / 2^27: vertex passes 0.76 -> 0.60 ms.
// Also the OR of the queued vertices' words, i.e. the roots whose traversal is still running, and,
// with new_id, the words copied to renumbered positions (next_r[new_id[v]]) for the pull gathers that
// go through the renumbered CSC sources.
__device__ __forceinline__ void queue_levels_work(const uint32_t* __restrict__ q, uint32_t n,
                                                  const unsigned long long* __restrict__ next,
                                                  const unsigned long long* visit, unsigned long long* planes,
                                                  uint64_t V, uint32_t lvl, unsigned long long* alive_out,
                                                  const uint32_t* __restrict__ new_id,
                                                  unsigned long long* __restrict__ next_r) {
    unsigned long long orr = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t v = q[i];
        const unsigned long long nb = next[v];
        if (new_id) next_r[new_id[v]] = nb;
        orr |= nb;
        if (!planes) continue;
        unsigned long long* p = planes + (uint64_t)v * 4;
        if (__ldcg(visit + v) == nb) {
            ulonglong2* p2 = reinterpret_cast<ulonglong2*>(p);
            p2[0] = make_ulonglong2(lvl & 1u ? nb : 0ull, lvl & 2u ? nb : 0ull);
            p2[1] = make_ulonglong2(lvl & 4u ? nb : 0ull, lvl & 8u ? nb : 0ull);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if ((lvl >> j) & 1u) p[j] |= nb;
        }
        if (lvl < 16) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if ((lvl >> (4 + j)) & 1u) p[4 * V + j] |= nb;
    }
    if (!alive_out) return;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) orr |= __shfl_xor_sync(0xffffffffu, orr, o);
    if ((threadIdx.x & 31) == 0 && orr) atomicOr(alive_out, orr);
}

__global__ void k_queue_levels(const uint32_t* __restrict__ q, const uint32_t* n_dev,
                               const unsigned long long* __restrict__ next, const unsigned long long* visit,
                               unsigned long long* planes, uint64_t V, uint32_t lvl, unsigned long long* alive_out,
                               const uint32_t* __restrict__ new_id, unsigned long long* __restrict__ next_r) {
    queue_levels_work(q, __ldcg(n_dev), next, visit, planes, V, lvl, alive_out, new_id, next_r);
}

// The upper planes (bits 4..7) are zeroed as this level begins, whose vertices are the first to have level 16: not
// ahead of time for traversals that hardly ever get there.
constexpr uint32_t kHighPlanes = 15;
__global__ void k_zero_planes(unsigned long long* __restrict__ planes, uint64_t n, const uint32_t* frontier) {
    if (!*frontier) return;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) planes[i] = 0ull;
}

// level bytes of 16 roots (16 q .. 16 q + 15) of vertex v, 0xFF where the root never reached it
__device__ __forceinline__ uint4 level_bytes(const unsigned long long* __restrict__ planes,
                                             const unsigned long long* __restrict__ visit, uint64_t V, uint64_t v, int q,
                                             int deep) {
    uint32_t w[4] = {0, 0, 0, 0};
    const uint32_t vis = (uint32_t)(__ldg(visit + v) >> (16 * q)) & 0xFFFFu;
    if (vis) {
        for (int h = 0; h <= deep; ++h) {
            const ulonglong2* p = reinterpret_cast<const ulonglong2*>(planes + 4 * (h * V + v));
            const ulonglong2 a = __ldg(p), b = __ldg(p + 1);
            const unsigned long long pl[4] = {a.x, a.y, b.x, b.y};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t bits = (uint32_t)(pl[j] >> (16 * q)) & 0xFFFFu;
#pragma unroll
                for (int k = 0; k < 4; ++k)  // bit i of the nibble -> byte i (the shifted copies never overlap)
                    w[k] |= (((bits >> (4 * k)) & 0xFu) * (0x00204081u << (4 * h + j))) & (0x01010101u << (4 * h + j));
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t m = ((((vis >> (4 * k)) & 0xFu) * 0x00204081u) & 0x01010101u) * 0xFFu;
        w[k] = (w[k] & m) | ~m;
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// level rows [V][64] of a graph batch (out: 16-byte aligned)
__global__ void __launch_bounds__(256) k_level_rows(const unsigned long long* __restrict__ planes,
                                                    const unsigned long long* __restrict__ visit, uint64_t V, int deep,
                                                    uint4* __restrict__ out) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < 4 * V; i += stride)
        __stcs(out + i, level_bytes(planes, visit, V, i >> 2, (int)(i & 3), deep));
}

// zero the frontier words (and their renumbered copies) of the vertices a queue lists: the only
// non-zero entries of a frontier array, cheaper than clearing all of it while frontiers are small
__global__ void k_clear_front(const uint32_t* __restrict__ q, uint32_t n, unsigned long long* __restrict__ word,
                              const uint32_t* __restrict__ new_id, unsigned long long* __restrict__ word_r) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t v = q[i];
        word[v] = 0ull;
        if (word_r) word_r[new_id[v]] = 0ull;
    }
}

// the renumbered copy of the first frontier (the roots), which no level has listed
__global__ void k_front_renumber(const uint32_t* __restrict__ q, const uint32_t* n_dev,
                                 const unsigned long long* __restrict__ word, const uint32_t* __restrict__ new_id,
                                 unsigned long long* __restrict__ word_r) {
    const uint32_t n = __ldcg(n_dev);
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        word_r[new_id[q[i]]] = word[q[i]];
}

// sum over vertices of popcount(visited word) * out-degree: the edges 64 single-root runs scan
__global__ void k_reach_edges(const unsigned long long* __restrict__ visit, const uint32_t* __restrict__ deg, uint64_t V,
                              unsigned long long* out) {
    unsigned long long acc = 0;
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V; v += (uint64_t)gridDim.x * blockDim.x)
        acc += (unsigned long long)__popcll(visit[v]) * deg[v];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0 && acc) atomicAdd(out, acc);
}

// level planes -> [n][V] root rows for the first n roots, 256 vertices per CTA: 64 level bytes per vertex
// into shared memory, 4 x 4 bytes at a time turned into 16 consecutive vertices of a root, and every
// root's row stored in whole 16-byte pieces of the output whatever its alignment (V odd: each row
// starts elsewhere), the row's first and last bytes one by one.  64 roots at 2^23: 0.28 ms (0.87 GB), one
// root 0.09 (0.24 with all columns made); from level rows, with a byte per load and 16-byte stores only where V allows,
// 0.26, and 2.0 at 2^23 - 1.
constexpr uint32_t kOutTile = 256;
constexpr uint32_t kOutStride = kOutTile / 4 + 4;  // words per root row in shared memory
__global__ void __launch_bounds__(256) k_levels_out(const unsigned long long* __restrict__ planes,
                                                    const unsigned long long* __restrict__ visit, uint32_t V, int n,
                                                    int deep, uint8_t* __restrict__ out) {
    __shared__ uint32_t t[kOutTile][17];                      // [vertex][root / 4]
    __shared__ __align__(16) uint32_t u[64][kOutStride];      // [root][vertex / 4]
    const uint64_t v0 = (uint64_t)blockIdx.x * kOutTile;
    const uint32_t quads = ((uint32_t)n + 15) / 16;  // of 16 columns that the call has
    for (uint32_t i = threadIdx.x; i < quads * kOutTile; i += blockDim.x) {
        const uint32_t r = i % kOutTile, q = i / kOutTile;
        const uint4 x = v0 + r < V ? level_bytes(planes, visit, V, v0 + r, (int)q, deep) : make_uint4(~0u, ~0u, ~0u, ~0u);
        t[r][4 * q] = x.x;
        t[r][4 * q + 1] = x.y;
        t[r][4 * q + 2] = x.z;
        t[r][4 * q + 3] = x.w;
    }
    __syncthreads();
    const uint32_t rq = threadIdx.x & 15, vg = threadIdx.x >> 4;  // roots 4 rq .. + 3, vertices 16 vg .. + 15
    if (4 * rq < (uint32_t)n) {
        uint32_t row[4][4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t a = t[16 * vg + 4 * k][rq], b = t[16 * vg + 4 * k + 1][rq];
            const uint32_t c = t[16 * vg + 4 * k + 2][rq], d = t[16 * vg + 4 * k + 3][rq];
            const uint32_t ab0 = __byte_perm(a, b, 0x5140), ab1 = __byte_perm(a, b, 0x7362);
            const uint32_t cd0 = __byte_perm(c, d, 0x5140), cd1 = __byte_perm(c, d, 0x7362);
            row[0][k] = __byte_perm(ab0, cd0, 0x5410);
            row[1][k] = __byte_perm(ab0, cd0, 0x7632);
            row[2][k] = __byte_perm(ab1, cd1, 0x5410);
            row[3][k] = __byte_perm(ab1, cd1, 0x7632);
        }
#pragma unroll
        for (int r = 0; r < 4; ++r)
            *reinterpret_cast<uint4*>(&u[4 * rq + r][4 * vg]) = make_uint4(row[r][0], row[r][1], row[r][2], row[r][3]);
    }
    __syncthreads();
    const uint32_t nv = V - v0 < kOutTile ? (uint32_t)(V - v0) : kOutTile;
    const uint32_t c = threadIdx.x & 15;
    for (uint32_t s = threadIdx.x >> 4; s < (uint32_t)n; s += 16) {
        uint8_t* o = out + (uint64_t)s * V + v0;
        const uint8_t* bytes = reinterpret_cast<const uint8_t*>(u[s]);
        const uint32_t first = (uint32_t)(-(uintptr_t)o & 15u);  // bytes before the first whole piece
        const uint32_t pieces = nv > first ? (nv - first) / 16 : 0u;
        if (c < pieces) {
            const uint32_t at = first + 16 * c, w = at >> 2, sh = (at & 3u) * 8;
            uint32_t x[5];
#pragma unroll
            for (int k = 0; k < 5; ++k) x[k] = u[s][w + k];
            *reinterpret_cast<uint4*>(o + at) =
                make_uint4(__funnelshift_r(x[0], x[1], sh), __funnelshift_r(x[1], x[2], sh), __funnelshift_r(x[2], x[3], sh),
                           __funnelshift_r(x[3], x[4], sh));
        }
        if (c < first && c < nv) o[c] = bytes[c];
        for (uint32_t i = first + 16 * pieces + c; i < nv; i += 16) o[i] = bytes[i];
    }
}

template <typename T>
__global__ void k_transpose_rows(const T* __restrict__ in, uint32_t V, int n, T* __restrict__ out, int width = 64) {
    __shared__ T t[64][33];
    const uint64_t v0 = (uint64_t)blockIdx.x * 32;
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        const uint64_t v = v0 + i;
        for (int s = threadIdx.x; s < width; s += blockDim.x) t[s][i] = v < V ? in[v * width + s] : T(0);
    }
    __syncthreads();
    for (int s = threadIdx.y; s < n; s += blockDim.y) {
        const uint64_t v = v0 + threadIdx.x;
        if (v < V) out[(uint64_t)s * V + v] = t[s][threadIdx.x];
    }
}

template <typename T>
__global__ void k_untranspose_rows(const T* __restrict__ in, uint32_t V, int n, T* __restrict__ out, int width) {
    __shared__ T t[64][33];
    const uint64_t v0 = (uint64_t)blockIdx.x * 32;
    for (int s = threadIdx.y; s < width; s += blockDim.y) {
        const uint64_t v = v0 + threadIdx.x;
        t[s][threadIdx.x] = (s < n && v < V) ? in[(uint64_t)s * V + v] : T(0);
    }
    __syncthreads();
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        const uint64_t v = v0 + i;
        for (int s = threadIdx.x; s < width; s += blockDim.x)
            if (v < V) out[v * width + s] = t[s][i];
    }
}

// ---------------------------------------------------------------------------------------------
// tasks: item i of a list index (begin[i], begin[i+1]) split into pieces of <= kTaskEdges edges.
// A task is one 16-byte record, so that a warp knows its edges, its vertex and where its result
// goes after a single load (which it issues one task ahead):
//   x  first edge, low 32 bits          z  vertex whose row the task reduces into
//   y  first edge, bits 32..39 in 0..7  w  slot of a list cut into several tasks, or kNoSlot
//      edges of the task << 8
struct TaskLoad {
    const uint64_t* begin;
    __device__ uint32_t operator()(uint64_t i) const {
        const uint64_t n = begin[i + 1] - begin[i];
        return (uint32_t)((n + kTaskEdges - 1) / kTaskEdges);
    }
};
struct TaskEpi {
    uint4* rec;
    const uint64_t* begin;
    const uint32_t* item_vertex;  // null: the item index is the vertex
    uint32_t* heavy_vertex;       // per slot
    uint32_t* nheavy;
    __device__ void operator()(uint64_t i, uint64_t excl, uint32_t cnt) const {
        if (!cnt) return;
        const uint32_t v = item_vertex ? item_vertex[i] : (uint32_t)i;
        uint32_t slot = kNoSlot;
        if (cnt > 1) {
            slot = atomicAdd(nheavy, 1u);
            heavy_vertex[slot] = v;
        }
        const uint64_t b = begin[i], e = begin[i + 1];
        for (uint32_t p = 0; p < cnt; ++p) {
            const uint64_t e0 = b + (uint64_t)p * kTaskEdges;
            const uint32_t len = (uint32_t)(e - e0 < kTaskEdges ? e - e0 : kTaskEdges);
            rec[excl + p] = make_uint4((uint32_t)e0, (uint32_t)(e0 >> 32) | (len << 8), v, slot);
        }
    }
};
__device__ __forceinline__ uint64_t task_begin(const uint4& t) { return ((uint64_t)(t.y & 0xFFu) << 32) | t.x; }
__device__ __forceinline__ uint32_t task_len(const uint4& t) { return t.y >> 8; }

struct RowTasks {
    DevBuf rec, heavy_vertex, counts, first;
    uint64_t ntasks = 0;
    uint32_t nheavy = 0;
    uint32_t nbatches = 0;  // first: [nbatches + 1]
};

// Batches of consecutive tasks, one per warp of the row kernels: batch b holds the tasks that begin in edges
// [b size, (b + 1) size).  Every warp is a CTA of its own, so the hardware hands batches to whichever SM
// is free: with 32 warps per SM taking tasks by stride, SMs were idle for a quarter of a PPR sweep.
__global__ void k_task_batches(const uint4* __restrict__ rec, uint64_t ntasks, uint32_t size, uint32_t nb,
                               uint32_t* __restrict__ first) {
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t <= ntasks; t += (uint64_t)gridDim.x * blockDim.x) {
        const int64_t lo = t ? (int64_t)(task_begin(rec[t - 1]) / size) : -1;
        const int64_t hi = t < ntasks ? (int64_t)(task_begin(rec[t]) / size) : (int64_t)nb;
        for (int64_t b = lo + 1; b <= hi; ++b) first[b] = (uint32_t)t;
    }
}

// 512 edges a batch, fewer on graphs that would not give every resident warp one.  50 PPR iterations on
// 1 M / 16 M: 35.8 ms with 256, 32.1 with 512, 31.0 with 1,024, whose batches come out as slow for the
// adjoint (27.3 against 26.5) and SSSP; 20,000 / 100,000: 1.43 with 16, 1.31 with 32 or 64.
constexpr uint64_t kBatchEdges = 512, kBatchEdgesMin = 32;
static int make_batches(eg_graph* g, RowTasks& t) {
    const uint64_t E = std::max<uint64_t>(g->E, 1), warps = g->num_sms * 32ull;
    const uint64_t size = std::min(kBatchEdges, std::max(kBatchEdgesMin, (E + warps - 1) / warps));
    t.nbatches = (uint32_t)((E + size - 1) / size);
    EG_TRY(t.first.reserve(4ull * (t.nbatches + 1)));
    k_task_batches<<<grid_for(t.ntasks + 1, 256), 256, 0, g->stream>>>(t.rec.as<uint4>(), t.ntasks, (uint32_t)size, t.nbatches,
                                                                       t.first.as<uint32_t>());
    EG_CHECK_LAUNCH("k_task_batches");
    return EG_OK;
}

static int make_tasks(eg_graph* g, RowTasks& t, const uint64_t* begin, uint64_t nitems, const uint32_t* item_vertex) {
    // upper bound on tasks: non-empty items + E / kTaskEdges
    const uint64_t cap = std::min<uint64_t>(nitems, g->E) + g->E / kTaskEdges + 2;
    EG_TRY(t.rec.reserve(sizeof(uint4) * cap));
    EG_TRY(t.heavy_vertex.reserve(sizeof(uint32_t) * (g->E / kTaskEdges + 2)));
    EG_TRY(t.counts.reserve(32));
    EG_CUDA(cudaMemsetAsync(t.counts.ptr, 0, 32, g->stream));
    uint64_t* d_total = t.counts.as<uint64_t>();
    uint32_t* d_nheavy = reinterpret_cast<uint32_t*>(t.counts.as<uint64_t>() + 1);
    TaskEpi ep{t.rec.as<uint4>(), begin, item_vertex, t.heavy_vertex.as<uint32_t>(), d_nheavy};
    EG_TRY(launch_scan(g, TaskLoad{begin}, ep, nitems, d_total, "row_tasks"));
    uint64_t h[2] = {0, 0};
    EG_CUDA(cudaMemcpyAsync(h, t.counts.ptr, 16, cudaMemcpyDeviceToHost, g->stream));
    EG_CUDA(cudaStreamSynchronize(g->stream));
    t.ntasks = nitems ? h[0] : 0;
    t.nheavy = (uint32_t)(h[1] & 0xFFFFFFFFu);
    return make_batches(g, t);
}

// ---------------------------------------------------------------------------------------------
// row kernels: a warp per batch of tasks, rows of 64 columns (256 bytes) or 32
struct RowArgs {
    const uint4* rec;
    const uint32_t* first;        // first task of every batch
    const uint32_t* adj;
    const float* w;               // per-edge weight (normalised for PPR, raw for SSSP)
};

// The PPR sweeps read a 256-byte row per edge, 8 bytes per lane.  A warp walks the edges of its batch
// without regard to where lists end: 16 rows are always on their way together, the next ids and
// weights behind them, and a list's sum is stored when its last edge has been added.  (A warp per
// task reads a list of three edges in a step for sixteen, and waits for a record, ids and rows each
// time.)  Rows are asked to stay in L2 (half of them evict-last), ids, weights and results pass through
// evict-first.  1 M vertices, 16 M edges, forward / adjoint sweep: a warp per task by stride, half a
// warp per row 0.53 / 0.75 ms, the walk in CTAs of 8 warps 0.38 / -, of 2 0.35 / 0.61, of 1 0.32 /
// 0.50 (12.9 / 8.2 TB/s of rows; random 256-byte rows out of 256 MB reach 10 TB/s, out of 64 MB 21).
constexpr int kWalkRows = 16;

// A lane's part of a row: two columns of 64 (float2), one of 32 (float)
__device__ __forceinline__ float2 ld_row(const float2* a, unsigned long long keep) {
    float2 v;
    asm volatile("ld.global.cg.L2::cache_hint.v2.f32 {%0, %1}, [%2], %3;" : "=f"(v.x), "=f"(v.y) : "l"(a), "l"(keep));
    return v;
}
__device__ __forceinline__ float ld_row(const float* a, unsigned long long keep) {
    float v;
    asm volatile("ld.global.cg.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(a), "l"(keep));
    return v;
}
__device__ __forceinline__ void row_zero(float2& a) { a = make_float2(0.f, 0.f); }
__device__ __forceinline__ void row_zero(float& a) { a = 0.f; }
__device__ __forceinline__ float2 row_scale(float f, float2 a) { return make_float2(f * a.x, f * a.y); }
__device__ __forceinline__ float row_scale(float f, float a) { return f * a; }
__device__ __forceinline__ float2 row_add(float2 acc, float w, float2 a) {
    return make_float2(fmaf(w, a.x, acc.x), fmaf(w, a.y, acc.y));
}
__device__ __forceinline__ float row_add(float acc, float w, float a) { return fmaf(w, a, acc); }
__device__ __forceinline__ float row_dot(float2 a, float2 b) { return fmaf(a.x, b.x, a.y * b.y); }
__device__ __forceinline__ float row_dot(float a, float b) { return a * b; }

// acc plus four weighted rows, which are added up by themselves first: a long list's sum takes a quarter of
// the roundings
__device__ __forceinline__ float add_four(float acc, const float4& w, float a, float b, float c, float d) {
    return acc + fmaf(w.w, d, fmaf(w.z, c, fmaf(w.y, b, w.x * a)));
}
__device__ __forceinline__ float2 add_four(float2 acc, const float4& w, float2 a, float2 b, float2 c, float2 d) {
    return make_float2(add_four(acc.x, w, a.x, b.x, c.x, d.x), add_four(acc.y, w, a.y, b.y, c.y, d.y));
}

// the seeds of a lane's columns
__device__ __forceinline__ uint2 seeds_at(const uint32_t* seeds, int n, uint32_t lane, float2) {
    return make_uint2(2 * lane < n ? __ldg(seeds + 2 * lane) : ~0u, 2 * lane + 1 < n ? __ldg(seeds + 2 * lane + 1) : ~0u);
}
__device__ __forceinline__ uint2 seeds_at(const uint32_t* seeds, int n, uint32_t lane, float) {
    return make_uint2(lane < n ? __ldg(seeds + lane) : ~0u, ~0u);
}
__device__ __forceinline__ float2 ppr_row(float2 acc, uint32_t v, uint2 seed, float alpha) {
    float2 r = row_scale(1.0f - alpha, acc);
    if (seed.x == v) r.x += alpha;
    if (seed.y == v) r.y += alpha;
    return r;
}
__device__ __forceinline__ float ppr_row(float acc, uint32_t v, uint2 seed, float alpha) {
    const float r = row_scale(1.0f - alpha, acc);
    return seed.x == v ? r + alpha : r;
}

// PPR forward: y[v] = (1-a) * sum_{u in in(v)} wn_uv * x[u] + a * e_seed[v]
template <class Row>
__global__ void __launch_bounds__(32, 32) k_row_spmm(RowArgs a, const Row* __restrict__ x, Row* __restrict__ y,
                                                  Row* __restrict__ heavy_acc, const uint32_t* __restrict__ seeds, int n_seeds,
                                                  float alpha) {
    __shared__ __align__(16) uint32_t id[32];
    __shared__ __align__(16) float wt[32];
    __shared__ __align__(16) uint4 task[32];  // end (from the batch's first edge), vertex, slot
    __shared__ __align__(8) uint2 s_seed[32];               // seeds of the lanes' columns
    const uint32_t lane = threadIdx.x;
    s_seed[lane] = seeds_at(seeds, n_seeds, lane, Row());
    unsigned long long keep;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 0.5;" : "=l"(keep));
    const uint32_t b = blockIdx.x;
    uint32_t t = __ldg(a.first + b);
    const uint32_t t1 = __ldg(a.first + b + 1);
    if (t == t1) return;
    const uint4 last = __ldg(a.rec + t1 - 1), tasks0 = t + lane < t1 ? __ldg(a.rec + t + lane) : last;
    const uint64_t e0 = __shfl_sync(0xffffffffu, task_begin(tasks0), 0);
    const uint32_t n = (uint32_t)(task_begin(last) - e0) + task_len(last);
    auto stage = [&](const uint4& r) {  // 32 tasks of the batch
        __syncwarp();
        task[lane] = make_uint4((uint32_t)(task_begin(r) - e0) + task_len(r), r.z, r.w, 0u);
        __syncwarp();
        t += 32;
    };
    const uint32_t* adj = a.adj + e0 + lane;
    const float* wts = a.w + e0 + lane;
    x += lane;
    uint32_t u = lane < n ? __ldcs(adj) : 0u;
    float w = lane < n ? __ldcs(wts) : 0.f;
    stage(tasks0);
    uint32_t k = 0, lists = t1 - t + 32;  // of the batch (t is 32 tasks ahead)
    uint32_t end = task[0].x;
    Row acc;
    row_zero(acc);
    auto finish = [&]() {
        const uint4 cur = task[k];
        if (cur.z == kNoSlot) __stcs(y + (uint64_t)cur.y * 32 + lane, ppr_row(acc, cur.y, s_seed[lane], alpha));
        else atomicAdd(heavy_acc + (uint64_t)cur.z * 32 + lane, acc);
        row_zero(acc);
        if (++k == 32) {
            stage(t + lane < t1 ? __ldg(a.rec + t + lane) : last);
            k = 0;
        }
        end = --lists ? task[k].x : ~0u;
    };
    for (uint32_t c = 0; c < n; c += 32) {
        __syncwarp();
        id[lane] = u;
        wt[lane] = w;
        __syncwarp();
        u = 0;
        if (c + 32 + lane < n) {
            u = __ldcs(adj + c + 32);
            w = __ldcs(wts + c + 32);
        }
        const uint32_t left = n - c < 32 ? n - c : 32;
        for (uint32_t s = 0; s < left; s += kWalkRows) {
            Row r[kWalkRows];
#pragma unroll
            for (int j = 0; j < kWalkRows; j += 4) {  // past the batch's last edge: row 0, not used
                const uint4 q = *reinterpret_cast<const uint4*>(id + s + j);
                r[j] = ld_row(x + (uint64_t)q.x * 32, keep);
                r[j + 1] = ld_row(x + (uint64_t)q.y * 32, keep);
                r[j + 2] = ld_row(x + (uint64_t)q.z * 32, keep);
                r[j + 3] = ld_row(x + (uint64_t)q.w * 32, keep);
            }
#pragma unroll
            for (int j = 0; j < kWalkRows; j += 4) {
                const float4 q = *reinterpret_cast<const float4*>(wt + s + j);
                const uint32_t at = c + s + j;
                if (at + 4 < end) {  // no list ends here
                    acc = add_four(acc, q, r[j], r[j + 1], r[j + 2], r[j + 3]);
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float qi = i == 0 ? q.x : i == 1 ? q.y : i == 2 ? q.z : q.w;
                        acc = row_add(acc, qi, r[j + i]);
                        if (at + i + 1 == end) finish();
                    }
                }
            }
        }
    }
}

// the rows of lists cut into several tasks (seeds null: no teleport), one warp each
template <class Row>
__global__ void k_row_heavy_finish(const uint32_t* __restrict__ heavy_vertex, uint32_t nheavy,
                                   Row* __restrict__ heavy_acc, Row* __restrict__ y, const uint32_t* __restrict__ seeds,
                                   int n_seeds, float alpha) {
    const uint32_t slot = (uint32_t)((blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (slot >= nheavy) return;
    const uint32_t v = heavy_vertex[slot];
    Row* p = heavy_acc + (uint64_t)slot * 32 + lane;
    y[(uint64_t)v * 32 + lane] = ppr_row(*p, v, seeds_at(seeds, n_seeds, lane, Row()), alpha);
    row_zero(*p);
}

// Seeds without in-edges: the sweeps leave their rows as they are, a at the seed's column, in nbuf
// consecutive row arrays.
__global__ void k_ppr_lone_seeds(const uint32_t* __restrict__ seeds, int n, const uint32_t* __restrict__ indeg,
                                 float* __restrict__ rows, uint64_t V, int nbuf, float alpha, int width) {
    const int s = threadIdx.x & 63;
    if (s >= n || indeg[seeds[s]]) return;
    for (int b = blockIdx.x; b < nbuf; b += gridDim.x) rows[((uint64_t)b * V + seeds[s]) * width + s] = alpha;
}
__global__ void k_ppr_init(const uint32_t* seeds, int n, float* x, int width) {
    const int s = threadIdx.x;
    if (s < n) x[(uint64_t)seeds[s] * width + s] = 1.0f;
}
// zero the rows that no sweep writes (deg = 0) in nbuf consecutive row arrays
__global__ void __launch_bounds__(256) k_zero_rows(const uint32_t* __restrict__ deg, uint64_t V, float4* __restrict__ rows,
                                                   int nbuf, int parts) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < V * parts; i += stride) {
        if (deg[i / (uint32_t)parts]) continue;
        for (int b = 0; b < nbuf; ++b) __stcs(rows + (uint64_t)b * V * parts + i, make_float4(0.f, 0.f, 0.f, 0.f));
    }
}

__device__ __forceinline__ double warp_sum_f64(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Row normalisation and its gradient over the CSR tasks (<= 512 edges of one source), a batch of them per warp:
// 32 tasks at a time, each lane those of up to kLane edges by itself (if a few of them are), the warp together the
// longer ones, so that neither a hub's list nor a graph of short lists leaves lanes idle.  A list of one task
// is finished here; of a longer one the FP64 partial sums meet in heavy[slot] and its tasks are finished by a
// second pass (finish_heavy).  Bound by the random 4-byte reads of the input-ordered weights.  Weights of the
// forward, with one thread per source / a warp per task by stride / so: 1 M R-MAT sources, 16 M edges
// 7.9 / 0.49 / 0.34 ms; 1 M uniform, 16 M 0.46 / 0.70 / 0.28; 8 M uniform, 8 M 0.34 / 2.8 / 0.24.
constexpr int kTaskThreads = 64;  // two batches per CTA, 64 warps per SM
constexpr int kLaneTasks = 4;
// Uniform lists of 32 edges: weights 0.25 ms with lists of up to 32 edges by a lane, 0.25 up to 16; gradients, with
// two FP64 reads per edge, 0.34 and 0.27.  Of 16 edges: 0.28 and 0.48; 0.38 and 0.52, as up to 24.
constexpr uint32_t kLaneWeights = 32, kLaneGrad = 24;

// f(task, k0, step): a lane's own short task with 0, 1; a long one with lane, 32, all lanes together
template <uint32_t kLane, class F>
__device__ __forceinline__ void each_task(const uint4* __restrict__ tasks, const uint32_t* __restrict__ first,
                                          uint32_t nbatches, F f) {
    const uint32_t lane = threadIdx.x & 31, b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (b >= nbatches) return;
    const uint32_t t1 = __ldg(first + b + 1);
    for (uint32_t t = __ldg(first + b); t < t1; t += 32) {
        const uint4 own = t + lane < t1 ? __ldg(tasks + t + lane) : make_uint4(0, 0, 0, kNoSlot);
        const uint32_t n = task_len(own);
        const uint32_t some = __ballot_sync(0xffffffffu, n != 0), lng = __ballot_sync(0xffffffffu, n > kLane);
        const bool lanes = __popc(some & ~lng) >= kLaneTasks;
        if (lanes && n && n <= kLane) f(own, 0u, 1u);
        for (uint32_t m = lanes ? lng : some; m; m &= m - 1) {
            const int l = __ffs(m) - 1;
            const uint4 rec = make_uint4(__shfl_sync(0xffffffffu, own.x, l), __shfl_sync(0xffffffffu, own.y, l),
                                         __shfl_sync(0xffffffffu, own.z, l), __shfl_sync(0xffffffffu, own.w, l));
            f(rec, lane, 32u);
        }
    }
}

// s[u] = sum of u's out-weights; wn[e] = w[eid[e]] / s[u] (null: not wanted)
__global__ void __launch_bounds__(kTaskThreads, 32) k_out_weights(const uint4* __restrict__ tasks,
                                                     const uint32_t* __restrict__ first, uint32_t nbatches,
                                                     const float* __restrict__ eid, const float* __restrict__ w_in,
                                                     float* __restrict__ s, float* __restrict__ wn,
                                                     double* __restrict__ heavy, int finish_heavy) {
    each_task<kLaneWeights>(tasks, first, nbatches, [&](const uint4& rec, uint32_t k0, uint32_t step) {
        if (finish_heavy && rec.w == kNoSlot) return;
        const uint64_t e0 = task_begin(rec);
        const uint32_t n = task_len(rec);
        float sum;
        if (finish_heavy) {
            sum = s[rec.z];
        } else {
            double acc = 0;
#pragma unroll 4
            for (uint32_t k = k0; k < n; k += step) acc += w_in[__float_as_uint(__ldg(eid + e0 + k))];
            if (step > 1) acc = warp_sum_f64(acc);
            sum = (float)acc;
            if (k0 == 0) {
                if (rec.w == kNoSlot) s[rec.z] = sum;
                else atomicAdd(heavy + rec.w, acc);
            }
            if (rec.w != kNoSlot) return;
        }
        if (wn)
#pragma unroll 4
            for (uint32_t k = k0; k < n; k += step) wn[e0 + k] = w_in[__float_as_uint(__ldg(eid + e0 + k))] / sum;
    });
}
__global__ void k_heavy_out_sums(const uint32_t* __restrict__ heavy_vertex, uint32_t nheavy,
                                 const double* __restrict__ heavy, float* __restrict__ s) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nheavy) s[heavy_vertex[i]] = (float)heavy[i];
}
__global__ void k_gather_norm_w(const uint32_t* __restrict__ nbr_is_src, const float* __restrict__ eid,
                                const float* __restrict__ w_in, const float* __restrict__ s, uint64_t E,
                                float* __restrict__ wn) {
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < E; e += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t id = __float_as_uint(eid[e]);
        wn[e] = w_in[id] / s[nbr_is_src[e]];
    }
}

// ---- adjoint sweep over the CSR: for a source row u,
//   lam_out[u] = (1-a) * sum_{v in out(u)} wn_uv * lam_in[v]
//   gA[e]     += (1-a) * <x_k[u], lam_in[v]>      (per CSR edge e = (u, v))
// The walk of k_row_spmm, with the source rows x_k[u] of the next 8 to 16 lists on their way to shared
// memory.  A step's 16 dot products <x_k[u], lam[v]> are summed over the warp by halving: at each
// stage a lane hands half of its partial sums to its partner and keeps the other half, so that 16
// products take 16 shuffles (one at a time: 80); lane 2 j and its neighbour end up with product j.  gA is
// kept in FP64: an edge's gradient is what is left of its gA minus the mean over the source's edges,
// and the roundings of K steps were most of its error (K = 50, 1 M / 16 M, two seeds: 1.1e-6 and
// 8.5e-7 with FP32 sums, 7.9e-7 and 5.4e-7 so, for 24.9 instead of 23.6 ms of sweeps).
__device__ __forceinline__ float dot_scatter(float (&d)[kWalkRows], uint32_t lane) {
    static_assert(kWalkRows == 16, "the four halving stages below leave one product of sixteen per lane pair");
#pragma unroll
    for (int o = 16, m = 8; o >= 2; o >>= 1, m >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int j = 0; j < m; ++j) {
            const float give = up ? d[j] : d[j + m], keep = up ? d[j + m] : d[j];
            d[j] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    return d[0] + __shfl_xor_sync(0xffffffffu, d[0], 1);
}

// 28 warps per SM (72 registers): 32 (64, spilled) 28.5 ms for 50 sweeps, 24 27.5, 28 25.4.
template <class Row>
__global__ void __launch_bounds__(32, 28) k_row_adjoint(RowArgs a, const Row* __restrict__ lam_in,
                                                     const Row* __restrict__ xk, Row* __restrict__ lam_out,
                                                     Row* __restrict__ heavy_acc, double* __restrict__ gA,
                                                     float scale) {
    __shared__ __align__(16) uint32_t id[32];
    __shared__ __align__(16) float wt[32];
    __shared__ __align__(16) uint4 task[16];      // ring of 16: end, vertex, slot
    __shared__ __align__(16) Row src[16][32];  // and their rows of x_k
    const uint32_t lane = threadIdx.x & 31;
    unsigned long long keep;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 0.5;" : "=l"(keep));
    const uint32_t b = blockIdx.x;
    const uint32_t t0 = __ldg(a.first + b), lists = __ldg(a.first + b + 1) - t0;
    if (!lists) return;
    auto tasks_at = [&](uint32_t i) {
        return lane < 8 && i + lane < lists ? __ldg(a.rec + t0 + i + lane) : make_uint4(0, 0, 0, 0);
    };
    const uint4 last = __ldg(a.rec + t0 + lists - 1), tasks0 = tasks_at(0), tasks8 = tasks_at(8);
    uint4 ahead = tasks_at(16);
    const uint64_t e0 = __shfl_sync(0xffffffffu, task_begin(tasks0), 0);
    const uint32_t n = (uint32_t)(task_begin(last) - e0) + task_len(last);
    auto stage = [&](const uint4& r, uint32_t slot) {  // 8 tasks (lanes 0..7) into the ring, their rows on the way
        if (lane < 8) task[slot + lane] = make_uint4((uint32_t)(task_begin(r) - e0) + task_len(r), r.z, r.w, 0u);
        constexpr uint32_t kLanes = 2 * sizeof(Row), kPart = 16 / sizeof(Row);  // lanes per row, 16 bytes each
#pragma unroll
        for (int i = 0; i < 8 * kLanes / 32; ++i) {
            const uint32_t q = 32 / kLanes * i + lane / kLanes, v = __shfl_sync(0xffffffffu, r.z, q);
            if (__shfl_sync(0xffffffffu, task_len(r), q))
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                                 (uint32_t)__cvta_generic_to_shared(&src[slot + q][kPart * (lane % kLanes)])),
                             "l"(xk + (uint64_t)v * 32 + kPart * (lane % kLanes))
                             : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const uint32_t* adj = a.adj + e0 + lane;
    const float* wts = a.w + e0 + lane;
    double* g = gA + e0 + (lane >> 1);
    lam_in += lane;
    uint32_t v = lane < n ? __ldcs(adj) : 0u;
    float w = lane < n ? __ldcs(wts) : 0.f;
    stage(tasks0, 0);
    stage(tasks8, 8);
    __syncwarp();
    uint32_t k = 0, end = task[0].x;
    Row xu, acc;
    row_zero(xu);
    row_zero(acc);
    auto finish = [&]() {
        const uint4 cur = task[k & 15];
        if (cur.z == kNoSlot) __stcs(lam_out + (uint64_t)cur.y * 32 + lane, row_scale(scale, acc));
        else atomicAdd(heavy_acc + (uint64_t)cur.z * 32 + lane, acc);
        row_zero(acc);
        ++k;
        if (!(k & 7)) {  // the finished eight make room
            __syncwarp();
            stage(ahead, (k + 8) & 15);
            ahead = tasks_at(k + 16);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncwarp();
        }
        end = k < lists ? task[k & 15].x : ~0u;
        xu = src[k & 15][lane];
    };
    for (uint32_t c = 0; c < n; c += 32) {
        __syncwarp();
        id[lane] = v;
        wt[lane] = w;
        __syncwarp();
        v = 0;
        if (c + 32 + lane < n) {
            v = __ldcs(adj + c + 32);
            w = __ldcs(wts + c + 32);
        }
        const uint32_t left = n - c < 32 ? n - c : 32;
        for (uint32_t s = 0; s < left; s += kWalkRows) {
            const bool have = !(lane & 1) && s + (lane >> 1) < left;
            const double g_old = have ? g[c + s] : 0.0;
            Row l[kWalkRows];
            float d[kWalkRows];
#pragma unroll
            for (int j = 0; j < kWalkRows; j += 4) {  // past the batch's last edge: row 0, not used
                const uint4 q = *reinterpret_cast<const uint4*>(id + s + j);
                l[j] = ld_row(lam_in + (uint64_t)q.x * 32, keep);
                l[j + 1] = ld_row(lam_in + (uint64_t)q.y * 32, keep);
                l[j + 2] = ld_row(lam_in + (uint64_t)q.z * 32, keep);
                l[j + 3] = ld_row(lam_in + (uint64_t)q.w * 32, keep);
            }
            if (c + s == 0) {  // the first source rows
                asm volatile("cp.async.wait_group 1;" ::: "memory");
                __syncwarp();
                xu = src[0][lane];
            }
#pragma unroll
            for (int j = 0; j < kWalkRows; j += 4) {
                const float4 q = *reinterpret_cast<const float4*>(wt + s + j);
                const uint32_t at = c + s + j;
                if (at + 4 < end) {  // no list ends here
                    acc = add_four(acc, q, l[j], l[j + 1], l[j + 2], l[j + 3]);
#pragma unroll
                    for (int i = 0; i < 4; ++i) d[j + i] = row_dot(xu, l[j + i]);
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float qi = i == 0 ? q.x : i == 1 ? q.y : i == 2 ? q.z : q.w;
                        acc = row_add(acc, qi, l[j + i]);
                        d[j + i] = row_dot(xu, l[j + i]);
                        if (at + i + 1 == end) finish();
                    }
                }
            }
            const float dot = dot_scatter(d, lane);
            if (have) g[c + s] = fma((double)scale, (double)dot, g_old);
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// dL/dw_e = (gA_e - sum_{e' in row(u)} wn_e' gA_e') / s_u, scattered to the input edge order
__global__ void __launch_bounds__(kTaskThreads, 32) k_weight_grad(const uint4* __restrict__ tasks,
                                                     const uint32_t* __restrict__ first, uint32_t nbatches,
                                                     const float* __restrict__ wn, const double* __restrict__ gA,
                                                     const float* __restrict__ s, const float* __restrict__ eid,
                                                     float* __restrict__ dw, double* __restrict__ heavy,
                                                     int finish_heavy) {
    each_task<kLaneGrad>(tasks, first, nbatches, [&](const uint4& rec, uint32_t k0, uint32_t step) {
        if (finish_heavy && rec.w == kNoSlot) return;
        const uint64_t e0 = task_begin(rec);
        const uint32_t n = task_len(rec);
        double dot = 0;
        if (finish_heavy) {
            dot = heavy[rec.w];
        } else {
#pragma unroll 4
            for (uint32_t k = k0; k < n; k += step) dot += wn[e0 + k] * gA[e0 + k];
            if (step > 1) dot = warp_sum_f64(dot);
            if (rec.w != kNoSlot) {
                if (k0 == 0) atomicAdd(heavy + rec.w, dot);
                return;
            }
        }
        const float inv = 1.0f / s[rec.z];
#pragma unroll 4
        for (uint32_t k = k0; k < n; k += step)
            dw[__float_as_uint(__ldg(eid + e0 + k))] = (float)((gA[e0 + k] - dot) * inv);
    });
}

// ---- batched SSSP: in place, skipping sources whose row did not change in the last sweep --------
// A warp walks the edges of its batch, 32 at a time: sources that did not change (one bit each, cached in
// L1: the bits do not change during a sweep) are dropped, the others queue up in shared memory, the
// sources of a list behind an entry for the list's own row.  16 queued rows are gathered together,
// whatever lists they belong to; a list whose row was not lowered costs nothing more, one without
// changed sources is never looked at.  Ids are on their way two steps ahead and bits one; the tasks are
// read when the first changed source turns up.  A destination with a single task is written by this
// warp alone and stored plainly; cut lists (and items of several partitions that share a vertex)
// take the minimum with atomics.  The sweep is bound by the row gathers.  64 graphs of 1k-500k vertices,
// 93 M edges, 64 sources, 24 sweeps: 107 ms with one row per warp load, byte flags and separate item /
// offset arrays; a task at a time, rows by half-warps, tasks by stride 47.5 ms, in batches with a
// warp per CTA 39.7; the walk 28.8 (10.8 E row gathers: 8.9 TB/s) at 32 warps per SM, 30.5 at 28,
// 33.7 at 24.
__device__ __forceinline__ float relaxed(float best, float msg, float w) { return fminf(best, msg + w); }  // toolkits/sssp.cpp:55
__device__ __forceinline__ float2 relaxed(float2 best, float2 msg, float w) {
    return make_float2(relaxed(best.x, msg.x, w), relaxed(best.y, msg.y, w));
}
__device__ __forceinline__ bool lower(float a, float b) { return a < b; }
__device__ __forceinline__ bool lower(float2 a, float2 b) { return a.x < b.x || a.y < b.y; }
// distances are >= 0: ordered like their bits
__device__ __forceinline__ bool lower_atomic(float* p, float a, float b) {
    return a < b && a < __int_as_float(atomicMin(reinterpret_cast<int*>(p), __float_as_int(a)));
}
__device__ __forceinline__ bool lower_atomic(float2* p, float2 a, float2 b) {
    const bool x = lower_atomic(&p->x, a.x, b.x), y = lower_atomic(&p->y, a.y, b.y);
    return x || y;
}

constexpr int kSsspRows = 16;
constexpr uint32_t kDestRow = 1u << 31;  // queue entry: the list's own row

template <class Row>
__global__ void __launch_bounds__(32, 32) k_row_sssp(RowArgs a, Row* __restrict__ dist,
                                                     const uint32_t* __restrict__ changed_prev,
                                                     uint32_t* __restrict__ changed_next, int shared_vertex,
                                                     int* __restrict__ any) {
    static_assert(kBatchEdges + kTaskEdges <= 32 * 32, "a batch's list starts are one bit per edge in s_head");
    __shared__ uint2 s_task[kBatchEdges];              // the batch's tasks: vertex, slot
    __shared__ uint32_t s_head[32];                    // bit e: a task begins with edge e of the batch
    __shared__ __align__(16) uint32_t q_row[kSsspRows + 64], q_edge[kSsspRows + 64];
    const uint32_t lane = threadIdx.x, lt = (1u << lane) - 1u, le = lt | (1u << lane);
    const uint32_t t0 = __ldg(a.first + blockIdx.x), tasks = __ldg(a.first + blockIdx.x + 1) - t0;
    if (!tasks) return;
    const uint4 begin = __ldg(a.rec + t0), last = __ldg(a.rec + t0 + tasks - 1);
    const uint64_t e0 = task_begin(begin);
    const uint32_t n = (uint32_t)(task_begin(last) - e0) + task_len(last);
    const uint32_t* adj = a.adj + e0 + lane;
    const float* wts = a.w + e0;
    dist += lane;
    bool loaded = false, any_lowered = false;
    uint32_t before = 0;       // tasks that begin before this chunk
    uint32_t queued = 0;
    uint32_t q_task = ~0u;     // task of the last queued source
    uint32_t cur = ~0u;        // task whose row is being reduced
    Row dv, best;
    row_zero(dv);
    row_zero(best);
    auto flush = [&]() {
        bool low = lower(best, dv);
        if (cur == ~0u || !__any_sync(0xffffffffu, low)) return;
        const uint2 tk = s_task[cur];
        Row* row = dist + (uint64_t)tk.x * 32;
        if (tk.y == kNoSlot && !shared_vertex) {
            if (low) __stcg(row, best);
        } else {
            low = lower_atomic(row, best, dv);
            if (!__any_sync(0xffffffffu, low)) return;
        }
        if (lane == 0) atomicOr(changed_next + (tk.x >> 5), 1u << (tk.x & 31));
        any_lowered = true;
    };
    auto reduce = [&](uint32_t base, uint32_t m) {  // entries [base, base + m) of the queue, m <= kSsspRows
        const uint32_t qe = lane < m ? q_edge[base + lane] : kDestRow;
        const float wl = qe & kDestRow ? 0.f : __ldg(wts + qe);
        Row r[kSsspRows];
#pragma unroll
        for (int j = 0; j < kSsspRows; j += 4) {
            const uint4 q = *reinterpret_cast<const uint4*>(q_row + base + j);
            if (j < m) r[j] = __ldcg(dist + (uint64_t)q.x * 32);
            if (j + 1 < m) r[j + 1] = __ldcg(dist + (uint64_t)q.y * 32);
            if (j + 2 < m) r[j + 2] = __ldcg(dist + (uint64_t)q.z * 32);
            if (j + 3 < m) r[j + 3] = __ldcg(dist + (uint64_t)q.w * 32);
        }
#pragma unroll
        for (int j = 0; j < kSsspRows; ++j) {
            if (j >= m) break;
            const uint32_t e = __shfl_sync(0xffffffffu, qe, j);
            const float w = __shfl_sync(0xffffffffu, wl, j);
            if (e & kDestRow) {
                flush();
                cur = e ^ kDestRow;
                dv = best = r[j];
            } else {
                best = relaxed(best, r[j], w);
            }
        }
    };
    uint32_t u0 = lane < n ? __ldg(adj) : 0u, u1 = lane + 32 < n ? __ldg(adj + 32) : 0u;
    uint32_t b0 = lane < n ? __ldg(changed_prev + (u0 >> 5)) : 0u;
    for (uint32_t c = 0; c < n; c += 32) {
        const uint32_t u2 = c + 64 + lane < n ? __ldg(adj + c + 64) : 0u;
        const uint32_t b1 = c + 32 + lane < n ? __ldg(changed_prev + (u1 >> 5)) : 0u;
        const bool active = (b0 >> (u0 & 31)) & 1u;
        const uint32_t m = __ballot_sync(0xffffffffu, active);
        if (m && !loaded) {
            loaded = true;
            s_head[lane] = 0;
            __syncwarp();
            for (uint32_t i = lane; i < tasks; i += 32) {
                const uint4 r = __ldg(a.rec + t0 + i);
                s_task[i] = make_uint2(r.z, r.w);
                const uint32_t at = (uint32_t)(task_begin(r) - e0);
                atomicOr(s_head + (at >> 5), 1u << (at & 31));
            }
            __syncwarp();
            before = __reduce_add_sync(0xffffffffu, lane < (c >> 5) ? __popc(s_head[lane]) : 0);
        }
        if (loaded) {
            const uint32_t heads = s_head[c >> 5];
            if (m) {
                const uint32_t task = before + __popc(heads & le) - 1;
                const uint32_t prev = m & lt;  // active sources before this one
                const uint32_t since = prev ? (2u << (31 - __clz(prev))) - 1u : 0u;
                const bool first = active && (prev ? (heads & le & ~since) != 0 : task != q_task);
                const uint32_t f = __ballot_sync(0xffffffffu, first);
                uint32_t at = queued + __popc(prev) + __popc(f & lt);
                if (first) {
                    q_row[at] = s_task[task].x;
                    q_edge[at++] = kDestRow | task;
                }
                if (active) {
                    q_row[at] = u0;
                    q_edge[at] = c + lane;
                }
                q_task = __shfl_sync(0xffffffffu, task, 31 - __clz(m));
                queued += __popc(m) + __popc(f);
                __syncwarp();
                uint32_t done = 0;
                for (; queued - done >= kSsspRows; done += kSsspRows) reduce(done, kSsspRows);
                if (done) {  // the rest to the front
                    queued -= done;
                    const uint32_t r = lane < queued ? q_row[done + lane] : 0u, e = lane < queued ? q_edge[done + lane] : 0u;
                    __syncwarp();
                    if (lane < queued) {
                        q_row[lane] = r;
                        q_edge[lane] = e;
                    }
                    __syncwarp();
                }
            }
            before += __popc(heads);
        }
        u0 = u1;
        u1 = u2;
        b0 = b1;
    }
    if (queued) reduce(0, queued);
    flush();
    if (any_lowered && lane == 0) *any = 1;
}

__global__ void k_fill_f32_rows(float* p, uint64_t n, float v) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) p[i] = v;
}

// {src, dst} records -> {src, dst, index} records: the index rides through the build in the weight
// slot, so every CSR / CSC position knows which input edge it holds
__global__ void k_expand_ids(const uint2* __restrict__ in, uint64_t E, uint32_t* __restrict__ out) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < E; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint2 r = in[i];
        out[3 * i] = r.x;
        out[3 * i + 1] = r.y;
        out[3 * i + 2] = (uint32_t)i;
    }
}

int expand_with_ids(eg_graph* g, const uint8_t* rec8_dev, uint64_t E) {
    if (!E) return EG_OK;
    k_expand_ids<<<grid_for(E, 256, 152u * 16u), 256, 0, g->stream>>>(reinterpret_cast<const uint2*>(rec8_dev), E,
                                                                      g->edges.as<uint32_t>());
    EG_CHECK_LAUNCH("k_expand_ids");
    return EG_OK;
}

// ---------------------------------------------------------------------------------------------
struct BatchState {
    DevBuf ticket, a64, b64, c64, lev, rows0, rows1, heavy, tmp_out, seeds, wn_csc, wn_csr, s_out, gA, heavy_sum, ck, seg;
    DevBuf ch0, ch1, flag, level_cnt, entries, n_entries, bm0, bm1, alive, ms_seg;
    DevBuf cap;      // captured level loop: per-level direction decisions and frontier edge counts
    DevBuf persist;  // persistent traversal: per-level counts, barrier words, error flag
    DevBuf wr0, wr1;  // frontier words in renumbered order (pull gathers through renumbered sources)
    RowTasks csc_tasks, csr_tasks;
    bool csc_ready = false, csr_ready = false;
    // captured MS-BFS level loop and the shapes it was captured for
    void* graph_exec = nullptr;
    uint64_t graph_V = 0;
    bool graph_lev = false;
    uint32_t graph_entries = 0;
    int graph_nbits = 0;
    int graph_div = 0;  // the switch's divisor the captured levels compare with
    ~BatchState() {
        if (graph_exec) cudaGraphExecDestroy((cudaGraphExec_t)graph_exec);
    }
};

static BatchState& bstate(eg_graph* g) {
    if (!g->batch) g->batch = new BatchState();
    return *static_cast<BatchState*>(g->batch);
}

void free_batch_state(eg_graph* g) {
    delete static_cast<BatchState*>(g->batch);
    g->batch = nullptr;
}

static int copy_small_in(eg_graph* g, DevBuf& dst, const uint32_t* src, int n, int where) {
    EG_TRY(dst.reserve(sizeof(uint32_t) * 64));
    EG_CUDA(cudaMemcpyAsync(dst.ptr, src, sizeof(uint32_t) * n,
                            where == EG_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, g->stream));
    return EG_OK;
}

static int check_roots(eg_graph* g, const uint32_t* roots, int n, int where, const char* fn) {
    if (!roots || n < 1 || n > 64) {
        set_error("%s: need 1..64 roots", fn);
        return EG_ERR_INVALID;
    }
    std::vector<uint32_t> h(n);
    EG_CUDA(cudaMemcpy(h.data(), roots, sizeof(uint32_t) * n,
                       where == EG_DEVICE ? cudaMemcpyDeviceToHost : cudaMemcpyHostToHost));
    for (int i = 0; i < n; ++i)
        if (h[i] >= g->V) {
            set_error("%s: root %u >= V %u", fn, h[i], g->V);
            return EG_ERR_INVALID;
        }
    return EG_OK;
}

// root entries (global vertex, bit) from n roots: entry s = (roots[s] + base, s)
__global__ void k_root_entries(const uint32_t* roots, int n, uint32_t base, uint2* ent) {
    const int s = threadIdx.x;
    if (s < n) ent[s] = make_uint2(roots[s] + base, (uint32_t)s);
}

// per-graph roots of a graph batch: entry (g * nper + s) = (voff[g] + roots[g * nper + s], s)
__global__ void k_root_entries_graphs(const uint32_t* roots, const uint64_t* voff, uint32_t ngraphs, int nper,
                                      uint2* ent) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i < (uint64_t)ngraphs * nper) {
        const uint64_t gi = i / nper;
        ent[i] = make_uint2((uint32_t)(voff[gi] + roots[i]), (uint32_t)(i % nper));
    }
}

__global__ void k_msbfs_init_entries(const uint2* ent, const uint32_t* n_dev, unsigned long long* visit,
                                     unsigned long long* front, unsigned long long* front_bm,
                                     unsigned long long* planes, uint32_t* q, uint32_t* nq, unsigned long long* act_edges, const uint32_t* deg) {
    const uint32_t n = *n_dev;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t v = ent[i].x, s = ent[i].y;
        const unsigned long long bit = 1ull << s;
        atomicOr(visit + v, bit);
        if (atomicOr(front + v, bit) == 0ull) {
            atomicOr(front_bm + (v >> 6), 1ull << (v & 63));
            q[atomicAdd(nq, 1u)] = v;
            atomicAdd(act_edges, (unsigned long long)deg[v]);
            if (planes) {  // level 0
                ulonglong2* p = reinterpret_cast<ulonglong2*>(planes + (uint64_t)v * 4);
                p[0] = p[1] = make_ulonglong2(0ull, 0ull);
            }
        }
    }
}

constexpr int kGraphLevels = 16;

// The captured level loop makes, on the device, the choice the host loop makes per level: each
// level's first kernel reads the frontier's length and out-edges and arms either the pull kernels
// (the full sweep for the first dense level, the early-exit pair after it on one graph) or the
// push (a scan and expansion whose item count it sets); the kernels of the other path find
// nothing to do.  After an empty frontier every later level is disarmed.
struct CapLevel {
    uint32_t n_push;   // queue length handed to the push scan and expansion (0: pull level)
    int skip_direct;   // k_pull_direct (MsBfsPullOp::stop)
    int skip_early;    // k_ms_head / k_ms_tail (MsBuArgs::stop)
    int pad;
};
struct CapState {
    CapLevel lv[kGraphLevels];
    unsigned long long act[kGraphLevels];  // out-edges of the frontier level L produced
    uint64_t push_total;                   // edges of the current push level (scan total)
    int dense_count;
    int stop;
};

__global__ void k_cap_decide(CapState* st, int L, const uint32_t* n_src, const unsigned long long* act_src,
                             unsigned long long dense_min, int early_after_first, int built_csr) {
    CapLevel& c = st->lv[L];
    const uint32_t n = *n_src;
    if (st->stop || n == 0) {
        st->stop = 1;
        c.n_push = 0;
        c.skip_direct = c.skip_early = 1;
        return;
    }
    const bool dense = !built_csr || *act_src >= dense_min;
    const bool early = dense && early_after_first && st->dense_count > 0;
    c.n_push = dense ? 0u : n;
    c.skip_direct = !(dense && !early);
    c.skip_early = !(dense && early);
    if (dense) ++st->dense_count;
}

// zero the frontier words a queue lists (its length read on the device), or the whole array when
// the queue is long; nothing once the loop has stopped
__global__ void k_clear_front_dev(const uint32_t* __restrict__ q, const uint32_t* n_dev, unsigned long long* word,
                                  uint64_t V, const CapState* st) {
    if (st->stop) return;
    const uint32_t n = __ldcg(n_dev);
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    if ((uint64_t)n > V / 32) {
        for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V; v += stride) word[v] = 0ull;
    } else {
        for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += stride) word[q[i]] = 0ull;
    }
}

// ---------------------------------------------------------------------------------------------
// The whole bit-parallel traversal in one persistent launch (EG_OPT_BATCH_LAUNCH = 1): every
// resident CTA runs every level, phase by phase, with a grid barrier between phases -- the same
// phases as the host-driven loop (clear, push or pull by the E / divisor switch, list the next
// frontier, level bytes), with the switch and the queue lengths read on the device.  A launch
// that could not keep all its CTAs resident is refused by the cooperative launch, and every
// barrier wait is bounded: on exhaustion the error flag is raised and the kernel returns.
constexpr int kMaxLevels = 256;

struct PersistWords {
    uint32_t cnt[kMaxLevels];          // queue length produced by level L
    unsigned long long act[kMaxLevels];  // out-edges of that queue
    uint32_t nseg[kMaxLevels];         // early-exit segments of level L
    uint32_t ticket[kMaxLevels];       // scan tile tickets of level L
    uint32_t chunk[kMaxLevels];        // pull chunk tickets of level L
    uint64_t total[kMaxLevels];        // push edges of level L
    unsigned bar_count, bar_gen;
    int err;
    uint32_t levels, pushes;
};

struct MsPersistArgs {
    uint64_t V, nwords;
    int P;
    const uint64_t* csr_off;
    const uint32_t* csr_adj;
    const uint32_t* gather_adj;
    const uint64_t* cidx;
    const uint32_t* cvert;
    uint64_t nitems;
    const uint32_t* pull_chunk_item;
    uint64_t E;
    const uint32_t* deg;
    unsigned long long* visit;
    unsigned long long* word0;
    unsigned long long* word1;
    unsigned long long* bm0;
    unsigned long long* bm1;
    uint32_t* q0;
    uint32_t* q1;
    const unsigned long long* alive_all;
    unsigned long long* lev;  // level planes
    unsigned long long* ms_seg;
    uint64_t* desc;
    uint64_t* ipref;
    uint32_t* push_chunk_item;
    const uint32_t* init_n;
    const unsigned long long* init_act;
    unsigned long long dense_min;
    int early_after_first, built_csr;
    PersistWords* w;
};

// bounded grid barrier (all CTAs resident): false when a wait ran out
__device__ __forceinline__ bool grid_barrier(PersistWords* w) {
    return grid_sync_bounded(&w->bar_count, &w->bar_gen, &w->err);
}

__global__ void __launch_bounds__(256, 4) k_msbfs_persistent(MsPersistArgs a) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    PersistWords* w = a.w;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t n = __ldcg(a.init_n);
    unsigned long long act = __ldcg(a.init_act);
    int dense_count = 0;
    for (uint32_t L = 0; L < 254 && n > 0; ++L) {
        const int c = L & 1;
        unsigned long long* front = c ? a.word1 : a.word0;
        unsigned long long* next = c ? a.word0 : a.word1;
        const unsigned long long* front_bm = c ? a.bm1 : a.bm0;
        unsigned long long* next_bm = c ? a.bm0 : a.bm1;
        const uint32_t* q = c ? a.q1 : a.q0;
        uint32_t* q_next = c ? a.q0 : a.q1;
        const bool dense = !a.built_csr || act >= a.dense_min;
        const bool early = dense && a.early_after_first && dense_count > 0;
        // clear: the next-frontier words (set two levels back, listed by q_next; level 0: all of
        // them), its bitmap, and the scan descriptors of a push level
        {
            const uint32_t n_old = L == 0 ? 0xFFFFFFFFu : (L == 1 ? __ldcg(a.init_n) : __ldcg(&w->cnt[L - 2]));
            if (n_old > a.V / 32) {
                for (uint64_t v = tid; v < a.V; v += stride) next[v] = 0ull;
            } else {
                for (uint64_t i = tid; i < n_old; i += stride) next[q_next[i]] = 0ull;
            }
            for (uint64_t i = tid; i < a.nwords; i += stride) next_bm[i] = 0ull;
            if (a.lev && L == kHighPlanes)
                for (uint64_t i = tid; i < 4 * a.V; i += stride) a.lev[4 * a.V + i] = 0ull;
            if (!dense) {
                const uint64_t tiles = ((uint64_t)n * a.P + kScanTile - 1) / kScanTile + 1;
                for (uint64_t i = tid; i < tiles; i += stride) a.desc[i] = 0ull;
            }
        }
        if (!grid_barrier(w)) return;
        if (dense && early) {
            MsBuArgs ma{a.gather_adj, a.cidx, a.cvert, a.nitems, (uint32_t)a.V, front, a.visit, next, next_bm,
                        a.alive_all, a.ms_seg, &w->nseg[L], nullptr};
            ms_head_work(ma);
            if (!grid_barrier(w)) return;
            ms_tail_work(ma);
        } else if (dense) {
            MsBfsPullOp op{front, front_bm, (uint64_t)n * 16 < a.V ? 1 : 0, a.visit, next, next_bm, a.alive_all, nullptr};
            pull_direct_chunks(op, a.gather_adj, a.cidx, a.cvert, a.pull_chunk_item, a.E, a.nitems, (uint32_t)a.V,
                               s_raw, &w->chunk[L]);
        } else {
            const uint64_t items = (uint64_t)n * a.P;
            scan_tiles(LoadItemLen{q, a.P, a.V + 1, a.csr_off}, EpiItemRank{a.ipref, a.push_chunk_item}, items, a.desc,
                       &w->ticket[L], &w->err, &w->total[L], kLookbackSpinCap);
            if (!grid_barrier(w)) return;
            PushArgs pa;
            pa.q = q;
            pa.nitems = items;
            pa.total_dev = &w->total[L];
            pa.P = a.P;
            pa.stride = a.V + 1;
            pa.off = a.csr_off;
            pa.adj = a.csr_adj;
            pa.w = nullptr;
            pa.ipref = a.ipref;
            pa.chunk_item = a.push_chunk_item;
            pa.q_out = nullptr;
            pa.n_out = nullptr;
            pa.act_edges = nullptr;
            pa.deg = nullptr;
            push_chunks(MsBfsPushOp{front, a.visit, next, next_bm}, pa);
        }
        if (!grid_barrier(w)) return;
        bm_compact_words(next_bm, a.nwords, q_next, &w->cnt[L], &w->act[L], a.deg);
        if (!grid_barrier(w)) return;
        n = __ldcg(&w->cnt[L]);
        act = __ldcg(&w->act[L]);
        if (dense) ++dense_count;
        if (a.lev) queue_levels_work(q_next, n, next, a.visit, a.lev, a.V, L + 1, nullptr, nullptr, nullptr);
        if (tid == 0) {
            w->levels = L + 1;
            w->pushes += dense ? 0u : 1u;
        }
    }
}

// one dense level as a full sweep (k_ms_sweep)
static int ms_sweep(eg_graph* g, const uint32_t* adj, const unsigned long long* front, const unsigned long long* front_bm,
                    int screen, unsigned long long* visit, unsigned long long* next, unsigned long long* next_bm,
                    const unsigned long long* alive, const int* stop, bool renumbered) {
    EngineState& s = g->eng;
    BatchState& b = bstate(g);
    if (!g->E) return EG_OK;
    if (g->partitions > 1) {  // a vertex has a list per partition, and sentinel entries lie between them
        MsBfsPullOp op{front, front_bm, screen, visit, next, next_bm, alive, stop};
        return launch_pull_direct(g, op, "msbfs_pull", adj, stop ? (unsigned)g->num_sms * 128u : 0u);
    }
    MsSweepArgs a;
    a.adj = adj;
    a.heads = s.pr_heads.as<uint32_t>();
    a.item_of = s.pr_item_of.as<uint32_t>();
    a.cvert = g->cvert.as<uint32_t>();
    a.E = g->E;
    a.shift = list_run_shift(g->E);
    a.nruns = (g->E + ((uint64_t)kPrBlock << a.shift) - 1) / ((uint64_t)kPrBlock << a.shift);
    a.nitems = (uint32_t)(g->ncompressed - 1);
    a.alive = g->batch_voff.empty() ? alive : nullptr;
    a.front = front;
    a.front_bm = front_bm;
    a.screen = screen;
    a.visit = visit;
    a.next = next;
    a.next_bm = next_bm;
    a.stop = stop;
    a.hot = renumbered ? std::min(kMsHot, relabel_lines((uint32_t)g->V)) : 0;
    a.ticket = b.ticket.as<uint32_t>();
    Timed t(&g->prof, g->stream, "msbfs_pull");
    EG_CUDA(cudaMemsetAsync(a.ticket, 0, 4, g->stream));
    k_ms_sweep<<<(unsigned)std::min<uint64_t>((a.nruns + kMsThreads / 32 - 1) / (kMsThreads / 32), (uint64_t)g->num_sms),
                 kMsThreads, kMsSmem, g->stream>>>(a);
    EG_CHECK_LAUNCH("k_ms_sweep");
    return EG_OK;
}

// MS-BFS over root entries already in b.entries (count in b.n_entries device word)
// lev: level planes (2 x [V][4] words) or null
static int msbfs_core(eg_graph* g, uint32_t n_entries, int nbits, unsigned long long* lev, uint64_t* reach_out,
                      int* sweeps_out, int* pushes_out) {
    BatchState& b = bstate(g);
    EngineState& s = g->eng;
    const uint64_t V = g->V;
    const uint64_t nwords = V / 64 + 1;
    const size_t bm_bytes = 8 * nwords;
    unsigned long long* visit = b.a64.as<unsigned long long>();
    unsigned long long* word[2] = {b.b64.as<unsigned long long>(), b.c64.as<unsigned long long>()};
    unsigned long long* bm[2] = {b.bm0.as<unsigned long long>(), b.bm1.as<unsigned long long>()};
    uint32_t* queue[2] = {s.q0.as<uint32_t>(), s.q1.as<uint32_t>()};
    unsigned long long* alive = b.alive.as<unsigned long long>();  // [0..1] per level parity, [2] all roots
    uint32_t* cnt = b.level_cnt.as<uint32_t>();  // [kGraphLevels + 1]
    unsigned long long* d_reach = s.counters.as<unsigned long long>() + 4;
    uint32_t* d_nq = reinterpret_cast<uint32_t*>(s.counters.as<unsigned long long>() + 2);
    unsigned long long* d_act = s.counters.as<unsigned long long>() + 3;
    const unsigned long long full = nbits == 64 ? ~0ull : ((1ull << nbits) - 1ull);
    const uint32_t* deg = g->outdeg.as<uint32_t>();
    const unsigned init_grid = std::max(1u, std::min<unsigned>((n_entries + 255) / 256, 4096u));
    const unsigned grid = (unsigned)g->num_sms * 8u;
    const bool one_graph = g->batch_voff.empty();
    constexpr uint64_t kUnknownQueue = ~0ull;
    // pull gathers through the CSC sources renumbered by out-degree class (hot frontier words share
    // cache lines), with a renumbered copy of each frontier; on one graph with the host-driven loop
    const bool renum = one_graph && !(g->use_cuda_graph & 1) && g->batch_launch != 1 && g->E > 0 && want_relabel(g);
    if (g->E && g->partitions == 1) {
        EG_TRY(setup_list_heads(g, renum));
        EG_TRY(b.ticket.reserve(16));
        EG_CUDA(cudaFuncSetAttribute(k_ms_sweep, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMsSmem));
    }
    if (renum) {
        EG_TRY(setup_relabel(g));
        EG_TRY(b.wr0.reserve(8 * V + 8));
        EG_TRY(b.wr1.reserve(8 * V + 8));
    }
    unsigned long long* word_r[2] = {b.wr0.as<unsigned long long>(), b.wr1.as<unsigned long long>()};
    const uint32_t* new_id = s.pr_new_id.as<uint32_t>();
    const uint32_t* gather_adj = renum ? s.pr_adj.as<uint32_t>() : g->csc_adj.as<uint32_t>();

    auto enqueue_init = [&]() -> int {
        EG_CUDA(cudaMemsetAsync(visit, 0, 8 * V, g->stream));
        EG_CUDA(cudaMemsetAsync(word[0], 0, 8 * V, g->stream));
        EG_CUDA(cudaMemsetAsync(bm[0], 0, bm_bytes, g->stream));
        EG_CUDA(cudaMemsetAsync(d_nq, 0, 16, g->stream));
        EG_CUDA(cudaMemsetAsync(cnt, 0, sizeof(uint32_t) * (kGraphLevels + 2), g->stream));
        EG_CUDA(cudaMemcpyAsync(alive + 2, &full, 8, cudaMemcpyHostToDevice, g->stream));
        EG_CUDA(cudaMemcpyAsync(alive, &full, 8, cudaMemcpyHostToDevice, g->stream));
        k_msbfs_init_entries<<<init_grid, 256, 0, g->stream>>>(b.entries.as<uint2>(), b.n_entries.as<uint32_t>(), visit,
                                                               word[0], bm[0], lev, queue[0], d_nq, d_act, deg);
        EG_CHECK_LAUNCH("k_msbfs_init_entries");
        if (renum) {
            EG_CUDA(cudaMemsetAsync(word_r[0], 0, 8 * V, g->stream));
            k_front_renumber<<<init_grid, 256, 0, g->stream>>>(queue[0], d_nq, word[0], new_id, word_r[0]);
            EG_CHECK_LAUNCH("k_front_renumber");
        }
        return EG_OK;
    };
    // one level L: frontier word[L&1] / bm[L&1] / queue[L&1] -> the same of parity (L+1)&1.  The
    // queue length lands in *count; captured loops (stop_flag set) pull every level and keep the
    // alive mask at "all roots".
    // The first dense level follows the frontier's explosion: most destinations miss most roots and
    // read all their in-edges, which the full sweep (k_ms_sweep) does best.  Later
    // dense levels find most destinations nearly covered and use the early-exit pair -- on one
    // graph.  In a batch of graphs the running-root mask is shared by all graphs, so a vertex
    // waits for bits its own graph can never deliver, and every level keeps the full sweep.
    // clear_n: how many vertices queue[x] lists from two levels back (the non-zero words of
    // word[x]); kUnknownQueue when not known on the host, and the arrays are cleared whole
    auto enqueue_level = [&](uint32_t L, uint64_t n_host, bool dense, bool screen, uint32_t* count, const int* stop_flag,
                             uint32_t* nout_host, unsigned long long* act_host, bool early_exit, uint64_t clear_n) -> int {
        const int c = L & 1, x = c ^ 1;
        if (clear_n <= V / 32) {
            if (clear_n) {
                Timed t(&g->prof, g->stream, "msbfs_vertex");
                k_clear_front<<<grid_for(clear_n, 256, grid), 256, 0, g->stream>>>(
                    queue[x], (uint32_t)clear_n, word[x], renum ? new_id : nullptr, renum ? word_r[x] : nullptr);
                EG_CHECK_LAUNCH("k_clear_front");
            }
        } else {
            EG_CUDA(cudaMemsetAsync(word[x], 0, 8 * V, g->stream));
            if (renum) EG_CUDA(cudaMemsetAsync(word_r[x], 0, 8 * V, g->stream));
        }
        EG_CUDA(cudaMemsetAsync(bm[x], 0, bm_bytes, g->stream));
        // renumbered gathers skip the frontier-bitmap screen (dense levels rarely screen)
        const unsigned long long* gather_word = renum ? word_r[c] : word[c];
        if (renum) screen = false;
        unsigned long long* alive_next = stop_flag ? nullptr : alive + x;
        if (alive_next) EG_CUDA(cudaMemsetAsync(alive_next, 0, 8, g->stream));
        if (dense) {
            EG_CUDA(cudaMemsetAsync(count, 0, 4, g->stream));
            if (!stop_flag) EG_CUDA(cudaMemsetAsync(d_act, 0, 8, g->stream));
            if (early_exit) {
                uint32_t* d_nseg = reinterpret_cast<uint32_t*>(cnt + kGraphLevels + 2);
                EG_CUDA(cudaMemsetAsync(d_nseg, 0, 4, g->stream));
                MsBuArgs ma{gather_adj, g->cidx.as<uint64_t>(), g->cvert.as<uint32_t>(),
                            g->ncompressed - 1, (uint32_t)V, gather_word, visit, word[x], bm[x],
                            stop_flag ? alive + 2 : alive + c, b.ms_seg.as<unsigned long long>(), d_nseg, stop_flag};
                Timed t(&g->prof, g->stream, "msbfs_pull");
                k_ms_head<<<grid_for(ma.nitems, 256, grid), 256, 0, g->stream>>>(ma);
                EG_CHECK_LAUNCH("k_ms_head");
                k_ms_tail<<<grid, 256, 0, g->stream>>>(ma);
                EG_CHECK_LAUNCH("k_ms_tail");
            } else {
                EG_TRY(ms_sweep(g, gather_adj, gather_word, bm[c], screen ? 1 : 0, visit, word[x], bm[x],
                                stop_flag ? alive + 2 : alive + c, stop_flag, renum));
            }
            Timed t(&g->prof, g->stream, "msbfs_vertex");
            k_bm_compact<<<grid_for(nwords, 256, grid), 256, 0, g->stream>>>(bm[x], nwords, queue[x], count,
                                                                            stop_flag ? nullptr : d_act, deg);
            EG_CHECK_LAUNCH("k_bm_compact");
        } else {
            MsBfsPushOp op{word[c], visit, word[x], bm[x]};
            EG_TRY(push_level(g, op, queue[c], n_host, queue[x], nout_host, nullptr, act_host, deg, "msbfs_push"));
        }
        if (lev || alive_next || renum) {
            Timed t(&g->prof, g->stream, "msbfs_vertex");
            if (lev && L == kHighPlanes)
                EG_CUDA(cudaMemsetAsync(lev + 4 * V, 0, 32 * V, g->stream));
            k_queue_levels<<<grid, 256, 0, g->stream>>>(queue[x], count, word[x], visit, lev, V, L + 1, alive_next,
                                                        renum ? new_id : nullptr, word_r[x]);
            EG_CHECK_LAUNCH("k_queue_levels");
        }
        return EG_OK;
    };

    int sweeps = 0, pushes = 0;
    uint32_t lvl = 0;
    // the host-driven level loop from level lvl on: the frontier (queue[lvl & 1]) lists n vertices
    // with act out-edges; q0len / q1len are how many vertices queue[0] / queue[1] list
    auto host_levels = [&](uint64_t n, unsigned long long act, uint64_t q0len, uint64_t q1len,
                           int dense_levels) -> int {
        struct {
            uint32_t n;
            uint32_t pad;
            unsigned long long act;
        } h;
        uint64_t qlen[2] = {q0len, q1len};
        while (n > 0) {
            if (lvl >= 254) {
                set_error("eg_msbfs: more than 254 levels");
                return EG_ERR_UNSUPPORTED;
            }
            // the Gemini switch on the union frontier; EG_OPT_BFS_DIRECTION concerns single-root BFS
            const bool dense = !g->built_csr || act >= g->E / (uint64_t)batch_divisor(g);
            uint32_t nout = 0;
            // a bitmap test before each gather pays only while the frontier is a small part of V
            EG_TRY(enqueue_level(lvl, n, dense, n * 16 < V, d_nq, nullptr, &nout, &act, one_graph && dense_levels > 0,
                                 qlen[(lvl & 1) ^ 1]));
            if (dense) {
                ++dense_levels;
                EG_CUDA(cudaMemcpyAsync(&h, d_nq, 16, cudaMemcpyDeviceToHost, g->stream));
                EG_CUDA(cudaStreamSynchronize(g->stream));
                nout = h.n;
                act = h.act;
            } else {
                ++pushes;
            }
            qlen[(lvl & 1) ^ 1] = nout;
            ++sweeps;
            n = nout;
            ++lvl;
        }
        return EG_OK;
    };
    if (g->batch_launch == 1) {
        // the whole traversal in one persistent cooperative launch
        EG_TRY(enqueue_init());
        EG_TRY(b.persist.reserve(sizeof(PersistWords)));
        PersistWords* pw = b.persist.as<PersistWords>();
        EG_CUDA(cudaMemsetAsync(pw, 0, sizeof(PersistWords), g->stream));
        const int P = g->partitions;
        const uint64_t max_tiles = ((V + 1) * (uint64_t)P + kScanTile - 1) / kScanTile + 2;
        EG_TRY(g->scan.desc.reserve(max_tiles * sizeof(uint64_t)));
        const size_t smem = 6 * ((size_t)kPullChunk + P + 3);
        EG_CUDA(cudaFuncSetAttribute(k_msbfs_persistent, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        int per_sm = 0;
        EG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_msbfs_persistent, 256, smem));
        if (per_sm < 1) {
            set_error("eg_msbfs: the persistent traversal does not fit an SM");
            return EG_ERR_UNSUPPORTED;
        }
        MsPersistArgs pa;
        pa.V = V;
        pa.nwords = nwords;
        pa.P = P;
        pa.csr_off = g->csr_off.as<uint64_t>();
        pa.csr_adj = g->csr_adj.as<uint32_t>();
        pa.gather_adj = gather_adj;
        pa.cidx = g->cidx.as<uint64_t>();
        pa.cvert = g->cvert.as<uint32_t>();
        pa.nitems = g->ncompressed - 1;
        pa.pull_chunk_item = s.pull_chunk_item.as<uint32_t>();
        pa.E = g->E;
        pa.deg = deg;
        pa.visit = visit;
        pa.word0 = word[0];
        pa.word1 = word[1];
        pa.bm0 = bm[0];
        pa.bm1 = bm[1];
        pa.q0 = queue[0];
        pa.q1 = queue[1];
        pa.alive_all = alive + 2;
        pa.lev = lev;
        pa.ms_seg = b.ms_seg.as<unsigned long long>();
        pa.desc = g->scan.desc.as<uint64_t>();
        pa.ipref = s.qdeg.as<uint64_t>();
        pa.push_chunk_item = s.chunk_item.as<uint32_t>();
        pa.init_n = d_nq;
        pa.init_act = d_act;
        pa.dense_min = g->E / (uint64_t)batch_divisor(g);
        pa.early_after_first = one_graph ? 1 : 0;
        pa.built_csr = g->built_csr ? 1 : 0;
        pa.w = pw;
        void* kargs[] = {&pa};
        {
            Timed t(&g->prof, g->stream, "msbfs_persistent");
            EG_CUDA(cudaLaunchCooperativeKernel((const void*)k_msbfs_persistent, dim3((unsigned)g->num_sms * per_sm),
                                                dim3(256), kargs, smem, g->stream));
            EG_CHECK_LAUNCH("k_msbfs_persistent");
        }
        PersistWords hw;
        EG_CUDA(cudaMemcpyAsync(&hw, pw, sizeof(PersistWords), cudaMemcpyDeviceToHost, g->stream));
        EG_CUDA(cudaStreamSynchronize(g->stream));
        if (hw.err) {
            set_error("eg_msbfs: a bounded wait of the persistent traversal gave up");
            return EG_ERR_TIMEOUT;
        }
        if (hw.levels >= 254 && hw.cnt[253] > 0) {
            set_error("eg_msbfs: more than 254 levels");
            return EG_ERR_UNSUPPORTED;
        }
        sweeps = (int)hw.levels;
        pushes = (int)hw.pushes;
        lvl = hw.levels;
    } else if (g->use_cuda_graph & 1) {
        // init + kGraphLevels levels replayed as one CUDA graph, each level choosing push or pull
        // on the device (k_cap_decide); levels after an empty frontier do nothing
        const bool key_ok = b.graph_exec && b.graph_V == V && b.graph_lev == (lev != nullptr) &&
                            b.graph_entries >= n_entries && b.graph_nbits == nbits &&
                            b.graph_div == batch_divisor(g);
        if (!key_ok) {
            if (b.graph_exec) cudaGraphExecDestroy((cudaGraphExec_t)b.graph_exec);
            b.graph_exec = nullptr;
            EG_TRY(b.cap.reserve(sizeof(CapState)));
            const int P = g->partitions;
            const uint64_t max_items = (V + 1) * (uint64_t)P;
            const uint64_t max_tiles = (max_items + kScanTile - 1) / kScanTile;
            EG_TRY(g->scan.desc.reserve(max_tiles * sizeof(uint64_t)));
            EG_TRY(g->scan.counter.reserve(16));
            const bool prof = g->prof.enabled;
            g->prof.enabled = false;
            EG_CUDA(cudaStreamBeginCapture(g->stream, cudaStreamCaptureModeThreadLocal));
            CapState* cs = b.cap.as<CapState>();
            int st = enqueue_init();
            auto ok = [&](cudaError_t e) {
                if (st == EG_OK && e != cudaSuccess) st = EG_ERR_CUDA;
            };
            ok(cudaMemsetAsync(cs, 0, sizeof(CapState), g->stream));
            ok(cudaMemsetAsync(word[1], 0, 8 * V, g->stream));
            const unsigned long long dense_min = g->E / (uint64_t)batch_divisor(g);
            for (uint32_t L = 0; st == EG_OK && L < (uint32_t)kGraphLevels; ++L) {
                const int c = L & 1, x = c ^ 1;
                const uint32_t* n_cur = L == 0 ? d_nq : cnt + L - 1;
                const unsigned long long* act_cur = L == 0 ? d_act : cs->act + L - 1;
                k_cap_decide<<<1, 1, 0, g->stream>>>(cs, (int)L, n_cur, act_cur, dense_min, one_graph ? 1 : 0,
                                                     g->built_csr ? 1 : 0);
                ok(cudaGetLastError());
                if (lev && L == kHighPlanes) {
                    k_zero_planes<<<grid, 256, 0, g->stream>>>(lev + 4 * V, 4 * V, n_cur);
                    ok(cudaGetLastError());
                }
                if (L >= 1) {  // the frontier words written two levels back (level 1: the roots)
                    const uint32_t* n_old = L == 1 ? d_nq : cnt + L - 2;
                    k_clear_front_dev<<<grid, 256, 0, g->stream>>>(queue[x], n_old, word[x], V, cs);
                    ok(cudaGetLastError());
                }
                ok(cudaMemsetAsync(bm[x], 0, bm_bytes, g->stream));
                // pull: the full sweep or the early-exit pair, whichever the level armed
                {
                    if (st == EG_OK)
                        st = ms_sweep(g, gather_adj, word[c], bm[c], 1, visit, word[x], bm[x], alive + 2,
                                      &cs->lv[L].skip_direct, false);
                    uint32_t* d_nseg = reinterpret_cast<uint32_t*>(cnt + kGraphLevels + 2);
                    ok(cudaMemsetAsync(d_nseg, 0, 4, g->stream));
                    MsBuArgs ma{gather_adj, g->cidx.as<uint64_t>(), g->cvert.as<uint32_t>(), g->ncompressed - 1,
                                (uint32_t)V, word[c], visit, word[x], bm[x], alive + 2,
                                b.ms_seg.as<unsigned long long>(), d_nseg, &cs->lv[L].skip_early};
                    k_ms_head<<<grid_for(ma.nitems, 256, grid), 256, 0, g->stream>>>(ma);
                    ok(cudaGetLastError());
                    k_ms_tail<<<grid, 256, 0, g->stream>>>(ma);
                    ok(cudaGetLastError());
                }
                // push: scan of the queued lists' lengths and the rank-balanced expansion, sized on
                // the device (zero items on pull levels)
                if (g->built_csr) {
                    const uint32_t* n_push = &cs->lv[L].n_push;
                    uint64_t* ipref = s.qdeg.as<uint64_t>();
                    ok(cudaMemsetAsync(g->scan.desc.ptr, 0, max_tiles * sizeof(uint64_t), g->stream));
                    ok(cudaMemsetAsync(g->scan.counter.ptr, 0, 4, g->stream));
                    LoadItemLen ld{queue[c], P, V + 1, g->csr_off.as<uint64_t>()};
                    EpiItemRank ep{ipref, s.chunk_item.as<uint32_t>()};
                    k_scan<<<(unsigned)std::min<uint64_t>(max_tiles, grid), kScanThreads, 0, g->stream>>>(
                        ld, ep, max_items, g->scan.desc.as<uint64_t>(), g->scan.counter.as<uint32_t>(),
                        g->err.as<int>(), &cs->push_total, kLookbackSpinCap, n_push, (uint32_t)P);
                    ok(cudaGetLastError());
                    PushArgs a;
                    a.q = queue[c];
                    a.nitems = 0;
                    a.n_dev = n_push;
                    a.total_dev = &cs->push_total;
                    a.P = P;
                    a.stride = V + 1;
                    a.off = g->csr_off.as<uint64_t>();
                    a.adj = g->csr_adj.as<uint32_t>();
                    a.w = nullptr;
                    a.ipref = ipref;
                    a.chunk_item = s.chunk_item.as<uint32_t>();
                    a.q_out = nullptr;
                    a.n_out = nullptr;
                    a.act_edges = nullptr;
                    a.deg = nullptr;
                    MsBfsPushOp pop{word[c], visit, word[x], bm[x]};
                    k_push<MsBfsPushOp><<<kPersistentGrid, kPushThreads, 0, g->stream>>>(pop, a);
                    ok(cudaGetLastError());
                }
                // the next frontier from its bitmap (either path), its out-edges and level bytes
                k_bm_compact<<<grid_for(nwords, 256, grid), 256, 0, g->stream>>>(bm[x], nwords, queue[x], cnt + L,
                                                                                cs->act + L, deg);
                ok(cudaGetLastError());
                if (lev) {
                    k_queue_levels<<<grid, 256, 0, g->stream>>>(queue[x], cnt + L, word[x], visit, lev, V, L + 1, nullptr,
                                                                nullptr, nullptr);
                    ok(cudaGetLastError());
                }
            }
            cudaGraph_t graph = nullptr;
            cudaError_t e = cudaStreamEndCapture(g->stream, &graph);
            g->prof.enabled = prof;
            EG_TRY(st);
            if (e != cudaSuccess) return cuda_fail(e, "cudaStreamEndCapture", __FILE__, __LINE__);
            cudaGraphExec_t exec = nullptr;
            e = cudaGraphInstantiate(&exec, graph, 0);
            cudaGraphDestroy(graph);
            if (e != cudaSuccess) return cuda_fail(e, "cudaGraphInstantiate", __FILE__, __LINE__);
            b.graph_exec = exec;
            b.graph_V = V;
            b.graph_lev = lev != nullptr;
            b.graph_entries = n_entries;
            b.graph_nbits = nbits;
            b.graph_div = batch_divisor(g);
        }
        {
            Timed t(&g->prof, g->stream, "msbfs_graph");
            EG_CUDA(cudaGraphLaunch((cudaGraphExec_t)b.graph_exec, g->stream));
        }
        std::vector<uint32_t> h(kGraphLevels);
        CapState hs;
        EG_CUDA(cudaMemcpyAsync(h.data(), cnt, sizeof(uint32_t) * kGraphLevels, cudaMemcpyDeviceToHost, g->stream));
        EG_CUDA(cudaMemcpyAsync(&hs, b.cap.ptr, sizeof(CapState), cudaMemcpyDeviceToHost, g->stream));
        EG_CUDA(cudaStreamSynchronize(g->stream));
        bool done = false;
        for (int L = 0; L < kGraphLevels && !done; ++L) {
            ++sweeps;
            if (hs.lv[L].n_push) ++pushes;
            done = h[L] == 0;
        }
        if (!done) {
            // deeper than the captured levels: the host-driven loop takes over at level
            // kGraphLevels (queue[0] lists the last captured level's output, queue[1] the one's before); the captured
            // levels kept no running-root masks, so every root counts as running
            lvl = kGraphLevels;
            EG_CUDA(cudaMemcpyAsync(alive + (lvl & 1), &full, 8, cudaMemcpyHostToDevice, g->stream));
            EG_TRY(host_levels(h[kGraphLevels - 1], hs.act[kGraphLevels - 1], h[kGraphLevels - 1], h[kGraphLevels - 2],
                               hs.dense_count));
        }
    } else {
        EG_TRY(enqueue_init());
        struct {
            uint32_t n;
            uint32_t pad;
            unsigned long long act;
        } h;
        EG_CUDA(cudaMemcpyAsync(&h, d_nq, 16, cudaMemcpyDeviceToHost, g->stream));
        EG_CUDA(cudaStreamSynchronize(g->stream));
        // queue[1] still holds an earlier call's list: its length is unknown
        EG_TRY(host_levels(h.n, h.act, h.n, kUnknownQueue, 0));
    }
    if (reach_out) {
        EG_CUDA(cudaMemsetAsync(d_reach, 0, 8, g->stream));
        Timed t(&g->prof, g->stream, "msbfs_vertex");
        k_reach_edges<<<grid_for(V, 256, grid), 256, 0, g->stream>>>(visit, deg, V, d_reach);
        EG_CHECK_LAUNCH("k_reach_edges");
        EG_CUDA(cudaMemcpyAsync(reach_out, d_reach, 8, cudaMemcpyDeviceToHost, g->stream));
        EG_CUDA(cudaStreamSynchronize(g->stream));
    }
    *sweeps_out = sweeps;
    if (pushes_out) *pushes_out = pushes;
    return EG_OK;
}

static int msbfs_buffers(eg_graph* g, uint32_t n_entries, bool with_levels) {
    BatchState& b = bstate(g);
    const uint64_t V = g->V;
    EG_TRY(ensure_engine(g));
    EG_TRY(setup_pull(g));
    EG_TRY(b.a64.reserve(8 * V + 8));
    EG_TRY(b.b64.reserve(8 * V + 8));
    EG_TRY(b.c64.reserve(8 * V + 8));
    EG_TRY(b.level_cnt.reserve(sizeof(uint32_t) * (kGraphLevels + 4)));
    EG_TRY(b.bm0.reserve(8 * (V / 64 + 1)));
    EG_TRY(b.bm1.reserve(8 * (V / 64 + 1)));
    EG_TRY(b.alive.reserve(64));
    {  // early-exit dense levels: at most one segment per entry longer than kMsHead plus one per kMsSeg
        const uint64_t nitems = g->ncompressed - 1;
        const uint64_t heavy = std::min<uint64_t>(nitems, g->E / (kMsHead + 1));
        EG_TRY(b.ms_seg.reserve(sizeof(unsigned long long) * (heavy + g->E / kMsSeg + 2)));
    }
    EG_TRY(b.entries.reserve(sizeof(uint2) * (n_entries + 1)));
    EG_TRY(b.n_entries.reserve(16));
    if (with_levels) EG_TRY(b.lev.reserve(64 * V + 64));
    EG_CUDA(cudaMemcpyAsync(b.n_entries.ptr, &n_entries, 4, cudaMemcpyHostToDevice, g->stream));
    return EG_OK;
}

int run_msbfs(eg_graph* g, const uint32_t* roots, int n, uint8_t* levels, int where, uint64_t* edges) {
    if (!g->built_csc) { set_error("eg_msbfs: CSC not built"); return EG_ERR_STATE; }
    EG_TRY(check_roots(g, roots, n, where, "eg_msbfs"));
    BatchState& b = bstate(g);
    const uint64_t V = g->V;
    EG_TRY(msbfs_buffers(g, (uint32_t)n, levels != nullptr));
    EG_TRY(copy_small_in(g, b.seeds, roots, n, where));
    k_root_entries<<<1, 64, 0, g->stream>>>(b.seeds.as<uint32_t>(), n, 0, b.entries.as<uint2>());
    EG_CHECK_LAUNCH("k_root_entries");
    unsigned long long* lev = levels ? b.lev.as<unsigned long long>() : nullptr;
    uint64_t reach = 0;
    int sweeps = 0, pushes = 0;
    EG_TRY(msbfs_core(g, (uint32_t)n, n, lev, &reach, &sweeps, &pushes));
    if (levels) {
        uint8_t* out = levels;
        if (where != EG_DEVICE) {
            EG_TRY(b.tmp_out.reserve((size_t)n * V + 64));
            out = b.tmp_out.as<uint8_t>();
        }
        {
            Timed t(&g->prof, g->stream, "msbfs_levels_out");
            k_levels_out<<<(unsigned)((V + kOutTile - 1) / kOutTile), 256, 0, g->stream>>>(
                lev, b.a64.as<unsigned long long>(), (uint32_t)V, n, sweeps >= 16 ? 1 : 0, out);
            EG_CHECK_LAUNCH("k_levels_out");
        }
        if (where != EG_DEVICE)
            EG_CUDA(cudaMemcpyAsync(levels, out, (size_t)n * V, cudaMemcpyDeviceToHost, g->stream));
    }
    EG_CUDA(cudaStreamSynchronize(g->stream));
    if (edges) *edges = reach;
    g->last_edges_processed = reach;
    g->last_iterations = sweeps;
    g->last_pushes = pushes;
    g->last_pulls = sweeps - pushes;
    return EG_OK;
}

// ---------------------------------------------------------------------------------------------
static int ensure_tasks(eg_graph* g, bool csr) {
    BatchState& b = bstate(g);
    if (csr) {
        if (!b.csr_ready) {
            EG_TRY(make_tasks(g, b.csr_tasks, g->csr_off.as<uint64_t>(), g->V, nullptr));
            b.csr_ready = true;
        }
    } else if (!b.csc_ready) {
        EG_TRY(make_tasks(g, b.csc_tasks, g->cidx.as<uint64_t>(), g->ncompressed - 1, g->cvert.as<uint32_t>()));
        b.csc_ready = true;
    }
    return EG_OK;
}

static RowArgs row_args(const RowTasks& t, const uint32_t* adj, const float* w) {
    return RowArgs{t.rec.as<uint4>(), t.first.as<uint32_t>(), adj, w};
}

// weights in CSC order (and, for the adjoint, in CSR order), row-normalised by the source's out-weight sum
static int prepare_ppr_weights(eg_graph* g, const float* w_in_dev, bool want_csr) {
    BatchState& b = bstate(g);
    const uint64_t E = g->E, V = g->V;
    const RowTasks& t = b.csr_tasks;
    EG_TRY(b.wn_csc.reserve(4 * E + 64));
    if (want_csr) EG_TRY(b.wn_csr.reserve(4 * E + 64));
    EG_TRY(b.s_out.reserve(4 * V + 64));
    EG_TRY(b.heavy_sum.reserve(8ull * t.nheavy + 64));
    const unsigned grid = (t.nbatches + kTaskThreads / 32 - 1) / (kTaskThreads / 32);
    const float* eid = g->csr_w.as<float>();
    float* wn = want_csr ? b.wn_csr.as<float>() : nullptr;
    Timed tm(&g->prof, g->stream, "ppr_weights");
    if (t.nheavy) EG_CUDA(cudaMemsetAsync(b.heavy_sum.ptr, 0, 8ull * t.nheavy, g->stream));
    if (g->partitions > 1) EG_CUDA(cudaMemsetAsync(b.s_out.ptr, 0, 4 * V, g->stream));  // sources without a task
    k_out_weights<<<grid, kTaskThreads, 0, g->stream>>>(t.rec.as<uint4>(), t.first.as<uint32_t>(), t.nbatches, eid, w_in_dev, b.s_out.as<float>(), wn,
                                               b.heavy_sum.as<double>(), 0);
    EG_CHECK_LAUNCH("k_out_weights");
    if (t.nheavy) {
        k_heavy_out_sums<<<(t.nheavy + 255) / 256, 256, 0, g->stream>>>(
            t.heavy_vertex.as<uint32_t>(), t.nheavy, b.heavy_sum.as<double>(), b.s_out.as<float>());
        EG_CHECK_LAUNCH("k_heavy_out_sums");
        if (wn) {
            k_out_weights<<<grid, kTaskThreads, 0, g->stream>>>(t.rec.as<uint4>(), t.first.as<uint32_t>(), t.nbatches, eid, w_in_dev, b.s_out.as<float>(),
                                                       wn, nullptr, 1);
            EG_CHECK_LAUNCH("k_out_weights");
        }
    }
    // CSC: the neighbour is the source
    k_gather_norm_w<<<grid_for(E, 256, 152u * 16u), 256, 0, g->stream>>>(
        g->csc_adj.as<uint32_t>(), g->csc_w.as<float>(), w_in_dev, b.s_out.as<float>(), E, b.wn_csc.as<float>());
    EG_CHECK_LAUNCH("k_gather_norm_w");
    return EG_OK;
}

// one forward step: y = a*e + (1-a) A^T x.  Rows of y without in-edges are as the caller left them: zero,
// and `a` at a seed's own column (lone_seeds).
template <class Row>
static int ppr_step_as(eg_graph* g, const float* x, float* y, float alpha, int n) {
    BatchState& b = bstate(g);
    const RowTasks& t = b.csc_tasks;
    RowArgs a = row_args(t, g->csc_adj.as<uint32_t>(), b.wn_csc.as<float>());
    Timed tm(&g->prof, g->stream, "ppr_spmm");
    k_row_spmm<Row><<<t.nbatches, 32, 0, g->stream>>>(a, reinterpret_cast<const Row*>(x), reinterpret_cast<Row*>(y),
                                                  b.heavy.as<Row>(), b.seeds.as<uint32_t>(), n, alpha);
    EG_CHECK_LAUNCH("k_row_spmm");
    if (t.nheavy) {
        k_row_heavy_finish<Row><<<(unsigned)((t.nheavy * 32ull + 255) / 256), 256, 0, g->stream>>>(
            t.heavy_vertex.as<uint32_t>(), t.nheavy, b.heavy.as<Row>(), reinterpret_cast<Row*>(y),
            b.seeds.as<uint32_t>(), n, alpha);
        EG_CHECK_LAUNCH("k_row_heavy_finish");
    }
    return EG_OK;
}
// Columns of a row: 32 for up to 32 seeds, which halves what the sweeps gather, else 64.  A step of 20
// iterations on 1 M / 16 M: 25.3 -> 20.5 ms with 32 seeds, 20.9 -> 17.5 with one.
static int row_width(int n) { return n <= 32 ? 32 : 64; }
static int ppr_step(eg_graph* g, const float* x, float* y, float alpha, int n) {
    return row_width(n) == 32 ? ppr_step_as<float>(g, x, y, alpha, n) : ppr_step_as<float2>(g, x, y, alpha, n);
}
template <class Row>
static int adjoint_step(eg_graph* g, const float* lam, const float* xk, float* lam2, float alpha) {
    BatchState& b = bstate(g);
    const RowTasks& t = b.csr_tasks;
    RowArgs a = row_args(t, g->csr_adj.as<uint32_t>(), b.wn_csr.as<float>());
    {
        Timed tm(&g->prof, g->stream, "ppr_adjoint");
        k_row_adjoint<Row><<<t.nbatches, 32, 0, g->stream>>>(
            a, reinterpret_cast<const Row*>(lam), reinterpret_cast<const Row*>(xk), reinterpret_cast<Row*>(lam2),
            b.heavy.as<Row>(), b.gA.as<double>(), 1.0f - alpha);
        EG_CHECK_LAUNCH("k_row_adjoint");
    }
    if (t.nheavy) {
        k_row_heavy_finish<Row><<<(unsigned)((t.nheavy * 32ull + 255) / 256), 256, 0, g->stream>>>(
            t.heavy_vertex.as<uint32_t>(), t.nheavy, b.heavy.as<Row>(), reinterpret_cast<Row*>(lam2), nullptr, 0, alpha);
        EG_CHECK_LAUNCH("k_row_heavy_finish");
    }
    return EG_OK;
}

static int lone_seeds(eg_graph* g, float* rows, int nbuf, int n, float alpha) {
    if (nbuf < 1) return EG_OK;
    k_ppr_lone_seeds<<<std::min(nbuf, 64), 64, 0, g->stream>>>(bstate(g).seeds.as<uint32_t>(), n, g->indeg.as<uint32_t>(), rows,
                                                               g->V, nbuf, alpha, row_width(n));
    EG_CHECK_LAUNCH("k_ppr_lone_seeds");
    return EG_OK;
}

static int ppr_common(eg_graph* g, const float* w_in, const uint32_t* seeds, int n, float alpha, int K, int where,
                      bool adjoint, const float** w_dev) {
    if (!g->built_csc || !g->built_csr) { set_error("eg_ppr: graph not built"); return EG_ERR_STATE; }
    if (!g->weighted || !g->edge_ids) {
        set_error("eg_ppr: load the graph with eg_load_directed_with_ids (per-edge ids select the weights)");
        return EG_ERR_STATE;
    }
    if (!w_in || K < 0 || !(alpha > 0.f && alpha <= 1.f)) { set_error("eg_ppr: need weights, K >= 0, 0 < alpha <= 1"); return EG_ERR_INVALID; }
    EG_TRY(check_roots(g, seeds, n, where, "eg_ppr"));
    BatchState& b = bstate(g);
    const uint64_t V = g->V, E = g->E_input;
    EG_TRY(copy_small_in(g, b.seeds, seeds, n, where));
    const float* wd = w_in;
    if (where != EG_DEVICE) {
        EG_TRY(b.tmp_out.reserve(4 * E + 64));
        EG_CUDA(cudaMemcpyAsync(b.tmp_out.ptr, w_in, 4 * E, cudaMemcpyHostToDevice, g->stream));
        wd = b.tmp_out.as<float>();
    }
    *w_dev = wd;
    EG_TRY(ensure_tasks(g, false));
    EG_TRY(ensure_tasks(g, true));
    EG_TRY(b.heavy.reserve(256ull * (std::max(b.csc_tasks.nheavy, b.csr_tasks.nheavy) + 1)));
    EG_CUDA(cudaMemsetAsync(b.heavy.ptr, 0, b.heavy.bytes, g->stream));
    EG_TRY(b.rows0.reserve(256 * V + 256));
    EG_TRY(b.rows1.reserve(256 * V + 256));
    return prepare_ppr_weights(g, wd, adjoint);
}

// one seed: the scalar chunked pull (4-byte gathers of x[src] times the normalised weight)
struct PprPullOp {
    using Acc = float;
    static constexpr bool kFilter = false;
    __device__ bool stopped() const { return false; }
    __device__ bool item_active(uint32_t) const { return true; }
    const float* x;
    const float* wn;
    float* y;
    float* acc;
    float scale;
    __device__ Acc identity() const { return 0.f; }
    __device__ Acc gather(uint32_t u, uint64_t e) const { return ld_keep(x + u) * __ldg(wn + e); }
    __device__ Acc combine(Acc a, Acc b) const { return a + b; }
    __device__ void smem_add(Acc* slot, Acc v) const { atomicAdd(slot, v); }
    __device__ void finish(bool ok, uint32_t v, Acc a, bool whole) const {
        if (!ok) return;
        if (whole) y[v] = scale * a;
        else atomicAdd(acc + v, a);
    }
};

__global__ void k_ppr_split(const uint32_t* __restrict__ split, const uint32_t* __restrict__ cvert, uint64_t nsplit,
                            float* y, float* acc, float scale) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nsplit; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t v = cvert[split[i]];
        y[v] = scale * acc[v];
        acc[v] = 0.f;
    }
}

__global__ void k_ppr_seed1(uint32_t seed, float* y, float value, int add) {
    if (add) y[seed] += value;
    else y[seed] = value;
}

static int run_ppr_single(eg_graph* g, uint32_t seed, float alpha, int K, float* out, int where) {
    BatchState& b = bstate(g);
    EngineState& s = g->eng;
    const uint64_t V = g->V;
    EG_TRY(ensure_engine(g));
    EG_TRY(setup_pull(g));
    float* x = s.vals0.as<float>();
    float* y = s.vals1.as<float>();
    EG_CUDA(cudaMemsetAsync(x, 0, 4 * V, g->stream));
    EG_CUDA(cudaMemsetAsync(s.acc.ptr, 0, 4 * V, g->stream));
    k_ppr_seed1<<<1, 1, 0, g->stream>>>(seed, x, 1.0f, 0);
    EG_CHECK_LAUNCH("k_ppr_seed1");
    for (int k = 0; k < K; ++k) {
        EG_CUDA(cudaMemsetAsync(y, 0, 4 * V, g->stream));
        // single = true: whole items write y directly, split items go through acc
        PprPullOp op{x, b.wn_csc.as<float>(), y, s.acc.as<float>(), 1.0f - alpha};
        EG_TRY(launch_pull(g, op, "ppr1_pull"));
        if (s.pull_nsplit) {
            k_ppr_split<<<grid_for(s.pull_nsplit, 256), 256, 0, g->stream>>>(s.pull_split.as<uint32_t>(), g->cvert.as<uint32_t>(),
                                                                             s.pull_nsplit, y, s.acc.as<float>(), 1.0f - alpha);
            EG_CHECK_LAUNCH("k_ppr_split");
        }
        k_ppr_seed1<<<1, 1, 0, g->stream>>>(seed, y, alpha, 1);
        EG_CHECK_LAUNCH("k_ppr_seed1");
        std::swap(x, y);
    }
    if (out)
        EG_CUDA(cudaMemcpyAsync(out, x, 4 * V, where == EG_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost,
                                g->stream));
    EG_CUDA(cudaStreamSynchronize(g->stream));
    g->last_edges_processed = g->E * (uint64_t)K;
    g->last_iterations = K;
    return EG_OK;
}

int run_ppr(eg_graph* g, const float* w_in, const uint32_t* seeds, int n, float alpha, int K, float* out, int where) {
    const float* wd = nullptr;
    EG_TRY(ppr_common(g, w_in, seeds, n, alpha, K, where, false, &wd));
    BatchState& b = bstate(g);
    const uint64_t V = g->V;
    if (n == 1 && g->partitions == 1) {
        uint32_t seed = 0;
        EG_CUDA(cudaMemcpyAsync(&seed, b.seeds.ptr, 4, cudaMemcpyDeviceToHost, g->stream));
        EG_CUDA(cudaStreamSynchronize(g->stream));
        return run_ppr_single(g, seed, alpha, K, out, where);
    }
    const int W = row_width(n);
    float* x = b.rows0.as<float>();
    float* y = b.rows1.as<float>();
    EG_CUDA(cudaMemsetAsync(x, 0, 4ull * W * V, g->stream));
    EG_CUDA(cudaMemsetAsync(y, 0, 4ull * W * V, g->stream));
    k_ppr_init<<<1, 64, 0, g->stream>>>(b.seeds.as<uint32_t>(), n, x, W);
    EG_CHECK_LAUNCH("k_ppr_init");
    for (int k = 0; k < K; ++k) {
        if (k < 2) EG_TRY(lone_seeds(g, y, 1, n, alpha));  // x_0 itself has 1 there
        EG_TRY(ppr_step(g, x, y, alpha, n));
        std::swap(x, y);
    }
    if (out) {
        float* dst = out;
        if (where != EG_DEVICE) {
            EG_TRY(b.tmp_out.reserve(4ull * n * V + 64));
            dst = b.tmp_out.as<float>();
        }
        dim3 blk(32, 8);
        k_transpose_rows<float><<<(unsigned)((V + 31) / 32), blk, 0, g->stream>>>(x, (uint32_t)V, n, dst, W);
        EG_CHECK_LAUNCH("k_transpose_rows");
        if (where != EG_DEVICE) EG_CUDA(cudaMemcpyAsync(out, dst, 4ull * n * V, cudaMemcpyDeviceToHost, g->stream));
    }
    EG_CUDA(cudaStreamSynchronize(g->stream));
    g->last_edges_processed = g->E * (uint64_t)K;
    g->last_iterations = K;
    return EG_OK;
}

// Checkpoint stride of the adjoint: the smallest one whose iterates fit EG_OPT_PPR_KEEP_MIB
// (all of x_0 .. x_{K-1} at stride 1, which recomputes nothing; else K / C checkpoints and a segment
// of C), at most ceil(sqrt(K)).  1 M vertices, K = 50: stride 1 keeps 12.8 GB and runs 99 forward
// sweeps in a forward and an adjoint, stride 8 keeps 4 GB and runs 143.
static uint64_t ppr_rows_kept(int K, int C) { return C == 1 ? (uint64_t)K : (uint64_t)((K + C - 1) / C) + C; }
static int ppr_stride(int K, uint64_t row, uint64_t budget) {
    const int most = std::max(1, (int)ceil(sqrt((double)std::max(K, 1))));
    int C = 1;
    while (C < most && ppr_rows_kept(K, C) * row > budget) ++C;
    return C;
}

static int zero_rows(eg_graph* g, const uint32_t* deg, float* rows, int nbuf, int width) {
    if (nbuf < 1) return EG_OK;
    k_zero_rows<<<grid_for(width / 4 * (uint64_t)g->V, 256, (unsigned)g->num_sms * 16u), 256, 0, g->stream>>>(
        deg, g->V, reinterpret_cast<float4*>(rows), nbuf, width / 4);
    EG_CHECK_LAUNCH("k_zero_rows");
    return EG_OK;
}

// adjoint of K forward steps from x_0 = e_seed; dL/dx_K given as [n][V]; dL/dw in input edge order
int run_ppr_backward(eg_graph* g, const float* w_in, const uint32_t* seeds, int n, float alpha, int K,
                     const float* dl_dx, float* dl_dw, int where) {
    const float* wd = nullptr;
    EG_TRY(ppr_common(g, w_in, seeds, n, alpha, K, where, true, &wd));
    if (!dl_dx || !dl_dw) { set_error("eg_ppr_backward: need dL/dx and the dL/dw output"); return EG_ERR_INVALID; }
    BatchState& b = bstate(g);
    const uint64_t V = g->V, E = g->E, Ein = g->E_input;
    const int W = row_width(n);
    const size_t row = 4ull * W * V;
    uint64_t budget = 0;
    if (g->ppr_keep_mib >= 0) {
        budget = (uint64_t)g->ppr_keep_mib << 20;
    } else if (ppr_rows_kept(K, 1) * row <= (1ull << 30)) {
        budget = 1ull << 30;  // not worth a look at what is free
    } else {
        size_t free_bytes = 0, total_bytes = 0;
        EG_CUDA(cudaMemGetInfo(&free_bytes, &total_bytes));
        budget = std::min<uint64_t>(total_bytes / 8, (free_bytes + b.ck.bytes + b.seg.bytes) / 2);
    }
    int C = ppr_stride(K, row, budget);
    while (true) {
        const size_t ck = row * ((std::max(K, 1) + C - 1) / C) + 256, seg = C > 1 ? row * C + 256 : 0;
        if (b.ck.bytes + b.seg.bytes > budget) {  // an earlier call was allowed more
            if (b.ck.bytes > ck) b.ck.release();
            if (b.seg.bytes > seg) b.seg.release();
        }
        int st = b.ck.reserve(ck);
        if (st == EG_OK && C > 1) st = b.seg.reserve(seg);
        if (st == EG_OK) break;
        const int most = ppr_stride(K, row, 0);  // the GPU is fuller than that: the fewest rows
        if (C == most) return st;
        C = most;
    }
    EG_TRY(b.gA.reserve(8 * E + 64));
    // forward with checkpoints x_0, x_C, x_2C, ... up to the last one before x_K
    float* ck = b.ck.as<float>();
    float* seg = b.seg.as<float>();
    const uint32_t* indeg = g->indeg.as<uint32_t>();
    const uint32_t* outdeg = g->outdeg.as<uint32_t>();
    EG_CUDA(cudaMemsetAsync(ck, 0, row, g->stream));
    k_ppr_init<<<1, 64, 0, g->stream>>>(b.seeds.as<uint32_t>(), n, ck, W);
    EG_CHECK_LAUNCH("k_ppr_init");
    if (C == 1) {
        EG_TRY(zero_rows(g, indeg, ck + W * V, K - 1, W));
        EG_TRY(lone_seeds(g, ck + W * V, K - 1, n, alpha));
        for (int k = 0; k + 1 < K; ++k) EG_TRY(ppr_step(g, ck + W * V * k, ck + W * V * (k + 1), alpha, n));
    } else {
        EG_TRY(zero_rows(g, indeg, seg, C, W));
        EG_TRY(lone_seeds(g, seg + W * V, C - 1, n, alpha));
        float* x = b.rows0.as<float>();
        float* y = b.rows1.as<float>();
        EG_CUDA(cudaMemcpyAsync(x, ck, row, cudaMemcpyDeviceToDevice, g->stream));
        EG_CUDA(cudaMemsetAsync(y, 0, row, g->stream));
        for (int k = 0; k < (K - 1) / C * C; ++k) {
            if (k < 2) EG_TRY(lone_seeds(g, y, 1, n, alpha));
            EG_TRY(ppr_step(g, x, y, alpha, n));
            std::swap(x, y);
            if ((k + 1) % C == 0)
                EG_CUDA(cudaMemcpyAsync(reinterpret_cast<char*>(ck) + row * ((k + 1) / C), x, row, cudaMemcpyDeviceToDevice,
                                        g->stream));
        }
    }
    // lambda_K from dL/dx_K ([n][V] -> [V][64])
    float* lam = b.rows0.as<float>();
    float* lam2 = b.rows1.as<float>();
    {
        const float* src = dl_dx;
        if (where != EG_DEVICE) {
            EG_TRY(b.tmp_out.reserve(4ull * n * V + 64));
            EG_CUDA(cudaMemcpyAsync(b.tmp_out.ptr, dl_dx, 4ull * n * V, cudaMemcpyHostToDevice, g->stream));
            src = b.tmp_out.as<float>();
        }
        dim3 blk(32, 8);
        k_untranspose_rows<float><<<(unsigned)((V + 31) / 32), blk, 0, g->stream>>>(src, (uint32_t)V, n, lam, W);
        EG_CHECK_LAUNCH("k_untranspose_rows");
    }
    EG_CUDA(cudaMemsetAsync(b.gA.ptr, 0, 8 * E, g->stream));
    const RowTasks& tr = b.csr_tasks;
    // the sweeps write only rows with out-edges; the others are zero from lambda_{K-1} on
    EG_TRY(zero_rows(g, outdeg, lam2, 1, W));
    for (int cp = (K - 1) / C; cp >= 0 && K > 0; --cp) {
        const int k0 = cp * C, k1 = std::min(K, k0 + C);
        const float* xs = ck + W * V * cp;  // x_k0 .. x_{k1-1}
        if (C > 1) {  // recomputed into the segment buffer
            EG_CUDA(cudaMemcpyAsync(seg, xs, row, cudaMemcpyDeviceToDevice, g->stream));
            for (int k = k0 + 1; k < k1; ++k)
                EG_TRY(ppr_step(g, seg + (size_t)(k - 1 - k0) * W * V, seg + (size_t)(k - k0) * W * V, alpha, n));
            xs = seg;
        }
        for (int k = k1 - 1; k >= k0; --k) {
            // lam holds lambda_{k+1}; gA += (1-a) <x_k[u], lam[v]>; lam2 = (1-a) A lam
            const float* xk = xs + (size_t)(k - k0) * W * V;
            EG_TRY(W == 32 ? adjoint_step<float>(g, lam, xk, lam2, alpha) : adjoint_step<float2>(g, lam, xk, lam2, alpha));
            if (k == K - 1) EG_TRY(zero_rows(g, outdeg, lam, 1, W));  // dL/dx_K itself is no longer needed
            std::swap(lam, lam2);
        }
    }
    // dL/dw
    float* dw = dl_dw;
    if (where != EG_DEVICE) {
        EG_TRY(b.tmp_out.reserve(4 * Ein + 64));
        dw = b.tmp_out.as<float>();
    }
    // every input edge sits in one CSR position; with several partitions only the first one's are tasks
    if (g->partitions > 1) EG_CUDA(cudaMemsetAsync(dw, 0, 4 * Ein, g->stream));
    if (tr.nheavy) EG_CUDA(cudaMemsetAsync(b.heavy_sum.ptr, 0, 8ull * tr.nheavy, g->stream));
    {
        Timed tm(&g->prof, g->stream, "ppr_weight_grad");
        for (int heavy = 0; heavy <= (tr.nheavy ? 1 : 0); ++heavy) {
            k_weight_grad<<<(tr.nbatches + kTaskThreads / 32 - 1) / (kTaskThreads / 32), kTaskThreads, 0, g->stream>>>(
                tr.rec.as<uint4>(), tr.first.as<uint32_t>(), tr.nbatches, b.wn_csr.as<float>(), b.gA.as<double>(), b.s_out.as<float>(),
                g->csr_w.as<float>(), dw, b.heavy_sum.as<double>(), heavy);
            EG_CHECK_LAUNCH("k_weight_grad");
        }
    }
    if (where != EG_DEVICE) EG_CUDA(cudaMemcpyAsync(dl_dw, dw, 4 * Ein, cudaMemcpyDeviceToHost, g->stream));
    EG_CUDA(cudaStreamSynchronize(g->stream));
    return EG_OK;
}

// ---------------------------------------------------------------------------------------------
__global__ void k_sssp_init_entries(const uint2* ent, uint32_t n, float* dist, int width, uint32_t* changed) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        dist[(uint64_t)ent[i].x * width + ent[i].y] = 0.f;
        atomicOr(changed + (ent[i].x >> 5), 1u << (ent[i].x & 31));
    }
}

// [V][32] rows -> [V][64], the columns past 32 unreached
__global__ void __launch_bounds__(256) k_widen_rows(const float* __restrict__ in, uint64_t V, float* __restrict__ out) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < 64 * V; i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = i & 32 ? 1e9f : __ldcs(in + (i >> 6) * 32 + (i & 31));
}

// Bellman-Ford sweeps from the root entries in b.entries; leaves dist [V][row_width(n)] in b.rows0.
// n: sources per row (32 columns for up to 32, which halves what the sweeps gather, else 64)
static int sssp_core(eg_graph* g, int n, uint32_t n_entries, int* sweeps_out) {
    const int W = row_width(n);
    EG_TRY(ensure_tasks(g, false));
    BatchState& b = bstate(g);
    const uint64_t V = g->V;
    EG_TRY(b.rows0.reserve(4ull * W * V + 256));
    const size_t ch_bytes = 4 * (V / 32 + 1);  // one bit per vertex: changed in the last sweep
    EG_TRY(b.ch0.reserve(ch_bytes));
    EG_TRY(b.ch1.reserve(ch_bytes));
    EG_TRY(b.flag.reserve(16));
    float* dist = b.rows0.as<float>();
    {
        Timed t(&g->prof, g->stream, "sssp_batch_init");
        k_fill_f32_rows<<<grid_for(W * V, 256, 152u * 16u), 256, 0, g->stream>>>(dist, W * V, 1e9f);
        EG_CHECK_LAUNCH("k_fill_f32_rows");
        EG_CUDA(cudaMemsetAsync(b.ch0.ptr, 0, ch_bytes, g->stream));
        k_sssp_init_entries<<<std::max(1u, std::min<unsigned>((n_entries + 255) / 256, 4096u)), 256, 0, g->stream>>>(
            b.entries.as<uint2>(), n_entries, dist, W, b.ch0.as<uint32_t>());
        EG_CHECK_LAUNCH("k_sssp_init_entries");
    }
    RowArgs a = row_args(b.csc_tasks, g->csc_adj.as<uint32_t>(), g->csc_w.as<float>());
    uint32_t* prev = b.ch0.as<uint32_t>();
    uint32_t* nxt = b.ch1.as<uint32_t>();
    int sweeps = 0;
    while (true) {
        EG_CUDA(cudaMemsetAsync(nxt, 0, ch_bytes, g->stream));
        EG_CUDA(cudaMemsetAsync(b.flag.ptr, 0, 4, g->stream));
        {
            Timed t(&g->prof, g->stream, "sssp_batch_sweep");
            if (W == 32)
                k_row_sssp<<<b.csc_tasks.nbatches, 32, 0, g->stream>>>(a, dist, prev, nxt, g->partitions > 1, b.flag.as<int>());
            else
                k_row_sssp<<<b.csc_tasks.nbatches, 32, 0, g->stream>>>(a, reinterpret_cast<float2*>(dist), prev, nxt,
                                                                      g->partitions > 1, b.flag.as<int>());
            EG_CHECK_LAUNCH("k_row_sssp");
        }
        ++sweeps;
        int any = 0;
        EG_CUDA(cudaMemcpyAsync(&any, b.flag.ptr, 4, cudaMemcpyDeviceToHost, g->stream));
        EG_CUDA(cudaStreamSynchronize(g->stream));
        if (!any) break;
        std::swap(prev, nxt);
    }
    *sweeps_out = sweeps;
    return EG_OK;
}

static int sssp_ready(eg_graph* g, const char* fn) {
    if (!g->built_csc) { set_error("%s: CSC not built", fn); return EG_ERR_STATE; }
    if (!g->weighted || g->edge_ids) { set_error("%s: graph needs float edge weights", fn); return EG_ERR_STATE; }
    return EG_OK;
}

int run_sssp_batch(eg_graph* g, const uint32_t* srcs, int n, float* out, int where) {
    EG_TRY(sssp_ready(g, "eg_sssp_batch"));
    EG_TRY(check_roots(g, srcs, n, where, "eg_sssp_batch"));
    BatchState& b = bstate(g);
    const uint64_t V = g->V;
    EG_TRY(copy_small_in(g, b.seeds, srcs, n, where));
    EG_TRY(b.entries.reserve(sizeof(uint2) * 64));
    k_root_entries<<<1, 64, 0, g->stream>>>(b.seeds.as<uint32_t>(), n, 0, b.entries.as<uint2>());
    EG_CHECK_LAUNCH("k_root_entries");
    int sweeps = 0;
    EG_TRY(sssp_core(g, n, (uint32_t)n, &sweeps));
    if (out) {
        float* dst = out;
        if (where != EG_DEVICE) {
            EG_TRY(b.tmp_out.reserve(4ull * n * V + 64));
            dst = b.tmp_out.as<float>();
        }
        dim3 blk(32, 8);
        k_transpose_rows<float><<<(unsigned)((V + 31) / 32), blk, 0, g->stream>>>(b.rows0.as<float>(), (uint32_t)V, n, dst,
                                                                                  row_width(n));
        EG_CHECK_LAUNCH("k_transpose_rows");
        if (where != EG_DEVICE) EG_CUDA(cudaMemcpyAsync(out, dst, 4ull * n * V, cudaMemcpyDeviceToHost, g->stream));
    }
    EG_CUDA(cudaStreamSynchronize(g->stream));
    g->last_iterations = sweeps;
    g->last_pulls = sweeps;
    g->last_pushes = 0;
    return EG_OK;
}

// ---------------------------------------------------------------------------------------------
// many small graphs: roots are local ids, nper per graph; outputs stay vertex-major [V_total][64]
static int graph_roots(eg_graph* g, const uint32_t* roots, int nper, int where, const char* fn, uint32_t* n_entries) {
    const uint64_t G = g->batch_voff.size() ? g->batch_voff.size() - 1 : 0;
    if (!G) { set_error("%s: no graph batch loaded (eg_load_graph_batch)", fn); return EG_ERR_STATE; }
    if (!roots || nper < 1 || nper > 64) { set_error("%s: need 1..64 roots per graph", fn); return EG_ERR_INVALID; }
    const uint64_t n = G * (uint64_t)nper;
    std::vector<uint32_t> h(n);
    EG_CUDA(cudaMemcpy(h.data(), roots, 4 * n, where == EG_DEVICE ? cudaMemcpyDeviceToHost : cudaMemcpyHostToHost));
    for (uint64_t i = 0; i < n; ++i) {
        const uint64_t gi = i / nper;
        if (h[i] >= g->batch_voff[gi + 1] - g->batch_voff[gi]) {
            set_error("%s: root %u of graph %llu out of range", fn, h[i], (unsigned long long)gi);
            return EG_ERR_INVALID;
        }
    }
    BatchState& b = bstate(g);
    EG_TRY(b.entries.reserve(sizeof(uint2) * (n + 1)));
    EG_TRY(b.tmp_out.reserve(4 * n + 64));
    EG_CUDA(cudaMemcpyAsync(b.tmp_out.ptr, h.data(), 4 * n, cudaMemcpyHostToDevice, g->stream));
    k_root_entries_graphs<<<(unsigned)((n + 255) / 256), 256, 0, g->stream>>>(
        b.tmp_out.as<uint32_t>(), g->d_batch_voff.as<uint64_t>(), (uint32_t)G, nper, b.entries.as<uint2>());
    EG_CHECK_LAUNCH("k_root_entries_graphs");
    EG_CUDA(cudaStreamSynchronize(g->stream));
    *n_entries = (uint32_t)n;
    return EG_OK;
}

int run_msbfs_graphs(eg_graph* g, const uint32_t* roots, int nper, uint8_t* levels, int where, uint64_t* edges) {
    if (!g->built_csc) { set_error("eg_msbfs_graphs: CSC not built"); return EG_ERR_STATE; }
    uint32_t n = 0;
    const uint64_t G = g->batch_voff.size() ? g->batch_voff.size() - 1 : 0;
    EG_TRY(msbfs_buffers(g, (uint32_t)(G * (uint64_t)std::max(nper, 1)), levels != nullptr));
    EG_TRY(graph_roots(g, roots, nper, where, "eg_msbfs_graphs", &n));
    BatchState& b = bstate(g);
    EG_CUDA(cudaMemcpyAsync(b.n_entries.ptr, &n, 4, cudaMemcpyHostToDevice, g->stream));
    uint64_t reach = 0;
    int sweeps = 0, pushes = 0;
    unsigned long long* lev = levels ? b.lev.as<unsigned long long>() : nullptr;
    EG_TRY(msbfs_core(g, n, nper, lev, &reach, &sweeps, &pushes));
    if (levels) {
        const uint64_t V = g->V;
        uint8_t* out = levels;
        const bool direct = where == EG_DEVICE && plain_device(g, levels, 16);
        if (!direct) {
            EG_TRY(b.tmp_out.reserve(64 * V + 64));
            out = b.tmp_out.as<uint8_t>();
        }
        {
            Timed t(&g->prof, g->stream, "msbfs_levels_out");
            k_level_rows<<<grid_for(4 * V, 256, (unsigned)g->num_sms * 16u), 256, 0, g->stream>>>(
                lev, b.a64.as<unsigned long long>(), V, sweeps >= 16 ? 1 : 0, reinterpret_cast<uint4*>(out));
            EG_CHECK_LAUNCH("k_level_rows");
        }
        if (!direct)
            EG_CUDA(cudaMemcpyAsync(levels, out, 64 * V, where == EG_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost,
                                    g->stream));
    }
    EG_CUDA(cudaStreamSynchronize(g->stream));
    if (edges) *edges = reach;
    g->last_edges_processed = reach;
    g->last_iterations = sweeps;
    g->last_pulls = sweeps - pushes;
    g->last_pushes = pushes;
    return EG_OK;
}

int run_sssp_graphs(eg_graph* g, const uint32_t* sources, int nper, float* dist, int where) {
    EG_TRY(sssp_ready(g, "eg_sssp_graphs"));
    uint32_t n = 0;
    EG_TRY(graph_roots(g, sources, nper, where, "eg_sssp_graphs", &n));
    int sweeps = 0;
    EG_TRY(sssp_core(g, nper, n, &sweeps));
    BatchState& b = bstate(g);
    const float* rows = b.rows0.as<float>();
    if (dist && row_width(nper) == 32) {
        float* wide = dist;
        if (where != EG_DEVICE || !plain_device(g, dist, 4)) {
            EG_TRY(b.tmp_out.reserve(256ull * g->V + 64));
            wide = b.tmp_out.as<float>();
        }
        k_widen_rows<<<grid_for(64ull * g->V, 256, 152u * 32u), 256, 0, g->stream>>>(rows, g->V, wide);
        EG_CHECK_LAUNCH("k_widen_rows");
        rows = wide;
    }
    if (dist && rows != dist)
        EG_CUDA(cudaMemcpyAsync(dist, rows, 256ull * g->V,
                                where == EG_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, g->stream));
    EG_CUDA(cudaStreamSynchronize(g->stream));
    g->last_iterations = sweeps;
    g->last_pulls = sweeps;
    g->last_pushes = 0;
    return EG_OK;
}

// graph i's edges occupy [eoff[i], eoff[i+1]); its vertex v becomes voff[i] + v
__global__ void k_relabel_batch(uint8_t* edges, int rec, uint64_t E, const uint64_t* __restrict__ eoff,
                                const uint64_t* __restrict__ voff, uint32_t G, int* bad) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < E; i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t lo = 0, hi = G;  // last graph with eoff <= i
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (__ldg(eoff + mid) <= i) lo = mid; else hi = mid;
        }
        uint32_t* r = reinterpret_cast<uint32_t*>(edges + i * (uint64_t)rec);
        const uint64_t base = voff[lo], nv = voff[lo + 1] - base;
        if (r[0] >= nv || r[1] >= nv) {
            atomicExch(bad, 1);
            continue;
        }
        r[0] = (uint32_t)(base + r[0]);
        r[1] = (uint32_t)(base + r[1]);
    }
}

int load_graph_batch(eg_graph* g, const void* edges, int rec, const uint64_t* eoff, const uint32_t* nverts, int G,
                     int where) {
    if ((rec != 8 && rec != 12) || G < 1 || !eoff || !nverts || eoff[0] != 0 || (where != EG_HOST && where != EG_DEVICE)) {
        set_error("eg_load_graph_batch: need 8/12-byte records, G >= 1, edge offsets starting at 0, vertex counts");
        return EG_ERR_INVALID;
    }
    std::vector<uint64_t> voff(G + 1, 0), eo(eoff, eoff + G + 1);
    for (int i = 0; i < G; ++i) {
        if (nverts[i] == 0 || eo[i + 1] < eo[i]) {
            set_error("eg_load_graph_batch: graph %d has no vertices or negative edge count", i);
            return EG_ERR_INVALID;
        }
        voff[i + 1] = voff[i] + nverts[i];
    }
    if (voff[G] >= (1ull << 32)) {
        set_error("eg_load_graph_batch: more than 2^32 vertices in total");
        return EG_ERR_INVALID;
    }
    const uint64_t E = eo[G];
    // the one-launch build reads the caller's device records itself
    EG_TRY(prepare_load(g, E, (uint32_t)voff[G], rec, 0));
    const bool one_launch = g->build_launch && persistent_build_fits(g);
    const bool direct = one_launch && edges && direct_records(g, edges, where);
    if (!direct) EG_TRY(load_edges_impl(g, edges, E, (uint32_t)voff[G], rec, 0, where, false));
    EG_TRY(g->d_batch_voff.reserve(8 * (G + 1)));
    EG_TRY(g->tmp64.reserve(8 * (G + 1)));
    EG_CUDA(cudaMemcpyAsync(g->d_batch_voff.ptr, voff.data(), 8 * (G + 1), cudaMemcpyHostToDevice, g->stream));
    EG_CUDA(cudaMemcpyAsync(g->tmp64.ptr, eo.data(), 8 * (G + 1), cudaMemcpyHostToDevice, g->stream));
    if (one_launch) {  // ids moved to the union inside the one launch
        EG_TRY(build_persistent(g, g->tmp64.as<uint64_t>(), g->d_batch_voff.as<uint64_t>(), (uint32_t)G,
                                direct ? edges : nullptr));
        g->batch_voff = voff;
        g->batch_eoff = eo;
        return EG_OK;
    }
    EG_CUDA(cudaMemsetAsync(g->err.as<int>() + 1, 0, sizeof(int), g->stream));
    if (E) {
        Timed t(&g->prof, g->stream, "relabel_batch");
        k_relabel_batch<<<grid_for(E, 256, 152u * 16u), 256, 0, g->stream>>>(
            g->edges.as<uint8_t>(), rec, E, g->tmp64.as<uint64_t>(), g->d_batch_voff.as<uint64_t>(), (uint32_t)G,
            g->err.as<int>() + 1);
        EG_CHECK_LAUNCH("k_relabel_batch");
    }
    int bad = 0;
    EG_CUDA(cudaMemcpyAsync(&bad, g->err.as<int>() + 1, sizeof(int), cudaMemcpyDeviceToHost, g->stream));
    EG_CUDA(cudaStreamSynchronize(g->stream));
    if (bad) {
        set_error("eg_load_graph_batch: a record holds a vertex id >= its graph's vertex count");
        return EG_ERR_INVALID;
    }
    g->batch_voff = voff;
    g->batch_eoff = eo;
    return build_structures(g, 1, 1);
}

}  // namespace eg
