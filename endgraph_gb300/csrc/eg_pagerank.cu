// eg_pagerank.cu — PageRank (toolkits/pagerank.cpp:26-98) on a one-partition graph: dense pull sweeps
// over the CSC by independent warps.
//
// A sweep is bound by the L1 lookups of its gathers (one per edge), so everything else is kept off
// that path.  Where a list starts is one bit per edge, read with the ids: no entry bounds to stage,
// no search for a thread's first entry.  A warp takes blocks of 512 edges, 8 consecutive ids per lane
// and half block, issues its 16 gathers, and sums lists with one segmented warp scan per half block;
// totals of lists that end in the block gather in shared memory and are finished one per lane, from
// degrees and places in entry order that were loaded behind the gathers.  The open list is carried
// from block to block, with what its roundings lose beside it; what a warp's run of blocks begins or ends in the middle
// of a list is added to the list's FP64 accumulator, and a second pass over the run boundaries finishes those
// lists.  (With both in FP32 a list of thousands of edges lost more than by 4,096-edge chunks: 17 M edges into
// 1,000 vertices 1.9e-7 off the FP64 value, relative L1, against 0.8e-7 by chunks; 0.4e-7 so.)  (Counting
// a list's pieces, so that the last warp finishes it, made the sweep wait for the counters of the
// hubs: 2.7 instead of 1.95 ms at 2^25 / 2^29, 2.8 with fences.)  Small graphs run every iteration in one
// persistent launch between grid barriers.
#include <math.h>

#include <algorithm>

#include "eg_pull.cuh"
#include "eg_queue.cuh"

namespace eg {

constexpr uint32_t kNoBoundary = 0xFFFFFFFFu;
constexpr int kPrGroup = 8;  // consecutive edges per lane: 4 or 16 were no faster (40.3 / 40.3 against 39.4 ms of sweeps)

constexpr uint32_t kPrSums = 32 * kPrGroup;  // lists that can end in a group of edges

struct PrArgs {
    const uint32_t* adj;
    const uint32_t* heads;    // bit e: edge e is the first of its list (one word of zeros past E)
    const uint32_t* item_of;  // per block: compressed entry that holds its first edge
    const uint32_t* dst;      // per entry: where its value goes in next
    const uint32_t* deg;      // per entry: its vertex's out-degree
    uint64_t E;
    uint64_t nruns;           // runs of 1 << shift blocks
    int shift;
    const float* curr;
    float* next;
    double* acc;              // per run boundary: the list that crosses it first there (split)
    const uint32_t* split;    // per run: boundary its first list's pieces meet at
    uint32_t hot;             // ranks that k_pr_sweep keeps in shared memory
    uint32_t* ticket;         // its next run
    float base, d;
    int divide;
};

__device__ __forceinline__ float pr_value(const PrArgs& a, float sum, uint32_t deg) {  // toolkits/pagerank.cpp:80-97
    const float x = a.base + a.d * sum;
    return a.divide && deg > 0 ? x / (float)deg : x;
}
__device__ __forceinline__ void pr_write(const PrArgs& a, uint32_t item, float sum) {
    const uint32_t to = __ldg(a.dst + item), deg = __ldg(a.deg + item);
    a.next[to] = pr_value(a, sum, deg);
}

// what a + b = s loses by rounding (Knuth's two-sum); nothing once the sum is infinite
__device__ __forceinline__ float sum_lost(float a, float b, float s) {
    const float v = s - a;
    return fabsf(s) < INFINITY ? (a - (s - v)) + (b - v) : 0.f;
}

// one run of blocks by one warp; s_sum: kPrSums floats of the warp's own
// kLong: runs of several blocks, whose carry is compensated (one block adds its two groups plainly)
template <bool kLong, class Gather>
__device__ __forceinline__ void pr_run(const PrArgs& a, uint64_t run, float* s_sum, Gather gather) {
    constexpr int G = kPrGroup, kGroups = (int)kPrBlock / (32 * G);
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t below = (1u << lane) - 1u;
    const uint64_t e_begin = (run << a.shift) * kPrBlock;
    const uint64_t e_end = min(a.E, ((run + 1) << a.shift) * kPrBlock);
    uint32_t item = __ldg(a.item_of + (run << a.shift));
    bool open_first = !(__ldg(a.heads + (e_begin >> 5)) & 1u);  // the first list began in an earlier run
    float carry = 0.f, carry_low = 0.f;  // sum of the open list so far, and what its roundings lost
    for (uint64_t e0 = e_begin; e0 < e_end; e0 += kPrBlock) {
        float val[kGroups][G];
        uint32_t head[kGroups];
#pragma unroll
        for (int g = 0; g < kGroups; ++g) {
            const uint64_t e = e0 + (uint64_t)g * (32 * G) + lane * G;
            uint32_t id[G];
            if (e + G <= a.E) {
#pragma unroll
                for (int q = 0; q < G / 4; ++q) {
                    const uint4 x = __ldcs(reinterpret_cast<const uint4*>(a.adj + e) + q);
                    id[4 * q] = x.x;
                    id[4 * q + 1] = x.y;
                    id[4 * q + 2] = x.z;
                    id[4 * q + 3] = x.w;
                }
#pragma unroll
                for (int j = 0; j < G; ++j) val[g][j] = gather(id[j]);
            } else {
#pragma unroll
                for (int j = 0; j < G; ++j) val[g][j] = e + j < a.E ? gather(a.adj[e + j]) : 0.f;
            }
            if (G == 16) head[g] = e < a.E ? __ldcs(reinterpret_cast<const uint16_t*>(a.heads) + e / 16) : 0u;
            else if (G == 8) head[g] = e < a.E ? __ldcs(reinterpret_cast<const uint8_t*>(a.heads) + e / 8) : 0u;
            else head[g] = e < a.E ? (__ldcs(reinterpret_cast<const uint8_t*>(a.heads) + e / 8) >> (e & 7)) & 0xFu : 0u;
            if (e == e_begin) head[g] &= ~1u;  // the run's first edge opens nothing new
        }
        // lists that end in earlier lanes (rank) and in the whole group
        uint32_t rank[kGroups], closed[kGroups], to[kGroups], deg[kGroups], at = item;
#pragma unroll
        for (int g = 0; g < kGroups; ++g) {
            rank[g] = closed[g] = 0;
#pragma unroll
            for (int j = 0; j < G; ++j) {
                const uint32_t b = __ballot_sync(0xffffffffu, (head[g] >> j) & 1u);
                rank[g] += __popc(b & below);
                closed[g] += __popc(b);
            }
            to[g] = lane < closed[g] ? __ldg(a.dst + at + lane) : 0u;
            deg[g] = lane < closed[g] ? __ldg(a.deg + at + lane) : 0u;
            at += closed[g];
        }
#pragma unroll
        for (int g = 0; g < kGroups; ++g) {
            const uint32_t f = head[g];
            float t = 0.f, first = 0.f;
            uint32_t k = rank[g];
            bool seen = false;
#pragma unroll
            for (int j = 0; j < G; ++j) {
                if ((f >> j) & 1u) {
                    if (seen) s_sum[k] = t;
                    else first = t;
                    ++k;
                    seen = true;
                    t = 0.f;
                }
                t += val[g][j];
            }
            // the open list along the lanes: t becomes its sum up to and including this lane
            const uint32_t m = __ballot_sync(0xffffffffu, seen);
            const int begin = 31 - __clz(m & (below | (1u << lane)));  // last lane that opened one, or -1
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float y = __shfl_up_sync(0xffffffffu, t, o);
                if ((int)lane - o >= max(begin, 0)) t += y;
            }
            float before = __shfl_up_sync(0xffffffffu, t, 1);
            if (lane == 0) before = 0.f;
            if (seen) {
                const float x = before + first, s = carry + x;
                s_sum[rank[g]] = m & below ? x : kLong ? s + (sum_lost(carry, x, s) + carry_low) : s;
            }
            const float rest = __shfl_sync(0xffffffffu, t, 31);
            if (m) {
                carry = rest;
                carry_low = 0.f;
            } else {
                const float s = carry + rest;
                if (kLong) carry_low += sum_lost(carry, rest, s);
                carry = s;
            }
            __syncwarp();
            for (uint32_t i = lane; i < closed[g]; i += 32) {
                const float sum = s_sum[i];
                if (i == 0 && open_first) atomicAdd(a.acc + __ldg(a.split + run), (double)sum);
                else if (i < 32) a.next[to[g]] = pr_value(a, sum, deg[g]);
                else pr_write(a, item + i, sum);
            }
            __syncwarp();
            if (closed[g]) open_first = false;
            item += closed[g];
        }
    }
    if (lane == 0) {
        const bool ends = e_end == a.E || ((__ldg(a.heads + (e_end >> 5)) >> (e_end & 31)) & 1u);
        if (open_first) atomicAdd(a.acc + __ldg(a.split + run), (double)carry + carry_low);
        else if (ends) pr_write(a, item, carry + carry_low);
        else atomicAdd(a.acc + __ldg(a.split + run + 1), (double)carry + carry_low);
    }
}

// the list that crosses the start of run r, if it began in the run before: its pieces are all in
__device__ __forceinline__ void pr_boundary(const PrArgs& a, uint64_t r) {
    if (__ldg(a.split + r) != (uint32_t)r) return;
    const double sum = __ldcg(a.acc + r);
    a.acc[r] = 0.0;  // for the next sweep
    pr_write(a, __ldg(a.item_of + (r << a.shift)), (float)sum);
}

// The sweep of a large graph: one CTA of 32 warps per SM, runs by ticket.  With renumbered sources the
// values of the first kPrHot ranks (rank r is id 32 r: see relabel_lines) are copied to shared memory
// by every SM, where a warp's gathers take a few cycles instead of a lookup each: on a power law
// a quarter of the gathers and more.  How many pays is set by the L1, whose lines hold the gathers in
// flight and which gets what shared memory leaves: 20 iterations at 2^25 / 2^29, 2^23 / 2^27 and 5 M /
// 40 M take 37.8 / 10.0 / 3.45 ms with none, 32.2 / 7.9 / - with 8,192, 29.8 / 7.3 / 2.65 with 16,384, 29.2 / 7.1
// / 2.64 with 24,576, 29.4 / 6.9 / 2.64 with 32,768, 36.2 / 7.0 / 2.69 with 33,760 and 66 / 10.9 / 3.8 with
// 40,960 (38.6 / 10.5 / 3.6 with CTAs of 8 warps, 48 warps per SM, a run per warp).
constexpr uint32_t kPrHot = 24576, kPrSweepThreads = 1024;
constexpr size_t kPrSweepSmem = sizeof(float) * (kPrHot + kPrSweepThreads / 32 * kPrSums);

__global__ void __launch_bounds__(kPrSweepThreads, 1) k_pr_sweep(PrArgs a) {
    extern __shared__ float s_dyn[];
    float* s_hot = s_dyn + kPrSweepThreads / 32 * kPrSums;
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t r = threadIdx.x; r < a.hot; r += kPrSweepThreads) s_hot[r] = __ldcg(a.curr + 32ull * r);
    const uint32_t hot_addr = (uint32_t)__cvta_generic_to_shared(s_hot), hot = a.hot;
    const float* curr = a.curr;
    unsigned long long keep;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 0.5;" : "=l"(keep));
    uint32_t next = 0;
    if (lane == 0) next = atomicAdd(a.ticket, 1u);
    __syncthreads();
    while (true) {
        const uint32_t run = __shfl_sync(0xffffffffu, next, 0);
        if (run >= a.nruns) break;
        if (lane == 0) next = atomicAdd(a.ticket, 1u);
        pr_run<true>(a, run, s_dyn + (threadIdx.x >> 5) * kPrSums, [&](uint32_t id) {
            const uint32_t rank = __funnelshift_r(id, id, 5);  // ids that are no multiple of 32 come out large
            float v;
            asm volatile(
                "{\n.reg .pred p;\nsetp.lt.u32 p, %1, %2;\n@p ld.shared.f32 %0, [%3];\n"
                "@!p ld.global.cg.L2::cache_hint.f32 %0, [%4], %5;\n}"
                : "=f"(v)
                : "r"(rank), "r"(hot), "r"(hot_addr + 4 * rank), "l"(curr + id), "l"(keep));
            return v;
        });
    }
}

__global__ void k_pr_boundaries(PrArgs a) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.ticket = 0;  // for the next sweep
    for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < a.nruns; r += (uint64_t)gridDim.x * blockDim.x)
        pr_boundary(a, r);
}

// Per entry: the bit of its first edge, its vertex's degree and (slot non-null) place; the entry of
// each block's first edge; per run the first run boundary that its first list crosses (none
// when the list starts with the run).
__global__ void k_pr_setup(const uint64_t* __restrict__ cidx, const uint32_t* __restrict__ cvert, uint64_t nitems,
                           const uint32_t* __restrict__ outdeg, const uint32_t* __restrict__ slot, int shift,
                           uint32_t* heads, uint32_t* __restrict__ item_of, uint32_t* __restrict__ deg,
                           uint32_t* __restrict__ place, uint32_t* __restrict__ split) {
    const uint64_t run = (uint64_t)kPrBlock << shift;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nitems; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t s = cidx[i], e = cidx[i + 1];
        if (e <= s) continue;
        atomicOr(heads + (s >> 5), 1u << (s & 31));
        for (uint64_t c = (s + kPrBlock - 1) / kPrBlock; c * kPrBlock < e; ++c) item_of[c] = (uint32_t)i;
        const uint32_t v = cvert[i];
        deg[i] = outdeg[v];
        if (slot) place[i] = slot[v];
        const uint64_t r0 = s / run + 1;
        if (s % run == 0) split[s / run] = kNoBoundary;
        for (uint64_t r = r0; r * run < e; ++r) split[r] = (uint32_t)r0;
    }
}

__device__ __forceinline__ void pr_start(float* curr, const uint32_t* __restrict__ outdeg, uint64_t V,
                                         const uint32_t* __restrict__ slot, double* acc, uint64_t nruns, uint64_t tid,
                                         uint64_t stride) {  // pagerank.cpp:36-45
    for (uint64_t v = tid; v < V; v += stride) {
        const uint32_t dg = outdeg[v];
        curr[slot ? slot[v] : v] = dg > 0 ? 1.0f / (float)dg : 1.0f;
    }
    for (uint64_t r = tid; r <= nruns; r += stride) acc[r] = 0.0;
}
// vertices without in-edges: next = 1-d (/ outdeg)
__device__ __forceinline__ void pr_no_in(float* next, const uint32_t* __restrict__ indeg, const uint32_t* __restrict__ outdeg,
                                         uint64_t V, float base, int divide, const uint32_t* __restrict__ slot, uint64_t tid,
                                         uint64_t stride) {
    for (uint64_t v = tid; v < V; v += stride) {
        if (indeg[v]) continue;
        const uint32_t dg = outdeg[v];
        next[slot ? slot[v] : v] = (divide && dg > 0) ? base / (float)dg : base;
    }
}
__global__ void k_pr_start(float* curr, const uint32_t* outdeg, uint64_t V, const uint32_t* slot, double* acc,
                           uint64_t nruns) {
    pr_start(curr, outdeg, V, slot, acc, nruns, blockIdx.x * (uint64_t)blockDim.x + threadIdx.x,
             (uint64_t)gridDim.x * blockDim.x);
}
__global__ void k_pr_no_in(float* next, const uint32_t* indeg, const uint32_t* outdeg, uint64_t V, float base, int divide,
                           const uint32_t* slot) {
    pr_no_in(next, indeg, outdeg, V, base, divide, slot, blockIdx.x * (uint64_t)blockDim.x + threadIdx.x,
             (uint64_t)gridDim.x * blockDim.x);
}

struct PrPersistArgs {
    PrArgs pr;              // curr, next, dst and divide are set per iteration
    uint64_t V;
    const uint32_t *indeg, *outdeg, *cvert;
    const uint32_t* order;  // slot of every vector but the last
    float* vec[2];
    float* out;             // the last vector
    int iterations;
    unsigned* words;        // barrier count, unused, error flag
    void* words_next;       // the next launch's, zeroed by this one
    uint32_t* finished;     // the pinned words: set when the last iteration is done
};

constexpr int kPrPersistThreads = 512, kPrPersistCtas = 2;

__global__ void __launch_bounds__(kPrPersistThreads, kPrPersistCtas) k_pr_persistent(PrPersistArgs a) {
    __shared__ float s_sum[kPrPersistThreads / 32][kPrSums];
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (uint64_t)gridDim.x * blockDim.x;
    unsigned arrived = 0;
    auto barrier = [&]() { return grid_sync_growing(a.words, reinterpret_cast<int*>(a.words + 2), a.finished + kPersistGaveUp, arrived); };
    pr_start(a.vec[0], a.outdeg, a.V, a.order, a.pr.acc, a.pr.nruns, tid, stride);
    for (int it = 0; it < a.iterations; ++it) {
        if (!barrier()) return;
        const bool last = it == a.iterations - 1;
        PrArgs p = a.pr;
        p.curr = a.vec[it & 1];
        p.next = last ? a.out : a.vec[(it & 1) ^ 1];
        if (last) p.dst = a.cvert;
        p.divide = !last;
        if (it < 2 || last) pr_no_in(p.next, a.indeg, a.outdeg, a.V, p.base, p.divide, last ? nullptr : a.order, tid, stride);
        for (uint64_t run = tid >> 5; run < p.nruns; run += stride >> 5) pr_run<false>(p, run, s_sum[threadIdx.x >> 5], [&](uint32_t id) { return ld_keep(p.curr + id); });
        if (!barrier()) return;
        for (uint64_t r = tid; r < p.nruns; r += stride) pr_boundary(p, r);
    }
    if (tid < 32) persist_clear(a.words_next);
    if (tid == 0) *a.finished = 1;
}

// Blocks per run: few boundaries (sweeps at 2^25 / 2^29 with 1 / 4 / 8 blocks: 41.2 / 38.6 / 38.0 ms), but runs
// enough for every resident warp several times (1 M / 16 M: 1.44 / 1.71 / 1.72).
int list_run_shift(uint64_t E) {
    int s = 0;
    while (s < 3 && (E >> (10 + s)) >= 24000) ++s;
    return s;
}

static int pr_setup(eg_graph* g, const uint32_t* order) {
    EngineState& s = g->eng;
    // with places it serves sweeps in vertex order too, so that calls of both kinds in turn make it once
    if (s.pr_heads_ready && (s.pr_heads_relabel || !order)) return EG_OK;
    const uint64_t E = g->E, nitems = g->ncompressed - 1;
    const size_t words = E / 32 + 2;
    const int shift = list_run_shift(E);
    EG_TRY(s.pr_heads.reserve(4 * words + 64));
    EG_TRY(s.pr_item_of.reserve(4 * (E / kPrBlock + 2)));
    EG_TRY(s.pr_split.reserve(4 * ((E / kPrBlock >> shift) + 3)));
    EG_TRY(s.pr_deg.reserve(4 * (nitems + 1)));
    if (order) EG_TRY(s.pr_place.reserve(4 * (nitems + 1)));
    Timed t(&g->prof, g->stream, "pr_setup");
    EG_CUDA(cudaMemsetAsync(s.pr_heads.ptr, 0, 4 * words, g->stream));
    k_pr_setup<<<grid_for(nitems, 256), 256, 0, g->stream>>>(
        g->cidx.as<uint64_t>(), g->cvert.as<uint32_t>(), nitems, g->outdeg.as<uint32_t>(), order, shift,
        s.pr_heads.as<uint32_t>(), s.pr_item_of.as<uint32_t>(), s.pr_deg.as<uint32_t>(), s.pr_place.as<uint32_t>(),
        s.pr_split.as<uint32_t>());
    EG_CHECK_LAUNCH("k_pr_setup");
    s.pr_heads_ready = true;
    s.pr_heads_relabel = order != nullptr;
    return EG_OK;
}

int setup_list_heads(eg_graph* g, bool relabel) {
    if (relabel) EG_TRY(setup_relabel(g));
    return pr_setup(g, relabel ? g->eng.pr_new_id.as<uint32_t>() : nullptr);
}

int run_pagerank_single(eg_graph* g, int iterations, float damping, float* out, int where) {
    EngineState& s = g->eng;
    const uint64_t V = g->V, E = g->E;
    for (DevBuf* b : {&s.vals0, &s.vals1}) EG_TRY(b->reserve(4 * (V + 1)));
    // with renumbered gathers every vector but the final one is kept in class order
    // Every iteration in one launch up to here: 20 iterations take 0.26 / 0.35 ms (one launch / sweeps) at
    // 65,536 / 2^20, 0.62 / 0.67 at 300,000 / 5 M, 1.45 / 1.33 and 0.1 for the renumbering at 1 M / 16 M, 2.70
    // / 1.91 at 2 M / 30 M.  Sweeps renumber by themselves when that comes back: 2^22 / 2^26 takes 0.30 ms to
    // renumber and 0.18 instead of 0.26 a sweep; a GPU too full for the second list goes without.  Passes over
    // many vertices want more threads than the one launch has: 3 iterations at 2^26 vertices take 2.23 / 1.33
    // with 1,000 edges, 2.86 / 1.96 with 2^24; 20 at 2^23 0.52 / 0.81 and 2.48 / 2.78.
    const bool small = E <= (1ull << 24) && V <= (1ull << 24) && list_run_shift(E) == 0;
    bool relabel = want_relabel(g);
    if (!relabel && !small && g->pr_relabel < 0 && iterations >= 4) relabel = setup_list_heads(g, true) == EG_OK;
    EG_TRY(setup_list_heads(g, relabel));
    const uint32_t* order = relabel ? s.pr_new_id.as<uint32_t>() : nullptr;
    float* vec[2] = {s.vals0.as<float>(), s.vals1.as<float>()};
    float* result = where == EG_DEVICE && plain_device(g, out, 4) ? out : vec[iterations & 1];
    PrArgs p;
    p.adj = relabel ? s.pr_adj.as<uint32_t>() : g->csc_adj.as<uint32_t>();
    p.heads = s.pr_heads.as<uint32_t>();
    p.item_of = s.pr_item_of.as<uint32_t>();
    p.dst = relabel ? s.pr_place.as<uint32_t>() : g->cvert.as<uint32_t>();
    p.deg = s.pr_deg.as<uint32_t>();
    p.E = E;
    p.shift = list_run_shift(E);
    p.nruns = (E + (kPrBlock << p.shift) - 1) / (kPrBlock << p.shift);
    EG_TRY(s.acc.reserve(8 * (p.nruns + 4)));
    p.acc = s.acc.as<double>();
    p.ticket = reinterpret_cast<uint32_t*>(p.acc + p.nruns + 3);
    // no more hot ranks than a quarter of an SM's edges: every SM copies them for every sweep
    p.hot = relabel ? (uint32_t)std::min<uint64_t>({kPrHot, relabel_lines((uint32_t)V), E / (4 * (uint64_t)g->num_sms)}) : 0;
    p.split = s.pr_split.as<uint32_t>();
    const uint32_t* outdeg = g->outdeg.as<uint32_t>();
    p.base = 1.0f - damping;
    p.d = damping;
    if (small) {
        void *block = nullptr, *next = nullptr;
        EG_TRY(persist_block(g, &block, &next));
        PrPersistArgs a{p, V, g->indeg.as<uint32_t>(), outdeg, g->cvert.as<uint32_t>(), order, {vec[0], vec[1]}, result, iterations,
                        static_cast<unsigned*>(block), next, reinterpret_cast<uint32_t*>(s.host_words)};
        // A warp per run, or what the vertices' values want where they are more: 20 iterations at 2^20 vertices
        // with 1,000 edges take 0.23 ms so and 2.7 by the one CTA that the runs want; the sum of both is
        // slower where the barriers dominate (0.41 instead of 0.32 ms at 2^20 / 2^20).
        const uint64_t warps = kPrPersistThreads / 32;
        const unsigned grid = (unsigned)std::min<uint64_t>((uint64_t)g->num_sms * kPrPersistCtas,
                                                           std::max((p.nruns + warps - 1) / warps, V / kVerticesPerCta));
        void* kargs[] = {&a};
        {
            Timed t(&g->prof, g->stream, "pr_persistent");
            EG_CUDA(cudaLaunchCooperativeKernel((const void*)k_pr_persistent, dim3(grid), dim3(kPrPersistThreads), kargs, 0,
                                                g->stream));
            EG_CHECK_LAUNCH("k_pr_persistent");
            persist_launched(g);
        }
    } else {
        const unsigned gv = grid_for(V, 256, 152u * 16u);
        EG_CUDA(cudaFuncSetAttribute(k_pr_sweep, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPrSweepSmem));
        EG_CUDA(cudaMemsetAsync(p.ticket, 0, 4, g->stream));
        {
            Timed t(&g->prof, g->stream, "pr_vertex");
            k_pr_start<<<gv, 256, 0, g->stream>>>(vec[0], outdeg, V, order, p.acc, p.nruns);
            EG_CHECK_LAUNCH("k_pr_start");
        }
        for (int it = 0; it < iterations; ++it) {
            const bool last = it == iterations - 1;
            p.curr = vec[it & 1];
            p.next = last ? result : vec[(it & 1) ^ 1];
            if (last) p.dst = g->cvert.as<uint32_t>();
            p.divide = !last;
            if (it < 2 || last) {
                Timed t(&g->prof, g->stream, "pr_vertex");
                k_pr_no_in<<<gv, 256, 0, g->stream>>>(p.next, g->indeg.as<uint32_t>(), outdeg, V, p.base, p.divide,
                                                       last ? nullptr : order);
                EG_CHECK_LAUNCH("k_pr_no_in");
            }
            {
                Timed t(&g->prof, g->stream, "pr_pull");
                k_pr_sweep<<<(unsigned)g->num_sms, kPrSweepThreads, kPrSweepSmem, g->stream>>>(p);
                EG_CHECK_LAUNCH("k_pr_sweep");
            }
            Timed t(&g->prof, g->stream, "pr_finish");
            k_pr_boundaries<<<grid_for(p.nruns, 256), 256, 0, g->stream>>>(p);
            EG_CHECK_LAUNCH("k_pr_boundaries");
        }
    }
    if (result != out) EG_TRY(copy_out(g, out, result, sizeof(float) * V, where));
    EG_CUDA(cudaStreamSynchronize(g->stream));
    if (small) EG_TRY(persist_finish(g, "eg_pagerank"));
    g->last_edges_processed = E * (uint64_t)iterations;
    g->last_iterations = iterations;
    g->last_pushes = 0;
    g->last_pulls = iterations;
    return EG_OK;
}

}  // namespace eg
