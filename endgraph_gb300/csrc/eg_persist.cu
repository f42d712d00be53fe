// eg_persist.cu — single-source traversals as one persistent cooperative launch: every level (or
// near/far step) runs inside the kernel between bounded grid barriers, so that a step costs a barrier
// instead of several launches and a host round trip.
//
// The frontier is a queue of list pieces {vertex, first edge, edges}, at most kPiece edges each, so
// that a hub's list is spread over the GPU without a scan over the frontier.  Warps take pieces by
// stride (piece i goes to warp i mod warps: the pieces of one hub lie next to each other in the
// queue), up to 32 at a time, and walk their edges together: a warp prefix sum of the lengths, kIlp
// edges per lane in flight.  Activated vertices are queued in shared memory and leave with one
// reservation of the global queue per CTA and step (with one per warp, all meeting in one L2 word, and
// with the lowered distance's old value awaited, an SSSP of 50,021 vertices and 800,017 edges took
// 0.60 ms instead of 0.37, one of 2^22 and 2^26 5.6 instead of 3.8).  Per edge the walk is bound by
// the latency of its gathers at 32 warps per SM (64 registers): 2 edges per lane in flight are 10-20 %
// slower, 6 spill.
#include <math.h>
#include <string.h>

#include <algorithm>

#include "eg_pull.cuh"
#include "eg_queue.cuh"

namespace eg {

constexpr int kIlp = 4;
constexpr uint32_t kStepsPerLaunch = 4096;  // then the host launches again: a kernel always ends

// what one step left behind, read by every CTA after the barrier that ends the step
struct alignas(16) StepSlot {
    uint32_t n;         // queue entries appended
    uint32_t min_bits;  // SSSP split: smallest parked distance
    uint32_t parked;    // SSSP split: vertices still parked
    uint32_t pad;
};

struct PersistState {
    unsigned bar_count, bar_pad;
    int err;
    uint32_t step;       // steps done so far
    StepSlot slot[4];    // step k reads slot k & 3, fills slot (k + 1) & 3 and clears slot (k + 2) & 3
    float thr, delta;    // SSSP near/far threshold and its step
    float weight_sum;    // sampled weights
    uint32_t pushes;
    unsigned long long edges;  // edges of the pieces walked
};

// what a launch tells the host, written to pinned memory by its first thread as it ends (persist_finish)
struct PersistResult {
    uint32_t valid, done, step, pushes, pulls, pad;
    unsigned long long reached, edges;
};
static_assert(sizeof(PersistResult) <= 4 * kPersistGaveUp, "the results lie in the handle's pinned words");

// one grid barrier; *s_slot gets the slot the finished step filled.  False: a wait gave up.
template <class State, class Slot>
__device__ __forceinline__ bool step_barrier(State* st, PersistResult* result, const Slot* slot, Slot* s_slot, unsigned& arrived) {
    if (!grid_sync_growing(&st->bar_count, &st->err, reinterpret_cast<uint32_t*>(result) + kPersistGaveUp, arrived)) return false;
    if (threadIdx.x < sizeof(Slot) / 16)
        reinterpret_cast<uint4*>(s_slot)[threadIdx.x] = __ldcg(reinterpret_cast<const uint4*>(slot) + threadIdx.x);
    __syncthreads();
    return true;
}

__device__ __forceinline__ uint32_t warp_incl(uint32_t x) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    return x;
}

// the first lane whose inclusive prefix exceeds rank r (lane 31 for ranks past the last)
__device__ __forceinline__ uint32_t warp_owner(uint32_t incl, uint32_t r) {
    uint32_t o = 0;
#pragma unroll
    for (int b = 16; b > 0; b >>= 1) {
        const uint32_t p = __shfl_sync(0xffffffffu, incl, o + b - 1);
        if (p <= r) o += b;
    }
    return o;
}

// The CTA's share of the next queue (eg_queue.cuh)
struct LocalQueue {
    uint4 e[kLocalQueue];
    uint32_t n;      // reserved
    uint32_t valid;  // reservations from here on did not fit
    uint32_t base;
};
__device__ __forceinline__ uint4 piece(uint32_t v, uint64_t beg, uint64_t end) {
    const uint32_t len = (uint32_t)(end - beg < kPiece ? end - beg : kPiece);
    return make_uint4(v, (uint32_t)beg, (uint32_t)(beg >> 32), len);
}

// every lane appends the pieces of its K vertices' lists [beg[j], end[j]) (empty: none)
template <int K>
__device__ __forceinline__ void append_pieces(LocalQueue& lq, WarpBlock& wb, const uint32_t (&v)[K],
                                              const uint64_t (&beg)[K], const uint64_t (&end)[K], uint4* q_out,
                                              uint32_t* n_out) {
    uint32_t cnt = 0;
#pragma unroll
    for (int j = 0; j < K; ++j) cnt += (uint32_t)((end[j] - beg[j] + kPiece - 1) / kPiece);
    if (!__any_sync(0xffffffffu, cnt != 0)) return;
    const uint32_t incl = warp_incl(cnt);
    const uint32_t tot = __shfl_sync(0xffffffffu, incl, 31);
    uint32_t at = kLocalQueue;
    if ((threadIdx.x & 31) == 31 && *(volatile uint32_t*)&lq.valid == 0xFFFFFFFFu) {
        at = atomicAdd(&lq.n, tot);
        if (at + tot > kLocalQueue) {
            atomicMin(&lq.valid, at);
            at = kLocalQueue;
        }
    }
    at = __shfl_sync(0xffffffffu, at, 31);
    uint32_t k = incl - cnt;  // this lane's first entry among the warp's
    if (at < kLocalQueue) {
#pragma unroll
        for (int j = 0; j < K; ++j)
            for (uint64_t b = beg[j]; b < end[j]; b += kPiece) lq.e[at + k++] = piece(v[j], b, end[j]);
        return;
    }
    const uint32_t room = wb.end - wb.pos, block = wb.wants(tot);
    uint32_t fresh = 0;
    if (block) {
        if ((threadIdx.x & 31) == 31) fresh = atomicAdd(n_out, block);
        fresh = __shfl_sync(0xffffffffu, fresh, 31);
    }
#pragma unroll
    for (int j = 0; j < K; ++j)
        for (uint64_t b = beg[j]; b < end[j]; b += kPiece, ++k)
            q_out[k < room ? wb.pos + k : fresh + (k - room)] = piece(v[j], b, end[j]);
    wb.took(tot, fresh, block);
}

// By the whole CTA, before the barrier that ends a phase.  What a warp has left of its block is filled with
// empty pieces, which a later phase of the step (behind that barrier) may overwrite.
__device__ __forceinline__ void flush_pieces(LocalQueue& lq, WarpBlock& wb, uint4* q_out, uint32_t* n_out,
                                             bool step_done = true) {
    for (uint32_t i = wb.pos + (threadIdx.x & 31); i < wb.end; i += 32) q_out[i] = make_uint4(0, 0, 0, 0);
    wb.phase_done(step_done);
    __syncthreads();
    const uint32_t n = min(lq.n, lq.valid);
    if (threadIdx.x == 0) lq.base = n ? atomicAdd(n_out, n) : 0u;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) q_out[lq.base + i] = lq.e[i];
    if (threadIdx.x == 0) {
        lq.n = 0;
        lq.valid = 0xFFFFFFFFu;
    }
}

// ---------------------------------------------------------------------------------------------
// SSSP (toolkits/sssp.cpp:52-64) with the near/far split of SsspOp: a lowered vertex below the
// threshold joins the next queue (once per step: its stamp holds the step that queued it), one
// above it is parked in the far bitmap.  When the queue runs empty a split step raises the
// threshold and moves the parked vertices below it.  Every relaxation is an exact float add and a
// minimum, so the fixpoint does not depend on the order.
struct SsspPersistArgs {
    uint64_t V, E, nwords;
    const uint64_t* off;
    const uint32_t* adj;
    const float* w;
    float* dist;
    uint32_t* stamp;
    unsigned long long* far_bm;
    uint4* q[2];
    uint32_t root;
    float delta;        // > 0: given; 0: plain sweeps; < 0: -delta x the sampled mean weight
    int resume;         // continue from the state an earlier launch left
    PersistState* st;
    void* st_next;      // the next launch's state, zeroed by this one
    PersistResult* result;
};

constexpr uint32_t kWeightSamples = 65536;

__global__ void __launch_bounds__(kPersistThreads, kPersistCtas) k_sssp_persistent(SsspPersistArgs a) {
    __shared__ StepSlot s_slot;
    extern __shared__ __align__(16) unsigned char s_raw[];
    LocalQueue& lq = *reinterpret_cast<LocalQueue*>(s_raw);
    WarpBlock wb;
    if (threadIdx.x == 0) {
        lq.n = 0;
        lq.valid = 0xFFFFFFFFu;
    }
    PersistState* st = a.st;
    unsigned arrived = 0;
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint32_t warp = (uint32_t)(tid >> 5), nwarps = (uint32_t)(stride >> 5);
    unsigned long long my_edges = 0;
    uint32_t step = 0, pushes = 0;
    float thr, delta;
    if (!a.resume) {
        for (uint64_t v = tid; v < a.V; v += stride) {
            a.dist[v] = v == a.root ? 0.f : 1e9f;
            a.stamp[v] = 0u;
        }
        for (uint64_t i = tid; i < a.nwords; i += stride) a.far_bm[i] = 0ull;
        if (a.delta < 0.f) {  // mean of a strided sample of the weights
            const uint64_t every = max(a.E / kWeightSamples, (uint64_t)1);
            float acc = 0.f;
            for (uint64_t i = tid; i < kWeightSamples && i * every < a.E; i += stride) acc += a.w[i * every];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (lane == 0 && acc != 0.f) atomicAdd(&st->weight_sum, acc);
        }
        if (tid < 32) {  // the root's pieces
            const uint64_t b = a.off[a.root], z = a.off[(uint64_t)a.root + 1];
            const uint32_t np = (uint32_t)((z - b + kPiece - 1) / kPiece);
            for (uint32_t p = lane; p < np; p += 32) a.q[0][p] = piece(a.root, b + (uint64_t)p * kPiece, z);
            if (lane == 0) st->slot[0].n = np;
        }
        if (!step_barrier(st, a.result, &st->slot[0], &s_slot, arrived)) return;
        delta = a.delta;
        if (delta < 0.f) {
            const uint64_t every = max(a.E / kWeightSamples, (uint64_t)1);
            const uint64_t taken = min((uint64_t)kWeightSamples, (a.E + every - 1) / every);
            const float mean_w = taken ? __ldcg(&st->weight_sum) / (float)taken : 0.f;
            delta = -delta * mean_w;
        }
        thr = delta > 0.f ? delta : INFINITY;
    } else {
        step = __ldcg(&st->step);
        thr = __ldcg(&st->thr);
        delta = __ldcg(&st->delta);
        if (threadIdx.x == 0) s_slot = st->slot[step & 3];
        __syncthreads();
    }
    const bool split = delta > 0.f;
    const uint32_t first = step;
    bool done = false;
    uint32_t last_kind = 0;  // 0: push, 1: split
    while (step - first < kStepsPerLaunch) {
        const uint32_t n = s_slot.n;
        StepSlot* out = &st->slot[(step + 1) & 3];
        uint4* q_out = a.q[(step + 1) & 1];
        const uint32_t mark = step + 1;
        if (n == 0) {
            if (!split || (last_kind == 1 && s_slot.parked == 0)) {
                done = true;
                break;
            }
            // after an empty split: jump to the nearest parked distance
            const float from = last_kind == 1 ? fmaxf(thr, __uint_as_float(s_slot.min_bits)) : thr;
            thr = from + delta > from ? from + delta : nextafterf(from, INFINITY);
        }
        __syncthreads();  // s_slot has been read
        if (tid == 0) {
            StepSlot* clear = &st->slot[(step + 2) & 3];
            clear->n = 0;
            clear->min_bits = 0x7F800000u;  // +inf
            clear->parked = 0;
        }
        if (n) {
            const uint4* q = a.q[step & 1];
            for (uint32_t base = 0; base < n; base += 32 * nwarps) {
                const uint64_t idx = (uint64_t)base + (uint64_t)lane * nwarps + warp;
                uint64_t beg = 0;
                uint32_t len = 0;
                float du = 0.f;
                if (idx < n) {
                    const uint4 e = __ldcg(q + idx);
                    du = __ldcg(a.dist + e.x);
                    beg = ((uint64_t)e.z << 32) | e.y;
                    len = e.w;
                }
                const uint32_t incl = warp_incl(len);
                const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
                if (lane == 0) my_edges += total;
                beg -= incl - len;  // rank r of the warp's edges sits at beg + r of its owner
                for (uint32_t r0 = 0; r0 < total; r0 += 32 * kIlp) {
                    uint32_t x[kIlp];
                    float nd[kIlp];
                    uint64_t lb[kIlp], le[kIlp];
#pragma unroll
                    for (int j = 0; j < kIlp; ++j) {
                        const uint32_t r = r0 + 32 * j + lane;
                        const uint32_t o = warp_owner(incl, r);
                        const uint64_t pos = __shfl_sync(0xffffffffu, beg, o) + r;
                        const float od = __shfl_sync(0xffffffffu, du, o);
                        x[j] = r < total ? __ldg(a.adj + pos) : 0u;
                        nd[j] = r < total ? od + __ldg(a.w + pos) : INFINITY;  // toolkits/sssp.cpp:55
                    }
                    float old[kIlp];
#pragma unroll
                    for (int j = 0; j < kIlp; ++j) old[j] = __ldcg(a.dist + x[j]);
#pragma unroll
                    for (int j = 0; j < kIlp; ++j) {
                        lb[j] = le[j] = 0;
                        if (nd[j] < old[j]) {
                            // whoever lowers x further in this step passes the same test and queues x too,
                            // so the minimum's old value is not needed
                            atomicMin(reinterpret_cast<int*>(a.dist + x[j]), __float_as_int(nd[j]));
                            const unsigned long long bit = 1ull << (x[j] & 63);
                            unsigned long long* fw = a.far_bm + (x[j] >> 6);
                            if (split && !(nd[j] < thr)) {
                                if (!(__ldcg(fw) & bit)) atomicOr(fw, bit);
                            } else {
                                const uint32_t prev = atomicExch(a.stamp + x[j], mark);
                                const uint64_t b = __ldg(a.off + x[j]), z = __ldg(a.off + (uint64_t)x[j] + 1);
                                if (split && (__ldcg(fw) & bit)) atomicAnd(fw, ~bit);  // queued: no longer parked
                                if (prev != mark) {
                                    lb[j] = b;
                                    le[j] = z;
                                }
                            }
                        }
                    }
                    append_pieces<kIlp>(lq, wb, x, lb, le, q_out, &out->n);
                }
            }
            ++pushes;
            last_kind = 0;
        } else {
            unsigned int mn = 0x7F800000u, left = 0;
            for (uint64_t base = tid & ~31ull; base < a.nwords; base += stride) {
                const uint64_t wi = base + lane;
                const unsigned long long word = wi < a.nwords ? __ldcg(a.far_bm + wi) : 0ull;
                unsigned long long move = 0;
                for (unsigned long long x = word; x; x &= x - 1) {
                    const int b = __ffsll((long long)x) - 1;
                    const float d = __ldcg(a.dist + wi * 64 + b);
                    if (d < thr) {
                        move |= 1ull << b;
                    } else {
                        ++left;
                        mn = min(mn, __float_as_uint(d));
                    }
                }
                if (move) a.far_bm[wi] = word & ~move;
                while (__any_sync(0xffffffffu, move != 0)) {
                    const uint32_t v[1] = {move ? (uint32_t)(wi * 64 + (uint64_t)(__ffsll((long long)move) - 1)) : 0u};
                    const uint64_t b[1] = {move ? __ldg(a.off + v[0]) : 0ull};
                    const uint64_t z[1] = {move ? __ldg(a.off + (uint64_t)v[0] + 1) : 0ull};
                    move &= move - 1;
                    append_pieces<1>(lq, wb, v, b, z, q_out, &out->n);
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
                left += __shfl_xor_sync(0xffffffffu, left, o);
            }
            if (lane == 0 && left) {
                atomicMin(&out->min_bits, mn);
                atomicAdd(&out->parked, left);
            }
            last_kind = 1;
        }
        ++step;
        flush_pieces(lq, wb, q_out, &out->n);
        if (!step_barrier(st, a.result, out, &s_slot, arrived)) return;
    }
    // every CTA leaves the loop at the same step; the edges walked are added up behind one more barrier
    if (lane == 0 && my_edges) atomicAdd(&st->edges, my_edges);
    if (!step_barrier(st, a.result, &st->slot[step & 3], &s_slot, arrived)) return;
    if (tid < 32) persist_clear(a.st_next);
    if (tid == 0) {
        st->step = step;
        st->thr = thr;
        st->delta = delta;
        st->pushes += pushes;
        *a.result = PersistResult{1u, done ? 1u : 0u, step, st->pushes, 0u, 0u, 0ull, __ldcg(&st->edges)};
    }
}

// The automatic threshold step, in mean weights.  A step costs a barrier and some L2 round trips
// (3.6 us with one CTA, 3.9 with 304) however few edges it relaxes, so graphs whose vertex arrays sit in L2 take steps so wide
// that R-MAT distances need one or two phases; larger ones gain more from relaxing less.  Times in
// ms with 0.7 / 3 / 100 x mean weight / mean degree: 20 k vertices, 300 k edges 1.14 / 0.51 / 0.28; 200 k,
// 4 M 1.99 / 0.87 / 0.56; 1 M, 8 M 1.42 / 1.07 / 0.88; 2 M, 64 M 4.4 / 2.9 / 3.7; 4 M, 20 M 1.8 / 2.4 / 3.1; 4 M,
// 67 M 3.8 / 3.8 / 5.4 (a tenth of the mean weight is 1.6 to 3.2 of these units there, and less than 0.7 of them on
// sparser graphs, which then take as many phases for nothing: with 0.1 / 0.7 / deg of the mean weight 4 M vertices,
// 8 M edges 5.7 / 2.5, a star of 4 M 0.57 / 0.17, a grid of 2000 x 2000 233 / 161).
// Few vertices with tens of thousands of edges each relax so many of them twice that steps matter less: with 10 / 100
// a uniform graph of 500 and 2^25 edges 2.0 / 4.9, R-MAT of 1,024 and 2^26 7.4 / 9.1, at degree 17,000 0.83 / 1.83 and,
// R-MAT of degree 2,048, 3.4 / 1.9.
static float auto_delta(uint64_t V, uint64_t E) {
    const float deg = (float)std::max((double)E / (double)V, 1.0);
    if (V <= (1u << 20)) return (deg > 32768.f ? 10.f : 100.f) / deg;
    if (V <= (1u << 23)) return std::max(0.1f, 0.7f / deg);
    return 0.7f / deg;
}

int run_sssp_persistent(eg_graph* g, uint32_t root, float* dist, int where) {
    const uint64_t V = g->V, E = g->E;
    EngineState& s = g->eng;
    EG_TRY(s.vals1.reserve(sizeof(uint32_t) * (V + 1)));
    EG_TRY(s.bm_visit.reserve(sizeof(uint64_t) * (V / 64 + 1)));
    const unsigned grid = (unsigned)persist_ctas(V, E, (uint64_t)g->num_sms);
    for (DevBuf* q : {&s.pieces0, &s.pieces1}) EG_TRY(q->reserve(sizeof(uint4) * queue_entries(V, E, grid)));
    float* d_dist = dist;
    if (where != EG_DEVICE || !plain_device(g, dist, 4)) {
        EG_TRY(s.vals0.reserve(sizeof(float) * (V + 1)));
        d_dist = s.vals0.as<float>();
    }
    SsspPersistArgs a;
    a.V = V;
    a.E = E;
    a.nwords = V / 64 + 1;
    a.off = g->csr_off.as<uint64_t>();
    a.adj = g->csr_adj.as<uint32_t>();
    a.w = g->csr_w.as<float>();
    a.dist = d_dist;
    a.stamp = s.vals1.as<uint32_t>();
    a.far_bm = s.bm_visit.as<unsigned long long>();
    a.q[0] = s.pieces0.as<uint4>();
    a.q[1] = s.pieces1.as<uint4>();
    a.root = root;
    a.delta = g->sssp_delta >= 0 ? (float)((double)g->sssp_delta * 1e-6) : -auto_delta(V, E);
    static_assert(sizeof(PersistState) <= kPersistBytes, "one block of the state words");
    void* block = nullptr;
    EG_TRY(persist_block(g, &block, &a.st_next));
    a.st = static_cast<PersistState*>(block);
    a.result = reinterpret_cast<PersistResult*>(s.host_words);
    const size_t smem = sizeof(LocalQueue);
    EG_CUDA(cudaFuncSetAttribute(k_sssp_persistent, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    volatile PersistResult* h = a.result;
    for (a.resume = 0;; a.resume = 1) {
        if (a.resume) EG_CUDA(cudaMemsetAsync(&a.st->bar_count, 0, sizeof(unsigned), g->stream));
        void* kargs[] = {&a};
        {
            Timed t(&g->prof, g->stream, "sssp_persistent");
            EG_CUDA(cudaLaunchCooperativeKernel((const void*)k_sssp_persistent, dim3(grid), dim3(kPersistThreads), kargs, smem,
                                                g->stream));
            EG_CHECK_LAUNCH("k_sssp_persistent");
            if (!a.resume) persist_launched(g);
        }
        EG_CUDA(cudaStreamSynchronize(g->stream));
        EG_TRY(persist_finish(g, "eg_sssp"));
        if (h->done) break;
        h->valid = 0;
    }
    g->last_edges_processed = h->edges;
    g->last_iterations = (int)h->pushes;
    g->last_pushes = (int)h->pushes;
    g->last_pulls = 0;
    if (dist && d_dist != dist) {
        EG_TRY(copy_out(g, dist, d_dist, sizeof(float) * V, where));
        EG_CUDA(cudaStreamSynchronize(g->stream));
    }
    return EG_OK;
}

// ---------------------------------------------------------------------------------------------
// BFS (toolkits/bfs.cpp:52-76): a push level claims unreached vertices through the level array; a
// dense level gives every compressed in-list of an unreached vertex a thread that looks at its first
// kBfsHead in-edges, then the warp walks what its 32 lists have left together, and lists longer than
// that are cut into segments that a second half of the level spreads over the GPU.  The frontier is
// "level == this level", or past 2^23 vertices the bits of kBits below.  Means of 16 roots, against the level loop driven
// from the host that it replaces (kernels per level, bitmaps, counters read back): 100,003 vertices,
// 1,000,003 edges 0.33 -> 0.08 ms; 2^22, 2^26 0.41 -> 0.26; 2^25, 2^29 2.11 -> 0.97 (1.29 by levels), most of it where the
// first dense level finds few parents in the lists' heads (5.04 -> 1.89 ms by levels: the rest of a list was one
// warp's).  A dense level is bound by its gathers: by levels, rounds of four in-edges, up to 12, took 1.29 ms, up
// to 8 1.34, up to 4 1.44, eight at once 1.54.
constexpr uint32_t kBfsHead = 12;
constexpr uint32_t kBfsSeg = 1024;
constexpr uint32_t kUnreached = 0xFFFFFFFFu;

struct alignas(16) BfsSlot {
    uint32_t n;               // queue entries appended
    uint32_t verts;           // vertices reached
    unsigned long long act;   // their out-edges
    uint32_t nseg;            // segments of the dense level
    uint32_t pad[3];
};

struct BfsPersistState {
    unsigned bar_count, bar_pad;
    int err;
    uint32_t step, pushes, pulls, pad[2];
    BfsSlot slot[4];  // as PersistState::slot
    unsigned long long reached, edges;
};

struct BfsPersistArgs {
    uint64_t V, nitems;
    const uint64_t* off;
    const uint32_t* adj;
    const uint32_t* csc_adj;
    const uint64_t* cidx;
    const uint32_t* cvert;
    uint32_t* level;
    uint32_t* parent;  // null: not wanted
    unsigned long long* vis;   // kBits: reached vertices, and those of before the dense level
    unsigned long long* snap;
    uint64_t nwords;
    uint4* q[2];
    unsigned long long* seg;  // (segment << 32) | compressed entry
    uint32_t root;
    int direction, has_csc;
    unsigned long long dense_min;
    int resume;
    BfsPersistState* st;
    void* st_next;  // the next launch's state, zeroed by this one
    PersistResult* result;
};

// Levels as the only record of what is reached are gathered from L2 while they fit it.  Past that (kBits) one bit per
// vertex says that it is reached (the level is stored before the bit may be seen; a bit that comes late costs a
// compare-and-swap that fails), and a dense level looks for parents in a copy of the bits from before it: a
// reached in-neighbour of an unreached vertex is in the frontier, or the vertex would have been reached with it.
__device__ __forceinline__ bool bit_at(const unsigned long long* w, uint32_t v) { return (__ldcg(w + (v >> 6)) >> (v & 63)) & 1ull; }
__device__ __forceinline__ void set_bit(unsigned long long* w, uint32_t v) { atomicOr(w + (v >> 6), 1ull << (v & 63)); }

template <bool kBits>
__global__ void __launch_bounds__(kPersistThreads, kPersistCtas) k_bfs_persistent(BfsPersistArgs a) {
    __shared__ BfsSlot s_slot;
    __shared__ uint32_t s_verts;
    __shared__ unsigned long long s_act;
    __shared__ uint32_t s_par[kPersistThreads];
    extern __shared__ __align__(16) unsigned char s_raw[];
    LocalQueue& lq = *reinterpret_cast<LocalQueue*>(s_raw);
    WarpBlock wb;
    if (threadIdx.x == 0) {
        lq.n = 0;
        lq.valid = 0xFFFFFFFFu;
        s_verts = 0;
        s_act = 0;
    }
    BfsPersistState* st = a.st;
    unsigned arrived = 0;
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint32_t warp = (uint32_t)(tid >> 5), nwarps = (uint32_t)(stride >> 5);
    uint32_t step = 0, pushes = 0, pulls = 0;
    unsigned long long reached = 0, edges = 0;
    if (!a.resume) {
        for (uint64_t v = tid; v < a.V; v += stride) {
            a.level[v] = v == a.root ? 0u : kUnreached;
            if (a.parent) a.parent[v] = v == a.root ? (uint32_t)v : (uint32_t)a.V;
        }
        if (kBits)
            for (uint64_t i = tid; i < a.nwords; i += stride) a.vis[i] = i == a.root >> 6 ? 1ull << (a.root & 63) : 0ull;
        if (tid < 32) {  // the root's pieces
            const uint64_t b = a.off[a.root], z = a.off[(uint64_t)a.root + 1];
            const uint32_t np = (uint32_t)((z - b + kPiece - 1) / kPiece);
            for (uint32_t p = lane; p < np; p += 32) a.q[0][p] = piece(a.root, b + (uint64_t)p * kPiece, z);
            if (lane == 0) {
                st->slot[0].n = np;
                st->slot[0].verts = 1;
                st->slot[0].act = z - b;
            }
        }
        if (!step_barrier(st, a.result, &st->slot[0], &s_slot, arrived)) return;
        reached = 1;
        edges = s_slot.act;
    } else {
        step = __ldcg(&st->step);
        if (threadIdx.x < sizeof(BfsSlot) / 16)
            reinterpret_cast<uint4*>(&s_slot)[threadIdx.x] =
                __ldcg(reinterpret_cast<const uint4*>(&st->slot[step & 3]) + threadIdx.x);
        __syncthreads();
        reached = __ldcg(&st->reached);
        edges = __ldcg(&st->edges);
    }
    const uint32_t first = step;
    while (s_slot.verts > 0 && step - first < kStepsPerLaunch) {
        const uint32_t n = s_slot.n;
        const bool dense = a.direction == 2 || (a.direction == 0 && a.has_csc && s_slot.act >= a.dense_min);
        BfsSlot* out = &st->slot[(step + 1) & 3];
        uint4* q_out = a.q[(step + 1) & 1];
        const uint32_t lvl = step;  // the frontier's level
        uint32_t my_verts = 0;
        unsigned long long my_act = 0;
        __syncthreads();  // s_slot has been read
        if (tid == 0) {
            BfsSlot* clear = &st->slot[(step + 2) & 3];
            clear->n = clear->verts = clear->nseg = 0;
            clear->act = 0;
        }
        // hand the step's totals and the gathered queue entries over; false: a barrier gave up
        auto end_phase = [&](bool step_done) -> bool {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                my_verts += __shfl_xor_sync(0xffffffffu, my_verts, o);
                my_act += __shfl_xor_sync(0xffffffffu, my_act, o);
            }
            if (lane == 0 && my_verts) {
                atomicAdd(&s_verts, my_verts);
                atomicAdd(&s_act, my_act);
            }
            my_verts = 0;
            my_act = 0;
            flush_pieces(lq, wb, q_out, &out->n, step_done);
            if (threadIdx.x == 0 && s_verts) {
                atomicAdd(&out->verts, s_verts);
                atomicAdd(&out->act, s_act);
                s_verts = 0;
                s_act = 0;
            }
            return step_barrier(st, a.result, out, &s_slot, arrived);
        };
        if (!dense) {
            const uint4* q = a.q[step & 1];
            for (uint32_t base = 0; base < n; base += 32 * nwarps) {
                const uint64_t idx = (uint64_t)base + (uint64_t)lane * nwarps + warp;
                uint64_t beg = 0;
                uint32_t len = 0, u = 0;
                if (idx < n) {
                    const uint4 e = __ldcg(q + idx);
                    u = e.x;
                    beg = ((uint64_t)e.z << 32) | e.y;
                    len = e.w;
                }
                const uint32_t incl = warp_incl(len);
                const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
                beg -= incl - len;
                for (uint32_t r0 = 0; r0 < total; r0 += 32 * kIlp) {
                    uint32_t x[kIlp], par[kIlp];
                    uint64_t lb[kIlp], le[kIlp];
                    bool open[kIlp];
#pragma unroll
                    for (int j = 0; j < kIlp; ++j) {
                        const uint32_t r = r0 + 32 * j + lane;
                        const uint32_t o = warp_owner(incl, r);
                        const uint64_t pos = __shfl_sync(0xffffffffu, beg, o) + r;
                        par[j] = __shfl_sync(0xffffffffu, u, o);
                        x[j] = r < total ? __ldg(a.adj + pos) : a.root;
                    }
#pragma unroll
                    for (int j = 0; j < kIlp; ++j)
                        open[j] = kBits ? !bit_at(a.vis, x[j]) : __ldcg(a.level + x[j]) == kUnreached;
#pragma unroll
                    for (int j = 0; j < kIlp; ++j) {
                        lb[j] = le[j] = 0;
                        if (open[j]) {
                            const uint32_t old = atomicCAS(a.level + x[j], kUnreached, lvl + 1);
                            const uint64_t b = __ldg(a.off + x[j]), z = __ldg(a.off + (uint64_t)x[j] + 1);
                            if (old == kUnreached) {
                                if (kBits) set_bit(a.vis, x[j]);
                                if (a.parent) a.parent[x[j]] = par[j];
                                lb[j] = b;
                                le[j] = z;
                                ++my_verts;
                                my_act += z - b;
                            }
                        }
                    }
                    append_pieces<kIlp>(lq, wb, x, lb, le, q_out, &out->n);
                }
            }
            ++pushes;
            if (!end_phase(true)) return;
        } else {
            if (kBits) {
                for (uint64_t i = tid; i < a.nwords; i += stride) a.snap[i] = __ldcg(a.vis + i);
                if (!step_barrier(st, a.result, &st->slot[step & 3], &s_slot, arrived)) return;
            }
            auto unreached = [&](uint32_t v) { return kBits ? !bit_at(a.vis, v) : __ldcg(a.level + v) == kUnreached; };
            auto in_front = [&](uint32_t u) { return kBits ? bit_at(a.snap, u) : __ldcg(a.level + u) == lvl; };
            // a list's vertex is loaded two rounds ahead, its level and bounds one round ahead
            uint64_t i = tid;
            uint32_t v1 = i < a.nitems ? __ldg(a.cvert + i) : kUnreached;
            uint32_t v2 = i + stride < a.nitems ? __ldg(a.cvert + i + stride) : kUnreached;
            bool open1 = v1 < a.V && unreached(v1);
            uint64_t p1 = i < a.nitems ? __ldg(a.cidx + i) : 0, e1 = i < a.nitems ? __ldg(a.cidx + i + 1) : 0;
            for (uint64_t base = tid & ~31ull; base < a.nitems; base += stride, i += stride) {
                const uint32_t v = v1;
                const bool open = open1;
                uint64_t p = p1;
                const uint64_t e = e1;
                uint32_t par = kUnreached, len = 0, nsg = 0;
                v1 = v2;
                v2 = i + 2 * stride < a.nitems ? __ldg(a.cvert + i + 2 * stride) : kUnreached;
                open1 = v1 < a.V && unreached(v1);
                if (i + stride < a.nitems) {
                    p1 = __ldg(a.cidx + i + stride);
                    e1 = __ldg(a.cidx + i + stride + 1);
                }
                if (open) {
                    const uint64_t h = e - p > kBfsHead ? p + kBfsHead : e;
                    for (uint64_t x = p; x < h && par == kUnreached; x += 4) {
                        uint32_t u[4];
                        bool hit[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) u[j] = x + j < h ? __ldg(a.csc_adj + x + j) : a.root;
#pragma unroll
                        for (int j = 0; j < 4; ++j) hit[j] = x + j < h && in_front(u[j]);
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            if (hit[j]) par = u[j];
                    }
                    if (par == kUnreached && e > h) {
                        p = h;
                        if (e - h <= kBfsSeg) len = (uint32_t)(e - h);
                        else nsg = (uint32_t)((e - h + kBfsSeg - 1) / kBfsSeg);
                    }
                }
                // the rest of the warp's lists, walked together
                const uint32_t incl = warp_incl(len);
                const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
                if (total) {
                    uint32_t* found = s_par + (threadIdx.x & ~31u);
                    found[lane] = kUnreached;
                    __syncwarp();
                    const uint64_t beg = p - (incl - len);
                    for (uint32_t r0 = 0; r0 < total; r0 += 32 * kIlp) {
                        uint32_t u[kIlp], o[kIlp];
                        bool want[kIlp];
#pragma unroll
                        for (int j = 0; j < kIlp; ++j) {
                            const uint32_t r = r0 + 32 * j + lane;
                            o[j] = warp_owner(incl, r);
                            const uint64_t pos = __shfl_sync(0xffffffffu, beg, o[j]) + r;
                            want[j] = r < total && *(volatile uint32_t*)(found + o[j]) == kUnreached;
                            u[j] = want[j] ? __ldg(a.csc_adj + pos) : a.root;
                        }
#pragma unroll
                        for (int j = 0; j < kIlp; ++j)
                            if (want[j] && in_front(u[j])) *(volatile uint32_t*)(found + o[j]) = u[j];
                    }
                    __syncwarp();
                    if (len) par = found[lane];
                    __syncwarp();
                }
                const uint32_t sincl = warp_incl(nsg);
                const uint32_t stot = __shfl_sync(0xffffffffu, sincl, 31);
                if (stot) {
                    uint32_t at = 0;
                    if (lane == 31) at = atomicAdd(&out->nseg, stot);
                    at = __shfl_sync(0xffffffffu, at, 31) + sincl - nsg;
                    for (uint32_t k = 0; k < nsg; ++k) a.seg[at + k] = ((unsigned long long)k << 32) | (uint32_t)i;
                }
                const uint32_t vv[1] = {v};
                uint64_t lb[1] = {0}, le[1] = {0};
                if (open && par != kUnreached) {  // this lane owns v's only list
                    a.level[v] = lvl + 1;
                    if (kBits) set_bit(a.vis, v);
                    if (a.parent) a.parent[v] = par;
                    lb[0] = __ldg(a.off + v);
                    le[0] = __ldg(a.off + (uint64_t)v + 1);
                    ++my_verts;
                    my_act += le[0] - lb[0];
                }
                append_pieces<1>(lq, wb, vv, lb, le, q_out, &out->n);
            }
            ++pulls;
            if (!end_phase(false)) return;  // whether there are segments is known behind the barrier
            const uint32_t nseg = s_slot.nseg;
            if (!nseg) wb.phase_done(true);
            if (nseg) {  // long lists, a warp per segment; the first segment to find a parent claims
                __syncthreads();  // s_slot has been read
                for (uint32_t t = warp; t < nseg; t += nwarps) {
                    const unsigned long long ent = __ldcg(a.seg + t);
                    const uint32_t i = (uint32_t)ent;
                    const uint32_t v = __ldg(a.cvert + i);
                    const uint64_t e = __ldg(a.cidx + i + 1);
                    uint64_t p = __ldg(a.cidx + i) + kBfsHead + (ent >> 32) * kBfsSeg;
                    const uint64_t pe = p + kBfsSeg < e ? p + kBfsSeg : e;
                    const uint32_t vv[1] = {v};
                    uint64_t lb[1] = {0}, le[1] = {0};
                    for (; p < pe; p += 32 * kIlp) {
                        if (__shfl_sync(0xffffffffu, __ldcg(a.level + v), 0) != kUnreached) break;
                        uint32_t cand = kUnreached;
#pragma unroll
                        for (int j = 0; j < kIlp; ++j) {
                            const uint64_t x = p + 32 * j + lane;
                            const uint32_t u = x < pe ? __ldg(a.csc_adj + x) : a.root;
                            if (x < pe && in_front(u)) cand = u;
                        }
                        const unsigned m = __ballot_sync(0xffffffffu, cand != kUnreached);
                        if (!m) continue;
                        const uint32_t par = __shfl_sync(0xffffffffu, cand, __ffs(m) - 1);
                        if (lane == 0 && atomicCAS(a.level + v, kUnreached, lvl + 1) == kUnreached) {
                            if (kBits) set_bit(a.vis, v);
                            if (a.parent) a.parent[v] = par;
                            lb[0] = __ldg(a.off + v);
                            le[0] = __ldg(a.off + (uint64_t)v + 1);
                            ++my_verts;
                            my_act += le[0] - lb[0];
                        }
                        break;
                    }
                    append_pieces<1>(lq, wb, vv, lb, le, q_out, &out->n);
                }
                if (!end_phase(true)) return;
            }
        }
        reached += s_slot.verts;
        edges += s_slot.act;
        ++step;
    }
    if (tid < 32) persist_clear(a.st_next);
    if (tid == 0) {  // every CTA leaves the loop at the same step
        st->step = step;
        st->reached = reached;
        st->edges = edges;
        st->pushes += pushes;
        st->pulls += pulls;
        *a.result = PersistResult{1u, s_slot.verts == 0 ? 1u : 0u, step, st->pushes, st->pulls, 0u, reached, edges};
    }
}

// Bits from more than this many vertices on.  Means of four roots, levels alone / host-driven levels with bitmaps
// before them / bits, in ms: R-MAT 2^22 / 2^26 0.21 / 0.52 / 0.22, 2^23 / 2^27 0.33 / 0.63 / 0.33, 2^24 / 2^28 0.59 / 0.88 /
// 0.55, 2^25 / 2^29 1.08 / 1.33 / 0.92, 2^27 / 2^30 3.91 / 3.54 / 2.47; uniform 2^20 / 2^24 0.17 / 1.00 / 0.19, 2^23 / 2^24
// 1.22 / 3.03 / 1.21, 2^26 / 2^27 10.6 / 9.8 / 8.1, 2^27 / 2^28 23.3 / 18.3 / 16.6.
constexpr uint64_t kBfsBits = 1ull << 23;

int run_bfs_persistent(eg_graph* g, uint32_t root, uint32_t* level, uint32_t* parent, int where, uint64_t* reached) {
    const uint64_t V = g->V, E = g->E;
    EngineState& s = g->eng;
    const unsigned grid = (unsigned)persist_ctas(V, E, (uint64_t)g->num_sms);
    for (DevBuf* q : {&s.pieces0, &s.pieces1}) EG_TRY(q->reserve(sizeof(uint4) * queue_entries(V, E, grid)));
    BfsPersistArgs a;
    a.level = level;
    a.parent = parent;
    if (where != EG_DEVICE || !plain_device(g, level, 4)) {
        EG_TRY(s.vals0.reserve(sizeof(uint32_t) * (V + 1)));
        a.level = s.vals0.as<uint32_t>();
    }
    if (parent && (where != EG_DEVICE || !plain_device(g, parent, 4))) {
        EG_TRY(s.vals1.reserve(sizeof(uint32_t) * (V + 1)));
        a.parent = s.vals1.as<uint32_t>();
    }
    a.V = V;
    a.nitems = g->built_csc ? g->ncompressed - 1 : 0;
    if (g->built_csc) EG_TRY(s.bu_seg.reserve(sizeof(unsigned long long) * (2 * (E / kBfsSeg) + 2)));
    a.off = g->csr_off.as<uint64_t>();
    a.adj = g->csr_adj.as<uint32_t>();
    a.csc_adj = g->csc_adj.as<uint32_t>();
    a.cidx = g->cidx.as<uint64_t>();
    a.cvert = g->cvert.as<uint32_t>();
    a.q[0] = s.pieces0.as<uint4>();
    a.q[1] = s.pieces1.as<uint4>();
    a.seg = s.bu_seg.as<unsigned long long>();
    a.root = root;
    a.direction = g->bfs_direction;
    a.has_csc = g->built_csc ? 1 : 0;
    a.dense_min = E / (uint64_t)g->dense_div;
    static_assert(sizeof(BfsPersistState) <= kPersistBytes, "one block of the state words");
    void* block = nullptr;
    EG_TRY(persist_block(g, &block, &a.st_next));
    a.st = static_cast<BfsPersistState*>(block);
    a.result = reinterpret_cast<PersistResult*>(s.host_words);
    const bool bits = V > kBfsBits;
    a.nwords = V / 64 + 1;
    if (bits)
        for (DevBuf* w : {&s.bm_visit, &s.bm_front}) EG_TRY(w->reserve(sizeof(uint64_t) * a.nwords));
    a.vis = s.bm_visit.as<unsigned long long>();
    a.snap = s.bm_front.as<unsigned long long>();
    const void* fn = bits ? (const void*)k_bfs_persistent<true> : (const void*)k_bfs_persistent<false>;
    const size_t smem = sizeof(LocalQueue);
    EG_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    volatile PersistResult* h = a.result;
    for (a.resume = 0;; a.resume = 1) {
        if (a.resume) EG_CUDA(cudaMemsetAsync(&a.st->bar_count, 0, sizeof(unsigned), g->stream));
        void* kargs[] = {&a};
        {
            Timed t(&g->prof, g->stream, "bfs_persistent");
            EG_CUDA(cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kPersistThreads), kargs, smem,
                                                g->stream));
            EG_CHECK_LAUNCH("k_bfs_persistent");
            if (!a.resume) persist_launched(g);
        }
        EG_CUDA(cudaStreamSynchronize(g->stream));
        EG_TRY(persist_finish(g, "eg_bfs"));
        if (h->done) break;
        h->valid = 0;
    }
    g->last_edges_processed = h->edges;  // sum of out-degrees of the reached vertices
    g->last_iterations = (int)h->step;
    g->last_pushes = (int)h->pushes;
    g->last_pulls = (int)h->pulls;
    if (reached) *reached = h->reached;
    if ((level && a.level != level) || a.parent != parent) {
        if (a.level != level) EG_TRY(copy_out(g, level, a.level, sizeof(uint32_t) * V, where));
        if (a.parent != parent) EG_TRY(copy_out(g, parent, a.parent, sizeof(uint32_t) * V, where));
        EG_CUDA(cudaStreamSynchronize(g->stream));
    }
    return EG_OK;
}

// ---------------------------------------------------------------------------------------------
// Connected components of a symmetrised graph (toolkits/cc.cpp's labels: the smallest vertex of each
// component) by union-find instead of label propagation: every vertex's parent is a smaller or equal
// vertex, a union hooks the larger of two roots under the smaller, so a component's root is its
// smallest vertex.  After the first two neighbours of every vertex are united, one component holds
// most of an R-MAT graph; the lists of its vertices need not be read (an edge that leaves it is in
// the other end's list too), and the rest go through the piece queue, so that long lists are spread
// over the GPU: the neighbour sampling of Afforest (Sutton, Ben-Nun and Barak, IPDPS 2018).
// Reads 2 V neighbours and a few lists instead of every edge several times: 10.4 M vertices, 734 M
// edges: 9.1 ms as three dense sweeps and a push, 1.6 ms so.  It is bound by walks up the trees that end at a
// few vertices: with loads past L1 2.9 ms, and 4.8 to 6.1 when the first neighbours were united with atomics.
struct alignas(16) CcSlot {
    uint32_t n;       // queue entries
    uint32_t common;  // the component that the lists are skipped for
    uint32_t pad[2];
};
struct CcState {
    unsigned bar_count, bar_pad;
    int err;
    uint32_t pad;
    CcSlot slot;
};
struct CcArgs {
    uint64_t V, nlists;
    const uint32_t* deg;
    const uint32_t* vert;  // kIndex: the vertices with neighbours (the compressed index); else list i is vertex i's
    const uint64_t* off;
    const uint32_t* adj;
    uint32_t* comp;
    uint4* q;
    CcState* st;
    void* st_next;  // the next launch's state, zeroed by this one
    PersistResult* result;
};
constexpr uint32_t kCcFirst = 2;      // neighbours united before the common component is looked for
constexpr int kCcSamples = 1024;

// The root of v's tree; parents get smaller on the way up, so the walk ends.  The loads may hit L1 (most
// walks end at the same few vertices, whose L2 lines would be read by every warp): a parent that is out
// of date is still an ancestor, and a grid barrier leaves no line of before it.
__device__ __forceinline__ uint32_t cc_root(const uint32_t* comp, uint32_t v) {
    for (uint32_t p = __ldca(comp + v); p != v; p = __ldca(comp + v)) v = p;
    return v;
}

// one tree out of u's and v's; a root that another thread hooked meanwhile leads on to its parent
__device__ __forceinline__ void cc_unite(uint32_t* comp, uint32_t u, uint32_t v) {
    while (true) {
        u = cc_root(comp, u);
        v = cc_root(comp, v);
        if (u == v) return;
        if (u < v) {
            const uint32_t x = u;
            u = v;
            v = x;
        }
        const uint32_t p = atomicCAS(comp + u, u, v);
        if (p == u) return;
        u = p;
    }
}

template <bool kIndex>
__device__ __forceinline__ uint32_t cc_vertex(const uint32_t* vert, uint64_t i) { return kIndex ? __ldg(vert + i) : (uint32_t)i; }

template <bool kIndex>
__device__ __forceinline__ void cc_compress(uint32_t* comp, const uint32_t* __restrict__ vert, uint64_t n, uint64_t tid,
                                            uint64_t stride) {
    for (uint64_t i = tid; i < n; i += stride) {
        const uint32_t v = cc_vertex<kIndex>(vert, i), p = __ldca(comp + v), r = cc_root(comp, p);
        if (r != p) comp[v] = r;
    }
}

template <bool kIndex>
__global__ void __launch_bounds__(kPersistThreads, kPersistCtas) k_cc_persistent(CcArgs a) {
    __shared__ CcSlot s_slot;
    __shared__ uint32_t s_sample[kCcSamples];
    __shared__ unsigned long long s_best;
    extern __shared__ __align__(16) unsigned char s_raw[];
    LocalQueue& lq = *reinterpret_cast<LocalQueue*>(s_raw);
    WarpBlock wb;
    if (threadIdx.x == 0) {
        lq.n = 0;
        lq.valid = 0xFFFFFFFFu;
        s_best = 0;
    }
    CcState* st = a.st;
    unsigned arrived = 0;
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint32_t warp = (uint32_t)(tid >> 5), nwarps = (uint32_t)(stride >> 5);
    // A vertex with neighbours starts under the smallest of itself and its first ones.  The others are done: what
    // follows passes over the compressed index (over all vertices, the 2^26 of a graph with 2^21 edges took 3.8 ms).
    for (uint64_t v = tid; v < a.V; v += stride)
        if (!__ldg(a.deg + v)) a.comp[v] = (uint32_t)v;
    for (uint64_t i = tid; i < a.nlists; i += stride) {
        const uint64_t b = __ldg(a.off + i), e = __ldg(a.off + i + 1);
        const uint32_t v = cc_vertex<kIndex>(a.vert, i);
        uint32_t p = v;
#pragma unroll
        for (uint32_t k = 0; k < kCcFirst; ++k)
            if (b + k < e) p = min(p, __ldg(a.adj + b + k));
        a.comp[v] = p;
    }
    if (!step_barrier(st, a.result, &st->slot, &s_slot, arrived)) return;
    cc_compress<kIndex>(a.comp, a.vert, a.nlists, tid, stride);
    if (!step_barrier(st, a.result, &st->slot, &s_slot, arrived)) return;
    for (uint32_t k = 0; k < kCcFirst; ++k) {
        for (uint64_t i = tid; i < a.nlists; i += stride) {
            const uint64_t b = __ldg(a.off + i) + k;
            if (b < __ldg(a.off + i + 1)) cc_unite(a.comp, cc_vertex<kIndex>(a.vert, i), __ldg(a.adj + b));
        }
        if (!step_barrier(st, a.result, &st->slot, &s_slot, arrived)) return;
        cc_compress<kIndex>(a.comp, a.vert, a.nlists, tid, stride);
        if (!step_barrier(st, a.result, &st->slot, &s_slot, arrived)) return;
    }
    // the component of most of a sample's vertices; one CTA decides for all
    if (blockIdx.x == 0) {
        for (int i = threadIdx.x; i < kCcSamples; i += blockDim.x)
            s_sample[i] = a.nlists ? __ldcg(a.comp + cc_vertex<kIndex>(a.vert, (uint64_t)(i * 2654435761u) * a.nlists / (1ull << 32))) : 0u;
        __syncthreads();
        for (int i = threadIdx.x; i < kCcSamples; i += blockDim.x) {
            uint32_t same = 0;
            for (int j = 0; j < kCcSamples; ++j) same += s_sample[j] == s_sample[i];
            atomicMax(&s_best, ((unsigned long long)same << 32) | s_sample[i]);
        }
        __syncthreads();
        if (threadIdx.x == 0) st->slot.common = (uint32_t)s_best;
    }
    if (!step_barrier(st, a.result, &st->slot, &s_slot, arrived)) return;
    const uint32_t common = s_slot.common;
    // the other components' lists, from the third neighbour on
    for (uint64_t base = tid & ~31ull; base < a.nlists; base += stride) {
        const uint64_t i = base + lane;
        const uint32_t vv[1] = {i < a.nlists ? cc_vertex<kIndex>(a.vert, i) : 0u};
        uint64_t lb[1] = {0}, le[1] = {0};
        if (i < a.nlists && __ldcg(a.comp + vv[0]) != common) {
            lb[0] = __ldg(a.off + i) + kCcFirst;
            le[0] = __ldg(a.off + i + 1);
            if (lb[0] >= le[0]) lb[0] = le[0] = 0;
        }
        append_pieces<1>(lq, wb, vv, lb, le, a.q, &st->slot.n);
    }
    flush_pieces(lq, wb, a.q, &st->slot.n);
    if (!step_barrier(st, a.result, &st->slot, &s_slot, arrived)) return;
    const uint32_t n = s_slot.n;
    if (n) {
        for (uint32_t base = 0; base < n; base += 32 * nwarps) {
            const uint64_t idx = (uint64_t)base + (uint64_t)lane * nwarps + warp;
            uint64_t beg = 0;
            uint32_t len = 0, u = 0;
            if (idx < n) {
                const uint4 e = __ldcg(a.q + idx);
                u = e.x;
                beg = ((uint64_t)e.z << 32) | e.y;
                len = e.w;
            }
            const uint32_t incl = warp_incl(len);
            const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
            beg -= incl - len;
            for (uint32_t r0 = 0; r0 < total; r0 += 32) {
                const uint32_t r = r0 + lane;
                const uint32_t o = warp_owner(incl, r);
                const uint64_t pos = __shfl_sync(0xffffffffu, beg, o) + r;
                const uint32_t ou = __shfl_sync(0xffffffffu, u, o);
                if (r < total) cc_unite(a.comp, ou, __ldg(a.adj + pos));
                __syncwarp();
            }
        }
        if (!step_barrier(st, a.result, &st->slot, &s_slot, arrived)) return;
        cc_compress<kIndex>(a.comp, a.vert, a.nlists, tid, stride);
    }
    if (tid < 32) persist_clear(a.st_next);
    if (tid == 0) a.result->valid = 1;
}

int run_cc_symmetric(eg_graph* g, uint32_t* label, int where) {
    const uint64_t V = g->V, E = g->E;
    EngineState& s = g->eng;
    const unsigned grid = (unsigned)persist_ctas(4 * V, E / 16, (uint64_t)g->num_sms);
    EG_TRY(s.pieces0.reserve(sizeof(uint4) * queue_entries(V, E, grid)));
    static_assert(sizeof(CcState) <= kPersistBytes, "one block of the state words");
    void *block = nullptr, *next = nullptr;
    EG_TRY(persist_block(g, &block, &next));
    PersistResult* h = reinterpret_cast<PersistResult*>(s.host_words);
    uint32_t* comp = label;
    if (where != EG_DEVICE || !plain_device(g, label, 4)) {
        EG_TRY(s.vals0.reserve(sizeof(uint32_t) * (V + 1)));
        comp = s.vals0.as<uint32_t>();
    }
    // The passes go over the compressed index where a quarter of the vertices and more have no neighbours: 2^26 with
    // 2,000 / 2^21 / 2^26 list entries take 1.84 / 3.8 / 10.0 ms over all vertices and 0.29 / 0.61 / 8.4 so, an
    // R-MAT of 2^23 / 2^27 1.10 and 0.93.  With next to none the index is 12 bytes a vertex for nothing: uniform
    // graphs of 2^26 / 2^28 take 14.8 and 17.0, of 2^23 / 2^25 1.45 and 1.65.
    const uint64_t nitems = g->ncompressed - 1;
    const bool index = nitems < V - V / 4;
    CcArgs a{V, index ? nitems : V, g->outdeg.as<uint32_t>(), index ? g->cvert.as<uint32_t>() : nullptr,
             index ? g->cidx.as<uint64_t>() : g->csr_off.as<uint64_t>(),
             index ? g->csc_adj.as<uint32_t>() : g->csr_adj.as<uint32_t>(), comp, s.pieces0.as<uint4>(),
             static_cast<CcState*>(block), next, h};
    const size_t smem = sizeof(LocalQueue);
    const void* fn = index ? (const void*)k_cc_persistent<true> : (const void*)k_cc_persistent<false>;
    EG_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    void* kargs[] = {&a};
    {
        Timed t(&g->prof, g->stream, "cc_persistent");
        EG_CUDA(cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kPersistThreads), kargs, smem,
                                            g->stream));
        EG_CHECK_LAUNCH("k_cc_persistent");
        persist_launched(g);
    }
    if (comp != label) EG_TRY(copy_out(g, label, comp, sizeof(uint32_t) * V, where));
    EG_CUDA(cudaStreamSynchronize(g->stream));
    EG_TRY(persist_finish(g, "eg_cc"));
    g->last_edges_processed = E;  // united once, or skipped because both ends were
    g->last_iterations = 1;
    g->last_pushes = 0;
    g->last_pulls = 1;
    return EG_OK;
}

}  // namespace eg
