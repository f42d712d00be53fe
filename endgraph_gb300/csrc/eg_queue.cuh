// eg_queue.cuh — how many entries a step of the persistent traversals (eg_persist.cu) can leave in its
// queue of list pieces, and the blocks that warps reserve in it.  No CUDA in here: the host sizes the
// queues with it, the kernels take their blocks by it, and a CPU test counts one against the other.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define EG_QUEUE_FN __host__ __device__ __forceinline__
#else
#define EG_QUEUE_FN inline
#endif

namespace eg {

constexpr uint32_t kPiece = 256;  // edges per queue entry
// Two CTAs of 512 threads per SM at 64 registers.  Measured on the first BFS kernel (levels alone, the rest of a long list
// walked by one thread): 2^25 / 2^29 1.61 ms (mean of 16 roots) against 1.66 with one CTA of 1,024, 1.70 with
// three of 512 (42 registers), 1.75 with two of 768 and 1.87 with two of 1,024; 2^22 / 2^26 0.29 against 0.30 / 0.28 /
// 0.29 / 0.32.
constexpr int kPersistThreads = 512;
constexpr int kPersistCtas = 2;
// A CTA's share of the next queue gathers in shared memory and goes out with one reservation.  What does
// not fit goes to the global queue in blocks of kQueueBlock entries that one warp reserves at a time (a
// reservation per warp and 128 edges made a push level of 2.7 M activations 0.38 ms long).
constexpr uint32_t kLocalQueue = 2048;
constexpr uint32_t kQueueBlock = 256;

// CTAs of a launch: one per kEdgesPerCta edges and per kVerticesPerCta vertices, whose values it sets up,
// up to the GPU's.  Fewer CTAs meet sooner at a barrier, but 2,048 edges were no slower than 4,096 or 8,192
// from 20 k edges on (0.134 / 0.142 / 0.159 ms at 2 k vertices, 20 k edges).  Without a share for
// the vertices an SSSP of 2^26 with 1,000 edges had one CTA to set them up and took 9.4 ms.
constexpr uint64_t kEdgesPerCta = 2048, kVerticesPerCta = 8192;
inline uint64_t persist_ctas(uint64_t V, uint64_t E, uint64_t num_sms) {
    const uint64_t want = E / kEdgesPerCta + V / kVerticesPerCta, most = num_sms * kPersistCtas;
    return want < 1 ? 1 : want < most ? want : most;
}

struct WarpBlock {  // the warp's block of the global queue, the same in every lane
    uint32_t pos = 0, end = 0;

    // entries to reserve before `tot` more are stored; 0: they fit what is left of the block
    EG_QUEUE_FN uint32_t wants(uint32_t tot) const {
        const uint32_t room = end - pos;
        return tot <= room ? 0u : tot - room > kQueueBlock ? tot - room : kQueueBlock;
    }
    // `tot` entries stored, the first ones in the room that was left, the rest from `fresh` on, where
    // `block` = wants(tot) entries were reserved
    EG_QUEUE_FN void took(uint32_t tot, uint32_t fresh, uint32_t block) {
        const uint32_t room = end - pos;
        if (tot > room) {
            pos = fresh + (tot - room);
            end = fresh + block;
        } else {
            pos += tot;
        }
    }
    // The queue's readers find [pos, end) filled with empty pieces.  A phase that another one of the same
    // step follows keeps the block, so that a warp leaves one unfinished block per step however many
    // phases it has (a dense BFS level with long lists has two).
    EG_QUEUE_FN void phase_done(bool step_done) {
        if (step_done) pos = end = 0;
    }
};

// Entries of one step's queue: the pieces (a vertex's list is queued at most once per step) and the
// unfinished blocks of the warps of CTAs that can fill their shared part at all.
inline uint64_t queue_entries(uint64_t V, uint64_t E, uint64_t ctas) {
    const uint64_t pieces = (V < E ? V : E) + E / kPiece, full = pieces / kLocalQueue;
    return pieces + (ctas < full ? ctas : full) * (kPersistThreads / 32) * kQueueBlock + 64;
}

}  // namespace eg
