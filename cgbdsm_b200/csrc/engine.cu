// B200 engine for the per-batch GPU path of continuous subgraph matching.
//
// Device data layout (HBM):
//   pool   u32 words holding every sorted neighbour run; runs start on 16-byte
//          boundaries; allocation is a bump pointer, updated runs are written
//          out of place and dead space is reclaimed by compaction.
//   rec    uint4 per (direction d, compressed vertex u), row-major [d][dvcap]:
//          x = run offset (words), y = run length, z = delta offset, w = delta length.
//          One 16-byte load resolves both the old list and this batch's delta
//          list of (d, u) (the two halves the reference keeps in index_gpu and
//          update_index, graph_gpu.h:41-49).
//   dval   this batch's delta values, sorted by (d, u, v), not deduplicated
//          (calig_helper_gamma.cu:569-573).
//
// Per batch (calig_helper_gamma.cu:485-597 + graph_gpu.cu:1261-1480):
//   1. edits = previous delta (deferred merge-back) + ins (add) + del (remove),
//      packed to (d,u,v,op) and radix-sorted; one warp per touched (d,u) writes
//      (old run U adds) \ removes.  One pass over each touched run per batch,
//      where the reference makes three (merge ins, remove del, merge delta).
//   2. delta keys packed + sorted -> dval and rec.z/.w for touched (d,u).
//   3. persistent warp DFS seeded from the delta edges of every query edge
//      (all query edges in one launch; the edge index ei travels with the seed).
//   4. rec.z/.w of touched (d,u) cleared; this batch's delta becomes the
//      pending merge-back of the next batch.
#include <cuda_runtime.h>
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdlib>
#include <cstdio>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "alloc_count.h"
#include "cgbdsm.h"
#include "query.h"
#include "seed_claim.h"

using cgb::EdgePlan;
using cgb::kMaxBN;
using cgb::kMaxDir;
using cgb::kMaxQE;
using cgb::kMaxQV;

namespace {

constexpr uint32_t kFull = 0xffffffffu;
constexpr int kDfsWarps = 8;  // warps per DFS block
constexpr uint32_t kTaskCap = 1u << 20;  // stolen-range ring capacity (64 MiB), a power of two
constexpr uint32_t kTaskSlack = 1u << 13; // tickets kept between the ring's tail and head
constexpr uint64_t kMaxBatchKeys = 1ull << 36;  // per key array of one batch: 512 GiB, beyond any HBM

// Plans belong to a handle (several handles may share a process and a
// device): they live in the handle's device memory, and the DFS copies them
// to shared memory as 32-bit words.
static_assert(sizeof(EdgePlan) % 4 == 0, "EdgePlan must be a whole number of words");

// ---------------------------------------------------------------------------
// key packing
// ---------------------------------------------------------------------------
struct PackInfo {
    uint32_t B;      // bits per vertex id
    uint32_t nd;     // directions
    uint32_t dv;     // compressed vertex count
    uint32_t pad_ok; // an all-ones key is padding (skipped), not an invalid key
};

__device__ __forceinline__ bool decode_ext(uint64_t k, const PackInfo& pi, uint32_t& d, uint32_t& u,
                                           uint32_t& v) {
    d = (uint32_t)(k >> 59);
    u = (uint32_t)((k >> 32) & 0x07FFFFFFu);
    v = (uint32_t)k;
    return d < pi.nd && u < pi.dv && v < pi.dv;
}

__device__ __forceinline__ uint64_t pack_duv(uint32_t d, uint32_t u, uint32_t v, uint32_t B) {
    return ((uint64_t)d << (2 * B)) | ((uint64_t)u << B) | (uint64_t)v;
}

// Edits of one merge, in up to three pieces: keys already packed as (d,u,v)
// with B0 bits per vertex (the delta kept for the merge-back, or selected
// deletions), and external keys to add and to remove.
struct EditSrc {
    const uint64_t* packed = nullptr;
    uint64_t n_packed = 0;
    uint32_t B0 = 0, packed_op = 0;
    const uint64_t* add = nullptr;
    uint64_t n_add = 0;
    const uint64_t* rem = nullptr;
    uint64_t n_rem = 0;
};

// Edits: ((d,u,v) << 1) | op, op 0 = add, 1 = remove.  Keys whose direction
// or vertex ids are out of range raise error bit 1 and become the all-ones
// marker, which sorts last and is skipped by the merge.
// Added keys with u == v (a self-loop in the data graph) set the sticky
// self_seen flag: until one appears no vertex lies in its own lists, which
// lets the matcher skip those exclusion tests (packed keys were checked when
// they were packed).
__global__ void k_pack_edits(EditSrc src, PackInfo pi, uint64_t* __restrict__ out, unsigned int* err,
                             unsigned int* self_seen) {
    const uint64_t n = src.n_packed + src.n_add + src.n_rem;
    const uint64_t m0 = (1ull << src.B0) - 1ull;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        if (i < src.n_packed) {
            const uint64_t k = src.packed[i];
            out[i] = k == ~0ull ? ~0ull
                                : (pack_duv((uint32_t)(k >> (2 * src.B0)), (uint32_t)((k >> src.B0) & m0),
                                            (uint32_t)(k & m0), pi.B) << 1) | src.packed_op;
            continue;
        }
        const uint32_t op = i < src.n_packed + src.n_add ? 0u : 1u;
        const uint64_t k = op ? src.rem[i - src.n_packed - src.n_add] : src.add[i - src.n_packed];
        uint32_t d, u, v;
        if (pi.pad_ok && k == ~0ull) {
            out[i] = ~0ull;
        } else if (decode_ext(k, pi, d, u, v)) {
            if (op == 0 && u == v) atomicOr(self_seen, 1u);
            out[i] = (pack_duv(d, u, v, pi.B) << 1) | op;
        } else {
            out[i] = ~0ull;
            atomicOr(err, 1u);
        }
    }
}

__global__ void k_pack_delta(const uint64_t* __restrict__ in, uint64_t n, PackInfo pi,
                             uint64_t* __restrict__ out, unsigned int* err, unsigned int* self_seen) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (; i < n; i += stride) {
        uint32_t d, u, v;
        if (decode_ext(in[i], pi, d, u, v)) {
            if (u == v) atomicOr(self_seen, 1u);
            out[i] = pack_duv(d, u, v, pi.B);
        } else {
            out[i] = ~0ull;
            atomicOr(err, 2u);
        }
    }
}

// ---------------------------------------------------------------------------
// fused edit merge of every touched (d, u): lane per run up to kTinyRun merged
// entries, warp per run below kBigRun, longer (hub) runs in tiles, a CTA each
// ---------------------------------------------------------------------------
constexpr uint32_t kTinyRun = 32;        // merged entries up to which one lane merges the run
// Merged entries (old run + edits) from which CTAs merge the run: a warp takes
// about 0.45 us per 32 entries (a chain of two dependent loads), a CTA about
// 3 us for a tile.
constexpr uint32_t kBigRun = 512;
constexpr uint32_t kMergeThreads = 256;
constexpr uint32_t kMergeItems = 11;     // merged entries per thread of a tile; odd: no bank conflicts
constexpr uint32_t kMergeTile = kMergeThreads * kMergeItems;
constexpr uint64_t kTileAggregate = 1ull << 62, kTilePrefix = 2ull << 62, kTileValue = kTileAggregate - 1;  // tile states
constexpr uint32_t kTileSpins = 1u << 24;
constexpr uint32_t kNoVal = 0xffffffffu; // window padding: above every vertex id (< 2^27)

struct MergeArgs {
    uint4* rec;
    uint32_t dvcap;
    uint32_t* pool;
    unsigned long long* pool_top;
    unsigned long long pool_cap;
    long long* live_words;       // sum of round4(len) over runs
    const uint64_t* edits;       // ((d,u,v)<<1|op), each run's edits together and sorted
    uint64_t n;
    uint2* runs[3];              // {first edit, edits} of the runs merged by a warp / in tiles / by a lane (k_edit_runs)
    unsigned int* list_ctr;      // [0] warp, [1] tiled, [2] lane, [4] tiles listed, [5] tiles taken
    unsigned long long* big_off; // tiled runs: where in the pool they go
    uint32_t* big_tile0;         //             their first tile
    uint32_t big_cap;
    uint2* tiles;                // {tiled run, tile of it}, a run's tiles in order
    unsigned long long* tile_state;  // per tile: its count, or the count up to it (zeroed before)
    uint32_t tile_cap;
    uint32_t B;
    unsigned int* err;
    unsigned long long* stats;   // [5] merge bytes (edits 8 B, old run 4 B/word, new run 4 B/word, record 32 B), [6] runs
    // run bit sets: a run that reaches rb_min_len without a bit set claims one
    // (slot table [d][dvcap], slot owners, claim counter, new-slot list)
    uint32_t* rb_slot;           // nullptr: not maintained by this merge
    uint32_t* rb_sel;
    unsigned int* rb_ctr;        // slots claimed
    unsigned int* rb_newc;       // of them by this merge
    uint32_t* rb_new;
    uint32_t rb_cap;
    uint32_t rb_min_len;
};

__device__ __forceinline__ uint32_t round4(uint32_t x) { return (x + 3u) & ~3u; }

// Number of entries of the ascending warp-held window w (lane k holds w[k],
// padded with kNoVal) that are < x (or <= x when le): binary lifting over
// shuffles, six steps.
__device__ __forceinline__ uint32_t win_rank(uint32_t w, uint32_t x, bool le) {
    uint32_t lo = 0;
#pragma unroll
    for (uint32_t step = 16; step >= 1; step >>= 1) {
        const uint32_t v = __shfl_sync(kFull, w, lo + step - 1);
        if (le ? v <= x : v < x) lo += step;
    }
    const uint32_t v = __shfl_sync(kFull, w, lo);
    return lo + ((le ? v <= x : v < x) ? 1u : 0u);
}

// Merge-path split of diagonal k of X (old run) and Y (edits) by one warp: the
// number of X entries among the first k merged entries, X winning ties (so
// for equal values the old entry precedes an add, and an add precedes a
// remove).  32 pivots a round.
__device__ __forceinline__ uint32_t merge_split(const uint32_t* __restrict__ X, uint32_t xl,
                                                const uint64_t* __restrict__ Y, uint32_t yl, uint32_t k,
                                                uint64_t vmask, uint32_t lane) {
    uint32_t lo = k > yl ? k - yl : 0;
    uint32_t hi = k < xl ? k : xl;
    while (hi > lo) {
        const uint32_t n = hi - lo, step = n > 32 ? n >> 5 : 1u;
        const uint32_t p = lo + (lane + 1) * step - 1;
        const bool below = p < hi && __ldg(X + p) <= (uint32_t)((__ldg(Y + (k - 1 - p)) >> 1) & vmask);
        const uint32_t c = __popc(__ballot_sync(kFull, below));
        if (n <= 32) return lo + c;
        const uint32_t base = lo;
        if (c) lo = base + c * step;
        if (c < 32) hi = base + (c + 1) * step - 1;
    }
    return lo;
}

// One window step of a warp merge: the next nout (<= 32) entries of the merge
// of X[i..) and Y[j..), from coalesced 32-entry windows of both.  Lane p
// gets entry p in *val and whether it is emitted: the last entry of its value
// group and not a remove, i.e. the set (X U adds) \ removes.  Advances i, j.
// sbuf: 32 words of this warp's shared memory.
__device__ __forceinline__ bool merge_window(const uint32_t* __restrict__ X, uint32_t xl,
                                             const uint64_t* __restrict__ Y, uint32_t yl, uint64_t vmask,
                                             uint32_t& i, uint32_t& j, uint32_t nout, uint32_t lane,
                                             uint32_t* sbuf, uint32_t& val) {
    const uint32_t xv = (i + lane < xl) ? __ldg(X + i + lane) : kNoVal;
    uint32_t yv = kNoVal, yop = 0;
    if (j + lane < yl) {
        const uint64_t e = __ldg(Y + j + lane);
        yv = (uint32_t)((e >> 1) & vmask);
        yop = (uint32_t)(e & 1ull);
    }
    // merged position: an old entry follows the edits strictly below it, an
    // edit follows the old entries up to and including its value
    const uint32_t px = lane + win_rank(yv, xv, false);
    const uint32_t py = lane + win_rank(xv, yv, true);
    if (px < nout) sbuf[px] = xv;
    if (py < nout) sbuf[py] = yv | (yop << 31);
    const uint32_t cx = __popc(__ballot_sync(kFull, px < nout));
    const uint32_t cy = nout - cx;
    // the entry after the window's last: first unconsumed entry of X or Y
    uint32_t nx = __shfl_sync(kFull, xv, cx & 31), ny = __shfl_sync(kFull, yv, cy & 31);
    if (cx == 32) nx = (i + 32 < xl) ? __ldg(X + i + 32) : kNoVal;
    if (cy == 32) ny = (j + 32 < yl) ? (uint32_t)((__ldg(Y + j + 32) >> 1) & vmask) : kNoVal;
    __syncwarp();
    bool emit = false;
    if (lane < nout) {
        const uint32_t e = sbuf[lane];
        val = e & 0x7fffffffu;
        const uint32_t nv = (lane + 1 < nout) ? (sbuf[lane + 1] & 0x7fffffffu) : min(nx, ny);
        emit = nv != val && !(e >> 31);
    }
    __syncwarp();
    i += cx;
    j += cy;
    return emit;
}

// Pool space for a merged run of at most `bound` entries (~0 when exhausted).
__device__ __forceinline__ unsigned long long pool_alloc(const MergeArgs& a, uint32_t bound) {
    unsigned long long off = atomicAdd(a.pool_top, (unsigned long long)round4(bound));
    if (off + round4(bound) > a.pool_cap) {
        atomicOr(a.err, 4u);
        off = ~0ull;
    }
    return off;
}

// Finds the runs of the edits (an edit whose (d,u) differs from the one before
// starts one; its end is searched by doubling steps) and lists them by merged
// length: one pass over the edits where a run-length encoding, a scan of the
// lengths and a classification took seven launches.  A run's place in its
// list is arbitrary; appends are one atomic per warp and list.
__global__ void k_edit_runs(MergeArgs a) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t vmask = (1ull << a.B) - 1ull;
    const uint32_t sh = a.B + 1;
    for (uint64_t base = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) & ~31ull; base < a.n;
         base += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = base + lane;
        uint32_t cls = 3, len = 0;
        if (i < a.n) {
            const uint64_t e = a.edits[i];
            const uint64_t du = e >> sh;
            if (e != ~0ull && (i == 0 || a.edits[i - 1] >> sh != du)) {
                uint64_t step = 1;
                while (i + step < a.n && a.edits[i + step] >> sh == du) step <<= 1;
                uint64_t lo = i + (step >> 1), hi = min(i + step, a.n);  // in the run / past it
                while (hi - lo > 1) {
                    const uint64_t mid = (lo + hi) >> 1;
                    if (a.edits[mid] >> sh == du) lo = mid; else hi = mid;
                }
                len = (uint32_t)(lo + 1 - i);
                const uint32_t total = a.rec[(size_t)(du >> a.B) * a.dvcap + (du & vmask)].y + len;
                cls = total > kTinyRun ? 0u : 2u;
                if (total >= kBigRun) {
                    // its tiles follow one another in the tile list; a run for which
                    // the lists have no room is left to a warp
                    const uint32_t nt = (total + kMergeTile - 1) / kMergeTile;
                    const uint32_t t0 = atomicAdd(a.list_ctr + 4, nt);
                    uint32_t r = a.big_cap;
                    if (t0 <= a.tile_cap && nt <= a.tile_cap - t0) r = atomicAdd(a.list_ctr + 1, 1u);
                    const bool fits = r < a.big_cap;
                    unsigned long long off = ~0ull;
                    if (fits) {
                        off = pool_alloc(a, total);
                        a.runs[1][r] = make_uint2((uint32_t)i, len);
                        a.big_off[r] = off;
                        a.big_tile0[r] = t0;
                        cls = 3;
                    }
                    for (uint32_t t = 0; t < nt && t0 + t < a.tile_cap; ++t)
                        a.tiles[t0 + t] = make_uint2(off != ~0ull ? r : kNoVal, t);
                }
            }
        }
#pragma unroll
        for (uint32_t k = 0; k < 3; k += 2) {
            const uint32_t bal = __ballot_sync(kFull, cls == k);
            if (!bal) continue;
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(a.list_ctr + k, (uint32_t)__popc(bal));
            at = __shfl_sync(kFull, at, 0);
            if (cls == k) a.runs[k][at + __popc(bal & ((1u << lane) - 1u))] = make_uint2((uint32_t)i, len);
        }
    }
}

// Accounting of the runs one warp merged, added to the launch's counters
// once per warp (per-run atomics on these few words serialised the merge).
struct MergeAcc {
    unsigned long long bytes = 0, runs = 0;
    long long live = 0;
    __device__ __forceinline__ void add(uint32_t xl, uint32_t yl, uint32_t outn) {
        bytes += 8ull * yl + 4ull * xl + 4ull * outn + 32ull;
        runs += 1;
        live += (long long)round4(outn) - (long long)round4(xl);
    }
    // every lane of the warp calls it; lane sums are combined
    __device__ __forceinline__ void flush(const MergeArgs& a, uint32_t lane) {
        for (int o = 16; o > 0; o >>= 1) {
            bytes += __shfl_xor_sync(kFull, bytes, o);
            runs += __shfl_xor_sync(kFull, runs, o);
            live += __shfl_xor_sync(kFull, live, o);
        }
        if (lane == 0) {
            if (bytes) atomicAdd(a.stats + 5, bytes);
            if (runs) atomicAdd(a.stats + 6, runs);
            if (live) atomicAdd((unsigned long long*)a.live_words, (unsigned long long)live);
        }
    }
};

// Record update after a run was merged (one thread); a run that reached the
// bit-set length without a bit set claims one.  The unused tail of the
// allocation is dead space until compaction.
__device__ __forceinline__ void merge_record(const MergeArgs& a, uint4* recp, uint4 old, unsigned long long off,
                                             uint32_t outn, uint32_t d, uint32_t u) {
    *recp = make_uint4((uint32_t)off, outn, old.z, old.w);
    if (a.rb_slot && outn >= a.rb_min_len) {
        uint32_t* sp = a.rb_slot + (size_t)d * a.dvcap + u;
        if (*sp == kNoVal) {
            const unsigned int c = atomicAdd(a.rb_ctr, 1u);
            if (c < a.rb_cap) {
                *sp = c;
                a.rb_sel[c] = d << 27 | u;
                a.rb_new[atomicAdd(a.rb_newc, 1u)] = c;
            }
        }
    }
}

// Lane per run for runs of at most kTinyRun merged entries (most runs of a
// batch touch a handful of entries): a serial merge per lane, one pool
// allocation per warp step (a warp prefix over the lanes' bounds).
__device__ __forceinline__ void merge_tiny(const MergeArgs& a, MergeAcc& acc) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t n = a.list_ctr[2];
    const uint64_t emask = (1ull << a.B) - 1ull;
    const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t base = gw * 32; base < n; base += nw * 32) {
        const uint32_t q = base + lane;
        const bool on = q < n;
        uint32_t d = 0, u = 0, yl = 0, y0 = 0;
        uint4 old = make_uint4(0, 0, 0, 0);
        uint4* recp = nullptr;
        if (on) {
            const uint2 r = a.runs[2][q];
            const uint64_t du = a.edits[r.x] >> (a.B + 1);
            d = (uint32_t)(du >> a.B);
            u = (uint32_t)(du & emask);
            y0 = r.x;
            yl = r.y;
            recp = a.rec + (size_t)d * a.dvcap + u;
            old = *recp;
        }
        const uint32_t bound = on ? round4(old.y + yl) : 0u;
        uint32_t pre = bound;  // inclusive prefix over the lanes
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(kFull, pre, o);
            if (lane >= (uint32_t)o) pre += v;
        }
        const uint32_t total = __shfl_sync(kFull, pre, 31);
        unsigned long long wbase = 0;
        if (lane == 0 && total) {
            wbase = atomicAdd(a.pool_top, (unsigned long long)total);
            if (wbase + total > a.pool_cap) {
                atomicOr(a.err, 4u);
                wbase = ~0ull;
            }
        }
        wbase = __shfl_sync(kFull, wbase, 0);
        if (!on || wbase == ~0ull) continue;  // pool exhausted: runs left unchanged, error raised
        const unsigned long long off = wbase + pre - bound;
        const uint32_t* X = a.pool + old.x;
        const uint64_t* Y = a.edits + y0;
        uint32_t* C = a.pool + off;
        uint32_t i = 0, j = 0, outn = 0;
        while (i < old.y || j < yl) {
            const uint32_t xv = i < old.y ? X[i] : kNoVal;
            const uint32_t yv = j < yl ? (uint32_t)((Y[j] >> 1) & emask) : kNoVal;
            const uint32_t v = min(xv, yv);
            bool present = false;
            if (xv == v) { present = true; ++i; }
            // the value's edits in order (adds before removes): the last decides
            while (j < yl && (uint32_t)((Y[j] >> 1) & emask) == v) { present = (Y[j] & 1ull) == 0; ++j; }
            if (present) C[outn++] = v;
        }
        merge_record(a, recp, old, off, outn, d, u);
        acc.add(old.y, yl, outn);
    }
}

// Warp per run: 32 merged entries per step from two coalesced windows.
__device__ __forceinline__ void merge_small(const MergeArgs& a, MergeAcc& acc, uint32_t* sbuf) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    const uint32_t nruns = a.list_ctr[0];
    const uint64_t vmask = (1ull << a.B) - 1ull;
    for (uint32_t q = gw; q < nruns; q += nw) {
        const uint2 r = a.runs[0][q];
        const uint64_t* Y = a.edits + r.x;
        const uint32_t yl = r.y;
        const uint64_t du = *Y >> (a.B + 1);
        const uint32_t d = (uint32_t)(du >> a.B), u = (uint32_t)(du & vmask);
        uint4* recp = a.rec + (size_t)d * a.dvcap + u;
        const uint4 old = *recp;
        const uint32_t* X = a.pool + old.x;
        const uint32_t xl = old.y;
        unsigned long long off = 0;
        if (lane == 0) off = pool_alloc(a, xl + yl);
        off = __shfl_sync(kFull, off, 0);
        if (off == ~0ull) continue;  // pool exhausted: run left unchanged, error raised
        uint32_t* C = a.pool + off;
        const uint32_t total = xl + yl;
        uint32_t outn = 0, i = 0, j = 0;
        for (uint32_t done = 0; done < total; done += 32) {
            const uint32_t nout = min(32u, total - done);
            uint32_t val = 0;
            const bool emit = merge_window(X, xl, Y, yl, vmask, i, j, nout, lane, sbuf, val);
            const uint32_t bal = __ballot_sync(kFull, emit);
            if (emit) C[outn + __popc(bal & ((1u << lane) - 1u))] = val;
            outn += __popc(bal);
        }
        if (lane == 0) {
            merge_record(a, recp, old, off, outn, d, u);
            acc.add(xl, yl, outn);
        }
    }
}

// Long runs, a tile of kMergeTile merged entries per CTA and step: the tile's
// part of X and Y staged in shared memory by coalesced loads, merged serially
// by each thread (kMergeItems entries), compacted, and written as one stretch
// behind the run's earlier tiles (their states; tiles are taken in list order,
// so every earlier one is done or running).  The run's last tile writes its
// record: by then every earlier tile has read the old one.
// One CTA per run and 2,048 entries per round (eight dependent windows a warp)
// took 98 us for the R-MAT 4M/34M tree's batch.
struct TileMem {
    uint32_t e[kMergeTile];  // [0, nx): X (value << 1), [nx, nt): Y (value << 1 | op); then the output
    uint32_t split[3];       // X entries before the tile, before its end; value after the tile
    uint32_t take;
    uint32_t base;
    typename cub::BlockScan<uint32_t, kMergeThreads>::TempStorage scan;
};
__device__ __forceinline__ void merge_tiles(const MergeArgs& a, MergeAcc& acc, TileMem& sm) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t ntiles = min(a.list_ctr[4], a.tile_cap);
    const uint64_t vmask = (1ull << a.B) - 1ull;
    for (;;) {
        __syncthreads();  // the previous tile's output has been written
        if (threadIdx.x == 0) sm.take = atomicAdd(a.list_ctr + 5, 1u);
        __syncthreads();
        const uint32_t ti = sm.take;
        if (ti >= ntiles) break;
        const uint2 tl = a.tiles[ti];
        if (tl.x == kNoVal) continue;  // no room for the run (error raised, run left unchanged) or merged by a warp
        const uint2 r = a.runs[1][tl.x];
        const uint32_t t0 = a.big_tile0[tl.x];
        const unsigned long long off = a.big_off[tl.x];
        const uint64_t* Y = a.edits + r.x;
        const uint32_t yl = r.y;
        const uint64_t du = *Y >> (a.B + 1);
        const uint32_t d = (uint32_t)(du >> a.B), u = (uint32_t)(du & vmask);
        uint4* recp = a.rec + (size_t)d * a.dvcap + u;
        const uint4 old = *recp;
        const uint32_t* X = a.pool + old.x;
        const uint32_t xl = old.y, total = xl + yl;
        const uint32_t k0 = tl.y * kMergeTile, k1 = min(k0 + kMergeTile, total), nt = k1 - k0;
        if (threadIdx.x < 32) {
            const uint32_t i0 = merge_split(X, xl, Y, yl, k0, vmask, lane);
            if (lane == 0) sm.split[0] = i0;
        } else if (threadIdx.x < 64) {
            const uint32_t i1 = merge_split(X, xl, Y, yl, k1, vmask, lane);
            if (lane == 0) {
                sm.split[1] = i1;
                uint32_t nxt = kNoVal;
                if (i1 < xl) nxt = __ldg(X + i1);
                if (k1 - i1 < yl) nxt = min(nxt, (uint32_t)((__ldg(Y + (k1 - i1)) >> 1) & vmask));
                sm.split[2] = nxt;
            }
        }
        __syncthreads();
        const uint32_t i0 = sm.split[0], nx = sm.split[1] - i0, ny = nt - nx, j0 = k0 - i0, after = sm.split[2];
        for (uint32_t t = threadIdx.x; t < nt; t += kMergeThreads) {
            uint32_t e;
            if (t < nx) {
                e = __ldg(X + i0 + t) << 1;
            } else {
                const uint64_t y = __ldg(Y + j0 + (t - nx));
                e = (uint32_t)((y >> 1) & vmask) << 1 | (uint32_t)(y & 1ull);
            }
            sm.e[t] = e;
        }
        __syncthreads();
        const uint32_t* sx = sm.e;
        const uint32_t* sy = sm.e + nx;
        const uint32_t a0 = min(threadIdx.x * kMergeItems, nt), a1 = min(a0 + kMergeItems, nt);
        uint32_t lo = a0 > ny ? a0 - ny : 0, hi = min(a0, nx);
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (sx[mid] <= (sy[a0 - 1 - mid] | 1u)) lo = mid + 1;  // by value, X first
            else hi = mid;
        }
        uint32_t i = lo, j = a0 - lo;
        uint32_t val[kMergeItems + 1];
#pragma unroll
        for (uint32_t q = 0; q <= kMergeItems; ++q) {
            if (a0 + q < a1 || (a0 + q == a1 && a1 < nt && a0 < a1)) {
                const bool fx = i < nx && (j >= ny || sx[i] <= (sy[j] | 1u));
                val[q] = fx ? sx[i] : sy[j];
                i += fx ? 1u : 0u;
                j += fx ? 0u : 1u;
            } else {
                val[q] = a0 + q == nt ? after << 1 : kNoVal;
            }
        }
        uint32_t emit = 0;
#pragma unroll
        for (uint32_t q = 0; q < kMergeItems; ++q)
            if (a0 + q < a1 && (val[q] >> 1) != (val[q + 1] >> 1) && !(val[q] & 1u)) emit |= 1u << q;
        uint32_t before = 0, all = 0;
        cub::BlockScan<uint32_t, kMergeThreads>(sm.scan).ExclusiveSum((uint32_t)__popc(emit), before, all);
        if (threadIdx.x < 32) {
            unsigned long long base = 0;
            if (tl.y) {
                if (lane == 0) atomicExch(a.tile_state + ti, kTileAggregate | all);
                int at = (int)(ti - 1);
                bool gave_up = false;
                for (;;) {
                    unsigned long long v = kTilePrefix;  // before the run's first tile: 0
                    if (at - (int)lane >= (int)t0) {
                        uint32_t spins = 0;
                        while ((v = *(volatile unsigned long long*)(a.tile_state + at - lane)) == 0 && ++spins < kTileSpins)
                            __nanosleep(20);
                    }
                    if (__any_sync(kFull, v == 0)) { gave_up = true; break; }
                    const uint32_t pre = __ballot_sync(kFull, (v & kTilePrefix) != 0);
                    const uint32_t last = pre ? __ffs(pre) - 1 : 31;
                    unsigned long long c = lane <= last ? (v & kTileValue) : 0ull;
                    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(kFull, c, o);
                    base += c;
                    if (pre) break;
                    at -= 32;
                }
                if (gave_up && lane == 0) atomicOr(a.err, 16u);
            }
            if (lane == 0) {
                atomicExch(a.tile_state + ti, kTilePrefix | (base + all));
                sm.base = (uint32_t)base;
                if (k1 == total) {
                    merge_record(a, recp, old, off, (uint32_t)base + all, d, u);
                    acc.add(xl, yl, (uint32_t)base + all);
                }
            }
        }
        __syncthreads();  // every entry of the tile is in registers: its memory takes the output
#pragma unroll
        for (uint32_t q = 0; q < kMergeItems; ++q)
            if ((emit >> q) & 1u) sm.e[before++] = val[q] >> 1;
        __syncthreads();
        uint32_t* C = a.pool + off + sm.base;
        for (uint32_t t = threadIdx.x; t < all; t += kMergeThreads) C[t] = sm.e[t];
    }
}

// Every listed run in one launch: each block takes tiles of the hub runs first
// (they take longest), then its share of the warp's and the lane's runs.
__global__ void __launch_bounds__(kMergeThreads) k_merge(MergeArgs a) {
    __shared__ TileMem sm;
    MergeAcc acc;
    merge_tiles(a, acc, sm);
    __syncthreads();
    merge_small(a, acc, sm.e + 32 * (threadIdx.x >> 5));
    merge_tiny(a, acc);
    acc.flush(a, threadIdx.x & 31);
}

// ---------------------------------------------------------------------------
// delta lists
// ---------------------------------------------------------------------------
// From the sorted packed keys ((d << lb | label bits) << 2B | u << B | v; lb =
// 0: no label bits): the delta values, and {offset, length} of every (d,u)'s
// stretch in its record, found as in k_edit_runs.  n keys, of which *nsel are
// real when given (the others become all-ones padding).
// clear: only takes the records' delta fields back to empty.
__device__ __forceinline__ void delta_lists(uint64_t* keys, uint64_t n, const int* nsel, uint32_t B, uint32_t lb,
                                            uint4* rec, uint32_t dvcap, uint32_t* __restrict__ dval, bool clear,
                                            uint32_t block, uint32_t blocks) {
    const uint64_t real = nsel ? (uint64_t)*nsel : n;
    const uint64_t vmask = (1ull << B) - 1ull;
    for (uint64_t i = (uint64_t)block * blockDim.x + threadIdx.x; i < (clear ? real : n);
         i += (uint64_t)blocks * blockDim.x) {
        if (i >= real) {
            keys[i] = ~0ull;
            continue;
        }
        const uint64_t k = keys[i];
        if (!clear) dval[i] = (uint32_t)(k & vmask);
        if (k == ~0ull) continue;
        const uint64_t du = k >> B;
        if (i > 0 && keys[i - 1] >> B == du) continue;
        uint2 f = make_uint2(0, 0);
        if (!clear) {
            uint64_t step = 1;
            while (i + step < real && keys[i + step] >> B == du) step <<= 1;
            uint64_t lo = i + (step >> 1), hi = min(i + step, real);
            while (hi - lo > 1) {
                const uint64_t mid = (lo + hi) >> 1;
                if (keys[mid] >> B == du) lo = mid; else hi = mid;
            }
            f = make_uint2((uint32_t)i, (uint32_t)(lo + 1 - i));
        }
        reinterpret_cast<uint2*>(rec + (size_t)(k >> (2 * B + lb)) * dvcap + (du & vmask))[1] = f;
    }
}
__global__ void k_delta_lists(uint64_t* keys, uint64_t n, const int* nsel, uint32_t B, uint32_t lb, uint4* rec,
                              uint32_t dvcap, uint32_t* dval, int clear) {
    delta_lists(keys, n, nsel, B, lb, rec, dvcap, dval, clear != 0, blockIdx.x, gridDim.x);
}

// Delta lists of the single-query engine and, in the last block, its seed
// ranges: the delta entries of direction seed_dir(ei) form one contiguous
// range of the sorted packed delta array.  One thread per range end (six per
// query edge: the searches are chains of dependent loads).
__global__ void __launch_bounds__(256) k_delta(uint64_t* dkeys, uint64_t n, uint32_t B, uint4* rec, uint32_t dvcap,
                                               uint32_t* dval, uint32_t qe, const EdgePlan* __restrict__ plans,
                                               const uint8_t* qe_dirs /*[qe][2]*/, const uint8_t* edge_ok, int have_ok,
                                               uint32_t* seed_lo, uint32_t* seed_pre) {
    if (blockIdx.x + 1 < gridDim.x) {
        delta_lists(dkeys, n, nullptr, B, 0, rec, dvcap, dval, false, blockIdx.x, gridDim.x - 1);
        return;
    }
    static_assert(cgb::kMaxQEKeyed * 6 <= 256, "one thread per range end");
    __shared__ uint32_t s_at[cgb::kMaxQEKeyed][6];
    __shared__ uint32_t s_cnt[cgb::kMaxQEKeyed];
    const uint32_t t = threadIdx.x / 6, w = threadIdx.x % 6;
    if (t < qe) {
        const uint32_t d = w < 2 ? plans[t].seed_dir : qe_dirs[2 * t + (w < 4 ? 0 : 1)];
        const uint64_t key = (uint64_t)(d + (w & 1u)) << (2 * B);
        uint64_t lo = 0, hi = n;
        while (lo < hi) {
            const uint64_t mid = (lo + hi) >> 1;
            if (dkeys[mid] < key) lo = mid + 1; else hi = mid;
        }
        s_at[t][w] = (uint32_t)lo;
    }
    __syncthreads();
    if (threadIdx.x < qe) {
        const uint32_t* p = s_at[threadIdx.x];
        const bool ok = have_ok ? edge_ok[threadIdx.x] != 0 : p[3] > p[2] && p[5] > p[4];
        seed_lo[threadIdx.x] = p[0];
        s_cnt[threadIdx.x] = ok ? p[1] - p[0] : 0;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t acc = 0;
        for (uint32_t e = 0; e < qe; ++e) { seed_pre[e] = acc; acc += s_cnt[e]; }
        seed_pre[qe] = acc;
    }
}

// ---------------------------------------------------------------------------
// run bit sets: every old run of at least kRunBitsMinLen entries is also kept
// as a bit set over the compressed ids, rebuilt each batch after the index
// update, so that a membership test in a long (hub) run, in the DFS probes
// and in the tail counts, is one load instead of a binary search
// ---------------------------------------------------------------------------
constexpr uint32_t kNoSlot = 0xffffffffu;
constexpr uint32_t kRunBitsMinLen = 128;        // $CGB_RUN_BITS_MIN_LEN overrides (tests use 1)
constexpr size_t kRunBitsBytes = 512ull << 20;  // runs beyond this budget are searched

// Full rebuild: the slot of every (direction, vertex) of the table (all
// dvcap rows) whose run is long enough, in claim order while slots last
// (ctr[0] counts claims), else kNoSlot; sel[slot] = dir << 27 | vertex.
// Afterwards each merge keeps the sets current (k_rb_update).
__global__ void k_rb_select(const uint4* __restrict__ rec, uint32_t dvcap, uint32_t nd, uint32_t min_len,
                            uint32_t cap, uint32_t* slot, uint32_t* sel, unsigned int* ctr) {
    const size_t n = (size_t)nd * dvcap;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        uint32_t sl = kNoSlot;
        if (rec[i].y >= min_len) {
            const unsigned int c = atomicAdd(ctr, 1u);
            if (c < cap) {
                sl = c;
                sel[c] = (uint32_t)(i / dvcap) << 27 | (uint32_t)(i % dvcap);
            }
        }
        slot[i] = sl;
    }
}

__global__ void k_rb_zero(uint32_t* bits, uint32_t words, uint32_t cap, const unsigned int* ctr) {
    const size_t n = (size_t)min(*ctr, cap) * words;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        bits[i] = 0;
}

// one warp per selected run: the bits of its words, set with atomicOr
// (lanes can share a word)
__global__ void k_rb_fill(const uint4* __restrict__ rec, uint32_t dvcap, const uint32_t* __restrict__ pool,
                          const uint32_t* __restrict__ sel, uint32_t cap, const unsigned int* ctr, uint32_t* bits,
                          uint32_t words) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t nsel = min(*ctr, cap);
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < nsel; c += nw) {
        const uint32_t du = sel[c];
        const uint4 r = rec[(size_t)(du >> 27) * dvcap + (du & ((1u << 27) - 1u))];
        uint32_t* b = bits + (size_t)c * words;
        for (uint32_t t = lane; t < r.y; t += 32) {
            const uint32_t v = __ldg(pool + r.x + t);
            atomicOr(b + (v >> 5), 1u << (v & 31));
        }
    }
}

// After a merge: slots claimed by runs that grew past the length threshold
// (*newc of them, listed in fresh) are zeroed and filled from the merged run,
// a warp each; and the merge's edits ((d,u,v) << 1 | op, each run's sorted) are
// applied to every bit set: the last edit of each (d,u,v) decides, as in the
// merge (an add sets the bit, a remove clears it).  Both may meet in a fresh
// set in any order: the fill sets exactly the merged run's bits, an added value
// is in it and a removed one is not.
__global__ void k_rb_update(const uint4* __restrict__ rec, uint32_t dvcap, const uint32_t* __restrict__ pool,
                            const uint32_t* __restrict__ sel, const uint32_t* __restrict__ fresh,
                            const unsigned int* newc, uint32_t* bits, uint32_t words,
                            const uint64_t* __restrict__ edits, uint64_t n, uint32_t B,
                            const uint32_t* __restrict__ slot) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t nnew = *newc;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < nnew; q += nw) {
        const uint32_t c = fresh[q];
        const uint32_t du = sel[c];
        const uint4 r = rec[(size_t)(du >> 27) * dvcap + (du & ((1u << 27) - 1u))];
        uint32_t* b = bits + (size_t)c * words;
        for (uint32_t t = lane; t < words; t += 32) atomicExch(b + t, 0u);
        __threadfence();
        __syncwarp();
        for (uint32_t t = lane; t < r.y; t += 32) {
            const uint32_t v = __ldg(pool + r.x + t);
            atomicOr(b + (v >> 5), 1u << (v & 31));
        }
    }
    const uint64_t vmask = (1ull << B) - 1ull;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t e = edits[i];
        if (e == ~0ull) continue;
        if (i + 1 < n && (edits[i + 1] >> 1) == (e >> 1)) continue;  // not the last edit of its value
        const uint64_t p = e >> 1;
        const uint32_t v = (uint32_t)(p & vmask), u = (uint32_t)((p >> B) & vmask), d = (uint32_t)(p >> (2 * B));
        const uint32_t sl = slot[(size_t)d * dvcap + u];
        if (sl == kNoSlot) continue;
        uint32_t* w = bits + (size_t)sl * words + (v >> 5);
        if (e & 1ull) atomicAnd(w, ~(1u << (v & 31)));
        else atomicOr(w, 1u << (v & 31));
    }
}

// Index symmetry: number of entries y in run (d, x) whose mirror entry (x in
// run (rev[d], y)) is missing.  Warp per run.
__global__ void k_asymmetry(const uint4* __restrict__ rec, uint32_t dvcap, uint32_t dv, uint32_t nd,
                            const uint32_t* __restrict__ pool, const uint8_t* __restrict__ rev,
                            unsigned long long* bad) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t total = (uint64_t)nd * dv;
    unsigned long long miss = 0;
    for (uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < total;
         i += ((uint64_t)gridDim.x * blockDim.x) >> 5) {
        const uint32_t d = (uint32_t)(i / dv), x = (uint32_t)(i % dv);
        const uint4 r = rec[(size_t)d * dvcap + x];
        const uint32_t rd = rev[d];
        for (uint32_t t = lane; t < r.y; t += 32) {
            const uint32_t y = pool[r.x + t];
            bool ok = false;
            if (y < dv && rd < nd) {
                const uint4 m = rec[(size_t)rd * dvcap + y];
                uint32_t lo = 0, hi = m.y;
                while (lo < hi) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (pool[m.x + mid] < x) lo = mid + 1; else hi = mid;
                }
                ok = lo < m.y && pool[m.x + lo] == x;
            }
            miss += ok ? 0 : 1;
        }
    }
    for (int o = 16; o > 0; o >>= 1) miss += __shfl_xor_sync(kFull, miss, o);
    if (lane == 0 && miss) atomicAdd(bad, miss);
}

// ---------------------------------------------------------------------------
// persistent warp DFS (count only)
// ---------------------------------------------------------------------------
// DFS queue counters (words), on 128-byte lines by who looks at them: tasks and
// tickets (every donor), finished units (every waiting block), and what only
// those that add to it touch
constexpr uint32_t kQReserved = 0, kQTickets = 1, kQDone = 32, kQMemo = 64, kQBusy = 66, kQWords = 96;
static_assert(kQDone / 32 != kQReserved / 32 && kQDone / 32 != kQMemo / 32 && kQMemo / 32 != kQReserved / 32 &&
                  kQBusy % 2 == 0 && kQBusy + 2 <= kQWords,
              "polled counters share no line with others; kQBusy holds 64 bits");
struct DfsArgs {
    const uint4* rec;
    uint32_t dvcap;
    const uint32_t* pool;
    const uint32_t* dval;
    const uint64_t* dkeys;
    uint32_t B;
    uint32_t qe;
    const uint32_t* seed_lo;
    const uint32_t* seed_pre;
    unsigned long long* counts;  // [qe]
    unsigned int* work_next;     // [0] seeds claimed behind the rows, [1] rows of seeds taken (seed_claim.h)
    unsigned int* err;
    unsigned long long* stats;   // [8]: seeds, chunks, tested, tails, algorithmic bytes read, .., .., stolen tasks
    unsigned long long budget_ns;  // per-launch wall-clock budget (0 = unlimited)
    uint32_t* tasks;             // stolen-range queue [task_cap][16 words]
    uint32_t task_cap;
    unsigned int* qctr;          // [kQWords]: kQReserved, kQTickets, kQDone
    uint32_t epoch;              // per-launch tag written as a task's ready flag (never 0)
    uint32_t force_split;        // publish unstarted work at every chunk, waited for or not (tests)
    uint32_t shard, num_shards;  // this engine expands the seed groups whose key hashes to shard (seed_shard)
    uint32_t steal;              // share long shallow ranges through the queue
    uint32_t tail_cache;         // count prefix-only tail subsets once per prefix
    const unsigned int* self_seen;  // sticky self-loop flag (see k_pack_edits)
    const uint32_t* vb;          // valid bits [qe][qv][vb_stride] or nullptr (no pruning)
    uint32_t vb_stride;
    uint32_t qv;
    const uint32_t* rb_slot;     // run bit sets: slot of (dir, vertex) [nd][dvcap] or nullptr (none)
    const uint32_t* rb_bits;     // [slot][rb_words]
    uint32_t rb_words;
    const EdgePlan* plans;       // [qe] (k_dfs_count<true>: every registered query's plans)
    const unsigned int* epoch_ptr;  // non-null: the launch tag is read here (k_epoch_bump)
    uint32_t* touched;           // footprint runs: bit per record resolved (nullptr: off)
    unsigned long long* lsum_tab;  // level-sum table [lsum_mask + 1][2], zeroed before the launch (nullptr: none)
    uint32_t lsum_mask;
    unsigned long long* memo_tab;  // subtree memos [memo_mask + 1][4], empty before and after a launch (nullptr: none)
    uint32_t memo_mask;
    uint32_t* memo_list;           // claimed slots (their number at kQMemo)
    const unsigned long long* wsum;  // dense level sums [array][dvcap] (nullptr: none)
    uint32_t pair_lane_max;      // pair counting: longest shorter list a lane scans alone
};

// Footprint of a matching launch: the bytes of every distinct record it
// resolved (16 B) and of that record's whole old and delta lists (4 B per
// entry), each counted once.  Added to *out.
__global__ void k_footprint(const uint4* __restrict__ rec, uint64_t n, const uint32_t* __restrict__ touched,
                            unsigned long long* out) {
    unsigned long long b = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        if ((touched[i >> 5] >> (i & 31)) & 1u) {
            const uint4 r = rec[i];
            b += 16ull + 4ull * ((unsigned long long)r.y + r.w);
        }
    for (int o = 16; o > 0; o >>= 1) b += __shfl_xor_sync(kFull, b, o);
    if ((threadIdx.x & 31) == 0 && b) atomicAdd(out, b);
}

// Next launch tag for a DFS launch that reads it from memory; the low 20
// bits (the tag's epoch field) are never 0.
__global__ void k_epoch_bump(unsigned int* e) {
    unsigned int v = *e + 1;
    if ((v & 0xfffffu) == 0) ++v;
    *e = v;
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Resolved candidate list of one (direction, vertex): the old run (pool) and,
// when visible, this batch's delta run (dval); the two are disjoint.
struct ListRef {
    const uint32_t* m;
    uint32_t ml;
    const uint32_t* d;
    uint32_t dl;
};

// Membership in the ascending p[0..n): halves the range with a select
// instead of a branch, so the trip count is ceil(log2 n) for every x.
// Invariant: if x is present it lies in [p, p + n).
__device__ __forceinline__ bool sorted_has_bl(const uint32_t* __restrict__ p, uint32_t n, uint32_t x) {
    if (n == 0) return false;
    while (n > 1) {
        const uint32_t half = n >> 1;
        p = (__ldg(p + half) <= x) ? p + half : p;
        n -= half;
    }
    return __ldg(p) == x;
}

__device__ __forceinline__ bool list_contains(const uint32_t* __restrict__ pool, const uint32_t* __restrict__ dval,
                                              const uint4& r, uint32_t x) {
    return sorted_has_bl(pool + r.x, r.y, x) || (r.w && sorted_has_bl(dval + r.z, r.w, x));
}

// Bit sets of the long old runs (rebuilt each batch): slot[(dir, vertex)]
// names a bit set over the compressed ids, or kNoSlot; a warp keeps the slot
// of every resolved record bn[k] in bslot[k].  slot == nullptr: none.
struct RunBits {
    const uint32_t* slot;
    const uint32_t* bits;
    uint32_t words;
    uint32_t* bslot;
    __device__ __forceinline__ void note(uint32_t k, size_t at) const {
        if (slot) bslot[k] = __ldg(slot + at);
    }
    // a lane's own record (not kept in bslot): nothing to note here
    __device__ __forceinline__ void touch(size_t) const {}
    __device__ __forceinline__ uint32_t slot_at(size_t at) const { return slot ? __ldg(slot + at) : kNoSlot; }
    // x in the list r whose old run has the bit set sl: one bit test for a long old run
    __device__ __forceinline__ bool has_slot(uint32_t sl, const uint4& r, const uint32_t* __restrict__ pool,
                                            const uint32_t* __restrict__ dval, uint32_t x) const {
        if (sl != kNoSlot) {
            if ((__ldg(bits + (size_t)sl * words + (x >> 5)) >> (x & 31)) & 1u) return true;
            return r.w && sorted_has_bl(dval + r.z, r.w, x);
        }
        return list_contains(pool, dval, r, x);
    }
    // x in the resolved list bn[k] = r
    __device__ __forceinline__ bool has(uint32_t k, const uint4& r, const uint32_t* __restrict__ pool,
                                       const uint32_t* __restrict__ dval, uint32_t x) const {
        return has_slot(slot ? bslot[k] : kNoSlot, r, pool, dval, x);
    }
};

// Footprint runs (a separate instantiation of the DFS, so that the timed
// kernel carries no trace of it): also sets the bit of every record resolved
// in touched (one bit per record).
struct RunBitsCount : RunBits {
    uint32_t* touched;
    __device__ __forceinline__ void note(uint32_t k, size_t at) const {
        RunBits::note(k, at);
        touch(at);
    }
    __device__ __forceinline__ void touch(size_t at) const { atomicOr(touched + (at >> 5), 1u << (at & 31)); }
};


// Tail counts (EdgePlan's subsets).  At the position being evaluated the prefix
// is fixed: a subset whose lists all hang off it has one count per prefix
// (s_tc), recounted only when a position it reads changed since (`dirty`, the
// shallowest position whose vertex changed; kClean: none); the others are
// counted per candidate, one lane each.
constexpr uint32_t kPairLaneMax = 0xffffffffu;  // pair counting: longest shorter list counted per lane ($CGB_PAIR_LANE_MAX)
constexpr uint32_t kClean = 0xffu;
constexpr uint32_t kNoPos = 0xffffffffu;

// Product of the lengths of c's own lists towards the tail vertices in
// sum_tails (1 when there are none): the weight of c in a level sum.
template <class RB>
__device__ __forceinline__ unsigned long long sum_lens(const EdgePlan& P, const uint4* __restrict__ rec,
                                                       uint32_t dvcap, uint32_t c, const RB& rb) {
    unsigned long long v = 1;
    for (uint32_t b = P.sum_tails; b; b &= b - 1) {
        const uint32_t q = P.bn_off[__ffs(b) - 1];
        const size_t at = (size_t)P.bn_dir[q] * dvcap + c;
        uint4 r = rec[at];
        if (!P.bn_dvis[q]) r.w = 0;
        rb.touch(at);
        v *= (unsigned long long)r.y + r.w;
    }
    return v;
}

// One value per lane with `on`, for its own candidate c at position d, over the
// lists of one subset (bits of `lists`, bn index sub_base + bit).  Lists of
// positions below d hang off the prefix (resolved in bn, the same for every
// lane); the others are c's own (their record is read here).
//   !sum: the number of x in every list with x not among the vertices matched
//         at the positions in ex (position d holds c);
//   sum:  the sum of sum_lens(x) over the one list.
// The lanes' shortest lists are laid end to end and walked 32 entries at a
// time by the whole warp, each entry with its owner's c (binary lifting over
// the prefix sums): a walk takes ceil(total / 32) steps whatever the lists'
// lengths, where one candidate at a time leaves most lanes idle (lists of a
// handful of entries) and one lane per candidate waits for the longest list.
template <class RB>
__device__ __forceinline__ unsigned long long flat_lists(const EdgePlan& P, uint32_t lists, uint32_t d, bool sum,
                                                         bool on, uint32_t c, uint32_t ex, const uint32_t* m,
                                                         const uint4* bn, const uint4* __restrict__ rec,
                                                         uint32_t dvcap, const uint32_t* __restrict__ pool,
                                                         const uint32_t* __restrict__ dval, uint32_t lane,
                                                         uint32_t& n_words, const RB& rb) {
    // this lane's shortest list: record fields x, y, z, length, bn index
    uint32_t gx = 0, gy = 0, gz = 0, glen = 0xffffffffu, gq = 0;
    for (uint32_t b = lists; b; b &= b - 1) {
        const uint32_t q = P.sub_base + __ffs(b) - 1;
        uint4 r = make_uint4(0, 0, 0, 0);
        if (P.bn_pos[q] < d) {
            r = bn[q];
        } else if (on) {
            const size_t at = (size_t)P.bn_dir[q] * dvcap + c;
            r = rec[at];
            if (!P.bn_dvis[q]) r.w = 0;
            rb.touch(at);
            n_words += 4;
        }
        if (r.y + r.w < glen) {
            glen = r.y + r.w;
            gx = r.x; gy = r.y; gz = r.z; gq = q;
        }
    }
    if (!on) glen = 0;
    unsigned long long res = 0;
    // 32 lists of at most 2^26 entries fit a 32-bit position; longer ones go one lane at a time
    uint32_t todo = __ballot_sync(kFull, glen != 0);
    const bool huge = __reduce_max_sync(kFull, glen) > (1u << 26);
    while (todo) {
        const uint32_t part = huge ? (todo & (0u - todo)) : todo;
        todo &= ~part;
        const uint32_t len = ((part >> lane) & 1u) ? glen : 0u;
        uint32_t incl = len;  // prefix sums of the lanes' lengths
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(kFull, incl, o);
            if (lane >= (uint32_t)o) incl += v;
        }
        const uint32_t total = __shfl_sync(kFull, incl, 31);
        const uint32_t first = incl - len;
        for (uint32_t b0 = 0; b0 < total; b0 += 32) {
            const uint32_t i = b0 + lane;
            uint32_t o = 0;  // owner of entry i: the number of lanes whose lists end at or before i
#pragma unroll
            for (uint32_t step = 16; step >= 1; step >>= 1)
                if (__shfl_sync(kFull, incl, o + step - 1) <= i) o += step;
            const uint32_t off = i - __shfl_sync(kFull, first, o);
            const uint32_t ox = __shfl_sync(kFull, gx, o), oy = __shfl_sync(kFull, gy, o);
            const uint32_t oz = __shfl_sync(kFull, gz, o);
            const uint32_t oc = __shfl_sync(kFull, c, o), oq = __shfl_sync(kFull, gq, o);
            bool ok = i < total;
            uint32_t x = 0;
            if (ok) {
                x = off < oy ? __ldg(pool + ox + off) : __ldg(dval + oz + (off - oy));
                n_words += 1;
            }
            if (sum) {
                unsigned long long v = ok ? sum_lens(P, rec, dvcap, x, rb) : 0ull;
                // inclusive sums within each owner's stretch, read at its last entry here
#pragma unroll
                for (int s = 1; s < 32; s <<= 1) {
                    const unsigned long long u = __shfl_up_sync(kFull, v, s);
                    const uint32_t uo = __shfl_up_sync(kFull, o, s);
                    if (lane >= (uint32_t)s && uo == o) v += u;
                }
                const bool any = len && first < b0 + 32u && incl > b0;
                const unsigned long long got = __shfl_sync(kFull, v, any ? min(incl - b0, 32u) - 1u : 0u);
                if (any) res += got;
            } else {
                if (ok) {
                    for (uint32_t e = ex; e; e &= e - 1) {
                        const uint32_t t = __ffs(e) - 1;
                        ok &= x != (t == d ? oc : m[t]);
                    }
                    for (uint32_t b = lists; b && ok; b &= b - 1) {
                        const uint32_t q = P.sub_base + __ffs(b) - 1;
                        if (q == oq) continue;
                        uint4 r;
                        uint32_t sl;
                        if (P.bn_pos[q] < d) {
                            r = bn[q];
                            sl = rb.slot ? rb.bslot[q] : kNoSlot;
                        } else {
                            const size_t at = (size_t)P.bn_dir[q] * dvcap + oc;
                            r = rec[at];
                            if (!P.bn_dvis[q]) r.w = 0;
                            sl = rb.slot_at(at);
                        }
                        n_words += 8u * (33u - __clz(r.y | 1u));
                        ok = rb.has_slot(sl, r, pool, dval, x);
                    }
                }
                const uint32_t bal = __ballot_sync(kFull, ok);
                if (len && first < b0 + 32u && incl > b0) {
                    const uint32_t lo = first > b0 ? first - b0 : 0u, hi = min(incl - b0, 32u);
                    res += __popc(bal >> lo & (0xffffffffu >> (32u - (hi - lo))));
                }
            }
        }
    }
    return res;
}

// Level-sum table: slots of {key, value}; key 0 = empty, K << 1 = claimed
// by a warp computing the value, K << 1 | 1 = value published, with
// K = (plan << 27 | vertex) + 1.  Zeroed before every launch, so values never
// outlive the index state they were computed on.  A lookup probes
// kLsumProbes slots; a warp that finds its key busy or every probe taken by
// other keys computes the value itself (nobody waits).
// A slot is claimed, read and published by 16-byte accesses alone (one memory
// operation each, so that key and value need no order between them).  Relaxed:
// an acquire at device scope drops the SM's whole L1, which the searches of
// the other 31 resident warps live in.
constexpr uint32_t kLsumProbes = 4;
constexpr uint32_t kLsumNone = 0xffffffffu;

__device__ __forceinline__ void lsum_load(const unsigned long long* slot, unsigned long long& k,
                                          unsigned long long& v) {
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(k), "=l"(v) : "l"(slot) : "memory");
}
__device__ __forceinline__ void lsum_publish(unsigned long long* slot, unsigned long long K, unsigned long long v) {
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}"
                 ::"l"(slot), "l"((K << 1) | 1ull), "l"(v) : "memory");
}
// Claims an empty slot for K; otherwise false, and what the slot holds.
__device__ __forceinline__ bool lsum_claim(unsigned long long* slot, unsigned long long K, unsigned long long& k,
                                           unsigned long long& v) {
    asm volatile("{\n\t.reg .b128 t, e, n;\n\tmov.b128 e, {%4, %4};\n\tmov.b128 n, {%3, %4};\n\t"
                 "atom.relaxed.gpu.global.cas.b128 t, [%2], e, n;\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(k), "=l"(v) : "l"(slot), "l"(K << 1), "l"(0ull) : "memory");
    return k == 0;
}

// One thread: the published value of K (hit = true), or the slot this
// thread claimed for K (to publish into), or kLsumNone.
__device__ __forceinline__ uint32_t lsum_find(unsigned long long* tab, uint32_t mask, unsigned long long K, bool& hit,
                                              unsigned long long& val) {
    uint32_t s = (uint32_t)((K * 0x9e3779b97f4a7c15ull) >> 32) & mask;
    for (uint32_t probe = 0; probe < kLsumProbes; ++probe, s = (s + 1) & mask) {
        unsigned long long* slot = tab + 2 * (size_t)s;
        unsigned long long k, v;
        lsum_load(slot, k, v);
        if (k == 0 && lsum_claim(slot, K, k, v)) return s;
        if ((k >> 1) == K) {
            if (k & 1ull) {
                hit = true;
                val = v;
            }
            return kLsumNone;  // published, or being computed by another warp
        }
    }
    return kLsumNone;
}

// Subtree memos.  The count S(x) of the subtree below a memo's level is a
// function of x = m[memo_pos] alone, so all the launch needs of it is
//     sum over x of S(x) * (sum of the weights of the prefixes that end in x).
// A slot {key, S, weight, -} gathers both: every prefix adds its weight; the
// one that claimed the slot expands the subtree, which may be handed to any
// number of warps (a task carries the slot), each adding its part of S;
// k_memo_finish multiplies.  Nobody waits for a value and no subtree is
// expanded twice.  (Publishing a finished S left the heaviest subtrees
// unpublished, their work being split among warps at once, and expanded by
// every warp that met them meanwhile.)  Slots are empty between launches.
constexpr uint32_t kMemoProbes = 8;

// key of the memo of plan ei at vertex x (never 0)
__device__ __forceinline__ unsigned long long memo_key(uint32_t ei, uint32_t x) {
    return (1ull << 63) | ((unsigned long long)ei << 27) | x;
}
// One thread: the slot of K, claimed if there is none (fresh) and `create`;
// kLsumNone when there is none or the probes are taken by other keys.
__device__ __forceinline__ uint32_t memo_slot(const DfsArgs& a, unsigned long long K, bool create, bool& fresh) {
    uint32_t s = (uint32_t)((K * 0x9e3779b97f4a7c15ull) >> 32) & a.memo_mask;
    for (uint32_t probe = 0; probe < kMemoProbes; ++probe, s = (s + 1) & a.memo_mask) {
        unsigned long long* slot = a.memo_tab + 4 * (size_t)s;
        unsigned long long k = *(volatile unsigned long long*)slot;
        if (k == 0) {
            if (!create) return kLsumNone;
            k = atomicCAS(slot, 0ull, K);
            if (k == 0) {
                fresh = true;
                a.memo_list[atomicAdd(a.qctr + kQMemo, 1u)] = s;
                return s;
            }
        }
        if (k == K) return s;
    }
    return kLsumNone;
}
// Adds S * weight of every claimed slot to its plan's count and empties it.
__global__ void k_memo_finish(unsigned long long* tab, const uint32_t* __restrict__ list, const unsigned int* n,
                              unsigned long long* counts) {
    const uint32_t total = *n;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        ulonglong2* slot = reinterpret_cast<ulonglong2*>(tab + 4 * (size_t)list[i]);
        const ulonglong2 ks = slot[0], wx = slot[1];
        const unsigned long long v = ks.y * wx.x;
        if (v) atomicAdd(counts + ((ks.x >> 27) & 0xffffu), v);
        slot[0] = make_ulonglong2(0, 0);
        slot[1] = make_ulonglong2(0, 0);
    }
}

__device__ __forceinline__ unsigned long long warp_sum(unsigned long long x) {
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(kFull, x, o);
    return x;
}

// Work units of the DFS: seeds (delta edges; seed_claim.h), ranges handed
// over inside a block through shared memory, and ranges handed to other blocks
// through a ring of tasks in device memory.  A task is 16 words: w0 = ei |
// depth << 16 | generator << 24, w1/w2 = [lo, hi) of the generator list, w3 =
// ready tag (ring only), w4..15 = the matched prefix.  At every chunk a busy
// warp that sees a waiting one publishes all the work it has not started at
// its shallowest level (top of its stack), so the biggest remaining subtrees
// move first: to a warp of its own block if one waits (s_wait; the task goes
// into that warp's mailbox), else to the ring while tickets outnumber reserved
// tasks.
// One waiting warp per block (s_poller) holds a ring ticket (atomicAdd on the
// ticket counter) and waits for task number `ticket`; tasks are numbered by an
// atomicAdd in the same order, so every task has exactly one consumer and
// neither side contends on a CAS.  The other waiting warps spin on their
// mailbox in shared memory.  What bounds a launch with little work is how fast
// that work spreads: with all 4,736 resident warps polling the ring and the
// termination counters (ld.acquire at device scope, which also drops the SM's
// L1), the counters' L2 slice saturated and a donor's own look at them took
// 15,000 cycles.
// Termination: completed == seeds + reserved, completed read first.  s_live
// counts a block's unfinished units (high word; a mailbox task counts from its
// donation) and its finished seeds and ring tasks not yet reported (low word);
// they are reported when no unit of the block is unfinished, so a reported
// unit has no part left anywhere but in the ring, where its reservation came
// before its report: equality means no unit is active and none can be created.
// Device-scope acquire load / release increment (cheaper than full fences).
__device__ __forceinline__ unsigned int ld_acquire(const unsigned int* p) {
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void add_release(unsigned int* p, unsigned int v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

constexpr uint32_t kTaskWords = 16;
constexpr uint32_t kTaskMemo = 15;  // word of a task: memo slot its counts go to (no prefix reaches position 11)
constexpr unsigned long long kLiveUnit = 1ull << 32;  // one unfinished unit in s_live
constexpr uint32_t kNoTicket = 0xffffffffu;

// tasks reserved (x) and tickets issued (y) in one load
__device__ __forceinline__ uint2 ld_relaxed_u2(const unsigned int* q) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(q) : "memory");
    return make_uint2((uint32_t)v, (uint32_t)(v >> 32));
}
constexpr uint32_t kNoVertex = 0xffffffffu;  // m[1] of a grouped unit: matches no candidate

// First index of the ascending X[0..n) whose value is >= c (> c when upper),
// for a warp-uniform c: 32-ary search, each round one load per lane.
__device__ __forceinline__ uint32_t warp_bound(const uint32_t* __restrict__ X, uint32_t n, uint32_t c, bool upper,
                                               uint32_t lane) {
    uint32_t lo = 0, hi = n;  // the answer lies in [lo, hi]
    while (hi - lo > 32) {
        const uint32_t span = hi - lo;
        bool below = false;  // lanes 0..30 test the pivots lo + floor(span * (lane + 1) / 32)
        if (lane < 31) {
            const uint32_t x = __ldg(X + lo + (uint32_t)(((uint64_t)span * (lane + 1)) >> 5));
            below = upper ? x <= c : x < c;
        }
        const uint32_t k = __popc(__ballot_sync(kFull, below));
        const uint32_t nlo = k ? lo + (uint32_t)(((uint64_t)span * k) >> 5) + 1u : lo;
        hi = k < 31 ? lo + (uint32_t)(((uint64_t)span * (k + 1)) >> 5) : hi;
        lo = nlo;
    }
    bool below = false;
    if (lo + lane < hi) {
        const uint32_t x = __ldg(X + lo + lane);
        below = upper ? x <= c : x < c;
    }
    return lo + __popc(__ballot_sync(kFull, below));
}

// Seed group of a grouped unit: X = the delta list of (seed_dir, m[0]), the
// x values of all seeds (x, m[0]) with multiplicity.  Up to 32 values live
// one per lane in xv.
struct SeedGroup {
    const uint32_t* x;
    uint32_t n;
    uint32_t xv;
    // multiplicity of the warp-uniform c in X
    __device__ __forceinline__ uint32_t mult(uint32_t c, uint32_t lane) const {
        if (n <= 32) return __popc(__ballot_sync(kFull, xv == c));
        return warp_bound(x, n, c, true, lane) - warp_bound(x, n, c, false, lane);
    }
    // per lane with `on`, the multiplicity of its own c: only the values of X
    // inside the chunk's range [cmin, cmax] are looked at
    __device__ __forceinline__ uint32_t mult_lane(uint32_t c, bool on, uint32_t lane) const {
        const uint32_t cmin = __reduce_min_sync(kFull, on ? c : 0xffffffffu);
        const uint32_t cmax = __reduce_max_sync(kFull, on ? c : 0u);
        if (cmin > cmax) return 0;
        uint32_t r = 0;
        if (n <= 32) {
            uint32_t bits = __ballot_sync(kFull, lane < n && xv >= cmin && xv <= cmax);
            while (bits) {
                const uint32_t i = __ffs(bits) - 1;
                bits &= bits - 1;
                r += (__shfl_sync(kFull, xv, i) == c) ? 1u : 0u;
            }
        } else {
            const uint32_t lo = warp_bound(x, n, cmin, false, lane), hi = warp_bound(x, n, cmax, true, lane);
            if (lo == hi) return 0;
            if (on) {
                uint32_t p = lo, len = hi - lo;
                while (len > 0) {
                    const uint32_t half = len >> 1;
                    if (__ldg(x + p + half) < c) { p += half + 1; len -= half + 1; }
                    else len = half;
                }
                for (; p < hi && __ldg(x + p) == c; ++p) ++r;
            }
        }
        return on ? r : 0u;
    }
};
// Ready tag of ticket t in launch `epoch`: the epoch's low 20 bits and the
// ring lap of t, so a slot reused in a later lap or launch never shows a
// stale tag to the consumer of t.
__device__ __forceinline__ uint32_t task_tag(uint32_t epoch, uint32_t t) {
    return ((epoch & 0xfffffu) << 12) | ((t / kTaskCap) & 0xfffu);
}
// Shard of the seed group (query edge ei, vertex x at the plan's first
// position): splitmix64's finaliser of (ei << 32 | x), modulo the shard
// count.  Seeds of one group (a grouped plan's run of equal first vertices)
// share the key, so a group is never split between shards.
__host__ __device__ __forceinline__ uint32_t seed_shard(uint32_t ei, uint32_t x, uint32_t num_shards) {
    uint64_t z = ((uint64_t)ei << 32 | x) + 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    z ^= z >> 31;
    return (uint32_t)(z % num_shards);
}

// s_cand entries: vertex id (< 2^27) | offset of the candidate in the
// generator chunk it came from << 27
constexpr uint32_t kCandBits = 27;
constexpr uint32_t kCandMask = (1u << kCandBits) - 1u;

// kMulti = false: one query, its plans (a.plans, one per edge, at most
// kMaxQEKeyed) and seed table copied to shared memory by every block.
// kMulti = true: the plans of every registered query in global memory
// (a.plans, one per (query, edge); a.qe of them), seed table searched in
// global memory, each warp's current plan copied to shared memory when its
// unit changes plan.  kSums = false compiles the level sums,
// memos and pair counting out: the kernel is bound by
// instruction fetch, and their code doubled its fetch stalls on patterns
// whose plans never use them.
template <bool kMulti, bool kFoot = false, bool kSums = true>
__global__ void __launch_bounds__(kDfsWarps * 32, 4) k_dfs_count(DfsArgs a) {
    __shared__ uint32_t s_cand[kDfsWarps][kMaxQV][32];
    __shared__ uint4 s_bn[kDfsWarps][kMaxBN];
    __shared__ uint32_t s_rbs[kDfsWarps][kMaxBN];  // run bit-set slot of each resolved record
    __shared__ uint32_t s_m[kDfsWarps][kMaxQV];
    __shared__ unsigned long long s_tc[kDfsWarps][cgb::kMaxSub];  // counts of the subsets off the prefix
    __shared__ uint32_t s_pre[kMulti ? 1 : kMaxQE + 1];
    __shared__ uint32_t s_lo[kMulti ? 1 : kMaxQE];
    __shared__ __align__(16) EdgePlan s_plan[kMulti ? kDfsWarps : cgb::kMaxQEKeyed];
    __shared__ uint32_t s_box[kDfsWarps][kTaskWords];  // mailboxes: tasks from this block's busy warps
    __shared__ uint32_t s_boxfull[kDfsWarps];
    __shared__ uint32_t s_wait;                        // bit w: warp w waits on its mailbox
    __shared__ uint32_t s_poller;                      // a warp of this block waits on the ring
    __shared__ uint32_t s_over;                        // the launch has no work left
    __shared__ unsigned long long s_live;              // unfinished units << 32 | finished, unreported
    __shared__ uint32_t s_row;                         // the block's row of seeds
    // lane 0's own (looked at between units only: registers are what the search is short of):
    // where the next seed comes from, its row, this warp's bit of s_wait was set, ticket of the ring
    __shared__ uint32_t s_acq[kDfsWarps][4];
    __shared__ unsigned long long s_stat[kDfsWarps][3];  // tail counts, bytes, busy cycles

    const uint32_t lane = threadIdx.x & 31;
    const uint32_t w = threadIdx.x >> 5;
    const bool self_loops = *(const volatile unsigned int*)a.self_seen != 0;
    // launch tag of the task ring: a kernel argument, or (in a replayed CUDA
    // graph, whose arguments are fixed) a device word bumped before the launch
    const uint32_t epoch = a.epoch_ptr ? *(const volatile unsigned int*)a.epoch_ptr : a.epoch;
    if (threadIdx.x == kDfsWarps * 32 - 1) s_row = atomicAdd(a.work_next + 1, 1u);  // beside the loads that follow
    if (!kMulti) {
        if (threadIdx.x <= a.qe) s_pre[threadIdx.x] = a.seed_pre[threadIdx.x];
        if (threadIdx.x < a.qe) s_lo[threadIdx.x] = a.seed_lo[threadIdx.x];
        const uint32_t* src = reinterpret_cast<const uint32_t*>(a.plans);
        uint32_t* dst = reinterpret_cast<uint32_t*>(s_plan);
        for (uint32_t t = threadIdx.x; t < a.qe * (uint32_t)(sizeof(EdgePlan) / 4); t += blockDim.x)
            dst[t] = __ldg(src + t);
    }
    if (threadIdx.x < kDfsWarps) {
        s_boxfull[threadIdx.x] = 0;
        s_stat[threadIdx.x][0] = s_stat[threadIdx.x][1] = s_stat[threadIdx.x][2] = 0;
        s_acq[threadIdx.x][0] = cgb::kSeedFirst;
        s_acq[threadIdx.x][2] = 0;
        s_acq[threadIdx.x][3] = kNoTicket;
    }
    if (threadIdx.x == 0) {
        s_wait = s_poller = s_over = 0;
        s_live = 0;
    }
    __syncthreads();
    auto pre_at = [&](uint32_t e) -> uint32_t { return kMulti ? __ldg(a.seed_pre + e) : s_pre[e]; };
    auto lo_at = [&](uint32_t e) -> uint32_t { return kMulti ? __ldg(a.seed_lo + e) : s_lo[e]; };
    auto grouped_at = [&](uint32_t e) -> bool { return kMulti ? a.plans[e].grouped != 0 : s_plan[e].grouped != 0; };
    int plan_in_smem = -1;  // kMulti: plan held in s_plan[w]
    // every engine walks all seeds; a sharded one skips the groups of other shards
    const uint32_t total = pre_at(a.qe);
    const uint64_t vmask = (1ull << a.B) - 1ull;
    uint32_t* m = s_m[w];
    uint4* bn = s_bn[w];
    using RB = typename std::conditional<kFoot, RunBitsCount, RunBits>::type;
    RB rb;
    rb.slot = a.rb_slot;
    rb.bits = a.rb_bits;
    rb.words = a.rb_words;
    rb.bslot = s_rbs[w];
    if constexpr (kFoot) rb.touched = a.touched;
    volatile unsigned int* vq = a.qctr;
    volatile uint32_t* vfull = s_boxfull;
    // per-depth state held by lane == depth
    uint32_t st_ncand = 0, st_pos = 0, st_next = 0, st_len = 0, st_gen = 0;
    uint32_t st_hs = 0;  // grouped units: X multiplicity of the vertices at hit positions < depth
    unsigned long long cnt = 0;  // lane-local partial count of the current edge
    // statistics: 32-bit counts in registers; tail counts and bytes (seed keys,
    // records, list words, probe sectors) gathered in shared memory, bytes
    // from a per-lane count of 4-byte words emptied every 64 steps and at every
    // unit's end (2^32 words a lane: some ten seconds of one warp's search)
    uint32_t n_seeds = 0, n_chunks = 0, n_tested = 0, n_tasks = 0, n_words = 0;
    auto count_tails = [&](uint32_t v) { s_stat[w][0] += v; };
    auto flush_bytes = [&]() {
        // in two halves: 32 lanes' sum has more than 32 bits
        const uint32_t lo = __reduce_add_sync(kFull, n_words & 0xffffu), hi = __reduce_add_sync(kFull, n_words >> 16);
        n_words = 0;
        if (lane == 0) s_stat[w][1] += 4ull * lo + ((unsigned long long)hi << 18);
    };
    int cur_ei = -1;
    const unsigned long long t_start = global_ns();
    uint32_t steps = 0;
    bool out_of_time = false;
    uint32_t &seeds = s_acq[w][0], &waiting = s_acq[w][2], &ticket = s_acq[w][3];
    uint32_t dirty = 0;  // shallowest position changed since the tail cache was filled (kClean: none)
    bool mb = false;              // counting (a part of) a subtree memo's S, unweighted, into mb_slot
    uint32_t mb_slot = kLsumNone;
    unsigned long long mb_base = 0;  // lane-local count when it was entered
    unsigned long long tail_k = 0;  // product of the tail groups that depend on the current prefix alone
    uint32_t idle_spins = 0;
    uint32_t kind = 0;
    uint32_t unit_clk = 0;  // kMulti: clock at the current unit's start

    for (;;) {
        // ---- acquire a unit: 1 = seed, 2 = ring task, 3 = all done, 4 = mailbox task, 0 = nothing yet
        if (kind) {
            // the unit before is finished; its report waits until no unit of the block is unfinished
            flush_bytes();
            if (lane == 0) {
                if (kMulti) s_stat[w][2] += (uint32_t)clock() - unit_clk;
                const unsigned long long dv = (kind != 4 ? 1ull : 0ull) - kLiveUnit;
                const unsigned long long nv = atomicAdd(&s_live, dv) + dv;
                if (nv < kLiveUnit && nv && atomicCAS(&s_live, nv, 0ull) == nv)
                    add_release(a.qctr + kQDone, (unsigned int)nv);
            }
        }
        kind = 0;
        uint32_t item = 0;
        if (lane == 0) {
            if (seeds <= cgb::kSeedNext) {
                item = cgb::seed_claim(seeds, s_acq[w][1], s_row, w, total, gridDim.x, kDfsWarps, a.steal != 0,
                                       [&](uint32_t i, uint32_t n) { return atomicAdd(a.work_next + i, n); },
                                       [&](uint32_t i) { return *(volatile unsigned int*)(a.work_next + i); });
                if (item < total) {
                    kind = 1;
                    atomicAdd(&s_live, kLiveUnit);
                }
            }
            if (!kind) {
                if (!a.steal) {
                    kind = 3;  // nothing is ever shared
                } else if (ticket == kNoTicket) {
                    if (!waiting) {
                        atomicOr(&s_wait, 1u << w);
                        waiting = true;
                    }
                    if (vfull[w]) {
                        kind = 4;
                        waiting = false;
                    } else if (*(volatile uint32_t*)&s_over) {
                        kind = 3;
                    } else if (!*(volatile uint32_t*)&s_poller && atomicCAS(&s_poller, 0u, 1u) == 0u) {
                        // wait on the ring for the block instead, unless a busy
                        // warp has just taken this warp's bit to fill its mailbox
                        if ((atomicAnd(&s_wait, ~(1u << w)) >> w) & 1u) {
                            waiting = false;
                            ticket = atomicAdd(a.qctr + kQTickets, 1u);
                        } else {
                            *(volatile uint32_t*)&s_poller = 0;
                        }
                    }
                }
                if (ticket != kNoTicket) {
                    const volatile uint32_t* tk = a.tasks + (size_t)(ticket & (a.task_cap - 1u)) * kTaskWords;
                    if (tk[3] == task_tag(epoch, ticket)) {
                        kind = 2;
                        item = ticket;
                        ticket = kNoTicket;
                        atomicAdd(&s_live, kLiveUnit);
                        *(volatile uint32_t*)&s_poller = 0;
                    } else if ((idle_spins & 3u) == 3u && vq[kQDone] == total + vq[kQReserved]) {
                        // a plain look said done: again in order, completed read with acquire before reserved
                        const unsigned int done = ld_acquire(a.qctr + kQDone);
                        if (done == total + ld_acquire(a.qctr + kQReserved)) {
                            *(volatile uint32_t*)&s_over = 1;
                            kind = 3;
                        }
                    }
                }
            }
        }
        kind = __shfl_sync(kFull, kind, 0);
        item = __shfl_sync(kFull, item, 0);
        if (kind == 3) break;
        if (kind == 0) {
            __nanosleep(idle_spins < 16 ? 40u : 200u);
            ++idle_spins;
            // rows left over now are those of blocks that cannot start
            if ((idle_spins & 63u) == 16u && lane == 0 && seeds == cgb::kSeedLater && ticket == kNoTicket) {
                if (*(volatile unsigned int*)(a.work_next + 1) >= gridDim.x) {
                    seeds = cgb::kSeedNone;
                } else if (!waiting || ((atomicAnd(&s_wait, ~(1u << w)) >> w) & 1u)) {
                    waiting = false;  // (otherwise a busy warp is filling this warp's mailbox)
                    seeds = cgb::kSeedNext;
                }
            }
            if ((idle_spins & 255u) == 0) {
                const bool late = a.budget_ns && (global_ns() - t_start) > a.budget_ns;
                if (__shfl_sync(kFull, late ? 1 : 0, 0)) { out_of_time = true; break; }
            }
            continue;
        }
        idle_spins = 0;
        if (kMulti) unit_clk = (uint32_t)clock();

        int ei = 0;
        uint32_t jbase = 2, tgen = 0, tlo = 0, thi = 0;
        mb_slot = kLsumNone;
        if (kind == 1) {
            if (kMulti) {
                // last plan whose seeds start at or before item (empty plans skipped)
                uint32_t lo = 0, hi = a.qe;
                while (hi - lo > 1) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (pre_at(mid) <= item) lo = mid; else hi = mid;
                }
                ei = (int)lo;
            } else {
                while (ei + 1 < (int)a.qe && s_pre[ei + 1] <= item) ++ei;
            }
            const uint32_t e_pre = pre_at(ei), e_lo = lo_at(ei);
            const uint64_t key = a.dkeys[e_lo + (item - e_pre)];
            ++n_seeds;
            if (grouped_at(ei) && item > e_pre) {
                // a grouped edge runs one DFS per first vertex: only the first
                // seed of each run of equal first vertices starts one
                const uint64_t prev = a.dkeys[e_lo + (item - e_pre) - 1];
                if (((prev ^ key) >> a.B & vmask) == 0) continue;
            }
            if (a.num_shards > 1 && seed_shard((uint32_t)ei, (uint32_t)((key >> a.B) & vmask), a.num_shards) != a.shard)
                continue;
            if (lane == 0) {
                m[0] = (uint32_t)((key >> a.B) & vmask);
                m[1] = grouped_at(ei) ? kNoVertex : (uint32_t)(key & vmask);
                n_words += 2;
            }
        } else {
            // lane 0 saw the ticket's ready tag, or its mailbox full: the task's words are published
            volatile uint32_t* tk = kind == 4 ? s_box[w] : a.tasks + (size_t)(item & (a.task_cap - 1u)) * kTaskWords;
            if (kind == 4) __threadfence_block(); else __threadfence();
            const uint32_t wv = lane < kTaskWords ? tk[lane] : 0;
            __syncwarp();
            if (kind == 4 && lane == 0) vfull[w] = 0;
            const uint32_t w0 = __shfl_sync(kFull, wv, 0);
            ei = (int)(w0 & 0xffffu);
            jbase = (w0 >> 16) & 0xffu;
            tgen = (w0 >> 24) & 0xffu;
            tlo = __shfl_sync(kFull, wv, 1);
            thi = __shfl_sync(kFull, wv, 2);
            if (kSums) mb_slot = __shfl_sync(kFull, wv, kTaskMemo);
            if (lane >= 4 && lane < 4 + kMaxQV) m[lane - 4] = wv;
            ++n_tasks;
        }
        __syncwarp();
        if (ei != cur_ei) {
            const unsigned long long c = warp_sum(cnt);
            if (cur_ei >= 0 && lane == 0 && c) atomicAdd(a.counts + cur_ei, c);
            cnt = 0;
            cur_ei = ei;
        }
        if (kMulti && plan_in_smem != ei) {
            const uint32_t* src = reinterpret_cast<const uint32_t*>(a.plans + ei);
            uint32_t* dst = reinterpret_cast<uint32_t*>(&s_plan[w]);
            for (uint32_t t = lane; t < sizeof(EdgePlan) / 4; t += 32) dst[t] = __ldg(src + t);
            __syncwarp();
            plan_in_smem = ei;
        }
        const EdgePlan& P = kMulti ? s_plan[w] : s_plan[ei];
        const bool tail_cache = a.tail_cache && !(P.flags & cgb::kPlanNoTailCache);
        const uint32_t nc = P.n_core;
        const bool has_tail = nc < P.n;
        const bool serial = has_tail && (!tail_cache || (P.flags & cgb::kPlanWarpTail));
        SeedGroup X{nullptr, 0u, kNoVertex};
        // weight of a grouped embedding with hs hits (1 inside a memo's subtree,
        // whose count is weighted once when it is complete)
        auto gw = [&](uint32_t hs) -> unsigned long long { return kSums && mb ? 1ull : (unsigned long long)(X.n - hs); };
        if (P.grouped) {
            const size_t xat = (size_t)P.seed_dir * a.dvcap + m[0];
            const uint4 xr = a.rec[xat];
            if (kFoot && lane == 0) atomicOr(a.touched + (xat >> 5), 1u << (xat & 31));
            X.x = a.dval + xr.z;
            X.n = xr.w;
            if (X.n <= 32 && lane < X.n) X.xv = __ldg(X.x + lane);
            if (lane == 0) n_words += 4 + min(X.n, 32u);
        }
        // set up depth j: resolve BN records, choose the shortest list as generator
        auto setup = [&](uint32_t j) {
            const uint32_t o0 = P.bn_off[j], o1 = P.bn_off[j + 1];
            const uint32_t nb = o1 - o0;
            uint32_t len = 0xffffffffu;
            if (lane < nb) {
                const uint32_t k = o0 + lane;
                const size_t at = (size_t)P.bn_dir[k] * a.dvcap + m[P.bn_pos[k]];
                uint4 r = a.rec[at];
                if (!P.bn_dvis[k]) r.w = 0;
                bn[k] = r;
                rb.note(k, at);
                len = r.y + r.w;
                n_words += 4;
            }
            // shortest list, lowest lane on ties: one redux over (length << 5 | lane)
            // (lengths are below 2^27; a longer one is only a worse generator)
            const uint32_t key = len == 0xffffffffu ? 0xffffffffu : (min(len, (1u << 27) - 1u) << 5) | lane;
            const uint32_t kmin = __reduce_min_sync(kFull, key);
            const uint32_t best = kmin >> 5, bl = kmin & 31u;
            if (lane == j) { st_ncand = 0; st_pos = 0; st_next = 0; st_len = nb ? best : 0; st_gen = bl; }
            __syncwarp();
        };

        dirty = 0;  // new unit: every cached tail count is stale
        const bool level_sum = kSums && P.sum_from && !a.vb && !self_loops && (!serial);
        const bool memo_on = kSums && P.memo_from && a.memo_tab && !a.vb && !self_loops;
        const bool pair_on = kSums && P.pair_last && !a.vb && !self_loops && (!serial);
        const bool sum_on = level_sum && !P.sum_dense;  // one-position sums, through the table
        const bool peek_on = memo_on && P.memo_from == P.memo_pos + 1;
        // position whose chunks are evaluated per lane besides the last one
        const uint32_t dpre = (pair_on || (sum_on && nc > 3)) ? nc - 2 : kNoPos;
        // depths where a chunk's passing candidates are partly counted at once:
        // what is not scanned yet is shared from them, then single survivors (a
        // unit that kept the survivors of a memo's position ran as long as the
        // whole launch: 2.2 ms of the R-MAT 4M/34M sparse pattern's batch)
        const uint32_t counted = (dpre != kNoPos ? 1u << dpre : 0u) | (peek_on ? 1u << P.memo_pos : 0u);
        mb = kSums && mb_slot != kLsumNone;  // a task inside a memo's subtree
        mb_base = cnt;
        if (nc > 2) {
            setup(jbase);
            if (kind != 1 && lane == jbase) { st_gen = tgen; st_next = tlo; st_len = thi; }
        }
        if (P.grouped) {
            uint32_t h = 0;
            for (uint32_t p = 2; p < jbase; ++p)
                if ((P.hit_mask >> p) & 1u) h += X.mult(m[p], lane);
            if (lane == jbase) st_hs = h;
        }
        __syncwarp();
        uint32_t j = jbase;
        for (;;) {
            if ((++steps & 63u) == 0) {
                flush_bytes();
                if (a.budget_ns && (steps & 1023u) == 0) {
                    // bounded run: give up (and report) once the budget is spent
                    unsigned long long now = global_ns();
                    out_of_time = __shfl_sync(kFull, (now - t_start) > a.budget_ns ? 1 : 0, 0) != 0;
                    if (out_of_time) break;
                }
            }
            // What this step evaluates: `ok` lanes, each with a candidate c at
            // position d, worth v0 times its tail count; or (node) no candidate
            // at all: lane 0 stands for the whole subtree below the prefix m[0..d).
            bool node = nc == 2, ok = false;
            uint32_t c = 0, d = j, gnext = 0, glen = 0;
            unsigned long long v0 = 1;
            if (nc > 2) {
                const uint32_t ncand = __shfl_sync(kFull, st_ncand, j);
                const uint32_t pos = __shfl_sync(kFull, st_pos, j);
                if (pos < ncand) {
                    if (lane == j) st_pos = pos + 1;
                    if (lane == 0) m[j] = s_cand[w][j][pos] & kCandMask;
                    __syncwarp();
                    dirty = min(dirty, j);
                    if (P.grouped) {
                        uint32_t h = __shfl_sync(kFull, st_hs, j);
                        if ((P.hit_mask >> j) & 1u) h += X.mult(m[j], lane);
                        if (lane == j + 1) st_hs = h;
                    }
                    ++j;
                    setup(j);
                    continue;
                }
                gnext = __shfl_sync(kFull, st_next, j);
                glen = __shfl_sync(kFull, st_len, j);
                if (gnext >= glen) {
                    if (kSums && mb && (j == P.memo_from || j == jbase)) {
                        // this warp's part of the memo's subtree is complete
                        const unsigned long long S = warp_sum(cnt - mb_base);
                        if (lane == 0 && S) atomicAdd(a.memo_tab + 4 * (size_t)mb_slot + 1, S);
                        cnt = mb_base;
                        mb = false;
                    }
                    if (j == jbase) break;
                    --j;
                    continue;
                }
                if (kSums && gnext == 0 && (memo_on || level_sum)) {
                    const uint4 gr = bn[P.bn_off[j] + __shfl_sync(kFull, st_gen, j)];
                    if (glen == gr.y + gr.w) {
                        if (memo_on && !mb && j == P.memo_from) {
                            // the whole level below m[memo_pos]: this prefix's weight goes to the
                            // memo; its subtree is expanded here if no other prefix did
                            uint32_t slot = kLsumNone;
                            bool fresh = false;
                            unsigned long long wt = 1;
                            if (P.grouped) wt = X.n - __shfl_sync(kFull, st_hs, j);
                            if (lane == 0) {
                                slot = memo_slot(a, memo_key((uint32_t)ei, m[P.memo_pos]), true, fresh);
                                if (slot != kLsumNone) atomicAdd(a.memo_tab + 4 * (size_t)slot + 2, wt);
                            }
                            slot = __shfl_sync(kFull, slot, 0);
                            if (slot != kLsumNone && !__shfl_sync(kFull, fresh ? 1u : 0u, 0)) {
                                if (lane == 0) count_tails(1);
                                if (lane == j) st_next = glen;
                                __syncwarp();
                                continue;
                            }
                            if (slot != kLsumNone) {
                                mb = true;
                                mb_slot = slot;
                                mb_base = cnt;
                            }
                        }
                        if (level_sum && P.sum_dense && a.wsum && j == P.sum_from) {
                            // positions [j, n_core) counted at once: the product of the
                            // precomputed sums of the positions owned by prefix positions
                            if (lane >= j && lane < nc) {
                                const uint32_t p = P.bn_pos[P.bn_off[lane]];
                                if (p < j) {
                                    v0 = __ldg(a.wsum + (size_t)(P.wslot + lane - j) * a.dvcap + m[p]);
                                    n_words += 2;
                                }
                            }
                            for (int o = 16; o > 0; o >>= 1) v0 *= __shfl_xor_sync(kFull, v0, o);
                            node = true;
                        } else if (sum_on && nc == 3) {
                            node = true;  // the last core position right below the seed
                        }
                    }
                }
                if (!node) {
                    // While warps wait for tasks, hand the work not yet started at the
                    // shallowest level of this unit to one of them: at a depth d < j
                    // the buffered survivors not yet descended plus the unscanned
                    // generator range, at d = j the range after this chunk.  The
                    // survivors are a contiguous stretch of the generator (their
                    // offsets in their chunk ride in the top bits of s_cand), so
                    // one range [lo, hi) of depth d's generator describes it all.
                    if (a.steal) {  // checked at every chunk: a waiting warp is served within one chunk's time
                        // 2: a warp of this block waits; 1: some block holds a ticket no task has been reserved for
                        uint32_t want = 0;
                        if (lane == 0) {
                            if (a.force_split) {
                                want = 1u;
                            } else if (*(volatile uint32_t*)&s_wait) {
                                want = 2u;
                            } else {
                                const uint2 q = ld_relaxed_u2(a.qctr);
                                want = (int)(q.y - q.x) > 0 ? 1u : 0u;
                            }
                        }
                        want = __shfl_sync(kFull, want, 0);
                        if (want) {
                            bool has = false;
                            if (lane >= jbase && lane < j) has = st_next < st_len || st_pos < st_ncand;
                            if (lane == j) has = glen > gnext + 32u;
                            const uint32_t hb = __ballot_sync(kFull, has);
                            uint32_t slot = 0xffffffffu;
                            if (hb && lane == 0) {
                                if (want == 2u) {
                                    const uint32_t wm = *(volatile uint32_t*)&s_wait;
                                    const uint32_t t = wm ? __ffs(wm) - 1 : 0u;
                                    if (wm && ((atomicAnd(&s_wait, ~(1u << t)) >> t) & 1u)) {
                                        slot = t;
                                        atomicAdd(&s_live, kLiveUnit);
                                    }
                                } else {
                                    // reserve the next task number while tickets wait for one (always, under
                                    // force_split).  atomicAdd never fails, so concurrent producers may
                                    // overshoot the demand by a few tasks; those wait in the ring for the
                                    // next idle warps, and the slack keeps the ring from lapping its head.
                                    const uint2 q = ld_relaxed_u2(a.qctr);
                                    if ((a.force_split || (int)(q.y - q.x) > 0) &&
                                        (int)(q.x - q.y) < (int)(a.task_cap - kTaskSlack))
                                        slot = atomicAdd(a.qctr + kQReserved, 1u);
                                }
                            }
                            slot = __shfl_sync(kFull, slot, 0);
                            if (slot != 0xffffffffu) {
                                const uint32_t d = __ffs(hb) - 1;
                                uint32_t lo = 0, hi = 0;
                                if (lane == d) {
                                    if (d == j) {
                                        lo = gnext + 32u;
                                        hi = glen;
                                    } else if (((counted >> d) & 1u) && st_next >= st_len) {
                                        // some of the chunk's candidates were counted at once, so the
                                        // survivors are no stretch: the last one goes alone
                                        lo = st_next - 32u + (s_cand[w][d][st_ncand - 1u] >> kCandBits);
                                        hi = lo + 1u;
                                    } else if ((counted >> d) & 1u) {
                                        lo = st_next;  // the buffered survivors stay for now
                                        hi = st_len;
                                    } else {
                                        lo = st_pos < st_ncand ? st_next - 32u + (s_cand[w][d][st_pos] >> kCandBits)
                                                               : st_next;
                                        hi = st_len;
                                    }
                                }
                                lo = __shfl_sync(kFull, lo, d);
                                hi = __shfl_sync(kFull, hi, d);
                                const uint32_t gd = __shfl_sync(kFull, st_gen, d);
                                uint32_t* tk =
                                    want == 2u ? s_box[slot] : a.tasks + (size_t)(slot & (a.task_cap - 1u)) * kTaskWords;
                                uint32_t v = 0;
                                if (lane == 0) v = (uint32_t)ei | (d << 16) | (gd << 24);
                                else if (lane == 1) v = lo;
                                else if (lane == 2) v = hi;
                                else if (lane == kTaskMemo) v = kSums && mb && d >= P.memo_from ? mb_slot : kLsumNone;
                                else if (lane >= 4 && lane < 4 + kMaxQV) v = (lane - 4 < d) ? m[lane - 4] : 0u;
                                if (lane < kTaskWords && lane != 3) tk[lane] = v;
                                if (want == 2u) __threadfence_block(); else __threadfence();
                                __syncwarp();
                                if (lane == 0) {
                                    if (want == 2u) vfull[slot] = 1;
                                    else *(volatile uint32_t*)(tk + 3) = task_tag(epoch, slot);
                                }
                                if (lane == d) {
                                    if (d == j) st_len = gnext + 32u;
                                    else if (((counted >> d) & 1u) && st_next >= st_len) --st_ncand;
                                    else if ((counted >> d) & 1u) st_len = st_next;
                                    else { st_len = st_next; st_ncand = st_pos; }
                                }
                                if (d == j) glen = gnext + 32u;
                            }
                        }
                    }
                    const uint32_t g = __shfl_sync(kFull, st_gen, j);
                    const uint32_t o0 = P.bn_off[j], o1 = P.bn_off[j + 1];
                    const uint4 gr = bn[o0 + g];
                    const uint32_t idx = gnext + lane;
                    ok = idx < glen;
                    if (ok) {
                        c = idx < gr.y ? __ldg(a.pool + gr.x + idx) : __ldg(a.dval + gr.z + (idx - gr.y));
                        n_words += 1;
                        for (uint32_t t = 0; t < j; ++t) ok &= (c != m[t]);
                        if (ok && a.vb)  // the valid bits are a sound superset: a clear bit cannot match
                            ok = (__ldg(a.vb + ((size_t)ei * a.qv + P.vs[j]) * a.vb_stride + (c >> 5)) >> (c & 31)) & 1u;
                    }
                    if (ok) {
                        // Each candidate is searched in every other backward list,
                        // stopping at the first miss.  All lanes search the same list
                        // with the same trip count, so the branch-free search keeps
                        // the warp converged, and the first steps of every lane hit
                        // the same words.
                        for (uint32_t k = o0; k < o1 && ok; ++k) {
                            if (k == o0 + g) continue;
                            const uint4 r = bn[k];
                            n_words += 8u * (33u - __clz(r.y | 1u));
                            ok = rb.has(k, r, a.pool, a.dval, c);
                        }
                        ++n_tested;
                    }
                    ++n_chunks;
                    if (j != nc - 1) {
                        bool desc = ok;  // survivors buffered for the descent
                        if (kSums && j == dpre) {
                            // counted below, per lane; pair counting leaves candidates
                            // whose shorter list is long to the descent
                            desc = false;
                            if (pair_on && a.pair_lane_max != kPairLaneMax) {
                                const size_t ata = (size_t)P.bn_dir[P.pair_a] * a.dvcap + m[P.bn_pos[P.pair_a]];
                                const size_t atb = (size_t)P.bn_dir[P.pair_b] * a.dvcap + c;
                                uint4 ra = a.rec[ata], rq = ok ? a.rec[atb] : make_uint4(0, 0, 0, 0);
                                const uint32_t la = ra.y + (P.bn_dvis[P.pair_a] ? ra.w : 0u);
                                const uint32_t lq = rq.y + (P.bn_dvis[P.pair_b] ? rq.w : 0u);
                                desc = ok && min(la, lq) > a.pair_lane_max;
                                ok = ok && !desc;
                            }
                        } else if (kSums && peek_on && j == P.memo_pos && !mb) {
                            // subtrees some warp expands already: only their weight is left to add
                            uint32_t slot = kLsumNone;
                            bool fresh = false;
                            if (ok) slot = memo_slot(a, memo_key((uint32_t)ei, c), false, fresh);
                            const bool hit = slot != kLsumNone;
                            unsigned long long wt = 1;
                            if (P.grouped) {
                                wt = X.n - __shfl_sync(kFull, st_hs, j);
                                if ((P.hit_mask >> j) & 1u) wt -= X.mult_lane(c, hit, lane);
                            }
                            if (hit) atomicAdd(a.memo_tab + 4 * (size_t)slot + 2, wt);
                            desc = ok && !hit;
                            ok = false;
                        } else {
                            ok = false;
                        }
                        const uint32_t bal = __ballot_sync(kFull, desc);
                        if (desc) s_cand[w][j][__popc(bal & ((1u << lane) - 1u))] = c | (lane << kCandBits);
                        if (lane == j) { st_ncand = __popc(bal); st_pos = 0; }
                    }
                }
            }
            if (node) ok = lane == 0;
            // the positions from n_core - 1 (one-position sums) or sum_from on are
            // counted by their sums, pendants included
            const bool summed = kSums && (sum_on ? node || j == dpre : node && nc > 2);
            uint32_t bal = __ballot_sync(kFull, ok);
            bool dead = false;  // no candidate of this level has a tail
            while (bal) {
                // one pass over the subsets for all lanes, or (serial) one embedding at a time
                bool on = ok;
                uint32_t de = d;
                if (serial && !node) {
                    const uint32_t l = __ffs(bal) - 1;
                    if (lane == l) m[j] = c;
                    __syncwarp();
                    on = lane == l;
                    de = nc;
                    dirty = tail_cache ? min(dirty, j) : 0u;
                }
                bal = serial && !node ? bal & (bal - 1u) : 0u;
                const uint32_t dmask = (1u << de) - 1u;
                const bool refresh = dirty < de && ((P.tail_reads & dmask) >> dirty) != 0;
                unsigned long long prod = on ? v0 : 0ull;
                if (refresh || dirty == 0) tail_k = 1;
                if (refresh) {
                    // records of the tail's (and the pair's) lists off changed prefix positions
                    for (uint32_t k = (pair_on ? P.sub_base : P.bn_off[nc]) + lane; k < P.bn_off[P.n]; k += 32) {
                        const uint32_t p = P.bn_pos[k];
                        if (p >= de || p < dirty) continue;
                        const size_t at = (size_t)P.bn_dir[k] * a.dvcap + m[p];
                        uint4 r = a.rec[at];
                        if (!P.bn_dvis[k]) r.w = 0;
                        bn[k] = r;
                        rb.note(k, at);
                        n_words += 4;
                    }
                    __syncwarp();
                }
                if (refresh || (P.sub_any >> de)) {
                    unsigned long long acc = 1, sc[3];
                    for (uint32_t i = 0; i < P.n_sub; ++i) {
                        const uint32_t sk = P.sub_kind[i];
                        const bool is_sum = kSums && (sk & cgb::kSubSum), is_pair = kSums && (sk & cgb::kSubPair);
                        if (kSums && ((is_sum && !(sum_on && summed)) || (is_pair && !(pair_on && j == dpre)) ||
                                      (summed && (sk & cgb::kSubPend))))
                            continue;
                        const bool live = is_sum || is_pair || (P.sub_group[i] >> de) != 0;
                        if (!live && !refresh) continue;
                        const uint32_t lists = P.sub_lists[i], pos = P.sub_pos[i];
                        const uint32_t ex = P.sub_excl[i] & ~(self_loops ? 0u : pos) & (dmask | 1u << de);
                        const bool stat = !is_sum && !(pos >> de);  // lists off the prefix only: cached
                        unsigned long long v;
                        if (stat && !(refresh && ((pos | (ex & dmask)) >> dirty))) {
                            v = s_tc[w][i];
                        } else {
                            bool fon = stat ? lane == 0 : prod != 0;
                            uint32_t fc = c, claim = kLsumNone;
                            unsigned long long hv = 0, K = 0;
                            bool hit = false;
                            uint32_t fd = de;
                            if (is_sum) {
                                // the sum over the list of its owner (this lane's candidate, or
                                // one vertex for the whole step): from the table, or walked here
                                // (and published when this lane claimed its slot)
                                const uint32_t p = P.bn_pos[P.sub_base];
                                if (p < de) { fc = m[p]; fon = lane == 0; }
                                fd = 0;
                                K = (((unsigned long long)ei << 27) | fc) + 1ull;
                                if (fon && a.lsum_tab) claim = lsum_find(a.lsum_tab, a.lsum_mask, K, hit, hv);
                                fon = fon && !hit;
                            }
                            if (!is_sum && !(lists & (lists - 1u))) {
                                // one list: its length less the excluded vertices in it
                                const uint32_t q = P.sub_base + __ffs(lists) - 1;
                                uint4 r = make_uint4(0, 0, 0, 0);
                                uint32_t sl = kNoSlot;
                                if (stat) {
                                    r = bn[q];
                                    sl = rb.slot ? rb.bslot[q] : kNoSlot;
                                } else if (fon) {
                                    const size_t at = (size_t)P.bn_dir[q] * a.dvcap + c;
                                    r = a.rec[at];
                                    if (!P.bn_dvis[q]) r.w = 0;
                                    if (ex) sl = rb.slot_at(at);
                                    rb.touch(at);
                                    n_words += 4;
                                }
                                v = (unsigned long long)r.y + r.w;
                                for (uint32_t e = stat ? ex & dmask : ex; e; e &= e - 1) {
                                    const uint32_t t = __ffs(e) - 1;
                                    const uint32_t x = t == de ? c : m[t];
                                    // a vertex held by two positions (a self-loop seed edge) is excluded once
                                    bool dup = x == kNoVertex;
                                    if (self_loops)
                                        for (uint32_t e2 = ex & ((1u << t) - 1u); e2; e2 &= e2 - 1) dup |= m[__ffs(e2) - 1] == x;
                                    if (!dup && v) v -= rb.has_slot(sl, r, a.pool, a.dval, x) ? 1ull : 0ull;
                                }
                            } else {
                                v = flat_lists(P, lists, fd, is_sum, fon, fc, stat ? ex & dmask : ex, m, bn, a.rec, a.dvcap,
                                               a.pool, a.dval, lane, n_words, rb);
                            }
                            if (stat) {
                                v = __shfl_sync(kFull, v, 0);
                                if (lane == 0) s_tc[w][i] = v;
                                __syncwarp();
                            } else if (is_sum) {
                                if (claim != kLsumNone) lsum_publish(a.lsum_tab + 2 * (size_t)claim, K, v);
                                if (hit) v = hv;
                                const uint32_t p = P.bn_pos[P.sub_base];
                                if (p < de) v = __shfl_sync(kFull, v, 0);
                                // less the matched prefix vertices in the list
                                const size_t at = (size_t)P.bn_dir[P.sub_base] * a.dvcap + fc;
                                for (uint32_t e = P.sum_same & (dmask | 1u << de); e; e &= e - 1) {
                                    const uint32_t t = __ffs(e) - 1;
                                    const uint32_t x = t == de ? c : m[t];
                                    if (!on || x == kNoVertex) continue;
                                    uint4 r = a.rec[at];
                                    if (!P.bn_dvis[P.sub_base]) r.w = 0;
                                    if (rb.has_slot(rb.slot_at(at), r, a.pool, a.dval, x))
                                        v -= sum_lens(P, a.rec, a.dvcap, x, rb);
                                }
                            }
                        }
                        if (stat && on && ((ex >> de) & 1u) && v) {
                            // the candidate itself may lie in every list of the subset
                            bool in = true;
                            for (uint32_t b = lists; b && in; b &= b - 1) {
                                const uint32_t q = P.sub_base + __ffs(b) - 1;
                                n_words += 8u * (33u - __clz(bn[q].y | 1u));
                                in = rb.has(q, bn[q], a.pool, a.dval, c);
                            }
                            v -= in ? 1ull : 0ull;
                        }
                        // inclusion-exclusion over the members that coincide
                        const uint32_t mem = sk & 7u;
                        if (!(mem & (mem - 1u))) {
                            acc = mem == 1u ? v : acc * v;
                            sc[mem >> 1] = v;
                        } else if (mem == 7u) {
                            acc += 2 * v;
                        } else {
                            acc -= (sk & cgb::kSubThree) ? v * sc[mem == 3u ? 2 : mem == 5u ? 1 : 0] : v;
                        }
                        if (sk & cgb::kSubLast) {
                            if (live) prod *= acc;
                            else tail_k *= acc;
                        }
                    }
                }
                dirty = kClean;
                if (tail_k == 0) dead = true;
                unsigned long long wt = 1;
                if (P.grouped) {
                    wt = gw(__shfl_sync(kFull, st_hs, d));
                    if (!node && ((P.hit_mask >> d) & 1u)) wt -= X.mult_lane(c, on, lane);
                }
                if (on) cnt += prod * tail_k * wt;
                const uint32_t non = __popc(__ballot_sync(kFull, on));
                if (lane == 0) count_tails(non);
            }
            if (nc == 2) break;
            // a level whose prefix-only tail count is 0 adds nothing however it goes
            // on; neither do survivors buffered from this chunk (pair counting), and
            // with st_next past the chunk their places could not be found again
            if (lane == j) {
                const bool done = node || (dead && !serial);
                st_next = done ? glen : gnext + 32u;
                if (kSums && done) st_ncand = st_pos;
            }
            __syncwarp();
        }
        if (out_of_time) {
            if (lane == 0) atomicOr(a.err, 8u);
            break;
        }
    }
    if (out_of_time && lane == 0) atomicOr(a.err, 8u);
    const unsigned long long c = warp_sum(cnt);
    if (cur_ei >= 0 && lane == 0 && c) atomicAdd(a.counts + cur_ei, c);
    const unsigned long long tested = warp_sum(n_tested);
    flush_bytes();
    if (lane == 0) {
        atomicAdd(a.stats + 0, n_seeds);
        atomicAdd(a.stats + 1, n_chunks);
        atomicAdd(a.stats + 2, tested);
        atomicAdd(a.stats + 3, s_stat[w][0]);
        atomicAdd(a.stats + 4, s_stat[w][1]);
        atomicAdd(a.stats + 7, n_tasks);
        // cycles spent on units (the autotuner's measure of a plan's work)
        if (kMulti) atomicAdd((unsigned long long*)(a.qctr + kQBusy), s_stat[w][2]);
    }
}

// ---------------------------------------------------------------------------
// dense level sums: W_k(x) for every vertex x of one level-sum position k of
// a plan (EdgePlan::sum_dense), computed children first before the DFS
// ---------------------------------------------------------------------------
struct WsumJob {
    uint32_t dir, dvis;  // G_k(x): the list of direction dir at x (delta part if dvis)
    uint32_t nt;         // pendant tails of k: lists of direction tdir at c (delta part if tvis)
    uint32_t tdir[cgb::kMaxSumTails], tvis[cgb::kMaxSumTails];
    uint32_t nch;        // positions owned by k: their sums at c
    const unsigned long long* child[cgb::kMaxSumChildren];
    unsigned long long* out;
};
constexpr uint32_t kWsumLane = 16;  // owners with lists up to this long are summed by one lane

// W(x) = sum over c in G(x) of (product of c's pendant list lengths) x
// (product of the children's W(c)), for every x < dv, for the job
// jobs[job0 + blockIdx.y] (the jobs of one launch are independent: their
// children are done).  Lane per owner for short lists (records read
// coalesced, 32 consecutive owners per warp), the whole warp for each longer
// one.
__global__ void k_wsum(const uint4* __restrict__ rec, uint32_t dvcap, const uint32_t* __restrict__ pool,
                       const uint32_t* __restrict__ dval, uint32_t dv, const WsumJob* __restrict__ jobs,
                       uint32_t job0) {
    __shared__ WsumJob sJ;
    static_assert(sizeof(WsumJob) % 4 == 0, "WsumJob is copied as words");
    for (uint32_t t = threadIdx.x; t < sizeof(WsumJob) / 4; t += blockDim.x)
        reinterpret_cast<uint32_t*>(&sJ)[t] = reinterpret_cast<const uint32_t*>(jobs + job0 + blockIdx.y)[t];
    __syncthreads();
    const WsumJob& J = sJ;
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    auto term = [&](uint32_t c) -> unsigned long long {
        unsigned long long v = 1;
#pragma unroll
        for (uint32_t i = 0; i < cgb::kMaxSumTails; ++i)
            if (i < J.nt) {
                const uint4 t = rec[(size_t)J.tdir[i] * dvcap + c];
                v *= (unsigned long long)t.y + (J.tvis[i] ? t.w : 0u);
            }
#pragma unroll
        for (uint32_t i = 0; i < cgb::kMaxSumChildren; ++i)
            if (i < J.nch) v *= __ldg(J.child[i] + c);
        return v;
    };
    for (uint64_t base = (((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) << 5; base < dv;
         base += nwarps * 32) {
        const uint64_t x = base + lane;
        uint4 r = make_uint4(0, 0, 0, 0);
        if (x < dv) {
            r = rec[(size_t)J.dir * dvcap + x];
            if (!J.dvis) r.w = 0;
        }
        const uint32_t len = r.y + r.w;
        unsigned long long acc = 0;
        if (len <= kWsumLane)
            for (uint32_t i = 0; i < len; ++i)
                acc += term(i < r.y ? __ldg(pool + r.x + i) : __ldg(dval + r.z + (i - r.y)));
        uint32_t big = __ballot_sync(kFull, len > kWsumLane);
        while (big) {
            const uint32_t i = __ffs(big) - 1;
            big &= big - 1;
            const uint32_t rx = __shfl_sync(kFull, r.x, i), ry = __shfl_sync(kFull, r.y, i);
            const uint32_t rz = __shfl_sync(kFull, r.z, i), rw = __shfl_sync(kFull, r.w, i);
            // four entries a lane and step: a hub's list is a chain of record
            // reads, and their latency is all there is to hide
            unsigned long long sv = 0;
            const uint32_t n = ry + rw;
            for (uint32_t t = lane; t < n; t += 128) {
                uint32_t c[4];
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) {
                    const uint32_t e = t + 32 * k;
                    c[k] = e < ry ? __ldg(pool + rx + e) : e < n ? __ldg(dval + rz + (e - ry)) : kNoVal;
                }
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k)
                    if (c[k] != kNoVal) sv += term(c[k]);
            }
            for (int o = 16; o > 0; o >>= 1) sv += __shfl_xor_sync(kFull, sv, o);
            if (lane == i) acc = sv;
        }
        if (x < dv) J.out[x] = acc;
    }
}

// ---------------------------------------------------------------------------
// valid bits (BuildLocalIndexBitAll with 1-bit masks, graph_gpu.cu:803-869,
// indexing.cu:2295-2379): vb[ei][u][w] holds bit (dv & 31) of word dv >> 5
// for query vertex u under query edge ei.  A sound superset of the vertices
// that some embedding mapping ei to a delta edge can place at u.
// ---------------------------------------------------------------------------
// Rebuilt (ei, u) start empty, the others all ones (graph_gpu.cu:818-828).
__global__ void k_vb_fill(const cgb::VbPlan* __restrict__ vbp, uint32_t* vb, uint32_t qe, uint32_t qv,
                          uint32_t stride) {
    const size_t n = (size_t)qe * qv * stride;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t ei = (uint32_t)(i / ((size_t)qv * stride));
        const uint32_t u = (uint32_t)((i / stride) % qv);
        vb[i] = ((vbp[ei].rebuild >> u) & 1u) ? 0u : 0xffffffffu;
    }
}

// Endpoints of ei: vertices with a delta list in ei's own direction
// (setInitialValidBitsAll1Bit, indexing.cu:2295-2317), set from the sorted
// packed delta keys (d << 2B | u << B | v): one bit per key, no full sweep.
__global__ void k_vb_seed(const cgb::VbPlan* __restrict__ vbp, const uint8_t* __restrict__ dir_edge,
                          const uint64_t* __restrict__ dkeys, uint64_t n, uint32_t B, uint32_t* vb, uint32_t qv,
                          uint32_t stride) {
    const uint64_t m = (1ull << B) - 1ull;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t k = dkeys[i];
        if (k == ~0ull) continue;  // a key out of range: the batch is rejected after this step
        const uint32_t d = (uint32_t)(k >> (2 * B)), u = (uint32_t)((k >> B) & m);
        const uint32_t ei = dir_edge[d];
        const cgb::VbPlan& P = vbp[ei];
        const uint32_t qu = d == P.d01 ? P.vs[0] : P.vs[1];
        atomicOr(vb + ((size_t)ei * qv + qu) * stride + (u >> 5), 1u << (u & 31));
    }
}

// Position `depth` of every query edge's indexing order (grid.y = ei): a
// vertex is valid if, for every backward neighbour, its list towards that
// neighbour (old run, plus the delta run when visible) holds a vertex whose
// bit is set (checkAllConstraintsAndSetBitsAll1Bit, indexing.cu:2319-2377).
// One warp per mask word, one lane per vertex.
__global__ void k_vb_depth(const cgb::VbPlan* __restrict__ vbp, const uint4* __restrict__ rec, uint32_t dvcap,
                           const uint32_t* __restrict__ pool, const uint32_t* __restrict__ dval, uint32_t dv,
                           uint32_t* vb, uint32_t qv, uint32_t stride, uint32_t depth) {
    const uint32_t ei = blockIdx.y;
    const cgb::VbPlan& P = vbp[ei];
    const uint32_t u = P.vs[depth];
    if (!((P.rebuild >> u) & 1u)) return;
    uint32_t* out = vb + ((size_t)ei * qv + u) * stride;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t wi = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; wi < stride; wi += nw) {
        const uint32_t x = wi * 32u + lane;
        bool valid = x < dv;
        for (uint32_t b = P.off[depth]; b < P.off[depth + 1] && valid; ++b) {
            const uint32_t* m1 = vb + ((size_t)ei * qv + P.vs[P.bpos[b]]) * stride;
            const uint4 r = rec[(size_t)P.bdir[b] * dvcap + x];
            bool sat = false;
            for (uint32_t t = 0; t < r.y && !sat; ++t) {
                const uint32_t nb = __ldg(pool + r.x + t);
                sat = (m1[nb >> 5] >> (nb & 31)) & 1u;
            }
            if (P.bvis[b])
                for (uint32_t t = 0; t < r.w && !sat; ++t) {
                    const uint32_t nb = __ldg(dval + r.z + t);
                    sat = (m1[nb >> 5] >> (nb & 31)) & 1u;
                }
            valid = sat;
        }
        const uint32_t word = __ballot_sync(kFull, valid);
        if (lane == 0) out[wi] = word;
    }
}

// ---------------------------------------------------------------------------
// maintenance kernels
// ---------------------------------------------------------------------------
__global__ void k_rec_sizes(const uint4* rec, uint32_t dvcap, uint32_t dv, uint32_t nd, uint32_t* out_round4) {
    uint64_t total = (uint64_t)nd * dv;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t d = (uint32_t)(i / dv), u = (uint32_t)(i % dv);
        uint32_t len = rec[(size_t)d * dvcap + u].y;
        out_round4[i] = round4(len);
    }
}

// Run lengths in (d, u) order, and a 0 after the last (scanned in place to offsets).
__global__ void k_rec_lens(const uint4* rec, uint32_t dvcap, uint32_t dv, uint32_t nd, unsigned long long* out) {
    const uint64_t total = (uint64_t)nd * dv;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= total; i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = i < total ? rec[(size_t)(i / dv) * dvcap + i % dv].y : 0;
}

// Copies every run to its compacted offset (warp per (d,u)).
__global__ void k_compact(uint4* rec, uint32_t dvcap, uint32_t dv, uint32_t nd, const uint32_t* src,
                          uint32_t* dst, const unsigned long long* new_off) {
    const uint32_t lane = threadIdx.x & 31;
    uint64_t total = (uint64_t)nd * dv;
    for (uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < total;
         i += ((uint64_t)gridDim.x * blockDim.x) >> 5) {
        uint32_t d = (uint32_t)(i / dv), u = (uint32_t)(i % dv);
        uint4* p = rec + (size_t)d * dvcap + u;
        uint4 r = *p;
        uint64_t no = new_off[i];
        for (uint32_t k = lane; k < r.y; k += 32) dst[no + k] = src[r.x + k];
        if (lane == 0) { r.x = (uint32_t)no; *p = r; }
    }
}

__global__ void k_dump(const uint4* rec, uint32_t dvcap, uint32_t dv, uint32_t nd, const uint32_t* pool,
                       const unsigned long long* off, uint64_t* out) {
    const uint32_t lane = threadIdx.x & 31;
    uint64_t total = (uint64_t)nd * dv;
    for (uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < total;
         i += ((uint64_t)gridDim.x * blockDim.x) >> 5) {
        uint32_t d = (uint32_t)(i / dv), u = (uint32_t)(i % dv);
        uint4 r = rec[(size_t)d * dvcap + u];
        uint64_t o = off[i];
        for (uint32_t k = lane; k < r.y; k += 32)
            out[o + k] = ((uint64_t)d << 59) | ((uint64_t)u << 32) | pool[r.x + k];
    }
}

__global__ void k_copy_rows(const uint4* src, uint32_t src_cap, uint4* dst, uint32_t dst_cap, uint32_t nd,
                            uint32_t dv) {
    uint64_t total = (uint64_t)nd * dv;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t d = (uint32_t)(i / dv), u = (uint32_t)(i % dv);
        dst[(size_t)d * dst_cap + u] = src[(size_t)d * src_cap + u];
    }
}

__global__ void k_u32_to_u64(const uint32_t* in, unsigned long long* out, uint64_t n) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = in[i];
}

inline uint32_t bits_for(uint32_t dv) {
    uint32_t b = 1;
    while ((1ull << b) < (uint64_t)dv) ++b;
    return b;
}

}  // namespace

// ===========================================================================
// host side
// ===========================================================================
struct cgb_handle {
    cgb_config cfg{};
    int device = 0;
    int num_sms = 148;
    int clock_khz = 0;      // asked for by the multi-query autotuner: a slow query
    int dfs_occupancy = 0;  // resident DFS blocks per SM
    uint32_t dfs_epoch = 0; // launch counter used as the task ready tag
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    std::string err;
    uint64_t launches = 0;

    // query
    bool have_query = false;
    cgb::QueryMeta q;
    EdgePlan plans[kMaxQE];
    EdgePlan* d_plans = nullptr;       // [kMaxQE] device copy of plans
    cgb::VbPlan* d_vbplans = nullptr;  // [kMaxQE] valid-bit plans
    uint8_t* d_dir_edge = nullptr;     // [kMaxDir] query edge of each direction
    uint8_t* d_qe_dirs = nullptr;  // [qe][2]
    uint8_t* d_edge_ok = nullptr;  // [kMaxQE]

    // index
    bool have_index = false;
    uint32_t nd = 0, dv = 0, dvcap = 0;
    uint4* rec = nullptr;
    uint32_t* pool = nullptr;
    uint32_t* pool_alt = nullptr;
    unsigned long long pool_cap = 0;
    // device scalars, one block (kCtl*): cleared by one memset from kCtlErr on
    // at every batch, read back by one copy
    unsigned long long* d_scal = nullptr;
    unsigned int* d_self = nullptr;  // sticky: some added key was a self-loop (u == v)
    unsigned long long* h_scal = nullptr;  // pinned mirror of d_scal
    unsigned long long h_pool_top = 0;
    long long h_live = 0;

    // per-batch buffers (grown on demand)
    uint64_t* d_keys_in = nullptr; size_t keys_in_cap = 0;       // uploaded ext keys (ins|del|delta)
    uint64_t* d_pending = nullptr; size_t pending_cap = 0; uint64_t n_pending = 0;  // delta keys to merge back, packed (d,u,v) and sorted by run
    uint32_t pending_B = 0;
    uint64_t* d_edits = nullptr; uint64_t* d_edits_alt = nullptr; size_t edits_cap = 0;
    uint2* d_runs[3] = {nullptr, nullptr, nullptr};  // merge lists (k_edit_runs)
    unsigned int* d_list_ctr = nullptr;  // MergeArgs::list_ctr, and [3] bit-set slots claimed by the last merge
    unsigned long long* d_big_off = nullptr; size_t big_off_cap = 0;
    uint32_t* d_big_tile0 = nullptr; size_t big_tile0_cap = 0;
    uint2* d_tiles = nullptr; size_t tiles_cap = 0;
    unsigned long long* d_tile_state = nullptr; size_t tile_state_cap = 0;
    uint64_t unsynced_edits = 0;  // edits merged since h_live and h_pool_top were read
    unsigned long long unsynced_need = 0;  // pool words those merges take at most
    uint64_t* d_dkeys = nullptr; uint64_t* d_dkeys_alt = nullptr; size_t dkeys_cap = 0;
    uint32_t* d_dval = nullptr;
    uint32_t* d_seed = nullptr;  // [0..kMaxQE) lo, [kMaxQE..2kMaxQE+1) pre
    unsigned long long* d_counts = nullptr;  // [kMaxQE]
    unsigned long long* d_stats = nullptr;   // [8]
    uint32_t* d_tasks = nullptr;             // stolen-range queue
    unsigned int* d_qctr = nullptr;          // DFS queue counters [kQWords]
    unsigned long long last_stats[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    void* d_temp = nullptr; size_t temp_cap = 0;
    unsigned long long* d_read_off = nullptr; size_t read_off_cap = 0;  // cgb_read_index
    uint64_t* d_read = nullptr; size_t read_cap = 0;

    // run bit sets: built in full on the first matched batch (and after the
    // record table grows), then kept current by every merge
    uint32_t* d_rb_slot = nullptr; size_t rb_slot_cap = 0;  // [nd][dvcap]
    uint32_t* d_rb_sel = nullptr; size_t rb_sel_cap = 0;
    uint32_t* d_rb_bits = nullptr; size_t rb_bits_cap = 0;
    uint32_t* d_rb_new = nullptr; size_t rb_new_cap = 0;    // slots claimed by the last merge
    unsigned int* d_rb_ctr = nullptr;  // slots claimed
    uint32_t rb_words = 0;             // words per bit set: (dvcap + 31) / 32
    uint32_t rb_cap = 0;               // bit sets the budget holds
    bool rb_valid = false;             // slot table and bit sets match the index
    uint32_t rb_min_len = kRunBitsMinLen;
    uint32_t rb_len_now = kRunBitsMinLen;  // doubled while the budget holds too few slots
    uint32_t pair_lane_max = kPairLaneMax;
    uint8_t* d_rev = nullptr;          // reverse direction of each direction
    uint32_t* d_touched = nullptr; size_t touched_cap = 0;  // footprint runs: record bit set
    unsigned long long* d_memo = nullptr;  // subtree memos [memo_slots][4], sized with the record table
    uint32_t* d_memo_list = nullptr;
    uint32_t memo_slots = 0;
    unsigned long long* d_lsum = nullptr;  // level-sum table, sized with the record table
    uint32_t lsum_slots = 0;
    unsigned long long* d_wsum = nullptr; size_t wsum_cap = 0;  // dense level sums [n_wsum][dvcap]
    uint32_t n_wsum = 0;
    WsumJob* d_wjobs = nullptr;                 // [n_wsum] jobs, ordered by height (children first)
    std::vector<uint32_t> wjob_level;           // job offsets of each height (size = heights + 1)
    const void* wjobs_for = nullptr;            // d_wsum the jobs were built for

    // label-keyed mode (the multi-query engine's data-graph index): the
    // "direction" of a key is the label of its target vertex, the delta keys
    // carry the source vertex's label (lb bits) between direction and source
    bool mq = false;
    uint32_t lb = 0;
    uint8_t* d_vlabel = nullptr;       // [dv] vertex labels
    unsigned int* d_epoch = nullptr;   // DFS launch tag read by replayed graphs

    // valid bits
    uint32_t vb_start[2] = {0, 0};   // starting edge (SelectStartingEdge)
    std::string vb_plan_error;       // set when the pattern has no consistent rebuild flags
    uint32_t* d_vb = nullptr; size_t vb_cap = 0;
    uint32_t vb_stride = 0;          // words per (ei, u) of the last matched batch; 0 = none
    float last_vb_ms = 0;

    uint64_t last_counts[kMaxQE] = {0};
    float last_t[4] = {0, 0, 0, 0};
    cudaEvent_t ev[7] = {};  // phases 0-3, caller-stream order 4, end 5, valid bits 6
};

namespace {

// Words of cgb_handle::d_scal.  The first three live as long as the handle.
constexpr uint32_t kCtlPoolTop = 0, kCtlLive = 1, kCtlRbClaimed = 2, kCtlErr = 3, kCtlWork = 4, kCtlList = 5,
                   kCtlStats = 8, kCtlCounts = 16, kCtlQueue = kCtlCounts + kMaxQE, kCtlWords = kCtlQueue + kQWords / 2;
static_assert(kCtlQueue % 16 == 0, "the polled queue counters start a 128-byte line");

cgb_status fail(cgb_handle* h, cgb_status s, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    if (h) h->err = buf;
    return s;
}

#define CK(call)                                                                                 \
    do {                                                                                         \
        cudaError_t e_ = (call);                                                                 \
        if (e_ != cudaSuccess) {                                                                 \
            return fail(h, e_ == cudaErrorMemoryAllocation ? CGB_ERR_OOM : CGB_ERR_CUDA,         \
                        "%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); \
        }                                                                                        \
    } while (0)

#define LAUNCHED() (h->launches++)

template <typename T>
cgb_status grow(cgb_handle* h, T*& p, size_t& cap, size_t need) {
    if (need <= cap && p) return CGB_OK;
    size_t nc = std::max<size_t>(need + need / 2, 1024);
    if (p) CK(cudaFree(p));
    p = nullptr;
    CK(cgb::device_malloc(&p, nc * sizeof(T)));
    cap = nc;
    return CGB_OK;
}

cgb_status grow_temp(cgb_handle* h, size_t need) {
    if (need <= h->temp_cap && h->d_temp) return CGB_OK;
    size_t nc = std::max<size_t>(need + need / 2, 1 << 20);
    if (h->d_temp) CK(cudaFree(h->d_temp));
    h->d_temp = nullptr;
    CK(cgb::device_malloc(&h->d_temp, nc));
    h->temp_cap = nc;
    return CGB_OK;
}

inline int grid_for(const cgb_handle* h, uint64_t n, int block = 256) {
    uint64_t g = (n + block - 1) / block;
    uint64_t cap = (uint64_t)h->num_sms * 8;
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    return (int)g;
}

// Level-sum table: about two slots per vertex, 2^12 to 2^24 slots (16 B each);
// subtree memos: up to 2^20 slots (32 B each), emptied by the launches that
// use them.  A table counts as there by its number of slots, which is set last:
// after a failed allocation the next call tries again.
cgb_status ensure_tables(cgb_handle* h) {
    uint32_t slots = 1u << 12;
    while (slots < (1u << 24) && slots < 2ull * h->dvcap) slots <<= 1;
    if (slots > h->lsum_slots) {
        h->lsum_slots = 0;
        if (h->d_lsum) CK(cudaFree(h->d_lsum));
        h->d_lsum = nullptr;
        CK(cgb::device_malloc(&h->d_lsum, (size_t)slots * 2 * sizeof(unsigned long long)));
        h->lsum_slots = slots;
    }
    slots = std::min(slots, 1u << 20);
    if (slots > h->memo_slots) {
        CK(cudaStreamSynchronize(h->stream));
        h->memo_slots = 0;
        if (h->d_memo) CK(cudaFree(h->d_memo));
        h->d_memo = nullptr;
        if (h->d_memo_list) CK(cudaFree(h->d_memo_list));
        h->d_memo_list = nullptr;
        CK(cgb::device_malloc(&h->d_memo, (size_t)slots * 4 * sizeof(unsigned long long)));
        CK(cgb::device_malloc(&h->d_memo_list, (size_t)slots * sizeof(uint32_t)));
        CK(cudaMemsetAsync(h->d_memo, 0, (size_t)slots * 4 * sizeof(unsigned long long), h->stream));
        h->memo_slots = slots;
    }
    return CGB_OK;
}

cgb_status ensure_dvcap(cgb_handle* h, uint32_t dv) {
    if (dv <= h->dvcap && h->rec) return ensure_tables(h);
    uint32_t nc = std::max<uint32_t>(dv + dv / 4 + 1024, h->dvcap * 2);
    uint4* nr = nullptr;
    CK(cgb::device_malloc(&nr, (size_t)h->nd * nc * sizeof(uint4)));
    CK(cudaMemsetAsync(nr, 0, (size_t)h->nd * nc * sizeof(uint4), h->stream));
    if (h->rec) {
        k_copy_rows<<<grid_for(h, (uint64_t)h->nd * h->dv), 256, 0, h->stream>>>(h->rec, h->dvcap, nr, nc, h->nd,
                                                                                   h->dv);
        LAUNCHED();
        CK(cudaGetLastError());
        CK(cudaStreamSynchronize(h->stream));
        CK(cudaFree(h->rec));
    }
    h->rec = nr;
    h->dvcap = nc;
    h->rb_valid = false;  // the slot table and the bit sets follow the record layout
    h->wjobs_for = nullptr;  // so do the arrays in the level-sum jobs, wherever d_wsum lies
    h->rb_len_now = h->rb_min_len;
    return ensure_tables(h);
}

// Dense level sums of every plan with sum_dense, children before parents
// (a position's children sit at higher positions), on the stream.
// The jobs are built (and uploaded) when the arrays move; one launch per
// height runs every job of that height of every plan.
cgb_status dense_level_sums(cgb_handle* h) {
    cgb_status s;
    if ((s = grow(h, h->d_wsum, h->wsum_cap, (size_t)h->n_wsum * h->dvcap)) != CGB_OK) return s;
    if (h->wjobs_for != h->d_wsum) {
        std::vector<std::vector<WsumJob>> by_height;
        for (uint32_t e = 0; e < h->q.qe; ++e) {
            const EdgePlan& P = h->plans[e];
            if (!P.sum_dense) continue;
            const uint32_t s0 = P.sum_from, nc = P.n_core;
            auto arr = [&](uint32_t k) { return h->d_wsum + (size_t)(P.wslot + k - s0) * h->dvcap; };
            uint32_t height[cgb::kMaxQV] = {0};
            for (uint32_t k = nc; k-- > s0;) {  // children sit at higher positions
                WsumJob J;
                std::memset(&J, 0, sizeof(J));
                J.dir = P.bn_dir[P.bn_off[k]];
                J.dvis = P.bn_dvis[P.bn_off[k]];
                for (uint32_t t = nc; t < P.n; ++t)
                    if (((P.sum_tails >> t) & 1u) && P.bn_pos[P.bn_off[t]] == k) {
                        J.tdir[J.nt] = P.bn_dir[P.bn_off[t]];
                        J.tvis[J.nt] = P.bn_dvis[P.bn_off[t]];
                        ++J.nt;
                    }
                for (uint32_t l = k + 1; l < nc; ++l)
                    if (P.bn_pos[P.bn_off[l]] == k) {
                        J.child[J.nch++] = arr(l);
                        height[k] = std::max(height[k], height[l] + 1);
                    }
                J.out = arr(k);
                if (by_height.size() <= height[k]) by_height.resize(height[k] + 1);
                by_height[height[k]].push_back(J);
            }
        }
        std::vector<WsumJob> all;
        h->wjob_level.assign(1, 0);
        for (auto& v : by_height) {
            all.insert(all.end(), v.begin(), v.end());
            h->wjob_level.push_back((uint32_t)all.size());
        }
        if (h->d_wjobs) CK(cudaFree(h->d_wjobs));
        h->d_wjobs = nullptr;
        CK(cgb::device_malloc(&h->d_wjobs, std::max<size_t>(all.size(), 1) * sizeof(WsumJob)));
        CK(cudaMemcpy(h->d_wjobs, all.data(), all.size() * sizeof(WsumJob), cudaMemcpyHostToDevice));
        h->wjobs_for = h->d_wsum;
    }
    for (size_t lv = 0; lv + 1 < h->wjob_level.size(); ++lv) {
        const uint32_t j0 = h->wjob_level[lv], nj = h->wjob_level[lv + 1] - j0;
        if (!nj) continue;
        const dim3 grid((unsigned)std::max<uint32_t>((uint32_t)h->num_sms * 2, (uint32_t)h->num_sms * 8 / nj), nj);
        k_wsum<<<grid, 256, 0, h->stream>>>(h->rec, h->dvcap, h->pool, h->d_dval, h->dv, h->d_wjobs, j0);
        LAUNCHED();
    }
    CK(cudaGetLastError());
    return CGB_OK;
}

// Level-sum table of a DFS launch (none when no plan uses level sums), zeroed
// by lsum_clear on the stream before each launch, and its subtree memos,
// multiplied into the counts by memo_finish after it.
void lsum_bind(const cgb_handle* h, bool any_sum, bool any_memo, DfsArgs& da) {
    const bool on = any_sum && h->lsum_slots;
    da.lsum_tab = on ? h->d_lsum : nullptr;
    da.lsum_mask = on ? h->lsum_slots - 1 : 0;
    const bool memo = any_memo && h->memo_slots;
    da.memo_tab = memo ? h->d_memo : nullptr;
    da.memo_mask = memo ? h->memo_slots - 1 : 0;
    da.memo_list = h->d_memo_list;
}
cgb_status lsum_clear(cgb_handle* h, const DfsArgs& da) {
    if (da.lsum_tab)
        CK(cudaMemsetAsync(da.lsum_tab, 0, ((size_t)da.lsum_mask + 1) * 2 * sizeof(unsigned long long), h->stream));
    return CGB_OK;
}
cgb_status memo_finish(cgb_handle* h, const DfsArgs& da) {
    if (da.memo_tab) {
        k_memo_finish<<<h->num_sms, 256, 0, h->stream>>>(da.memo_tab, da.memo_list, da.qctr + kQMemo, da.counts);
        LAUNCHED();
        CK(cudaGetLastError());
    }
    return CGB_OK;
}

// Compacts the pool into pool_alt (allocating or growing it to new_cap words)
// and swaps.  Synchronous.
cgb_status compact_pool(cgb_handle* h, unsigned long long new_cap) {
    const uint64_t n = (uint64_t)h->nd * h->dv;
    if (new_cap < h->pool_cap) new_cap = h->pool_cap;
    uint32_t* sizes = nullptr;
    unsigned long long* offs = nullptr;
    unsigned long long live = 0;
    CK(cgb::device_malloc(&sizes, std::max<uint64_t>(n, 1) * sizeof(uint32_t)));
    CK(cgb::device_malloc(&offs, (n + 1) * sizeof(unsigned long long)));
    CK(cudaMemsetAsync(offs, 0, (n + 1) * sizeof(unsigned long long), h->stream));
    if (n > 0) {
        k_rec_sizes<<<grid_for(h, n), 256, 0, h->stream>>>(h->rec, h->dvcap, h->dv, h->nd, sizes);
        LAUNCHED();
        k_u32_to_u64<<<grid_for(h, n), 256, 0, h->stream>>>(sizes, offs, n);
        LAUNCHED();
    }
    size_t tb = 0;
    CK(cub::DeviceScan::ExclusiveSum(nullptr, tb, offs, offs, (int64_t)n + 1, h->stream));
    if (grow_temp(h, tb) != CGB_OK) return CGB_ERR_OOM;
    CK(cub::DeviceScan::ExclusiveSum(h->d_temp, tb, offs, offs, (int64_t)n + 1, h->stream));
    LAUNCHED();
    CK(cudaMemcpyAsync(&live, offs + n, sizeof(live), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    // the destination must hold every live run plus the headroom requested
    while (new_cap < live + (16ull << 20)) new_cap *= 2;
    uint32_t* dst = nullptr;
    if (h->pool_alt && new_cap == h->pool_cap) {
        dst = h->pool_alt;
    } else {
        if (h->pool_alt) CK(cudaFree(h->pool_alt));
        h->pool_alt = nullptr;
        CK(cgb::device_malloc(&dst, new_cap * sizeof(uint32_t)));
    }
    if (n > 0) {
        k_compact<<<grid_for(h, n * 32), 256, 0, h->stream>>>(h->rec, h->dvcap, h->dv, h->nd, h->pool, dst, offs);
        LAUNCHED();
        CK(cudaGetLastError());
    }
    CK(cudaStreamSynchronize(h->stream));
    CK(cudaFree(sizes));
    CK(cudaFree(offs));
    uint32_t* old = h->pool;
    h->pool = dst;
    if (new_cap == h->pool_cap) {
        h->pool_alt = old;
    } else {
        CK(cudaFree(old));
        h->pool_alt = nullptr;
        h->pool_cap = new_cap;
    }
    h->h_pool_top = live;
    h->h_live = (long long)live;
    h->unsynced_edits = 0;
    h->unsynced_need = 0;
    unsigned long long sc[2] = {live, live};  // kCtlPoolTop, kCtlLive
    CK(cudaMemcpyAsync(h->d_scal, sc, sizeof(sc), cudaMemcpyHostToDevice, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return CGB_OK;
}

cgb_status sync_scalars(cgb_handle* h);

// Ensures the pool can absorb a merge of n_edits edits in the worst case: every
// run is written anew.  The pool's top is known as of the last read-back; the
// merges enqueued since count by their own worst case, and where that says no
// the pool is asked.
cgb_status reserve_pool(cgb_handle* h, uint64_t n_edits) {
    cgb_status s;
    auto need = [&] {
        return (unsigned long long)std::max<long long>(h->h_live, 0) + 4ull * (h->unsynced_edits + n_edits) + 64;
    };
    if (h->unsynced_need && h->h_pool_top + h->unsynced_need + need() > h->pool_cap &&
        (s = sync_scalars(h)) != CGB_OK)
        return s;
    if (h->h_pool_top + h->unsynced_need + need() <= h->pool_cap) {
        h->unsynced_need += need();
        return CGB_OK;
    }
    unsigned long long cap = h->pool_cap;
    while ((unsigned long long)std::max<long long>(h->h_live, 0) + need() > cap * 3 / 4) cap = cap * 2;
    if ((s = compact_pool(h, cap)) != CGB_OK) return s;
    h->unsynced_need = need();
    return CGB_OK;
}

// Sorts packed keys in place (alt buffer used as ping-pong); returns sorted pointer.
cgb_status radix_sort(cgb_handle* h, uint64_t*& keys, uint64_t*& alt, uint64_t n, int begin_bit, int end_bit) {
    if (n == 0) return CGB_OK;
    cub::DoubleBuffer<uint64_t> db(keys, alt);
    size_t tb = 0;
    CK(cub::DeviceRadixSort::SortKeys(nullptr, tb, db, (int64_t)n, begin_bit, end_bit, h->stream));
    if (grow_temp(h, tb) != CGB_OK) return CGB_ERR_OOM;
    CK(cub::DeviceRadixSort::SortKeys(h->d_temp, tb, db, (int64_t)n, begin_bit, end_bit, h->stream));
    LAUNCHED();
    if (db.Current() != keys) std::swap(keys, alt);
    return CGB_OK;
}

// Grow-only per-batch buffers (reallocated only when a batch is larger than any before).
cgb_status ensure_edit_buffers(cgb_handle* h, uint64_t n) {
    if (n <= h->edits_cap && h->d_edits) return CGB_OK;
    size_t nc = std::max<size_t>(n + n / 2, 1 << 16);
    CK(cudaStreamSynchronize(h->stream));
    void* olds[] = {h->d_edits, h->d_edits_alt, h->d_runs[0], h->d_runs[1], h->d_runs[2]};
    for (void* p : olds) if (p) CK(cudaFree(p));
    for (auto& p : h->d_runs) p = nullptr;
    h->d_edits = h->d_edits_alt = nullptr;
    h->edits_cap = 0;
    CK(cgb::device_malloc(&h->d_edits, nc * sizeof(uint64_t)));
    CK(cgb::device_malloc(&h->d_edits_alt, nc * sizeof(uint64_t)));
    for (auto& p : h->d_runs) CK(cgb::device_malloc(&p, nc * sizeof(uint2)));
    h->edits_cap = nc;
    return CGB_OK;
}

// The kept delta's buffer is one of them (same size: it changes places with
// the sorted keys after a batch); it is free here, merged back before.
cgb_status ensure_delta_buffers(cgb_handle* h, uint64_t n) {
    if (n <= h->dkeys_cap && h->d_dkeys) return CGB_OK;
    size_t nc = std::max<size_t>(n + n / 2, 1 << 16);
    CK(cudaStreamSynchronize(h->stream));
    void* olds[] = {h->d_dkeys, h->d_dkeys_alt, h->d_pending, h->d_dval};
    for (void* p : olds) if (p) CK(cudaFree(p));
    h->d_dkeys = h->d_dkeys_alt = h->d_pending = nullptr;
    h->d_dval = nullptr;
    h->dkeys_cap = h->pending_cap = 0;
    CK(cgb::device_malloc(&h->d_pending, nc * sizeof(uint64_t)));
    CK(cgb::device_malloc(&h->d_dkeys, nc * sizeof(uint64_t)));
    CK(cgb::device_malloc(&h->d_dkeys_alt, nc * sizeof(uint64_t)));
    CK(cgb::device_malloc(&h->d_dval, nc * sizeof(uint32_t)));
    h->dkeys_cap = h->pending_cap = nc;
    return CGB_OK;
}

// Applies the edits to the index.  Packed edits alone are in run order already
// (they were sorted as a delta) and are not sorted again.
cgb_status apply_edits(cgb_handle* h, const EditSrc& src) {
    const uint64_t n = src.n_packed + src.n_add + src.n_rem;
    if (n == 0) return CGB_OK;
    cgb_status s;
    if ((s = reserve_pool(h, n)) != CGB_OK) return s;
    if ((s = ensure_edit_buffers(h, n)) != CGB_OK) return s;
    PackInfo pi{bits_for(h->dv), h->nd, h->dv, h->mq ? 1u : 0u};
    unsigned int* d_err = (unsigned int*)(h->d_scal + kCtlErr);
    k_pack_edits<<<grid_for(h, n), 256, 0, h->stream>>>(src, pi, h->d_edits, d_err, h->d_self);
    LAUNCHED();
    CK(cudaGetLastError());
    // by (d,u,v), and one bit more that makes the all-ones invalid marker sort
    // last; the op bit is left out: the sort is stable and adds come first
    if (src.n_add + src.n_rem)
        if ((s = radix_sort(h, h->d_edits, h->d_edits_alt, n, 1, 2 * (int)pi.B + (int)bits_for(h->nd) + 2)) != CGB_OK)
            return s;
    // tiled runs and tiles this merge can list at most: every run entry in the
    // index (and those merged since the last read-back) and every edit
    const uint64_t entries = (uint64_t)std::max<long long>(h->h_live, 0) + 4 * h->unsynced_edits + n;
    h->unsynced_edits += n;
    const uint64_t big_cap = std::min<uint64_t>(entries / kBigRun, n) + 1;
    const uint64_t tile_cap = std::min<uint64_t>(entries / kMergeTile + big_cap, 1u << 30);
    if ((s = grow(h, h->d_big_off, h->big_off_cap, (size_t)big_cap)) != CGB_OK) return s;
    if ((s = grow(h, h->d_big_tile0, h->big_tile0_cap, (size_t)big_cap)) != CGB_OK) return s;
    if ((s = grow(h, h->d_tiles, h->tiles_cap, (size_t)tile_cap)) != CGB_OK) return s;
    if ((s = grow(h, h->d_tile_state, h->tile_state_cap, (size_t)tile_cap)) != CGB_OK) return s;
    MergeArgs ma;
    ma.big_off = h->d_big_off;
    ma.big_tile0 = h->d_big_tile0;
    ma.big_cap = (uint32_t)big_cap;
    ma.tiles = h->d_tiles;
    ma.tile_state = h->d_tile_state;
    ma.tile_cap = (uint32_t)tile_cap;
    ma.rec = h->rec;
    ma.dvcap = h->dvcap;
    ma.pool = h->pool;
    ma.pool_top = h->d_scal + kCtlPoolTop;
    ma.pool_cap = h->pool_cap;
    ma.live_words = (long long*)(h->d_scal + kCtlLive);
    ma.edits = h->d_edits;
    ma.n = n;
    for (int k = 0; k < 3; ++k) ma.runs[k] = h->d_runs[k];
    ma.list_ctr = h->d_list_ctr;
    ma.B = pi.B;
    ma.err = d_err;
    ma.stats = h->d_stats;
    // bit sets are kept current by the merge once built (k_rb_update)
    const bool rb = h->rb_valid && !(h->cfg.flags & CGB_FLAG_NO_RUN_BITS);
    ma.rb_slot = rb ? h->d_rb_slot : nullptr;
    ma.rb_sel = h->d_rb_sel;
    ma.rb_ctr = h->d_rb_ctr;
    ma.rb_newc = h->d_list_ctr + 3;
    ma.rb_cap = h->rb_cap;
    ma.rb_min_len = h->rb_len_now;
    if (rb && (s = grow(h, h->d_rb_new, h->rb_new_cap, std::max<size_t>(h->rb_cap, 1))) != CGB_OK) return s;
    ma.rb_new = h->d_rb_new;
    CK(cudaMemsetAsync(h->d_list_ctr, 0, 6 * sizeof(unsigned int), h->stream));
    CK(cudaMemsetAsync(h->d_tile_state, 0, tile_cap * sizeof(unsigned long long), h->stream));
    k_edit_runs<<<grid_for(h, n), 256, 0, h->stream>>>(ma);
    LAUNCHED();
    // a warp per run at most, up to the blocks that can be resident; a block per SM for the tiles
    const int mg = std::max(h->num_sms, (int)std::min<uint64_t>((n * 32 + 255) / 256, (uint64_t)h->num_sms * 8));
    k_merge<<<mg, kMergeThreads, 0, h->stream>>>(ma);
    LAUNCHED();
    if (rb) {
        k_rb_update<<<std::max(grid_for(h, n), h->num_sms), 256, 0, h->stream>>>(
            h->rec, h->dvcap, h->pool, h->d_rb_sel, h->d_rb_new, h->d_list_ctr + 3, h->d_rb_bits, h->rb_words,
            h->d_edits, n, pi.B, h->d_rb_slot);
        LAUNCHED();
    }
    CK(cudaGetLastError());
    return CGB_OK;
}

// Builds the run bit sets in full: a slot for every run of at least
// rb_min_len entries while the budget lasts (later merges keep them current).
cgb_status rebuild_run_bits(cgb_handle* h) {
    cgb_status s;
    h->rb_words = (h->dvcap + 31) / 32;
    // as many bit sets as the budget holds, never more than records exist
    h->rb_cap = (uint32_t)std::min<size_t>(kRunBitsBytes / 4 / std::max(h->rb_words, 1u),
                                           std::max<size_t>((size_t)h->nd * h->dvcap, 1));
    const uint32_t cap = h->rb_cap;
    if ((s = grow(h, h->d_rb_slot, h->rb_slot_cap, (size_t)h->nd * h->dvcap)) != CGB_OK) return s;
    if ((s = grow(h, h->d_rb_sel, h->rb_sel_cap, (size_t)cap)) != CGB_OK) return s;
    if ((s = grow(h, h->d_rb_bits, h->rb_bits_cap, (size_t)cap * h->rb_words)) != CGB_OK) return s;
    CK(cudaMemsetAsync(h->d_rb_ctr, 0, sizeof(unsigned int), h->stream));
    k_rb_select<<<grid_for(h, (uint64_t)h->nd * h->dvcap), 256, 0, h->stream>>>(
        h->rec, h->dvcap, h->nd, h->rb_len_now, cap, h->d_rb_slot, h->d_rb_sel, h->d_rb_ctr);
    LAUNCHED();
    k_rb_zero<<<h->num_sms * 8, 256, 0, h->stream>>>(h->d_rb_bits, h->rb_words, cap, h->d_rb_ctr);
    LAUNCHED();
    k_rb_fill<<<h->num_sms * 8, 256, 0, h->stream>>>(h->rec, h->dvcap, h->pool, h->d_rb_sel, cap, h->d_rb_ctr,
                                                     h->d_rb_bits, h->rb_words);
    LAUNCHED();
    CK(cudaGetLastError());
    h->rb_valid = true;
    return CGB_OK;
}

cgb_status sync_scalars(cgb_handle* h) {
    CK(cudaMemcpyAsync(h->h_scal, h->d_scal, kCtlQueue * sizeof(unsigned long long), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    // every slot claimed: rebuild on the next batch with runs of twice the
    // length, so the longest runs of the index get them (at one length the
    // sets were rebuilt on every batch: 0.55 ms of a 16 ms batch on R-MAT
    // 2M/17M with 32 labels)
    if (h->rb_valid && (uint32_t)h->h_scal[kCtlRbClaimed] >= h->rb_cap) {
        h->rb_valid = false;
        if (h->rb_len_now < (1u << 26)) h->rb_len_now *= 2;
    }
    h->h_pool_top = h->h_scal[kCtlPoolTop];
    h->h_live = (long long)h->h_scal[kCtlLive];
    h->unsynced_edits = 0;
    h->unsynced_need = 0;
    return CGB_OK;
}

cgb_status flush_pending(cgb_handle* h) {
    if (h->n_pending == 0) return CGB_OK;
    EditSrc src;
    src.packed = h->d_pending;
    src.n_packed = h->n_pending;
    src.B0 = h->pending_B;
    cgb_status s = apply_edits(h, src);
    if (s != CGB_OK) return s;
    h->n_pending = 0;
    return sync_scalars(h);
}

}  // namespace

extern "C" {

void cgb_default_config(cgb_config* cfg) {
    if (!cfg) return;
    std::memset(cfg, 0, sizeof(*cfg));
}

cgb_status cgb_create(const cgb_config* cfg, cgb_handle** out) {
    if (!out) return CGB_ERR_ARG;
    *out = nullptr;
    cgb_handle* h = new cgb_handle();
    if (cfg) h->cfg = *cfg; else cgb_default_config(&h->cfg);
    h->device = h->cfg.device;
    if (const char* e = std::getenv("CGB_RUN_BITS_MIN_LEN")) h->rb_len_now = h->rb_min_len = (uint32_t)std::max(1l, std::atol(e));
    if (const char* e = std::getenv("CGB_PAIR_LANE_MAX")) h->pair_lane_max = (uint32_t)std::max(0l, std::atol(e));
    int ndev = 0;
    cudaError_t e = cudaGetDeviceCount(&ndev);
    if (e != cudaSuccess || ndev == 0) {
        cgb_status s = fail(h, CGB_ERR_CUDA, "no CUDA device: %s", cudaGetErrorString(e));
        *out = h;
        return s;
    }
    if (h->device < 0 || h->device >= ndev) { *out = h; return fail(h, CGB_ERR_ARG, "bad device %d", h->device); }
#define CKC(call) do { cudaError_t e_ = (call); if (e_ != cudaSuccess) { *out = h; return fail(h, CGB_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); } } while (0)
    CKC(cudaSetDevice(h->device));
    CKC(cudaDeviceGetAttribute(&h->num_sms, cudaDevAttrMultiProcessorCount, h->device));
    CKC(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking));
    h->own_stream = true;
    CKC(cgb::device_malloc(&h->d_scal, kCtlWords * sizeof(unsigned long long)));
    CKC(cudaMemset(h->d_scal, 0, kCtlWords * sizeof(unsigned long long)));
    h->d_rb_ctr = (unsigned int*)(h->d_scal + kCtlRbClaimed);
    h->d_list_ctr = (unsigned int*)(h->d_scal + kCtlList);
    h->d_stats = h->d_scal + kCtlStats;
    h->d_counts = h->d_scal + kCtlCounts;
    h->d_qctr = (unsigned int*)(h->d_scal + kCtlQueue);
    CKC(cgb::device_malloc(&h->d_self, sizeof(unsigned int)));
    CKC(cudaMemset(h->d_self, 0, sizeof(unsigned int)));
    CKC(cudaMallocHost(&h->h_scal, kCtlWords * sizeof(unsigned long long)));
    CKC(cgb::device_malloc(&h->d_rev, kMaxDir));
    CKC(cgb::device_malloc(&h->d_seed, (3 * kMaxQE + 2) * sizeof(uint32_t)));
    CKC(cgb::device_malloc(&h->d_tasks, (size_t)kTaskCap * kTaskWords * sizeof(uint32_t)));
    CKC(cudaMemset(h->d_tasks, 0, (size_t)kTaskCap * kTaskWords * sizeof(uint32_t)));
    CKC(cgb::device_malloc(&h->d_qe_dirs, 2 * kMaxQE));
    CKC(cgb::device_malloc(&h->d_edge_ok, kMaxQE));
    CKC(cgb::device_malloc(&h->d_plans, sizeof(EdgePlan) * kMaxQE));
    CKC(cgb::device_malloc(&h->d_vbplans, sizeof(cgb::VbPlan) * kMaxQE));
    CKC(cgb::device_malloc(&h->d_dir_edge, kMaxDir));
    for (auto& ev : h->ev) CKC(cudaEventCreate(&ev));
#undef CKC
    *out = h;
    return CGB_OK;
}

void cgb_destroy(cgb_handle* h) {
    if (!h) return;
    cudaSetDevice(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    void* ptrs[] = {h->rec, h->pool, h->pool_alt, h->d_scal, h->d_self, h->d_keys_in, h->d_pending, h->d_edits,
                    h->d_edits_alt, h->d_runs[0], h->d_runs[1], h->d_runs[2],
                    h->d_dkeys, h->d_dkeys_alt, h->d_dval,
                    h->d_seed, h->d_tasks, h->d_temp, h->d_read_off, h->d_read, h->d_big_off, h->d_big_tile0, h->d_tiles,
                    h->d_tile_state, h->d_memo, h->d_memo_list, h->d_qe_dirs, h->d_edge_ok,
                    h->d_vb, h->d_rb_slot, h->d_rb_sel, h->d_rb_bits, h->d_rb_new, h->d_rev, h->d_touched, h->d_plans,
                    h->d_vbplans, h->d_dir_edge, h->d_lsum, h->d_wsum, h->d_wjobs};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    if (h->h_scal) cudaFreeHost(h->h_scal);
    for (auto& ev : h->ev)
        if (ev) cudaEventDestroy(ev);
    if (h->own_stream && h->stream) cudaStreamDestroy(h->stream);
    delete h;
}

const char* cgb_last_error(const cgb_handle* h) { return h ? h->err.c_str() : "null handle"; }

cgb_status cgb_load_query(cgb_handle* h, uint32_t qv, const uint32_t* labels, uint32_t qe, const uint32_t* edges) {
    if (!h || !edges) return CGB_ERR_ARG;
    if (h->have_index) return fail(h, CGB_ERR_STATE, "query must be loaded before the index");
    std::string e = cgb::build_query_meta(qv, qe, edges, labels, h->q);
    if (!e.empty()) return fail(h, CGB_ERR_ARG, "%s", e.c_str());
    h->nd = h->q.nd;
    uint8_t dirs[2 * kMaxQE];
    for (uint32_t i = 0; i < h->q.qe; ++i) { dirs[2 * i] = h->q.qe_dir[i][0]; dirs[2 * i + 1] = h->q.qe_dir[i][1]; }
    CK(cudaSetDevice(h->device));
    CK(cudaMemcpy(h->d_qe_dirs, dirs, 2 * h->q.qe, cudaMemcpyHostToDevice));
    uint8_t rev[kMaxDir];
    std::memset(rev, 255, sizeof(rev));
    for (uint32_t d = 0; d < h->q.nd; ++d) rev[d] = h->q.eidx[h->q.dir_dst[d] * kMaxQV + h->q.dir_src[d]];
    CK(cudaMemcpy(h->d_rev, rev, kMaxDir, cudaMemcpyHostToDevice));
    h->have_query = true;
    return CGB_OK;
}

cgb_status cgb_load_query_file(cgb_handle* h, const char* path) {
    if (!h || !path) return CGB_ERR_ARG;
    std::vector<uint32_t> labels, edges;
    uint32_t qv = 0;
    std::string e = cgb::parse_query_file(path, labels, edges, qv);
    if (!e.empty()) return fail(h, CGB_ERR_IO, "%s", e.c_str());
    return cgb_load_query(h, qv, labels.data(), (uint32_t)(edges.size() / 2), edges.data());
}

uint32_t cgb_query_dir(const cgb_handle* h, uint32_t a, uint32_t b) {
    if (!h || !h->have_query || a >= h->q.qv || b >= h->q.qv) return 255;
    return h->q.eidx[a * kMaxQV + b];
}

cgb_status cgb_build_index(cgb_handle* h, const uint64_t* keys, uint64_t n, uint32_t dv_count) {
    if (!h) return CGB_ERR_ARG;
    if (!h->have_query) return fail(h, CGB_ERR_STATE, "load a query first");
    if (h->have_index) return fail(h, CGB_ERR_STATE, "index already built");
    if (dv_count > CGB_MAX_VID) return fail(h, CGB_ERR_LIMIT, "dv_count %u exceeds 2^27-1", dv_count);
    if (n && !keys) return CGB_ERR_ARG;
    CK(cudaSetDevice(h->device));
    // planner statistics (calig_helper_gamma.cu:304-311): entries and
    // non-empty vertices per direction -> mean run length
    std::vector<uint64_t> card(h->nd, 0), nodes(h->nd, 0);
    {
        std::vector<uint8_t> seen((size_t)h->nd * std::max<uint32_t>(dv_count, 1), 0);
        for (uint64_t i = 0; i < n; ++i) {
            uint32_t d = (uint32_t)(keys[i] >> 59), u = (uint32_t)((keys[i] >> 32) & 0x07FFFFFFu);
            uint32_t v = (uint32_t)keys[i];
            if (d >= h->nd || u >= dv_count || v >= dv_count)
                return fail(h, CGB_ERR_ARG, "key %llu out of range (dir %u u %u v %u, dv %u)",
                            (unsigned long long)i, d, u, v, dv_count);
            card[d]++;
            uint8_t& s = seen[(size_t)d * dv_count + u];
            if (!s) { s = 1; nodes[d]++; }
        }
    }
    float avg[kMaxDir] = {0};
    for (uint32_t d = 0; d < h->nd; ++d) avg[d] = nodes[d] ? (float)card[d] / (float)nodes[d] : 0.f;
    cgb::plan_edges(h->q, avg, h->plans, !(h->cfg.flags & CGB_FLAG_ENUMERATE_TAIL),
                    !(h->cfg.flags & CGB_FLAG_PLAIN_CORE_ORDER), !(h->cfg.flags & CGB_FLAG_NO_SEED_GROUPS),
                    !(h->cfg.flags & CGB_FLAG_WARP_TAIL), !(h->cfg.flags & CGB_FLAG_NO_LEVEL_SUM), true, cgb::kFoldLists);
    h->n_wsum = 0;
    h->wjobs_for = nullptr;  // the plans changed: rebuild the level-sum jobs
    for (uint32_t e = 0; e < h->q.qe; ++e)
        if (h->plans[e].sum_dense) {
            h->plans[e].wslot = (uint8_t)h->n_wsum;
            h->n_wsum += h->plans[e].n_core - h->plans[e].sum_from;
        }
    CK(cudaMemcpy(h->d_plans, h->plans, sizeof(EdgePlan) * kMaxQE, cudaMemcpyHostToDevice));
    {
        // valid-bit plans from the reference's starting edge
        cgb::select_starting_edge(h->q, card.data(), avg, h->vb_start);
        cgb::VbPlan vbp[kMaxQE];
        std::memset(vbp, 0, sizeof(vbp));
        h->vb_plan_error = cgb::plan_valid_bits(h->q, h->vb_start, vbp);
        if (!h->vb_plan_error.empty() && (h->cfg.flags & (CGB_FLAG_VALID_BITS | CGB_FLAG_MASK_PRUNE)))
            return fail(h, CGB_ERR_ARG, "valid bits: %s", h->vb_plan_error.c_str());
        CK(cudaMemcpy(h->d_vbplans, vbp, sizeof(vbp), cudaMemcpyHostToDevice));
        CK(cudaMemcpy(h->d_dir_edge, h->q.dir_to_edge, sizeof(h->q.dir_to_edge), cudaMemcpyHostToDevice));
    }

    h->dv = dv_count;
    cgb_status s;
    if ((s = ensure_dvcap(h, std::max<uint32_t>(dv_count, 1))) != CGB_OK) return s;
    unsigned long long cap = h->cfg.pool_words;
    // out-of-place merges write every touched run anew, so the pool carries
    // headroom for many batches between compactions (HBM is plentiful)
    if (cap == 0) cap = std::max<unsigned long long>(4ull * n + (128ull << 20), 192ull << 20);
    CK(cgb::device_malloc(&h->pool, cap * sizeof(uint32_t)));
    h->pool_cap = cap;
    h->h_pool_top = 0;
    h->h_live = 0;
    CK(cudaMemsetAsync(h->d_scal, 0, kCtlWords * sizeof(unsigned long long), h->stream));
    if ((s = grow(h, h->d_keys_in, h->keys_in_cap, std::max<uint64_t>(n, 1))) != CGB_OK) return s;
    if (n) CK(cudaMemcpyAsync(h->d_keys_in, keys, n * sizeof(uint64_t), cudaMemcpyHostToDevice, h->stream));
    EditSrc src;
    src.add = h->d_keys_in;
    src.n_add = n;
    if ((s = apply_edits(h, src)) != CGB_OK) return s;
    if ((s = sync_scalars(h)) != CGB_OK) return s;
    if (h->h_scal[kCtlErr]) return fail(h, CGB_ERR_ARG, "invalid keys (error bits %llu)", h->h_scal[kCtlErr]);
    h->have_index = true;
    return CGB_OK;
}

cgb_status cgb_apply_batch_device(cgb_handle* h, uint32_t dv_count, const uint64_t* ins, uint64_t n_ins,
                                  const uint64_t* del, uint64_t n_del, const uint64_t* delta, uint64_t n_delta,
                                  const uint8_t* edge_ok, void* stream, uint64_t* out_count) {
    if (!h || !out_count) return CGB_ERR_ARG;
    *out_count = 0;
    if (!h->have_index) return fail(h, CGB_ERR_STATE, "build the index first");
    if (dv_count < h->dv) return fail(h, CGB_ERR_ARG, "dv_count must not decrease (%u < %u)", dv_count, h->dv);
    if (dv_count > CGB_MAX_VID) return fail(h, CGB_ERR_LIMIT, "dv_count exceeds 2^27-1");
    if ((n_ins && !ins) || (n_del && !del) || (n_delta && !delta)) return CGB_ERR_ARG;
    if (n_ins > kMaxBatchKeys || n_del > kMaxBatchKeys) return fail(h, CGB_ERR_LIMIT, "edit batch too large");
    if (n_delta > 0xffffffffull) return fail(h, CGB_ERR_LIMIT, "delta batch too large");
    CK(cudaSetDevice(h->device));
    cudaStream_t user = (cudaStream_t)stream;
    if (user && user != h->stream) {
        // order this batch after the caller's prior work on `user`
        CK(cudaEventRecord(h->ev[4], user));
        CK(cudaStreamWaitEvent(h->stream, h->ev[4], 0));
    }
    cgb_status s;
    if ((s = ensure_dvcap(h, dv_count)) != CGB_OK) return s;
    h->dv = dv_count;
    const uint32_t B = bits_for(dv_count);
    PackInfo pi{B, h->nd, dv_count};
    unsigned int* d_err = (unsigned int*)(h->d_scal + kCtlErr);
    CK(cudaMemsetAsync(h->d_scal + kCtlErr, 0, (kCtlWords - kCtlErr) * sizeof(unsigned long long), h->stream));
    CK(cudaEventRecord(h->ev[0], h->stream));

    // 1. index update: pending delta (add) + ins (add) + del (remove)
    EditSrc src;
    src.packed = h->d_pending;
    src.n_packed = h->n_pending;
    src.B0 = h->pending_B;
    src.add = ins;
    src.n_add = n_ins;
    src.rem = del;
    src.n_rem = n_del;
    if ((s = apply_edits(h, src)) != CGB_OK) return s;
    h->n_pending = 0;
    CK(cudaEventRecord(h->ev[1], h->stream));

    // 2. delta lists
    const bool match = n_delta > 0;
    if (match) {
        if ((s = ensure_delta_buffers(h, n_delta)) != CGB_OK) return s;
        k_pack_delta<<<grid_for(h, n_delta), 256, 0, h->stream>>>(delta, n_delta, pi, h->d_dkeys, d_err, h->d_self);
        LAUNCHED();
        if ((s = radix_sort(h, h->d_dkeys, h->d_dkeys_alt, n_delta, 0, 2 * (int)B + (int)bits_for(h->nd) + 1)) != CGB_OK) return s;
        if (edge_ok) CK(cudaMemcpyAsync(h->d_edge_ok, edge_ok, h->q.qe, cudaMemcpyHostToDevice, h->stream));
        k_delta<<<grid_for(h, n_delta) + 1, 256, 0, h->stream>>>(h->d_dkeys, n_delta, B, h->rec, h->dvcap, h->d_dval,
                                                                 h->q.qe, h->d_plans, h->d_qe_dirs, h->d_edge_ok,
                                                                 edge_ok ? 1 : 0, h->d_seed, h->d_seed + kMaxQE);
        LAUNCHED();
        CK(cudaGetLastError());
        const bool vb_on = (h->cfg.flags & (CGB_FLAG_VALID_BITS | CGB_FLAG_MASK_PRUNE)) != 0;
        h->vb_stride = 0;
        if (vb_on) {
            // 2b. valid bits: fill, endpoints from the delta keys, then one
            // launch per indexing-order position (all query edges at once)
            const uint32_t stride = (dv_count + 31) / 32, qv = h->q.qv, qe = h->q.qe;
            if ((s = grow(h, h->d_vb, h->vb_cap, (size_t)qe * qv * stride)) != CGB_OK) return s;
            CK(cudaEventRecord(h->ev[6], h->stream));
            const size_t words = (size_t)qe * qv * stride;
            k_vb_fill<<<(unsigned)std::min<size_t>((words + 255) / 256, (size_t)h->num_sms * 16), 256, 0,
                        h->stream>>>(h->d_vbplans, h->d_vb, qe, qv, stride);
            LAUNCHED();
            k_vb_seed<<<grid_for(h, n_delta), 256, 0, h->stream>>>(h->d_vbplans, h->d_dir_edge, h->d_dkeys, n_delta,
                                                                   B, h->d_vb, qv, stride);
            LAUNCHED();
            const dim3 g((unsigned)std::min<uint32_t>((stride + 7) / 8, (uint32_t)h->num_sms * 8), qe);
            for (uint32_t d = 2; d < qv; ++d) {
                k_vb_depth<<<g, 256, 0, h->stream>>>(h->d_vbplans, h->rec, h->dvcap, h->pool, h->d_dval, dv_count,
                                                     h->d_vb, qv, stride, d);
                LAUNCHED();
            }
            CK(cudaGetLastError());
            h->vb_stride = stride;
        }
        CK(cudaEventRecord(h->ev[2], h->stream));

        // 2c. bit sets of the long old runs (this batch's index): built in full
        // once (and after the record table grows), since then kept current by
        // every merge; rebuilt when the slots ran out so that the longest runs
        // of today's index hold them
        const bool rb_on = !(h->cfg.flags & CGB_FLAG_NO_RUN_BITS);
        if (rb_on && !h->rb_valid && (s = rebuild_run_bits(h)) != CGB_OK) return s;

        // 3. matching
        DfsArgs da;
        da.rec = h->rec;
        da.dvcap = h->dvcap;
        da.pool = h->pool;
        da.dval = h->d_dval;
        da.dkeys = h->d_dkeys;
        da.B = B;
        da.qe = h->q.qe;
        da.seed_lo = h->d_seed;
        da.seed_pre = h->d_seed + kMaxQE;
        da.counts = h->d_counts;
        da.work_next = (unsigned int*)(h->d_scal + kCtlWork);
        da.err = d_err;
        da.stats = h->d_stats;
        da.tasks = h->d_tasks;
        da.task_cap = kTaskCap;
        da.qctr = h->d_qctr;
        do {  // the tag's epoch field must never be 0 (the ring starts zeroed)
            ++h->dfs_epoch;
        } while ((h->dfs_epoch & 0xfffffu) == 0);
        da.epoch = h->dfs_epoch;
        da.force_split = (h->cfg.flags & CGB_FLAG_FORCE_SPLIT) ? 1u : 0u;
        da.num_shards = h->cfg.num_shards ? h->cfg.num_shards : 1u;
        da.steal = (h->cfg.flags & CGB_FLAG_NO_STEAL) ? 0u : 1u;
        da.tail_cache = (h->cfg.flags & CGB_FLAG_NO_TAIL_CACHE) ? 0u : 1u;
        da.pair_lane_max = h->pair_lane_max;
        da.shard = h->cfg.shard_index < da.num_shards ? h->cfg.shard_index : 0u;
        da.self_seen = h->d_self;
        da.vb = (h->cfg.flags & CGB_FLAG_MASK_PRUNE) ? h->d_vb : nullptr;
        da.vb_stride = h->vb_stride;
        da.qv = h->q.qv;
        da.rb_slot = rb_on ? h->d_rb_slot : nullptr;
        da.rb_bits = h->d_rb_bits;
        da.rb_words = h->rb_words;
        da.plans = h->d_plans;
        da.epoch_ptr = nullptr;
        da.touched = nullptr;
        const bool footprint = (h->cfg.flags & CGB_FLAG_FOOTPRINT) != 0;
        const uint64_t nrec = (uint64_t)h->nd * h->dvcap;
        if (footprint) {
            if ((s = grow(h, h->d_touched, h->touched_cap, (size_t)(nrec + 31) / 32)) != CGB_OK) return s;
            CK(cudaMemsetAsync(h->d_touched, 0, ((nrec + 31) / 32) * sizeof(uint32_t), h->stream));
            da.touched = h->d_touched;
        }
        da.budget_ns = h->cfg.dfs_budget_ms ? (unsigned long long)h->cfg.dfs_budget_ms * 1000000ull
                                            : 600ull * 1000000000ull;
        // persistent grid: the blocks that an empty device holds at once (fewer may
        // run while another handle's kernels do: seed_claim.h)
        if (h->dfs_occupancy == 0) {
            int occ = 0;
            CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_dfs_count<false>, kDfsWarps * 32, 0));
            h->dfs_occupancy = std::max(occ, 1);
        }
        int bps = h->dfs_occupancy;
        if (h->cfg.dfs_blocks_per_sm) bps = std::min(bps, (int)h->cfg.dfs_blocks_per_sm);
        bool any_sum = false, any_memo = false;
        for (uint32_t e = 0; e < h->q.qe; ++e) {
            any_sum |= h->plans[e].sum_from != 0 && !h->plans[e].sum_dense;
            any_memo |= h->plans[e].memo_from != 0;
        }
        da.wsum = nullptr;
        if (h->n_wsum && !da.vb && da.tail_cache) {
            if ((s = dense_level_sums(h)) != CGB_OK) return s;
            da.wsum = h->d_wsum;
        }
        lsum_bind(h, any_sum, any_memo, da);
        if ((s = lsum_clear(h, da)) != CGB_OK) return s;
        bool uses_sums = false;
        for (uint32_t e = 0; e < h->q.qe; ++e)
            uses_sums |= h->plans[e].sum_from != 0 || h->plans[e].memo_from != 0 || h->plans[e].pair_last != 0;
        const dim3 grid(h->num_sms * bps), block(kDfsWarps * 32);
        if (footprint && uses_sums) k_dfs_count<false, true, true><<<grid, block, 0, h->stream>>>(da);
        else if (footprint) k_dfs_count<false, true, false><<<grid, block, 0, h->stream>>>(da);
        else if (uses_sums) k_dfs_count<false, false, true><<<grid, block, 0, h->stream>>>(da);
        else k_dfs_count<false, false, false><<<grid, block, 0, h->stream>>>(da);
        LAUNCHED();
        CK(cudaGetLastError());
        if ((s = memo_finish(h, da)) != CGB_OK) return s;
        CK(cudaEventRecord(h->ev[3], h->stream));
        if (footprint) {  // stats[4] := the launch's footprint (bytes of distinct records and lists)
            CK(cudaMemsetAsync(h->d_stats + 4, 0, sizeof(unsigned long long), h->stream));
            k_footprint<<<grid_for(h, nrec), 256, 0, h->stream>>>(h->rec, nrec, h->d_touched, h->d_stats + 4);
            LAUNCHED();
        }

        // 4. clear delta records; this delta becomes the pending merge-back
        k_delta_lists<<<grid_for(h, n_delta), 256, 0, h->stream>>>(h->d_dkeys, n_delta, nullptr, B, 0, h->rec,
                                                                   h->dvcap, nullptr, 1);
        LAUNCHED();
        std::swap(h->d_pending, h->d_dkeys);  // the sorted delta itself: nothing is copied
        h->pending_B = B;
        h->n_pending = n_delta;
    } else {
        CK(cudaEventRecord(h->ev[2], h->stream));
        CK(cudaEventRecord(h->ev[3], h->stream));
    }
    CK(cudaEventRecord(h->ev[5], h->stream));
    if ((s = sync_scalars(h)) != CGB_OK) return s;
    float t01 = 0, t12 = 0, t23 = 0, t03 = 0;
    cudaEventElapsedTime(&t01, h->ev[0], h->ev[1]);
    cudaEventElapsedTime(&t12, h->ev[1], h->ev[2]);
    cudaEventElapsedTime(&t23, h->ev[2], h->ev[3]);
    cudaEventElapsedTime(&t03, h->ev[0], h->ev[5]);
    h->last_vb_ms = 0;
    if (h->vb_stride) cudaEventElapsedTime(&h->last_vb_ms, h->ev[6], h->ev[2]);
    h->last_t[0] = t01; h->last_t[1] = t12; h->last_t[2] = t23; h->last_t[3] = t03;
    for (int i = 0; i < 8; ++i) h->last_stats[i] = h->h_scal[kCtlStats + i];
    if (h->h_scal[kCtlErr]) {
        h->n_pending = 0;
        h->rb_valid = false;  // a rejected batch may have left runs and bit sets apart
        cgb_status st = (h->h_scal[kCtlErr] & 24u) ? CGB_ERR_TIMEOUT : (h->h_scal[kCtlErr] & 4u) ? CGB_ERR_OOM : CGB_ERR_ARG;
        return fail(h, st,
                    "batch rejected: error bits %llu (1/2 = key out of range, 4 = pool exhausted, "
                    "8 = matching exceeded its time budget, 16 = a queued task was never published)",
                    h->h_scal[kCtlErr]);
    }
    uint64_t total = 0;
    for (uint32_t e = 0; e < h->q.qe; ++e) { h->last_counts[e] = h->h_scal[kCtlCounts + e]; total += h->h_scal[kCtlCounts + e]; }
    for (int i = 0; i < 8; ++i) h->last_stats[i] = h->h_scal[kCtlStats + i];
    *out_count = total;
    if (h->cfg.flags & CGB_FLAG_NO_MERGE_BACK_DEFER) {
        if ((s = flush_pending(h)) != CGB_OK) return s;
    }
    return CGB_OK;
}

cgb_status cgb_apply_batch(cgb_handle* h, uint32_t dv_count, const uint64_t* ins, uint64_t n_ins,
                           const uint64_t* del, uint64_t n_del, const uint64_t* delta, uint64_t n_delta,
                           const uint8_t* edge_ok, uint64_t* out_count) {
    if (!h || !out_count) return CGB_ERR_ARG;
    if ((n_ins && !ins) || (n_del && !del) || (n_delta && !delta)) return CGB_ERR_ARG;
    // bounded before the sum below, which must not wrap
    if (n_ins > kMaxBatchKeys || n_del > kMaxBatchKeys || n_delta > kMaxBatchKeys)
        return fail(h, CGB_ERR_LIMIT, "batch too large");
    CK(cudaSetDevice(h->device));
    const uint64_t n = n_ins + n_del + n_delta;
    cgb_status s;
    if ((s = grow(h, h->d_keys_in, h->keys_in_cap, std::max<uint64_t>(n, 1))) != CGB_OK) return s;
    uint64_t* d = h->d_keys_in;
    if (n_ins) CK(cudaMemcpyAsync(d, ins, n_ins * 8, cudaMemcpyHostToDevice, h->stream));
    if (n_del) CK(cudaMemcpyAsync(d + n_ins, del, n_del * 8, cudaMemcpyHostToDevice, h->stream));
    if (n_delta) CK(cudaMemcpyAsync(d + n_ins + n_del, delta, n_delta * 8, cudaMemcpyHostToDevice, h->stream));
    return cgb_apply_batch_device(h, dv_count, d, n_ins, d + n_ins, n_del, d + n_ins + n_del, n_delta, edge_ok,
                                  nullptr, out_count);
}

cgb_status cgb_last_edge_counts(const cgb_handle* h, uint64_t* out, uint32_t cap) {
    if (!h || !out) return CGB_ERR_ARG;
    for (uint32_t e = 0; e < cap && e < h->q.qe; ++e) out[e] = h->last_counts[e];
    return CGB_OK;
}

cgb_status cgb_last_timings(const cgb_handle* h, float* t4) {
    if (!h || !t4) return CGB_ERR_ARG;
    for (int i = 0; i < 4; ++i) t4[i] = h->last_t[i];
    return CGB_OK;
}

uint64_t cgb_kernel_launches(const cgb_handle* h) { return h ? h->launches : 0; }

cgb_status cgb_last_stats(const cgb_handle* h, uint64_t* out8) {
    if (!h || !out8) return CGB_ERR_ARG;
    for (int i = 0; i < 8; ++i) out8[i] = h->last_stats[i];
    return CGB_OK;
}

void* cgb_stream(const cgb_handle* h) { return h ? (void*)h->stream : nullptr; }

cgb_status cgb_plan_anchor(const cgb_handle* h, uint32_t ei, uint32_t* qvertex) {
    if (!h || !qvertex) return CGB_ERR_ARG;
    if (!h->have_index) return CGB_ERR_STATE;
    if (ei >= h->q.qe) return CGB_ERR_ARG;
    *qvertex = h->plans[ei].vs[0];
    return CGB_OK;
}

cgb_status cgb_plan_info(const cgb_handle* h, uint32_t ei, uint32_t* out4) {
    if (!h || !out4) return CGB_ERR_ARG;
    if (!h->have_index) return CGB_ERR_STATE;
    if (ei >= h->q.qe) return CGB_ERR_ARG;
    const EdgePlan& P = h->plans[ei];
    out4[0] = P.n_core;
    out4[1] = P.sum_from;
    out4[2] = P.sum_dense;
    out4[3] = P.tail_lane | (uint32_t)P.memo_from << 8 | (uint32_t)P.memo_pos << 16;
    return CGB_OK;
}

cgb_status cgb_check_symmetry(cgb_handle* h, uint64_t* n_asym) {
    if (!h || !n_asym) return CGB_ERR_ARG;
    *n_asym = 0;
    if (!h->have_index) return fail(h, CGB_ERR_STATE, "no index");
    CK(cudaSetDevice(h->device));
    cgb_status s;
    if ((s = flush_pending(h)) != CGB_OK) return s;
    unsigned long long* d_bad = nullptr;
    CK(cgb::device_malloc(&d_bad, sizeof(unsigned long long)));
    CK(cudaMemsetAsync(d_bad, 0, sizeof(unsigned long long), h->stream));
    const uint64_t n = (uint64_t)h->nd * h->dv;
    if (n) {
        k_asymmetry<<<grid_for(h, n * 32), 256, 0, h->stream>>>(h->rec, h->dvcap, h->dv, h->nd, h->pool, h->d_rev, d_bad);
        LAUNCHED();
    }
    unsigned long long bad = 0;
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(&bad, d_bad, sizeof(bad), cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    cudaFree(d_bad);
    CK(e);
    *n_asym = bad;
    return CGB_OK;
}

cgb_status cgb_starting_edge(const cgb_handle* h, uint32_t* out2) {
    if (!h || !out2) return CGB_ERR_ARG;
    if (!h->have_index) return CGB_ERR_STATE;
    out2[0] = h->vb_start[0];
    out2[1] = h->vb_start[1];
    return CGB_OK;
}

cgb_status cgb_valid_bits(cgb_handle* h, uint32_t* out, uint64_t cap, uint64_t* n_words, float* ms) {
    if (!h || !n_words) return CGB_ERR_ARG;
    *n_words = 0;
    if (!h->vb_stride) return fail(h, CGB_ERR_STATE, "no valid bits: enable CGB_FLAG_VALID_BITS and match a batch");
    const uint64_t n = (uint64_t)h->q.qe * h->q.qv * h->vb_stride;
    *n_words = n;
    if (ms) *ms = h->last_vb_ms;
    if (!out) return CGB_OK;
    if (cap < n) return fail(h, CGB_ERR_ARG, "buffer holds %llu of %llu words", (unsigned long long)cap,
                             (unsigned long long)n);
    CK(cudaSetDevice(h->device));
    CK(cudaMemcpyAsync(out, h->d_vb, n * sizeof(uint32_t), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return CGB_OK;
}

cgb_status cgb_read_index(cgb_handle* h, uint64_t* out, uint64_t cap, uint64_t* n_out) {
    if (!h || !n_out) return CGB_ERR_ARG;
    if (!h->have_index) return fail(h, CGB_ERR_STATE, "no index");
    CK(cudaSetDevice(h->device));
    cgb_status s;
    if ((s = flush_pending(h)) != CGB_OK) return s;
    const uint64_t n = (uint64_t)h->nd * h->dv;
    // the offsets of the runs and the key buffer stay with the handle up to
    // kReadKeep words each (allocating them took 1 of a small index's 1.2 ms);
    // larger ones are the call's own
    constexpr size_t kReadKeep = (64u << 20) / sizeof(uint64_t);
    struct Own {
        void* p = nullptr;
        ~Own() { if (p) cudaFree(p); }
    } own_off, own_keys;
    unsigned long long* offs = nullptr;
    if (n + 1 > kReadKeep) {
        CK(cgb::device_malloc(&own_off.p, (n + 1) * sizeof(unsigned long long)));
        offs = (unsigned long long*)own_off.p;
    } else {
        if ((s = grow(h, h->d_read_off, h->read_off_cap, n + 1)) != CGB_OK) return s;
        offs = h->d_read_off;
    }
    k_rec_lens<<<grid_for(h, n + 1), 256, 0, h->stream>>>(h->rec, h->dvcap, h->dv, h->nd, offs);
    LAUNCHED();
    size_t tb = 0;
    CK(cub::DeviceScan::ExclusiveSum(nullptr, tb, offs, offs, (int64_t)n + 1, h->stream));
    if ((s = grow_temp(h, tb)) != CGB_OK) return s;
    CK(cub::DeviceScan::ExclusiveSum(h->d_temp, tb, offs, offs, (int64_t)n + 1, h->stream));
    LAUNCHED();
    unsigned long long total = 0;
    CK(cudaMemcpyAsync(&total, offs + n, sizeof(total), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    *n_out = total;
    if (out && cap < total) return fail(h, CGB_ERR_ARG, "output capacity %llu < %llu", (unsigned long long)cap, total);
    if (out && total > 0) {
        uint64_t* keys = nullptr;
        if (total > kReadKeep) {
            CK(cgb::device_malloc(&own_keys.p, total * sizeof(uint64_t)));
            keys = (uint64_t*)own_keys.p;
        } else {
            if ((s = grow(h, h->d_read, h->read_cap, (size_t)total)) != CGB_OK) return s;
            keys = h->d_read;
        }
        k_dump<<<grid_for(h, n * 32), 256, 0, h->stream>>>(h->rec, h->dvcap, h->dv, h->nd, h->pool, offs, keys);
        LAUNCHED();
        CK(cudaMemcpyAsync(out, keys, total * sizeof(uint64_t), cudaMemcpyDeviceToHost, h->stream));
        CK(cudaStreamSynchronize(h->stream));
    }
    return CGB_OK;
}

}  // extern "C"

#include "multiquery.cuh"
