// Packed-memory-array layout of the index (the reference's GPMA:
// Multi_GPMA gpma/gpma.cuh:36-111, CGCSM_GPMA index/gpma_wrapper.cu:26-116,
// rebalance gpma/gpma.cu:493-665), rebuilt for sm_100a without device-side
// launches (the reference's rebalance uses CDP1, which sm_90+ lacks).
//
// Layout: one PMA per query direction d, `cap_d = kSeg * 2^h_d` slots of
// full 64-bit keys (d << 59 | u << 32 | v) plus a valid byte per slot; the
// directions are packed back to back, so the whole slot array is
// non-decreasing.  A slot that holds no key keeps a copy of an earlier key
// value (order is all that matters for it), so a plain lower_bound over the
// slots finds the first slot whose value is >= x, and x is present iff that
// slot is valid and holds x.
//
// Batch update, set semantics (index + ins) - del (the same as the engine's
// k_merge; the reference's GPMA is bulk-loaded once and never updated
// or read by its matcher, calig_helper_gpma.cu:284-296, 383-414, so its
// update semantics are not a parity target):
//   1. sort the edits (key, op), one effect per distinct key: a present key
//      that is deleted loses its valid flag in place; an absent key that is
//      inserted is queued for its leaf (the leaf of its lower_bound slot)
//   2. per leaf with queued inserts, the smallest enclosing tree node whose
//      density after the batch is within the upper bound of its level
//      (0.92 at the leaves to 0.84 at the root, gpma.cuh:55-58) is its
//      window; windows are tree nodes, so keeping only the maximal ones (sort
//      by start, prefix max of end) leaves disjoint windows
//   3. each window's valid keys and queued inserts are gathered, sorted
//      (segmented) and spread evenly over the window's slots
//   4. if a root would exceed its bound, the whole structure is rebuilt with
//      capacities at density <= 1/2 (amortised doubling)
// Lower density bounds are not enforced: deletions leave slots invalid until
// a window rewrites them (space is reclaimed by later windows and rebuilds).
#include <cuda_runtime.h>
#include <cub/cub.cuh>

#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <string>
#include <vector>

#include "cgbdsm.h"
#include "kept_buffers.h"

namespace {

constexpr uint32_t kSeg = 32;               // slots per leaf
constexpr double kUpLeaf = 0.92, kUpRoot = 0.84;

struct GpmaDir {
    uint64_t off = 0;      // first slot
    uint64_t cap = 0;      // slots (kSeg << h)
    uint32_t h = 0;        // tree height (leaves = 2^h)
    uint64_t leaf0 = 0;    // first leaf (global leaf index)
};

__device__ __forceinline__ uint64_t lower_bound_u64(const uint64_t* __restrict__ a, uint64_t lo, uint64_t hi,
                                                    uint64_t x) {
    uint64_t len = hi - lo;
    while (len > 0) {
        const uint64_t half = len >> 1;
        if (a[lo + half] < x) { lo += half + 1; len -= half + 1; }
        else len = half;
    }
    return lo;
}

// Per-direction tables on the device.
struct DirTab {
    const uint64_t* off;
    const uint64_t* cap;
    const uint32_t* h;
    const uint64_t* leaf0;
};

// The batch's keys with their op (0 insert, 1 delete).
__global__ void k_gp_edits(const uint64_t* __restrict__ ins, uint64_t n_ins, const uint64_t* __restrict__ del, uint64_t n_del,
                           uint64_t* __restrict__ key, uint8_t* __restrict__ op) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n_ins + n_del;
         i += (uint64_t)gridDim.x * blockDim.x) {
        key[i] = i < n_ins ? ins[i] : del[i - n_ins];
        op[i] = i < n_ins ? 0 : 1;
    }
}

// One thread per sorted edit; the first of each run of equal keys applies
// the run's effect (any delete wins: (S + ins) - del).
__global__ void k_gp_effect(const uint64_t* __restrict__ key, const uint8_t* __restrict__ op, uint64_t n,
                            uint64_t* slots, uint8_t* valid, DirTab dt, uint32_t nd, uint64_t* ins_key,
                            uint64_t* ins_leaf, unsigned long long* n_ins, int* leaf_delta, uint32_t* leaf_ins,
                            unsigned int* err) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t k = key[i];
        if (i > 0 && key[i - 1] == k) continue;
        bool del = false, ins = false;
        for (uint64_t t = i; t < n && key[t] == k; ++t) {
            del |= op[t] != 0;
            ins |= op[t] == 0;
        }
        const uint32_t d = (uint32_t)(k >> 59);
        if (d >= nd) { atomicOr(err, 1u); continue; }
        const uint64_t s0 = dt.off[d], s1 = s0 + dt.cap[d];
        const uint64_t p = lower_bound_u64(slots, s0, s1, k);
        const bool present = p < s1 && valid[p] && slots[p] == k;
        const uint64_t leaf = dt.leaf0[d] + min((p - s0) / kSeg, (dt.cap[d] / kSeg) - 1);
        if (del) {
            if (present) {
                valid[p] = 0;
                atomicAdd(leaf_delta + leaf, -1);
            }
        } else if (ins && !present) {
            const unsigned long long q = atomicAdd(n_ins, 1ull);
            ins_key[q] = k;
            ins_leaf[q] = leaf;
            atomicAdd(leaf_delta + leaf, 1);
            atomicAdd(leaf_ins + leaf, 1u);
        }
    }
}

// Valid keys per leaf (one warp per leaf) and per direction (added to dir_n).
__global__ void k_gp_leafcount(const uint8_t* valid, uint64_t n_leaves, const uint32_t* __restrict__ leaf_dir,
                               uint32_t* cnt, unsigned long long* dir_n) {
    __shared__ unsigned int s_n[CGB_MAX_DIR];
    for (uint32_t t = threadIdx.x; t < CGB_MAX_DIR; t += blockDim.x) s_n[t] = 0;
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t l = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; l < n_leaves; l += nw) {
        const uint32_t b = __ballot_sync(0xffffffffu, valid[l * kSeg + lane] != 0);
        if (lane == 0) {
            cnt[l] = __popc(b);
            if (b) atomicAdd(s_n + leaf_dir[l], (unsigned int)__popc(b));
        }
    }
    __syncthreads();
    for (uint32_t t = threadIdx.x; t < CGB_MAX_DIR; t += blockDim.x)
        if (s_n[t]) atomicAdd(dir_n + t, (unsigned long long)s_n[t]);
}

// Per leaf, the keys after the batch (newc) and the keys kept in place
// (without the queued inserts); both are prefix-summed next.
__global__ void k_gp_newcount(const uint32_t* cnt, const int* delta, const uint32_t* leaf_ins, uint64_t n,
                              uint64_t* newc, uint64_t* kept) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t c = (uint64_t)((int64_t)cnt[i] + delta[i]);
        newc[i] = c;
        kept[i] = c - leaf_ins[i];
    }
}

// Window of each leaf with queued inserts: smallest node within its level's
// upper density bound, entered at its first leaf as the largest level there
// (wlv: level + 1; 0: no window starts at the leaf).  P = inclusive prefix
// sums of the new per-leaf counts (P[l] = sum over leaves <= l).
__global__ void k_gp_window(const uint32_t* __restrict__ leaf_ins, const uint64_t* __restrict__ P,
                            const uint32_t* __restrict__ leaf_dir, DirTab dt, uint64_t n_leaves, uint32_t* wlv,
                            unsigned int* resize) {
    for (uint64_t l = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; l < n_leaves;
         l += (uint64_t)gridDim.x * blockDim.x) {
        if (!leaf_ins[l]) continue;
        const uint32_t d = leaf_dir[l];
        const uint64_t base = dt.leaf0[d], rel = l - base;
        const uint32_t h = dt.h[d];
        bool found = false;
        for (uint32_t lv = 0; lv <= h; ++lv) {
            const uint64_t a = base + ((rel >> lv) << lv), b = a + (1ull << lv);
            const uint64_t c = P[b - 1] - (a > 0 ? P[a - 1] : 0);
            const double up = h ? kUpLeaf - (kUpLeaf - kUpRoot) * (double)lv / (double)h : kUpRoot;
            if ((double)c <= up * (double)((uint64_t)kSeg << lv)) {
                atomicMax(wlv + a, lv + 1);
                found = true;
                break;
            }
        }
        if (!found) atomicOr(resize, 1u);
    }
}

// End (first leaf past it) of the window starting at each leaf, 0 if none.
__global__ void k_gp_end(const uint32_t* __restrict__ wlv, uint64_t n, uint64_t* end) {
    for (uint64_t l = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; l < n; l += (uint64_t)gridDim.x * blockDim.x)
        end[l] = wlv[l] ? l + (1ull << (wlv[l] - 1)) : 0;
}

// A window is maximal when its end exceeds every end before it (pmax: running
// maximum): 1 at its first leaf.  The running sum of these numbers the windows
// and, with pmax, says which leaves lie in one: nothing is sorted or searched.
__global__ void k_gp_maximal(const uint32_t* __restrict__ wlv, const uint64_t* __restrict__ pmax, uint64_t n,
                             uint32_t* flag) {
    for (uint64_t l = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; l < n; l += (uint64_t)gridDim.x * blockDim.x)
        flag[l] = wlv[l] && pmax[l] > (l ? pmax[l - 1] : 0ull) ? 1u : 0u;
}

// Window w (flag at leaf l, widx[l] = w + 1): first leaf and level, new key
// count, the keys kept in place (the inserts go behind them), and the value
// before it (read before any rewrite).  The last leaf writes the counts.
struct GpWin {
    uint64_t a, b, count, pred;
};
__global__ void k_gp_wininfo(const uint32_t* __restrict__ flag, const uint32_t* __restrict__ widx,
                             const uint64_t* __restrict__ pmax, uint64_t n_leaves, const uint64_t* __restrict__ P,
                             const uint64_t* __restrict__ Q, const uint64_t* __restrict__ slots, GpWin* win,
                             uint64_t* wcount, unsigned long long* wfill, unsigned long long* n_win) {
    for (uint64_t l = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; l < n_leaves;
         l += (uint64_t)gridDim.x * blockDim.x) {
        if (l == n_leaves - 1) *n_win = widx[l];
        if (!flag[l]) continue;
        const uint32_t w = widx[l] - 1;
        const uint64_t b = pmax[l];
        const uint64_t c = P[b - 1] - (l > 0 ? P[l - 1] : 0);
        win[w] = {l, b, c, l > 0 ? slots[l * kSeg - 1] : 0ull};
        wcount[w] = c;
        wfill[w] = Q[b - 1] - (l > 0 ? Q[l - 1] : 0);
    }
}

// The windows' valid keys to tmp, in slot order: a warp per leaf that lies in
// a window (a block per window left most threads idle: nearly every window
// is one leaf; 98 -> 12 us for 100 k inserts into 2 M keys).
__global__ void k_gp_gather(const GpWin* __restrict__ win, const uint32_t* __restrict__ widx,
                            const uint64_t* __restrict__ pmax, uint64_t n_leaves, const uint64_t* __restrict__ woff,
                            const uint64_t* __restrict__ Q, const uint64_t* __restrict__ slots,
                            const uint8_t* __restrict__ valid, uint64_t* tmp, unsigned int* bad) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t l = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; l < n_leaves; l += nw) {
        if (pmax[l] <= l) continue;
        const uint32_t w = widx[l] - 1;
        const uint64_t a = win[w].a, n = win[w].count;
        const uint64_t at = (l > 0 ? Q[l - 1] : 0) - (a > 0 ? Q[a - 1] : 0);
        const bool f = valid[l * kSeg + lane] != 0;
        const uint32_t b = __ballot_sync(0xffffffffu, f);
        const uint64_t p = at + __popc(b & ((1u << lane) - 1u));
        if (f) {
            if (p < n) tmp[woff[w] + p] = slots[l * kSeg + lane];
            else atomicOr(bad, 1u);
        }
    }
}

// Queued inserts join their window, behind the keys kept in place.  Every
// such leaf lies in a window and every window's slots in tmp number its new
// count; a violation of either sets `bad` and writes nothing.
__global__ void k_gp_place_ins(const uint64_t* __restrict__ ins_key, const uint64_t* __restrict__ ins_leaf,
                               uint64_t n, const uint32_t* __restrict__ widx, const uint64_t* __restrict__ pmax,
                               const uint64_t* __restrict__ woff, const GpWin* __restrict__ win,
                               unsigned long long* wfill, uint64_t* tmp, unsigned int* bad) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t leaf = ins_leaf[i];
        if (pmax[leaf] <= leaf) { atomicOr(bad, 1u); continue; }
        const uint32_t w = widx[leaf] - 1;
        const unsigned long long q = atomicAdd(wfill + w, 1ull);
        if (q >= win[w].count) { atomicOr(bad, 1u); continue; }
        tmp[woff[w] + q] = ins_key[i];
    }
}

// Spread each window's sorted keys evenly: key i to slot s0 + floor(i W / n);
// every other slot copies the last key before it (or the value before the
// window).  A warp per leaf in a window; W is a power of two, and whether slot
// r holds key i needs no division (r n <= i W < (r + 1) n).
__global__ void k_gp_scatter(const GpWin* __restrict__ win, const uint32_t* __restrict__ widx,
                             const uint64_t* __restrict__ pmax, uint64_t n_leaves, const uint64_t* __restrict__ woff,
                             const uint64_t* __restrict__ sorted, uint64_t* slots, uint8_t* valid) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t l = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; l < n_leaves; l += nw) {
        if (pmax[l] <= l) continue;
        const uint32_t w = widx[l] - 1;
        const GpWin W = win[w];
        const uint32_t sh = 31 - __clz((uint32_t)(W.b - W.a)) + 5;  // log2 of its slots
        static_assert(kSeg == 32, "a lane per slot of a leaf");
        const uint64_t r = (l - W.a) * kSeg + lane, n = W.count;
        // last key index placed at or before slot r: ceil((r + 1) n / W) - 1
        const uint64_t im = n ? ((r + 1) * n + (1ull << sh) - 1) >> sh : 0;
        const uint64_t at = l * kSeg + lane;
        if (im == 0) {
            slots[at] = W.pred;
            valid[at] = 0;
        } else {
            const uint64_t i = im - 1;
            slots[at] = sorted[woff[w] + i];
            valid[at] = (i << sh) >= r * n && (i << sh) < (r + 1) * n ? 1 : 0;
        }
    }
}

// Rebuild: sorted unique keys spread over fresh capacities (density <= 1/2).
__global__ void k_gp_spread(const uint64_t* __restrict__ keys, uint64_t n, const uint64_t* __restrict__ dir_start,
                            const uint64_t* __restrict__ dir_n, DirTab dt, uint32_t nd, uint64_t* slots,
                            uint8_t* valid, uint64_t total_slots) {
    for (uint64_t s = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; s < total_slots;
         s += (uint64_t)gridDim.x * blockDim.x) {
        // direction of slot s
        uint32_t lo = 0, len = nd;
        while (len > 0) {
            const uint32_t half = len >> 1;
            if (dt.off[lo + half] <= s) { lo += half + 1; len -= half + 1; }
            else len = half;
        }
        const uint32_t d = lo - 1;
        const uint64_t r = s - dt.off[d], W = dt.cap[d], m = dir_n[d], st = dir_start[d];
        const uint64_t im = m ? ((r + 1) * m + W - 1) / W : 0;
        if (im == 0) {
            slots[s] = st > 0 ? keys[st - 1] : 0ull;
            valid[s] = 0;
        } else {
            const uint64_t i = im - 1;
            slots[s] = keys[st + i];
            valid[s] = (i * W / m == r) ? 1 : 0;
        }
    }
}

__global__ void k_gp_dir_hist(const uint64_t* keys, uint64_t n, uint32_t nd, unsigned long long* hist,
                              unsigned int* err) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t d = (uint32_t)(keys[i] >> 59);
        if (d < nd) atomicAdd(hist + d, 1ull);
        else atomicOr(err, 1u);
    }
}

__global__ void k_gp_leafdir(uint32_t* leaf_dir, const uint64_t* leaf0, uint32_t nd, uint64_t n_leaves) {
    for (uint64_t l = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; l < n_leaves;
         l += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t lo = 0, len = nd;
        while (len > 0) {
            const uint32_t half = len >> 1;
            if (leaf0[lo + half] <= l) { lo += half + 1; len -= half + 1; }
            else len = half;
        }
        leaf_dir[l] = lo - 1;
    }
}

__global__ void k_gp_valid_flags(const uint8_t* valid, uint64_t n, uint8_t* out) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = valid[i];
}

// The keys of a direction's leaves, ascending, without their direction: a
// warp per leaf, at the scanned leaf counts.
__global__ void k_gp_extract(const uint64_t* __restrict__ slots, const uint8_t* __restrict__ valid, uint64_t n_leaves,
                             const uint64_t* __restrict__ off, uint64_t* __restrict__ out) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t l = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; l < n_leaves; l += nw) {
        const bool f = valid[l * kSeg + lane] != 0;
        const uint32_t b = __ballot_sync(0xffffffffu, f);
        if (f) out[off[l] + __popc(b & ((1u << lane) - 1u))] = slots[l * kSeg + lane] & ((1ull << 59) - 1ull);
    }
}

struct MaxOp {
    __device__ __forceinline__ uint64_t operator()(uint64_t a, uint64_t b) const { return a > b ? a : b; }
};

}  // namespace

struct cgb_gpma {
    int device = 0;
    cudaStream_t stream = nullptr;
    uint32_t nd = 0;
    std::string err;
    std::vector<GpmaDir> dirs;
    uint64_t total_slots = 0, n_leaves = 0, n_keys = 0;
    uint64_t dir_n[CGB_MAX_DIR] = {0};  // keys per direction
    bool counts_stale = false;  // an update failed after its deletes: leaf and direction counts are behind
    uint64_t* slots = nullptr;
    uint8_t* valid = nullptr;
    uint32_t* leaf_cnt = nullptr;
    int* leaf_delta = nullptr;
    uint32_t* leaf_ins = nullptr;
    uint32_t* leaf_dir = nullptr;
    uint64_t* d_off = nullptr; uint64_t* d_cap = nullptr; uint32_t* d_h = nullptr; uint64_t* d_leaf0 = nullptr;
    unsigned long long* d_scal = nullptr;  // [0] n_ins, [1] n_win, [2] resize|err<<1 (u32 pair), [3..] hist
    void* temp = nullptr; size_t temp_cap = 0;
    // per-call buffers, kept between calls: a call's 16 cudaMalloc and cudaFree
    // took 14 of a 100k + 100k update's 17 ms
    cgb::KeptBuffers bufs;
    uint64_t stats[6] = {0, 0, 0, 0, 0, 0};
    cudaEvent_t e0 = nullptr, e1 = nullptr;
};

namespace {

cgb_status gfail(cgb_gpma* g, cgb_status s, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    if (g) g->err = buf;
    return s;
}

#define GCK(x)                                                                                    \
    do {                                                                                          \
        cudaError_t e_ = (x);                                                                     \
        if (e_ != cudaSuccess) return gfail(g, e_ == cudaErrorMemoryAllocation ? CGB_ERR_OOM : CGB_ERR_CUDA, \
                                            "%s: %s", #x, cudaGetErrorString(e_));                \
    } while (0)

unsigned grid_of(uint64_t n) { return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((n + 255) / 256, 148ull * 16)); }

// A buffer of n T for the current call.
template <typename T>
cgb_status galloc(cgb_gpma* g, T*& p, uint64_t n) {
    cudaError_t e = cudaSuccess;
    p = (T*)g->bufs.take(std::max<uint64_t>(n, 1) * sizeof(T), [&](size_t bytes) {
        void* q = nullptr;
        e = cudaMalloc(&q, bytes);
        return e == cudaSuccess ? q : nullptr;
    }, [](void* q) { cudaFree(q); });
    GCK(e);
    return CGB_OK;
}

cgb_status gtemp(cgb_gpma* g, size_t need) {
    if (need <= g->temp_cap && g->temp) return CGB_OK;
    const size_t bytes = need + need / 2;
    if (g->temp) cudaFree(g->temp);
    g->temp = nullptr;
    g->temp_cap = 0;
    GCK(cudaMalloc(&g->temp, bytes));
    g->temp_cap = bytes;
    return CGB_OK;
}

void free_structure(cgb_gpma* g) {
    for (void* p : {(void*)g->slots, (void*)g->valid, (void*)g->leaf_cnt, (void*)g->leaf_delta, (void*)g->leaf_ins,
                    (void*)g->leaf_dir})
        if (p) cudaFree(p);
    g->slots = nullptr; g->valid = nullptr; g->leaf_cnt = nullptr; g->leaf_delta = nullptr;
    g->leaf_ins = nullptr; g->leaf_dir = nullptr;
}

// Returns the call's buffers to the handle.
void reclaim(cgb_gpma* g) {
    g->bufs.give_back([](void* p) { cudaFree(p); });
}

// The caller's key arrays may come from work queued on the default stream.
cgb_status after_default_stream(cgb_gpma* g) {
    GCK(cudaEventRecord(g->e0, cudaStreamLegacy));
    GCK(cudaStreamWaitEvent(g->stream, g->e0, 0));
    return CGB_OK;
}

// Rebuilds the structure from n sorted unique keys (device).
cgb_status rebuild(cgb_gpma* g, const uint64_t* keys, uint64_t n) {
    unsigned int* d_err = (unsigned int*)(g->d_scal + 2);
    unsigned long long* hist = g->d_scal + 3;
    GCK(cudaMemsetAsync(g->d_scal + 2, 0, (1 + g->nd) * sizeof(unsigned long long), g->stream));
    if (n) k_gp_dir_hist<<<grid_of(n), 256, 0, g->stream>>>(keys, n, g->nd, hist, d_err);
    std::vector<unsigned long long> h(1 + g->nd);
    GCK(cudaMemcpyAsync(h.data(), g->d_scal + 2, h.size() * sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                        g->stream));
    GCK(cudaStreamSynchronize(g->stream));
    if (h[0]) return gfail(g, CGB_ERR_ARG, "key direction out of range (>= %u)", g->nd);
    free_structure(g);
    g->dirs.assign(g->nd, {});
    uint64_t off = 0, leaf = 0;
    std::vector<uint64_t> start(g->nd), cnt(g->nd);
    uint64_t acc = 0;
    for (uint32_t d = 0; d < g->nd; ++d) {
        cnt[d] = g->dir_n[d] = h[1 + d];
        start[d] = acc;
        acc += cnt[d];
        uint32_t hh = 0;
        while (((uint64_t)kSeg << hh) < 2 * cnt[d]) ++hh;  // density <= 1/2
        g->dirs[d] = {off, (uint64_t)kSeg << hh, hh, leaf};
        off += (uint64_t)kSeg << hh;
        leaf += 1ull << hh;
    }
    g->total_slots = off;
    g->n_leaves = leaf;
    g->n_keys = n;
    GCK(cudaMalloc(&g->slots, off * sizeof(uint64_t)));
    GCK(cudaMalloc(&g->valid, off));
    GCK(cudaMalloc(&g->leaf_cnt, leaf * sizeof(uint32_t)));
    GCK(cudaMalloc(&g->leaf_delta, leaf * sizeof(int)));
    GCK(cudaMalloc(&g->leaf_ins, leaf * sizeof(uint32_t)));
    GCK(cudaMalloc(&g->leaf_dir, leaf * sizeof(uint32_t)));
    std::vector<uint64_t> o(g->nd), c(g->nd), l0(g->nd);
    std::vector<uint32_t> hh(g->nd);
    for (uint32_t d = 0; d < g->nd; ++d) { o[d] = g->dirs[d].off; c[d] = g->dirs[d].cap; hh[d] = g->dirs[d].h; l0[d] = g->dirs[d].leaf0; }
    GCK(cudaMemcpyAsync(g->d_off, o.data(), g->nd * 8, cudaMemcpyHostToDevice, g->stream));
    GCK(cudaMemcpyAsync(g->d_cap, c.data(), g->nd * 8, cudaMemcpyHostToDevice, g->stream));
    GCK(cudaMemcpyAsync(g->d_h, hh.data(), g->nd * 4, cudaMemcpyHostToDevice, g->stream));
    GCK(cudaMemcpyAsync(g->d_leaf0, l0.data(), g->nd * 8, cudaMemcpyHostToDevice, g->stream));
    uint64_t *d_start = nullptr, *d_cnt = nullptr;
    cgb_status s;
    if ((s = galloc(g, d_start, g->nd)) != CGB_OK) return s;
    if ((s = galloc(g, d_cnt, g->nd)) != CGB_OK) return s;
    GCK(cudaMemcpyAsync(d_start, start.data(), g->nd * 8, cudaMemcpyHostToDevice, g->stream));
    GCK(cudaMemcpyAsync(d_cnt, cnt.data(), g->nd * 8, cudaMemcpyHostToDevice, g->stream));
    DirTab dt{g->d_off, g->d_cap, g->d_h, g->d_leaf0};
    k_gp_spread<<<grid_of(off), 256, 0, g->stream>>>(keys, n, d_start, d_cnt, dt, g->nd, g->slots, g->valid, off);
    k_gp_leafdir<<<grid_of(leaf), 256, 0, g->stream>>>(g->leaf_dir, g->d_leaf0, g->nd, leaf);
    k_gp_leafcount<<<grid_of(leaf * 32), 256, 0, g->stream>>>(g->valid, leaf, g->leaf_dir, g->leaf_cnt, hist);
    GCK(cudaGetLastError());
    GCK(cudaStreamSynchronize(g->stream));
    g->counts_stale = false;
    reclaim(g);
    return CGB_OK;
}

// Leaf counts and direction counts from the valid flags.
cgb_status recount(cgb_gpma* g) {
    GCK(cudaMemsetAsync(g->d_scal + 3, 0, CGB_MAX_DIR * sizeof(unsigned long long), g->stream));
    k_gp_leafcount<<<grid_of(g->n_leaves * 32), 256, 0, g->stream>>>(g->valid, g->n_leaves, g->leaf_dir, g->leaf_cnt,
                                                                     g->d_scal + 3);
    GCK(cudaGetLastError());
    unsigned long long dn[CGB_MAX_DIR];
    GCK(cudaMemcpyAsync(dn, g->d_scal + 3, sizeof(dn), cudaMemcpyDeviceToHost, g->stream));
    GCK(cudaStreamSynchronize(g->stream));
    g->n_keys = 0;
    for (uint32_t d = 0; d < g->nd; ++d) g->n_keys += g->dir_n[d] = dn[d];
    g->counts_stale = false;
    return CGB_OK;
}

// Sorted unique copy of keys (device) into *out (allocated in bufs).
cgb_status sort_unique(cgb_gpma* g, const uint64_t* keys, uint64_t n, uint64_t*& out, uint64_t& m) {
    uint64_t *a = nullptr, *b = nullptr;
    cgb_status s;
    if ((s = galloc(g, a, n)) != CGB_OK) return s;
    if ((s = galloc(g, b, n)) != CGB_OK) return s;
    size_t bytes = 0;
    GCK(cub::DeviceRadixSort::SortKeys(nullptr, bytes, keys, a, n, 0, 64, g->stream));
    if ((s = gtemp(g, bytes)) != CGB_OK) return s;
    GCK(cub::DeviceRadixSort::SortKeys(g->temp, bytes, keys, a, n, 0, 64, g->stream));
    unsigned long long* d_m = g->d_scal + 0;
    bytes = 0;
    GCK(cub::DeviceSelect::Unique(nullptr, bytes, a, b, d_m, n, g->stream));
    if ((s = gtemp(g, bytes)) != CGB_OK) return s;
    GCK(cub::DeviceSelect::Unique(g->temp, bytes, a, b, d_m, n, g->stream));
    unsigned long long hm = 0;
    GCK(cudaMemcpyAsync(&hm, d_m, 8, cudaMemcpyDeviceToHost, g->stream));
    GCK(cudaStreamSynchronize(g->stream));
    out = b;
    m = hm;
    return CGB_OK;
}

}  // namespace

extern "C" {

cgb_status cgb_gpma_create(int device, uint32_t num_dirs, cgb_gpma** out) {
    if (!out || num_dirs == 0 || num_dirs > CGB_MAX_DIR) return CGB_ERR_ARG;
    auto* g = new cgb_gpma();
    *out = g;
    g->device = device;
    g->nd = num_dirs;
    GCK(cudaSetDevice(device));
    GCK(cudaStreamCreateWithFlags(&g->stream, cudaStreamNonBlocking));
    GCK(cudaMalloc(&g->d_off, num_dirs * 8));
    GCK(cudaMalloc(&g->d_cap, num_dirs * 8));
    GCK(cudaMalloc(&g->d_h, num_dirs * 4));
    GCK(cudaMalloc(&g->d_leaf0, num_dirs * 8));
    GCK(cudaMalloc(&g->d_scal, (3 + CGB_MAX_DIR) * sizeof(unsigned long long)));
    GCK(cudaEventCreate(&g->e0));
    GCK(cudaEventCreate(&g->e1));
    uint64_t none = 0;
    return rebuild(g, &none, 0);
}

void cgb_gpma_destroy(cgb_gpma* g) {
    if (!g) return;
    cudaSetDevice(g->device);
    if (g->stream) cudaStreamSynchronize(g->stream);
    free_structure(g);
    g->bufs.release_all([](void* p) { cudaFree(p); });
    for (void* p : {(void*)g->d_off, (void*)g->d_cap, (void*)g->d_h, (void*)g->d_leaf0, (void*)g->d_scal, g->temp})
        if (p) cudaFree(p);
    if (g->e0) cudaEventDestroy(g->e0);
    if (g->e1) cudaEventDestroy(g->e1);
    if (g->stream) cudaStreamDestroy(g->stream);
    delete g;
}

const char* cgb_gpma_last_error(const cgb_gpma* g) { return g ? g->err.c_str() : "null handle"; }

cgb_status cgb_gpma_bulk_load(cgb_gpma* g, const uint64_t* keys_device, uint64_t n) {
    if (!g || (n && !keys_device)) return CGB_ERR_ARG;
    GCK(cudaSetDevice(g->device));
    uint64_t* u = nullptr;
    uint64_t m = 0;
    cgb_status s;
    reclaim(g);  // a call that failed left its buffers out
    if ((s = after_default_stream(g)) != CGB_OK) return s;
    if (n) {
        if ((s = sort_unique(g, keys_device, n, u, m)) != CGB_OK) return s;
    }
    const uint64_t none = 0;
    s = rebuild(g, n ? u : &none, m);
    return s;
}

cgb_status cgb_gpma_batch_update(cgb_gpma* g, const uint64_t* ins_device, uint64_t n_ins,
                                 const uint64_t* del_device, uint64_t n_del) {
    if (!g || (n_ins && !ins_device) || (n_del && !del_device)) return CGB_ERR_ARG;
    // bounded before the sum below, which must not wrap (2^36 keys = 512 GiB, beyond any HBM)
    if (n_ins > (1ull << 36) || n_del > (1ull << 36)) return gfail(g, CGB_ERR_LIMIT, "edit batch too large");
    GCK(cudaSetDevice(g->device));
    for (auto& x : g->stats) x = 0;
    const uint64_t n = n_ins + n_del;
    if (n == 0) return CGB_OK;
    cgb_status s;
    if (g->counts_stale && (s = recount(g)) != CGB_OK) return s;
    reclaim(g);
    if ((s = after_default_stream(g)) != CGB_OK) return s;
    GCK(cudaEventRecord(g->e0, g->stream));
    // 1. edits sorted by key with their op (0 insert, 1 delete)
    uint64_t *k_in = nullptr, *k_out = nullptr;
    uint8_t *o_in = nullptr, *o_out = nullptr;
    if ((s = galloc(g, k_in, n)) != CGB_OK) return s;
    if ((s = galloc(g, k_out, n)) != CGB_OK) return s;
    if ((s = galloc(g, o_in, n)) != CGB_OK) return s;
    if ((s = galloc(g, o_out, n)) != CGB_OK) return s;
    k_gp_edits<<<grid_of(n), 256, 0, g->stream>>>(ins_device, n_ins, del_device, n_del, k_in, o_in);
    size_t bytes = 0;
    GCK(cub::DeviceRadixSort::SortPairs(nullptr, bytes, k_in, k_out, o_in, o_out, n, 0, 64, g->stream));
    if ((s = gtemp(g, bytes)) != CGB_OK) return s;
    GCK(cub::DeviceRadixSort::SortPairs(g->temp, bytes, k_in, k_out, o_in, o_out, n, 0, 64, g->stream));
    // 2. effects: deletes in place, inserts queued per leaf
    uint64_t *ins_key = nullptr, *ins_leaf = nullptr;
    if ((s = galloc(g, ins_key, n)) != CGB_OK) return s;
    if ((s = galloc(g, ins_leaf, n)) != CGB_OK) return s;
    GCK(cudaMemsetAsync(g->d_scal, 0, (3 + CGB_MAX_DIR) * sizeof(unsigned long long), g->stream));
    GCK(cudaMemsetAsync(g->leaf_delta, 0, g->n_leaves * sizeof(int), g->stream));
    GCK(cudaMemsetAsync(g->leaf_ins, 0, g->n_leaves * sizeof(uint32_t), g->stream));
    DirTab dt{g->d_off, g->d_cap, g->d_h, g->d_leaf0};
    g->counts_stale = true;
    unsigned int* d_flags = (unsigned int*)(g->d_scal + 2);  // [0] resize, [1] error
    k_gp_effect<<<grid_of(n), 256, 0, g->stream>>>(k_out, o_out, n, g->slots, g->valid, dt, g->nd, ins_key, ins_leaf,
                                                   g->d_scal + 0, g->leaf_delta, g->leaf_ins, d_flags + 1);
    // 3. windows: per leaf, the level of the window starting there; the maximal
    // ones numbered by a running sum
    uint64_t *newc = nullptr, *kept = nullptr, *P = nullptr, *Q = nullptr, *wend = nullptr, *pmax = nullptr;
    uint32_t *wlv = nullptr, *flag = nullptr, *widx = nullptr;
    GpWin* win = nullptr;
    uint64_t* wcount = nullptr;
    unsigned long long* wfill = nullptr;
    const uint64_t L = g->n_leaves, maxwin = std::min(L, n);
    if ((s = galloc(g, newc, L)) != CGB_OK) return s;
    if ((s = galloc(g, kept, L)) != CGB_OK) return s;
    if ((s = galloc(g, P, L)) != CGB_OK) return s;
    if ((s = galloc(g, Q, L)) != CGB_OK) return s;
    if ((s = galloc(g, wend, L)) != CGB_OK) return s;
    if ((s = galloc(g, pmax, L)) != CGB_OK) return s;
    if ((s = galloc(g, wlv, L)) != CGB_OK) return s;
    if ((s = galloc(g, flag, L)) != CGB_OK) return s;
    if ((s = galloc(g, widx, L)) != CGB_OK) return s;
    if ((s = galloc(g, win, maxwin)) != CGB_OK) return s;
    if ((s = galloc(g, wcount, maxwin)) != CGB_OK) return s;
    if ((s = galloc(g, wfill, maxwin)) != CGB_OK) return s;
    GCK(cudaMemsetAsync(wlv, 0, L * sizeof(uint32_t), g->stream));
    k_gp_newcount<<<grid_of(L), 256, 0, g->stream>>>(g->leaf_cnt, g->leaf_delta, g->leaf_ins, L, newc, kept);
    size_t b1 = 0, b2 = 0, b3 = 0;
    GCK(cub::DeviceScan::InclusiveSum(nullptr, b1, newc, P, L, g->stream));
    GCK(cub::DeviceScan::InclusiveScan(nullptr, b2, wend, pmax, MaxOp(), L, g->stream));
    GCK(cub::DeviceScan::InclusiveSum(nullptr, b3, flag, widx, L, g->stream));
    if ((s = gtemp(g, std::max(b1, std::max(b2, b3)))) != CGB_OK) return s;
    GCK(cub::DeviceScan::InclusiveSum(g->temp, b1, newc, P, L, g->stream));
    GCK(cub::DeviceScan::InclusiveSum(g->temp, b1, kept, Q, L, g->stream));
    k_gp_window<<<grid_of(L), 256, 0, g->stream>>>(g->leaf_ins, P, g->leaf_dir, dt, L, wlv, d_flags);
    k_gp_end<<<grid_of(L), 256, 0, g->stream>>>(wlv, L, wend);
    GCK(cub::DeviceScan::InclusiveScan(g->temp, b2, wend, pmax, MaxOp(), L, g->stream));
    k_gp_maximal<<<grid_of(L), 256, 0, g->stream>>>(wlv, pmax, L, flag);
    GCK(cub::DeviceScan::InclusiveSum(g->temp, b3, flag, widx, L, g->stream));
    k_gp_wininfo<<<grid_of(L), 256, 0, g->stream>>>(flag, widx, pmax, L, P, Q, g->slots, win, wcount, wfill,
                                                    g->d_scal + 1);
    unsigned long long h3[3];
    GCK(cudaMemcpyAsync(h3, g->d_scal, sizeof(h3), cudaMemcpyDeviceToHost, g->stream));
    GCK(cudaStreamSynchronize(g->stream));
    const uint64_t nins = h3[0], nwin = h3[1];
    const unsigned int resize = (unsigned int)(h3[2] & 0xffffffffull), kerr = (unsigned int)(h3[2] >> 32);
    if (kerr) return gfail(g, CGB_ERR_ARG, "key direction out of range (>= %u)", g->nd);
    if (resize) {
        // 4. a root is over its bound: rebuild from the valid keys plus the inserts
        uint64_t *all = nullptr;
        if ((s = galloc(g, all, g->total_slots + nins)) != CGB_OK) return s;
        uint8_t* flags = nullptr;
        if ((s = galloc(g, flags, g->total_slots)) != CGB_OK) return s;
        k_gp_valid_flags<<<grid_of(g->total_slots), 256, 0, g->stream>>>(g->valid, g->total_slots, flags);
        bytes = 0;
        GCK(cub::DeviceSelect::Flagged(nullptr, bytes, g->slots, flags, all, g->d_scal + 1, g->total_slots, g->stream));
        if ((s = gtemp(g, bytes)) != CGB_OK) return s;
        GCK(cub::DeviceSelect::Flagged(g->temp, bytes, g->slots, flags, all, g->d_scal + 1, g->total_slots,
                                       g->stream));
        unsigned long long nv = 0;
        GCK(cudaMemcpyAsync(&nv, g->d_scal + 1, 8, cudaMemcpyDeviceToHost, g->stream));
        GCK(cudaStreamSynchronize(g->stream));
        if (nins) GCK(cudaMemcpyAsync(all + nv, ins_key, nins * 8, cudaMemcpyDeviceToDevice, g->stream));
        uint64_t* u = nullptr;
        uint64_t m = 0;
        if ((s = sort_unique(g, all, nv + nins, u, m)) != CGB_OK) return s;
        g->stats[3] = 1;
        s = rebuild(g, u, m);
        GCK(cudaEventRecord(g->e1, g->stream));
        GCK(cudaEventSynchronize(g->e1));
        float ms = 0;
        cudaEventElapsedTime(&ms, g->e0, g->e1);
        g->stats[0] = g->total_slots;
        g->stats[4] = (uint64_t)(ms * 1000.0f);
        g->stats[5] = g->n_keys;
        return s;
    }
    uint64_t rewritten = 0;
    if (nwin) {
        // 5. rewrite the windows: gather, sort, spread
        uint64_t* woff = nullptr;
        if ((s = galloc(g, woff, nwin + 1)) != CGB_OK) return s;
        bytes = 0;
        GCK(cub::DeviceScan::ExclusiveSum(nullptr, bytes, wcount, woff, nwin, g->stream));
        if ((s = gtemp(g, bytes)) != CGB_OK) return s;
        GCK(cub::DeviceScan::ExclusiveSum(g->temp, bytes, wcount, woff, nwin, g->stream));
        unsigned long long tail[2];
        GCK(cudaMemcpyAsync(&tail[0], woff + nwin - 1, 8, cudaMemcpyDeviceToHost, g->stream));
        GCK(cudaMemcpyAsync(&tail[1], wcount + nwin - 1, 8, cudaMemcpyDeviceToHost, g->stream));
        GCK(cudaStreamSynchronize(g->stream));
        const uint64_t total = tail[0] + tail[1];
        uint64_t *tmp = nullptr, *srt = nullptr;
        if ((s = galloc(g, tmp, total)) != CGB_OK) return s;
        if ((s = galloc(g, srt, total)) != CGB_OK) return s;
        GCK(cudaMemcpyAsync(woff + nwin, &total, 8, cudaMemcpyHostToDevice, g->stream));
        unsigned int* d_bad = d_flags + 1;  // cleared at the start of the batch
        k_gp_gather<<<grid_of(L * 32), 256, 0, g->stream>>>(win, widx, pmax, L, woff, Q, g->slots, g->valid, tmp, d_bad);
        if (nins)
            k_gp_place_ins<<<grid_of(nins), 256, 0, g->stream>>>(ins_key, ins_leaf, nins, widx, pmax, woff, win, wfill,
                                                                 tmp, d_bad);
        unsigned int hb = 0;
        GCK(cudaMemcpyAsync(&hb, d_bad, 4, cudaMemcpyDeviceToHost, g->stream));
        GCK(cudaStreamSynchronize(g->stream));
        if (hb) return gfail(g, CGB_ERR_STATE, "internal: window bookkeeping inconsistent (no key written out of place)");
        bytes = 0;
        GCK(cub::DeviceSegmentedSort::SortKeys(nullptr, bytes, tmp, srt, total, nwin, woff, woff + 1, g->stream));
        if ((s = gtemp(g, bytes)) != CGB_OK) return s;
        GCK(cub::DeviceSegmentedSort::SortKeys(g->temp, bytes, tmp, srt, total, nwin, woff, woff + 1, g->stream));
        k_gp_scatter<<<grid_of(L * 32), 256, 0, g->stream>>>(win, widx, pmax, L, woff, srt, g->slots, g->valid);
        rewritten = total;
    }
    GCK(cudaGetLastError());
    GCK(cudaEventRecord(g->e1, g->stream));
    if ((s = recount(g)) != CGB_OK) return s;
    float ms = 0;
    cudaEventElapsedTime(&ms, g->e0, g->e1);
    g->stats[0] = g->total_slots;
    g->stats[1] = nwin;
    g->stats[2] = rewritten;
    g->stats[3] = 0;
    g->stats[4] = (uint64_t)(ms * 1000.0f);
    g->stats[5] = g->n_keys;
    reclaim(g);
    return CGB_OK;
}

cgb_status cgb_gpma_extract(cgb_gpma* g, uint32_t dir, uint64_t* out_device, uint64_t cap, uint64_t* n_out) {
    if (!g || !n_out || dir >= g->nd) return CGB_ERR_ARG;
    GCK(cudaSetDevice(g->device));
    const GpmaDir& D = g->dirs[dir];
    cgb_status s;
    if (g->counts_stale && (s = recount(g)) != CGB_OK) return s;
    const uint64_t m = g->dir_n[dir];  // kept by every load and update
    *n_out = m;
    if (!out_device) return CGB_OK;
    if (cap < m) return gfail(g, CGB_ERR_ARG, "buffer holds %llu of %llu keys", (unsigned long long)cap, (unsigned long long)m);
    if (!m) return CGB_OK;
    reclaim(g);
    if ((s = after_default_stream(g)) != CGB_OK) return s;
    const uint64_t L = D.cap / kSeg;
    uint64_t* off = nullptr;
    if ((s = galloc(g, off, L)) != CGB_OK) return s;
    size_t bytes = 0;
    GCK(cub::DeviceScan::ExclusiveSum(nullptr, bytes, g->leaf_cnt + D.leaf0, off, L, g->stream));
    if ((s = gtemp(g, bytes)) != CGB_OK) return s;
    GCK(cub::DeviceScan::ExclusiveSum(g->temp, bytes, g->leaf_cnt + D.leaf0, off, L, g->stream));
    k_gp_extract<<<grid_of(L * 32), 256, 0, g->stream>>>(g->slots + D.off, g->valid + D.off, L, off, out_device);
    GCK(cudaGetLastError());
    GCK(cudaStreamSynchronize(g->stream));
    reclaim(g);
    return CGB_OK;
}

cgb_status cgb_gpma_stats(const cgb_gpma* g, uint64_t* out6) {
    if (!g || !out6) return CGB_ERR_ARG;
    for (int i = 0; i < 6; ++i) out6[i] = g->stats[i];
    return CGB_OK;
}

}  // extern "C"
