// Device engine: slack CSR/CSC build, persistent peel, incremental row
// transitions, skyline assembly and dense row expansion.
//
// Reference path (llysdal/d-core-cuda):
//   graph upload      moveGraphToDevice, src/cuda_memory.h:32-41
//   peel pass         scan + process kernels driven by KListInplace,
//                     main.cu:27-141, 171-195
//   decomposition     dcore, main.cu:197-262 (kmax via swapInOut, then one
//                     pass per k = 0..kmax)
// The engine computes the same numbers with a different schedule: one
// persistent cooperative kernel per pass (levels and rows follow one another
// without a barrier, a device work queue for cascades, no host round trip per
// level), and rows k >= 1 derived from row k-1 by h-index refinement instead
// of one fresh peel per row (see k_trans2).
#include <atomic>
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <vector>

#include "dc_engine.cuh"
#include "dc_internal.h"

namespace dc {

// Kernel launches issued by the engine since load (host counter).
std::atomic<unsigned long long> g_launches{0};

#define DC_CUDA(call)                                                                        \
    do {                                                                                     \
        cudaError_t _e = (call);                                                             \
        if (_e != cudaSuccess)                                                               \
            return set_error(DC_ERR_CUDA, "%s failed: %s (%s:%d)", #call, cudaGetErrorString(_e), \
                             __FILE__, __LINE__);                                            \
    } while (0)

static constexpr int kThreads = 256;
static constexpr int kWarpsPerBlock = kThreads / 32;

// ---------------------------------------------------------------------------
// small helpers
// ---------------------------------------------------------------------------

// Device buffers of a handle come from the device's stream-ordered pool on
// the handle's stream: no implicit device-wide synchronisation, so handles on
// different streams (the serving loop runs many) keep their kernels
// overlapping while they allocate and free.
template <typename T>
static int dmalloc(cudaStream_t st, T** p, uint64_t n) {
    *p = nullptr;
    if (n == 0) n = 1;
    cudaError_t e = cudaMallocAsync((void**)p, n * sizeof(T), st);
    if (e != cudaSuccess) {
        *p = nullptr;
        cudaGetLastError();
        return set_error(DC_ERR_NOMEM, "device allocation of %llu bytes failed: %s",
                         (unsigned long long)(n * sizeof(T)), cudaGetErrorString(e));
    }
    return DC_OK;
}
template <typename T>
static void dfree(cudaStream_t st, T*& p) {
    if (p) cudaFreeAsync((void*)p, st);
    p = nullptr;
}

__device__ __forceinline__ unsigned warp_incl_scan(unsigned x) {
    const unsigned lane = threadIdx.x & 31u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= (unsigned)o) x += y;
    }
    return x;
}

__device__ __forceinline__ unsigned long long warp_incl_scan64(unsigned long long x) {
    const unsigned lane = threadIdx.x & 31u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= (unsigned)o) x += y;
    }
    return x;
}

// Block-wide exclusive scan of one 64-bit value per thread; returns the block
// total through *total.
__device__ unsigned long long block_excl_scan64(unsigned long long x, unsigned long long* total) {
    __shared__ unsigned long long s_w[33];  // exclusive sums of up to 32 warps, total
    const unsigned lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    unsigned long long inc = warp_incl_scan64(x);
    if (lane == 31) s_w[w] = inc;
    __syncthreads();
    if (w == 0) {
        unsigned nw = blockDim.x >> 5;
        unsigned long long v = lane < nw ? s_w[lane] : 0ull;
        unsigned long long vi = warp_incl_scan64(v);
        if (lane < nw) s_w[lane] = vi - v;
        if (lane == nw - 1) s_w[32] = vi;
    }
    __syncthreads();
    unsigned long long res = inc - x + s_w[w];
    *total = s_w[32];
    __syncthreads();
    return res;
}

// Block-wide append: threads with pred get consecutive positions of a list
// (counter *ctr), one atomic per block.  All threads of the block call it.
__device__ __forceinline__ unsigned block_append(unsigned* ctr, bool pred) {
    __shared__ unsigned s_base;
    unsigned long long tot;
    const unsigned long long ex = block_excl_scan64(pred ? 1ull : 0ull, &tot);
    if (threadIdx.x == 0) s_base = tot ? atomicAdd(ctr, (unsigned)tot) : 0u;
    __syncthreads();
    const unsigned pos = s_base + (unsigned)ex;
    __syncthreads();
    return pos;
}

// ---------------------------------------------------------------------------
// exclusive prefix sums of one or two arrays, n elements each
// ---------------------------------------------------------------------------
// Two plain launches: every block sums its range (the last one to finish
// scans the sums), then every block writes its range.  A grid of small arrays
// is bound by launches and round trips: 10,000 elements took 14 us in one
// cooperative launch with two grid barriers, plus 6 us in the kernels that
// widened and narrowed the values around it, once per side; these take 6 us
// for both sides.  Long arrays are bound by memory, read twice.
constexpr int kScanThreads = 256, kScanTile = 4 * kScanThreads;
struct WordsInPlace {  // data[0 .. n] becomes the sums, data[n] the total
    unsigned long long* data;
    __device__ unsigned long long get(int, uint64_t i) const { return data[i]; }
    __device__ void put(int, uint64_t i, unsigned long long x) const { data[i] = x; }
};
struct ListStarts {  // starts of lists with room for max(gap_min, len / gap_div) more entries each
    const int32_t* len[2];
    uint32_t* off[2];
    uint32_t gap_min, gap_div;
    __device__ unsigned long long get(int side, uint64_t i) const {
        const uint32_t l = (uint32_t)len[side][i];
        return (unsigned long long)l + (gap_div ? max(gap_min, l / gap_div) : gap_min);
    }
    __device__ void put(int side, uint64_t i, unsigned long long x) const { off[side][i] = (uint32_t)x; }
};
__device__ __forceinline__ uint64_t scan_range(uint64_t n) {  // elements per block
    const uint64_t per = (n + gridDim.x - 1) / gridDim.x;
    return (per + kScanTile - 1) / kScanTile * kScanTile;
}
// part: gridDim.x + 1 words per side; *ticket is 0 before and after.
// total (optional): one word per side.
template <class A>
__global__ void __launch_bounds__(kScanThreads) k_scan_sums(A a, uint64_t n, unsigned long long* part, unsigned* ticket,
                                                            unsigned long long* total) {
    __shared__ bool s_last;
    const uint64_t per = scan_range(n), lo = min(n, per * blockIdx.x), hi = min(n, lo + per);
    unsigned long long s = 0, tot;
    for (uint64_t i = lo + threadIdx.x; i < hi; i += kScanThreads) s += a.get(blockIdx.y, i);
    block_excl_scan64(s, &tot);
    if (threadIdx.x == 0) {
        part[blockIdx.y * (gridDim.x + 1) + blockIdx.x] = tot;
        __threadfence();
        s_last = atomicAdd(ticket, 1u) == gridDim.x * gridDim.y - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (unsigned side = 0; side < gridDim.y; ++side) {
        volatile unsigned long long* q = part + side * (gridDim.x + 1);
        unsigned long long carry = 0;
        for (unsigned b0 = 0; b0 < gridDim.x; b0 += kScanThreads) {
            const unsigned b = b0 + threadIdx.x;
            const unsigned long long x = b < gridDim.x ? q[b] : 0ull;
            const unsigned long long ex = block_excl_scan64(x, &tot);
            if (b < gridDim.x) q[b] = ex + carry;
            carry += tot;
        }
        if (threadIdx.x == 0) {
            q[gridDim.x] = carry;
            if (total) total[side] = carry;
        }
    }
    if (threadIdx.x == 0) *ticket = 0;
}
template <class A>
__global__ void __launch_bounds__(kScanThreads) k_scan_apply(A a, uint64_t n, const unsigned long long* part) {
    const uint64_t per = scan_range(n), lo = min(n, per * blockIdx.x), hi = min(n, lo + per);
    const unsigned long long* q = part + blockIdx.y * (gridDim.x + 1);
    unsigned long long carry = q[blockIdx.x];
    for (uint64_t b0 = lo; b0 < hi; b0 += kScanTile) {
        const uint64_t i0 = b0 + 4 * threadIdx.x;
        unsigned long long x[4], tot;
#pragma unroll
        for (int j = 0; j < 4; ++j) x[j] = i0 + j < hi ? a.get(blockIdx.y, i0 + j) : 0ull;
        unsigned long long at = carry + block_excl_scan64(x[0] + x[1] + x[2] + x[3], &tot);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (i0 + j < hi) a.put(blockIdx.y, i0 + j, at);
            at += x[j];
        }
        carry += tot;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) a.put(blockIdx.y, n, q[gridDim.x]);
}

// ---------------------------------------------------------------------------
// graph build
// ---------------------------------------------------------------------------
// Edge lists usually come grouped by source (files, generators, a rebuilt
// store): a warp takes 128 consecutive edges, and each run of equal sources in
// a row of 32 is one atomic.  Bound by L2 atomics (65 M edges: one per edge and
// side took 1.0 ms to count and 2.2 ms to place); ungrouped edges form runs
// of one.
// Lane's place in its run of equal x and the run's length; lanes of a run are
// consecutive.
__device__ __forceinline__ void warp_run(uint32_t x, unsigned* first, unsigned* length) {
    const unsigned lane = threadIdx.x & 31u;
    const uint32_t prev = __shfl_up_sync(0xFFFFFFFFu, x, 1);
    const unsigned heads = __ballot_sync(0xFFFFFFFFu, lane == 0 || x != prev);
    *first = 31u - __clz(heads & (0xFFFFFFFFu >> (31u - lane)));
    const unsigned after = lane == 31 ? 0u : heads & (0xFFFFFFFFu << (lane + 1u));
    *length = (after ? __ffs(after) - 1u : 32u) - *first;
}

__global__ void k_count_degrees(uint32_t V, uint64_t E, const uint32_t* src, const uint32_t* dst, int32_t* out_len,
                                int32_t* in_len, EngineCtl* c) {
    const unsigned lane = threadIdx.x & 31u;
    const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t b = gw * 128; b < E; b += nw * 128) {
        uint32_t s[4], d[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const uint64_t e = b + 32 * r + lane;
            s[r] = d[r] = 0xFFFFFFFFu;
            if (e < E) {
                s[r] = src[e];
                d[r] = dst[e];
                if (s[r] >= V || d[r] >= V) {
                    set_dev_error(c, DC_DEV_ERR_BADID, 10);
                    s[r] = d[r] = 0xFFFFFFFFu;
                }
            }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            unsigned first, length;
            warp_run(s[r], &first, &length);
            if (s[r] != 0xFFFFFFFFu) {
                if (first == lane) atomicAdd(&out_len[s[r]], (int)length);
                atomicAdd(&in_len[d[r]], 1);
            }
        }
    }
}

__global__ void k_scatter_edges(uint64_t E, const uint32_t* src, const uint32_t* dst, const uint32_t* out_off,
                                int32_t* out_fill, uint32_t* out_nbr, const uint32_t* in_off, int32_t* in_fill,
                                uint32_t* in_nbr) {
    const unsigned lane = threadIdx.x & 31u;
    const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t b = gw * 128; b < E; b += nw * 128) {
        uint32_t s[4], d[4], oo[4], io[4];
        unsigned first[4];
        int po[4], pi[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const uint64_t e = b + 32 * r + lane;
            s[r] = e < E ? src[e] : 0xFFFFFFFFu;
            d[r] = e < E ? dst[e] : 0xFFFFFFFFu;
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            unsigned length;
            warp_run(s[r], &first[r], &length);
            po[r] = pi[r] = 0;
            oo[r] = io[r] = 0;
            if (s[r] != 0xFFFFFFFFu) {
                if (first[r] == lane) po[r] = atomicAdd(&out_fill[s[r]], (int)length);
                pi[r] = atomicAdd(&in_fill[d[r]], 1);
                oo[r] = out_off[s[r]];
                io[r] = in_off[d[r]];
            }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int at = __shfl_sync(0xFFFFFFFFu, po[r], first[r]) + (int)(lane - first[r]);
            if (s[r] != 0xFFFFFFFFu) {
                out_nbr[oo[r] + (uint32_t)at] = d[r];
                in_nbr[io[r] + (uint32_t)pi[r]] = s[r];
            }
        }
    }
}

// ---------------------------------------------------------------------------
// incremental rows: shared helpers
// ---------------------------------------------------------------------------
static constexpr int kWin = 64;

// Per-vertex queue state for the transition drain: bit 0 = requested, bit 1
// = being evaluated.  A vertex is never evaluated by two warps at once, and a
// request that lands during an evaluation re-queues the vertex when that
// evaluation ends.  Returns true when the caller must push the vertex.
__device__ __forceinline__ bool mark_request(uint32_t* m) { return atomicOr(m, 1u) == 0u; }

// ---------------------------------------------------------------------------
// fused peel
// ---------------------------------------------------------------------------
struct PeelInst {
    const uint32_t* a_off;
    const int32_t* a_len;
    const uint32_t* a_nbr;
    const uint32_t* b_off;
    const int32_t* b_len;
    const uint32_t* b_nbr;
    const int32_t* member;  // nullptr: all vertices
    int32_t k;              // constraint threshold (0: none)
    int32_t* key;
    int32_t* cdeg;
    int32_t* val;
    uint32_t* rem0;
    uint32_t* rem1;
};

struct Peel2Params {
    uint32_t V;
    int ninst;
    unsigned chunk;  // a list longer than 4 chunks is split into items of that size
    PeelInst in[2];
    uint32_t* bag;  // [2 V] vertices handed to other warps
    TicketQueue q;
    EngineCtl* ctl;
};

// Queue items: a removed vertex (piece 0: its taker queues the other pieces of
// a long list), a further piece of a long list, or a bag of up to 32 removed
// vertices (start in the bag array, count).
constexpr unsigned long long kPeelInst = 1ull << 32, kPeelBag = 1ull << 33;
constexpr int kPeelDetail = 34;  // 20 bits: piece or count
// Vertices in a warp's stack and in the bags carry their instance in the top
// bit (2^31 vertices would not fit the device: the scratch alone takes 88
// bytes per vertex).
constexpr uint32_t kPeelTop = 0x80000000u;
constexpr int kPeelEnd = 0x7FFFFFFF;  // level: nothing remains

constexpr unsigned kPeelStack = 384;   // vertices in a warp's stack
// 256 and 96 or 384 entries measure the same within 1 %.
constexpr unsigned kPeelBatch = 512;   // entries a warp starts on at a time
constexpr unsigned kPeelShare = 192;   // entries a warp keeps for itself when others wait
// and vertices: where lists are short and a removal's turn comes with the last
// of its neighbours, as in a grid or a layered graph, one warp removes most of
// a wave and every further batch of 32 is a link of the chain.  8 / 16 / 24 / 32
// / any number: 400 x 400 grid 2.0 / 2.0 / 2.6 / 2.6 / 14.0 ms, 300 layers of
// 500 1.2 / 1.2 / 1.3 / 1.7 / 5.1, 100 layers of 2,000 with eight edges 0.61 /
// 0.66 / 0.80 / 0.80 / 0.79, R-MAT 20 4.29 / 4.30 / 4.29 / 4.27 / 4.23.
constexpr unsigned kPeelKeep = 16;

// Entries per item of a list of len entries (piece numbers have 20 bits).
__device__ __forceinline__ unsigned peel_unit(unsigned chunk, unsigned len) {
    unsigned u = 4 * chunk;
    while (len > ((unsigned long long)u << 20)) u <<= 1;
    return u;
}

struct PeelHook {
    int ninst;
    unsigned blocks;
    __device__ unsigned begin(unsigned) const { return blocks; }
    __device__ __forceinline__ int operator()(EngineCtl* c, int level, bool worked, int bound) const {
        for (int i = 0; i < ninst; ++i) {
            unsigned n = ld_vol(&c->rc_cur[i]);
            if (ld_vol(&c->peel_compact[i])) {
                n = ld_vol(&c->rc_next[i].v);
                c->rc_cur[i] = n;
                c->rc_next[i].v = 0;
                c->peel_list[i] = ld_vol(&c->peel_list[i]) == 0 ? 1 : 0;
                c->removed_at[i] = ld_vol(&c->removed[i]);
                c->peel_compact[i] = 0;
            } else {
                // the list is written anew once a quarter of it is gone
                c->peel_compact[i] = 4ull * (ld_vol(&c->removed[i]) - ld_vol(&c->removed_at[i])) > n;
            }
        }
        // a level whose scan found nothing to remove changed no degree: the
        // levels up to the least degree kept are empty too
        return worked ? level + 1 : bound == kNoBound ? kPeelEnd : max(level + 1, bound);
    }
};
// Run by the last block to finish the initialisation.
struct PeelStart {
    int ninst;
    uint32_t V;
    bool member;
    __device__ void operator()(EngineCtl* c) const {
        for (int i = 0; i < ninst; ++i) {
            c->rc_cur[i] = c->members[i] = member ? c->rc_next[i].v : V;
            c->rc_next[i].v = 0;
            c->peel_list[i] = member ? 0 : -1;
            c->peel_compact[i] = 1;
        }
        __threadfence();
    }
};

// One warp's part of the peel: removed vertices wait on the warp's own stack
// in shared memory, and what it cannot hold or others can start on at once
// goes to them through the queue.
template <bool kBoth>
struct PeelWarp {
    const Peel2Params& p;
    EngineCtl* c;
    uint32_t* stack;
    unsigned n;  // vertices on the stack (the same on every lane)
    int L;
    unsigned long long tag;
    unsigned peeled0, peeled1;  // this warp's removals not reported yet, per peel
    int maxv0, maxv1;           // last level with one

    // nb bags of sz (<= 32) vertices each from the stack's top to the queue.
    __device__ void spill(unsigned nb, unsigned sz) {
        const unsigned lane = threadIdx.x & 31u, total = nb * sz;
        unsigned at = 0;
        if (lane == 0) at = atomicAdd(&c->bag_tail, total);
        at = __shfl_sync(0xFFFFFFFFu, at, 0);
        n -= total;
        __syncwarp();
        for (unsigned k = lane; k < total; k += 32) *(volatile uint32_t*)&p.bag[at + k] = stack[n + k];
        __threadfence();
        __syncwarp();
        const unsigned base = step_reserve(c, nb);
        for (unsigned k = lane; k < nb; k += 32)
            step_put(p.q, base + k, (unsigned long long)(at + k * sz) | kPeelBag |
                                        ((unsigned long long)sz << kPeelDetail) | tag);
    }

    // A vertex's lists end to end: the constraint list, if any, then the other.
    struct List {
        unsigned len, la;      // entries in all, entries of the constraint list
        uint32_t aoff, boff;   // starts
    };
    __device__ __forceinline__ List list_of(uint32_t v, int i) const {
        const PeelInst& I0 = p.in[0];
        const PeelInst& I1 = p.in[1];
        List l{0u, 0u, 0u, 0u};
        l.len = (unsigned)__ldg((i ? I1.b_len : I0.b_len) + v);
        l.boff = __ldg((i ? I1.b_off : I0.b_off) + v);
        if (kBoth) {
            l.la = (unsigned)__ldg((i ? I1.a_len : I0.a_len) + v);
            l.aoff = __ldg((i ? I1.a_off : I0.a_off) + v);
            l.len += l.la;
        }
        return l;
    }

    // Lanes with cnt > 0 hold the entries [e0, e0 + cnt) of a vertex's lists
    // (instance i): all of them are spread over the warp's lanes, four in
    // flight per lane; every entry takes one from its neighbour's degree.
    __device__ void entries(const List& l, int i, unsigned e0, unsigned cnt) {
        const unsigned lane = threadIdx.x & 31u;
        const unsigned incl = warp_incl_scan(cnt);
        const unsigned T = __shfl_sync(0xFFFFFFFFu, incl, 31);
        const PeelInst& I0 = p.in[0];
        const PeelInst& I1 = p.in[1];
        // entry of t: rel + t; rel and the bases may be "negative", so the sums
        // with t are taken in 32 bits before they index anything
        const unsigned rel = e0 - (incl - cnt);
        const unsigned la = l.la, abase = l.aoff, bbase = l.boff + rel - la;
        for (unsigned t0 = 0; t0 < T; t0 += 128) {
            if (n > kPeelStack - 128) spill(4, 32);
            uint32_t u[4];
            int io[4], old[4];
            bool isa[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const unsigned t = t0 + 32 * r + lane;
                unsigned o = 0;
#pragma unroll
                for (unsigned s = 16; s; s >>= 1)
                    if (__shfl_sync(0xFFFFFFFFu, incl, o + s - 1) <= t) o += s;
                o = min(o, 31u);
                const unsigned bb = __shfl_sync(0xFFFFFFFFu, bbase, o);
                io[r] = __shfl_sync(0xFFFFFFFFu, i, o);
                isa[r] = false;
                if (kBoth) {
                    const unsigned ab = __shfl_sync(0xFFFFFFFFu, abase, o), re = __shfl_sync(0xFFFFFFFFu, rel, o);
                    isa[r] = re + t < __shfl_sync(0xFFFFFFFFu, la, o);
                    if (isa[r] && t < T) u[r] = __ldg((io[r] ? I1.a_nbr : I0.a_nbr) + (ab + re + t));
                }
                if (!isa[r]) u[r] = t < T ? __ldg((io[r] ? I1.b_nbr : I0.b_nbr) + (bb + t)) : 0u;
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const unsigned t = t0 + 32 * r + lane;
                old[r] = 0x80000000;
                if (t < T)
                    old[r] = atomicSub(isa[r] ? (io[r] ? I1.cdeg : I0.cdeg) + u[r] : (io[r] ? I1.key : I0.key) + u[r], 1);
            }
            bool any = false;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int lim = isa[r] ? (io[r] ? I1.k : I0.k) : L + 1;
                old[r] = (t0 + 32 * r + lane < T && old[r] == lim) ? 1 : 0;
                any |= old[r] != 0;
            }
            if (__any_sync(0xFFFFFFFFu, any)) {
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    if (old[r]) old[r] = atomicCAS((io[r] ? I1.val : I0.val) + u[r], -1, L) == -1 ? 1 : 0;
#pragma unroll
                for (int r = 0; r < 4; ++r) take_removed(old[r] != 0, u[r], io[r]);
            }
        }
    }

    // Converged warp: lanes with pred add vertex v to the stack.
    __device__ __forceinline__ void take_removed(bool pred, uint32_t v, int i) {
        const unsigned lane = threadIdx.x & 31u;
        const unsigned m = __ballot_sync(0xFFFFFFFFu, pred);
        if (!m) return;
        if (pred) stack[n + __popc(m & ((1u << lane) - 1u))] = v | (i ? kPeelTop : 0u);
        n += __popc(m);
        const unsigned m1 = __ballot_sync(0xFFFFFFFFu, pred && i != 0);
        peeled0 += __popc(m & ~m1);
        peeled1 += __popc(m1);
        if (m & ~m1) maxv0 = L;
        if (m1) maxv1 = L;
    }

    // Converged warp: the pieces after the first of the long lists (lanes with
    // len > unit) go to the queue.
    __device__ void push_pieces(uint32_t v, int i, unsigned len, unsigned unit) {
        const unsigned lane = threadIdx.x & 31u;
        unsigned m = __ballot_sync(0xFFFFFFFFu, len > unit);
        while (m) {
            const unsigned o = __ffs(m) - 1;
            m &= m - 1u;
            const uint32_t x = __shfl_sync(0xFFFFFFFFu, v, o);
            const int ix = __shfl_sync(0xFFFFFFFFu, i, o);
            const unsigned l = __shfl_sync(0xFFFFFFFFu, len, o), un = __shfl_sync(0xFFFFFFFFu, unit, o);
            const unsigned more = (l - 1) / un;
            const unsigned base = step_reserve(c, more);
            for (unsigned k = lane; k < more; k += 32)
                step_put(p.q, base + k, (unsigned long long)x | (ix ? kPeelInst : 0ull) |
                                            ((unsigned long long)(k + 1) << kPeelDetail) | tag);
        }
    }

    // nb vertices from the stack's top to the queue, one item each.
    __device__ void give(unsigned nb) {
        n -= nb;
        const unsigned base = step_reserve(c, nb);
        for (unsigned k = threadIdx.x & 31u; k < nb; k += 32) {
            const uint32_t e = stack[n + k];
            step_put(p.q, base + k, (unsigned long long)(e & ~kPeelTop) | ((e & kPeelTop) ? kPeelInst : 0ull) | tag);
        }
    }

    // The stack's only vertex (lane 0's l, i; at most 32 entries), an entry per
    // lane without a search for its place: chains of single removals are the
    // peel's longest (60,000 links 113 -> 71 ms, 104 with an item per vertex).
    __device__ __forceinline__ void single(const List& l0, int i0) {
        const unsigned lane = threadIdx.x & 31u;
        const unsigned len = __shfl_sync(0xFFFFFFFFu, l0.len, 0), la = kBoth ? __shfl_sync(0xFFFFFFFFu, l0.la, 0) : 0u;
        const unsigned ab = kBoth ? __shfl_sync(0xFFFFFFFFu, l0.aoff, 0) : 0u, bb = __shfl_sync(0xFFFFFFFFu, l0.boff, 0);
        const int i = __shfl_sync(0xFFFFFFFFu, i0, 0);
        const PeelInst& I0 = p.in[0];
        const PeelInst& I1 = p.in[1];
        n = 0;
        uint32_t u = 0;
        bool gone = false;
        if (lane < len) {
            const bool isa = kBoth && lane < la;
            u = isa ? __ldg((i ? I1.a_nbr : I0.a_nbr) + (ab + lane)) : __ldg((i ? I1.b_nbr : I0.b_nbr) + (bb + (lane - la)));
            const int old = atomicSub(isa ? (i ? I1.cdeg : I0.cdeg) + u : (i ? I1.key : I0.key) + u, 1);
            gone = old == (isa ? (i ? I1.k : I0.k) : L + 1) && atomicCAS((i ? I1.val : I0.val) + u, -1, L) == -1;
        }
        __syncwarp();
        take_removed(gone, u, i);
    }

    // Works off the stack, 32 vertices at a time from its top (fewer when
    // their lists are long).  What remains is shared once it is more than
    // half a batch or a moment's work and warps wait: one vertex each while
    // they last, else bags of 32.  (Sharing by the number of vertices alone left one warp with
    // 2.8 ms of long lists in one level of R-MAT 22.)
    __device__ void drain() {
        const unsigned lane = threadIdx.x & 31u;
        while (n) {
            __syncwarp();
            const bool has = lane < n;
            const uint32_t e = has ? stack[n - 1 - lane] : 0u;
            const uint32_t v = e & ~kPeelTop;
            const int i = e >> 31;
            List l{0u, 0u, 0u, 0u};
            if (has) l = list_of(v, i);
            if (n == 1 && __shfl_sync(0xFFFFFFFFu, l.len, 0) <= 32u) {
                single(l, i);
                continue;
            }
            const unsigned unit = peel_unit(p.chunk, l.len);
            unsigned cnt = min(l.len, unit);
            const unsigned before = warp_incl_scan(cnt) - cnt;
            const bool mine = has && before < kPeelBatch;
            const unsigned m = __popc(__ballot_sync(0xFFFFFFFFu, mine));
            const unsigned total = __shfl_sync(0xFFFFFFFFu, before + cnt, m - 1);
            n -= m;
            __syncwarp();
            if (!mine) cnt = l.len = 0;
            push_pieces(v, i, l.len, unit);
            entries(l, i, 0u, cnt);
            __syncwarp();
            if (n > kPeelKeep || (n > 1 && (unsigned long long)n * total > (unsigned long long)kPeelShare * m)) {
                const int idle = (int)(ld_vol(&c->t_head) -
                                       (unsigned)*reinterpret_cast<volatile unsigned long long*>(&c->t_work));
                const unsigned own = min(kPeelKeep, max(1u, kPeelShare * m / max(total, 1u)));
                if (idle > 0 && n > own) {
                    const unsigned more = n - own;
                    if (more <= 32 || (unsigned)idle >= more) give(min((unsigned)idle, more));
                    else spill(min((unsigned)idle, more / 32), 32);
                }
            }
        }
        __syncwarp();
    }

    // A queue item.
    __device__ void item(unsigned long long it) {
        const unsigned lane = threadIdx.x & 31u;
        const unsigned detail = (unsigned)(it >> kPeelDetail) & 0xFFFFFu;
        uint32_t v = (uint32_t)it;
        int i = (it & kPeelInst) ? 1 : 0;
        unsigned e0 = 0, cnt = 0, unit = 1;
        List l{0u, 0u, 0u, 0u};
        if (it & kPeelBag) {
            if (lane < detail) {
                const uint32_t e = ld_vol(&p.bag[v + lane]);
                v = e & ~kPeelTop;
                i = e >> 31;
                l = list_of(v, i);
                unit = peel_unit(p.chunk, l.len);
                cnt = min(l.len, unit);
            }
            push_pieces(v, i, l.len, unit);
        } else {
            if (lane == 0) {
                l = list_of(v, i);
                unit = peel_unit(p.chunk, l.len);
                e0 = detail * unit;
                cnt = min(unit, l.len - e0);
            }
            if (!detail) push_pieces(v, i, l.len, unit);
        }
        __syncwarp();
        entries(l, i, e0, cnt);
        drain();
    }
};

// Up to two independent peels advance level by level in one grid: the kmax
// pass (peeling in-degree, swapInOut + KListInplace(k = 0), main.cu:218-220)
// and row 0 (peeling out-degree), or two rows of the per-row method.  Level
// L of each peel removes every remaining vertex whose peeling degree is at
// most L (scan, main.cu:37-56) and the cascade that follows (process,
// main.cu:100-135) with value L.
//
// Bound by latency in the light levels and, with one queue item per removed
// vertex, by the queue's same-address atomics in the heavy ones (2.5 ns per
// item, 4 M items in 14 levels of R-MAT 22).  So a removed vertex stays with
// the warp that removed it, on a stack in shared memory; 32 of them are worked
// off together, their lists laid end to end over the lanes with four entries
// in flight per lane; the queue carries only the pieces of long lists and
// vertices that waiting warps can start on.  Levels advance without a grid
// barrier.  The remaining vertices' list is scanned once per level for both
// peels together and written anew only when a quarter of it is gone.
// kBoth: the instances have a constraint list too (rows k >= 1).
#ifndef DC_PEEL_MIN_BLOCKS
#define DC_PEEL_MIN_BLOCKS 4
#endif
template <bool kBoth>
__global__ void __launch_bounds__(kThreads, DC_PEEL_MIN_BLOCKS) k_peel2(Peel2Params p) {
    const unsigned lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
    const unsigned gwarp = blockIdx.x * kWarpsPerBlock + wib;
    const unsigned nwarps = gridDim.x * kWarpsPerBlock;
    EngineCtl* c = p.ctl;
    __shared__ uint32_t s_stack[kWarpsPerBlock][kPeelStack];
    __shared__ StepBlock s_step;
    const bool tracing = c->trace != nullptr;

    // ---- init
    for (int i = 0; i < p.ninst; ++i) {
        const PeelInst& I = p.in[i];
        for (uint64_t base = (uint64_t)blockIdx.x * kThreads; base < p.V; base += (uint64_t)gridDim.x * kThreads) {
            const uint64_t vi = base + threadIdx.x;
            const uint32_t v = (uint32_t)vi;
            if (!kBoth) {
                if (vi < p.V) {
                    I.val[v] = -1;
                    I.key[v] = __ldg(I.a_len + v);
                }
                continue;
            }
            const bool in = vi < p.V && I.member[v] >= I.k;
            if (vi < p.V && !in) I.val[v] = 0;
            if (in) {
                I.val[v] = -1;
                int kd = 0, cd = 0;
                uint32_t o = I.a_off[v], e = o + (uint32_t)I.a_len[v];
                for (; o < e; ++o) kd += (I.member[I.a_nbr[o]] >= I.k);
                o = I.b_off[v];
                e = o + (uint32_t)I.b_len[v];
                for (; o < e; ++o) cd += (I.member[I.b_nbr[o]] >= I.k);
                I.key[v] = kd;
                I.cdeg[v] = cd;
            }
            const unsigned pos = block_append(&c->rc_next[i].v, in);
            if (in) I.rem0[pos] = v;
        }
    }
    if (!grid_sync_hook(c, PeelStart{p.ninst, p.V, kBoth})) return;

    const PeelHook next{p.ninst, gridDim.x};
    PeelWarp<kBoth> w{p, c, s_stack[wib], 0u, 0, 0ull, 0u, 0u, 0, 0};
    unsigned ticket = kNoTicket;
    step_block_init(&s_step, c);
    unsigned long long word = step_block_word(&s_step);
    for (;;) {
        const int L = step_level(word);
        if (word == kStopWord || L == kPeelEnd) break;
        if (tracing && threadIdx.x == 0) trace_wake(c, word);
        w.L = L;
        w.tag = step_tag(word);
        int pending = 0;
        int bound = kNoBound;
        // ---- scan of the remaining vertices, both peels together
        unsigned nr[2] = {0, 0};
        bool compact[2] = {false, false};
        const uint32_t* from[2] = {nullptr, nullptr};
        uint32_t* to[2] = {nullptr, nullptr};
        bool wrote = false;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if (i >= p.ninst) continue;
            const int l = ld_vol(&c->peel_list[i]);
            nr[i] = ld_vol(&c->rc_cur[i]);
            compact[i] = ld_vol(&c->peel_compact[i]) != 0;
            from[i] = l < 0 ? nullptr : l == 0 ? p.in[i].rem0 : p.in[i].rem1;
            to[i] = l == 0 ? p.in[i].rem1 : p.in[i].rem0;
        }
        const unsigned before = w.peeled0 + w.peeled1;
        for (uint64_t base = 0; base < max(nr[0], nr[1]); base += 64ull * nwarps) {
            uint32_t v[4];
            int val[4], key[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int i = r >> 1;
                const uint64_t idx = base + (uint64_t)(r & 1) * 32u * nwarps + 32u * gwarp + lane;
                v[r] = 0xFFFFFFFFu;
                if (idx < nr[i]) v[r] = from[i] ? ld_vol(from[i] + idx) : (uint32_t)idx;
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const PeelInst& I = p.in[r >> 1];
                val[r] = 0;
                key[r] = 0;
                if (v[r] != 0xFFFFFFFFu) {
                    val[r] = ld_vol(&I.val[v[r]]);
                    key[r] = ld_vol(&I.key[v[r]]);
                }
            }
#pragma unroll
            for (int r = 0; r < 4; ++r)
                if (val[r] == -1) {
                    if (key[r] <= L) val[r] = atomicCAS(&p.in[r >> 1].val[v[r]], -1, L) == -1 ? -2 : 0;
                    else bound = min(bound, key[r]);
                }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                if (compact[i]) {
                    const unsigned m0 = __ballot_sync(0xFFFFFFFFu, val[2 * i] == -1);
                    const unsigned m1 = __ballot_sync(0xFFFFFFFFu, val[2 * i + 1] == -1);
                    if (m0 | m1) {
                        unsigned at = 0;
                        if (lane == 0) at = atomicAdd(&c->rc_next[i].v, (unsigned)(__popc(m0) + __popc(m1)));
                        at = __shfl_sync(0xFFFFFFFFu, at, 0);
                        const unsigned below = (1u << lane) - 1u;
                        if (val[2 * i] == -1) to[i][at + __popc(m0 & below)] = v[2 * i];
                        if (val[2 * i + 1] == -1) to[i][at + __popc(m0) + __popc(m1 & below)] = v[2 * i + 1];
                        wrote = true;
                    }
                }
                w.take_removed(val[2 * i] == -2, v[2 * i], i);
                w.take_removed(val[2 * i + 1] == -2, v[2 * i + 1], i);
            }
            if (w.n > kPeelStack - 128) w.drain();
        }
        const bool worked = w.peeled0 + w.peeled1 != before;
        w.drain();
        // removals counted so far (those of queue items follow in a later level)
        if (lane == 0) {
            if (w.peeled0) atomicAdd(&s_step.count[0], w.peeled0);
            if (w.peeled1) atomicAdd(&s_step.count[1], w.peeled1);
        }
        w.peeled0 = w.peeled1 = 0;
        if (wrote) __threadfence();
        step_seeded(c, &s_step, bound, worked, word, tracing, next);
        // ---- the queue
        unsigned long long item = 0;
        int state;
        while ((state = step_take(c, p.q, &s_step, &ticket, &item, &pending, &word, next)) == kTakeItem) {
            w.item(item);
            ++pending;
        }
        if (state == kTakeStop) break;
    }
    if (lane == 0) {
        if (w.maxv0) atomicMax(&c->maxv[0], w.maxv0);
        if (w.maxv1) atomicMax(&c->maxv[1], w.maxv1);
    }
}

// The peels of a small graph, one block each: degrees and the removed vertices
// in shared memory, a level's removals in rounds with a block barrier between
// them (a vertex is listed once, when it is removed, so the list never exceeds
// V entries).  The grid's version spends about 10 us on an empty level and 1.2
// us on every link of a chain of removals, here they take about 1 us and 0.5; what bounds it is the entries one SM can take (shared-memory atomics,
// about 2,000 per us), and the other SMs are free for other handles.
struct SmallPeel {
    PeelInst in[2];
    uint32_t V;
    EngineCtl* ctl;
};
constexpr int kSmallPeelThreads = 1024;
constexpr uint32_t kSmallPeelV = 36000;           // 6 bytes of shared memory per vertex
// Faster than the grid's kernel, small / grid in ms: R-MAT 12 0.21 / 0.71,
// 13 (24 edges per vertex) 0.39 / 1.04, 14 (40) 0.75 / 1.45, 15 (32) 1.09 /
// 1.73; ER 1,000 0.05 / 0.15, 10,000 (20) 0.14 / 0.19, but (when the line was
// drawn) 20,000 (20) 0.22 / 0.21 and 30,000 (50) 0.49 / 0.31: where all
// degrees are alike the removals are a few wide cascades, which want the
// chip's atomics.  Hence by the longest list, as it was when the lists were
// built (any choice gives the same result).
static bool peel_fits_block(const DevGraph& g) {
    const bool skewed = g.max_len >= 8 * (g.E / std::max<uint32_t>(g.V, 1) + 4);
    return g.V >= 1 && (skewed ? g.V <= kSmallPeelV && g.E <= 2000000u : g.V <= 16384 && g.E <= 500000u);
}
// longest list of either side
__global__ void k_max_len(uint32_t V, const int32_t* a, const int32_t* b, int* out) {
    int m = 0;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) m = max(m, max(a[v], b[v]));
    m = __reduce_max_sync(0xFFFFFFFFu, m);
    if ((threadIdx.x & 31u) == 0) atomicMax(out, m);
}
constexpr int kSmallPeelGone = 1 << 30;           // taken from the degree of a removed vertex
constexpr unsigned kSmallPeelLong = 256, kSmallPeelLongs = 64;  // lists that the whole block reads
__global__ void __launch_bounds__(kSmallPeelThreads, 1) k_peel_small(SmallPeel p) {
    extern __shared__ int s_key[];
    uint16_t* s_list = reinterpret_cast<uint16_t*>(s_key + p.V);
    __shared__ unsigned s_tail, s_longs, s_long[kSmallPeelLongs];
    __shared__ int s_min;
    const PeelInst& I = p.in[blockIdx.x];
    const unsigned t = threadIdx.x, lane = t & 31u, V = p.V;
    for (unsigned v = t; v < V; v += kSmallPeelThreads) s_key[v] = __ldg(I.a_len + v);
    if (t == 0) s_tail = s_longs = 0;
    int level = 0;
    unsigned head = 0;
    // an entry of a removed vertex's list: one from the neighbour's degree
    auto entry = [&](uint32_t u) {
        if (atomicSub(&s_key[u], 1) == level + 1) {
            atomicSub(&s_key[u], kSmallPeelGone);
            I.val[u] = level;
            s_list[atomicAdd(&s_tail, 1u)] = (uint16_t)u;
        }
    };
    while (head < V) {
        // the next level: the least degree left
        __syncthreads();
        if (t == 0) s_min = 0x7FFFFFFF;
        __syncthreads();
        int m = 0x7FFFFFFF;
        for (unsigned v = t; v < V; v += kSmallPeelThreads) {
            const int k = s_key[v];
            if (k >= 0) m = min(m, k);
        }
        m = __reduce_min_sync(0xFFFFFFFFu, m);
        if (lane == 0) atomicMin(&s_min, m);
        __syncthreads();
        level = s_min;
        if (level == 0x7FFFFFFF) break;  // (no vertex left: head is V)
        for (unsigned b = t - lane; b < V; b += kSmallPeelThreads) {
            const unsigned v = b + lane;
            const int k = v < V ? s_key[v] : -1;
            const bool gone = k >= 0 && k <= level;
            const unsigned mask = __ballot_sync(0xFFFFFFFFu, gone);
            if (!mask) continue;
            unsigned at = 0;
            if (lane == 0) at = atomicAdd(&s_tail, (unsigned)__popc(mask));
            at = __shfl_sync(0xFFFFFFFFu, at, 0);
            if (gone) {
                s_key[v] = k - kSmallPeelGone;
                I.val[v] = level;
                s_list[at + __popc(mask & ((1u << lane) - 1u))] = (uint16_t)v;
            }
        }
        __syncthreads();
        unsigned tail = s_tail;
        __syncthreads();
        while (head < tail) {
            // eight lanes per vertex, four entries in flight each
            for (unsigned i = head + (t >> 3); i < tail; i += kSmallPeelThreads / 8) {
                const uint32_t v = s_list[i], off = __ldg(I.b_off + v);
                const unsigned n = (unsigned)__ldg(I.b_len + v);
                if (n > kSmallPeelLong) {
                    unsigned at = kSmallPeelLongs;
                    if ((t & 7u) == 0) at = atomicAdd(&s_longs, 1u);
                    at = __shfl_sync(0xFFu << (lane & ~7u), at, lane & ~7u);
                    if (at < kSmallPeelLongs) {
                        if ((t & 7u) == 0) s_long[at] = v;
                        continue;
                    }
                }
                for (unsigned e = t & 7u; e < n; e += 32) {
                    uint32_t u[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) u[q] = e + 8 * q < n ? __ldg(I.b_nbr + off + e + 8 * q) : 0xFFFFFFFFu;
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (u[q] != 0xFFFFFFFFu) entry(u[q]);
                }
            }
            __syncthreads();
            const unsigned longs = min(s_longs, kSmallPeelLongs);
            for (unsigned i = 0; i < longs; ++i) {
                const uint32_t v = s_long[i], off = __ldg(I.b_off + v);
                const unsigned n = (unsigned)__ldg(I.b_len + v);
                for (unsigned e = t; e < n; e += kSmallPeelThreads) entry(__ldg(I.b_nbr + off + e));
            }
            __syncthreads();
            head = tail;
            tail = s_tail;
            if (t == 0) s_longs = 0;
            __syncthreads();
        }
    }
    if (t == 0) {
        p.ctl->maxv[blockIdx.x] = level;
        p.ctl->removed[blockIdx.x] = head;
        p.ctl->members[blockIdx.x] = V;
    }
}

// ---------------------------------------------------------------------------
// incremental rows with exact support counters
// ---------------------------------------------------------------------------
// State of a group of blocks that works on a run of rows: the vertices of the
// run's first core (the ids below |C_a| of the relabeled graph), or all.
struct RowGroup {
    int32_t* cur;
    int32_t* cnt_out;  // #{u in N_out(v) : cur[u] >= cur[v]}  (never above the truth)
    int32_t* cnt_in;   // #{w in N_in(v)  : cur[w] >= cur[v]}
    uint32_t* mark;
    int32_t* stamp;
    uint32_t* logidx;
    TicketQueue q;
    EngineCtl* ctl;
};

// What the groups share (device memory).
struct RowPlan {
    PadW span[kRowGroups];  // (last row << 32) | current row of each group's run; 0: none
    struct alignas(128) Own {
        unsigned long long t_row;  // start of the current row
        unsigned row_ns;           // what the last row took
        int lo;                    // first row of the run to start
        unsigned flush_n, flush_off;  // values of the finished run's last row to leave in the seam array
        unsigned spare_n, spare_off;  // place in the seam array that an attempt to take rows over did not use
        int from;                     // group whose values the run to start begins with (-1: row 0)
        unsigned ready;               // the group's values belong to its run
        unsigned readers;             // groups about to copy its values
        unsigned members;             // blocks of the group, those that joined included
        unsigned long long step_blocks;  // (step << 32) | blocks that seed it: members 0 .. blocks - 1
        int prev;                     // row before the current one (the current one if it is the run's first)
        int join;                     // group that this one's blocks go to
    } own[kRowGroups];
    alignas(128) unsigned seam_tail;
    alignas(128) unsigned log_count;
    unsigned long long voids;
};

struct Trans2Params {
    const uint32_t* out_off;
    int32_t* out_len;
    uint32_t* out_nbr;
    const uint32_t* in_off;
    int32_t* in_len;
    uint32_t* in_nbr;
    const int32_t* kmax;
    const int32_t* row0;
    int32_t K;
    int32_t K0;     // first row to compute; group 0's cur holds row 0 inside C_K0, -1 outside
    int32_t Kstop;  // last row to compute (rows above stay untouched)
    uint32_t n;     // vertices group 0 has state for
    int sorted;     // lists ordered by neighbour kmax, descending
    const uint32_t* order;  // C_k = order[0 .. ck[k]); nullptr: the graph is relabeled, C_k = ids 0 .. ck[k]-1
    const uint32_t* ck;
    uint32_t* log_v;
    int32_t* log_k;
    int32_t* log_l;
    unsigned long long log_cap;
    // groups (1: no plan, one run)
    int n_groups;
    unsigned first_block[kRowGroups + 1];
    RowGroup g[kRowGroups];
    RowPlan* plan;
    int32_t run_min;    // least first row a run may have (its core fits the groups' state)
    uint32_t* seam_of;  // [K + 2] 1 + place in `seam` of the values of row k - 1, where a run starts at row k
    int32_t* seam;
    unsigned seam_cap;
};

// Levels of the row kernel's steps other than rows.
constexpr int kRowsEnd = 0x7FFFFFFF;  // the group leaves
constexpr int kRowsInit = -1;         // start values of the group's next run
constexpr int kRowsCount = -2;        // its counters
constexpr int kRowsWait = -3;         // nothing to take over yet
constexpr int kRowsJoin = -4;         // the group is over, its blocks go on in another one

// Next step of a group (run by the warp that finished the step).  After a row
// that needed no work the run jumps to the first row whose leaving set or
// seed set can be non-empty (the step's bound).  A group whose run is over
// takes over the upper half of what another group has left: the costs of rows
// differ by orders of magnitude and cluster just below the values of k where
// the core collapses, so no fixed cut balances them (eight equal runs of
// R-MAT 22 took 0.006 to 17.8 ms each, 71 ms together).  It begins with the
// other group's values as they are: values only fall, within a row and from
// row to row, so any of them bounds the later row's from above (from row 0
// the first row of such a run took up to 8 ms).
// When no group has rows worth taking over, the group's blocks join the one
// with the most left for good: they take items of its current row at once and
// seed with its own blocks from the next step on.  The last rows below a cliff
// of |C_k| are the heaviest and cannot be cut any more: one group's blocks
// alone took the last 30 % of the rows of R-MAT 20 and 22 for them (joining,
// with counts in shared memory instead of spilled registers, saves a tenth of
// the rows).  A group that others join has a run at
// that time, a finished group's run is cleared before it looks for one to
// join, and it never gets another: no two groups join each other.
struct RowsNext {
    const Trans2Params& p;
    int gid;
    unsigned blocks;  // of a launch without groups

    __device__ unsigned begin(unsigned step) const {
        if (p.n_groups == 1) return blocks;
        RowPlan::Own& own = p.plan->own[gid];
        const unsigned b = ld_vol(&own.members);
        *(volatile unsigned long long*)&own.step_blocks = ((unsigned long long)step << 32) | b;
        return b;
    }

    __device__ int operator()(EngineCtl*, int level, bool worked, int bound) const {
        const int r = worked ? level + 1 : max(level + 1, bound);
        if (p.n_groups == 1) return r > p.Kstop ? kRowsEnd : r;
        RowPlan* pl = p.plan;
        RowPlan::Own& own = pl->own[gid];
        const unsigned long long now = gtimer();
        if (level == kRowsInit) {  // the values are copied
            own.flush_n = 0;
            if (own.from >= 0) {
                __threadfence();  // the copies are made before the other group may overwrite what they read
                atomicSub(&pl->own[own.from].readers, 1u);
            }
            return kRowsCount;
        }
        if (level == kRowsCount) {
            own.t_row = now;
            own.row_ns = 0;
            __threadfence();
            *(volatile unsigned*)&own.ready = 1u;
            const int lo = ld_vol(&own.lo);
            *(volatile int*)&own.prev = lo;
            return lo;
        }
        bool flush = false;
        if (level > 0) {
            unsigned long long s = ld_acquire(&pl->span[gid].v);
            for (;;) {  // ends: others only shorten the run
                const int stop = (int)(s >> 32);
                const unsigned long long to = r > stop ? 0ull : ((unsigned long long)stop << 32) | (unsigned)r;
                const unsigned long long o = atomicCAS(&pl->span[gid].v, s, to);
                if (o != s) {
                    s = o;
                    continue;
                }
                if (to) {
                    const unsigned long long t = *(volatile unsigned long long*)&own.t_row;
                    if (t) *(volatile unsigned*)&own.row_ns = (unsigned)min(now - t, 0xFFFFFFFFull);
                    *(volatile unsigned long long*)&own.t_row = now;
                    *(volatile int*)&own.prev = level;
                    return r;
                }
                // the run is over: the run that starts at stop + 1 needs its last row's values
                *(volatile unsigned*)&own.ready = 0u;
                __threadfence();
                if (stop < p.Kstop) {
                    own.flush_n = __ldg(p.ck + stop + 1);
                    own.flush_off = ld_vol(p.seam_of + stop + 1) - 1u;
                    flush = true;
                }
                break;
            }
        } else {
            own.flush_n = 0;
        }
        bool any = false, wanted = false;
        // (a group that others still copy from keeps its values)
        const bool busy = ld_acquire(&own.readers) != 0u;
        for (int attempt = 0; attempt < 4; ++attempt) {
            int best = -1, best_start = 0;
            unsigned long long best_s = 0, best_score = 0;
            any = false;
            for (int h = 0; h < p.n_groups; ++h) {
                const unsigned long long s = h == gid ? 0ull : ld_acquire(&pl->span[h].v);
                if (!s) continue;
                any = true;
                const int row = (int)(uint32_t)s, stop = (int)(s >> 32), left = stop - row;
                const int start = max(row + 1 + left / 2, p.run_min);
                if (left < 2 || start > stop || ld_vol(p.seam_of + start)) continue;
                // worth it when what is left there takes longer than the start
                // of a run (a pass over its core's lists, about 10 ns per
                // vertex); a row takes as long as the last one or the current
                // one so far
                unsigned long long ns = 100000ull;
                if (ld_vol(&pl->own[h].ready)) {
                    const unsigned long long t = *(volatile unsigned long long*)&pl->own[h].t_row;
                    ns = max((unsigned long long)ld_vol(&pl->own[h].row_ns), t && now > t ? now - t : 0ull);
                }
                const unsigned long long score = (unsigned long long)left * ns;
                if (score > best_score && score > 40000ull + 10ull * __ldg(p.ck + start)) {
                    best = h;
                    best_start = start;
                    best_s = s;
                    best_score = score;
                }
            }
            wanted = best >= 0;
            if (best < 0 || busy) break;
            const unsigned n = __ldg(p.ck + best_start);
            if (own.spare_n < n) {
                if (ld_vol(&pl->seam_tail) + (unsigned long long)n > p.seam_cap) break;
                own.spare_off = atomicAdd(&pl->seam_tail, n);
                if (own.spare_off + (unsigned long long)n > p.seam_cap) {
                    own.spare_n = 0;
                    break;
                }
                own.spare_n = n;
            }
            // the seam is there, and the other group knows that its values
            // are wanted, before its run is shortened (its last step reads
            // both after the exchange on its span that ends the run, with a
            // fence between)
            if (atomicCAS(p.seam_of + best_start, 0u, own.spare_off + 1u) != 0u) continue;
            atomicAdd(&pl->own[best].readers, 1u);
            __threadfence();
            const unsigned long long stop = best_s >> 32;
            for (int again = 0; again < 8; ++again) {  // the other group may move on meanwhile
                const unsigned long long o = atomicCAS(
                    &pl->span[best].v, best_s, ((unsigned long long)(best_start - 1) << 32) | (best_s & 0xFFFFFFFFull));
                if (o == best_s) {
                    own.from = ld_acquire(&pl->own[best].ready) ? best : -1;
                    if (own.from < 0) atomicSub(&pl->own[best].readers, 1u);
                    own.spare_n = 0;
                    own.lo = best_start;
                    *(volatile unsigned long long*)&pl->span[gid].v = (stop << 32) | (unsigned)best_start;
                    return kRowsInit;
                }
                if ((o >> 32) != stop || (int)(uint32_t)o >= best_start) break;
                best_s = o;
            }
            atomicExch(p.seam_of + best_start, 0u);
            atomicSub(&pl->own[best].readers, 1u);
        }
        if (flush) return kRowsWait;  // leaves the values first
        // nothing to wait for, or a group that stopped on an error
        for (int h = 0; h < p.n_groups; ++h)
            if (ld_vol(&p.g[h].ctl->error)) any = false;
        if (!any) return kRowsEnd;
        if (!wanted) {
            int to = -1;
            unsigned long long most = 0;
            for (int h = 0; h < p.n_groups; ++h) {
                const unsigned long long s = h == gid ? 0ull : ld_acquire(&pl->span[h].v);
                if (!s) continue;
                const unsigned long long t = *(volatile unsigned long long*)&pl->own[h].t_row;
                const unsigned long long ns = max((unsigned long long)ld_vol(&pl->own[h].row_ns), t && now > t ? now - t : 0ull);
                const unsigned long long left = (s >> 32) - (uint32_t)s + 1ull, score = left * (ns + 1ull);
                if (score > most) {
                    most = score;
                    to = h;
                }
            }
            if (to < 0) return kRowsWait;  // the last run ended meanwhile
            *(volatile int*)&own.join = to;
            return kRowsJoin;
        }
        __nanosleep(10000);
        return kRowsWait;
    }
};

// Starting values of a run of rows that starts at row a on the handle's own
// graph: row 0 inside C_a, -1 (left) outside.
__global__ void k_preleft_cur(uint32_t V, const int32_t* kmax, const int32_t* row0, int32_t a, int32_t* cur) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V; v += (uint64_t)gridDim.x * blockDim.x)
        cur[v] = kmax[v] >= a ? row0[v] : -1;
}

// Converged warp: when the warp holds no item of its own yet (*keep ==
// kNoKeep), it keeps the first request of the lowest requesting lane to
// evaluate next itself instead of queueing it: the link from a drop to the
// neighbour's evaluation skips the queue's publish and take.
constexpr uint32_t kNoKeep = 0xFFFFFFFFu;
// Requests of a lane: bit r of *req set = u[r] is requested (r < 4); the
// items stay in registers (no dynamically indexed array).
__device__ __forceinline__ uint32_t first_requested(unsigned req, const uint32_t u[4]) {
    return (req & 1u) ? u[0] : (req & 2u) ? u[1] : (req & 4u) ? u[2] : u[3];
}
// Returns true (on every lane) when an item was kept.
__device__ __forceinline__ bool keep_one(uint32_t* keep, unsigned* req, const uint32_t u[4]) {
    if (*keep != kNoKeep) return false;
    const unsigned m = __ballot_sync(0xFFFFFFFFu, *req != 0u);
    if (!m) return false;
    const unsigned src = __ffs(m) - 1;
    const uint32_t item = __shfl_sync(0xFFFFFFFFu, first_requested(*req, u), src);
    if ((threadIdx.x & 31u) == src) *req &= *req - 1u;  // drop the kept request
    *keep = item;
    return true;
}

// ---- list passes of the row kernel ----------------------------------------
// Lists are read in windows of 128 entries, four per lane (entries b + lane,
// b + 32 + lane, ..): neighbouring lanes hold neighbouring entries, and with
// lists in id order their values share cache lines -- in the dense cores,
// where the work is, 32 consecutive neighbours lie in a few lines, so a
// window's gathers and decrements take a fraction of the transactions that
// 32 scattered ones would.  Ids past the list's end read as 0xFFFFFFFF, which
// is outside every id range.
__device__ __forceinline__ void load_ids4(const uint32_t* nbr, uint32_t o, int n, int b, bool active, uint32_t u[4]) {
    const int e = b + (int)(threadIdx.x & 31u);
#pragma unroll
    for (int q = 0; q < 4; ++q) u[q] = (active && e + 32 * q < n) ? __ldg(nbr + o + (uint32_t)(e + 32 * q)) : 0xFFFFFFFFu;
}
// Values of a window's four entries of this lane (-1 for ids from `ids` on).
__device__ __forceinline__ void gather4(const int32_t* cur, uint32_t ids, const uint32_t u[4], int v[4]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = u[q] < ids ? ld_vol(&cur[u[q]]) : -1;
}

// Counts the neighbours at each value of [lo, hi] (both lists) into the bins
// bo / bi; values above hi are not counted (the caller carries them).  On
// kmax-sorted lists a list ends at its first neighbour outside C_j.  Returns
// the entries read.
__device__ __forceinline__ int hist_pass2v(const int32_t* cur, uint32_t ids, const uint32_t* onbr, uint32_t oo, int no,
                                           const uint32_t* inbr, uint32_t io, int ni, int lo, int hi, bool sorted,
                                           int* bo, int* bi) {
    const unsigned lane = threadIdx.x & 31u;
    int to = 0, ti = 0, entries = 0;
    bool ao = no > 0, ai = ni > 0;
    for (int b = 0; ao || ai; b += 128) {
        uint32_t uo[4], ui[4];
        int vo[4], vi[4];
        load_ids4(onbr, oo, no, b, ao, uo);
        load_ids4(inbr, io, ni, b, ai, ui);
        gather4(cur, ao ? ids : 0u, uo, vo);
        gather4(cur, ai ? ids : 0u, ui, vi);
        entries += (ao ? min(128, no - b) : 0) + (ai ? min(128, ni - b) : 0);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            to += vo[q] == hi;
            ti += vi[q] == hi;
            if (vo[q] >= lo && vo[q] < hi) atomicAdd(&bo[vo[q] - lo], 1);
            if (vi[q] >= lo && vi[q] < hi) atomicAdd(&bi[vi[q] - lo], 1);
        }
        ao = ao && b + 128 < no;
        ai = ai && b + 128 < ni;
        if (sorted && ao && __shfl_sync(0xFFFFFFFFu, vo[3], 31) == -1) ao = false;
        if (sorted && ai && __shfl_sync(0xFFFFFFFFu, vi[3], 31) == -1) ai = false;
    }
    to = __reduce_add_sync(0xFFFFFFFFu, to);
    ti = __reduce_add_sync(0xFFFFFFFFu, ti);
    if (lane == 0) {
        if (to) atomicAdd(&bo[hi - lo], to);
        if (ti) atomicAdd(&bi[hi - lo], ti);
    }
    return entries;
}

// Converged warp: each lane pushes items_a[r] for bits r of ma and items_b[r]
// for bits r of mb (r < 4) with the step's tag, one reservation for the warp.
__device__ __forceinline__ void step_push_mask8(EngineCtl* c, TicketQueue q, unsigned ma, const uint32_t items_a[4],
                                                   unsigned mb, const uint32_t items_b[4], unsigned long long tag) {
    const unsigned lane = threadIdx.x & 31u;
    const unsigned cnt = __popc(ma) + __popc(mb);
    if (!__any_sync(0xFFFFFFFFu, cnt != 0u)) return;
    unsigned x = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= (unsigned)o) x += y;
    }
    const unsigned total = __shfl_sync(0xFFFFFFFFu, x, 31);
    unsigned base = step_reserve(c, total) + (x - cnt);
#pragma unroll
    for (unsigned r = 0; r < 4; ++r)
        if (ma & (1u << r)) step_put(q, base + __popc(ma & ((1u << r) - 1u)), (unsigned long long)items_a[r] | tag);
    base += __popc(ma);
#pragma unroll
    for (unsigned r = 0; r < 4; ++r)
        if (mb & (1u << r)) step_put(q, base + __popc(mb & ((1u << r) - 1u)), (unsigned long long)items_b[r] | tag);
}

// Both lists of a vertex and the ids of their first window.
struct RowLists {
    uint32_t oo, io;  // list starts
    int no, ni;       // lengths
    uint32_t uo[4], ui[4];
};

// The lists never change while the kernel runs: read through the read-only
// path, so that the loads may be issued ahead of fences.
__device__ __forceinline__ RowLists row_lists(const Trans2Params& p, uint32_t x) {
    RowLists L;
    L.oo = __ldg(p.out_off + x);
    L.io = __ldg(p.in_off + x);
    L.no = __ldg(p.out_len + x);
    L.ni = __ldg(p.in_len + x);
    load_ids4(p.out_nbr, L.oo, L.no, 0, true, L.uo);
    load_ids4(p.in_nbr, L.io, L.ni, 0, true, L.ui);
    return L;
}

// Counts, over both lists, the neighbours at each of the T values cap,
// cap - 1, .. (a drop is rarely larger), this lane's share in go / gi.  The
// next window's ids are in flight while a window's values are gathered, so a
// step of 128 entries per list costs one memory latency.  Returns the entries
// read.
constexpr int kThr = 4;
template <int T>
__device__ __forceinline__ int count_pass(const Trans2Params& p, const int32_t* cur, uint32_t ids, const RowLists& L,
                                          int cap, int go[T], int gi[T]) {
    uint32_t uo[4], ui[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        uo[q] = L.uo[q];
        ui[q] = L.ui[q];
    }
#pragma unroll
    for (int r = 0; r < T; ++r) go[r] = gi[r] = 0;
    bool ao = L.no > 0, ai = L.ni > 0;
    int entries = 0;
    for (int b = 0; ao || ai; b += 128) {
        int vo[4], vi[4];
        gather4(cur, ao ? ids : 0u, uo, vo);
        gather4(cur, ai ? ids : 0u, ui, vi);
        entries += (ao ? min(128, L.no - b) : 0) + (ai ? min(128, L.ni - b) : 0);
        ao = ao && b + 128 < L.no;
        ai = ai && b + 128 < L.ni;
        load_ids4(p.out_nbr, L.oo, L.no, b + 128, ao, uo);
        load_ids4(p.in_nbr, L.io, L.ni, b + 128, ai, ui);
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int r = 0; r < T; ++r) {
                go[r] += vo[q] >= cap - r;
                gi[r] += vi[q] >= cap - r;
            }
        // kmax-sorted lists end at the first neighbour outside C_j
        if (p.sorted && ao && __shfl_sync(0xFFFFFFFFu, vo[3], 31) == -1) ao = false;
        if (p.sorted && ai && __shfl_sync(0xFFFFFFFFu, vi[3], 31) == -1) ai = false;
    }
    return entries;
}

// Counters of the first run's vertices on the handle's own graph (the sorts
// count those of the relabeled one) against every neighbour, at the
// vertex's starting value in group 0's cur (vertices with a value below 1 get
// zero counts: they are never evaluated and no counter includes them).
__global__ void k_counters_init(Trans2Params p) {
    const unsigned lane = threadIdx.x & 31u;
    const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const RowGroup& G = p.g[0];
    for (uint64_t v = gw; v < p.n; v += nw) {
        int go[1] = {0}, gi[1] = {0};
        const int cv = ld_vol(&G.cur[v]);
        if (cv >= 1) {
            count_pass<1>(p, G.cur, p.n, row_lists(p, (uint32_t)v), cv, go, gi);
            go[0] = __reduce_add_sync(0xFFFFFFFFu, go[0]);
            gi[0] = __reduce_add_sync(0xFFFFFFFFu, gi[0]);
        }
        if (lane == 0) {
            G.cnt_out[v] = go[0];
            G.cnt_in[v] = gi[0];
        }
    }
}

// One pass over both lists of x after its value fell from cap to nv: counts
// the neighbours with value >= nv into *cnt_o / *cnt_i (this lane's share)
// and takes x's support away from the neighbours whose level lies in
// (nv, cap] (out-neighbours lose a unit of cnt_in, in-neighbours one of
// cnt_out), requesting those that fall below what they need.  The next
// window's values and the ids after it are in flight while a window's
// decrements return.  kLeave: x leaves C_j (nv = 0, cap = its old value); the
// requests kept are counted as outstanding, and *lmin bounds the next row
// that can need work.  Returns the entries read.
template <bool kLeave>
__device__ __forceinline__ int drop_pass(const Trans2Params& p, const RowGroup& G, uint32_t ids, const RowLists& L, int nv, int cap,
                                         int j, unsigned long long word, int* cnt_o, int* cnt_i, uint32_t* keep,
                                         int* pending, int* lmin) {
    bool ao = L.no > 0, ai = L.ni > 0;
    if (!ao && !ai) return 0;
    int entries = 0;
    uint32_t uo[4], ui[4], no[4], ni[4];
    int vo[4], vi[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        uo[q] = L.uo[q];
        ui[q] = L.ui[q];
    }
    gather4(G.cur, ids, uo, vo);
    gather4(G.cur, ids, ui, vi);
    load_ids4(p.out_nbr, L.oo, L.no, 128, ao, no);
    load_ids4(p.in_nbr, L.io, L.ni, 128, ai, ni);
    for (int b = 0;; b += 128) {
        entries += (ao ? min(128, L.no - b) : 0) + (ai ? min(128, L.ni - b) : 0);
        bool mo = ao && b + 128 < L.no, mi = ai && b + 128 < L.ni;
        if (p.sorted && mo && __shfl_sync(0xFFFFFFFFu, vo[3], 31) == -1) mo = false;
        if (p.sorted && mi && __shfl_sync(0xFFFFFFFFu, vi[3], 31) == -1) mi = false;
        int oldo[4], oldi[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (!kLeave) {
                *cnt_o += vo[q] >= nv;
                *cnt_i += vi[q] >= nv;
            }
            oldo[q] = (vo[q] > nv && vo[q] <= cap) ? atomicSub(&G.cnt_in[uo[q]], 1) : 0x7FFFFFFF;
            oldi[q] = (vi[q] > nv && vi[q] <= cap) ? atomicSub(&G.cnt_out[ui[q]], 1) : 0x7FFFFFFF;
        }
        int wo[4], wi[4];
        gather4(G.cur, mo ? ids : 0u, no, wo);
        gather4(G.cur, mi ? ids : 0u, ni, wi);
        unsigned ro = 0, ri = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (oldo[q] - 1 < j) ro |= 1u << q;
            else if (kLeave) *lmin = min(*lmin, oldo[q]);
            if (oldi[q] != 0x7FFFFFFF && oldi[q] - 1 < vi[q]) ri |= 1u << q;
        }
        if (__any_sync(0xFFFFFFFFu, (ro | ri) != 0u)) {
            unsigned so_[4], si_[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                so_[q] = (ro >> q) & 1u ? atomicOr(&G.mark[uo[q]], 1u) : 1u;
                si_[q] = (ri >> q) & 1u ? atomicOr(&G.mark[ui[q]], 1u) : 1u;
            }
            ro = ri = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (so_[q] == 0u) ro |= 1u << q;
                if (si_[q] == 0u) ri |= 1u << q;
            }
            if (keep_one(keep, &ro, uo) || keep_one(keep, &ri, ui)) {
                if (kLeave) step_count_kept(G.ctl);
                else --*pending;  // the item being finished pays for the kept one
            }
            step_push_mask8(G.ctl, G.q, ro, uo, ri, ui, step_tag(word));
        }
        if (!mo && !mi) break;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            uo[q] = no[q];
            ui[q] = ni[q];
            vo[q] = wo[q];
            vi[q] = wi[q];
        }
        load_ids4(p.out_nbr, L.oo, L.no, b + 256, mo, no);
        load_ids4(p.in_nbr, L.io, L.ni, b + 256, mi, ni);
        ao = mo;
        ai = mi;
    }
    return entries;
}

// The value of x when it fell more than kThr - 1 below cap: windows of kWin
// values below hi, histograms in shared memory; carry_o / carry_i = counts
// above hi.  Counts at the value found go to *c_o / *c_i.
__device__ __forceinline__ int window_value(const Trans2Params& p, const RowGroup& G, uint32_t ids, const RowLists& L, int j, int hi, int carry_o,
                                            int carry_i, int* ho, int* hi_, int* c_o, int* c_i, int* entries) {
    const unsigned lane = threadIdx.x & 31u;
    for (;;) {
        int lo = max(0, hi - (kWin - 1));
        ho[lane] = 0;
        ho[lane + 32] = 0;
        hi_[lane] = 0;
        hi_[lane + 32] = 0;
        __syncwarp();
        *entries += hist_pass2v(G.cur, ids, p.out_nbr, L.oo, L.no, p.in_nbr, L.io, L.ni, lo, hi, p.sorted != 0, ho, hi_);
        __syncwarp();
        int b0 = 2 * lane, b1 = 2 * lane + 1;
        int o0 = ho[b0], o1 = ho[b1], i0 = hi_[b0], i1 = hi_[b1];
        int po = o0 + o1, pi = i0 + i1;
        int so = po, si = pi;
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) {
            int yo = __shfl_down_sync(0xFFFFFFFFu, so, s);
            int yi = __shfl_down_sync(0xFFFFFFFFu, si, s);
            if (lane + s < 32) {
                so += yo;
                si += yi;
            }
        }
        int cum_o1 = carry_o + (so - po) + o1, cum_i1 = carry_i + (si - pi) + i1;
        int cum_o0 = cum_o1 + o0, cum_i0 = cum_i1 + i0;
        int L0 = lo + b0, L1 = lo + b1;
        bool ok1 = (L1 <= hi) && cum_o1 >= L1 && cum_i1 >= j;
        bool ok0 = (L0 <= hi) && cum_o0 >= L0 && cum_i0 >= j;
        unsigned m1 = __ballot_sync(0xFFFFFFFFu, ok1), m0 = __ballot_sync(0xFFFFFFFFu, ok0);
        int t1 = m1 ? 31 - __clz(m1) : -1, t0 = m0 ? 31 - __clz(m0) : -1;
        int best = -1, bt = 0, bodd = 0;
        if (t1 >= 0) {
            best = lo + 2 * t1 + 1;
            bt = t1;
            bodd = 1;
        }
        if (t0 >= 0 && lo + 2 * t0 > best) {
            best = lo + 2 * t0;
            bt = t0;
            bodd = 0;
        }
        if (best >= 0) {
            int xo = bodd ? cum_o1 : cum_o0, xi = bodd ? cum_i1 : cum_i0;
            *c_o = __shfl_sync(0xFFFFFFFFu, xo, bt);
            *c_i = __shfl_sync(0xFFFFFFFFu, xi, bt);
            return best;
        }
        carry_o += __shfl_sync(0xFFFFFFFFu, so, 0);
        carry_i += __shfl_sync(0xFFFFFFFFu, si, 0);
        if (lo == 0) {  // unreachable for members of C_j
            *c_o = carry_o;
            *c_i = carry_i;
            return 0;
        }
        hi = lo - 1;
        __syncwarp();
    }
}

// Corner records a warp takes from the log at a time.
static constexpr unsigned kLogChunk = 8;

// Latency-bound: a row's changes run through dependent evaluations (a chain of
// 20,000 takes 4.9 us per link, 7.8 with two more fences and a queue item per
// link), so what counts is the number of memory round trips and fences from
// one vertex's drop to the next one's evaluation.  Hence: the static data of a
// vertex is loaded while its mark is set, its value and counters come with it,
// the new value is found with register counters at the four highest candidates
// (the shared-memory histogram only for larger drops), a corner record's place
// is in hand before the drop, one fence stands between the new value (with its
// record) and the neighbours' values and one before the vertex is released, a
// request is one atomicOr, a warp keeps one of the items it requests, and rows
// advance without a grid barrier.  Rows 1..kmax as one run, R-MAT 18 / 20 / 22
// and ER of 10,000: 9.7 / 14.4 / 35.4 / 0.47 ms; in groups (RowsNext) 2.3 / 5.2 /
// 19.0 ms.  80 registers for three blocks per SM (64 spill).
#ifndef DC_TRANS2_MIN_BLOCKS
#define DC_TRANS2_MIN_BLOCKS 3
#endif
struct RowWarp {
    unsigned long long entries, log_at;
    unsigned evals, drops, log, log_left;
};
// kGroups: several groups of blocks (RowPlan); else one run, no plan.
template <bool kGroups>
__global__ void __launch_bounds__(kThreads, DC_TRANS2_MIN_BLOCKS) k_trans2(Trans2Params p) {
    const unsigned lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
    int gid = 0;
    while (kGroups && gid + 1 < p.n_groups && blockIdx.x >= p.first_block[gid + 1]) ++gid;
    unsigned block = blockIdx.x - p.first_block[gid];  // number within the group
    EngineCtl* c = p.g[gid].ctl;
    __shared__ int s_ho[kWarpsPerBlock][kWin];
    __shared__ int s_hi[kWarpsPerBlock][kWin];
    __shared__ StepBlock s_step;
    __shared__ unsigned s_member;
    bool tracing = c->trace != nullptr;
    // failure-detection tests: this block never reports, the others' waits run out
    if (c->test_skip_block && (int)blockIdx.x == c->test_skip_block - 1) return;
    // lane 0's counts of its warp and the records left in its log chunk: in
    // shared memory, the loop has no registers to spare
    __shared__ RowWarp s_warp[kWarpsPerBlock];
    RowWarp& my = s_warp[wib];
    if (lane == 0) my = RowWarp{0ull, 0ull, 0u, 0u, 0u, 0u};
    unsigned ticket = kNoTicket;
    unsigned* const log_count = kGroups ? &p.plan->log_count : &c->log_count;
    step_block_init(&s_step, c);
    unsigned long long word = step_block_word(&s_step);
    int jprev = p.K0;    // row before this step's (the row itself: the first of its run)
    uint32_t ids = p.n;  // vertices with state
    for (;;) {
        const int j = step_level(word);
        if (word == kStopWord || j == kRowsEnd) break;
        if (kGroups && j == kRowsJoin) {
            // the whole block goes over: a new number, the other group's word
            // (which every warp reads before one of them can replace it)
            gid = ld_vol(&p.plan->own[gid].join);
            c = p.g[gid].ctl;
            tracing = c->trace != nullptr;
            __syncthreads();
            if (threadIdx.x == 0) s_member = atomicAdd(&p.plan->own[gid].members, 1u);
            step_block_init(&s_step, c);
            word = step_block_word(&s_step);
            block = s_member;
            __syncthreads();
            ticket = kNoTicket;
            continue;
        }
        const RowGroup& G = p.g[gid];
        const RowPlan::Own* own = kGroups ? &p.plan->own[gid] : nullptr;
        unsigned blocks = gridDim.x;
        bool seeds = true;  // the block has a share of this step's seeding
        if (kGroups) {
            const unsigned long long sb = *(const volatile unsigned long long*)&own->step_blocks;
            blocks = (unsigned)sb;
            // (another step's number: this one is over)
            seeds = (unsigned)(sb >> 32) == step_number(word) && block < blocks;
            ids = __ldg(p.ck + ld_vol(&own->lo));
            jprev = ld_vol(&own->prev);
        }
        const bool seed_out = jprev == j;  // first row of a run: members are seeded by their out-counts too
        const RowsNext next{p, gid, blocks};
        const unsigned gwarp = block * kWarpsPerBlock + wib;
        const unsigned nwarps = blocks * kWarpsPerBlock;
        const unsigned long long tag = step_tag(word);
        if (tracing && threadIdx.x == 0) trace_wake(c, word);
        uint32_t keep = kNoKeep;
        int pending = 0;
        if (kGroups && j < 0) {
            // between runs: the finished run's last row to the seam, then the
            // next run's start values and counters (every value is read from
            // row 0, a thread clears what it has copied itself)
            const unsigned fn = seeds ? ld_vol(&own->flush_n) : 0u, fo = ld_vol(&own->flush_off);
            for (uint32_t i = block * kThreads + threadIdx.x; i < fn; i += blocks * kThreads)
                p.seam[fo + i] = ld_vol(&G.cur[i]);
            if (j == kRowsInit && seeds) {
                const int from = ld_vol(&own->from);
                const int32_t* src = from < 0 ? p.row0 : p.g[from].cur;
                for (uint32_t i = block * kThreads + threadIdx.x; i < ids; i += blocks * kThreads) {
                    G.cur[i] = ld_vol(&src[i]);
                    G.mark[i] = 0;
                    G.stamp[i] = -1;
                }
            } else if (j == kRowsCount && seeds) {
                for (uint32_t v = gwarp; v < ids; v += nwarps) {
                    int go[1] = {0}, gi[1] = {0};
                    const int cv = ld_vol(&G.cur[v]);
                    if (cv >= 1) {
                        count_pass<1>(p, G.cur, ids, row_lists(p, v), cv, go, gi);
                        go[0] = __reduce_add_sync(0xFFFFFFFFu, go[0]);
                        gi[0] = __reduce_add_sync(0xFFFFFFFFu, gi[0]);
                    }
                    if (lane == 0) {
                        G.cnt_out[v] = go[0];
                        G.cnt_in[v] = gi[0];
                    }
                }
            }
            __threadfence();
            if (seeds) step_seeded(c, &s_step, kNoBound, false, word, tracing, next);
            unsigned long long none;
            if (step_take(c, G.q, &s_step, &ticket, &none, &pending, &word, next) == kTakeStop) break;
            continue;
        }
        // rows jprev+1 .. j-1 equal row jprev; vertices with kmax in
        // [jprev, j-1] leave now (all but those with kmax == j-1 have value 0)
        const uint32_t vj = seeds ? __ldg(p.ck + j) : 0u, vprev = seeds ? __ldg(p.ck + jprev) : 0u;
        // ---- vertices leaving C_j: value -1; neighbours they supported lose one count
        int bound = kNoBound;  // on the next row that can need work
        // spread over all warps; a warp's share (up to 32 at a time) is cleared
        // with one fence, and the next one's lists are loaded while one's are read
        const uint32_t share = vprev > vj ? min(32u, (vprev - vj + nwarps - 1) / nwarps) : 1u;
        for (uint32_t base = vj + gwarp * share; base < vprev; base += nwarps * share) {
            const uint32_t i = base + lane;
            uint32_t xl = 0;
            int al = 0;
            if (lane < share && i < vprev) {
                xl = p.order ? __ldg(p.order + i) : i;
                al = ld_vol(&G.cur[xl]);
                *(volatile int32_t*)&G.cur[xl] = -1;
            }
            unsigned m = __ballot_sync(0xFFFFFFFFu, al >= 1);
            if (!m) continue;
            RowLists L = row_lists(p, __shfl_sync(0xFFFFFFFFu, xl, __ffs(m) - 1));
            __threadfence();
            while (m) {
                const int a = __shfl_sync(0xFFFFFFFFu, al, __ffs(m) - 1);
                const RowLists cur_l = L;
                m &= m - 1u;
                if (m) L = row_lists(p, __shfl_sync(0xFFFFFFFFu, xl, __ffs(m) - 1));
                drop_pass<true>(p, G, ids, cur_l, 0, a, j, word, nullptr, nullptr, &keep, &pending, &bound);
            }
        }
        // ---- seeds: members whose in-count at their own level is below j;
        // the least min(cnt_in, kmax) + 1 of the others bounds the next row
        // that can need work
        for (uint32_t base = gwarp * 32; base < vj; base += nwarps * 32) {
            const uint32_t i = base + lane;
            unsigned req = 0;
            uint32_t v = 0;
            if (i < vj) {
                v = p.order ? __ldg(p.order + i) : i;
                const int cv = ld_vol(&G.cur[v]), ci = ld_vol(&G.cnt_in[v]);
                const int co = seed_out ? ld_vol(&G.cnt_out[v]) : 0x7FFFFFFF;
                const int km = __ldg(p.kmax + v);
                if (cv >= 1) {
                    if (ci < j || co < cv) req = mark_request(&G.mark[v]) ? 1u : 0u;
                    else bound = min(bound, min(ci, km) + 1);
                }
            }
            if (__any_sync(0xFFFFFFFFu, req != 0u)) {
                const uint32_t u[4] = {v, 0u, 0u, 0u};
                if (keep_one(&keep, &req, u)) step_count_kept(c);
                step_push(c, G.q, req != 0u, (unsigned long long)v | tag);
            }
        }
        if (seeds) step_seeded(c, &s_step, bound, keep != kNoKeep, word, tracing, next);

        // ---- drain: the warp's kept item first, else the queue; finished
        // items are counted off in batches (before the warp waits)
        unsigned long long item = 0;
        int state = kTakeItem;
        for (;;) {
            uint32_t x;
            if (keep != kNoKeep) {
                x = keep;
                keep = kNoKeep;
            } else {
                state = step_take(c, G.q, &s_step, &ticket, &item, &pending, &word, next);
                if (state != kTakeItem) break;
                x = (uint32_t)item;
            }
            // The mark says "being evaluated" before any neighbour is read (a
            // request made before it belongs to a drop that is seen below, one
            // made after it has x evaluated again), and so is the snapshot of
            // the counters: one read after a neighbour's decrement, beside that
            // neighbour's value from before it, would leave the counter too
            // high for good, and a later drop unseen.  (A decrement that lands
            // after the snapshot, beside the neighbour's new value, only makes
            // the counter too low, which costs an evaluation.)  So all of x's
            // state is read by acquire loads, a word per lane, in one latency;
            // lane 0's load of the mark returns after its exchange.
            if (lane == 0) atomicExch(&G.mark[x], 2u);
            const int km = __ldg(p.kmax + x);
            const RowLists L = row_lists(p, x);
            const void* at = lane == 0   ? (const void*)G.mark
                             : lane == 1 ? (const void*)G.cnt_out
                             : lane == 2 ? (const void*)G.cnt_in
                             : lane == 3 ? (const void*)G.cur
                             : lane == 4 ? (const void*)G.stamp
                                         : (const void*)G.logidx;
            const unsigned state_word = ld_acquire((const unsigned*)at + x);
            __syncwarp();
            const int s0o = (int)__shfl_sync(0xFFFFFFFFu, state_word, 1), s0i = (int)__shfl_sync(0xFFFFFFFFu, state_word, 2);
            const int cap = (int)__shfl_sync(0xFFFFFFFFu, state_word, 3);
            const int stamp = (int)__shfl_sync(0xFFFFFFFFu, state_word, 4);
            const uint32_t logidx = __shfl_sync(0xFFFFFFFFu, state_word, 5);
            if (km < j || cap < 1) {
                if (lane == 0) atomicExch(&G.mark[x], 0u);
                ++pending;
                continue;
            }
            // ---- new value
            int c_o = 0, c_i = 0, nv = -1, entries;
            {
                int go[kThr], gi[kThr];
                entries = count_pass<kThr>(p, G.cur, ids, L, cap, go, gi);
#pragma unroll
                for (int r = 0; r < kThr; ++r) {
                    go[r] = __reduce_add_sync(0xFFFFFFFFu, go[r]);
                    gi[r] = __reduce_add_sync(0xFFFFFFFFu, gi[r]);
                }
#pragma unroll
                for (int r = kThr - 1; r >= 0; --r)
                    if (cap - r >= 0 && go[r] >= cap - r && gi[r] >= j) {
                        nv = cap - r;
                        c_o = go[r];
                        c_i = gi[r];
                    }
                if (nv < 0) {
                    if (cap >= kThr) {
                        nv = window_value(p, G, ids, L, j, cap - kThr, go[kThr - 1], gi[kThr - 1], s_ho[wib], s_hi[wib], &c_o,
                                          &c_i, &entries);
                    } else {  // unreachable for members of C_j
                        nv = 0;
                    }
                }
            }
            if (nv < cap) {
                if (lane == 0) {
                    ++my.drops;
                    // the value and its corner record
                    unsigned long long li = logidx;
                    const bool fresh = stamp != j;
                    if (fresh) {
                        if (!my.log_left) {
                            my.log_at = atomicAdd(log_count, kLogChunk);
                            my.log_left = kLogChunk;
                        }
                        li = my.log_at++;
                        --my.log_left;
                        ++my.log;
                    }
                    if (li < p.log_cap) {
                        if (fresh) {
                            G.stamp[x] = j;
                            G.logidx[x] = (uint32_t)li;
                            p.log_v[li] = x;
                            p.log_k[li] = j;
                        }
                        p.log_l[li] = nv;
                    } else {
                        set_dev_error(c, DC_DEV_ERR_CAPACITY, 20);
                    }
                    *(volatile int32_t*)&G.cur[x] = nv;
                }
                __syncwarp();
                __threadfence();
                // recount at nv after the write, and take x's support away
                // from neighbours whose level lies in (nv, cap]: out-neighbours
                // hold x in cnt_in, in-neighbours in cnt_out
                c_o = 0;
                c_i = 0;
                entries += drop_pass<false>(p, G, ids, L, nv, cap, j, word, &c_o, &c_i, &keep, &pending, nullptr);
                c_o = __reduce_add_sync(0xFFFFFFFFu, c_o);
                c_i = __reduce_add_sync(0xFFFFFFFFu, c_i);
            }
            if (lane == 0) {
                ++my.evals;
                my.entries += (unsigned)entries;
            }
            if (tracing && lane == 0 && step_number(word) - 1 < c->trace_cap)
                atomicMax(&c->trace[8 * (step_number(word) - 1) + 7], (unsigned long long)entries);
            unsigned again = 0;
            if (lane == 0) {
                const int no = atomicAdd(&G.cnt_out[x], c_o - s0o) + (c_o - s0o);
                const int ni = atomicAdd(&G.cnt_in[x], c_i - s0i) + (c_i - s0i);
                const bool stable = nv < 1 || (no >= nv && ni >= j);
                // released once the counters are performed everywhere;
                // requested meanwhile or unstable: evaluated again, and the
                // mark says so before another warp can take the item (an
                // exchange that came after the taker's would leave the mark
                // set with nobody queued, and drop every later request)
                fence_acq_rel();
                if (!stable || atomicCAS(&G.mark[x], 2u, 0u) == 3u) {
                    atomicExch(&G.mark[x], 1u);
                    fence_acq_rel();
                    again = 1u;
                }
            }
            if (__shfl_sync(0xFFFFFFFFu, again, 0)) {
                if (keep == kNoKeep) {
                    keep = x;  // at once: still the item being finished
                    continue;
                }
                step_push(c, G.q, lane == 0, (unsigned long long)x | tag);
            }
            ++pending;
        }
        if (state == kTakeStop) break;
        if (!kGroups) jprev = j;
    }
    if (lane == 0) {
        // unused records of the last chunk are void
        for (; my.log_left; --my.log_left, ++my.log_at)
            if (my.log_at < p.log_cap) p.log_k[my.log_at] = -1;
        atomicAdd(&c->log_used, my.log);
        atomicAdd(&c->evals, (unsigned long long)my.evals);
        atomicAdd(&c->drops, (unsigned long long)my.drops);
        atomicAdd(&c->edges_scanned, my.entries);
    }
}

// ---------------------------------------------------------------------------
// lists of the relabeled graph, in id order
// ---------------------------------------------------------------------------
// New ids are positions in kmax-descending order, so a list in id order has
// the neighbours inside C_j = {kmax >= j} as a prefix for every j (row
// evaluations read only that) and close neighbours side by side (their values
// share cache lines).  List i is copied from list order[i] of the handle's
// graph with every entry renamed by pos.
static constexpr int kSortShort = 32;
static constexpr int kSortWarp = 256;
static constexpr int kSortMid = 4096;
static constexpr int kSortThreads = 256;

// Both sides of the relabeled graph in one launch (blockIdx.y).  Along with its
// list every vertex gets its support count on that side at its row 0: the
// neighbours below n0 (|C_k0|) whose row 0 is no smaller.  The entries are in
// registers here; a pass of its own over both sides took 0.43 ms of R-MAT 20.
struct SortSide {
    const uint32_t* off;    // starts and lengths of the new lists
    const int32_t* len;
    uint32_t* nbr;
    const uint32_t* src;    // the handle's lists, and where each list starts there
    const uint32_t* start;
    uint32_t* list[3];      // longer lists: for the warp, the block and the counting sort
    int32_t* support;
};
struct SortArgs {
    SortSide side[2];
    unsigned* cnt;        // [6] longer lists by side and sort, zero before
    const uint2* pos;     // new id and row 0 by the handle's id: one gather per entry
    const int32_t* kmax;  // by new id
    const int32_t* row0;
    uint32_t n0;
    int K;
};
// Least value that supports v (0x7FFFFFFF: v is never evaluated, no counts).
__device__ __forceinline__ int support_level(const SortArgs& p, uint32_t v) {
    const int r = v < p.n0 ? p.row0[v] : 0;
    return r >= 1 ? r : 0x7FFFFFFF;
}
// Entry u renamed; *sup counts it if it supports.
__device__ __forceinline__ uint32_t rename(const SortArgs& p, uint32_t u, int level, int* sup) {
    const uint2 x = __ldg(p.pos + u);
    *sup += x.x < p.n0 && (int)x.y >= level;
    return x.x;
}

// Lists of at most kSortShort entries, eight lanes each with T entries per
// lane (entry 8 t + lane in k[t], bitonic as below): four lists per warp, their
// entries read and written side by side.  Bound by the latency of the two
// dependent loads (entry, new id).  One thread per list, an insertion
// sort in local memory and the list found through two more loads took 148 us
// of R-MAT 20 and 23 us of 10,000 vertices (both sides, no counts).
template <int T>
__device__ __forceinline__ void oct_sort(const SortArgs& p, const uint32_t* in, int n, int level, uint32_t* a, int* sup) {
    const int sl = (int)(threadIdx.x & 7u);
    uint32_t k[T];
    int c = 0;
#pragma unroll
    for (int t = 0; t < T; ++t) k[t] = 8 * t + sl < n ? in[8 * t + sl] : 0xFFFFFFFFu;
#pragma unroll
    for (int t = 0; t < T; ++t)
        if (8 * t + sl < n) k[t] = rename(p, k[t], level, &c);
#pragma unroll
    for (int size = 2; size <= 8 * T; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride; stride >>= 1) {
#pragma unroll
            for (int t = 0; t < T; ++t) {
                const bool up = ((8 * t + sl) & size) == 0;
                if (stride >= 8) {
                    const int o = t ^ (stride >> 3);
                    if (o > t) {
                        const uint32_t lo = min(k[t], k[o]), hi = max(k[t], k[o]);
                        k[t] = up ? lo : hi;
                        k[o] = up ? hi : lo;
                    }
                } else {
                    const uint32_t o = __shfl_xor_sync(0xFFFFFFFFu, k[t], stride);
                    k[t] = ((sl & stride) == 0) == up ? min(k[t], o) : max(k[t], o);
                }
            }
        }
    }
#pragma unroll
    for (int t = 0; t < T; ++t)
        if (8 * t + sl < n) a[8 * t + sl] = k[t];
    c += __shfl_xor_sync(0xFFFFFFFFu, c, 4);
    c += __shfl_xor_sync(0xFFFFFFFFu, c, 2);
    *sup = c + __shfl_xor_sync(0xFFFFFFFFu, c, 1);
}
__global__ void k_sort_short(uint32_t V, SortArgs p) {
    const SortSide& S = p.side[blockIdx.y];
    const unsigned lane = threadIdx.x & 31u;
    const uint64_t stride = (((uint64_t)gridDim.x * blockDim.x) >> 5) * 4;
    for (uint64_t b = ((blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5) * 4; b < V; b += stride) {
        const uint64_t i = b + (lane >> 3);
        const int len = i < V ? S.len[i] : 0, n = len <= kSortShort ? len : 0;
        const uint32_t v = i < V ? (uint32_t)i : 0u;
        const uint32_t* in = S.src + S.start[v];
        uint32_t* a = S.nbr + S.off[v];
        const int level = support_level(p, v), most = (int)__reduce_max_sync(0xFFFFFFFFu, (unsigned)n);
        int sup = 0;
        if (most > 16) oct_sort<4>(p, in, n, level, a, &sup);
        else if (most > 8) oct_sort<2>(p, in, n, level, a, &sup);
        else if (most) oct_sort<1>(p, in, n, level, a, &sup);
        if ((lane & 7u) == 0 && i < p.n0 && len <= kSortShort) S.support[i] = sup;
    }
}

// Bitonic stages size (compile time, > 1) with strides from..1 on 32 T
// entries in registers, entry 32 t + lane in k[t]; `at` = index of the first
// entry in the whole list (a multiple of 32 T).
template <int T>
__device__ __forceinline__ void warp_stages(uint32_t k[T], int size, int from, int at) {
    const int lane = (int)(threadIdx.x & 31u);
#pragma unroll
    for (int stride = 16 * T; stride; stride >>= 1) {
        if (stride > from) continue;
#pragma unroll
        for (int t = 0; t < T; ++t) {
            const bool up = ((at + 32 * t + lane) & size) == 0;
            if (stride >= 32) {
                const int o = t ^ (stride >> 5);
                if (o > t) {
                    const uint32_t lo = min(k[t], k[o]), hi = max(k[t], k[o]);
                    k[t] = up ? lo : hi;
                    k[o] = up ? hi : lo;
                }
            } else {
                const uint32_t o = __shfl_xor_sync(0xFFFFFFFFu, k[t], stride);
                k[t] = ((lane & stride) == 0) == up ? min(k[t], o) : max(k[t], o);
            }
        }
    }
}
// One warp per list of kSortShort+1 .. 32 T entries: bitonic sort in
// registers (the places past the end hold the largest value and stay last).
// 240 shuffles for 256 entries, where ranking every entry against every other
// took 2,048 comparisons per lane.  Returns the support count.
template <int T>
__device__ __forceinline__ int warp_sort(const SortArgs& p, const uint32_t* in, int n, int level, uint32_t* a) {
    const int lane = (int)(threadIdx.x & 31u);
    uint32_t k[T];
    int c = 0;
#pragma unroll
    for (int t = 0; t < T; ++t) k[t] = 32 * t + lane < n ? in[32 * t + lane] : 0xFFFFFFFFu;
#pragma unroll
    for (int t = 0; t < T; ++t)
        if (32 * t + lane < n) k[t] = rename(p, k[t], level, &c);
#pragma unroll
    for (int size = 2; size <= 32 * T; size <<= 1) warp_stages<T>(k, size, size >> 1, 0);
#pragma unroll
    for (int t = 0; t < T; ++t)
        if (32 * t + lane < n) a[32 * t + lane] = k[t];
    return __reduce_add_sync(0xFFFFFFFFu, c);
}
__global__ void __launch_bounds__(kSortThreads) k_sort_warp(SortArgs p) {
    static_assert(kSortWarp == 256, "eight entries per lane");
    const SortSide& S = p.side[blockIdx.y];
    const unsigned nl = p.cnt[3 * blockIdx.y], nw = gridDim.x * (kSortThreads / 32);
    for (unsigned li = blockIdx.x * (kSortThreads / 32) + (threadIdx.x >> 5); li < nl; li += nw) {
        const uint32_t v = S.list[0][li];
        const int n = S.len[v], level = support_level(p, v);
        uint32_t* a = S.nbr + S.off[v];
        const uint32_t* in = S.src + S.start[v];
        const int sup = n <= 64    ? warp_sort<2>(p, in, n, level, a)
                        : n <= 128 ? warp_sort<4>(p, in, n, level, a)
                                   : warp_sort<8>(p, in, n, level, a);
        if ((threadIdx.x & 31u) == 0 && v < p.n0) S.support[v] = sup;
    }
}

// One block per list of kSortWarp+1 .. kSortMid entries: bitonic sort.  Runs of
// 256 entries are sorted in registers by a warp each; of the later stages only
// the strides of 256 and more go through shared memory (10 block-wide passes
// for 4,096 entries instead of 78).
__global__ void __launch_bounds__(kSortThreads) k_sort_mid(SortArgs p) {
    __shared__ uint32_t s[kSortMid];
    __shared__ int s_sup;
    const SortSide& S = p.side[blockIdx.y];
    const int lane = (int)(threadIdx.x & 31u), w = (int)(threadIdx.x >> 5);
    const unsigned nl = p.cnt[3 * blockIdx.y + 1];
    if (threadIdx.x == 0) s_sup = 0;
    __syncthreads();
    for (unsigned li = blockIdx.x; li < nl; li += gridDim.x) {
        const uint32_t v = S.list[1][li];
        const int n = S.len[v], level = support_level(p, v);
        uint32_t* a = S.nbr + S.off[v];
        const uint32_t* in = S.src + S.start[v];
        int sup = 0;
        int N = 512;
        while (N < n) N <<= 1;
        for (int c = 256 * w; c < N; c += 8 * kSortThreads) {  // one run per warp and turn
            uint32_t k[8];
#pragma unroll
            for (int t = 0; t < 8; ++t) k[t] = c + 32 * t + lane < n ? in[c + 32 * t + lane] : 0xFFFFFFFFu;
#pragma unroll
            for (int t = 0; t < 8; ++t)
                if (c + 32 * t + lane < n) k[t] = rename(p, k[t], level, &sup);
#pragma unroll
            for (int size = 2; size <= 256; size <<= 1) warp_stages<8>(k, size, size >> 1, c);
#pragma unroll
            for (int t = 0; t < 8; ++t) s[c + 32 * t + lane] = k[t];
        }
        sup = __reduce_add_sync(0xFFFFFFFFu, sup);
        if (lane == 0 && sup) atomicAdd(&s_sup, sup);
        __syncthreads();
        if (threadIdx.x == 0) {
            if (v < p.n0) S.support[v] = s_sup;
            s_sup = 0;
        }
        for (int size = 512; size <= N; size <<= 1) {
            for (int stride = size >> 1; stride >= 256; stride >>= 1) {
                for (int q = threadIdx.x; q < N / 2; q += kSortThreads) {
                    const int i = ((q & ~(stride - 1)) << 1) | (q & (stride - 1)), o = i | stride;
                    const uint32_t x = s[i], y = s[o];
                    if ((x > y) == ((i & size) == 0)) {
                        s[i] = y;
                        s[o] = x;
                    }
                }
                __syncthreads();
            }
            for (int c = 256 * w; c < N; c += 8 * kSortThreads) {
                uint32_t k[8];
#pragma unroll
                for (int t = 0; t < 8; ++t) k[t] = s[c + 32 * t + lane];
                warp_stages<8>(k, size, 128, c);
                if (size < N) {
#pragma unroll
                    for (int t = 0; t < 8; ++t) s[c + 32 * t + lane] = k[t];
                } else {
#pragma unroll
                    for (int t = 0; t < 8; ++t)
                        if (c + 32 * t + lane < n) a[c + 32 * t + lane] = k[t];
                }
            }
            __syncthreads();
        }
    }
}

// One block per longer list: counting sort.  Bin of an id: its 32-id line (a
// cache line of values) while there are bins for lines, plus K - kmax, which
// grows with the id and keeps the classes of kmax apart; entries of a bin keep
// no particular order.  The list fits no shared memory, so its entries are
// renamed twice.  Bound by the longest list: 1,024 threads, four entries each.
static constexpr int kSortBigBins = 11264;
__global__ void __launch_bounds__(1024) k_sort_big(SortArgs p) {
    __shared__ unsigned bins[kSortBigBins];
    __shared__ int s_sup;
    const SortSide& S = p.side[blockIdx.y];
    const unsigned nl = p.cnt[3 * blockIdx.y + 2];
    const int K = p.K;
    const uint32_t lines = (uint32_t)(kSortBigBins - 1 - K);
    auto bin_of = [&](uint32_t u) { return (int)min(u >> 5, lines) + (K - p.kmax[u]); };
    for (unsigned li = blockIdx.x; li < nl; li += gridDim.x) {
        const uint32_t v = S.list[2][li];
        const int n = S.len[v], level = support_level(p, v);
        uint32_t* a = S.nbr + S.off[v];
        const uint32_t* in = S.src + S.start[v];
        int sup = 0;
        if (threadIdx.x == 0) s_sup = 0;
        for (int i = threadIdx.x; i < kSortBigBins; i += blockDim.x) bins[i] = 0;
        __syncthreads();
        // four entries in flight per thread (three dependent loads each)
        for (int i0 = threadIdx.x; i0 < n; i0 += 4 * blockDim.x) {
            uint32_t u[4];
            int b[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) u[q] = i0 + q * (int)blockDim.x < n ? in[i0 + q * blockDim.x] : 0xFFFFFFFFu;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (u[q] != 0xFFFFFFFFu) u[q] = rename(p, u[q], level, &sup);
#pragma unroll
            for (int q = 0; q < 4; ++q) b[q] = u[q] != 0xFFFFFFFFu ? bin_of(u[q]) : -1;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (b[q] >= 0) atomicAdd(&bins[b[q]], 1u);
        }
        if (sup) atomicAdd(&s_sup, sup);
        __syncthreads();
        if (threadIdx.x == 0 && v < p.n0) S.support[v] = s_sup;
        // exclusive scan of the bins, blockDim at a time
        unsigned long long carry = 0;
        for (int b0 = 0; b0 < kSortBigBins; b0 += blockDim.x) {
            const int b = b0 + threadIdx.x;
            const unsigned long long x = b < kSortBigBins ? bins[b] : 0ull;
            unsigned long long tot;
            const unsigned long long ex = block_excl_scan64(x, &tot);
            if (b < kSortBigBins) bins[b] = (unsigned)(ex + carry);
            carry += tot;
            __syncthreads();
        }
        for (int i0 = threadIdx.x; i0 < n; i0 += 4 * blockDim.x) {
            uint32_t u[4];
            int b[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) u[q] = i0 + q * (int)blockDim.x < n ? in[i0 + q * blockDim.x] : 0xFFFFFFFFu;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (u[q] != 0xFFFFFFFFu) u[q] = __ldg(p.pos + u[q]).x;
#pragma unroll
            for (int q = 0; q < 4; ++q) b[q] = u[q] != 0xFFFFFFFFu ? bin_of(u[q]) : -1;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (b[q] >= 0) a[atomicAdd(&bins[b[q]], 1u)] = u[q];
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// order by kmax, skyline assembly, expansion
// ---------------------------------------------------------------------------
// One pass over the vertices: counts per kmax value, the number of corners rows
// 1.. can have (min(kmax, row 0) each: *corners) and sum of (in + out degree) x
// kmax, the list entries a pass over rows 1..kmax scans, a deterministic
// measure of a graph's row work (*work).  Most vertices share a few small kmax
// values, so the counts go to per-block shared bins first (when kmax + 1 <=
// kHistShared).  Three kernels, each with its own read-back, took 30 us more.
constexpr int kHistShared = 8192;
__global__ void k_row_stats(uint32_t V, const int32_t* kmax, const int32_t* row0, const int32_t* in_len,
                            const int32_t* out_len, uint32_t* hist, int32_t K, unsigned long long* corners,
                            unsigned long long* work) {
    extern __shared__ uint32_t sh[];
    const bool shared = K + 1 <= kHistShared;
    if (shared)
        for (int i = threadIdx.x; i <= K; i += blockDim.x) sh[i] = 0;
    __syncthreads();
    unsigned long long c = 0, w = 0;
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V; v += (uint64_t)gridDim.x * blockDim.x) {
        const int k = kmax[v];
        atomicAdd(shared ? &sh[k] : &hist[k], 1u);
        c += (unsigned long long)min(k, row0[v]);
        w += (unsigned long long)(in_len[v] + out_len[v]) * (unsigned long long)k;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        c += __shfl_xor_sync(0xFFFFFFFFu, c, o);
        w += __shfl_xor_sync(0xFFFFFFFFu, w, o);
    }
    if ((threadIdx.x & 31u) == 0) {
        atomicAdd(corners, c);
        atomicAdd(work, w);
    }
    __syncthreads();
    if (shared)
        for (int i = threadIdx.x; i <= K; i += blockDim.x)
            if (sh[i]) atomicAdd(&hist[i], sh[i]);
}

// w[k] += in + out degree of every vertex with kmax == k (shared-memory
// bins when the range fits, else global atomics)
__global__ void k_kmax_degree_hist(uint32_t V, const int32_t* kmax, const int32_t* in_len, const int32_t* out_len,
                                   int32_t K, unsigned long long* w) {
    extern __shared__ unsigned long long sw[];
    const bool shared = K + 1 <= 4096;
    if (shared)
        for (int i = threadIdx.x; i <= K; i += blockDim.x) sw[i] = 0;
    __syncthreads();
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V; v += (uint64_t)gridDim.x * blockDim.x) {
        unsigned long long dgr = (unsigned long long)(in_len[v] + out_len[v]);
        if (shared) atomicAdd(&sw[kmax[v]], dgr);
        else atomicAdd(&w[kmax[v]], dgr);
    }
    __syncthreads();
    if (shared)
        for (int i = threadIdx.x; i <= K; i += blockDim.x)
            if (sw[i]) atomicAdd(&w[i], sw[i]);
}

// cursor[k] = first position of bucket k in descending-kmax order.  Most
// vertices share a few small kmax values, whose cursors bound the pass: the
// lanes of a warp that hold the same kmax count as one in the block's bins,
// and a block takes the positions of a bin's vertices with one atomic (one
// per warp and value: 73 us of R-MAT 20).  Values past the bins go to the
// cursor one warp at a time.
constexpr int kOrderBins = 1024, kOrderItems = 8;
__global__ void __launch_bounds__(kThreads) k_order_scatter(uint32_t V, const int32_t* kmax, int K, uint32_t* cursor,
                                                            uint32_t* order) {
    __shared__ uint32_t bin[kOrderBins];
    const unsigned lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    const int bins = min(K + 1, kOrderBins);
    for (uint64_t b = (uint64_t)blockIdx.x * kThreads * kOrderItems; b < V; b += (uint64_t)gridDim.x * kThreads * kOrderItems) {
        int key[kOrderItems];
        uint32_t at[kOrderItems];
        for (int i = threadIdx.x; i < bins; i += kThreads) bin[i] = 0;
        __syncthreads();
#pragma unroll
        for (int q = 0; q < kOrderItems; ++q) {
            const uint64_t v = b + q * kThreads + threadIdx.x;
            key[q] = v < V ? kmax[v] : -1;
        }
#pragma unroll
        for (int q = 0; q < kOrderItems; ++q) {
            const unsigned peers = __match_any_sync(0xFFFFFFFFu, key[q]), leader = __ffs(peers) - 1;
            uint32_t p0 = 0;
            if (key[q] >= 0 && lane == leader)
                p0 = atomicAdd(key[q] < bins ? &bin[key[q]] : &cursor[key[q]], (unsigned)__popc(peers));
            at[q] = __shfl_sync(0xFFFFFFFFu, p0, leader) + __popc(peers & below);
        }
        __syncthreads();
        for (int i = threadIdx.x; i < bins; i += kThreads)
            if (bin[i]) bin[i] = atomicAdd(&cursor[i], bin[i]);
        __syncthreads();
#pragma unroll
        for (int q = 0; q < kOrderItems; ++q)
            if (key[q] >= 0)
                order[at[q] + (key[q] < bins ? bin[key[q]] : 0u)] = (uint32_t)(b + q * kThreads + threadIdx.x);
        __syncthreads();
    }
}

// log entries with a negative row are void (dropped corners)
__global__ void k_sky_count(uint32_t V, uint64_t nlog, const uint32_t* log_v, const int32_t* log_k,
                            unsigned long long* cnt) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nlog; i += (uint64_t)gridDim.x * blockDim.x)
        if (log_k[i] >= 0) atomicAdd(&cnt[log_v[i]], 1ull);
}
__global__ void k_set_one(uint32_t V, unsigned long long* cnt) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V; v += (uint64_t)gridDim.x * blockDim.x)
        cnt[v] = 1ull;
}
__global__ void k_sky_fill_row0(uint32_t V, const unsigned long long* off, const int32_t* row0, int32_t* sky_k,
                                int32_t* sky_l, uint32_t* fill) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V; v += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t o = off[v];
        sky_k[o] = 0;
        sky_l[o] = row0[v];
        fill[v] = 1;
    }
}
__global__ void k_sky_fill_log(uint64_t nlog, const uint32_t* log_v, const int32_t* log_k, const int32_t* log_l,
                               const unsigned long long* off, int32_t* sky_k, int32_t* sky_l, uint32_t* fill) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nlog; i += (uint64_t)gridDim.x * blockDim.x) {
        if (log_k[i] < 0) continue;
        uint32_t v = log_v[i];
        uint32_t pos = atomicAdd(&fill[v], 1u);
        sky_k[off[v] + pos] = log_k[i];
        sky_l[off[v] + pos] = log_l[i];
    }
}
// sort each vertex's corners by k (insertion sort; lists are short)
__global__ void k_sky_sort(uint32_t V, const unsigned long long* off, int32_t* sky_k, int32_t* sky_l, uint32_t* off32) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V; v += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t a = off[v], b = off[v + 1];
        for (uint64_t i = a + 1; i < b; ++i) {
            int kk = sky_k[i], ll = sky_l[i];
            uint64_t jj = i;
            while (jj > a && sky_k[jj - 1] > kk) {
                sky_k[jj] = sky_k[jj - 1];
                sky_l[jj] = sky_l[jj - 1];
                --jj;
            }
            sky_k[jj] = kk;
            sky_l[jj] = ll;
        }
        off32[v] = (uint32_t)a;
        if (v == V - 1) off32[V] = (uint32_t)b;
    }
}

// Dense rows [k0, k0+n): rows[(k-k0)*V + v]
// Four consecutive vertices per thread and one 16-byte streaming store per
// row (V a multiple of 4, so every row starts 16-byte aligned); the output is
// far larger than L2, hence the streaming (evict-first) stores.
__global__ void k_expand4(uint32_t V, uint32_t k0, uint32_t n, const int32_t* kmax, const uint32_t* sky_off,
                          const int32_t* sky_k, const int32_t* sky_l, int32_t* rows) {
    const uint32_t V4 = V / 4;
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < V4; t += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t ci[4], b[4];
        int val[4], nextk[4], km[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t v = 4 * (uint32_t)t + q;
            const uint32_t a = sky_off[v];
            b[q] = sky_off[v + 1];
            km[q] = kmax[v];
            uint32_t c = a;
            while (c + 1 < b[q] && (uint32_t)sky_k[c + 1] <= k0) ++c;
            ci[q] = c;
            val[q] = sky_l[c];
            nextk[q] = (c + 1 < b[q]) ? sky_k[c + 1] : 0x7FFFFFFF;
        }
        int4* out = reinterpret_cast<int4*>(rows) + t;
        for (uint32_t r = 0; r < n; ++r) {
            const int k = (int)(k0 + r);
            int o[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                while (k >= nextk[q]) {
                    ++ci[q];
                    val[q] = sky_l[ci[q]];
                    nextk[q] = (ci[q] + 1 < b[q]) ? sky_k[ci[q] + 1] : 0x7FFFFFFF;
                }
                o[q] = (k <= km[q]) ? val[q] : 0;
            }
            __stcs(out + (uint64_t)r * V4, make_int4(o[0], o[1], o[2], o[3]));
        }
    }
}

__global__ void k_expand(uint32_t V, uint32_t k0, uint32_t n, const int32_t* kmax, const uint32_t* sky_off,
                         const int32_t* sky_k, const int32_t* sky_l, int32_t* rows) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V; v += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t a = sky_off[v], b = sky_off[v + 1];
        int km = kmax[v];
        uint32_t ci = a;
        while (ci + 1 < b && (uint32_t)sky_k[ci + 1] <= k0) ++ci;
        int val = sky_l[ci];
        int nextk = (ci + 1 < b) ? sky_k[ci + 1] : 0x7FFFFFFF;
        for (uint32_t r = 0; r < n; ++r) {
            int k = (int)(k0 + r);
            while (k >= nextk) {
                ++ci;
                val = sky_l[ci];
                nextk = (ci + 1 < b) ? sky_k[ci + 1] : 0x7FFFFFFF;
            }
            rows[(uint64_t)r * V + v] = (k <= km) ? val : 0;
        }
    }
}

// skyline from dense rows (per-row peel method)
__global__ void k_rows_corner_count(uint32_t V, uint32_t K, const int32_t* kmax, const int32_t* rows,
                                    unsigned long long* cnt) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V; v += (uint64_t)gridDim.x * blockDim.x) {
        int km = kmax[v];
        unsigned long long c = 1;
        for (int k = 1; k <= km; ++k) c += rows[(uint64_t)k * V + v] != rows[(uint64_t)(k - 1) * V + v];
        cnt[v] = c;
    }
}
__global__ void k_rows_corner_fill(uint32_t V, const int32_t* kmax, const int32_t* rows, const unsigned long long* off,
                                   int32_t* sky_k, int32_t* sky_l, uint32_t* off32) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V; v += (uint64_t)gridDim.x * blockDim.x) {
        int km = kmax[v];
        uint64_t o = off[v];
        sky_k[o] = 0;
        sky_l[o] = rows[v];
        ++o;
        for (int k = 1; k <= km; ++k) {
            int x = rows[(uint64_t)k * V + v];
            if (x != rows[(uint64_t)(k - 1) * V + v]) {
                sky_k[o] = k;
                sky_l[o] = x;
                ++o;
            }
        }
        off32[v] = (uint32_t)off[v];
        if (v == V - 1) off32[V] = (uint32_t)off[V];
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static int grid_for(dc_graph* h, uint64_t n) {
    uint64_t b = (n + kThreads - 1) / kThreads;
    uint64_t cap = (uint64_t)h->geom.sms * 16;
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return (int)b;
}

int coop_launch(dc_graph* h, const void* fn, void** args, int threads, const char* name) {
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, 0);
    if (e != cudaSuccess || per_sm < 1)
        return set_error(DC_ERR_CUDA, "%s: occupancy query failed (%s)", name, cudaGetErrorString(e));
    per_sm = std::min(per_sm, 1024 / threads);
    dim3 grid((unsigned)(per_sm * h->geom.sms)), block((unsigned)threads);
    DC_CUDA(cudaMemsetAsync(h->ctl, 0, sizeof(EngineCtl), h->stream));
    e = cudaLaunchCooperativeKernel(fn, grid, block, args, 0, h->stream);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return set_error(DC_ERR_CUDA, "%s: cooperative launch failed (%s)", name, cudaGetErrorString(e));
    }
    return DC_OK;
}

int check_ctl(dc_graph* h, EngineCtl* hc, const char* what) { return check_ctl_on(h->ctl, h->stream, hc, what); }

int check_ctl_on(EngineCtl* ctl, cudaStream_t st, EngineCtl* hc, const char* what) {
    DC_CUDA(cudaMemcpyAsync(hc, ctl, sizeof(EngineCtl), cudaMemcpyDeviceToHost, st));
    DC_CUDA(cudaStreamSynchronize(st));
    if (hc->error) {
        if (hc->error & DC_DEV_ERR_TIMEOUT)
            return set_error(DC_ERR_TIMEOUT, "%s: bounded device wait expired (site %u)", what, hc->err_where);
        if (hc->error & DC_DEV_ERR_BADID) return set_error(DC_ERR_INVALID, "%s: vertex id out of range", what);
        if (hc->error & DC_DEV_ERR_CAPACITY) return set_error(DC_ERR_CAPACITY, "%s: device buffer capacity exceeded", what);
        return set_error(DC_ERR_CUDA, "%s: device error 0x%x (site %u)", what, hc->error, hc->err_where);
    }
    return DC_OK;
}

int init_handle(dc_graph* h) {
    DC_CUDA(cudaGetDevice(&h->device));
    // two attributes, not the whole property set (cudaGetDeviceProperties is
    // slow, and every handle pays this)
    int coop = 0, sms = 0;
    DC_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, h->device));
    DC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->device));
    if (!coop) return set_error(DC_ERR_NO_DEVICE, "device lacks cooperative launch");
    h->geom.sms = sms;
    h->geom.threads = kThreads;
    DC_CUDA(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking));
    // Freed blocks stay in the device's default pool for reuse instead of
    // going back to the driver at every synchronisation.
    cudaMemPool_t pool;
    DC_CUDA(cudaDeviceGetDefaultMemPool(&pool, h->device));
    uint64_t keep = ~0ull;
    DC_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    if (dmalloc(h->stream, &h->ctl, 1)) return DC_ERR_NOMEM;
    for (auto& e : h->ev) DC_CUDA(cudaEventCreate(&e));
    return DC_OK;
}

void free_graph_arrays(DevGraph& g, cudaStream_t st) {
    dfree(st, g.out_off);
    dfree(st, g.out_len);
    dfree(st, g.out_nbr);
    dfree(st, g.in_off);
    dfree(st, g.in_len);
    dfree(st, g.in_nbr);
    g.out_cap = g.in_cap = 0;
}

int sky_take_spare(dc_graph* h, int slot, uint64_t n, uint32_t** off, int32_t** k, int32_t** l, uint64_t* cap) {
    Decomp& d = h->d;
    if (d.spare_cap[slot] < n || !d.spare_k[slot]) {
        dfree(h->stream, d.spare_k[slot]);
        dfree(h->stream, d.spare_l[slot]);
        d.spare_cap[slot] = 0;
        const uint64_t want = n + n / 4 + 1;
        if (dmalloc(h->stream, &d.spare_k[slot], want) || dmalloc(h->stream, &d.spare_l[slot], want))
            return DC_ERR_NOMEM;
        d.spare_cap[slot] = want;
    }
    if (!d.spare_off[slot] && dmalloc(h->stream, &d.spare_off[slot], (uint64_t)h->g.V + 1)) return DC_ERR_NOMEM;
    *off = d.spare_off[slot];
    *k = d.spare_k[slot];
    *l = d.spare_l[slot];
    *cap = d.spare_cap[slot];
    d.spare_off[slot] = nullptr;
    d.spare_k[slot] = nullptr;
    d.spare_l[slot] = nullptr;
    d.spare_cap[slot] = 0;
    return DC_OK;
}

void sky_put_spare(dc_graph* h, int slot, uint32_t* off, int32_t* k, int32_t* l, uint64_t cap) {
    Decomp& d = h->d;
    dfree(h->stream, d.spare_off[slot]);
    dfree(h->stream, d.spare_k[slot]);
    dfree(h->stream, d.spare_l[slot]);
    d.spare_off[slot] = off;
    d.spare_k[slot] = k;
    d.spare_l[slot] = l;
    d.spare_cap[slot] = (k && l) ? cap : 0;
}

void free_decomp(Decomp& d, cudaStream_t st) {
    dfree(st, d.kmax_v);
    dfree(st, d.row0);
    dfree(st, d.sky_off);
    dfree(st, d.sky_k);
    dfree(st, d.sky_l);
    dfree(st, d.rows);
    for (int i = 0; i < 2; ++i) {
        dfree(st, d.spare_off[i]);
        dfree(st, d.spare_k[i]);
        dfree(st, d.spare_l[i]);
        d.spare_cap[i] = 0;
    }
    d.rows_cap = 0;
    d.corner_cap = 0;
    d.valid = false;
    d.rows_valid = false;
}

// The row groups' state; returns whether there was any.
static bool free_groups(dc_graph* h) {
    Scratch* s = h->scratch;
    bool any = s->seam != nullptr;
    for (RowSegment& g : s->seg) {
        any = any || g.cur || g.tring;
        dfree(h->stream, g.cur);
        dfree(h->stream, g.cnt_out);
        dfree(h->stream, g.cnt_in);
        dfree(h->stream, g.mark);
        dfree(h->stream, g.stamp);
        dfree(h->stream, g.logidx);
        dfree(h->stream, g.tring);
        dfree(h->stream, g.ctl);
        g.cap_V = 0;
        g.tring_cap = 0;
    }
    dfree(h->stream, s->seam_of);
    dfree(h->stream, s->seam);
    s->seam_of_cap = 0;
    s->seam_cap = 0;
    return any;
}

void free_scratch(dc_graph* h) {
    Scratch* s = h->scratch;
    if (!s) return;
    free_groups(h);
    dfree(h->stream, s->key);
    dfree(h->stream, s->cdeg);
    dfree(h->stream, s->cur);
    dfree(h->stream, s->row0);
    dfree(h->stream, s->mark);
    dfree(h->stream, s->stamp);
    dfree(h->stream, s->logidx);
    dfree(h->stream, s->rem0);
    dfree(h->stream, s->rem1);
    dfree(h->stream, s->order);
    dfree(h->stream, s->ck);
    dfree(h->stream, s->log_v);
    dfree(h->stream, s->log_k);
    dfree(h->stream, s->log_l);
    dfree(h->stream, s->tmp64);
    dfree(h->stream, s->partial);
    dfree(h->stream, s->cursor);
    dfree(h->stream, s->key2);
    dfree(h->stream, s->cdeg2);
    dfree(h->stream, s->rem2);
    dfree(h->stream, s->rem3);
    dfree(h->stream, s->cnt_out);
    dfree(h->stream, s->tring);
    dfree(h->stream, s->kmax_old);
    dfree(h->stream, s->row0_old);
    dfree(h->stream, s->plan);
    dfree(h->stream, s->pos);
    dfree(h->stream, s->kmax_r);
    dfree(h->stream, s->row0_r);
    for (int i = 0; i < 2; ++i) {
        dfree(h->stream, s->r_off[i]);
        dfree(h->stream, s->r_len[i]);
        dfree(h->stream, s->r_nbr[i]);
    }
    delete s;
    h->scratch = nullptr;
}

static uint64_t scan_words(const dc_graph* h) { return (uint64_t)h->geom.sms * 64 + 64; }
static unsigned* scan_ticket(dc_graph* h) { return (unsigned*)(h->scratch->partial + scan_words(h) - 1); }

int ensure_scratch(dc_graph* h, uint32_t V) {
    if (!h->scratch) h->scratch = new Scratch();
    Scratch* s = h->scratch;
    if (s->cap_V >= V && s->key) return DC_OK;
    // release V-sized buffers and reallocate
    dfree(h->stream, s->key); dfree(h->stream, s->cdeg); dfree(h->stream, s->cur); dfree(h->stream, s->row0); dfree(h->stream, s->mark); dfree(h->stream, s->stamp);
    dfree(h->stream, s->logidx); dfree(h->stream, s->rem0); dfree(h->stream, s->rem1); dfree(h->stream, s->order); dfree(h->stream, s->tmp64);
    dfree(h->stream, s->partial); dfree(h->stream, s->cursor);
    dfree(h->stream, s->key2); dfree(h->stream, s->cdeg2); dfree(h->stream, s->rem2); dfree(h->stream, s->rem3); dfree(h->stream, s->cnt_out);
    uint64_t n = (uint64_t)V + 1;
    if (dmalloc(h->stream, &s->key, n) || dmalloc(h->stream, &s->cdeg, n) || dmalloc(h->stream, &s->cur, n) || dmalloc(h->stream, &s->row0, n) ||
        dmalloc(h->stream, &s->mark, n) || dmalloc(h->stream, &s->stamp, n) || dmalloc(h->stream, &s->logidx, n) || dmalloc(h->stream, &s->rem0, n) ||
        dmalloc(h->stream, &s->rem1, n) || dmalloc(h->stream, &s->order, n) || dmalloc(h->stream, &s->tmp64, n + 1) ||
        dmalloc(h->stream, &s->partial, scan_words(h)) || dmalloc(h->stream, &s->cursor, n + 1) ||
        dmalloc(h->stream, &s->key2, n) || dmalloc(h->stream, &s->cdeg2, n) || dmalloc(h->stream, &s->rem2, n) || dmalloc(h->stream, &s->rem3, n) ||
        dmalloc(h->stream, &s->cnt_out, n))
        return DC_ERR_NOMEM;
    DC_CUDA(cudaMemsetAsync(scan_ticket(h), 0, sizeof(unsigned), h->stream));
    s->cap_V = V;
    return DC_OK;
}

uint64_t device_footprint(const dc_graph* h) {
    const DevGraph& g = h->g;
    const Decomp& d = h->d;
    uint64_t V1 = (uint64_t)g.V + 1;
    uint64_t b = sizeof(EngineCtl);
    if (g.out_off) b += 2 * 4 * (2 * V1) + 4 * (g.out_cap + g.in_cap);
    if (d.kmax_v) b += 4 * (3 * V1) + 8 * d.corner_cap;
    for (int i = 0; i < 2; ++i) b += 8 * d.spare_cap[i] + (d.spare_off[i] ? 4 * V1 : 0);
    b += 4 * d.rows_cap;
    if (const Scratch* s = h->scratch) {
        uint64_t n = (uint64_t)s->cap_V + 1;
        if (s->key) b += 4 * (16 * n + 1) + 8 * (n + 1) + 8 * ((uint64_t)h->geom.sms * 64 + 64);
        b += 8ull * s->ck_cap + 12 * s->log_cap + 8 * s->tring_cap;
        if (s->kmax_old) b += 8 * n;
        for (const RowSegment& sg : s->seg)
            b += (sg.cur ? 24 * ((uint64_t)sg.cap_V + 1) : 0) + 8 * sg.tring_cap + (sg.ctl ? sizeof(EngineCtl) : 0);
        b += (s->plan ? sizeof(RowPlan) : 0) + 4ull * s->seam_of_cap + 4 * s->seam_cap;
        if (s->pos) b += 4 * 8 * ((uint64_t)s->r_cap_V + 1);     // relabeled graph: ids, kmax, row 0, offsets, lengths
        if (s->r_nbr[0]) b += 2 * 4 * s->r_cap;     // its lists
    }
    return b;
}

// Grid of the prefix sums over n elements: at most 16 blocks per SM (two sides'
// sums fit s->partial), a tile each at least.
static unsigned scan_blocks(const dc_graph* h, uint64_t n) {
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((n + kScanTile - 1) / kScanTile, 16ull * h->geom.sms));
}

template <class A>
static void scan_sums(dc_graph* h, const A& a, int sides, uint64_t n, unsigned long long* total = nullptr) {
    ++g_launches;
    k_scan_sums<A><<<dim3(scan_blocks(h, n), sides), kScanThreads, 0, h->stream>>>(
        a, n, (unsigned long long*)h->scratch->partial, scan_ticket(h), total);
}
template <class A>
static void scan_apply(dc_graph* h, const A& a, int sides, uint64_t n) {
    ++g_launches;
    k_scan_apply<A><<<dim3(scan_blocks(h, n), sides), kScanThreads, 0, h->stream>>>(
        a, n, (const unsigned long long*)h->scratch->partial);
}

// Exclusive scan of n u64 values in s->tmp64 (tmp64[n] receives the total).
int scan_tmp64(dc_graph* h, uint64_t n) {
    const WordsInPlace a{(unsigned long long*)h->scratch->tmp64};
    scan_sums(h, a, 1, n);
    scan_apply(h, a, 1, n);
    DC_CUDA(cudaGetLastError());
    return DC_OK;
}

int build_from_device_edges(dc_graph* h, uint32_t V, uint64_t E, const uint32_t* d_src, const uint32_t* d_dst) {
    free_graph_arrays(h->g, h->stream);
    free_decomp(h->d, h->stream);
    if (int rc = ensure_scratch(h, V)) return rc;
    DevGraph& g = h->g;
    if (dmalloc(h->stream, &g.out_len, (uint64_t)V + 1) || dmalloc(h->stream, &g.in_len, (uint64_t)V + 1)) return DC_ERR_NOMEM;
    DC_CUDA(cudaMemsetAsync(g.out_len, 0, sizeof(int32_t) * ((uint64_t)V + 1), h->stream));
    DC_CUDA(cudaMemsetAsync(g.in_len, 0, sizeof(int32_t) * ((uint64_t)V + 1), h->stream));
    DC_CUDA(cudaMemsetAsync(h->ctl, 0, sizeof(EngineCtl), h->stream));
    if (E) {
        ++g_launches;
        k_count_degrees<<<grid_for(h, E), kThreads, 0, h->stream>>>(V, E, d_src, d_dst, g.out_len, g.in_len, h->ctl);
    }
    // list starts; the totals come back with the status of the count
    ListStarts ls{{g.out_len, g.in_len}, {nullptr, nullptr}, h->gap_min, h->gap_div};
    static_assert(offsetof(EngineCtl, drops) == offsetof(EngineCtl, evals) + 8, "two totals side by side");
    scan_sums(h, ls, 2, V, &h->ctl->evals);
    if (V <= kSmallPeelV) {  // (other peels do not ask)
        ++g_launches;
        k_max_len<<<grid_for(h, V), kThreads, 0, h->stream>>>(V, g.out_len, g.in_len, &h->ctl->maxv[0]);
    }
    EngineCtl hc;
    if (int rc = check_ctl(h, &hc, "graph build")) return rc;
    g.max_len = (uint32_t)hc.maxv[0];
    if (hc.evals >= 0xFFFFFFFFull || hc.drops >= 0xFFFFFFFFull)
        return set_error(DC_ERR_CAPACITY, "adjacency with slack exceeds 2^32 entries (u32 offsets)");
    if (dmalloc(h->stream, &g.out_off, (uint64_t)V + 1) || dmalloc(h->stream, &g.out_nbr, hc.evals) ||
        dmalloc(h->stream, &g.in_off, (uint64_t)V + 1) || dmalloc(h->stream, &g.in_nbr, hc.drops))
        return DC_ERR_NOMEM;
    g.out_cap = hc.evals;
    g.in_cap = hc.drops;
    ls.off[0] = g.out_off;
    ls.off[1] = g.in_off;
    scan_apply(h, ls, 2, V);
    DC_CUDA(cudaMemsetAsync(g.out_len, 0, sizeof(int32_t) * V, h->stream));
    DC_CUDA(cudaMemsetAsync(g.in_len, 0, sizeof(int32_t) * V, h->stream));
    if (E) {
        ++g_launches;
        k_scatter_edges<<<grid_for(h, E), kThreads, 0, h->stream>>>(E, d_src, d_dst, g.out_off, g.out_len, g.out_nbr,
                                                                     g.in_off, g.in_len, g.in_nbr);
    }
    DC_CUDA(cudaGetLastError());
    g.V = V;
    g.E = E;
    return DC_OK;
}

// Expands a CSR with arbitrary per-list slots into an edge list on device.
__global__ void k_csr_to_edges(uint32_t V, const uint32_t* off, const int32_t* len, const unsigned long long* eoff,
                               const uint32_t* nbr, uint32_t* src, uint32_t* dst, int swap) {
    const unsigned lane = threadIdx.x & 31u;
    const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t v = gw; v < V; v += nw) {
        uint32_t o = off[v];
        int n = len[v];
        uint64_t e0 = eoff[v];
        for (int i = lane; i < n; i += 32) {
            uint32_t u = nbr[o + i];
            if (!swap) {
                src[e0 + i] = (uint32_t)v;
                dst[e0 + i] = u;
            } else {
                src[e0 + i] = u;
                dst[e0 + i] = (uint32_t)v;
            }
        }
    }
}

int build_from_host_csr(dc_graph* h, uint32_t V, uint64_t E, const int32_t* in_deg, const int32_t* out_deg,
                        const uint32_t* in_off, const uint32_t* out_off, const uint32_t* in_nbr,
                        const uint32_t* out_nbr, uint64_t nbr_len) {
    (void)in_deg;
    (void)in_off;
    (void)in_nbr;
    // The reference binary stores both directions; the out-lists define the
    // edge multiset, so the device rebuilds both sides from them.
    free_graph_arrays(h->g, h->stream);
    free_decomp(h->d, h->stream);
    if (int rc = ensure_scratch(h, V)) return rc;
    uint32_t *d_off = nullptr, *d_nbr = nullptr, *d_src = nullptr, *d_dst = nullptr;
    int32_t* d_deg = nullptr;
    int rc = DC_OK;
    if ((rc = dmalloc(h->stream, &d_off, (uint64_t)V + 1)) || (rc = dmalloc(h->stream, &d_nbr, nbr_len)) || (rc = dmalloc(h->stream, &d_deg, V)) ||
        (rc = dmalloc(h->stream, &d_src, E)) || (rc = dmalloc(h->stream, &d_dst, E))) {
        dfree(h->stream, d_off); dfree(h->stream, d_nbr); dfree(h->stream, d_deg); dfree(h->stream, d_src); dfree(h->stream, d_dst);
        return rc;
    }
    Scratch* s = h->scratch;
    cudaMemcpyAsync(d_off, out_off, sizeof(uint32_t) * ((uint64_t)V + 1), cudaMemcpyHostToDevice, h->stream);
    cudaMemcpyAsync(d_nbr, out_nbr, sizeof(uint32_t) * nbr_len, cudaMemcpyHostToDevice, h->stream);
    cudaMemcpyAsync(d_deg, out_deg, sizeof(int32_t) * V, cudaMemcpyHostToDevice, h->stream);
    // edge offsets = exclusive scan of degrees
    std::vector<unsigned long long> eo((size_t)V + 1);
    unsigned long long acc = 0;
    for (uint32_t v = 0; v < V; ++v) {
        eo[v] = acc;
        acc += (unsigned long long)out_deg[v];
    }
    eo[V] = acc;
    if (acc != E) {
        dfree(h->stream, d_off); dfree(h->stream, d_nbr); dfree(h->stream, d_deg); dfree(h->stream, d_src); dfree(h->stream, d_dst);
        return set_error(DC_ERR_INVALID, "binary graph: out-degrees sum to %llu, header says %llu", acc,
                         (unsigned long long)E);
    }
    cudaMemcpyAsync(s->tmp64, eo.data(), sizeof(unsigned long long) * ((size_t)V + 1), cudaMemcpyHostToDevice,
                    h->stream);
    ++g_launches;
    k_csr_to_edges<<<grid_for(h, (uint64_t)V * 32), kThreads, 0, h->stream>>>(
        V, d_off, d_deg, (const unsigned long long*)s->tmp64, d_nbr, d_src, d_dst, 0);
    cudaError_t e = cudaStreamSynchronize(h->stream);
    dfree(h->stream, d_off);
    dfree(h->stream, d_nbr);
    dfree(h->stream, d_deg);
    if (e != cudaSuccess) {
        dfree(h->stream, d_src); dfree(h->stream, d_dst);
        return set_error(DC_ERR_CUDA, "binary graph upload failed: %s", cudaGetErrorString(e));
    }
    rc = build_from_device_edges(h, V, E, d_src, d_dst);
    cudaStreamSynchronize(h->stream);
    dfree(h->stream, d_src);
    dfree(h->stream, d_dst);
    return rc;
}

int ensure_tring(dc_graph* h, uint64_t need) {
    Scratch* s = h->scratch;
    uint64_t cap = 1024;
    while (cap < need) cap <<= 1;
    if (s->tring_cap >= cap && s->tring) return DC_OK;
    dfree(h->stream, s->tring);
    s->tring_cap = 0;
    if (dmalloc(h->stream, &s->tring, cap)) return DC_ERR_NOMEM;
    s->tring_cap = cap;
    DC_CUDA(cudaMemsetAsync(s->tring, 0xFF, sizeof(unsigned long long) * cap, h->stream));
    return DC_OK;
}

// Two 256-thread blocks per SM where nothing better is known (the autotuner
// refines it).
static constexpr int kDefaultBlocksPerSm = 2;

static int persistent_grid(dc_graph* h, const void* fn, int bps, int* blocks) {
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kThreads, 0);
    if (e != cudaSuccess || per_sm < 1)
        return set_error(DC_ERR_CUDA, "occupancy query failed (%s)", cudaGetErrorString(e));
    if (bps <= 0) bps = h->blocks_per_sm > 0 ? h->blocks_per_sm : kDefaultBlocksPerSm;
    *blocks = std::min(bps, per_sm) * h->geom.sms;
    return DC_OK;
}

// A control block as persistent_launch prepares it (no trace, no test
// hook), written by the device: usable inside a captured CUDA graph.
__global__ void k_ctl_init(EngineCtl* c, unsigned long long wait_ns) {
    uint32_t* w = reinterpret_cast<uint32_t*>(c);
    for (uint32_t i = threadIdx.x; i < sizeof(EngineCtl) / 4; i += blockDim.x) w[i] = 0;
    __syncthreads();
    if (threadIdx.x == 0) {
        c->step = -1;
        c->wait_ns = wait_ns;
    }
}

int ctl_init_enqueue(dc_graph* h, EngineCtl* ctl, cudaStream_t st) {
    ++g_launches;
    k_ctl_init<<<1, 256, 0, st>>>(ctl, h->wait_ns);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? DC_OK : set_error(DC_ERR_CUDA, "control block init: %s", cudaGetErrorString(e));
}

// Capture-safe persistent launch: the control block is initialised by a
// kernel and nothing is waited for (the caller reads the block's status
// later).
int persistent_enqueue(dc_graph* h, const void* fn, void** args, const char* name, EngineCtl* ctl, cudaStream_t st,
                       int bps) {
    int blocks = 0;
    if (int rc = persistent_grid(h, fn, bps, &blocks)) return rc;
    if (int rc = ctl_init_enqueue(h, ctl, st)) return rc;
    ++g_launches;
    cudaError_t e = cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(kThreads), args, 0, st);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return set_error(DC_ERR_CUDA, "%s: cooperative launch failed (%s)", name, cudaGetErrorString(e));
    }
    return DC_OK;
}

// Initialises a control block (on stream st) and launches a persistent
// kernel there without waiting.  The handle's own block carries the trace.
// first: the kernel's first step (nullptr: it starts with a grid barrier);
// grid: blocks (0: by blocks per SM).
static int persistent_launch(dc_graph* h, const void* fn, void** args, const char* name, EngineCtl* ctl,
                             cudaStream_t st, int bps, const FirstStep* first = nullptr, int grid = 0) {
    int blocks = grid;
    if (!blocks)
        if (int rc = persistent_grid(h, fn, bps, &blocks)) return rc;
    const bool own = ctl == h->ctl;
    EngineCtl& init = h->ctl_init;
    memset(&init, 0, sizeof(init));
    init.step = -1;
    init.wait_ns = h->wait_ns;
    if (first) {
        init.step = 0;
        init.t_work = (unsigned long long)(first->blocks ? first->blocks : blocks) << kWorkShift;
        for (auto& w : init.step_word) w.v = (1ull << 32) | (unsigned long long)(uint32_t)first->level;
    }
    if (own) {
        init.trace = h->trace_dev;
        init.trace_cap = h->trace_cap;
        if (h->barrier_fault_block >= 0) {  // one launch only
            init.test_skip_block = h->barrier_fault_block + 1;
            h->barrier_fault_block = -1;
        }
    }
    DC_CUDA(cudaMemcpyAsync(ctl, &init, sizeof(EngineCtl), cudaMemcpyHostToDevice, st));
    if (own && h->trace_dev) DC_CUDA(cudaMemsetAsync(h->trace_dev, 0, 64ull * h->trace_cap, st));
    ++g_launches;
    cudaError_t e = cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(kThreads), args, 0, st);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return set_error(DC_ERR_CUDA, "%s: cooperative launch failed (%s)", name, cudaGetErrorString(e));
    }
    return DC_OK;
}

// Waits for a persistent kernel launched on stream st with control block ctl
// and converts its device status; the handle's own block also delivers the
// trace.  A failed phase may leave items in its ring, which is cleared.
static int finish_persistent(dc_graph* h, EngineCtl* ctl, cudaStream_t st, const char* name, EngineCtl* out) {
    int rc = check_ctl_on(ctl, st, out, name);
    const bool own = ctl == h->ctl;
    if (own && h->trace_dev && h->trace_host) {
        cudaMemcpy(h->trace_host, h->trace_dev, 64ull * h->trace_cap, cudaMemcpyDeviceToHost);
        h->trace_steps = (unsigned)std::max(0, out->step);
        if (h->trace_cb) h->trace_cb(name, h->trace_host, h->trace_steps, h->trace_user);
    }
    if (rc != DC_OK) {
        Scratch* s = h->scratch;
        cudaMemsetAsync(s->tring, 0xFF, sizeof(unsigned long long) * s->tring_cap, st);
        cudaStreamSynchronize(st);
    }
    return rc;
}

// Launches a persistent kernel, waits, and converts its device status.
int run_persistent(dc_graph* h, const void* fn, void** args, const char* name, EngineCtl* out, int bps,
                   const FirstStep* first) {
    if (int rc = persistent_launch(h, fn, args, name, h->ctl, h->stream, bps, first)) return rc;
    return finish_persistent(h, h->ctl, h->stream, name, out);
}

// State of row group i + 1 for the ids below n of the relabeled graph, with
// an eighth of headroom.
static int ensure_segment(dc_graph* h, int i, uint32_t n) {
    RowSegment& g = h->scratch->seg[i];
    if (!g.ctl && dmalloc(h->stream, &g.ctl, 1)) return DC_ERR_NOMEM;
    if (g.cap_V < n || !g.cur) {
        dfree(h->stream, g.cur);
        dfree(h->stream, g.cnt_out);
        dfree(h->stream, g.cnt_in);
        dfree(h->stream, g.mark);
        dfree(h->stream, g.stamp);
        dfree(h->stream, g.logidx);
        g.cap_V = 0;
        const uint64_t m = (uint64_t)n + n / 8 + 1;
        if (dmalloc(h->stream, &g.cur, m) || dmalloc(h->stream, &g.cnt_out, m) || dmalloc(h->stream, &g.cnt_in, m) ||
            dmalloc(h->stream, &g.mark, m) || dmalloc(h->stream, &g.stamp, m) || dmalloc(h->stream, &g.logidx, m))
            return DC_ERR_NOMEM;
        g.cap_V = (uint32_t)std::min<uint64_t>(m - 1, 0xFFFFFFFFull);
    }
    uint64_t need = 2ull * n + (uint64_t)h->geom.sms * 64 + 4096, cap = 1024;
    while (cap < need) cap <<= 1;
    if (g.tring_cap < cap || !g.tring) {
        dfree(h->stream, g.tring);
        g.tring_cap = 0;
        if (dmalloc(h->stream, &g.tring, cap)) return DC_ERR_NOMEM;
        g.tring_cap = cap;
        DC_CUDA(cudaMemsetAsync(g.tring, 0xFF, sizeof(unsigned long long) * cap, h->stream));
    }
    return DC_OK;
}

PeelInst make_inst(dc_graph* h, int which, const int32_t* member, int32_t k, int32_t* val, int slot) {
    DevGraph& g = h->g;
    Scratch* s = h->scratch;
    PeelInst I;
    if (which == 0) {
        I.a_off = g.in_off; I.a_len = g.in_len; I.a_nbr = g.in_nbr;
        I.b_off = g.out_off; I.b_len = g.out_len; I.b_nbr = g.out_nbr;
    } else {
        I.a_off = g.out_off; I.a_len = g.out_len; I.a_nbr = g.out_nbr;
        I.b_off = g.in_off; I.b_len = g.in_len; I.b_nbr = g.in_nbr;
    }
    I.member = member;
    I.k = k;
    I.val = val;
    if (slot == 0) {
        I.key = s->key; I.cdeg = s->cdeg; I.rem0 = s->rem0; I.rem1 = s->rem1;
    } else {
        I.key = s->key2; I.cdeg = s->cdeg2; I.rem0 = s->rem2; I.rem1 = s->rem3;
    }
    return I;
}

// A peel is over when every vertex is removed (the last level's scan reports
// what its warps removed before); a vertex left would go into the rows with
// -1 for its kmax, an index there.
static int peel_status(const EngineCtl& c, int ninst, int32_t* maxv) {
    for (int i = 0; i < ninst; ++i) {
        if (c.removed[i] != c.members[i])
            return set_error(DC_ERR_CUDA, "peel: ended with %u of %u vertices removed", c.removed[i], c.members[i]);
        maxv[i] = c.maxv[i];
    }
    return DC_OK;
}

// Runs one or two peels in one persistent launch; maxv[i] = largest value.
int run_peel2(dc_graph* h, int ninst, const PeelInst* inst, int32_t* maxv) {
    Scratch* s = h->scratch;
    DevGraph& g = h->g;
    // one block per peel where the shapes were never set (a trace or a barrier
    // test wants the grid's kernel)
    if (h->peel_bps <= 0 && h->blocks_per_sm <= 0 && !inst[0].member && peel_fits_block(g) && !h->trace_dev &&
        h->barrier_fault_block < 0) {
        SmallPeel sp;
        sp.in[0] = inst[0];
        sp.in[1] = ninst > 1 ? inst[1] : inst[0];
        sp.V = g.V;
        sp.ctl = h->ctl;
        const int shm = (int)(6u * g.V + 8u);
        DC_CUDA(cudaFuncSetAttribute((const void*)k_peel_small, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(6u * kSmallPeelV + 8u)));
        DC_CUDA(cudaMemsetAsync(h->ctl, 0, sizeof(EngineCtl), h->stream));
        ++g_launches;
        k_peel_small<<<ninst, kSmallPeelThreads, shm, h->stream>>>(sp);
        DC_CUDA(cudaGetLastError());
        EngineCtl hc;
        if (int rc = check_ctl(h, &hc, "peel")) return rc;
        return peel_status(hc, ninst, maxv);
    }
    const unsigned chunk = h->peel_chunk ? h->peel_chunk : 64;
    // bags (at least 8 of the 2 V vertices each) and pieces of long lists
    uint64_t need = 2ull * g.V + 2ull * (g.out_cap + g.in_cap) / (4ull * chunk) + (uint64_t)h->geom.sms * 64 + 4096;
    if (int rc = ensure_tring(h, need)) return rc;
    Peel2Params p;
    p.V = g.V;
    p.ninst = ninst;
    p.chunk = chunk;
    p.in[0] = inst[0];
    p.in[1] = ninst > 1 ? inst[1] : inst[0];
    p.bag = (uint32_t*)s->tmp64;  // V + 2 words of 8 bytes; no scan runs meanwhile
    p.q.slots = s->tring;
    p.q.mask = (unsigned)(s->tring_cap - 1);
    p.ctl = h->ctl;
    void* args[] = {&p};
    EngineCtl hc;
    const void* fn = inst[0].member ? (const void*)k_peel2<true> : (const void*)k_peel2<false>;
    // Blocks on a handle that was not told: every block adds about 9 ns to a
    // light level, and large levels want more warps.  1 / 2 / 3 blocks per SM:
    // R-MAT 13 0.87 / 0.91 / 0.99 ms, R-MAT 15 1.15 / 1.23 / 1.32, ER of 10,000
    // 0.19 / 0.20 / 0.22, of 60,000 (60 edges per vertex) 0.47 / 0.43 / 0.45,
    // of 100,000 0.23 / 0.22 / 0.22, R-MAT 20 4.5 / 4.4 / 4.6, R-MAT 21 6.3 /
    // 5.7 / 5.9, R-MAT 22 10.0 / 8.5 / 8.6, ER of 3 M 2.99 / 1.79 / 1.42.
    int bps = h->peel_bps;
    if (bps <= 0 && h->blocks_per_sm <= 0 && !inst[0].member) bps = g.V <= 50000u ? 1 : g.V >= 3000000u ? 3 : 2;
    const FirstStep first{0, 0};
    if (int rc = run_persistent(h, fn, args, "peel", &hc, bps, &first)) return rc;
    return peel_status(hc, ninst, maxv);
}

int peel_kmax_row0(dc_graph* h, int32_t* kmax, int32_t* lmax) {
    int32_t mv[2] = {0, 0};
    PeelInst I[2] = {make_inst(h, 0, nullptr, 0, h->d.kmax_v, 0), make_inst(h, 1, nullptr, 0, h->scratch->row0, 1)};
    if (int rc = run_peel2(h, 2, I, mv)) return rc;
    *kmax = mv[0];
    *lmax = mv[1];
    return DC_OK;
}

// which: 0 = kmax pass (peel in-degree), 1 = row pass (peel out-degree)
int run_peel(dc_graph* h, int which, const int32_t* member, int32_t k, int32_t* d_val, int32_t* maxval, int sync) {
    (void)sync;
    PeelInst I = make_inst(h, which, member, k, d_val, 0);
    int32_t mv = 0;
    if (int rc = run_peel2(h, 1, &I, &mv)) return rc;
    if (maxval) *maxval = mv;
    return DC_OK;
}

// Skyline from row 0 and the corner log of the last run of rows (nlog
// entries, h->log_used of them records, the others void).
int build_skyline_from_log(dc_graph* h, uint64_t nlog) {
    Scratch* s = h->scratch;
    Decomp& d = h->d;
    uint32_t V = h->g.V;
    unsigned long long* cnt = (unsigned long long*)s->tmp64;
    const uint64_t total = (uint64_t)V + (nlog ? h->log_used : 0);
    ++g_launches;
    k_set_one<<<grid_for(h, V), kThreads, 0, h->stream>>>(V, cnt);
    if (nlog) {
        ++g_launches;
        k_sky_count<<<grid_for(h, nlog), kThreads, 0, h->stream>>>(V, nlog, s->log_v, s->log_k, cnt);
    }
    if (int rc = scan_tmp64(h, V)) return rc;
    if (d.corner_cap < total || !d.sky_k) {
        // a quarter of headroom: maintenance batches rarely grow it again
        dfree(h->stream, d.sky_k);
        dfree(h->stream, d.sky_l);
        d.corner_cap = 0;
        const uint64_t want = total + total / 4 + 1;
        if (dmalloc(h->stream, &d.sky_k, want) || dmalloc(h->stream, &d.sky_l, want)) {
            dfree(h->stream, d.sky_k);
            if (!free_groups(h) || dmalloc(h->stream, &d.sky_k, want) || dmalloc(h->stream, &d.sky_l, want)) return DC_ERR_NOMEM;
        }
        d.corner_cap = want;
    }
    if (!d.sky_off && dmalloc(h->stream, &d.sky_off, (uint64_t)V + 1)) return DC_ERR_NOMEM;
    ++g_launches;
    k_sky_fill_row0<<<grid_for(h, V), kThreads, 0, h->stream>>>(V, cnt, s->row0, d.sky_k, d.sky_l, s->cursor);
    if (nlog) {
        ++g_launches;
        k_sky_fill_log<<<grid_for(h, nlog), kThreads, 0, h->stream>>>(nlog, s->log_v, s->log_k, s->log_l, cnt, d.sky_k,
                                                                      d.sky_l, s->cursor);
    }
    ++g_launches;
    k_sky_sort<<<grid_for(h, V), kThreads, 0, h->stream>>>(V, cnt, d.sky_k, d.sky_l, d.sky_off);
    d.n_corners = total;
    DC_CUDA(cudaGetLastError());
    return DC_OK;
}

static int ensure_rows(dc_graph* h, uint64_t elems) {
    Decomp& d = h->d;
    if (d.rows_cap >= elems && d.rows) return DC_OK;
    dfree(h->stream, d.rows);
    d.rows_cap = 0;
    if (dmalloc(h->stream, &d.rows, elems) && !(free_groups(h) && dmalloc(h->stream, &d.rows, elems) == DC_OK))
        return DC_ERR_NOMEM;
    d.rows_cap = elems;
    return DC_OK;
}

int expand_rows(dc_graph* h, uint32_t k0, uint32_t n, int32_t* d_dst) {
    Decomp& d = h->d;
    if (!d.valid) return set_error(DC_ERR_STATE, "no decomposition on this graph");
    if (n == 0) return DC_OK;
    ++g_launches;
    if (h->g.V % 4 == 0 && ((uintptr_t)d_dst & 15u) == 0)
        k_expand4<<<grid_for(h, h->g.V / 4), kThreads, 0, h->stream>>>(h->g.V, k0, n, d.kmax_v, d.sky_off, d.sky_k,
                                                                         d.sky_l, d_dst);
    else
        k_expand<<<grid_for(h, h->g.V), kThreads, 0, h->stream>>>(h->g.V, k0, n, d.kmax_v, d.sky_off, d.sky_k,
                                                                   d.sky_l, d_dst);
    DC_CUDA(cudaGetLastError());
    return DC_OK;
}

// ---------------------------------------------------------------------------
// the graph relabeled in kmax order for the row kernel
// ---------------------------------------------------------------------------
// New id i = position of a vertex in kmax-descending order (s->order), so
// C_k = {new ids < |C_k|} is a prefix of the id space: the row kernel's scans
// of C_k read its state contiguously, and the dense core's state (the
// vertices of the heavy rows) packs into a small range that stays in the
// SMs' caches.  Lists hold new ids, ordered by neighbour kmax.
// Starts and lengths of both lists go along, and the lists too long for
// k_sort_short are listed for the other sorts (one atomic per warp and sort).
struct GatherSide {
    const uint32_t* off;
    const int32_t* len;
    uint32_t* start;
    int32_t* len_r;
    uint32_t* list[3];
};
__global__ void k_relabel_gather(uint32_t V, const uint32_t* order, const int32_t* kmax, const int32_t* row0,
                                 uint2* pos, int32_t* kmax_r, int32_t* row0_r, GatherSide out, GatherSide in,
                                 unsigned* cnt) {
    const unsigned lane = threadIdx.x & 31u;
    for (uint64_t b = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) & ~31ull; b < V;
         b += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = b + lane;
        int n[2] = {0, 0};
        if (i < V) {
            const uint32_t v = order[i];
            const int r0 = row0[v];
            pos[v] = make_uint2((uint32_t)i, (uint32_t)r0);
            kmax_r[i] = kmax[v];
            row0_r[i] = r0;
            out.start[i] = out.off[v];
            in.start[i] = in.off[v];
            out.len_r[i] = n[0] = out.len[v];
            in.len_r[i] = n[1] = in.len[v];
        }
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            const GatherSide& S = side == 0 ? out : in;
            const int to = n[side] > kSortMid ? 2 : n[side] > kSortWarp ? 1 : n[side] > kSortShort ? 0 : -1;
#pragma unroll
            for (int l = 0; l < 3; ++l) {
                const unsigned m = __ballot_sync(0xFFFFFFFFu, to == l);
                if (!m) continue;
                unsigned at = 0;
                if (lane == 0) at = atomicAdd(&cnt[3 * side + l], (unsigned)__popc(m));
                at = __shfl_sync(0xFFFFFFFFu, at, 0);
                if (to == l) S.list[l][at + __popc(m & ((1u << lane) - 1u))] = (uint32_t)i;
            }
        }
    }
}

// Corner records of the relabeled run back to original ids.  A run that
// jumped from row 0 to row k logs vertex v at row k whenever its value differs
// from row 0; where another run computed row k - 1 the corner is void when the
// value equals that row's (in the seam array).  *n: records in the log.
__global__ void k_log_finish(const unsigned* n, unsigned long long cap, const uint32_t* order, uint32_t* log_v,
                             int32_t* log_k, const int32_t* log_l, const uint32_t* seam_of, const int32_t* seam,
                             unsigned long long* voids) {
    const uint64_t m = min((unsigned long long)*n, cap);
    unsigned t = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x) {
        const int32_t k = log_k[i];
        if (k < 0) continue;
        const uint32_t v = log_v[i];
        const uint32_t at = seam_of ? seam_of[k] : 0u;
        if (at && log_l[i] == seam[at - 1u + v]) {
            log_k[i] = -1;
            ++t;
        } else {
            log_v[i] = order[v];
        }
    }
    t = __reduce_add_sync(0xFFFFFFFFu, t);
    if ((threadIdx.x & 31u) == 0 && t) atomicAdd(voids, (unsigned long long)t);
}

// Control blocks of the groups after the first (group 0's is the handle's own,
// initialised by its launch) and the plan's runs.
struct RowsStart {
    int n_groups;
    EngineCtl* ctl[kRowGroups];
    unsigned blocks[kRowGroups];
    unsigned long long span[kRowGroups];
    uint32_t seam_row[kRowGroups], seam_at[kRowGroups];  // first rows of the runs after the first, their seams
    unsigned seam_tail;
    unsigned long long wait_ns;
};
__global__ void k_rows_start(RowsStart r, RowPlan* plan, uint32_t* seam_of, uint32_t n_seam_of) {
    // one block: clear, then set
    for (uint32_t i = threadIdx.x; i < sizeof(RowPlan) / 4; i += blockDim.x) reinterpret_cast<uint32_t*>(plan)[i] = 0;
    for (uint32_t i = threadIdx.x; i < n_seam_of; i += blockDim.x) seam_of[i] = 0;
    for (int g = 1; g < r.n_groups; ++g)
        for (uint32_t i = threadIdx.x; i < sizeof(EngineCtl) / 4; i += blockDim.x)
            reinterpret_cast<uint32_t*>(r.ctl[g])[i] = 0;
    __syncthreads();
    if (threadIdx.x < (unsigned)r.n_groups) {
        const int g = threadIdx.x;
        plan->span[g].v = r.span[g];
        plan->own[g].lo = plan->own[g].prev = (int)(uint32_t)r.span[g];
        plan->own[g].members = r.blocks[g];
        plan->own[g].step_blocks = (1ull << 32) | r.blocks[g];
        plan->own[g].from = -1;
        plan->own[g].ready = g == 0;
        if (r.seam_row[g]) seam_of[r.seam_row[g]] = r.seam_at[g] + 1u;
        if (g) {
            EngineCtl* c = r.ctl[g];
            // a group with a run starts it, one without looks for one
            const int level = r.span[g] ? kRowsInit : kRowsWait;
            for (int i = 0; i < kStepWords; ++i) c->step_word[i].v = (1ull << 32) | (unsigned long long)(uint32_t)level;
            c->t_work = (unsigned long long)r.blocks[g] << kWorkShift;
            c->wait_ns = r.wait_ns;
        }
    }
    if (threadIdx.x == 0) plan->seam_tail = r.seam_tail;
}
// The groups' status and statistics into group 0's control block.
__global__ void k_rows_collect(RowsStart r, const RowPlan* plan) {
    EngineCtl* c0 = r.ctl[0];
    for (int g = 1; g < r.n_groups; ++g) {
        const EngineCtl* c = r.ctl[g];
        if (c->error && !c0->error) c0->err_where = c->err_where;
        c0->error |= c->error;
        c0->log_used += c->log_used;
        c0->evals += c->evals;
        c0->drops += c->drops;
        c0->edges_scanned += c->edges_scanned;
    }
    c0->log_count = plan->log_count;
    c0->pushes = plan->voids;
}

// Builds the relabeled graph (s->order must hold the kmax order of the
// current kmax) with its lists sorted by neighbour kmax, plus kmax and row 0
// by new id.
static int build_relabeled(dc_graph* h, int32_t K, uint32_t n0, unsigned* sort_cnt) {
    DevGraph& g = h->g;
    Scratch* s = h->scratch;
    const uint32_t V = g.V;
    const uint64_t n = (uint64_t)V + 1;
    if (s->r_cap_V < V || !s->pos) {
        dfree(h->stream, s->pos);
        dfree(h->stream, s->kmax_r);
        dfree(h->stream, s->row0_r);
        for (int i = 0; i < 2; ++i) {
            dfree(h->stream, s->r_off[i]);
            dfree(h->stream, s->r_len[i]);
        }
        s->r_cap_V = 0;
        if (dmalloc(h->stream, &s->pos, n) || dmalloc(h->stream, &s->kmax_r, n) || dmalloc(h->stream, &s->row0_r, n) ||
            dmalloc(h->stream, &s->r_off[0], n) || dmalloc(h->stream, &s->r_off[1], n) ||
            dmalloc(h->stream, &s->r_len[0], n) || dmalloc(h->stream, &s->r_len[1], n))
            return DC_ERR_NOMEM;
        s->r_cap_V = V;
    }
    const uint64_t cap = g.E + 1;
    if (s->r_cap < cap || !s->r_nbr[0]) {
        for (int i = 0; i < 2; ++i) {
            dfree(h->stream, s->r_nbr[i]);
        }
        s->r_cap = 0;
        const uint64_t want = cap + cap / 8;  // headroom for later, larger graphs of the handle
        for (int i = 0; i < 2; ++i) {
            if (dmalloc(h->stream, &s->r_nbr[i], want)) return DC_ERR_NOMEM;
        }
        s->r_cap = want;
    }
    uint32_t* start = (uint32_t*)s->tmp64;  // of every list in the handle's, out then in
    SortArgs so;
    so.side[0] = SortSide{s->r_off[0], s->r_len[0], s->r_nbr[0], g.out_nbr, start, {s->rem0, s->rem2, s->rem1}, s->cnt_out};
    so.side[1] = SortSide{s->r_off[1], s->r_len[1], s->r_nbr[1], g.in_nbr, start + n,
                          {s->rem3, (uint32_t*)s->cdeg, (uint32_t*)s->cdeg2}, s->key};
    so.cnt = sort_cnt;
    so.pos = s->pos;
    so.kmax = s->kmax_r;
    so.row0 = s->row0_r;
    so.n0 = n0;
    so.K = K;
    GatherSide gs[2];
    for (int side = 0; side < 2; ++side) {
        gs[side] = GatherSide{side == 0 ? g.out_off : g.in_off, side == 0 ? g.out_len : g.in_len, start + side * n,
                              s->r_len[side], {}};
        for (int l = 0; l < 3; ++l) gs[side].list[l] = so.side[side].list[l];
    }
    ++g_launches;
    k_relabel_gather<<<grid_for(h, V), kThreads, 0, h->stream>>>(V, s->order, h->d.kmax_v, s->row0, s->pos, s->kmax_r,
                                                                  s->row0_r, gs[0], gs[1], sort_cnt);
    const ListStarts ls{{s->r_len[0], s->r_len[1]}, {s->r_off[0], s->r_off[1]}, 0, 0};
    scan_sums(h, ls, 2, V);
    scan_apply(h, ls, 2, V);
    // every relabeled list is read from its original list, renamed and
    // sorted in one pass; most lists go to the short and the warp sort, the
    // others read their counts on the device
    // The counting sort has a few long lists, one block each; on a graph where
    // that takes a while the others run beside it (preparation of R-MAT 22
    // 3.06 -> 2.64 ms, R-MAT 20 0.76 -> 0.67; the fork and the join cost about
    // 15 us, a handle's first one the stream as well).
    const bool beside = g.E >= (8ull << 20);
    if (beside) {
        if (!h->side_stream) DC_CUDA(cudaStreamCreateWithFlags(&h->side_stream, cudaStreamNonBlocking));
        for (auto& e : h->side_ev)
            if (!e) DC_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        DC_CUDA(cudaEventRecord(h->side_ev[0], h->stream));
        DC_CUDA(cudaStreamWaitEvent(h->side_stream, h->side_ev[0], 0));
    }
    g_launches += 4;
    k_sort_big<<<dim3(h->geom.sms, 2), 1024, 0, beside ? h->side_stream : h->stream>>>(so);
    k_sort_short<<<dim3(grid_for(h, 8ull * V), 2), kThreads, 0, h->stream>>>(V, so);
    k_sort_warp<<<dim3(h->geom.sms * 8, 2), kSortThreads, 0, h->stream>>>(so);
    k_sort_mid<<<dim3(h->geom.sms * 8, 2), kSortThreads, 0, h->stream>>>(so);
    if (beside) {
        DC_CUDA(cudaEventRecord(h->side_ev[1], h->side_stream));
        DC_CUDA(cudaStreamWaitEvent(h->stream, h->side_ev[1], 0));
    }
    DC_CUDA(cudaGetLastError());
    return DC_OK;
}

// Rows 1..Kstop from row 0 (scratch row0) and kmax (d.kmax_v): orders
// vertices by kmax, initialises the support counters and runs the
// row-to-row kernel.  Corners of rows 1..Kstop are left in the scratch log
// (*nlog entries).  allow_sort: order adjacency lists by neighbour kmax
// first (otherwise lists are read whole).
// cut: the engine may cut the rows by itself.
static int rows_run(dc_graph* h, int32_t K, int32_t Kstop, bool allow_sort, uint64_t* nlog_out, int32_t K0, bool cut) {
    DevGraph& g = h->g;
    Decomp& d = h->d;
    Scratch* s = h->scratch;
    const uint32_t V = g.V;
    *nlog_out = 0;
    h->log_used = 0;
    cudaEventRecord(h->ev[2], h->stream);
    // |C_k| and first positions by kmax (K + 2 words each, sized by kmax: it
    // exceeds V where edges are parallel), two sums, the sorts' counters
    const uint64_t nk = (uint64_t)K + 2;
    if (s->ck_cap < nk) {
        dfree(h->stream, s->ck);
        s->ck_cap = 0;
        if (dmalloc(h->stream, &s->ck, 2 * nk + kRowPrepWords)) return DC_ERR_NOMEM;
        s->ck_cap = (uint32_t)nk;
    }
    unsigned long long* sums = (unsigned long long*)s->ck;  // corners, row work
    unsigned* sort_cnt = s->ck + 4;
    uint32_t* d_ck = s->ck + kRowPrepWords;
    uint32_t* hist = d_ck + nk;
    static_assert(kRowPrepWords >= 4 + 6, "two sums, six counters");
    DC_CUDA(cudaMemsetAsync(s->ck, 0, sizeof(uint32_t) * (2 * nk + kRowPrepWords), h->stream));
    ++g_launches;
    k_row_stats<<<grid_for(h, V), kThreads, K + 1 <= kHistShared ? 4 * (K + 1) : 0, h->stream>>>(
        V, d.kmax_v, s->row0, g.in_len, g.out_len, hist, K, sums, sums + 1);
    std::vector<uint32_t> host(2 * nk + kRowPrepWords);
    DC_CUDA(cudaMemcpyAsync(host.data(), s->ck, sizeof(uint32_t) * host.size(), cudaMemcpyDeviceToHost, h->stream));
    DC_CUDA(cudaStreamSynchronize(h->stream));
    unsigned long long bound = 0;
    memcpy(&bound, host.data(), sizeof(bound));
    memcpy(&h->row_work, host.data() + 2, sizeof(h->row_work));
    uint32_t* ck = host.data() + kRowPrepWords;
    {
        uint32_t* start = ck + nk;  // counts, then first positions
        uint32_t run = 0;
        ck[K + 1] = 0;
        for (int32_t k = K; k >= 0; --k) {
            const uint32_t c = start[k];
            start[k] = run;
            run += c;
            ck[k] = run;
        }
    }
    DC_CUDA(cudaMemcpyAsync(d_ck, ck, sizeof(uint32_t) * 2 * nk, cudaMemcpyHostToDevice, h->stream));
    ++g_launches;
    k_order_scatter<<<grid_for(h, ((uint64_t)V + kOrderItems - 1) / kOrderItems), kThreads, 0, h->stream>>>(
        V, d.kmax_v, K, hist, s->order);
    // The graph the row kernel reads: where sorting is allowed, the graph
    // relabeled in kmax order with kmax-sorted lists (C_k a prefix of the
    // ids); else the handle's own lists (kmax-sorted when they still are from
    // an earlier run) with C_k listed by `order`.
    const bool relabel = allow_sort && K + 1 <= kSortBigBins;
    // A run from row 1 on the relabeled graph (a full decomposition, or rows
    // 1..R of a maintenance batch) may be cut in runs of rows that groups of
    // blocks work on at the same time: group 0 starts at row 1, a run starting
    // at row a starts from row 0 inside C_a, with state for the ids below
    // |C_a|.  Groups whose run is over take over rows of others (RowsNext).
    const int32_t k0 = std::max(1, K0);
    int32_t first_row[kRowGroups] = {k0};  // of each run, ascending
    int nrun = 1, ngroups = 1;
    int32_t run_min = Kstop + 1;
    int first_share = 1;   // blocks of the first run, in shares of the others'
    uint32_t n_state = 0;  // vertices every group after the first has state for
    if (relabel && k0 == 1 && Kstop >= kMinSplitRows && (cut || !h->auto_cuts)) {
        if (h->auto_cuts) {
            // A handle whose launch shapes were never set is cut where the
            // core a run starts from is small: a start costs a pass over its
            // core's lists and a refinement from row 0 there.  With skewed
            // degrees (|C_k| a few per cent of |C_1| after a tenth of the
            // rows) they take the rows from 3.0 / 9.7 / 14.4 / 35 ms to 0.7 /
            // 2.3 / 5.2 / 19 (ragged R-MAT 17, R-MAT 18 / 20 / 22); where every
            // vertex is in almost every core (ER, 100 edges per vertex) fixed
            // cuts took them from 3.6 to 11.0 ms.
            // Hence an eighth of |C_1| at most (a quarter up to 65,536
            // vertices), which also bounds the groups' state, and no cut
            // where that leaves more than half of the rows to the first run.
            n_state = std::max(ck[1] / 8, std::min(ck[1] / 4, 65536u));
            run_min = 2;
            while (run_min <= Kstop && ck[run_min] > n_state) ++run_min;
            // Small graphs: eight groups hide each other's latency best, equal
            // runs (8 / 6 / 5 / 4 groups: R-MAT 18, 3.9 M edges 2.1 / 2.5 /
            // 2.7 / 3.0 ms).  From 8 M edges on the rows want more warps each
            // and the cores are large for longer: five groups, first rows at
            // 0.6, 0.3, 0.15 and 0.075 of the rows, which took the rows of
            // nine R-MAT graphs of 2^19 to 2^22 vertices from 6.5 / 11.1 /
            // 21.4 ms (five or six equal runs, 16 / 32 / 64 M edges) to 5.9 /
            // 10.0 / 18.6, between 17 % less and 3 % more.
            first_share = g.E < (8ull << 20) ? 2 : 1;
            if (2 * (run_min - 1) <= Kstop) {
                const int32_t rows = Kstop - run_min + 1, runs = std::min<int32_t>(kRowGroups - 1, rows / 2);
                if (first_share == 2) {
                    for (int32_t i = 0; i < runs; ++i) first_row[nrun++] = run_min + (int32_t)((int64_t)rows * i / runs);
                } else {
                    for (int64_t f : {75, 150, 300, 600}) {
                        const int32_t c = (int32_t)(Kstop * f / 1000);
                        if (c >= run_min && c > first_row[nrun - 1]) first_row[nrun++] = c;
                    }
                    if (nrun == 1) first_row[nrun++] = run_min;
                    run_min = first_row[1];
                }
                n_state = ck[run_min];
                ngroups = nrun == 1 ? 1 : first_share == 2 ? kRowGroups : 5;
            }
        } else {
            for (int i = 0; i < kMaxRowSegments - 1 && nrun < kRowGroups; ++i) {
                const int32_t c = (int32_t)((int64_t)K * h->rows_split[i] / 1000);
                if (c >= 1 && c < Kstop && c + 1 > first_row[nrun - 1]) first_row[nrun++] = c + 1;
            }
            if (nrun > 1) {
                run_min = first_row[1];
                n_state = ck[run_min];
                ngroups = nrun;
            }
        }
    }
    // blocks: what fits at the same time
    const void* rows_fn = ngroups > 1 ? (const void*)k_trans2<true> : (const void*)k_trans2<false>;
    int grid = 0;
    // (engine's cuts, 1 / 2 / 3 blocks per SM: 53,000 edges 0.39 / 0.42 / 0.45
    // ms, 228,000 0.55 / 0.53 / 0.56, 518,000 0.93 / 0.99 / 1.03, 0.96 M 1.10 /
    // 1.00 / 1.01, 1.9 M 1.67 / 1.44 / 1.38, 3.9 M 3.2 / 2.4 / 2.3)
    const int most_bps = !h->auto_cuts ? 8
                         : h->blocks_per_sm > 0 ? h->blocks_per_sm  // dc_set_launch bounds the launch
                         : g.E < 300000u ? 1 : g.E < 1500000u ? 2 : 8;
    if (int rc = persistent_grid(h, rows_fn, ngroups > 1 ? most_bps : h->rows_bps, &grid)) return rc;
    // (cuts of the caller's: blocks per SM for every run, as for separate launches)
    const int run_bps = h->rows_bps > 0 ? h->rows_bps : h->blocks_per_sm;
    if (ngroups > 1 && !h->auto_cuts && run_bps > 0) grid = std::min(grid, run_bps * ngroups * h->geom.sms);
    const uint64_t spare = (uint64_t)kLogChunk * kWarpsPerBlock * grid;  // records left over in the warps' chunks
    // seams: the values of row a - 1 in C_a for every run that starts at a,
    // with room for rows taken over (a void record each at most)
    uint64_t seam_cap = 0;
    for (int i = 1; i < nrun; ++i) seam_cap += ck[first_row[i]];
    if (nrun > 1) seam_cap = std::min<uint64_t>(seam_cap + 8ull * n_state, 0xFFFFFFF0ull);
    const uint64_t lc = bound + 1 + spare + seam_cap;
    if (s->log_cap < lc) {
        // a quarter of headroom: later runs (maintenance batches) rarely grow it again
        const uint64_t cap = lc + lc / 4;
        dfree(h->stream, s->log_v);
        dfree(h->stream, s->log_k);
        dfree(h->stream, s->log_l);
        s->log_cap = 0;
        if (dmalloc(h->stream, &s->log_v, cap) || dmalloc(h->stream, &s->log_k, cap) || dmalloc(h->stream, &s->log_l, cap)) return DC_ERR_NOMEM;
        s->log_cap = cap;
    }
    const uint32_t n0 = relabel ? ck[std::min(k0, K + 1)] : V;
    int sorted = 0;
    const uint32_t *G_out_off = g.out_off, *G_in_off = g.in_off, *G_order = s->order;
    int32_t *G_out_len = g.out_len, *G_in_len = g.in_len;
    uint32_t *G_out_nbr = g.out_nbr, *G_in_nbr = g.in_nbr;
    const int32_t *G_kmax = d.kmax_v, *G_row0 = s->row0;
    if (relabel) {
        if (int rc = build_relabeled(h, K, n0, sort_cnt)) return rc;
        sorted = 1;
        G_out_off = s->r_off[0];
        G_in_off = s->r_off[1];
        G_out_len = s->r_len[0];
        G_in_len = s->r_len[1];
        G_out_nbr = s->r_nbr[0];
        G_in_nbr = s->r_nbr[1];
        G_kmax = s->kmax_r;
        G_row0 = s->row0_r;
        G_order = nullptr;
    }
    // starting values and counters of the first run: row 0 inside C_k0 with
    // the vertices outside already left (for k0 = 1 those of kmax 0), so its
    // first step has no leaving pass; the marks of all V vertices, because the
    // local core update expects them clear
    if (int rc = ensure_tring(h, 2ull * V + (uint64_t)h->geom.sms * 64 + 4096)) return rc;
    Trans2Params tp;
    memset(&tp, 0, sizeof(tp));
    tp.out_off = G_out_off; tp.out_len = G_out_len; tp.out_nbr = G_out_nbr;
    tp.in_off = G_in_off; tp.in_len = G_in_len; tp.in_nbr = G_in_nbr;
    tp.kmax = G_kmax;
    tp.row0 = G_row0;
    tp.K = K;
    tp.K0 = k0;
    tp.Kstop = Kstop;
    tp.n = n0;
    tp.sorted = sorted;
    tp.order = G_order;
    tp.ck = d_ck;
    tp.log_v = s->log_v;
    tp.log_k = s->log_k;
    tp.log_l = s->log_l;
    tp.log_cap = s->log_cap;
    tp.n_groups = ngroups;
    tp.g[0] = RowGroup{s->cur, s->cnt_out, s->key, s->mark, s->stamp, s->logidx,
                       TicketQueue{s->tring, (unsigned)(s->tring_cap - 1)}, h->ctl};
    DC_CUDA(cudaMemsetAsync(s->mark, 0, sizeof(uint32_t) * V, h->stream));
    if (n0) {
        if (relabel) {
            DC_CUDA(cudaMemcpyAsync(s->cur, G_row0, 4ull * n0, cudaMemcpyDeviceToDevice, h->stream));
        } else {
            g_launches += 2;
            k_preleft_cur<<<grid_for(h, n0), kThreads, 0, h->stream>>>(n0, G_kmax, G_row0, k0, s->cur);
            k_counters_init<<<grid_for(h, (uint64_t)n0 * 32), kThreads, 0, h->stream>>>(tp);
        }
        DC_CUDA(cudaMemsetAsync(s->stamp, 0xFF, sizeof(int32_t) * n0, h->stream));
    }
    RowsStart rs;
    memset(&rs, 0, sizeof(rs));
    if (ngroups > 1) {
        const int shares = ngroups + first_share - 1;
        tp.first_block[0] = 0;
        for (int i = 0; i < ngroups; ++i)
            tp.first_block[i + 1] = (unsigned)((int64_t)grid * (i + first_share) / shares);
        for (int i = 1; i < ngroups; ++i) {
            if (int rc = ensure_segment(h, i - 1, n_state)) return rc;
            const RowSegment& sg = s->seg[i - 1];
            tp.g[i] = RowGroup{sg.cur, sg.cnt_out, sg.cnt_in, sg.mark, sg.stamp, sg.logidx,
                               TicketQueue{sg.tring, (unsigned)(sg.tring_cap - 1)}, sg.ctl};
        }
        if (!s->plan && dmalloc(h->stream, &s->plan, 1)) return DC_ERR_NOMEM;
        if (s->seam_of_cap < (uint32_t)K + 2 || !s->seam_of) {
            dfree(h->stream, s->seam_of);
            s->seam_of_cap = 0;
            if (dmalloc(h->stream, &s->seam_of, (uint64_t)K + 2)) return DC_ERR_NOMEM;
            s->seam_of_cap = (uint32_t)K + 2;
        }
        if (s->seam_cap < seam_cap || !s->seam) {
            dfree(h->stream, s->seam);
            s->seam_cap = 0;
            const uint64_t want = seam_cap + seam_cap / 8;
            if (dmalloc(h->stream, &s->seam, want)) return DC_ERR_NOMEM;
            s->seam_cap = want;
        }
        tp.plan = s->plan;
        tp.run_min = run_min;
        tp.seam_of = s->seam_of;
        tp.seam = s->seam;
        tp.seam_cap = (unsigned)seam_cap;
        rs.n_groups = ngroups;
        rs.wait_ns = h->wait_ns;
        for (int i = 0; i < ngroups; ++i) {
            rs.ctl[i] = tp.g[i].ctl;
            rs.blocks[i] = tp.first_block[i + 1] - tp.first_block[i];
            if (i >= nrun) continue;
            const int32_t last = i + 1 < nrun ? first_row[i + 1] - 1 : Kstop;
            rs.span[i] = ((unsigned long long)last << 32) | (unsigned long long)first_row[i];
            if (i) {
                rs.seam_row[i] = (uint32_t)first_row[i];
                rs.seam_at[i] = rs.seam_tail;
                rs.seam_tail += ck[first_row[i]];
            }
        }
        ++g_launches;
        k_rows_start<<<1, 512, 0, h->stream>>>(rs, s->plan, s->seam_of, (uint32_t)K + 2);
    } else {
        tp.first_block[1] = (unsigned)grid;
    }
    uint64_t nlog = 0;
    cudaEventRecord(h->ev[3], h->stream);
    if (Kstop >= k0) {
        void* args[] = {&tp};
        const FirstStep first{k0, (int)(tp.first_block[1] - tp.first_block[0])};
        if (int rc = persistent_launch(h, rows_fn, args, "transitions", h->ctl, h->stream, 0, &first, grid))
            return rc;
        if (ngroups > 1) {
            ++g_launches;
            k_rows_collect<<<1, 1, 0, h->stream>>>(rs, s->plan);
        }
        if (relabel) {
            ++g_launches;
            k_log_finish<<<grid_for(h, lc / 4), kThreads, 0, h->stream>>>(
                &h->ctl->log_count, s->log_cap, s->order, s->log_v, s->log_k, s->log_l,
                ngroups > 1 ? s->seam_of : nullptr, s->seam, &h->ctl->pushes);
        }
        EngineCtl hc;
        const int rc = finish_persistent(h, h->ctl, h->stream, "transitions", &hc);
        if (rc != DC_OK) {
            for (RowSegment& sg : s->seg)
                if (sg.tring) cudaMemsetAsync(sg.tring, 0xFF, sizeof(unsigned long long) * sg.tring_cap, h->stream);
            cudaStreamSynchronize(h->stream);
            return rc;
        }
        nlog = hc.log_count;
        h->log_used = hc.log_used - hc.pushes;
        h->stat_evals = hc.evals;
        h->stat_drops = hc.drops;
        h->stat_entries = hc.edges_scanned;
    }
    cudaEventRecord(h->ev[4], h->stream);
    *nlog_out = nlog;
    return DC_OK;
}

int rows_from_row0(dc_graph* h, int32_t K, int32_t Kstop, bool allow_sort, uint64_t* nlog_out, int32_t K0) {
    const int rc = rows_run(h, K, Kstop, allow_sort, nlog_out, K0, true);
    // cuts of the engine's own choice are not worth a refusal: one run needs
    // no groups (all memory is taken before the kernel starts)
    if (rc != DC_ERR_NOMEM || !h->auto_cuts || !free_groups(h)) return rc;
    return rows_run(h, K, Kstop, allow_sort, nlog_out, K0, false);
}

int decompose(dc_graph* h, int method, int materialize_rows) {
    DevGraph& g = h->g;
    Decomp& d = h->d;
    const uint32_t V = g.V;
    d.valid = false;
    d.rows_valid = false;
    if (int rc = ensure_scratch(h, V)) return rc;
    Scratch* s = h->scratch;
    if (!d.kmax_v && dmalloc(h->stream, &d.kmax_v, (uint64_t)V + 1)) return DC_ERR_NOMEM;
    d.peel_valid = false;
    if (V == 0) {
        d.kmax = 0;
        d.lmax = 0;
        d.n_corners = 0;
        if (!d.sky_off && dmalloc(h->stream, &d.sky_off, 1)) return DC_ERR_NOMEM;
        DC_CUDA(cudaMemsetAsync(d.sky_off, 0, sizeof(uint32_t), h->stream));
        d.row_lo = 1;
        d.row_hi = 0;
        d.peel_valid = true;
        d.valid = true;
        return DC_OK;
    }
    cudaEventRecord(h->ev[0], h->stream);
    // kmax (in-degree peel) and row 0 (out-degree peel) in one grid
    int32_t mv[2] = {0, 0};
    {
        PeelInst I[2] = {make_inst(h, 0, nullptr, 0, d.kmax_v, 0), make_inst(h, 1, nullptr, 0, s->row0, 1)};
        if (int rc = run_peel2(h, 2, I, mv)) return rc;
    }
    cudaEventRecord(h->ev[1], h->stream);
    const int32_t K = mv[0];
    d.kmax = K;
    d.lmax = mv[1];
    if (!d.row0 && dmalloc(h->stream, &d.row0, (uint64_t)V + 1)) return DC_ERR_NOMEM;
    DC_CUDA(cudaMemcpyAsync(d.row0, s->row0, 4ull * V, cudaMemcpyDeviceToDevice, h->stream));
    d.peel_valid = true;
    d.row_lo = 1;
    d.row_hi = K;
    if (method == 1) {
        // one fresh peel per row (the reference's schedule, main.cu:238-244),
        // two rows per launch
        if (int rc = ensure_rows(h, (uint64_t)(K + 1) * V)) return rc;
        DC_CUDA(cudaMemcpyAsync(d.rows, s->row0, 4ull * V, cudaMemcpyDeviceToDevice, h->stream));
        for (int32_t k = 1; k <= K; k += 2) {
            int n = (k + 1 <= K) ? 2 : 1;
            PeelInst I[2] = {make_inst(h, 1, d.kmax_v, k, d.rows + (uint64_t)k * V, 0),
                             make_inst(h, 1, d.kmax_v, k + 1, d.rows + (uint64_t)(k + 1) * V, 1)};
            int32_t m2[2];
            if (int rc = run_peel2(h, n, I, m2)) return rc;
        }
        cudaEventRecord(h->ev[2], h->stream);
        cudaEventRecord(h->ev[3], h->stream);
        unsigned long long* cnt = (unsigned long long*)s->tmp64;
        ++g_launches;
        k_rows_corner_count<<<grid_for(h, V), kThreads, 0, h->stream>>>(V, K, d.kmax_v, d.rows, cnt);
        if (int rc = scan_tmp64(h, V)) return rc;
        unsigned long long total = 0;
        DC_CUDA(cudaMemcpyAsync(&total, s->tmp64 + V, sizeof(total), cudaMemcpyDeviceToHost, h->stream));
        DC_CUDA(cudaStreamSynchronize(h->stream));
        if (d.corner_cap < total) {
            dfree(h->stream, d.sky_k);
            dfree(h->stream, d.sky_l);
            if (dmalloc(h->stream, &d.sky_k, total) || dmalloc(h->stream, &d.sky_l, total)) return DC_ERR_NOMEM;
            d.corner_cap = total;
        }
        if (!d.sky_off && dmalloc(h->stream, &d.sky_off, (uint64_t)V + 1)) return DC_ERR_NOMEM;
        ++g_launches;
        k_rows_corner_fill<<<grid_for(h, V), kThreads, 0, h->stream>>>(V, d.kmax_v, d.rows, cnt, d.sky_k, d.sky_l,
                                                                        d.sky_off);
        d.n_corners = total;
        d.rows_valid = true;
        if (int rc = degree_kmax_sum(h, &h->full_work)) return rc;
        cudaEventRecord(h->ev[4], h->stream);
        cudaEventRecord(h->ev[5], h->stream);
        cudaEventRecord(h->ev[6], h->stream);
        DC_CUDA(cudaStreamSynchronize(h->stream));
        d.valid = true;
        float ms = 0;
        cudaEventElapsedTime(&ms, h->ev[0], h->ev[1]);
        h->times.kmax_ms = ms;
        h->times.row0_ms = 0;
        cudaEventElapsedTime(&ms, h->ev[1], h->ev[2]);
        h->times.trans_ms = ms;
        h->full_rows_ms = ms;
        cudaEventElapsedTime(&ms, h->ev[3], h->ev[4]);
        h->times.sky_ms = ms;
        h->times.expand_ms = 0;
        return DC_OK;
    }
    // ---- method 0: rows 1..K derived row to row
    uint64_t nlog = 0;
    if (int rc = rows_from_row0(h, K, K, true, &nlog)) return rc;
    h->full_work = h->row_work;
    if (int rc = build_skyline_from_log(h, nlog)) return rc;
    cudaEventRecord(h->ev[5], h->stream);
    d.valid = true;
    if (materialize_rows) {
        if (int rc = ensure_rows(h, (uint64_t)(K + 1) * V)) return rc;
        if (int rc = expand_rows(h, 0, (uint32_t)K + 1, d.rows)) return rc;
        d.rows_valid = true;
    }
    cudaEventRecord(h->ev[6], h->stream);
    DC_CUDA(cudaStreamSynchronize(h->stream));
    float ms = 0;
    cudaEventElapsedTime(&ms, h->ev[0], h->ev[1]);
    h->times.kmax_ms = ms;
    cudaEventElapsedTime(&ms, h->ev[1], h->ev[3]);
    h->times.row0_ms = ms;
    cudaEventElapsedTime(&ms, h->ev[3], h->ev[4]);
    h->times.trans_ms = ms;
    h->full_rows_ms = ms;
    cudaEventElapsedTime(&ms, h->ev[4], h->ev[5]);
    h->times.sky_ms = ms;
    cudaEventElapsedTime(&ms, h->ev[5], h->ev[6]);
    h->times.expand_ms = ms;
    return DC_OK;
}

int row_weights(dc_graph* h, uint64_t* out) {
    const DevGraph& g = h->g;
    const Decomp& d = h->d;
    const int32_t K = d.kmax;
    unsigned long long* w = nullptr;
    if (dmalloc(h->stream, &w, (uint64_t)K + 1)) return DC_ERR_NOMEM;
    DC_CUDA(cudaMemsetAsync(w, 0, 8ull * (K + 1), h->stream));
    if (g.V) {
        ++g_launches;
        size_t shm = K + 1 <= 4096 ? 8ull * (K + 1) : 0;
        k_kmax_degree_hist<<<grid_for(h, g.V), kThreads, shm, h->stream>>>(g.V, d.kmax_v, g.in_len, g.out_len, K, w);
    }
    std::vector<uint64_t> hw((size_t)K + 1);
    DC_CUDA(cudaMemcpyAsync(hw.data(), w, 8ull * (K + 1), cudaMemcpyDeviceToHost, h->stream));
    dfree(h->stream, w);
    DC_CUDA(cudaStreamSynchronize(h->stream));
    uint64_t run = 0;
    for (int32_t k = K; k >= 0; --k) {
        run += hw[k];
        out[k] = run;
    }
    return DC_OK;
}

// the row work alone (k_row_stats)
__global__ void k_deg_kmax_sum(uint32_t V, const int32_t* kmax, const int32_t* in_len, const int32_t* out_len,
                               unsigned long long* acc) {
    unsigned long long w = 0;
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V; v += (uint64_t)gridDim.x * blockDim.x)
        w += (unsigned long long)(in_len[v] + out_len[v]) * (unsigned long long)max(kmax[v], 0);
#pragma unroll
    for (int s = 16; s; s >>= 1) w += __shfl_xor_sync(0xFFFFFFFFu, w, s);
    if ((threadIdx.x & 31u) == 0) atomicAdd(acc, w);
}

int degree_kmax_sum(dc_graph* h, uint64_t* out) {
    unsigned long long* acc = (unsigned long long*)h->scratch->tmp64;
    DC_CUDA(cudaMemsetAsync(acc, 0, sizeof(unsigned long long), h->stream));
    ++g_launches;
    k_deg_kmax_sum<<<grid_for(h, h->g.V), kThreads, 0, h->stream>>>(h->g.V, h->d.kmax_v, h->g.in_len, h->g.out_len,
                                                                     acc);
    unsigned long long w = 0;
    DC_CUDA(cudaMemcpyAsync(&w, acc, sizeof(w), cudaMemcpyDeviceToHost, h->stream));
    DC_CUDA(cudaStreamSynchronize(h->stream));
    *out = w;
    return DC_OK;
}

int decompose_range(dc_graph* h, int32_t k_first, int32_t k_last) {
    DevGraph& g = h->g;
    Decomp& d = h->d;
    const uint32_t V = g.V;
    if (k_first <= 0 || !d.peel_valid || !d.kmax_v || !d.row0) {
        // kmax and row 0 (fused peel)
        if (int rc = ensure_scratch(h, V)) return rc;
        Scratch* s = h->scratch;
        if (!d.kmax_v && dmalloc(h->stream, &d.kmax_v, (uint64_t)V + 1)) return DC_ERR_NOMEM;
        if (V == 0) return decompose(h, 0, 0);
        d.valid = false;
        d.rows_valid = false;
        cudaEventRecord(h->ev[0], h->stream);
        int32_t mv[2] = {0, 0};
        PeelInst I[2] = {make_inst(h, 0, nullptr, 0, d.kmax_v, 0), make_inst(h, 1, nullptr, 0, s->row0, 1)};
        if (int rc = run_peel2(h, 2, I, mv)) return rc;
        cudaEventRecord(h->ev[1], h->stream);
        d.kmax = mv[0];
        d.lmax = mv[1];
        if (!d.row0 && dmalloc(h->stream, &d.row0, (uint64_t)V + 1)) return DC_ERR_NOMEM;
        DC_CUDA(cudaMemcpyAsync(d.row0, s->row0, 4ull * V, cudaMemcpyDeviceToDevice, h->stream));
        DC_CUDA(cudaStreamSynchronize(h->stream));
        float ms = 0;
        cudaEventElapsedTime(&ms, h->ev[0], h->ev[1]);
        h->times.kmax_ms = ms;
        d.peel_valid = true;
    } else {
        h->times.kmax_ms = 0;
    }
    if (int rc = ensure_scratch(h, V)) return rc;
    Scratch* s = h->scratch;
    const int32_t K = d.kmax;
    const int32_t k0 = std::max(1, k_first), k1 = std::min(k_last, K);
    d.rows_valid = false;
    // the row kernel starts from row 0 in scratch
    DC_CUDA(cudaMemcpyAsync(s->row0, d.row0, 4ull * V, cudaMemcpyDeviceToDevice, h->stream));
    uint64_t nlog = 0;
    if (int rc = rows_from_row0(h, K, k1, true, &nlog, k0)) return rc;
    if (int rc = build_skyline_from_log(h, nlog)) return rc;
    cudaEventRecord(h->ev[5], h->stream);
    DC_CUDA(cudaStreamSynchronize(h->stream));
    float ms = 0;
    cudaEventElapsedTime(&ms, h->ev[3], h->ev[4]);
    h->times.trans_ms = ms;
    cudaEventElapsedTime(&ms, h->ev[4], h->ev[5]);
    h->times.sky_ms = ms;
    h->times.row0_ms = 0;
    h->times.expand_ms = 0;
    d.row_lo = k0;
    d.row_hi = k1;
    d.valid = true;
    return DC_OK;
}


}  // namespace dc
