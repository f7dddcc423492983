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
// persistent cooperative kernel per pass (software grid barrier per level, a
// device work queue for cascades, no host round trip per level), and rows
// k >= 1 derived from row k-1 by h-index refinement instead of one fresh
// peel per row (see k_transitions).
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
    __shared__ unsigned long long s_w[32];
    const unsigned lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    unsigned long long inc = warp_incl_scan64(x);
    if (lane == 31) s_w[w] = inc;
    __syncthreads();
    if (w == 0) {
        unsigned nw = blockDim.x >> 5;
        unsigned long long v = lane < nw ? s_w[lane] : 0ull;
        unsigned long long vi = warp_incl_scan64(v);
        if (lane < nw) s_w[lane] = vi - v;
        if (lane == nw - 1) s_w[31] = vi;
    }
    __syncthreads();
    unsigned long long res = inc - x + s_w[w];
    *total = s_w[31];
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
// cooperative exclusive scan (u64), n elements in place; out[n] = total
// ---------------------------------------------------------------------------
__global__ void k_scan_coop(unsigned long long* data, uint64_t n, unsigned long long* partial, EngineCtl* c) {
    const uint64_t nb = gridDim.x;
    const uint64_t per = (n + nb - 1) / nb;
    const uint64_t lo = min(n, per * blockIdx.x), hi = min(n, lo + per);
    // phase 1: block sums
    unsigned long long s = 0;
    for (uint64_t i = lo + threadIdx.x; i < hi; i += blockDim.x) s += data[i];
    unsigned long long tot;
    block_excl_scan64(s, &tot);
    if (threadIdx.x == 0) partial[blockIdx.x] = tot;
    if (!grid_sync(c)) return;
    // phase 2: block 0 scans the partials
    if (blockIdx.x == 0) {
        unsigned long long carry = 0;
        for (uint64_t b0 = 0; b0 < nb; b0 += blockDim.x) {
            uint64_t b = b0 + threadIdx.x;
            unsigned long long v = b < nb ? partial[b] : 0ull;
            unsigned long long t2;
            unsigned long long ex = block_excl_scan64(v, &t2);
            if (b < nb) partial[b] = ex + carry;
            carry += t2;
            __syncthreads();
        }
        if (threadIdx.x == 0) data[n] = carry;
    }
    if (!grid_sync(c)) return;
    // phase 3: scan own range
    unsigned long long carry = partial[blockIdx.x];
    for (uint64_t b0 = lo; b0 < hi; b0 += blockDim.x) {
        uint64_t i = b0 + threadIdx.x;
        unsigned long long v = i < hi ? data[i] : 0ull;
        unsigned long long t2;
        unsigned long long ex = block_excl_scan64(v, &t2);
        if (i < hi) data[i] = ex + carry;
        carry += t2;
    }
}

// ---------------------------------------------------------------------------
// graph build
// ---------------------------------------------------------------------------
__global__ void k_count_degrees(uint32_t V, uint64_t E, const uint32_t* src, const uint32_t* dst, int32_t* out_len,
                                int32_t* in_len, EngineCtl* c) {
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < E; e += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t s = src[e], d = dst[e];
        if (s >= V || d >= V) {
            set_dev_error(c, DC_DEV_ERR_BADID, 10);
            continue;
        }
        atomicAdd(&out_len[s], 1);
        atomicAdd(&in_len[d], 1);
    }
}

// capacity of v's list = len + max(gap_min, len / gap_div)
__global__ void k_capacity(uint32_t V, const int32_t* len, uint32_t gap_min, uint32_t gap_div, unsigned long long* cap) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V; v += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t l = (uint32_t)len[v];
        uint32_t g = gap_min;
        if (gap_div) g = max(g, l / gap_div);
        cap[v] = (unsigned long long)l + g;
    }
}

__global__ void k_off_to_u32(uint32_t V, const unsigned long long* in, uint32_t* out) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v <= V; v += (uint64_t)gridDim.x * blockDim.x)
        out[v] = (uint32_t)in[v];
}

__global__ void k_scatter_edges(uint64_t E, const uint32_t* src, const uint32_t* dst, const uint32_t* out_off,
                                int32_t* out_fill, uint32_t* out_nbr, const uint32_t* in_off, int32_t* in_fill,
                                uint32_t* in_nbr) {
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < E; e += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t s = src[e], d = dst[e];
        int po = atomicAdd(&out_fill[s], 1);
        out_nbr[out_off[s] + po] = d;
        int pi = atomicAdd(&in_fill[d], 1);
        in_nbr[in_off[d] + pi] = s;
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

// Entries per item of a list of len entries (piece numbers have 20 bits).
__device__ __forceinline__ unsigned peel_unit(unsigned chunk, unsigned len) {
    unsigned u = 4 * chunk;
    while (len > ((unsigned long long)u << 20)) u <<= 1;
    return u;
}

struct PeelHook {
    int ninst;
    __device__ __forceinline__ int operator()(EngineCtl* c, int level, bool worked, int bound) const {
        for (int i = 0; i < ninst; ++i) {
            unsigned n = ld_vol(&c->rc_cur[i]);
            if (ld_vol(&c->peel_compact[i])) {
                n = ld_vol(&c->rc_next[i].v);
                c->rc_cur[i] = n;
                c->rc_next[i].v = 0;
                c->peel_list[i] = ld_vol(&c->peel_list[i]) == 0 ? 1 : 0;
                c->removed[i] = 0;
                c->peel_compact[i] = 0;
            } else {
                // the list is written anew once a quarter of it is gone
                c->peel_compact[i] = 4ull * ld_vol(&c->removed[i]) > n;
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
            c->rc_cur[i] = member ? c->rc_next[i].v : V;
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

    // Works off the stack, 32 vertices at a time from its top (fewer when
    // their lists are long).  What remains is shared once it is more than a
    // moment's work and warps wait: one vertex each while they last, else
    // bags of 32.  (Sharing by the number of vertices alone left one warp with
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
            if (n > 1 && (unsigned long long)n * total > (unsigned long long)kPeelShare * m) {
                const int idle = (int)(ld_vol(&c->t_head) -
                                       (unsigned)*reinterpret_cast<volatile unsigned long long*>(&c->t_work));
                const unsigned own = max(1u, kPeelShare * m / max(total, 1u));
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

    const PeelHook next{p.ninst};
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

// ---------------------------------------------------------------------------
// incremental rows with exact support counters
// ---------------------------------------------------------------------------
struct Trans2Params {
    uint32_t n;  // vertices with state: V, or |C_K0| of the relabeled graph (ids from n on are outside C_K0)
    const uint32_t* out_off;
    int32_t* out_len;
    uint32_t* out_nbr;
    const uint32_t* in_off;
    int32_t* in_len;
    uint32_t* in_nbr;
    const int32_t* kmax;
    int32_t K;
    int32_t K0;     // first row to compute; cur holds row 0 (K0 > 1 jumps straight to row K0)
    // preleft: cur already holds -1 for the vertices outside C_K0 and the
    // counters ignore them, so the first row has no leaving set and seeds
    // every member whose out-count is below its value as well (the host
    // always starts runs this way; 0 = the leaving pass removes them)
    int preleft;
    int32_t Kstop;  // last row to compute (rows above stay untouched)
    int sorted;     // lists ordered by neighbour kmax, descending
    const uint32_t* order;  // C_k = order[0 .. ck[k]); nullptr: the graph is relabeled, C_k = ids 0 .. ck[k]-1
    const uint32_t* ck;
    int32_t* cur;
    int32_t* cnt_out;  // #{u in N_out(v) : cur[u] >= cur[v]}  (never above the truth)
    int32_t* cnt_in;   // #{w in N_in(v)  : cur[w] >= cur[v]}
    uint32_t* mark;
    int32_t* stamp;
    uint32_t* logidx;
    uint32_t* log_v;
    int32_t* log_k;
    int32_t* log_l;
    unsigned long long log_cap;
    TicketQueue q;
    EngineCtl* ctl;
};

// Next row (run by the warp that finished the step): after a row that needed
// no work, jump to the first row whose leaving set or seed set can be
// non-empty (the step's bound).
struct TransHook {
    __device__ __forceinline__ int operator()(EngineCtl*, int row, bool worked, int bound) const {
        return worked ? row + 1 : max(row + 1, bound);
    }
};

// Starting values of a run of rows that starts at row a on the handle's own
// graph: row 0 inside C_a, -1 (left) outside.
__global__ void k_preleft_cur(uint32_t V, const int32_t* kmax, const int32_t* row0, int32_t a, int32_t* cur) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V; v += (uint64_t)gridDim.x * blockDim.x)
        cur[v] = kmax[v] >= a ? row0[v] : -1;
}

// This lane's share of #{entries u of list a[0..n) : cur[u] >= cv}, 128
// entries per warp step; on kmax-sorted lists (sorted != 0) the count stops
// after the step whose last entry is outside C_a (cur == -1, or an id from
// `ids` on: so is every later entry).
__device__ __forceinline__ int count_at_least(const int32_t* cur, uint32_t ids, const uint32_t* a, int n, int cv,
                                              int sorted) {
    const unsigned lane = threadIdx.x & 31u;
    int c = 0;
    for (int b = 0; b < n; b += 128) {
        uint32_t u[4];
        int x[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int e = b + 32 * r + (int)lane;
            u[r] = e < n ? a[e] : ids;
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) x[r] = u[r] < ids ? cur[u[r]] : -1;
#pragma unroll
        for (int r = 0; r < 4; ++r) c += (x[r] >= cv);
        if (sorted && b + 128 < n && __shfl_sync(0xFFFFFFFFu, x[3], 31) == -1) break;
    }
    return c;
}

// Counters of the first n vertices against every neighbour, at the vertex's
// starting value (vertices with a value below 1 get zero counts: they are
// never evaluated and no counter includes them).  On kmax-sorted lists
// (sorted != 0) a list ends at its first neighbour outside C_a, which counts
// nothing.
__global__ void k_counters_init(uint32_t n, const uint32_t* out_off, const int32_t* out_len, const uint32_t* out_nbr,
                                const uint32_t* in_off, const int32_t* in_len, const uint32_t* in_nbr,
                                const int32_t* cur, int32_t* cnt_out, int32_t* cnt_in, int sorted) {
    const unsigned lane = threadIdx.x & 31u;
    const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t v = gw; v < n; v += nw) {
        int cv = cur[v];
        int co = 0, ci = 0;
        if (cv < 1) {  // never evaluated, never counted: no support needed
            if (lane == 0) {
                cnt_out[v] = 0;
                cnt_in[v] = 0;
            }
            continue;
        }
        co = count_at_least(cur, n, out_nbr + out_off[v], out_len[v], cv, sorted);
        ci = count_at_least(cur, n, in_nbr + in_off[v], in_len[v], cv, sorted);
        co = __reduce_add_sync(0xFFFFFFFFu, co);
        ci = __reduce_add_sync(0xFFFFFFFFu, ci);
        if (lane == 0) {
            cnt_out[v] = co;
            cnt_in[v] = ci;
        }
    }
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

// ---- vectorised list passes of the row kernel ----------------------------
// A list is read with 16-byte id loads: the list at element offset o of its
// array, length n, is covered by the virtual indices t in [o & 3, (o & 3) + n)
// of the 16-byte aligned window starting at o - (o & 3); lane l takes the
// four ids at t = b + 4 l .. b + 4 l + 3 of the step starting at b (128
// entries per list and step), so eight neighbour values per lane (both
// lists) are gathered in flight at once.  The adjacency arrays are 16-byte
// aligned and padded so that the last window of the last list stays inside.
__device__ __forceinline__ void load_ids4(const uint32_t* nbr, uint32_t o, int end, int b, bool active, uint32_t u[4]) {
    const int t0 = b + 4 * (int)(threadIdx.x & 31u);
    uint4 w = make_uint4(0u, 0u, 0u, 0u);
    if (active && t0 < end) w = *reinterpret_cast<const uint4*>(nbr + (o - (o & 3u)) + t0);
    u[0] = w.x;
    u[1] = w.y;
    u[2] = w.z;
    u[3] = w.w;
}

__device__ __forceinline__ int sel4(const int x[4], int q) { return q == 0 ? x[0] : q == 1 ? x[1] : q == 2 ? x[2] : x[3]; }

// Value of the step's last entry (virtual index last >= b) for the early stop
// on kmax-sorted lists.
__device__ __forceinline__ int last_value(const int x[4], int b, int last) {
    const int r = last - b;
    return __shfl_sync(0xFFFFFFFFu, sel4(x, r & 3), r >> 2);
}

// Counts the neighbours at each value of [lo, hi] (both lists) into the bins
// bo / bi; values above hi are not counted (the caller carries them).  On
// kmax-sorted lists a list ends at its first neighbour outside C_j.  Returns
// the entries read.
__device__ __forceinline__ int hist_pass2v(const int32_t* cur, uint32_t ids, const uint32_t* onbr, uint32_t oo, int no,
                                           const uint32_t* inbr, uint32_t io, int ni, int lo, int hi, bool sorted,
                                           int* bo, int* bi) {
    const unsigned lane = threadIdx.x & 31u;
    const int so = (int)(oo & 3u), si = (int)(io & 3u), endo = so + no, endi = si + ni;
    int to = 0, ti = 0, entries = 0;
    bool doneo = no <= 0, donei = ni <= 0;
    for (int b = 0; !(doneo && donei); b += 128) {
        uint32_t uo[4], ui[4];
        load_ids4(onbr, oo, endo, b, !doneo, uo);
        load_ids4(inbr, io, endi, b, !donei, ui);
        const int t0 = b + 4 * (int)lane;
        int co[4], ci[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int t = t0 + q;
            co[q] = (!doneo && t >= so && t < endo && uo[q] < ids) ? ld_vol(&cur[uo[q]]) : -1;
            ci[q] = (!donei && t >= si && t < endi && ui[q] < ids) ? ld_vol(&cur[ui[q]]) : -1;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            int x = co[q];
            to += (x == hi);
            if (x >= lo && x < hi) atomicAdd(&bo[x - lo], 1);
            x = ci[q];
            ti += (x == hi);
            if (x >= lo && x < hi) atomicAdd(&bi[x - lo], 1);
        }
        if (!doneo) {
            const int last = min(b + 127, endo - 1);
            entries += last + 1 - max(b, so);
            const int lv = last_value(co, b, last);
            if (b + 128 >= endo || (sorted && lv == -1)) doneo = true;
        }
        if (!donei) {
            const int last = min(b + 127, endi - 1);
            entries += last + 1 - max(b, si);
            const int lv = last_value(ci, b, last);
            if (b + 128 >= endi || (sorted && lv == -1)) donei = true;
        }
    }
#pragma unroll
    for (int s = 16; s; s >>= 1) {
        to += __shfl_xor_sync(0xFFFFFFFFu, to, s);
        ti += __shfl_xor_sync(0xFFFFFFFFu, ti, s);
    }
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
    load_ids4(p.out_nbr, L.oo, (int)(L.oo & 3u) + L.no, 0, L.no > 0, L.uo);
    load_ids4(p.in_nbr, L.io, (int)(L.io & 3u) + L.ni, 0, L.ni > 0, L.ui);
    return L;
}

// Values of the window's four entries of this lane (-1 outside the list, and
// for ids from `ids` on).
__device__ __forceinline__ void gather4(const int32_t* cur, uint32_t ids, const uint32_t u[4], int b, int start,
                                        int end, bool active, int v[4]) {
    const int t0 = b + 4 * (int)(threadIdx.x & 31u);
#pragma unroll
    for (int q = 0; q < 4; ++q)
        v[q] = (active && t0 + q >= start && t0 + q < end && u[q] < ids) ? ld_vol(&cur[u[q]]) : -1;
}

// Counts, over both lists, the neighbours at each of the kThr values cap,
// cap - 1, .. (a drop is rarely larger), this lane's share in go / gi.  The
// next window's ids are in flight while a window's values are gathered, so a
// step of 128 entries per list costs one memory latency.  Returns the entries
// read.
constexpr int kThr = 4;
__device__ __forceinline__ int count_pass(const Trans2Params& p, const RowLists& L, int cap, int go[kThr],
                                          int gi[kThr]) {
    const int so = (int)(L.oo & 3u), si = (int)(L.io & 3u), endo = so + L.no, endi = si + L.ni;
    uint32_t uo[4], ui[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        uo[q] = L.uo[q];
        ui[q] = L.ui[q];
    }
#pragma unroll
    for (int r = 0; r < kThr; ++r) go[r] = gi[r] = 0;
    bool ao = L.no > 0, ai = L.ni > 0;
    int entries = 0;
    for (int b = 0; ao || ai; b += 128) {
        int vo[4], vi[4];
        gather4(p.cur, p.n, uo, b, so, endo, ao, vo);
        gather4(p.cur, p.n, ui, b, si, endi, ai, vi);
        entries += (ao ? min(128, endo - b) : 0) + (ai ? min(128, endi - b) : 0);
        ao = ao && b + 128 < endo;
        ai = ai && b + 128 < endi;
        load_ids4(p.out_nbr, L.oo, endo, b + 128, ao, uo);
        load_ids4(p.in_nbr, L.io, endi, b + 128, ai, ui);
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int r = 0; r < kThr; ++r) {
                go[r] += vo[q] >= cap - r;
                gi[r] += vi[q] >= cap - r;
            }
        // kmax-sorted lists end at the first neighbour outside C_j
        if (p.sorted && ao && __shfl_sync(0xFFFFFFFFu, vo[3], 31) == -1) ao = false;
        if (p.sorted && ai && __shfl_sync(0xFFFFFFFFu, vi[3], 31) == -1) ai = false;
    }
    return entries;
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
__device__ __forceinline__ int drop_pass(const Trans2Params& p, EngineCtl* c, const RowLists& L, int nv, int cap,
                                         int j, unsigned long long word, int* cnt_o, int* cnt_i, uint32_t* keep,
                                         int* pending, int* lmin) {
    const int so = (int)(L.oo & 3u), si = (int)(L.io & 3u), endo = so + L.no, endi = si + L.ni;
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
    gather4(p.cur, p.n, uo, 0, so, endo, ao, vo);
    gather4(p.cur, p.n, ui, 0, si, endi, ai, vi);
    load_ids4(p.out_nbr, L.oo, endo, 128, ao, no);
    load_ids4(p.in_nbr, L.io, endi, 128, ai, ni);
    for (int b = 0;; b += 128) {
        entries += (ao ? min(128, endo - b) : 0) + (ai ? min(128, endi - b) : 0);
        bool mo = ao && b + 128 < endo, mi = ai && b + 128 < endi;
        if (p.sorted && mo && __shfl_sync(0xFFFFFFFFu, vo[3], 31) == -1) mo = false;
        if (p.sorted && mi && __shfl_sync(0xFFFFFFFFu, vi[3], 31) == -1) mi = false;
        int oldo[4], oldi[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (!kLeave) {
                *cnt_o += vo[q] >= nv;
                *cnt_i += vi[q] >= nv;
            }
            oldo[q] = (vo[q] > nv && vo[q] <= cap) ? atomicSub(&p.cnt_in[uo[q]], 1) : 0x7FFFFFFF;
            oldi[q] = (vi[q] > nv && vi[q] <= cap) ? atomicSub(&p.cnt_out[ui[q]], 1) : 0x7FFFFFFF;
        }
        int wo[4], wi[4];
        gather4(p.cur, p.n, no, b + 128, so, endo, mo, wo);
        gather4(p.cur, p.n, ni, b + 128, si, endi, mi, wi);
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
                so_[q] = (ro >> q) & 1u ? atomicOr(&p.mark[uo[q]], 1u) : 1u;
                si_[q] = (ri >> q) & 1u ? atomicOr(&p.mark[ui[q]], 1u) : 1u;
            }
            ro = ri = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (so_[q] == 0u) ro |= 1u << q;
                if (si_[q] == 0u) ri |= 1u << q;
            }
            if (keep_one(keep, &ro, uo) || keep_one(keep, &ri, ui)) {
                if (kLeave) step_count_kept(c, word);
                else --*pending;  // the item being finished pays for the kept one
            }
            step_push_mask8(c, p.q, ro, uo, ri, ui, step_tag(word));
        }
        if (!mo && !mi) break;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            uo[q] = no[q];
            ui[q] = ni[q];
            vo[q] = wo[q];
            vi[q] = wi[q];
        }
        load_ids4(p.out_nbr, L.oo, endo, b + 256, mo, no);
        load_ids4(p.in_nbr, L.io, endi, b + 256, mi, ni);
        ao = mo;
        ai = mi;
    }
    return entries;
}

// The value of x when it fell more than kThr - 1 below cap: windows of kWin
// values below hi, histograms in shared memory; carry_o / carry_i = counts
// above hi.  Counts at the value found go to *c_o / *c_i.
__device__ __forceinline__ int window_value(const Trans2Params& p, const RowLists& L, int j, int hi, int carry_o,
                                            int carry_i, int* ho, int* hi_, int* c_o, int* c_i, int* entries) {
    const unsigned lane = threadIdx.x & 31u;
    for (;;) {
        int lo = max(0, hi - (kWin - 1));
        ho[lane] = 0;
        ho[lane + 32] = 0;
        hi_[lane] = 0;
        hi_[lane + 32] = 0;
        __syncwarp();
        *entries += hist_pass2v(p.cur, p.n, p.out_nbr, L.oo, L.no, p.in_nbr, L.io, L.ni, lo, hi, p.sorted != 0, ho, hi_);
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

// Latency-bound: a row's changes run through dependent evaluations (one row
// of R-MAT 20 takes 480 us for 178 evaluations), so what counts is the number
// of memory round trips and fences from one vertex's drop to the next one's
// evaluation.  Hence: the static data of a vertex is loaded while its mark is
// set, its value and counters come with it, the new value is found with
// register counters at the four highest candidates (the shared-memory
// histogram only for larger drops), a corner record's place is in hand before
// the drop, one fence stands between the new value (with its record) and the
// neighbours' values, a request is one atomicOr, a warp keeps one of the items
// it requests, and rows advance without a grid barrier.  Together: rows
// 1..kmax of R-MAT 18 / 20 / 22 in one launch 16.5 / 25.8 / 53.5 -> 9.6 / 17.6 /
// 38.5 ms, ER 10,000 / 100,000 0.71 -> 0.39 ms.  80 registers for three
// blocks per SM (64 spill); one to four blocks measure within 7 %.
#ifndef DC_TRANS2_MIN_BLOCKS
#define DC_TRANS2_MIN_BLOCKS 3
#endif
__global__ void __launch_bounds__(kThreads, DC_TRANS2_MIN_BLOCKS) k_trans2(Trans2Params p) {
    const unsigned lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
    const unsigned gwarp = blockIdx.x * kWarpsPerBlock + wib;
    const unsigned nwarps = gridDim.x * kWarpsPerBlock;
    EngineCtl* c = p.ctl;
    __shared__ int s_ho[kWarpsPerBlock][kWin];
    __shared__ int s_hi[kWarpsPerBlock][kWin];
    __shared__ StepBlock s_step;
    const bool tracing = c->trace != nullptr;
    // failure-detection tests: this block never reports, the others' waits run out
    if (c->test_skip_block && (int)blockIdx.x == c->test_skip_block - 1) return;
    const TransHook next;
    unsigned my_evals = 0, my_drops = 0, my_log = 0;
    unsigned long long my_entries = 0;
    unsigned ticket = kNoTicket;
    unsigned long long log_at = 0;  // lane 0: the records of the warp's chunk
    unsigned log_left = 0;
    step_block_init(&s_step, c);
    unsigned long long word = step_block_word(&s_step);
    int jprev = p.preleft ? p.K0 : 0;  // row currently held in cur
    bool seed_out = p.preleft != 0;
    for (;;) {
        const int j = step_level(word);
        if (word == kStopWord || j > p.Kstop) break;
        const unsigned long long tag = step_tag(word);
        if (tracing && threadIdx.x == 0) trace_wake(c, word);
        uint32_t keep = kNoKeep;
        int pending = 0;
        // rows jprev+1 .. j-1 equal row jprev; vertices with kmax in
        // [jprev, j-1] leave now (all but those with kmax == j-1 have value 0)
        const uint32_t vj = __ldg(p.ck + j), vprev = __ldg(p.ck + jprev);
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
                al = ld_vol(&p.cur[xl]);
                *(volatile int32_t*)&p.cur[xl] = -1;
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
                drop_pass<true>(p, c, cur_l, 0, a, j, word, nullptr, nullptr, &keep, &pending, &bound);
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
                const int cv = ld_vol(&p.cur[v]), ci = ld_vol(&p.cnt_in[v]);
                const int co = seed_out ? ld_vol(&p.cnt_out[v]) : 0x7FFFFFFF;
                const int km = __ldg(p.kmax + v);
                if (cv >= 1) {
                    if (ci < j || co < cv) req = mark_request(&p.mark[v]) ? 1u : 0u;
                    else bound = min(bound, min(ci, km) + 1);
                }
            }
            if (__any_sync(0xFFFFFFFFu, req != 0u)) {
                const uint32_t u[4] = {v, 0u, 0u, 0u};
                if (keep_one(&keep, &req, u)) step_count_kept(c, word);
                step_push(c, p.q, req != 0u, (unsigned long long)v | tag);
            }
        }
        step_seeded(c, &s_step, bound, false, word, tracing, next);

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
                state = step_take(c, p.q, &s_step, &ticket, &item, &pending, &word, next);
                if (state != kTakeItem) break;
                x = (uint32_t)item;
            }
            // the mark says "being evaluated" before any neighbour is read (a
            // request made before it belongs to a drop that is seen below, one
            // made after it has x evaluated again); a decrement that lands
            // between the counter snapshot and the mark only makes the counter
            // too low, which costs an evaluation
            unsigned mk = 0;
            if (lane == 0) mk = atomicExch(&p.mark[x], 2u);
            const int cap = ld_vol(&p.cur[x]);
            const int s0o = ld_vol(&p.cnt_out[x]), s0i = ld_vol(&p.cnt_in[x]);
            const int stamp = ld_vol(&p.stamp[x]);
            const uint32_t logidx = ld_vol(&p.logidx[x]);
            const int km = __ldg(p.kmax + x);
            const RowLists L = row_lists(p, x);
            if (lane == 0) used_result(mk, ld_acquire(&p.mark[x]));
            __syncwarp();
            if (km < j || cap < 1) {
                if (lane == 0) atomicExch(&p.mark[x], 0u);
                ++pending;
                continue;
            }
            // ---- new value
            int c_o = 0, c_i = 0, nv = -1, entries;
            {
                int go[kThr], gi[kThr];
                entries = count_pass(p, L, cap, go, gi);
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
                        nv = window_value(p, L, j, cap - kThr, go[kThr - 1], gi[kThr - 1], s_ho[wib], s_hi[wib], &c_o,
                                          &c_i, &entries);
                    } else {  // unreachable for members of C_j
                        nv = 0;
                    }
                }
            }
            ++my_evals;
            if (nv < cap) {
                ++my_drops;
                if (lane == 0) {
                    // the value and its corner record
                    unsigned long long li = logidx;
                    const bool fresh = stamp != j;
                    if (fresh) {
                        if (!log_left) {
                            log_at = atomicAdd(&c->log_count, kLogChunk);
                            log_left = kLogChunk;
                        }
                        li = log_at++;
                        --log_left;
                        ++my_log;
                    }
                    if (li < p.log_cap) {
                        if (fresh) {
                            p.stamp[x] = j;
                            p.logidx[x] = (uint32_t)li;
                            p.log_v[li] = x;
                            p.log_k[li] = j;
                        }
                        p.log_l[li] = nv;
                    } else {
                        set_dev_error(c, DC_DEV_ERR_CAPACITY, 20);
                    }
                    *(volatile int32_t*)&p.cur[x] = nv;
                }
                __syncwarp();
                __threadfence();
                // recount at nv after the write, and take x's support away
                // from neighbours whose level lies in (nv, cap]: out-neighbours
                // hold x in cnt_in, in-neighbours in cnt_out
                c_o = 0;
                c_i = 0;
                entries += drop_pass<false>(p, c, L, nv, cap, j, word, &c_o, &c_i, &keep, &pending, nullptr);
                c_o = __reduce_add_sync(0xFFFFFFFFu, c_o);
                c_i = __reduce_add_sync(0xFFFFFFFFu, c_i);
            }
            my_entries += (unsigned)entries;
            if (tracing && lane == 0 && step_number(word) - 1 < c->trace_cap)
                atomicMax(&c->trace[8 * (step_number(word) - 1) + 7], (unsigned long long)entries);
            unsigned again = 0;
            if (lane == 0) {
                const int no = atomicAdd(&p.cnt_out[x], c_o - s0o) + (c_o - s0o);
                const int ni = atomicAdd(&p.cnt_in[x], c_i - s0i) + (c_i - s0i);
                const bool stable = nv < 1 || (no >= nv && ni >= j);
                // released once the counters are; requested meanwhile or
                // unstable: evaluated again
                if (!stable || atomicCAS(&p.mark[x], 2u, 0u) == 3u) {
                    used_result(atomicExch(&p.mark[x], 1u));
                    again = 1u;
                }
            }
            if (__shfl_sync(0xFFFFFFFFu, again, 0)) {
                if (keep == kNoKeep) {
                    keep = x;  // at once: still the item being finished
                    continue;
                }
                step_push(c, p.q, lane == 0, (unsigned long long)x | tag);
            }
            ++pending;
        }
        if (state == kTakeStop) break;
        jprev = j;
        seed_out = false;
    }
    if (lane == 0) {
        // unused records of the last chunk are void
        for (; log_left; --log_left, ++log_at)
            if (log_at < p.log_cap) p.log_k[log_at] = -1;
        atomicAdd(&c->log_used, my_log);
        atomicAdd(&c->evals, (unsigned long long)my_evals);
        atomicAdd(&c->drops, (unsigned long long)my_drops);
        atomicAdd(&c->edges_scanned, my_entries);
    }
}

// ---------------------------------------------------------------------------
// adjacency lists ordered by neighbour kmax, descending
// ---------------------------------------------------------------------------
// With every list in this order, the neighbours inside C_j = {kmax >= j}
// form a prefix of the list, so row-to-row evaluations read only that
// prefix.  Short lists: one thread, insertion sort.  Medium lists: one block,
// bitonic sort of (kmax, id) pairs in shared memory.  Long lists: one block,
// counting sort by kmax through a scratch copy of the list.
static constexpr int kSortShort = 32;
static constexpr int kSortWarp = 256;
static constexpr int kSortMid = 4096;

// Where the entries of list i come from: the list itself (sorted in place),
// or, when the relabeled graph is built, list order[i] of the handle's graph
// with every entry renamed by pos (copy, rename and sort in one pass).
struct ListSrc {
    const uint32_t* off;
    const uint32_t* nbr;
    const uint32_t* order;  // nullptr: in place
    const uint32_t* pos;
};
__device__ __forceinline__ const uint32_t* src_list(const ListSrc& s, uint32_t i, const uint32_t* own) {
    return s.order ? s.nbr + s.off[s.order[i]] : own;
}
__device__ __forceinline__ uint32_t src_id(const ListSrc& s, uint32_t u) { return s.order ? s.pos[u] : u; }

// Lists of at most kSortShort entries are sorted here, one thread each;
// longer ones are listed for the warp sort (up to kSortWarp), the block
// sort (up to kSortMid) or the counting sort.
__global__ void k_sort_short(uint32_t V, const uint32_t* off, const int32_t* len, uint32_t* nbr, const int32_t* kmax,
                             uint32_t* warp_list, uint32_t* mid_list, uint32_t* big_list, unsigned* cnt, ListSrc src) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V; v += (uint64_t)gridDim.x * blockDim.x) {
        int n = len[v];
        if (n > kSortMid) {
            big_list[atomicAdd(&cnt[2], 1u)] = (uint32_t)v;
            continue;
        }
        if (n > kSortWarp) {
            mid_list[atomicAdd(&cnt[1], 1u)] = (uint32_t)v;
            continue;
        }
        if (n > kSortShort) {
            warp_list[atomicAdd(&cnt[0], 1u)] = (uint32_t)v;
            continue;
        }
        uint32_t* a = nbr + off[v];
        const uint32_t* in = src_list(src, (uint32_t)v, a);
        if (n < 2) {
            if (n == 1 && src.order) a[0] = src_id(src, in[0]);
            continue;
        }
        uint32_t ids[kSortShort];
        int ks[kSortShort];
        for (int i = 0; i < n; ++i) {
            ids[i] = src_id(src, in[i]);
            ks[i] = kmax[ids[i]];
        }
        for (int i = 1; i < n; ++i) {
            uint32_t x = ids[i];
            int kx = ks[i];
            int jj = i - 1;
            while (jj >= 0 && ks[jj] < kx) {
                ids[jj + 1] = ids[jj];
                ks[jj + 1] = ks[jj];
                --jj;
            }
            ids[jj + 1] = x;
            ks[jj + 1] = kx;
        }
        for (int i = 0; i < n; ++i) a[i] = ids[i];
    }
}

// One warp per list of kSortShort+1 .. kSortWarp entries: the list and its
// neighbours' kmax go to the warp's shared buffer, every entry's place is its
// rank (entries with a larger kmax, or an equal kmax and a smaller index, go
// before it), and the entries are written back at their places.  The list
// count is read on the device (no host round trip).
constexpr int kSortWarpThreads = 256;
// Lane-strided entries i = lane + 32 t, t < T: rank among the n staged
// entries, written to a[rank].  Staged keys are (kmax << 8) | (255 - index),
// all distinct, so the rank (kmax descending, index ascending on ties) is the
// number of larger keys.
template <int T>
__device__ __forceinline__ void warp_rank_place(const uint32_t* ids, const uint32_t* ks, int n, uint32_t* a) {
    const unsigned lane = threadIdx.x & 31u;
    uint32_t mk[T];
    int rank[T];
#pragma unroll
    for (int t = 0; t < T; ++t) {
        const int i = (int)lane + 32 * t;
        mk[t] = i < n ? ks[i] : 0xFFFFFFFFu;
        rank[t] = 0;
    }
    for (int j = 0; j < n; ++j) {
        const uint32_t kj = ks[j];
#pragma unroll
        for (int t = 0; t < T; ++t) rank[t] += kj > mk[t];
    }
#pragma unroll
    for (int t = 0; t < T; ++t) {
        const int i = (int)lane + 32 * t;
        if (i < n) a[rank[t]] = ids[i];
    }
}
__global__ void __launch_bounds__(kSortWarpThreads) k_sort_warp(const uint32_t* off, const int32_t* len,
                                                                 uint32_t* nbr, const int32_t* kmax,
                                                                 const uint32_t* list, const unsigned* n_list,
                                                                 ListSrc src) {
    constexpr int kW = kSortWarpThreads / 32;
    static_assert(kSortWarp <= 256, "index part of the staged keys is 8 bits");
    __shared__ uint32_t s_id[kW][kSortWarp];
    __shared__ uint32_t s_k[kW][kSortWarp];
    const unsigned lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    const unsigned nl = *n_list;
    for (unsigned li = blockIdx.x * kW + w; li < nl; li += gridDim.x * kW) {
        const uint32_t v = list[li];
        const int n = len[v];
        uint32_t* a = nbr + off[v];
        const uint32_t* in = src_list(src, v, a);
        for (int i = lane; i < n; i += 32) {
            const uint32_t u = src_id(src, in[i]);
            s_id[w][i] = u;
            s_k[w][i] = ((uint32_t)kmax[u] << 8) | (uint32_t)(255 - i);
        }
        __syncwarp();
        switch ((n + 31) >> 5) {  // chunks of 32 entries (uniform over the warp)
            case 1: warp_rank_place<1>(s_id[w], s_k[w], n, a); break;
            case 2: warp_rank_place<2>(s_id[w], s_k[w], n, a); break;
            case 3: warp_rank_place<3>(s_id[w], s_k[w], n, a); break;
            case 4: warp_rank_place<4>(s_id[w], s_k[w], n, a); break;
            case 5: warp_rank_place<5>(s_id[w], s_k[w], n, a); break;
            case 6: warp_rank_place<6>(s_id[w], s_k[w], n, a); break;
            case 7: warp_rank_place<7>(s_id[w], s_k[w], n, a); break;
            default: warp_rank_place<8>(s_id[w], s_k[w], n, a); break;
        }
        __syncwarp();
    }
}

// One block per list of kSortWarp+1 .. kSortMid entries: a counting sort by
// neighbour kmax in shared memory (K + 1 bins, the list staged in shared
// memory), written back in place.  Entries of equal kmax keep no particular
// order; only the kmax order matters to the readers.  Dynamic shared memory:
// 4 (K + 1) + 8 kSortMid bytes.
__global__ void k_sort_mid(const uint32_t* off, const int32_t* len, uint32_t* nbr, const int32_t* kmax, int K,
                           const uint32_t* list, unsigned n_list, ListSrc src) {
    extern __shared__ unsigned s_mid[];
    unsigned* bins = s_mid;                   // K + 1
    uint32_t* ids = s_mid + (K + 1);          // kSortMid
    int* ks = (int*)(ids + kSortMid);         // kSortMid
    for (unsigned li = blockIdx.x; li < n_list; li += gridDim.x) {
        const uint32_t v = list[li];
        const int n = len[v];
        uint32_t* a = nbr + off[v];
        const uint32_t* in = src_list(src, v, a);
        for (int i = threadIdx.x; i <= K; i += blockDim.x) bins[i] = 0;
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const uint32_t u = src_id(src, in[i]);
            const int k = kmax[u];
            ids[i] = u;
            ks[i] = k;
            atomicAdd(&bins[K - k], 1u);
        }
        __syncthreads();
        unsigned long long carry = 0;
        for (int b0 = 0; b0 <= K; b0 += blockDim.x) {
            const int b = b0 + threadIdx.x;
            const unsigned long long x = b <= K ? bins[b] : 0ull;
            unsigned long long tot;
            const unsigned long long ex = block_excl_scan64(x, &tot);
            if (b <= K) bins[b] = (unsigned)(ex + carry);
            carry += tot;
            __syncthreads();
        }
        for (int i = threadIdx.x; i < n; i += blockDim.x) a[atomicAdd(&bins[K - ks[i]], 1u)] = ids[i];
        __syncthreads();
    }
}

// bins = K + 1 counters in shared memory (K < kSortBigBins)
static constexpr int kSortBigBins = 11264;
__global__ void k_sort_big(const uint32_t* off, const int32_t* len, uint32_t* nbr, uint32_t* tmp, const int32_t* kmax,
                           int K, const uint32_t* list, unsigned n_list, ListSrc src) {
    __shared__ unsigned bins[kSortBigBins];
    for (unsigned li = blockIdx.x; li < n_list; li += gridDim.x) {
        uint32_t v = list[li];
        const int n = len[v];
        uint32_t* a = nbr + off[v];
        // in place: staged through tmp; from a source list: straight into a
        uint32_t* t = src.order ? a : tmp + off[v];
        const uint32_t* in = src_list(src, v, a);
        for (int i = threadIdx.x; i <= K; i += blockDim.x) bins[i] = 0;
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += blockDim.x) atomicAdd(&bins[K - kmax[src_id(src, in[i])]], 1u);
        __syncthreads();
        // exclusive scan of bins (K+1 values), chunked by blockDim
        unsigned long long carry = 0;
        for (int b0 = 0; b0 <= K; b0 += blockDim.x) {
            int b = b0 + threadIdx.x;
            unsigned long long x = b <= K ? bins[b] : 0ull;
            unsigned long long tot;
            unsigned long long ex = block_excl_scan64(x, &tot);
            if (b <= K) bins[b] = (unsigned)(ex + carry);
            carry += tot;
            __syncthreads();
        }
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            uint32_t u = src_id(src, in[i]);
            unsigned pos = atomicAdd(&bins[K - kmax[u]], 1u);
            t[pos] = u;
        }
        __syncthreads();
        if (!src.order)
            for (int i = threadIdx.x; i < n; i += blockDim.x) a[i] = t[i];
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// order by kmax, skyline assembly, expansion
// ---------------------------------------------------------------------------
// Counts per kmax value.  Most vertices share a few small values, so the
// counts go to per-block shared bins first (when kmax + 1 <= kHistShared).
constexpr int kHistShared = 8192;
__global__ void k_kmax_hist(uint32_t V, const int32_t* kmax, uint32_t* hist, int32_t K) {
    extern __shared__ uint32_t sh[];
    const bool shared = K + 1 <= kHistShared;
    if (shared)
        for (int i = threadIdx.x; i <= K; i += blockDim.x) sh[i] = 0;
    __syncthreads();
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V; v += (uint64_t)gridDim.x * blockDim.x)
        atomicAdd(shared ? &sh[kmax[v]] : &hist[kmax[v]], 1u);
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

// cursor[k] = first position of bucket k in descending-kmax order
// Warp-aggregated: lanes holding the same kmax take their positions with one
// atomic (the leader's) instead of one each.
__global__ void k_order_scatter(uint32_t V, const int32_t* kmax, uint32_t* cursor, uint32_t* order) {
    const unsigned lane = threadIdx.x & 31u;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t base = (blockIdx.x * (uint64_t)blockDim.x) & ~31ull; base < V; base += stride) {
        const uint64_t v = base + (threadIdx.x & ~31u) % blockDim.x + lane;
        const bool ok = v < V;
        const int key = ok ? kmax[v] : -1;
        const unsigned peers = __match_any_sync(0xFFFFFFFFu, key);
        const unsigned leader = __ffs(peers) - 1;
        unsigned p0 = 0;
        if (ok && lane == leader) p0 = atomicAdd(&cursor[key], (unsigned)__popc(peers));
        p0 = __shfl_sync(0xFFFFFFFFu, p0, leader);
        if (ok) order[p0 + __popc(peers & ((1u << lane) - 1u))] = (uint32_t)v;
    }
}

// corner bound per vertex: min(kmax, row0) + 1
__global__ void k_corner_bound(uint32_t V, const int32_t* kmax, const int32_t* row0, unsigned long long* acc) {
    unsigned long long s = 0;
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V; v += (uint64_t)gridDim.x * blockDim.x)
        s += (unsigned long long)min(kmax[v], row0[v]);
#pragma unroll
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
    if ((threadIdx.x & 31u) == 0) atomicAdd(acc, s);
}

// Row ranges of the segments of a split run of rows.
struct SegBounds {
    int32_t lo[kMaxRowSegments], hi[kMaxRowSegments];
    int n;
};
// Corner bounds per segment: acc[i] = corners of rows lo[i]..hi[i] (a
// vertex's value drops at least one per corner, so it has at most
// min(rows it belongs to, row 0 value) of them; the first corner of a
// segment that starts from row 0 is one of them).
__global__ void k_corner_bounds(uint32_t V, const int32_t* kmax, const int32_t* row0, SegBounds b,
                                unsigned long long* acc) {
    unsigned long long t[kMaxRowSegments] = {};
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V; v += (uint64_t)gridDim.x * blockDim.x) {
        const int32_t km = kmax[v], r0 = row0[v];
#pragma unroll
        for (int i = 0; i < kMaxRowSegments; ++i)
            if (i < b.n) t[i] += (unsigned long long)max(0, min(min(km, b.hi[i]) - b.lo[i] + 1, r0));
    }
#pragma unroll
    for (int i = 0; i < kMaxRowSegments; ++i) {
#pragma unroll
        for (int o = 16; o; o >>= 1) t[i] += __shfl_xor_sync(0xFFFFFFFFu, t[i], o);
        if ((threadIdx.x & 31u) == 0 && i < b.n && t[i]) atomicAdd(&acc[i], t[i]);
    }
}

// log entries with a negative row are void (dropped corners)
__global__ void k_sky_count(uint32_t V, uint64_t nlog, const uint32_t* log_v, const int32_t* log_k,
                            unsigned long long* cnt) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nlog; i += (uint64_t)gridDim.x * blockDim.x)
        if (log_k[i] >= 0) atomicAdd(&cnt[log_v[i]], 1ull);
}
// A row segment that jumped from row 0 to row k logs vertex v at row k
// whenever its value differs from row 0; the corner is void when the value
// equals row k-1's (cur after the previous segment).  Counts the void entries.
__global__ void k_seg_void(uint64_t n, const uint32_t* log_v, int32_t* log_k, const int32_t* log_l, int32_t k,
                           const int32_t* cur, unsigned long long* dropped) {
    unsigned long long t = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        if (log_k[i] == k && log_l[i] == cur[log_v[i]]) {
            log_k[i] = -1;
            ++t;
        }
#pragma unroll
    for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xFFFFFFFFu, t, o);
    if ((threadIdx.x & 31u) == 0 && t) atomicAdd(dropped, t);
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

__global__ void k_max_reduce(uint64_t n, const int32_t* a, int* out) {
    int m = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        m = max(m, a[i]);
#pragma unroll
    for (int o = 16; o; o >>= 1) m = max(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
    if ((threadIdx.x & 31u) == 0) atomicMax(out, m);
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
    dfree(st, g.out_nbr_alloc);
    g.out_nbr = nullptr;
    dfree(st, g.in_off);
    dfree(st, g.in_len);
    dfree(st, g.in_nbr_alloc);
    g.in_nbr = nullptr;
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

void free_scratch(dc_graph* h) {
    Scratch* s = h->scratch;
    if (!s) return;
    for (RowSegment& g : s->seg) {
        if (g.stream) cudaStreamSynchronize(g.stream);
        dfree(h->stream, g.cur);
        dfree(h->stream, g.cnt_out);
        dfree(h->stream, g.cnt_in);
        dfree(h->stream, g.mark);
        dfree(h->stream, g.stamp);
        dfree(h->stream, g.logidx);
        dfree(h->stream, g.tring);
        dfree(h->stream, g.ctl);
        if (g.stream) cudaStreamDestroy(g.stream);
        for (auto& e : g.ev)
            if (e) cudaEventDestroy(e);
    }
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
    dfree(h->stream, s->ring);
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
    dfree(h->stream, s->w_out_len);
    dfree(h->stream, s->w_in_len);
    dfree(h->stream, s->w_out_nbr);
    dfree(h->stream, s->w_in_nbr);
    dfree(h->stream, s->kmax_old);
    dfree(h->stream, s->row0_old);
    dfree(h->stream, s->pos);
    dfree(h->stream, s->kmax_r);
    dfree(h->stream, s->row0_r);
    for (int i = 0; i < 2; ++i) {
        dfree(h->stream, s->r_off[i]);
        dfree(h->stream, s->r_len[i]);
        dfree(h->stream, s->r_nbr_alloc[i]);
    }
    delete s;
    h->scratch = nullptr;
}

int ensure_scratch(dc_graph* h, uint32_t V) {
    if (!h->scratch) h->scratch = new Scratch();
    Scratch* s = h->scratch;
    if (s->cap_V >= V && s->key) return DC_OK;
    // release V-sized buffers and reallocate
    dfree(h->stream, s->key); dfree(h->stream, s->cdeg); dfree(h->stream, s->cur); dfree(h->stream, s->row0); dfree(h->stream, s->mark); dfree(h->stream, s->stamp);
    dfree(h->stream, s->logidx); dfree(h->stream, s->rem0); dfree(h->stream, s->rem1); dfree(h->stream, s->order); dfree(h->stream, s->ring); dfree(h->stream, s->tmp64);
    dfree(h->stream, s->partial); dfree(h->stream, s->cursor);
    dfree(h->stream, s->key2); dfree(h->stream, s->cdeg2); dfree(h->stream, s->rem2); dfree(h->stream, s->rem3); dfree(h->stream, s->cnt_out);
    uint64_t n = (uint64_t)V + 1;
    if (dmalloc(h->stream, &s->key, n) || dmalloc(h->stream, &s->cdeg, n) || dmalloc(h->stream, &s->cur, n) || dmalloc(h->stream, &s->row0, n) ||
        dmalloc(h->stream, &s->mark, n) || dmalloc(h->stream, &s->stamp, n) || dmalloc(h->stream, &s->logidx, n) || dmalloc(h->stream, &s->rem0, n) ||
        dmalloc(h->stream, &s->rem1, n) || dmalloc(h->stream, &s->order, n) || dmalloc(h->stream, &s->tmp64, n + 1) ||
        dmalloc(h->stream, &s->partial, (uint64_t)h->geom.sms * 64 + 64) || dmalloc(h->stream, &s->cursor, n + 1) ||
        dmalloc(h->stream, &s->key2, n) || dmalloc(h->stream, &s->cdeg2, n) || dmalloc(h->stream, &s->rem2, n) || dmalloc(h->stream, &s->rem3, n) ||
        dmalloc(h->stream, &s->cnt_out, n))
        return DC_ERR_NOMEM;
    uint64_t need = (uint64_t)V + (uint64_t)h->geom.sms * 64 * 32 + 64;
    uint64_t rc = 1024;
    while (rc < need) rc <<= 1;
    if (dmalloc(h->stream, &s->ring, rc)) return DC_ERR_NOMEM;
    s->ring_mask = (uint32_t)(rc - 1);
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
        if (s->key) b += 4 * (16 * n + 1) + 8 * (n + 1) + 8 * ((uint64_t)h->geom.sms * 64 + 64) + 4ull * (s->ring_mask + 1ull);
        b += 4ull * s->ck_cap + 12 * s->log_cap + 8 * s->tring_cap;
        b += 4 * (s->w_out_cap + s->w_in_cap);
        if (s->kmax_old) b += 8 * n;
        for (const RowSegment& sg : s->seg)
            b += (sg.cur ? 24 * ((uint64_t)sg.cap_V + 1) : 0) + 8 * sg.tring_cap + (sg.ctl ? sizeof(EngineCtl) : 0);
        if (s->pos) b += 4 * 7 * ((uint64_t)s->r_cap_V + 1);     // relabeled graph: ids, kmax, row 0, offsets, lengths
        if (s->r_nbr_alloc[0]) b += 2 * 4 * (s->r_cap + 7);     // its lists
    }
    return b;
}

// Exclusive scan of n u64 values in s->tmp64 (tmp64[n] receives the total).
int scan_tmp64(dc_graph* h, uint64_t n) {
    Scratch* s = h->scratch;
    unsigned long long* data = (unsigned long long*)s->tmp64;
    unsigned long long* part = (unsigned long long*)s->partial;
    void* args[] = {&data, &n, &part, &h->ctl};
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)k_scan_coop, 256, 0);
    per_sm = std::max(1, std::min(per_sm, 8));
    DC_CUDA(cudaMemsetAsync(h->ctl, 0, sizeof(EngineCtl), h->stream));
    ++g_launches;
    cudaError_t e = cudaLaunchCooperativeKernel((const void*)k_scan_coop, dim3(per_sm * h->geom.sms), dim3(256), args,
                                                0, h->stream);
    if (e != cudaSuccess) return set_error(DC_ERR_CUDA, "scan launch failed: %s", cudaGetErrorString(e));
    return DC_OK;
}

static int finish_build(dc_graph* h, uint32_t V, uint64_t E, const uint32_t* d_src, const uint32_t* d_dst) {
    DevGraph& g = h->g;
    Scratch* s = h->scratch;
    // capacities -> offsets (out)
    for (int side = 0; side < 2; ++side) {
        int32_t* len = side == 0 ? g.out_len : g.in_len;
        ++g_launches;
        k_capacity<<<grid_for(h, V), kThreads, 0, h->stream>>>(V, len, h->gap_min, h->gap_div,
                                                               (unsigned long long*)s->tmp64);
        if (int rc = scan_tmp64(h, V)) return rc;
        unsigned long long total = 0;
        DC_CUDA(cudaMemcpyAsync(&total, s->tmp64 + V, sizeof(total), cudaMemcpyDeviceToHost, h->stream));
        DC_CUDA(cudaStreamSynchronize(h->stream));
        if (total >= 0xFFFFFFFFull)
            return set_error(DC_ERR_CAPACITY, "adjacency with slack exceeds 2^32 entries (u32 offsets)");
        uint32_t** off = side == 0 ? &g.out_off : &g.in_off;
        uint32_t** nbr = side == 0 ? &g.out_nbr : &g.in_nbr;
        uint32_t** alloc = side == 0 ? &g.out_nbr_alloc : &g.in_nbr_alloc;
        // the row kernel reads ids in aligned 16-byte groups: the lists
        // start at a 16-byte boundary (three spare entries in front cover
        // any alignment of the allocation) and four spare entries at the end
        // cover the last group of the last list
        if (dmalloc(h->stream, off, (uint64_t)V + 1) || dmalloc(h->stream, alloc, total + 7)) return DC_ERR_NOMEM;
        *nbr = (uint32_t*)(((uintptr_t)*alloc + 15u) & ~(uintptr_t)15u);
        ++g_launches;
        k_off_to_u32<<<grid_for(h, (uint64_t)V + 1), kThreads, 0, h->stream>>>(V, (unsigned long long*)s->tmp64, *off);
        if (side == 0) g.out_cap = total;
        else g.in_cap = total;
    }
    DC_CUDA(cudaMemsetAsync(g.out_len, 0, sizeof(int32_t) * V, h->stream));
    DC_CUDA(cudaMemsetAsync(g.in_len, 0, sizeof(int32_t) * V, h->stream));
    if (E)
        ++g_launches;
        k_scatter_edges<<<grid_for(h, E), kThreads, 0, h->stream>>>(E, d_src, d_dst, g.out_off, g.out_len, g.out_nbr,
                                                                     g.in_off, g.in_len, g.in_nbr);
    DC_CUDA(cudaGetLastError());
    g.V = V;
    g.E = E;
    g.sorted_kmax = false;
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
    if (E) k_count_degrees<<<grid_for(h, E), kThreads, 0, h->stream>>>(V, E, d_src, d_dst, g.out_len, g.in_len, h->ctl);
    EngineCtl hc;
    if (int rc = check_ctl(h, &hc, "graph build")) return rc;
    return finish_build(h, V, E, d_src, d_dst);
}

__global__ void k_host_csr_len(uint32_t V, const int32_t* deg, int32_t* len) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V; v += (uint64_t)gridDim.x * blockDim.x)
        len[v] = deg[v];
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

// Two 256-thread blocks per SM: measured best or near it from R-MAT 19 to 22
// once the queue counters sit on separate lines (the autotuner refines it).
static constexpr int kDefaultBlocksPerSm = 2;

static int persistent_grid(dc_graph* h, const void* fn, int bps, int* blocks, int share = 1) {
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kThreads, 0);
    if (e != cudaSuccess || per_sm < 1)
        return set_error(DC_ERR_CUDA, "occupancy query failed (%s)", cudaGetErrorString(e));
    if (bps <= 0) bps = h->blocks_per_sm > 0 ? h->blocks_per_sm : kDefaultBlocksPerSm;
    // launches that share the SMs get an equal part of the resident blocks each
    *blocks = std::max(1, std::min(bps * h->geom.sms, per_sm * h->geom.sms / share));
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
// share: the launch is one of that many which run at the same time.
static int persistent_launch(dc_graph* h, const void* fn, void** args, const char* name, EngineCtl* ctl,
                             cudaStream_t st, int bps, const FirstStep* first = nullptr, int share = 1) {
    int blocks = 0;
    if (int rc = persistent_grid(h, fn, bps, &blocks, share)) return rc;
    const bool own = ctl == h->ctl;
    EngineCtl* initp = &h->ctl_init;
    for (int i = 0; i < kMaxRowSegments - 1; ++i)
        if (ctl == h->scratch->seg[i].ctl) initp = &h->ctl_init_seg[i];
    EngineCtl& init = *initp;
    memset(&init, 0, sizeof(init));
    init.step = -1;
    init.wait_ns = h->wait_ns;
    if (first) {
        init.step = 0;
        init.t_work = (unsigned long long)blocks << kWorkShift;
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
        unsigned long long* ring = s->tring;
        uint64_t cap = s->tring_cap;
        for (const RowSegment& g : s->seg)
            if (ctl == g.ctl) {
                ring = g.tring;
                cap = g.tring_cap;
            }
        cudaMemsetAsync(ring, 0xFF, sizeof(unsigned long long) * cap, st);
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

// Stream, events and control block of row segment i + 1 (seg[i]).
static int ensure_segment_stream(dc_graph* h, int i) {
    RowSegment& g = h->scratch->seg[i];
    if (!g.stream) {
        DC_CUDA(cudaStreamCreateWithFlags(&g.stream, cudaStreamNonBlocking));
        for (auto& e : g.ev) DC_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
    if (!g.ctl && dmalloc(h->stream, &g.ctl, 1)) return DC_ERR_NOMEM;
    return DC_OK;
}

// State of row segment i + 1 for the n vertices of its first row's core (ids
// below n of the relabeled graph), with an eighth of headroom.
static int ensure_segment(dc_graph* h, int i, uint32_t n) {
    if (int rc = ensure_segment_stream(h, i)) return rc;
    RowSegment& g = h->scratch->seg[i];
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

// Creates the streams of the row segments the handle's cuts ask for (their
// state is sized for the graph's cores by the first run that uses them).
int prepare_row_segments(dc_graph* h) {
    const uint32_t V = h->g.V;
    if (!V) return DC_OK;
    int n = 0;
    while (n < kMaxRowSegments - 1 && h->rows_split[n] > 0) ++n;
    if (!n) return DC_OK;
    if (int rc = ensure_scratch(h, V)) return rc;
    for (int i = 0; i < n; ++i)
        if (int rc = ensure_segment_stream(h, i)) return rc;
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

// Runs one or two peels in one persistent launch; maxv[i] = largest value.
int run_peel2(dc_graph* h, int ninst, const PeelInst* inst, int32_t* maxv) {
    Scratch* s = h->scratch;
    DevGraph& g = h->g;
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
    const FirstStep first{0};
    if (int rc = run_persistent(h, fn, args, "peel", &hc, h->peel_bps, &first)) return rc;
    for (int i = 0; i < ninst; ++i) maxv[i] = hc.maxv[i];
    return DC_OK;
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

// Skyline from row 0 and the corner logs of the last run of rows: the
// first segment's nlog entries at the log's start (h->log_used of them
// records, the others void) and the other segments' ranges (h->seg_off /
// seg_n, void entries skipped).
int build_skyline_from_log(dc_graph* h, uint64_t nlog) {
    Scratch* s = h->scratch;
    Decomp& d = h->d;
    uint32_t V = h->g.V;
    unsigned long long* cnt = (unsigned long long*)s->tmp64;
    uint64_t lo[kMaxRowSegments], n[kMaxRowSegments];
    int nr = 0;
    uint64_t total = (uint64_t)V;
    if (nlog) {
        lo[nr] = 0;
        n[nr++] = nlog;
        total += h->log_used;
    }
    for (int i = 0; i < h->nseg_extra; ++i)
        if (h->seg_n[i]) {
            lo[nr] = h->seg_off[i];
            n[nr++] = h->seg_n[i];
            total += h->seg_n[i] - h->seg_void[i];
        }
    ++g_launches;
    k_set_one<<<grid_for(h, V), kThreads, 0, h->stream>>>(V, cnt);
    for (int r = 0; r < nr; ++r) {
        ++g_launches;
        k_sky_count<<<grid_for(h, n[r]), kThreads, 0, h->stream>>>(V, n[r], s->log_v + lo[r], s->log_k + lo[r], cnt);
    }
    if (int rc = scan_tmp64(h, V)) return rc;
    if (d.corner_cap < total || !d.sky_k) {
        // a quarter of headroom: maintenance batches rarely grow it again
        dfree(h->stream, d.sky_k);
        dfree(h->stream, d.sky_l);
        d.corner_cap = 0;
        const uint64_t want = total + total / 4 + 1;
        if (dmalloc(h->stream, &d.sky_k, want) || dmalloc(h->stream, &d.sky_l, want)) return DC_ERR_NOMEM;
        d.corner_cap = want;
    }
    if (!d.sky_off && dmalloc(h->stream, &d.sky_off, (uint64_t)V + 1)) return DC_ERR_NOMEM;
    ++g_launches;
    k_sky_fill_row0<<<grid_for(h, V), kThreads, 0, h->stream>>>(V, cnt, s->row0, d.sky_k, d.sky_l, s->cursor);
    for (int r = 0; r < nr; ++r) {
        ++g_launches;
        k_sky_fill_log<<<grid_for(h, n[r]), kThreads, 0, h->stream>>>(n[r], s->log_v + lo[r], s->log_k + lo[r],
                                                                      s->log_l + lo[r], cnt, d.sky_k, d.sky_l,
                                                                      s->cursor);
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
    if (dmalloc(h->stream, &d.rows, elems)) return DC_ERR_NOMEM;
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

// Orders every adjacency list by neighbour kmax, descending.  *sorted = 0
// when kmax is too large for the long-list counting sort (lists then stay
// in arbitrary order and evaluations read them whole).
// Orders every list of one side by neighbour kmax, descending (kmax[u] of
// each entry u of the graph the lists belong to).  cap = entries the lists'
// array spans (the long-list sort stages through a scratch copy that size).
static int sort_side(dc_graph* h, int32_t K, uint32_t V, const uint32_t* off, const int32_t* len, uint32_t* nbr,
                     uint64_t cap, const int32_t* kmax, int side, ListSrc src) {
    Scratch* s = h->scratch;
    unsigned* cnt = s->cursor;
    DC_CUDA(cudaMemsetAsync(cnt, 0, 3 * sizeof(unsigned), h->stream));
    ++g_launches;
    k_sort_short<<<grid_for(h, V), kThreads, 0, h->stream>>>(V, off, len, nbr, kmax, s->rem0, s->rem2, s->rem1, cnt,
                                                              src);
    // most lists go to the warp sort, which reads its count on the device
    ++g_launches;
    k_sort_warp<<<h->geom.sms * 8, kSortWarpThreads, 0, h->stream>>>(off, len, nbr, kmax, s->rem0, &cnt[0], src);
    unsigned hc[3] = {0, 0, 0};
    DC_CUDA(cudaMemcpyAsync(hc, cnt, sizeof(hc), cudaMemcpyDeviceToHost, h->stream));
    DC_CUDA(cudaStreamSynchronize(h->stream));
    if (hc[1]) {
        const size_t shm = 4ull * (K + 1) + 8ull * kSortMid;
        // the kernel's limit is set to its largest need, the same value on
        // every call: handles sorting on other threads at the same time
        // (the serving loop) must never see it lowered below their launch
        constexpr size_t kMidMax = 4ull * kSortBigBins + 8ull * kSortMid;
        static_assert(kMidMax <= 227ull * 1024, "mid-list sort shared memory");
        DC_CUDA(cudaFuncSetAttribute(k_sort_mid, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMidMax));
        int blocks = (int)std::min<unsigned>(hc[1], (unsigned)h->geom.sms * 8);
        ++g_launches;
        k_sort_mid<<<blocks, 256, shm, h->stream>>>(off, len, nbr, kmax, K, s->rem2, hc[1], src);
    }
    if (hc[2]) {
        uint32_t*& tmp = side == 0 ? s->w_out_nbr : s->w_in_nbr;
        uint64_t& tcap = side == 0 ? s->w_out_cap : s->w_in_cap;
        if (!src.order && (tcap < cap || !tmp)) {  // in place: staging copy of the lists' span
            dfree(h->stream, tmp);
            if (dmalloc(h->stream, &tmp, cap)) return DC_ERR_NOMEM;
            tcap = cap;
        }
        int blocks = (int)std::min<unsigned>(hc[2], (unsigned)h->geom.sms * 2);
        ++g_launches;
        k_sort_big<<<blocks, 512, 0, h->stream>>>(off, len, nbr, tmp, kmax, K, s->rem1, hc[2], src);
    }
    DC_CUDA(cudaGetLastError());
    return DC_OK;
}

// Orders every adjacency list of the graph by neighbour kmax, descending.
// *sorted = 0 when kmax is too large for the long-list counting sort (lists
// then stay in arbitrary order and evaluations read them whole).
static int sort_lists_by_kmax(dc_graph* h, int32_t K, int* sorted) {
    DevGraph& g = h->g;
    *sorted = 0;
    if (g.sorted_kmax) {
        *sorted = 1;
        return DC_OK;
    }
    if (K + 1 > kSortBigBins) return DC_OK;
    for (int side = 0; side < 2; ++side)
        if (int rc = sort_side(h, K, g.V, side == 0 ? g.out_off : g.in_off, side == 0 ? g.out_len : g.in_len,
                               side == 0 ? g.out_nbr : g.in_nbr, side == 0 ? g.out_cap : g.in_cap, h->d.kmax_v, side,
                               ListSrc{nullptr, nullptr, nullptr, nullptr}))
            return rc;
    g.sorted_kmax = true;
    *sorted = 1;
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
__global__ void k_relabel_gather(uint32_t V, const uint32_t* order, const int32_t* kmax, const int32_t* row0,
                                 const int32_t* out_len, const int32_t* in_len, uint32_t* pos, int32_t* kmax_r,
                                 int32_t* row0_r, int32_t* len_o, int32_t* len_i) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < V; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t v = order[i];
        pos[v] = (uint32_t)i;
        kmax_r[i] = kmax[v];
        row0_r[i] = row0[v];
        len_o[i] = out_len[v];
        len_i[i] = in_len[v];
    }
}

__global__ void k_len_to_u64e(uint32_t V, const int32_t* len, unsigned long long* out) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < V; i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = (unsigned long long)len[i];
}

// corner records of the relabeled run back to original ids (void ones hold none)
__global__ void k_unlabel_log(uint64_t n, const uint32_t* order, uint32_t* log_v, const int32_t* log_k) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        if (log_k[i] >= 0) log_v[i] = order[log_v[i]];
}

// Builds the relabeled graph (s->order must hold the kmax order of the
// current kmax) with its lists sorted by neighbour kmax, plus kmax and row 0
// by new id.
static int build_relabeled(dc_graph* h, int32_t K) {
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
    // list arrays: three spare entries in front for the 16-byte alignment of
    // the array start, four at the end for the last 16-byte id group
    const uint64_t cap = g.E + 8;
    if (s->r_cap < cap || !s->r_nbr_alloc[0]) {
        for (int i = 0; i < 2; ++i) {
            dfree(h->stream, s->r_nbr_alloc[i]);
            s->r_nbr[i] = nullptr;
        }
        s->r_cap = 0;
        const uint64_t want = cap + cap / 8;  // headroom for later, larger graphs of the handle
        for (int i = 0; i < 2; ++i) {
            if (dmalloc(h->stream, &s->r_nbr_alloc[i], want + 7)) return DC_ERR_NOMEM;
            s->r_nbr[i] = (uint32_t*)(((uintptr_t)s->r_nbr_alloc[i] + 15u) & ~(uintptr_t)15u);
        }
        s->r_cap = want;
    }
    ++g_launches;
    k_relabel_gather<<<grid_for(h, V), kThreads, 0, h->stream>>>(V, s->order, h->d.kmax_v, s->row0, g.out_len,
                                                                  g.in_len, s->pos, s->kmax_r, s->row0_r, s->r_len[0],
                                                                  s->r_len[1]);
    for (int side = 0; side < 2; ++side) {
        ++g_launches;
        k_len_to_u64e<<<grid_for(h, V), kThreads, 0, h->stream>>>(V, s->r_len[side], (unsigned long long*)s->tmp64);
        if (int rc = scan_tmp64(h, V)) return rc;
        ++g_launches;
        k_off_to_u32<<<grid_for(h, n), kThreads, 0, h->stream>>>(V, (unsigned long long*)s->tmp64, s->r_off[side]);
    }
    // every relabeled list is read from its original list, renamed and
    // sorted by neighbour kmax in one pass
    for (int side = 0; side < 2; ++side) {
        const ListSrc src{side == 0 ? g.out_off : g.in_off, side == 0 ? g.out_nbr : g.in_nbr, s->order, s->pos};
        if (int rc = sort_side(h, K, V, s->r_off[side], s->r_len[side], s->r_nbr[side], s->r_cap, s->kmax_r, side, src))
            return rc;
    }
    return DC_OK;
}

// Rows 1..Kstop from row 0 (scratch row0) and kmax (d.kmax_v): orders
// vertices by kmax, initialises the support counters and runs the
// row-to-row kernel.  Corners of rows 1..Kstop are left in the scratch log
// (*nlog entries).  allow_sort: order adjacency lists by neighbour kmax
// first (otherwise lists are read whole).
int rows_from_row0(dc_graph* h, int32_t K, int32_t Kstop, bool allow_sort, uint64_t* nlog_out, int32_t K0,
                   bool allow_relabel) {
    DevGraph& g = h->g;
    Decomp& d = h->d;
    Scratch* s = h->scratch;
    const uint32_t V = g.V;
    *nlog_out = 0;
    h->log_used = 0;
    h->nseg_extra = 0;
    cudaEventRecord(h->ev[2], h->stream);
    if (s->ck_cap < (uint32_t)K + 2) {
        dfree(h->stream, s->ck);
        if (dmalloc(h->stream, &s->ck, (uint64_t)K + 2)) return DC_ERR_NOMEM;
        s->ck_cap = K + 2;
    }
    uint32_t* hist = s->cursor;
    DC_CUDA(cudaMemsetAsync(hist, 0, sizeof(uint32_t) * ((uint64_t)K + 2), h->stream));
    ++g_launches;
    k_kmax_hist<<<grid_for(h, V), kThreads, K + 1 <= kHistShared ? 4 * (K + 1) : 0, h->stream>>>(V, d.kmax_v, hist, K);
    std::vector<uint32_t> hh((size_t)K + 2), ck((size_t)K + 2), start((size_t)K + 2);
    DC_CUDA(cudaMemcpyAsync(hh.data(), hist, sizeof(uint32_t) * ((size_t)K + 2), cudaMemcpyDeviceToHost, h->stream));
    unsigned long long* acc = (unsigned long long*)s->tmp64;
    DC_CUDA(cudaMemsetAsync(acc, 0, sizeof(unsigned long long), h->stream));
    ++g_launches;
    k_corner_bound<<<grid_for(h, V), kThreads, 0, h->stream>>>(V, d.kmax_v, s->row0, acc);
    unsigned long long bound = 0;
    DC_CUDA(cudaMemcpyAsync(&bound, acc, sizeof(bound), cudaMemcpyDeviceToHost, h->stream));
    DC_CUDA(cudaStreamSynchronize(h->stream));
    {
        uint64_t run = 0;
        ck[K + 1] = 0;
        for (int32_t k = K; k >= 0; --k) {
            start[k] = (uint32_t)run;
            run += hh[k];
            ck[k] = (uint32_t)run;
        }
    }
    DC_CUDA(cudaMemcpyAsync(s->ck, ck.data(), sizeof(uint32_t) * ((size_t)K + 2), cudaMemcpyHostToDevice, h->stream));
    DC_CUDA(cudaMemcpyAsync(hist, start.data(), sizeof(uint32_t) * ((size_t)K + 2), cudaMemcpyHostToDevice, h->stream));
    ++g_launches;
    k_order_scatter<<<grid_for(h, V), kThreads, 0, h->stream>>>(V, d.kmax_v, hist, s->order);
    // The graph the row kernel reads: where sorting is allowed, the graph
    // relabeled in kmax order with kmax-sorted lists (C_k a prefix of the
    // ids); else the handle's own lists (kmax-sorted when they still are from
    // an earlier run) with C_k listed by `order`.
    const bool relabel = allow_sort && allow_relabel && K + 1 <= kSortBigBins;
    // a run from row 1 on the relabeled graph (a full decomposition, or rows
    // 1..R of a maintenance batch) may be split in row segments run concurrently: segment 0 (rows
    // 1..cut[0]) on the handle's stream, segment i (rows cut[i-1]+1..cut[i],
    // starting there from row 0) on seg[i-1]'s stream, each with its own
    // state (for the vertices of its first row's core: the ids below |C_a|)
    // and its own range of the corner log; runs of fewer than kMinSplitRows
    // rows stay whole
    const int32_t k0 = std::max(1, K0);
    int32_t cut[kMaxRowSegments];
    int nseg = 1;
    if (relabel && k0 == 1 && Kstop >= kMinSplitRows) {
        int32_t split[kMaxRowSegments - 1] = {};
        for (int i = 0; i < kMaxRowSegments - 1; ++i)
            split[i] = (int32_t)((int64_t)K * (h->auto_cuts ? (i + 1) * 1000 / kMaxRowSegments : h->rows_split[i]) / 1000);
        if (h->auto_cuts) {
            // Cuts of a handle whose launch shapes were never set: equal runs
            // of rows, where the core a run starts from is small.  A run's
            // start costs a pass over its first core's lists and a refinement
            // from row 0 there: with skewed degrees (|C_k| a few per cent of
            // |C_1| at the first cut) eight runs at a time take the rows from
            // 3.46 / 8.92 / 34.2 ms to 1.30 / 3.66 / 19.6 (R-MAT 17 / 18 / 22,
            // the best of 13 sets of cuts 1.27 / 3.23 / 18.1); where every
            // vertex is in almost every core (ER, 100 edges per vertex) the
            // same cuts take them from 3.6 to 11.0 ms.  Hence a quarter of
            // |C_1| at most for a run's core, half of it for all together
            // (which also bounds the runs' state).
            uint64_t sum = 0;
            for (int i = kMaxRowSegments - 2; i >= 0; --i) {
                const uint64_t m = split[i] >= 1 && split[i] < Kstop ? ck[split[i] + 1] : 0;
                if (4 * m > ck[1] || 2 * (sum + m) > ck[1]) split[i] = 0;
                else sum += m;
            }
        }
        for (int i = 0; i < kMaxRowSegments - 1; ++i) {
            const int32_t c = split[i];
            if (c >= 1 && c < Kstop && (nseg == 1 || c > cut[nseg - 2])) cut[nseg++ - 1] = c;
        }
    }
    cut[nseg - 1] = Kstop;
    // log ranges: [off[i], off[i] + cap[i]) per segment
    uint64_t off[kMaxRowSegments] = {}, capn[kMaxRowSegments] = {};
    // records every warp of the largest grid may leave unused in its last chunk
    const uint64_t spare = (uint64_t)kLogChunk * kWarpsPerBlock * 8 * h->geom.sms / nseg;
    uint64_t lc = bound + 1 + spare;
    if (nseg > 1) {
        SegBounds sb;
        sb.n = nseg;
        for (int i = 0; i < nseg; ++i) {
            sb.lo[i] = i == 0 ? k0 : cut[i - 1] + 1;
            sb.hi[i] = cut[i];
        }
        DC_CUDA(cudaMemsetAsync(acc, 0, nseg * sizeof(unsigned long long), h->stream));
        ++g_launches;
        k_corner_bounds<<<grid_for(h, V), kThreads, 0, h->stream>>>(V, d.kmax_v, s->row0, sb, acc);
        unsigned long long bs[kMaxRowSegments] = {};
        DC_CUDA(cudaMemcpyAsync(bs, acc, nseg * sizeof(unsigned long long), cudaMemcpyDeviceToHost, h->stream));
        DC_CUDA(cudaStreamSynchronize(h->stream));
        lc = 0;
        for (int i = 0; i < nseg; ++i) {
            off[i] = lc;
            capn[i] = bs[i] + 1 + spare;
            lc += capn[i];
        }
    }
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
    if (nseg == 1) capn[0] = s->log_cap;
    int sorted = 0;
    const uint32_t *G_out_off = g.out_off, *G_in_off = g.in_off, *G_order = s->order;
    int32_t *G_out_len = g.out_len, *G_in_len = g.in_len;
    uint32_t *G_out_nbr = g.out_nbr, *G_in_nbr = g.in_nbr;
    const int32_t *G_kmax = d.kmax_v, *G_row0 = s->row0;
    if (relabel) {
        if (int rc = build_relabeled(h, K)) return rc;
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
    } else if (allow_sort || g.sorted_kmax) {
        if (int rc = sort_lists_by_kmax(h, K, &sorted)) return rc;
    }
    // starting values and counters of a run that starts at row a: row 0
    // inside C_a with the vertices outside already left (for a = 1 those of
    // kmax 0), so the run's first step has no leaving pass
    auto start_state = [&](cudaStream_t st, int32_t a, int32_t* cur, int32_t* co, int32_t* ci, uint32_t* mark,
                           uint64_t n_mark, int32_t* stamp) -> int {
        const uint32_t n = relabel ? ck[std::min(a, K + 1)] : V;
        DC_CUDA(cudaMemsetAsync(mark, 0, sizeof(uint32_t) * n_mark, st));
        if (!n) return DC_OK;
        if (relabel) {
            DC_CUDA(cudaMemcpyAsync(cur, G_row0, 4ull * n, cudaMemcpyDeviceToDevice, st));
        } else {
            ++g_launches;
            k_preleft_cur<<<grid_for(h, n), kThreads, 0, st>>>(n, G_kmax, G_row0, a, cur);
        }
        ++g_launches;
        k_counters_init<<<grid_for(h, (uint64_t)n * 32), kThreads, 0, st>>>(
            n, G_out_off, G_out_len, G_out_nbr, G_in_off, G_in_len, G_in_nbr, cur, co, ci, sorted);
        DC_CUDA(cudaMemsetAsync(stamp, 0xFF, sizeof(int32_t) * n, st));
        return DC_OK;
    };
    if (int rc = start_state(h->stream, k0, s->cur, s->cnt_out, s->key, s->mark, V, s->stamp))
        return rc;  // (the marks of all V vertices: the local core update expects them clear)
    if (int rc = ensure_tring(h, 2ull * V + (uint64_t)h->geom.sms * 64 + 4096)) return rc;
    Trans2Params tp[kMaxRowSegments];
    tp[0].n = relabel ? ck[std::min(k0, K + 1)] : V;
    tp[0].out_off = G_out_off; tp[0].out_len = G_out_len; tp[0].out_nbr = G_out_nbr;
    tp[0].in_off = G_in_off; tp[0].in_len = G_in_len; tp[0].in_nbr = G_in_nbr;
    tp[0].kmax = G_kmax;
    tp[0].K = K;
    tp[0].K0 = k0;
    tp[0].preleft = 1;
    tp[0].Kstop = cut[0];
    tp[0].sorted = sorted;
    tp[0].order = G_order;
    tp[0].ck = s->ck;
    tp[0].cur = s->cur;
    tp[0].cnt_out = s->cnt_out;
    tp[0].cnt_in = s->key;
    tp[0].mark = s->mark;
    tp[0].stamp = s->stamp;
    tp[0].logidx = s->logidx;
    tp[0].log_v = s->log_v;
    tp[0].log_k = s->log_k;
    tp[0].log_l = s->log_l;
    tp[0].log_cap = capn[0];
    tp[0].q.slots = s->tring;
    tp[0].q.mask = (unsigned)(s->tring_cap - 1);
    tp[0].ctl = h->ctl;
    for (int i = 1; i < nseg; ++i)
        if (int rc = ensure_segment(h, i - 1, ck[cut[i - 1] + 1])) return rc;
    if (nseg > 1) {
        // the other segments start once the shared preparation is done
        DC_CUDA(cudaEventRecord(s->seg[0].ev[0], h->stream));
        for (int i = 1; i < nseg; ++i) {
            RowSegment& sg = s->seg[i - 1];
            DC_CUDA(cudaStreamWaitEvent(sg.stream, s->seg[0].ev[0], 0));
            const uint32_t t_n = ck[cut[i - 1] + 1];
            if (int rc = start_state(sg.stream, cut[i - 1] + 1, sg.cur, sg.cnt_out, sg.cnt_in, sg.mark, t_n, sg.stamp))
                return rc;
            Trans2Params& t = tp[i];
            t = tp[0];
            t.n = t_n;
            t.K0 = cut[i - 1] + 1;
            t.preleft = 1;
            t.Kstop = cut[i];
            t.cur = sg.cur;
            t.cnt_out = sg.cnt_out;
            t.cnt_in = sg.cnt_in;
            t.mark = sg.mark;
            t.stamp = sg.stamp;
            t.logidx = sg.logidx;
            t.log_v = s->log_v + off[i];
            t.log_k = s->log_k + off[i];
            t.log_l = s->log_l + off[i];
            t.log_cap = capn[i];
            t.q.slots = sg.tring;
            t.q.mask = (unsigned)(sg.tring_cap - 1);
            t.ctl = sg.ctl;
        }
    }
    uint64_t nlog = 0;
    uint64_t nseg_log[kMaxRowSegments] = {}, nseg_used[kMaxRowSegments] = {};
    unsigned long long voids[kMaxRowSegments] = {};
    cudaEventRecord(h->ev[3], h->stream);
    if (tp[0].Kstop >= tp[0].K0) {
        static const char* const kNames[8] = {"transitions",           "transitions (segment 2)",
                                              "transitions (segment 3)", "transitions (segment 4)",
                                              "transitions (segment 5)", "transitions (segment 6)",
                                              "transitions (segment 7)", "transitions (segment 8)"};
        static_assert(kMaxRowSegments <= 8, "one name per segment");
        void* args[kMaxRowSegments][1];
        int launched = 0, rc = DC_OK;
        for (int i = 0; i < nseg && rc == DC_OK; ++i) {
            args[i][0] = &tp[i];
            EngineCtl* ctl = i == 0 ? h->ctl : s->seg[i - 1].ctl;
            cudaStream_t st = i == 0 ? h->stream : s->seg[i - 1].stream;
            const FirstStep first{tp[i].K0};
            rc = persistent_launch(h, (const void*)k_trans2, args[i], kNames[i], ctl, st, h->rows_bps, &first, nseg);
            if (rc == DC_OK) ++launched;
        }
        h->stat_evals = h->stat_drops = h->stat_entries = 0;
        for (int i = 0; i < launched; ++i) {
            EngineCtl hc;
            EngineCtl* ctl = i == 0 ? h->ctl : s->seg[i - 1].ctl;
            cudaStream_t st = i == 0 ? h->stream : s->seg[i - 1].stream;
            const int r = finish_persistent(h, ctl, st, kNames[i], &hc);
            if (r != DC_OK) {
                if (rc == DC_OK) rc = r;
                continue;
            }
            nseg_log[i] = hc.log_count;
            nseg_used[i] = hc.log_used;
            h->stat_evals += hc.evals;
            h->stat_drops += hc.drops;
            h->stat_entries += hc.edges_scanned;
        }
        if (rc) return rc;
        nlog = nseg_log[0];
        h->log_used = nseg_used[0];
        if (nseg > 1) {
            DC_CUDA(cudaMemsetAsync(acc, 0, nseg * sizeof(unsigned long long), h->stream));
            for (int i = 1; i < nseg; ++i) {
                RowSegment& sg = s->seg[i - 1];
                DC_CUDA(cudaEventRecord(sg.ev[1], sg.stream));
                DC_CUDA(cudaStreamWaitEvent(h->stream, sg.ev[1], 0));
                if (!nseg_log[i]) continue;
                // a corner at the segment's first row is void where the value
                // equals the previous segment's last row
                const int32_t* prev = i == 1 ? s->cur : s->seg[i - 2].cur;
                ++g_launches;
                k_seg_void<<<grid_for(h, nseg_log[i]), kThreads, 0, h->stream>>>(
                    nseg_log[i], s->log_v + off[i], s->log_k + off[i], s->log_l + off[i], cut[i - 1] + 1, prev,
                    acc + i);
            }
            DC_CUDA(cudaMemcpyAsync(voids, acc, nseg * sizeof(unsigned long long), cudaMemcpyDeviceToHost, h->stream));
            DC_CUDA(cudaStreamSynchronize(h->stream));
            h->nseg_extra = nseg - 1;
            for (int i = 1; i < nseg; ++i) {
                h->seg_off[i - 1] = off[i];
                h->seg_n[i - 1] = nseg_log[i];
                h->seg_void[i - 1] = nseg_log[i] - nseg_used[i] + voids[i];
            }
        }
        if (relabel)  // corner records back to original ids (the seam check above compares relabeled state)
            for (int i = 0; i < nseg; ++i)
                if (nseg_log[i]) {
                    ++g_launches;
                    k_unlabel_log<<<grid_for(h, nseg_log[i]), kThreads, 0, h->stream>>>(nseg_log[i], s->order,
                                                                                       s->log_v + off[i],
                                                                                       s->log_k + off[i]);
                }
    }
    cudaEventRecord(h->ev[4], h->stream);
    *nlog_out = nlog;
    return DC_OK;
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
    if (int rc = degree_kmax_sum(h, &h->full_work)) return rc;
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

// sum over vertices of (in + out degree) x kmax: the list entries a per-row
// pass over rows 1..kmax scans, a deterministic measure of a graph's row work
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
