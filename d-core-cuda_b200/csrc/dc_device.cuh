// Device-side building blocks shared by the persistent engine kernels:
//   - EngineCtl: counters, error word and grid-barrier state in device memory
//   - grid_sync: software grid barrier with a bounded wait (cooperative launch)
//   - ticket queue, and steps on it that follow one another without a barrier
//   - warp-aggregated append
// Every spin in here is bounded by the control block's wait limit
// (EngineCtl::wait_ns, kWaitNs when 0) of %globaltimer time; on expiry the
// waiter sets DC_DEV_ERR_TIMEOUT in EngineCtl::error and returns, so a fault
// in the protocol ends the kernel with a status instead of a hang.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace dc {

constexpr unsigned DC_DEV_ERR_TIMEOUT = 1u;   // a bounded wait ran out
constexpr unsigned DC_DEV_ERR_BADID = 4u;     // vertex id out of range
constexpr unsigned DC_DEV_ERR_CAPACITY = 8u;  // a log or list buffer overflowed
constexpr unsigned DC_DEV_ERR_NOTFOUND = 16u; // delete of an absent edge

constexpr uint32_t kEmptySlot = 0xFFFFFFFFu;
constexpr unsigned long long kWaitNs = 4000000000ull;  // default limit of one wait: 4 s
constexpr int kMaxRowSegments = 8;  // runs the rows' cuts (dc_tuning) may ask for
constexpr int kRowGroups = 8;       // groups of blocks that work on runs of rows at the same time
constexpr int kMinSplitRows = 32;   // runs of fewer rows are never split

// A counter on a 128-byte line of its own.
struct alignas(128) PadU {
    unsigned v;
};
struct alignas(128) PadW {
    unsigned long long v;
};
constexpr int kStepWords = 8;  // copies of the step word, each block polls one

// The counters every warp hits (ticket head and tail, the outstanding count,
// the barrier) and the flags idle warps poll (phase_done, error) each sit in
// a 128-byte line of their own: on one line they all land in one L2 slice,
// which then serialises the grid.
struct EngineCtl {
    // grid barrier
    alignas(128) unsigned bar_count;
    unsigned bar_gen;
    // polled by idle warps
    alignas(128) unsigned error;
    unsigned err_where;
    unsigned worked;               // last step of which an item was kept by the warp that found it
    unsigned log_used;             // corner records written (the log's ranges have holes)
    unsigned phase_done;    // set by whoever brings outstanding to 0
    // results / statistics
    alignas(128) unsigned log_count;
    unsigned long long evals;
    unsigned long long drops;
    unsigned long long pushes;
    unsigned long long edges_scanned;
    // ticket queue (see TicketQueue)
    alignas(128) unsigned t_head;  // next ticket
    alignas(128) unsigned t_tail;  // next slot to reserve
    alignas(128) int outstanding;  // unfinished producers + pushed, unfinished items
    PadW step_word[kStepWords];                // (step number << 32) | level, see "Steps without a barrier"
    alignas(128) unsigned long long t_work;    // steps without a barrier: both in one word
    alignas(128) unsigned bag_tail;            // fused peel: vertices put into bags
    int peel_list[2];       // per peel: remaining vertices in rem0 / rem1, or all (-1)
    int peel_compact[2];    // the level writes the list anew
    unsigned removed[2];    // removed so far
    unsigned removed_at[2]; // removed when the list was written
    unsigned members[2];    // vertices to remove
    alignas(128) unsigned long long next_low;  // (step << 32) | (2^31 - 1 - least next level)
    alignas(128) unsigned rc_cur[2];  // remaining-list sizes per peel instance
    PadU rc_next[2];        // next level's remaining-list sizes (appended by every warp)
    int maxv[2];            // largest value per peel instance
    int step;               // level / transition index
    int level;              // row repair: last row taken
    // optional per-step timing trace: 8 words per step
    //   [0] %globaltimer at step start, [1] when its work ran out,
    //   [2] queue items of the step, [3] %globaltimer at the closing barrier,
    //   [4] latest block wake-up after the opening barrier,
    //   [5] latest block seeding done, [6] earliest block wake-up
    unsigned long long* trace;
    unsigned trace_cap;
    unsigned trace_tail0;
    // limit of one bounded wait in ns (0: kWaitNs)
    unsigned long long wait_ns;
    // failure-detection tests: block test_skip_block - 1 leaves at its first
    // grid barrier without arriving, so every other block's barrier wait runs
    // out (0: off)
    int test_skip_block;
};

// Decisions and results of one maintenance batch run as a captured CUDA
// graph: every branch the host-driven batch takes between its kernels is
// taken on the device, by small kernels writing these fields, and the
// kernels after a branch act only while their run flag is set.
struct BatchStatus {
    int run_apply;      // the batch is valid: no missing deletion, insertions fit their free slots
    int run_repair;     // rows 1..R are repaired in place
    int run_merge;      // a new skyline is merged (the repair's changes, or new row-0 corners only)
    int run_chg;        // the merge reads change lists (the repair logged changes)
    int fallback;       // rows 1..R must be recomputed (repair not expected to pay, or it gave up)
    int merge_overflow; // the merged skyline outgrew its buffer: the host merges instead
    int notfound;       // a deleted edge is not in the graph (nothing applied)
    int need_rebuild;   // an inserted edge does not fit its list (nothing applied)
    int R, Knew, lmax;  // row bound, kmax and lmax after the batch
    unsigned err, err_where;  // device error bits of the persistent kernels
    unsigned n_leave;   // vertices whose kmax fell (deletions) or rose (insertions)
    unsigned pad;
    unsigned long long nlog, total, cap, work, region, scanned;
    unsigned long long deadline_ns;  // time limit of the repair (0: none)
};

__device__ __forceinline__ unsigned long long wait_limit(const EngineCtl* c) {
    const unsigned long long w = *reinterpret_cast<const volatile unsigned long long*>(&c->wait_ns);
    return w ? w : kWaitNs;
}

__device__ __forceinline__ unsigned ld_vol(const unsigned* p) {
    return *reinterpret_cast<const volatile unsigned*>(p);
}
__device__ __forceinline__ int ld_vol(const int* p) {
    return *reinterpret_cast<const volatile int*>(p);
}
__device__ __forceinline__ unsigned long long gtimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void set_dev_error(EngineCtl* c, unsigned code, unsigned where) {
    atomicOr(&c->error, code);
    atomicExch(&c->err_where, where);
}

// Software grid barrier.  All blocks of a cooperative launch are co-resident,
// so every block reaches it unless one has already bailed out on an error;
// waiters then leave on the error word or after the wait limit.
// Returns true when the grid may continue.
__device__ __forceinline__ bool grid_sync(EngineCtl* c) {
    __shared__ unsigned s_ok;
    if (c->test_skip_block && (int)blockIdx.x == c->test_skip_block - 1) return false;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned nb = gridDim.x;
        unsigned gen = ld_vol(&c->bar_gen);
        __threadfence();
        unsigned arrived = atomicAdd(&c->bar_count, 1u);
        if (arrived == nb - 1) {
            atomicExch(&c->bar_count, 0u);
            __threadfence();
            atomicAdd(&c->bar_gen, 1u);
        } else {
            const unsigned long long t0 = gtimer(), lim = wait_limit(c);
            while (ld_vol(&c->bar_gen) == gen) {
                if (ld_vol(&c->error)) break;
                if (gtimer() - t0 > lim) {
                    set_dev_error(c, DC_DEV_ERR_TIMEOUT, 1);
                    break;
                }
                __nanosleep(32);
            }
        }
        __threadfence();
        s_ok = (ld_vol(&c->error) == 0u);
    }
    __syncthreads();
    return s_ok != 0u;
}

// Grid barrier whose last arriving block runs hook(c) before releasing the
// others, so per-phase counters can be reset with no other block running.
template <typename Hook>
__device__ __forceinline__ bool grid_sync_hook(EngineCtl* c, Hook hook) {
    __shared__ unsigned s_ok2;
    if (c->test_skip_block && (int)blockIdx.x == c->test_skip_block - 1) return false;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned nb = gridDim.x;
        unsigned gen = ld_vol(&c->bar_gen);
        __threadfence();
        unsigned arrived = atomicAdd(&c->bar_count, 1u);
        if (arrived == nb - 1) {
            hook(c);
            atomicExch(&c->bar_count, 0u);
            __threadfence();
            atomicAdd(&c->bar_gen, 1u);
        } else {
            const unsigned long long t0 = gtimer(), lim = wait_limit(c);
            while (ld_vol(&c->bar_gen) == gen) {
                if (ld_vol(&c->error)) break;
                if (gtimer() - t0 > lim) {
                    set_dev_error(c, DC_DEV_ERR_TIMEOUT, 4);
                    break;
                }
                __nanosleep(32);
            }
        }
        __threadfence();
        s_ok2 = (ld_vol(&c->error) == 0u);
        if (c->trace) {
            int st = ld_vol(&c->step);
            if (st >= 0 && (unsigned)st < c->trace_cap) {
                unsigned long long now = gtimer();
                atomicMax(&c->trace[8 * st + 4], now);
                atomicMin(&c->trace[8 * st + 6], now);
            }
        }
    }
    __syncthreads();
    return s_ok2 != 0u;
}

// Warp-aggregated append: every lane of a converged warp calls this; lanes
// with pred get consecutive positions from *counter.
__device__ __forceinline__ unsigned warp_append(unsigned* counter, bool pred, unsigned* total = nullptr) {
    const unsigned lane = threadIdx.x & 31u;
    unsigned mask = __ballot_sync(0xFFFFFFFFu, pred);
    if (total) *total = __popc(mask);
    if (!mask) return 0;
    unsigned leader = __ffs(mask) - 1;
    unsigned base = 0;
    if (lane == leader) base = atomicAdd(counter, (unsigned)__popc(mask));
    base = __shfl_sync(0xFFFFFFFFu, base, leader);
    return base + __popc(mask & ((1u << lane) - 1u));
}

// ---------------------------------------------------------------------------
// Ticket queue.  Items are 64-bit words in a ring of slots (kEmptyItem =
// free).  A consumer warp takes a ticket with one atomicAdd on t_head and
// polls only its own slot, so idle warps do not contend on shared counters.
// Termination uses one counter: `outstanding` starts at the number of
// producer warps; each producer subtracts 1 when its seeding share is done,
// each push adds the number of pushed items before they become visible, and
// each finished item subtracts 1 after its own pushes.  Whoever brings it to
// 0 sets phase_done; a consumer whose slot is still empty then leaves.  At
// the barrier that ends the phase the abandoned tickets are skipped by
// setting t_tail = t_head (grid_sync_hook).
// ---------------------------------------------------------------------------
constexpr unsigned long long kEmptyItem = ~0ull;

struct TicketQueue {
    unsigned long long* slots;
    unsigned mask;
};

__device__ __forceinline__ void tq_finish(EngineCtl* c, int n) {
    __threadfence();
    if (atomicSub(&c->outstanding, n) == n) {
        atomicExch(&c->phase_done, 1u);
        if (c->trace && (unsigned)c->step < c->trace_cap) c->trace[8 * c->step + 1] = gtimer();
    }
}

// Converged warp: lanes with pred push `cnt` consecutive items item0,
// item0 + inc, ... (cnt may be 0).
__device__ __forceinline__ void tq_push_warp_multi(EngineCtl* c, TicketQueue q, unsigned cnt,
                                                   unsigned long long item0, unsigned long long inc) {
    const unsigned lane = threadIdx.x & 31u;
    unsigned x = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= (unsigned)o) x += y;
    }
    unsigned total = __shfl_sync(0xFFFFFFFFu, x, 31);
    if (total == 0) return;
    unsigned base = 0;
    if (lane == 0) {
        atomicAdd(&c->outstanding, (int)total);
        base = atomicAdd(&c->t_tail, total);
    }
    base = __shfl_sync(0xFFFFFFFFu, base, 0) + (x - cnt);
    if (cnt) __threadfence();
    for (unsigned i = 0; i < cnt; ++i) {
        volatile unsigned long long* s = &q.slots[(base + i) & q.mask];
        *s = item0 + inc * i;
    }
}

__device__ __forceinline__ void tq_push_warp(EngineCtl* c, TicketQueue q, bool pred, unsigned long long item) {
    const unsigned lane = threadIdx.x & 31u;
    unsigned m = __ballot_sync(0xFFFFFFFFu, pred);
    if (!m) return;
    unsigned base = 0;
    if (lane == 0) {
        atomicAdd(&c->outstanding, (int)__popc(m));
        base = atomicAdd(&c->t_tail, (unsigned)__popc(m));
    }
    base = __shfl_sync(0xFFFFFFFFu, base, 0);
    if (pred) {
        __threadfence();
        volatile unsigned long long* s = &q.slots[(base + __popc(m & ((1u << lane) - 1u))) & q.mask];
        *s = item;
    }
}

// Converged warp: each lane pushes items[r] for every bit r set in mask
// (r < 4), in bit order.
__device__ __forceinline__ void tq_push_warp_mask4(EngineCtl* c, TicketQueue q, unsigned mask,
                                                   const uint32_t items[4]) {
    const unsigned lane = threadIdx.x & 31u;
    const unsigned cnt = __popc(mask);
    unsigned x = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= (unsigned)o) x += y;
    }
    unsigned total = __shfl_sync(0xFFFFFFFFu, x, 31);
    if (total == 0) return;
    unsigned base = 0;
    if (lane == 0) {
        atomicAdd(&c->outstanding, (int)total);
        base = atomicAdd(&c->t_tail, total);
    }
    base = __shfl_sync(0xFFFFFFFFu, base, 0) + (x - cnt);
    if (cnt) __threadfence();
#pragma unroll
    for (unsigned r = 0; r < 4; ++r) {
        if (mask & (1u << r)) {
            volatile unsigned long long* s = &q.slots[(base + __popc(mask & ((1u << r) - 1u))) & q.mask];
            *s = (unsigned long long)items[r];
        }
    }
}

// Converged warp: returns true with *item set, or false when the phase is
// over (or an error / timeout occurred).  *ticket holds the warp's current
// ticket between calls (kNoTicket initially).
constexpr unsigned kNoTicket = 0xFFFFFFFFu;
__device__ __forceinline__ bool tq_take_warp(EngineCtl* c, TicketQueue q, unsigned* ticket,
                                             unsigned long long* item) {
    const unsigned lane = threadIdx.x & 31u;
    unsigned long long it = kEmptyItem;
    int state = 0;  // 1 = got item, 2 = phase over
    if (lane == 0) {
        if (*ticket == kNoTicket) *ticket = atomicAdd(&c->t_head, 1u);
        volatile unsigned long long* s = &q.slots[*ticket & q.mask];
        unsigned long long t0 = 0;
        unsigned spins = 0, seen_tail = 0;
        int seen_out = 0;
        for (;;) {
            it = *s;
            if (it != kEmptyItem) {
                *s = kEmptyItem;
                *ticket = kNoTicket;
                state = 1;
                break;
            }
            // the shared flags are polled every 4th spin once the wait is long
            if ((spins < 16 || (spins & 3) == 0) && (ld_vol(&c->phase_done) || ld_vol(&c->error))) {
                // abandon the ticket: the phase-ending barrier skips it
                *ticket = kNoTicket;
                state = 2;
                break;
            }
            if (++spins == 64) {
                t0 = gtimer();
                seen_tail = ld_vol(&c->t_tail);
                seen_out = ld_vol(&c->outstanding);
            }
            // the limit bounds a wait without progress: while the phase's
            // other warps still push or finish items the clock restarts
            if (spins > 64 && (spins & 63) == 0) {
                const unsigned tl = ld_vol(&c->t_tail);
                const int ou = ld_vol(&c->outstanding);
                if (tl != seen_tail || ou != seen_out) {
                    seen_tail = tl;
                    seen_out = ou;
                    t0 = gtimer();
                } else if (gtimer() - t0 > wait_limit(c)) {
                    set_dev_error(c, DC_DEV_ERR_TIMEOUT, 5);
                    *ticket = kNoTicket;
                    state = 2;
                    break;
                }
            }
            if (spins > 16) __nanosleep(spins > 256 ? 256 : 32);
        }
    }
    state = __shfl_sync(0xFFFFFFFFu, state, 0);
    it = __shfl_sync(0xFFFFFFFFu, it, 0);
    __threadfence();
    *item = it;
    return state == 1;
}

// ---------------------------------------------------------------------------
// Steps without a barrier.  A step (level or row) is over when every block has
// reported its seeding and every item is finished; no warp works on it any
// more then, so the one that finished last prepares the next step itself and
// publishes it in step_word, and the others, which wait for items, see the
// word change and start it.  Nothing arrives at a barrier: a grid barrier per
// step cost its arrival and release round trips on top of the queue's own
// termination (an empty step took 16-17 us with 296 blocks, 10 this way).
//   - t_work holds the queue's tail (low 33 bits) and the number of unfinished
//     producers and items (high 31 bits) in one word: a push is one atomic,
//     and the count can never lag behind the items it covers
//   - counters that belong to a step carry its number, so none is reset
//     between steps
//   - one warp of each block polls one of the copies of the step word and
//     passes it on through shared memory (2,368 pollers of one line kept its
//     L2 slice busy for longer than the light steps last)
//   - a warp keeps its ticket from one step to the next (a ticket dropped by
//     one warp while another advances the step would lose an item), and items
//     carry their step: a warp that finds an item of a newer step in its slot
//     has not started that step yet and leaves the item there until it has
// Memory order: atomics on different addresses are not ordered by themselves,
// not even by a result that was waited for.  Whatever a warp did in a step is
// released by the subtraction on t_work that reports it; the one that ends the
// step acquires all of it with a fence, reads the step's counters, and releases
// the next step with the fence before its words; the polling warp acquires the
// word and hands it on inside the block with fences of the block's scope.
// (Without the release the end of a step could be seen before its bound, and a
// peel ended early or a row was jumped, about once in 5,000 decompositions
// while other kernels kept L2 busy.)  Acquire loads cost no more than relaxed
// ones here (327 clocks), a fence 280-900, so readers acquire, and a writer
// fences once, between its value and whatever makes another warp look at it.
// ---------------------------------------------------------------------------
constexpr int kWorkShift = 33;

__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void fence_acq_rel() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
// Atomic addition after everything this thread wrote, or saw from its warp or
// block through their barriers, is performed.
__device__ __forceinline__ unsigned long long add_release(unsigned long long* p, unsigned long long x) {
    unsigned long long v;
    asm volatile("atom.add.release.gpu.global.u64 %0, [%1], %2;" : "=l"(v) : "l"(p), "l"(x) : "memory");
    return v;
}

__device__ __forceinline__ int step_level(unsigned long long w) { return (int)(uint32_t)w; }
__device__ __forceinline__ unsigned step_number(unsigned long long w) { return (unsigned)(w >> 32); }
// 9 bits above 32 bits of payload and 22 of detail; the top bit stays 0, so
// no item equals kEmptyItem
__device__ __forceinline__ unsigned long long step_tag(unsigned long long w) { return ((w >> 32) & 0x1FFull) << 54; }

constexpr unsigned long long kStopWord = ~0ull;  // the block leaves (error or wait limit)
constexpr int kNoBound = 0x7FFFFFFF;

// Shared state of a block.
struct StepBlock {
    unsigned long long word;  // the step word as the polling warp saw it last
    unsigned done;            // warps that finished their seeding share
    int bound;                // least next level they found
    unsigned worked;          // one of them found work that is not in the queue
    unsigned count[2];        // fused peel: vertices they removed
};
// All threads, at kernel start.
__device__ __forceinline__ void step_block_init(StepBlock* b, const EngineCtl* c) {
    if (threadIdx.x == 0) {
        b->word = ld_acquire(&c->step_word[blockIdx.x % kStepWords].v);
        b->done = 0;
        b->bound = kNoBound;
        b->worked = 0;
        b->count[0] = b->count[1] = 0;
    }
    __syncthreads();
}
__device__ __forceinline__ unsigned long long step_block_word(const StepBlock* b) {
    return *reinterpret_cast<const volatile unsigned long long*>(&b->word);
}

// One thread (after a warp barrier): n producers or items of step `word` are
// finished; the last one advances the step.  next(c, level, worked, bound): the next level;
// next.begin(step): the blocks that seed that step, before it is published.
template <typename Next>
__device__ __forceinline__ void step_finish(EngineCtl* c, int n, unsigned long long word, const Next& next) {
    const unsigned long long old = add_release(&c->t_work, 0ull - ((unsigned long long)n << kWorkShift));
    if ((old >> kWorkShift) != (unsigned long long)n) return;
    fence_acq_rel();
    const unsigned step = step_number(word);
    const unsigned tail = (unsigned)old;
    const unsigned tail0 = ld_vol(&c->trace_tail0);
    const unsigned long long low = *reinterpret_cast<const volatile unsigned long long*>(&c->next_low);
    const bool worked = tail != tail0 || ld_vol(&c->worked) == step;
    const int bound = (unsigned)(low >> 32) == step ? kNoBound - (int)(uint32_t)low : kNoBound;
    const int level = next(c, step_level(word), worked, bound);
    if (c->trace) {
        const unsigned long long now = gtimer();
        const unsigned st = step - 1;
        if (st < c->trace_cap) {
            c->trace[8 * st + 1] = now;
            c->trace[8 * st + 2] = tail - tail0;
            c->trace[8 * st + 3] = now;
        }
        if (st + 1 < c->trace_cap) {
            c->trace[8 * (st + 1)] = now;
            c->trace[8 * (st + 1) + 6] = ~0ull;
        }
    }
    c->step = (int)step;
    c->trace_tail0 = tail;
    atomicAdd(&c->t_work, (unsigned long long)next.begin(step + 1) << kWorkShift);
    __threadfence();
    const unsigned long long w = ((unsigned long long)(step + 1) << 32) | (unsigned long long)(uint32_t)level;
#pragma unroll
    for (int i = 0; i < kStepWords; ++i) *reinterpret_cast<volatile unsigned long long*>(&c->step_word[i].v) = w;
}

// Converged warp: its seeding share of the step is done; bound (any lane's):
// no level below it can have work that this warp saw; worked: it found work
// (queued items say so by themselves).  The last warp of a block reports the
// block.
template <typename Next>
__device__ __forceinline__ void step_seeded(EngineCtl* c, StepBlock* b, int bound, bool worked,
                                            unsigned long long word, bool tracing, const Next& next) {
    bound = __reduce_min_sync(0xFFFFFFFFu, bound);
    __syncwarp();
    if ((threadIdx.x & 31u) == 0) {
        if (bound != kNoBound) atomicMin(&b->bound, bound);
        if (worked) atomicOr(&b->worked, 1u);
        __threadfence_block();
        if (atomicAdd(&b->done, 1u) == (blockDim.x >> 5) - 1) {
            b->done = 0;
            __threadfence_block();
            const int m = atomicExch(&b->bound, kNoBound);
            const unsigned step = step_number(word);
            if (atomicExch(&b->worked, 0u)) atomicMax(&c->worked, step);
            for (int i = 0; i < 2; ++i)
                if (const unsigned k = atomicExch(&b->count[i], 0u)) atomicAdd(&c->removed[i], k);
            if (tracing && step - 1 < c->trace_cap) atomicMax(&c->trace[8 * (step - 1) + 5], gtimer());
            if (m != kNoBound)
                atomicMax(&c->next_low, ((unsigned long long)step << 32) | (unsigned long long)(kNoBound - m));
            step_finish(c, 1, word, next);
        }
    }
    __syncwarp();
}

// Converged warp, while the step is being seeded: an item kept by the warp
// counts like a queued one (before the block's report, which another warp may
// make).  The warp reports work with its share (step_seeded).
__device__ __forceinline__ void step_count_kept(EngineCtl* c) {
    if ((threadIdx.x & 31u) == 0) {
        atomicAdd(&c->t_work, 1ull << kWorkShift);
        fence_acq_rel();
    }
    __syncwarp();
}

// Start of a step in the optional trace (one thread per block).
__device__ __forceinline__ void trace_wake(EngineCtl* c, unsigned long long word) {
    const unsigned st = step_number(word) - 1;
    if (st < c->trace_cap) {
        const unsigned long long now = gtimer();
        atomicMax(&c->trace[8 * st + 4], now);
        atomicMin(&c->trace[8 * st + 6], now);
    }
}

// Converged warp: reserves `total` slots for items (lane 0's value counts);
// returns the first one's number on every lane.
__device__ __forceinline__ unsigned step_reserve(EngineCtl* c, unsigned total) {
    unsigned base = 0;
    if ((threadIdx.x & 31u) == 0)
        base = (unsigned)atomicAdd(&c->t_work, ((unsigned long long)total << kWorkShift) | total);
    return __shfl_sync(0xFFFFFFFFu, base, 0);
}
__device__ __forceinline__ void step_put(TicketQueue q, unsigned at, unsigned long long item) {
    *reinterpret_cast<volatile unsigned long long*>(&q.slots[at & q.mask]) = item;
}
// Converged warp: lanes with pred push one item each.
__device__ __forceinline__ void step_push(EngineCtl* c, TicketQueue q, bool pred, unsigned long long item) {
    const unsigned m = __ballot_sync(0xFFFFFFFFu, pred);
    if (!m) return;
    const unsigned base = step_reserve(c, __popc(m));
    if (pred) step_put(q, base + __popc(m & ((1u << (threadIdx.x & 31u)) - 1u)), item);
}

// Converged warp: the next item (kTakeItem, *item), or the start of the next
// step (kTakeStep, *word updated), or kTakeStop after an error.  *pending
// (lane 0): items this warp finished and has not counted off; they are
// counted off before the warp waits.
enum : int { kTakeItem = 1, kTakeStep = 2, kTakeStop = 3 };
template <typename Next>
__device__ __forceinline__ int step_take(EngineCtl* c, TicketQueue q, StepBlock* b, unsigned* ticket,
                                         unsigned long long* item, int* pending, unsigned long long* word,
                                         const Next& next) {
    const unsigned lane = threadIdx.x & 31u;
    unsigned long long it = kEmptyItem, w = *word;
    int state = 0;
    __syncwarp();
    if (lane == 0) {
        const bool poller = threadIdx.x == 0;
        if (*ticket == kNoTicket) *ticket = atomicAdd(&c->t_head, 1u);
        unsigned long long* s = &q.slots[*ticket & q.mask];
        const unsigned long long tag = step_tag(w) >> 54;
        it = ld_acquire(s);
        if (it == kEmptyItem && *pending > 0) {
            step_finish(c, *pending, w, next);
            *pending = 0;
        }
        unsigned long long t0 = 0, seen = 0;
        unsigned spins = 0;
        while ((it >> 54) != tag) {
            if (poller) {
                w = ld_acquire(&c->step_word[blockIdx.x % kStepWords].v);
                if ((++spins & 15u) == 0) {
                    // the limit bounds a wait without progress: while the
                    // step's other warps still push or finish items the clock
                    // restarts
                    const unsigned long long tw = *reinterpret_cast<volatile unsigned long long*>(&c->t_work);
                    if (ld_vol(&c->error)) {
                        w = kStopWord;
                    } else if (spins == 64 || tw != seen) {
                        seen = tw;
                        t0 = gtimer();
                    } else if (spins > 64 && gtimer() - t0 > wait_limit(c)) {
                        set_dev_error(c, DC_DEV_ERR_TIMEOUT, 5);
                        w = kStopWord;
                    }
                }
                if (w != *word) {
                    __threadfence_block();
                    *reinterpret_cast<volatile unsigned long long*>(&b->word) = w;
                }
            } else {
                w = step_block_word(b);
                ++spins;
            }
            if (w != *word) break;
            if (!poller) __nanosleep(spins > 16 ? 200 : 100);
            it = ld_acquire(s);
        }
        if ((it >> 54) == tag) {
            *reinterpret_cast<volatile unsigned long long*>(s) = kEmptyItem;
            *ticket = kNoTicket;
            state = kTakeItem;
        } else {
            __threadfence_block();
            state = w == kStopWord ? kTakeStop : kTakeStep;
        }
    }
    __syncwarp();
    state = __shfl_sync(0xFFFFFFFFu, state, 0);
    if (state == kTakeItem) it = __shfl_sync(0xFFFFFFFFu, it, 0);
    else w = __shfl_sync(0xFFFFFFFFu, w, 0);
    *item = it;
    *word = w;
    return state;
}

}  // namespace dc
