// Net effect of a large maintenance batch on the GPU: what net_batch and
// group_by (dc_maint.cu) compute on the host for small ones.  A batch has
// sequential semantics and is applied as its net effect per edge (insertions
// minus deletions), with the deletions grouped by list on both sides.
//   1. stable radix sort of the operations by (source, destination)
//   2. runs of equal edges, the net count of each
//   3. one scan over the runs places distinct deleted pairs, deleted entries
//      and inserted entries (all in edge order, as the host's)
//   4. deleted entries grouped by source as they are, and by destination after
//      a stable sort by it
// The host sorted and grouped 250,000 operations in 40 ms, half of such a
// batch at R-MAT 22; this takes about 1 ms.
#include <algorithm>
#include <atomic>
#include <cstdint>

#include "dc_netbatch.cuh"

namespace dc {
extern std::atomic<unsigned long long> g_launches;

namespace {

constexpr int kNT = 256;               // threads per block
constexpr int kNItems = 8;             // consecutive items per thread
constexpr int kNTile = kNT * kNItems;  // items per block

struct Sum3 {
    uint32_t a, b, c;
};

__device__ __forceinline__ Sum3 warp_incl(Sum3 x) {
    const unsigned lane = threadIdx.x & 31u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t ya = __shfl_up_sync(0xFFFFFFFFu, x.a, o), yb = __shfl_up_sync(0xFFFFFFFFu, x.b, o),
                       yc = __shfl_up_sync(0xFFFFFFFFu, x.c, o);
        if (lane >= (unsigned)o) {
            x.a += ya;
            x.b += yb;
            x.c += yc;
        }
    }
    return x;
}
// Exclusive scan over the block's threads; *total: the block's sum.
__device__ Sum3 block_excl(Sum3 x, Sum3* total) {
    __shared__ Sum3 s_w[kNT / 32 + 1];
    const unsigned lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    const Sum3 inc = warp_incl(x);
    if (lane == 31) s_w[w] = inc;
    __syncthreads();
    if (threadIdx.x == 0) {
        Sum3 run{0, 0, 0};
        for (int i = 0; i < kNT / 32; ++i) {
            const Sum3 t = s_w[i];
            s_w[i] = run;
            run.a += t.a;
            run.b += t.b;
            run.c += t.c;
        }
        s_w[kNT / 32] = run;
    }
    __syncthreads();
    const Sum3 r{inc.a - x.a + s_w[w].a, inc.b - x.b + s_w[w].b, inc.c - x.c + s_w[w].c};
    *total = s_w[kNT / 32];
    __syncthreads();
    return r;
}
// Exclusive scan of part[0 .. n) in place by one block; part[n] = total.
__global__ void k_nb_scan_parts(Sum3* part, uint32_t n) {
    Sum3 carry{0, 0, 0};
    for (uint32_t b = 0; b < n; b += kNT) {
        const uint32_t i = b + threadIdx.x;
        const Sum3 x = i < n ? part[i] : Sum3{0, 0, 0};
        Sum3 tot;
        const Sum3 ex = block_excl(x, &tot);
        if (i < n) part[i] = Sum3{ex.a + carry.a, ex.b + carry.b, ex.c + carry.c};
        carry.a += tot.a;
        carry.b += tot.b;
        carry.c += tot.c;
    }
    if (threadIdx.x == 0) part[n] = carry;
}

__global__ void k_nb_load(uint32_t n, const uint32_t* pairs, uint32_t* key, uint32_t* val) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        key[i] = pairs[2 * (uint64_t)i + 1];
        val[i] = i;
    }
}
// keys of the second sort: the sources, in the order of the first
__global__ void k_nb_source(uint32_t n, const uint32_t* pairs, const uint32_t* val, uint32_t* key) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        key[i] = pairs[2 * (uint64_t)val[i]];
}

// Whether sorted operation i starts a run of equal edges.
__device__ __forceinline__ bool run_start(uint32_t i, const uint32_t* pairs, const uint32_t* key, const uint32_t* val) {
    return i == 0 || key[i] != key[i - 1] ||
           pairs[2 * (uint64_t)val[i] + 1] != pairs[2 * (uint64_t)val[i - 1] + 1];
}
__global__ void k_nb_run_count(uint32_t n, const uint32_t* pairs, const uint32_t* key, const uint32_t* val, Sum3* part) {
    const uint32_t t0 = blockIdx.x * kNTile + threadIdx.x * kNItems;
    Sum3 s{0, 0, 0};
    for (int j = 0; j < kNItems; ++j)
        if (t0 + j < n) s.a += run_start(t0 + j, pairs, key, val);
    Sum3 tot;
    block_excl(s, &tot);
    if (threadIdx.x == 0) part[blockIdx.x] = tot;
}
// first[r] = operation that starts run r; net[r] += insertions - deletions
__global__ void k_nb_runs(uint32_t n, const uint32_t* pairs, const uint8_t* is_del, const uint32_t* key,
                          const uint32_t* val, const Sum3* part, uint32_t* first, int32_t* net) {
    const uint32_t t0 = blockIdx.x * kNTile + threadIdx.x * kNItems;
    Sum3 s{0, 0, 0};
    for (int j = 0; j < kNItems; ++j)
        if (t0 + j < n) s.a += run_start(t0 + j, pairs, key, val);
    Sum3 tot;
    uint32_t r = block_excl(s, &tot).a + part[blockIdx.x].a;  // runs started before this thread's items
    for (int j = 0; j < kNItems; ++j) {
        const uint32_t i = t0 + j;
        if (i >= n) break;
        if (run_start(i, pairs, key, val)) first[r++] = i;
        atomicAdd(&net[r - 1], is_del && is_del[val[i]] ? -1 : 1);
    }
}
__global__ void k_nb_net_count(const Sum3* n_runs, const int32_t* net, Sum3* part) {
    const uint32_t n = n_runs->a, t0 = blockIdx.x * kNTile + threadIdx.x * kNItems;
    Sum3 s{0, 0, 0};
    for (int j = 0; j < kNItems; ++j)
        if (t0 + j < n) {
            const int32_t x = net[t0 + j];
            s.a += x < 0;
            s.b += (uint32_t)max(-x, 0);
            s.c += (uint32_t)max(x, 0);
        }
    Sum3 tot;
    block_excl(s, &tot);
    if (threadIdx.x == 0) part[blockIdx.x] = tot;
}
__global__ void k_nb_emit(const Sum3* n_runs, const uint32_t* pairs, const uint32_t* val, const uint32_t* first,
                          const int32_t* net, const Sum3* part, uint32_t* del_u, uint32_t* del_v, int32_t* del_n,
                          uint32_t* occ_u, uint32_t* occ_v, uint32_t* ins_u, uint32_t* ins_v) {
    const uint32_t n = n_runs->a, t0 = blockIdx.x * kNTile + threadIdx.x * kNItems;
    Sum3 s{0, 0, 0};
    for (int j = 0; j < kNItems; ++j)
        if (t0 + j < n) {
            const int32_t x = net[t0 + j];
            s.a += x < 0;
            s.b += (uint32_t)max(-x, 0);
            s.c += (uint32_t)max(x, 0);
        }
    Sum3 tot;
    Sum3 at = block_excl(s, &tot);
    at.a += part[blockIdx.x].a;
    at.b += part[blockIdx.x].b;
    at.c += part[blockIdx.x].c;
    for (int j = 0; j < kNItems; ++j) {
        const uint32_t r = t0 + j;
        if (r >= n) break;
        const int32_t x = net[r];
        if (!x) continue;
        const uint32_t e = val[first[r]], u = pairs[2 * (uint64_t)e], v = pairs[2 * (uint64_t)e + 1];
        if (x < 0) {
            del_u[at.a] = u;
            del_v[at.a] = v;
            del_n[at.a++] = -x;
            for (int32_t k = 0; k < -x; ++k, ++at.b) {
                occ_u[at.b] = u;
                occ_v[at.b] = v;
            }
        } else {
            for (int32_t k = 0; k < x; ++k, ++at.c) {
                ins_u[at.c] = u;
                ins_v[at.c] = v;
            }
        }
    }
}

// Groups of equal consecutive keys: gvert[g], goff[g], goff[number of groups] = n.
__global__ void k_nb_group_count(uint32_t n, const uint32_t* key, Sum3* part) {
    const uint32_t t0 = blockIdx.x * kNTile + threadIdx.x * kNItems;
    Sum3 s{0, 0, 0};
    for (int j = 0; j < kNItems; ++j) {
        const uint32_t i = t0 + j;
        if (i < n) s.a += i == 0 || key[i] != key[i - 1];
    }
    Sum3 tot;
    block_excl(s, &tot);
    if (threadIdx.x == 0) part[blockIdx.x] = tot;
}
__global__ void k_nb_groups(uint32_t n, const uint32_t* key, const Sum3* part, uint32_t* gvert, uint32_t* goff) {
    const uint32_t t0 = blockIdx.x * kNTile + threadIdx.x * kNItems;
    Sum3 s{0, 0, 0};
    for (int j = 0; j < kNItems; ++j) {
        const uint32_t i = t0 + j;
        if (i < n) s.a += i == 0 || key[i] != key[i - 1];
    }
    Sum3 tot;
    uint32_t g = block_excl(s, &tot).a + part[blockIdx.x].a;
    for (int j = 0; j < kNItems; ++j) {
        const uint32_t i = t0 + j;
        if (i < n && (i == 0 || key[i] != key[i - 1])) {
            gvert[g] = key[i];
            goff[g++] = i;
        }
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) goff[part[gridDim.x].a] = n;
}
__global__ void k_nb_take(uint32_t n, const uint32_t* from, const uint32_t* val, uint32_t* to) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) to[i] = from[val[i]];
}
__global__ void k_nb_iota(uint32_t n, const uint32_t* from, uint32_t* key, uint32_t* val) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        key[i] = from[i];
        val[i] = i;
    }
}

template <typename T>
int nb_alloc(cudaStream_t st, T** p, uint64_t n) {
    if (cudaMallocAsync((void**)p, std::max<uint64_t>(n, 1) * sizeof(T), st) != cudaSuccess) {
        *p = nullptr;
        cudaGetLastError();
        return set_error(DC_ERR_NOMEM, "maintenance batch: device allocation failed");
    }
    return DC_OK;
}

}  // namespace

void device_batch_free(dc_graph* h, DeviceBatch* d) {
    for (void* p : {(void*)d->del_u, (void*)d->del_v, (void*)d->del_n, (void*)d->ins_u, (void*)d->ins_v, (void*)d->gvert[0],
                    (void*)d->gvert[1], (void*)d->goff[0], (void*)d->goff[1], (void*)d->gof[0], (void*)d->gof[1],
                    (void*)d->gnbr[0], (void*)d->gnbr[1]})
        if (p) cudaFreeAsync(p, h->stream);
    *d = DeviceBatch();
}

int net_batch_device(dc_graph* h, const uint32_t* pairs, const uint8_t* is_del, uint64_t b, DeviceBatch* out) {
    *out = DeviceBatch();
    if (b == 0 || b >= (1ull << 30)) return set_error(DC_ERR_INVALID, "net_batch_device: batch size");
    cudaStream_t st = h->stream;
    const uint32_t V = h->g.V, n = (uint32_t)b;
    const int bits = V > 1 ? 32 - __builtin_clz(V - 1) : 1;
    const uint32_t tiles = (n + kNTile - 1) / kNTile;
    const int grid = (int)std::min<uint32_t>((n + kNT - 1) / kNT, (uint32_t)h->geom.sms * 8);
    uint32_t *d_pairs = nullptr, *key = nullptr, *val = nullptr, *key2 = nullptr, *val2 = nullptr, *cnt = nullptr,
             *first = nullptr;
    uint8_t* d_del = nullptr;
    int32_t* net = nullptr;
    Sum3 *part = nullptr, *part2 = nullptr;
    auto release = [&]() {
        for (void* p : {(void*)d_pairs, (void*)key, (void*)val, (void*)key2, (void*)val2, (void*)cnt, (void*)first,
                        (void*)d_del, (void*)net, (void*)part, (void*)part2})
            if (p) cudaFreeAsync(p, st);
    };
    DeviceBatch& d = *out;
    int rc = DC_OK;
    auto fail = [&](int code) {
        release();
        device_batch_free(h, out);
        return code;
    };
    if ((rc = nb_alloc(st, &d_pairs, 2ull * n)) || (is_del && (rc = nb_alloc(st, &d_del, n))) ||
        (rc = nb_alloc(st, &key, n)) || (rc = nb_alloc(st, &val, n)) || (rc = nb_alloc(st, &key2, n)) ||
        (rc = nb_alloc(st, &val2, n)) || (rc = nb_alloc(st, &cnt, radix_count_words(n))) ||
        (rc = nb_alloc(st, &first, n)) || (rc = nb_alloc(st, &net, n)) || (rc = nb_alloc(st, &part, tiles + 1)) ||
        (rc = nb_alloc(st, &part2, tiles + 1)) || (rc = nb_alloc(st, &d.del_u, n)) || (rc = nb_alloc(st, &d.del_v, n)) ||
        (rc = nb_alloc(st, &d.del_n, n)) || (rc = nb_alloc(st, &d.ins_u, n)) || (rc = nb_alloc(st, &d.ins_v, n)) ||
        (rc = nb_alloc(st, &d.gof[0], n)) || (rc = nb_alloc(st, &d.gnbr[0], n)))
        return fail(rc);
    bool ok = cudaMemcpyAsync(d_pairs, pairs, 8ull * n, cudaMemcpyHostToDevice, st) == cudaSuccess &&
              (!is_del || cudaMemcpyAsync(d_del, is_del, n, cudaMemcpyHostToDevice, st) == cudaSuccess) &&
              cudaMemsetAsync(net, 0, 4ull * n, st) == cudaSuccess;
    if (!ok) return fail(set_error(DC_ERR_CUDA, "maintenance batch: upload failed"));
    g_launches += 8;
    k_nb_load<<<grid, kNT, 0, st>>>(n, d_pairs, key, val);
    radix_sort_pairs(st, n, bits, &key, &val, &key2, &val2, cnt);
    k_nb_source<<<grid, kNT, 0, st>>>(n, d_pairs, val, key);
    radix_sort_pairs(st, n, bits, &key, &val, &key2, &val2, cnt);
    k_nb_run_count<<<tiles, kNT, 0, st>>>(n, d_pairs, key, val, part);
    k_nb_scan_parts<<<1, kNT, 0, st>>>(part, tiles);
    k_nb_runs<<<tiles, kNT, 0, st>>>(n, d_pairs, d_del, key, val, part, first, net);
    k_nb_net_count<<<tiles, kNT, 0, st>>>(part + tiles, net, part2);
    k_nb_scan_parts<<<1, kNT, 0, st>>>(part2, tiles);
    k_nb_emit<<<tiles, kNT, 0, st>>>(part + tiles, d_pairs, val, first, net, part2, d.del_u, d.del_v, d.del_n, d.gof[0],
                                     d.gnbr[0], d.ins_u, d.ins_v);
    Sum3 tot{0, 0, 0};
    if (cudaMemcpyAsync(&tot, part2 + tiles, sizeof(tot), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return fail(set_error(DC_ERR_CUDA, "maintenance batch: %s", cudaGetErrorString(cudaGetLastError())));
    d.n_pairs = tot.a;
    d.n_del = tot.b;
    d.n_ins = tot.c;
    if (d.n_del) {
        const uint32_t m = d.n_del, mt = (m + kNTile - 1) / kNTile;
        const int mg = (int)std::min<uint32_t>((m + kNT - 1) / kNT, (uint32_t)h->geom.sms * 8);
        if ((rc = nb_alloc(st, &d.gof[1], m)) || (rc = nb_alloc(st, &d.gnbr[1], m))) return fail(rc);
        for (int side = 0; side < 2; ++side)
            if ((rc = nb_alloc(st, &d.gvert[side], m)) || (rc = nb_alloc(st, &d.goff[side], m + 1ull))) return fail(rc);
        // by destination: the entries in edge order, stably sorted
        g_launches += 8;
        k_nb_iota<<<mg, kNT, 0, st>>>(m, d.gnbr[0], key, val);
        radix_sort_pairs(st, m, bits, &key, &val, &key2, &val2, cnt);
        k_nb_take<<<mg, kNT, 0, st>>>(m, d.gof[0], val, d.gnbr[1]);
        cudaMemcpyAsync(d.gof[1], key, 4ull * m, cudaMemcpyDeviceToDevice, st);
        Sum3 ng[2];
        for (int side = 0; side < 2; ++side) {
            Sum3* pt = side == 0 ? part : part2;
            k_nb_group_count<<<mt, kNT, 0, st>>>(m, d.gof[side], pt);
            k_nb_scan_parts<<<1, kNT, 0, st>>>(pt, mt);
            k_nb_groups<<<mt, kNT, 0, st>>>(m, d.gof[side], pt, d.gvert[side], d.goff[side]);
            cudaMemcpyAsync(&ng[side], pt + mt, sizeof(Sum3), cudaMemcpyDeviceToHost, st);
        }
        if (cudaStreamSynchronize(st) != cudaSuccess)
            return fail(set_error(DC_ERR_CUDA, "maintenance batch: %s", cudaGetErrorString(cudaGetLastError())));
        d.ngroups[0] = ng[0].a;
        d.ngroups[1] = ng[1].a;
    }
    release();
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        device_batch_free(h, out);
        return set_error(DC_ERR_CUDA, "maintenance batch: %s", cudaGetErrorString(e));
    }
    return DC_OK;
}

}  // namespace dc
