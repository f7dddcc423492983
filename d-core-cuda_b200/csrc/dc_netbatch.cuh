// A maintenance batch's net effect in device memory (dc_netbatch.cu).
#pragma once
#include <cstdint>

#include "dc_engine.cuh"
#include "dc_internal.h"

namespace dc {

struct DeviceBatch {
    // distinct deleted pairs with their counts, and inserted entries (one per
    // occurrence), in edge order
    uint32_t n_pairs = 0, n_del = 0, n_ins = 0;
    uint32_t *del_u = nullptr, *del_v = nullptr;
    int32_t* del_n = nullptr;
    uint32_t *ins_u = nullptr, *ins_v = nullptr;
    // deleted entries grouped by list, side 0 out-lists, side 1 in-lists:
    // entry t takes gnbr[t] out of the list of gof[t]; group g holds entries
    // goff[g] .. goff[g + 1] of list gvert[g]
    uint32_t ngroups[2] = {0, 0};
    uint32_t *gvert[2] = {nullptr, nullptr}, *goff[2] = {nullptr, nullptr};
    uint32_t *gof[2] = {nullptr, nullptr}, *gnbr[2] = {nullptr, nullptr};
};

// Net effect of b updates (vertex ids checked by the caller) on the handle's
// stream; the arrays belong to *out until device_batch_free.
int net_batch_device(dc_graph* h, const uint32_t* pairs, const uint8_t* is_del, uint64_t b, DeviceBatch* out);
void device_batch_free(dc_graph* h, DeviceBatch* d);

// Stable sort of (key, val) by the low `bits` bits of key on stream st
// (dc_partition.cu); the sorted arrays end up in *key, *val (the pairs of
// pointers are exchanged as needed); cnt holds radix_count_words(m) words of
// some m >= n.
void radix_sort_pairs(cudaStream_t st, uint64_t n, int bits, uint32_t** key, uint32_t** val, uint32_t** key2,
                      uint32_t** val2, uint32_t* cnt);
uint64_t radix_count_words(uint64_t n);

}  // namespace dc
