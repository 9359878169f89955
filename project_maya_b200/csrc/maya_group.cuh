// maya_group.cuh - the grouping of a window's plan entries by expert, by one block.
#pragma once

#include "maya_common.cuh"

namespace maya {

struct GroupOut {
    unsigned long long* ptr;     // [groups] blob address
    int* start;                  // [groups + 1] entry ranges
    int* ent;                    // [entries] entry numbers, a group's side by side in ascending order
    int* n_groups;
};
struct GroupShared {
    alignas(16) unsigned long long ptr[128];
    int start[128], leaders[4], entries[4];
};

// Entries i < n <= 128 (i = 8 token + slot) with a non-zero blob address p are grouped by address: groups in order of first
// appearance, members in ascending i.  Thread i < 128 brings p (0: no entry); the whole block calls (at least 128 threads).
// Every entry compares itself with all the others - independent shared-memory reads, two to a load - instead of walking to its
// first match and then scanning counts (9.4 us for 16 tokens, one dependent read after another).
__device__ __forceinline__ void group_entries(unsigned long long p, int n, const GroupOut& G, GroupShared& sh) {
    const int i = threadIdx.x, lane = i & 31, warp = i >> 5;
    if (i < 128) sh.ptr[i] = i < n ? p : 0ull;
    __syncthreads();
    int cnt = 0, rank = 0, first = 128;
    bool leader = false;
    unsigned lead_mask = 0u;
    int incl = 0;
    if (i < 128) {
        p = sh.ptr[i];
        const ulonglong2* s2 = (const ulonglong2*) sh.ptr;
#pragma unroll 8
        for (int f = 0; f < (n + 1) / 2; ++f) {
            const ulonglong2 o = s2[f];
            const int a = o.x == p, b = o.y == p;
            cnt += a + b;
            rank += (a && 2 * f < i) + (b && 2 * f + 1 < i);
            first = min(first, a ? 2 * f : b ? 2 * f + 1 : 128);
        }
        leader = p != 0ull && first == i;
        lead_mask = __ballot_sync(0xffffffffu, leader);
        incl = leader ? cnt : 0;                     // entries of the groups led up to here
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) { sh.leaders[warp] = __popc(lead_mask); sh.entries[warp] = incl; }
    }
    __syncthreads();
    if (i < 128) {
        int g0 = 0, e0 = 0;
        for (int w = 0; w < warp; ++w) { g0 += sh.leaders[w]; e0 += sh.entries[w]; }
        if (leader) {
            const int g = g0 + __popc(lead_mask & ((1u << lane) - 1u)), s = e0 + incl - cnt;
            sh.start[i] = s;
            G.ptr[g] = p;
            G.start[g] = s;
        }
        if (i == 0) {
            const int ng = sh.leaders[0] + sh.leaders[1] + sh.leaders[2] + sh.leaders[3];
            G.start[ng] = sh.entries[0] + sh.entries[1] + sh.entries[2] + sh.entries[3];
            *G.n_groups = ng;
        }
    }
    __syncthreads();
    if (i < 128 && p != 0ull) G.ent[sh.start[first] + rank] = i;
}

}  // namespace maya
