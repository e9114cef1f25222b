// cluster_sort.cuh — stable sort of up to 131,072 particles (or given keys) by
// one thread-block cluster, in one launch.
//
// The onesweep sort (radix_sort.cuh) takes thirteen graph nodes per step: two
// clears, two key kernels, the plan and one launch per digit, active or not.
// Below some 100,000 keys each of them is a launch with a few microseconds of
// latency and hardly any work. Here up to 16 thread blocks of 1024 threads hold
// the keys: every digit pass ranks them in the blocks, exchanges the blocks'
// digit counts and scatters keys and indices through distributed shared
// memory, with two hardware cluster barriers per pass and nothing in global
// memory but the input and the permutation. No wait is polled.
//
// Only key bits that decide an order are sorted, packed into 32-bit words: the
// 63-bit Morton keys of a scene of 32 cells per axis hold 15 to 18 of them.
//
// What bounds it: barrier and shared-memory latency up to some 16 k keys, the
// 16 SMs' scatter above. The variants of 4, 6 and 8 items per thread (above 49,152
// keys) keep the full keys in registers until the deciding bits are known and
// spill 20, 132 and 256 bytes at their 64 registers. Device time of keys + sort + hash clear, against the
// kernels it replaced: 2 k particles 13 us (53), 33 k 18 (61), 79 k 32 (61);
// 65,536 given keys with 24 deciding bits 28 us (three passes of 8 us).
#pragma once
#include "sph_common.cuh"

namespace wcsph {

constexpr u32 CLUSTER_SORT_MAX = 131072u;

struct ClusterSortArgs {
    // input: positions (with `scene`: the batched keys), or keys when pos is null
    const float4* pos;
    const u32* scene;
    const u64* keys_in;
    u32 n;
    float cs;
    u64* keys_out;      // positions: the full keys in input order (nullptr: not wanted)
    u32* perm;          // sorted -> input index
    // step bookkeeping (nullptr / 0: none): sort_sel names perm as the first
    // index buffer, the unit list is emptied, the cell hash is cleared
    DevState* st;
    u64* table;
    u32 table_size;
};

// Enqueues the sort on `stream`. *launched = false, and nothing is enqueued,
// where it does not apply: too many keys, a device on which the cluster does not
// fit, or a test hook of the onesweep is on (its waits, or its results at sizes
// that the cluster takes).
cudaError_t enqueue_cluster_sort(const ClusterSortArgs& a, cudaStream_t stream, bool* launched);

}  // namespace wcsph
