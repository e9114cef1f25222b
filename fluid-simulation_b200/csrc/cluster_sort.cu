// cluster_sort.cu — see cluster_sort.cuh for the design.
#include "cluster_sort.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>

#include "radix_sort.cuh"
#include "radix_sort_dev.cuh"

namespace cg = cooperative_groups;

namespace wcsph {

namespace {

constexpr u32 CS_THREADS = 1024;
constexpr u32 CS_WARPS = CS_THREADS / 32;
constexpr u32 CS_MAX_BLOCKS = 16;   // a non-portable cluster size (24 bits of 32,768 keys: 23 us; 8 blocks 32, 4 blocks 54)

enum SortInput : int { SORT_SCENE = 0, SORT_BATCH = 1, SORT_KEYS = 2 };

template <int IPT>
struct ClusterSmem {
    static constexpr u32 items = CS_THREADS * IPT;
    u64 recv[items];           // the block's items (key << 32 | index), written by all blocks
    u32 wcnt[CS_WARPS][256];   // per warp: digit counts, then exclusive prefixes over the warps
    u32 part[2][4][256];       // partial sums of the four thread groups
    u32 count[2][256];         // the block's digit counts, read by the other blocks (alternating)
    u32 base[256];             // first output rank of each digit of this block
    u32 wsum[8];
    u32 varies[4];             // bits in which the block's keys (and their relations) differ from key 0's
    u32 bits;                  // deciding key bits, and their runs: (key >> src) & mask, moved to dst
    u32 runs;
    u32 src[32], dst[32];
    u64 mask[32];
};

// Lanes of the warp that hold the same 8-bit digit, among the lanes in `among`
// (every lane calls it). Eight ballots instead of match.any, which takes a step
// per distinct value: a pass over random digits 10.4 -> 8 us at 65,536 keys. The
// onesweep tiles keep match.any: between steps their keys come nearly sorted, a
// warp holds a few cells, and the ballots cost 8 us more at 1 M particles.
__device__ __forceinline__ u32 same_digit(u32 d, u32 among) {
    u32 peers = among;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool bit = (d >> b) & 1u;
        const u32 set = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? set : ~set;
    }
    return peers;
}

__device__ __forceinline__ void cluster_barrier(cg::cluster_group& cluster, u32 blocks) {
    if (blocks == 1u) __syncthreads();
    else cluster.sync();
}

// Digit passes over bits [0, bits) of the 32-bit keys held in registers:
// thread t of warp w holds items w * 32 * IPT + k * 32 + lane of its block's
// IPT * 1024, and the blocks' items follow one another. The last pass of the
// last word writes the permutation.
template <int IPT>
__device__ __forceinline__ void cluster_passes(cg::cluster_group& cluster, ClusterSmem<IPT>& S, u32 (&key)[IPT],
                                               u32 (&idx)[IPT], u32 n, u32 bits, bool last_word, u32& parity,
                                               u32* perm) {
    constexpr u32 items = ClusterSmem<IPT>::items;
    const u32 tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const u32 blocks = cluster.num_blocks(), me = cluster.block_rank();
    const u32 mine = warp * (32u * IPT) + lane;            // position of item k in the block: mine + 32 k
    const u32 held = n > me * items ? min(n - me * items, items) : 0u;   // items of this block
    const u32 lt = sortdev::lanemask_lt();
    const u32 dig = tid & 255u, grp = tid >> 8;            // four threads per digit
    for (u32 shift = 0; shift < bits; shift += 8u) {
        const bool last = last_word && shift + 8u >= bits;
        for (u32 t = tid; t < CS_WARPS * 256u / 4u; t += CS_THREADS)
            reinterpret_cast<uint4*>(&S.wcnt[0][0])[t] = make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();
        u32 rank[IPT];
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
            const bool valid = mine + 32u * k < held;
            const u32 d = (key[k] >> shift) & 255u;
            const u32 peers = same_digit(d, __ballot_sync(0xffffffffu, valid));
            const u32 base = valid ? S.wcnt[warp][d] : 0u;
            rank[k] = base + __popc(peers & lt);
            __syncwarp();
            if (valid && (peers >> lane) == 1u) S.wcnt[warp][d] = base + __popc(peers);
            __syncwarp();
        }
        __syncthreads();
        // prefixes over the warps: each of a digit's four threads takes eight warps
        u32 c[8], run = 0;
#pragma unroll
        for (u32 w = 0; w < 8u; ++w) {
            c[w] = run;
            run += S.wcnt[8u * grp + w][dig];
        }
        S.part[0][grp][dig] = run;
        __syncthreads();
        u32 lower = 0, sum = 0;
#pragma unroll
        for (u32 g = 0; g < 4u; ++g) {
            const u32 p = S.part[0][g][dig];
            lower += g < grp ? p : 0u;
            sum += p;
        }
#pragma unroll
        for (u32 w = 0; w < 8u; ++w) S.wcnt[8u * grp + w][dig] = lower + c[w];
        u32 before = 0, total = sum;
        if (blocks > 1u) {
            if (grp == 0) S.count[parity][dig] = sum;
            cluster.sync();   // the blocks' counts are there
            total = 0;
            for (u32 b = grp; b < blocks; b += 4u) {
                const u32 v = *cluster.map_shared_rank(&S.count[parity][dig], b);
                before += b < me ? v : 0u;
                total += v;
            }
            S.part[0][grp][dig] = before;
            S.part[1][grp][dig] = total;
            __syncthreads();
        }
        // first output rank of every digit (threads of the first group)
        u32 incl = 0;
        if (grp == 0) {
            if (blocks > 1u) {
                before = S.part[0][0][dig] + S.part[0][1][dig] + S.part[0][2][dig] + S.part[0][3][dig];
                total = S.part[1][0][dig] + S.part[1][1][dig] + S.part[1][2][dig] + S.part[1][3][dig];
            }
            incl = total;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const u32 t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= static_cast<u32>(o)) incl += t;
            }
            if (lane == 31u) S.wsum[warp] = incl;
        }
        __syncthreads();
        if (grp == 0) {
            u32 low = 0;
#pragma unroll
            for (u32 w = 0; w < 8u; ++w) low += w < warp ? S.wsum[w] : 0u;
            S.base[dig] = low + incl - total + before;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
            if (mine + 32u * k < held) {
                const u32 d = (key[k] >> shift) & 255u;
                const u32 dst = S.base[d] + S.wcnt[warp][d] + rank[k];   // < n: the ranks are a permutation
                if (last) {
                    perm[dst] = idx[k];
                } else {
                    const u32 b = dst / items;
                    *cluster.map_shared_rank(&S.recv[dst - b * items], b) = (static_cast<u64>(key[k]) << 32) | idx[k];
                }
            }
        }
        cluster_barrier(cluster, blocks);   // the scattered items are there; no block leaves while others read its counts
        if (last) return;
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
            const u64 it = S.recv[mine + 32u * k];
            key[k] = static_cast<u32>(it >> 32);
            idx[k] = static_cast<u32>(it);
        }
        parity ^= 1u;
    }
}

template <int IPT, int INPUT>
__global__ void __launch_bounds__(CS_THREADS, 1) cluster_sort_kernel(const ClusterSortArgs a) {
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    ClusterSmem<IPT>& S = *reinterpret_cast<ClusterSmem<IPT>*>(dyn_smem);
    cg::cluster_group cluster = cg::this_cluster();
    const u32 tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const u32 blocks = cluster.num_blocks(), me = cluster.block_rank();
    const u32 n = a.n;
    const u32 first = me * ClusterSmem<IPT>::items + warp * (32u * IPT) + lane;   // item k: first + 32 k
    if (tid < 4u) S.varies[tid] = 0u;
    __syncthreads();

    auto load_key = [&](u32 i) -> u64 {
        if constexpr (INPUT == SORT_KEYS) return a.keys_in[i];
        else if constexpr (INPUT == SORT_BATCH) return batch_key(a.scene[i], cell_of(a.pos[i], a.cs));
        else return morton_key(cell_of(a.pos[i], a.cs));
    };
    const u64 key0 = load_key(0);
    u64 full[IPT];
    u32 idx[IPT];
    u64 diff = 0, rel = 0;
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const u32 i = first + 32u * k;
        idx[k] = i;
        full[k] = key0;
        if (i < n) {
            full[k] = load_key(i);
            if (INPUT != SORT_KEYS && a.keys_out) a.keys_out[i] = full[k];
        }
        const u64 d = full[k] ^ key0;
        diff |= d;
        rel |= d ^ (d >> 3);
    }
    const u32 v[4] = {static_cast<u32>(diff), static_cast<u32>(diff >> 32), static_cast<u32>(rel),
                      static_cast<u32>(rel >> 32)};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const u32 r = __reduce_or_sync(0xffffffffu, v[q]);
        if (lane == 0 && r) atomicOr(&S.varies[q], r);
    }
    // the step's bookkeeping, while the bits are gathered
    if (me == 0 && tid == 0 && a.st) {
        a.st->sort_sel[SORT_DIGITS] = 1u;
        a.st->unit_count = 0;
        a.st->unit_next = 0;
        a.st->thin_count = 0;
        a.st->thin_rows = 0;
    }
    for (u32 t = me * CS_THREADS + tid; t < a.table_size; t += blocks * CS_THREADS) a.table[t] = EMPTY_HASH;
    cluster_barrier(cluster, blocks);
    // A bit decides an order only if it differs between keys and is not the
    // same function (copy or inverse) of the bit three above it in all of
    // them: keys that agree on the higher of the two then agree on both. In
    // Morton keys that drops an axis's copies of its sign.
    if (warp == 0) {   // one warp per block reads the others' masks (lane = block)
        u32 all[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            all[q] = __reduce_or_sync(0xffffffffu, lane < blocks ? *cluster.map_shared_rank(&S.varies[q], lane) : 0u);
        u64 deciding = ((static_cast<u64>(all[1]) << 32) | all[0]) & ((static_cast<u64>(all[3]) << 32) | all[2]);
        if (lane == 0) {
            u32 r = 0, to = 0;
            while (deciding) {
                const u32 src = static_cast<u32>(__ffsll(static_cast<long long>(deciding))) - 1u;
                const u64 rest = ~(deciding >> src);
                const u32 len = rest ? static_cast<u32>(__ffsll(static_cast<long long>(rest))) - 1u : 64u;
                const u64 m = len >= 64u ? ~0ull : (1ull << len) - 1ull;
                S.src[r] = src;
                S.mask[r] = m;
                S.dst[r] = to;
                to += len;
                ++r;
                deciding &= ~(m << src);
            }
            S.runs = r;
            S.bits = to;
        }
    }
    cluster_barrier(cluster, blocks);   // no block leaves (no deciding bit) while others read its masks
    const u32 bits = S.bits;
    auto compressed = [&](u64 k) {
        u64 c = 0;
        for (u32 r = 0; r < S.runs; ++r) c |= ((k >> S.src[r]) & S.mask[r]) << S.dst[r];
        return c;
    };
    if (bits == 0u) {
#pragma unroll
        for (int k = 0; k < IPT; ++k)
            if (idx[k] < n) a.perm[idx[k]] = idx[k];
        return;
    }
    u32 key[IPT];
    u32 parity = 0;
#pragma unroll
    for (int k = 0; k < IPT; ++k) key[k] = static_cast<u32>(compressed(full[k]));
    cluster_passes<IPT>(cluster, S, key, idx, n, min(bits, 32u), bits <= 32u, parity, a.perm);
    if (bits > 32u) {   // the upper word of the keys, in the order of the lower one
#pragma unroll
        for (int k = 0; k < IPT; ++k)
            key[k] = first + 32u * k < n ? static_cast<u32>(compressed(load_key(idx[k])) >> 32) : 0u;
        cluster_passes<IPT>(cluster, S, key, idx, n, bits - 32u, true, parity, a.perm);
    }
}

template <int IPT, int INPUT>
cudaError_t launch(const ClusterSortArgs& a, u32 blocks, cudaStream_t stream, bool* launched) {
    constexpr int kMaxDevices = 64;
    static std::atomic<int> fits[kMaxDevices];   // 0 = not yet asked, 1 = yes, 2 = no
    const auto fn = cluster_sort_kernel<IPT, INPUT>;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= kMaxDevices || fits[dev].load() == 2) return cudaSuccess;
    // set on every call: the attributes belong to the current context
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sizeof(ClusterSmem<IPT>)));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(CS_MAX_BLOCKS);
    cfg.blockDim = dim3(CS_THREADS);
    cfg.dynamicSmemBytes = sizeof(ClusterSmem<IPT>);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CS_MAX_BLOCKS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (fits[dev].load() == 0) {   // asked for the largest cluster
        int active = 0;
        const bool ok = cudaOccupancyMaxActiveClusters(&active, fn, &cfg) == cudaSuccess && active > 0;
        if (!ok) cudaGetLastError();
        fits[dev].store(ok ? 1 : 2);
        if (!ok) return cudaSuccess;
    }
    cfg.gridDim = dim3(blocks);
    attr[0].val.clusterDim.x = blocks;
    e = cudaLaunchKernelEx(&cfg, fn, a);
    *launched = e == cudaSuccess;
    return e;
}

template <int INPUT>
cudaError_t launch_ipt(const ClusterSortArgs& a, cudaStream_t stream, bool* launched) {
    u32 blocks = 1;   // a power of two, one item per thread until the cluster is full
    while (blocks < CS_MAX_BLOCKS && blocks * CS_THREADS < a.n) blocks *= 2;
    const u32 ipt = (a.n + blocks * CS_THREADS - 1) / (blocks * CS_THREADS);
    if (ipt <= 1) return launch<1, INPUT>(a, blocks, stream, launched);
    if (ipt <= 2) return launch<2, INPUT>(a, blocks, stream, launched);
    if (ipt <= 3) return launch<3, INPUT>(a, blocks, stream, launched);
    if (ipt <= 4) return launch<4, INPUT>(a, blocks, stream, launched);
    if (ipt <= 6) return launch<6, INPUT>(a, blocks, stream, launched);
    return launch<8, INPUT>(a, blocks, stream, launched);
}

}  // namespace

cudaError_t enqueue_cluster_sort(const ClusterSortArgs& a, cudaStream_t stream, bool* launched) {
    *launched = false;
    if (a.n == 0 || a.n > CLUSTER_SORT_MAX || sort_stall_test() || large_sort_test()) return cudaSuccess;
    if (!a.pos) return launch_ipt<SORT_KEYS>(a, stream, launched);
    if (a.scene) return launch_ipt<SORT_BATCH>(a, stream, launched);
    return launch_ipt<SORT_SCENE>(a, stream, launched);
}

}  // namespace wcsph
