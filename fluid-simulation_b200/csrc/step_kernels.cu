// step_kernels.cu — see step_kernels.cuh for the decomposition.
#include "step_kernels.cuh"

#include <algorithm>
#include <atomic>
#include <climits>

#include "simulator.cuh"
#include "step_device.cuh"

namespace wcsph {

namespace {

template <int KIND, int WPB, bool BATCH>
__global__ void __launch_bounds__(WPB * 32, KindCfg<KIND>::min_warps / WPB) cell_pass_kernel(const DevParams P, const TravArgs a) {
    if (a.st->error_flags & ERR_LOOKBACK_TIMEOUT) return;   // no sorted state this step (reorder skipped)
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    const u32 lane = lane_id();
    const u32 warp = threadIdx.x >> 5;
    const WarpView<KIND> S = warp_view<KIND>(a, dyn_smem, warp);

    float dt = 0.f, np_dt = 0.f;
    if constexpr (KIND == PASS_SURFACE) {
        // every warp reads the CFL step itself (no block barrier); the flip of
        // the max-speed parity happens only after every warp has finished
        float t = 0.f;
        if (lane == 0) t = cfl_time_step(a, P);
        dt = __shfl_sync(FULL, t, 0);
        np_dt = a.delta < a.np_max_dt ? a.delta : a.np_max_dt;
    }
    float red_max = 0.f, red_speed = 0.f, red_speed2 = 0.f;
    cell_pass_chunk<KIND, BATCH>(P, a, S, blockIdx.x * WPB + warp, dt, np_dt, red_max, red_speed, red_speed2);

    if constexpr (KIND == PASS_ADJ_FORCE) {
        double v = static_cast<double>(red_speed);
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
        if (lane == 0 && v != 0.0) atomicAdd(a.adj_accum, v);
    }
    if constexpr (KIND == PASS_SURFACE) surface_reduce<WPB>(a, dt, np_dt, red_max, red_speed, red_speed2);
}


// Density pass over blocks of 2^LEVEL cells (density_blocks.cuh).
template <int LEVEL, bool BATCH>
__global__ void __launch_bounds__(BlockCfg<LEVEL>::nt, BlockCfg<LEVEL>::min_blocks)
density_block_kernel(const DevParams P, const TravArgs a) {
    if (a.st->error_flags & ERR_LOOKBACK_TIMEOUT) return;   // no sorted state this step (reorder skipped)
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    density_units<BlockCfg<LEVEL>, BATCH>(P, a, *reinterpret_cast<BlockSmem<BlockCfg<LEVEL>>*>(dyn_smem));
}

// Neighbours summed together (list_rows' DEPTH) and resident warps per SM the
// register allocation of the list kernels must allow (36 -> 56 registers, 48 ->
// 40). Both passes wait on neighbour gathers.
// From 2^17 particles on the force pass sums two neighbours at a time, with the
// next two in flight, and gains more than the warps it costs: 1 M particles
// 141 -> 121 us, 4 M 497 -> 430 (28 warps 126 / 461, 40 warps spill: 166 / 629,
// three at a time 136 / 505). The surface pass keeps one at a time, all the
// warps that fit and 8-warp blocks: 1 M 139 us, 4 M 474 (two at a time at 32
// warps 143 / 516; 2-warp blocks 141 / 502); the batched one, which looks its
// scene up, would spill at 40 registers and takes 48 (12 and 100 scenes 256 / 1090
// -> 252 / 1088 us a step).
// Smaller scenes leave the SMs a few warps each, so three at a time are summed
// with 128 registers to spare: force / surface 27 / 27 -> 20 / 16 us at 33 k
// particles with walls, 55 / 55 -> 27 / 25 at 79 k (half of that by full warps:
// these scenes took 8 rows per warp before). Rows without usable lists are
// summed two at a time there (`spilled`; four would take 121 registers: the 79 k
// step 128 -> 143 us): all rows of 79 k particles with 32 list slots 540 -> 459
// us a step, 513 with 8 rows per warp.
template <int KIND, bool SMALL, bool BATCH>
struct ListCfg {
    static constexpr int min_warps = SMALL ? 16 : (KIND == PASS_FORCE ? 36 : (BATCH ? 40 : 48));
    static constexpr int depth = SMALL ? 3 : (KIND == PASS_FORCE ? 2 : 1);
    static constexpr int spilled = SMALL ? 2 : 1;
};

// Force / surface pass over the neighbour lists written by the density pass.
template <int KIND, int WPB, bool BATCH, bool SMALL, int SHARE>
__global__ void __launch_bounds__(WPB * 32, ListCfg<KIND, SMALL, BATCH>::min_warps / WPB)
list_pass_kernel(const DevParams P, const TravArgs a) {
    if (a.st->error_flags & ERR_LOOKBACK_TIMEOUT) return;   // no sorted state this step (reorder skipped)
    const u32 lane = lane_id();
    const u32 warp = threadIdx.x >> 5;
    float dt = 0.f, np_dt = 0.f;
    if constexpr (KIND == PASS_SURFACE) {
        float t = 0.f;
        if (lane == 0) t = cfl_time_step(a, P);
        dt = __shfl_sync(FULL, t, 0);
        np_dt = a.delta < a.np_max_dt ? a.delta : a.np_max_dt;
    }
    float red_max = 0.f, red_speed = 0.f, red_speed2 = 0.f;
    const u32 gw = blockIdx.x * WPB + warp;
    const u32 base = gw / SHARE * LIST_ROWS;
    if (base < a.n)
        list_rows<KIND, BATCH, ListCfg<KIND, SMALL, BATCH>::depth, ListCfg<KIND, SMALL, BATCH>::spilled, SHARE>(
            P, a, base, min(LIST_ROWS, a.n - base), dt, np_dt, red_max, red_speed, red_speed2, gw % SHARE);
    if constexpr (KIND == PASS_SURFACE) surface_reduce<WPB>(a, dt, np_dt, red_max, red_speed, red_speed2);
}

template <bool BATCH>
__global__ void reorder_cells_kernel(const float4* __restrict__ pos_in, const float4* __restrict__ vel_in,
                                     const u32* __restrict__ v1, const u32* __restrict__ v2,
                                     const DevState* st, u32 n, float cs, float4* __restrict__ pos_out,
                                     float4* __restrict__ vel_out, u32* __restrict__ perm_out,
                                     u64* __restrict__ ckey_out, u64* table, u32* cstart, u32* cend,
                                     u32 tmask, DevState* st_err, const u32* __restrict__ scene_in,
                                     u32* __restrict__ units, u32 unit_level) {
    // a sort whose look-back wait ran out left no permutation: keep the
    // previous sorted state and hash (every later pass returns at once too)
    if (st->error_flags & ERR_LOOKBACK_TIMEOUT) return;
    reorder_cell_item<BATCH>(pos_in, vel_in, v1, v2, st, n, cs, pos_out, vel_out, perm_out, ckey_out, table, cstart,
                             cend, tmask, st_err, scene_in, blockIdx.x * blockDim.x + threadIdx.x, units, unit_level);
}

__global__ void init_cfl_kernel(const float4* __restrict__ vel, u32 n, DevState* st) {
    float m = 0.f;
    for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 v = vel[i];
        m = fmaxf(m, dot3(v, v));
    }
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(FULL, m, o));
    if ((threadIdx.x & 31u) == 0) atomicMax(&st->vmax2_bits[st->parity], __float_as_uint(m));
}

__global__ void metrics_kernel(const float4* __restrict__ vel, u32 n, float mass, float* out2) {
    // single block, deterministic order (used outside the step)
    __shared__ double s1[32], s2[32];
    double a = 0.0, b = 0.0;
    for (u32 i = threadIdx.x; i < n; i += blockDim.x) {
        const float4 v = vel[i];
        const float d = dot3(v, v);
        a += static_cast<double>(sqrtf(d));
        b += static_cast<double>(d);
    }
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(FULL, a, o);
        b += __shfl_xor_sync(FULL, b, o);
    }
    if ((threadIdx.x & 31u) == 0) { s1[threadIdx.x >> 5] = a; s2[threadIdx.x >> 5] = b; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t1 = 0.0, t2 = 0.0;
        for (u32 w = 0; w < blockDim.x / 32; ++w) { t1 += s1[w]; t2 += s2[w]; }
        out2[0] = n ? static_cast<float>(t1 / static_cast<double>(n)) : 0.f;
        out2[1] = static_cast<float>(0.5 * static_cast<double>(mass) * t2);
    }
}

template <bool BATCH>
__global__ void boundary_mass_kernel(const DevParams P, const float4* __restrict__ bpos, u32 nb, HashView bh,
                                     float* __restrict__ bmass, const u64* __restrict__ bckey) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nb) return;
    const float4 xi = bpos[i];
    const int3 c = cell_of(xi, P.h);
    const u32 scene = BATCH ? static_cast<u32>(bckey[i] >> 48) : 0u;
    float sum = P.w0;  // cubic_spline(0, h)
    for (int x = -1; x <= 1; ++x)
        for (int y = -1; y <= 1; ++y)
            for (int z = -1; z <= 1; ++z) {
                u64 pk;
                if constexpr (BATCH)
                    pk = pack_cell_batch(scene, offset_coord(c.x) + x, offset_coord(c.y) + y, offset_coord(c.z) + z);
                else
                    pk = pack_cell(offset_coord(c.x) + x, offset_coord(c.y) + y, offset_coord(c.z) + z);
                const u32 slot = hash_find<BATCH>(bh.table, bh.tmask, pk);
                if (slot == EMPTY_CELL) continue;
                const u32 s = bh.cstart[slot], e = bh.cend[slot];
                for (u32 j = s; j < e; ++j) {
                    const float4 xj = bpos[j];
                    const float r2 = dist2(xi, xj);
                    if (j != i && r2 <= P.h2) sum += cubic_w(sqrtf(r2) * P.inv_h, P);
                }
            }
    bmass[i] = P.rest_density / sum;
}

}  // namespace

u32 pass_grid(u32 n, int wpb, u32 chunk) {
    const u32 chunks = (n + chunk - 1) / chunk;
    return (chunks + wpb - 1) / wpb;
}

void launch_reorder_cells(const float4* pos_in, const float4* vel_in, const u32* perm_src1, const u32* perm_src2,
                          const DevState* st, u32 n, float cs, float4* pos_out, float4* vel_out, u32* perm_out,
                          u64* ckey_out, u64* table, u32* cstart, u32* cend, u32 tmask, DevState* st_err,
                          cudaStream_t stream, const u32* scene_in, u32* units, u32 unit_level) {
    if (n == 0) return;
    const u32 threads = 256;
    const u32 grid = (n + threads - 1) / threads;
    if (scene_in)
        reorder_cells_kernel<true><<<grid, threads, 0, stream>>>(pos_in, vel_in, perm_src1, perm_src2, st, n, cs,
                                                                 pos_out, vel_out, perm_out, ckey_out, table, cstart,
                                                                 cend, tmask, st_err, scene_in, units, unit_level);
    else
        reorder_cells_kernel<false><<<grid, threads, 0, stream>>>(pos_in, vel_in, perm_src1, perm_src2, st, n, cs,
                                                                  pos_out, vel_out, perm_out, ckey_out, table, cstart,
                                                                  cend, tmask, st_err, nullptr, units, unit_level);
}

template <int KIND, int WPB, bool BATCH>
static void launch_wpb(const DevParams& P, const TravArgs& a, cudaStream_t stream, u32 grid) {
    // per-warp candidate staging sized by the bit-matrix capacity 32 * mask_words
    if constexpr (KIND == PASS_FORCE || KIND == PASS_SURFACE) {
        if (a.nbr) {   // the list kernels use no shared memory (all of it serves as L1)
            const dim3 block(WPB * 32);
            if (list_share(a.n) > 1u) list_pass_kernel<KIND, WPB, BATCH, true, LIST_SHARE><<<grid, block, 0, stream>>>(P, a);
            else if (a.n < LIST_SMALL) list_pass_kernel<KIND, WPB, BATCH, true, 1><<<grid, block, 0, stream>>>(P, a);
            else list_pass_kernel<KIND, WPB, BATCH, false, 1><<<grid, block, 0, stream>>>(P, a);
            return;
        }
    }
    const u32 ncell = static_cast<u32>((2 * a.range + 1) * (2 * a.range + 1) * (2 * a.range + 1));
    const size_t bytes = warp_smem_bytes<KIND>(a.mask_words * 32u, ncell, a.nb > 0) * WPB;
    static bool configured = false;  // per instantiation; the attribute is per device function
    if (!configured) {
        cudaFuncSetAttribute(cell_pass_kernel<KIND, WPB, BATCH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(warp_smem_bytes<KIND>(32u * MAX_MASK_WORDS, MAX_RANGE_CELLS, true) * WPB));
        configured = true;
    }
    cell_pass_kernel<KIND, WPB, BATCH><<<grid, WPB * 32, bytes, stream>>>(P, a);
}

template <int LEVEL, bool BATCH>
static void launch_density_blocks(const DevParams& P, const TravArgs& a, cudaStream_t stream) {
    using C = BlockCfg<LEVEL>;
    constexpr int kMaxDevices = 64;
    static std::atomic<u32> resident[kMaxDevices];   // resident blocks of the device, 0 = not yet asked
    int dev = 0;
    WCSPH_CUDA(cudaGetDevice(&dev));
    u32 blocks = dev < kMaxDevices ? resident[dev].load() : 0u;
    // on every call: the attribute belongs to the current context
    WCSPH_CUDA(cudaFuncSetAttribute(density_block_kernel<LEVEL, BATCH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    static_cast<int>(sizeof(BlockSmem<C>))));
    if (blocks == 0) {
        int per_sm = 0, sms = 0;
        WCSPH_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, density_block_kernel<LEVEL, BATCH>, C::nt,
                                                                 sizeof(BlockSmem<C>)));
        WCSPH_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        blocks = static_cast<u32>(std::max(per_sm, 1) * std::max(sms, 1));
        if (dev < kMaxDevices) resident[dev].store(blocks);
    }
    density_block_kernel<LEVEL, BATCH><<<std::min(blocks, a.n), C::nt, sizeof(BlockSmem<C>), stream>>>(P, a);
    WCSPH_CUDA(cudaGetLastError());
}

template <int KIND, bool BATCH>
static void launch_kind(const DevParams& P, const TravArgs& a, cudaStream_t stream, int wpb) {
    const bool listed = (KIND == PASS_FORCE || KIND == PASS_SURFACE) && a.nbr != nullptr;
    const u32 groups = (a.n + LIST_ROWS - 1) / LIST_ROWS;   // each of list_share warps
    const u32 grid = listed ? pass_grid(groups * list_share(a.n), wpb, 1u) : pass_grid(a.n, wpb, a.chunk);
    if (grid == 0) return;
    if constexpr (KIND == PASS_DENSITY) {
        if (a.units) {
            if (a.unit_level == 3u) launch_density_blocks<3, BATCH>(P, a, stream);
            else if (a.unit_level == 6u) launch_density_blocks<6, BATCH>(P, a, stream);
            else launch_density_blocks<5, BATCH>(P, a, stream);
            return;
        }
    }
    switch (wpb) {
    case 2: launch_wpb<KIND, 2, BATCH>(P, a, stream, grid); break;
    case 8: launch_wpb<KIND, 8, BATCH>(P, a, stream, grid); break;
    default: launch_wpb<KIND, 4, BATCH>(P, a, stream, grid); break;
    }
}

template <bool BATCH>
static void launch_pass_t(int kind, const DevParams& P, const TravArgs& a, cudaStream_t stream, int wpb) {
    switch (kind) {
    case PASS_DENSITY: launch_kind<PASS_DENSITY, BATCH>(P, a, stream, wpb); break;
    case PASS_FORCE: launch_kind<PASS_FORCE, BATCH>(P, a, stream, wpb); break;
    case PASS_SURFACE: launch_kind<PASS_SURFACE, BATCH>(P, a, stream, wpb); break;
    case PASS_COUNT: launch_kind<PASS_COUNT, BATCH>(P, a, stream, wpb); break;
    case PASS_FILL: launch_kind<PASS_FILL, BATCH>(P, a, stream, wpb); break;
    case PASS_ADJ_FORCE: launch_kind<PASS_ADJ_FORCE, BATCH>(P, a, stream, wpb); break;
    case PASS_ADJ_DENSITY: launch_kind<PASS_ADJ_DENSITY, BATCH>(P, a, stream, wpb); break;
    default: break;
    }
}

void launch_pass(int kind, const DevParams& P, const TravArgs& a, cudaStream_t stream, int wpb, bool batch) {
    if (wpb != 2 && wpb != 8) wpb = 4;
    if (batch) launch_pass_t<true>(kind, P, a, stream, wpb);
    else launch_pass_t<false>(kind, P, a, stream, wpb);
}

void launch_init_cfl(const float4* vel, u32 n, DevState* st, cudaStream_t stream) {
    if (n == 0) return;
    const u32 blocks = std::min<u32>((n + 255) / 256, 1184);
    init_cfl_kernel<<<blocks, 256, 0, stream>>>(vel, n, st);
}

void launch_boundary_mass(const DevParams& P, const float4* bpos, u32 nb, HashView bh, float* bmass,
                          cudaStream_t stream, const u64* bckey) {
    if (nb == 0) return;
    if (bckey) boundary_mass_kernel<true><<<(nb + 127) / 128, 128, 0, stream>>>(P, bpos, nb, bh, bmass, bckey);
    else boundary_mass_kernel<false><<<(nb + 127) / 128, 128, 0, stream>>>(P, bpos, nb, bh, bmass, nullptr);
}

void launch_metrics(const float4* vel, u32 n, float mass, float* out2, cudaStream_t stream) {
    metrics_kernel<<<1, 1024, 0, stream>>>(vel, n, mass, out2);
}

}  // namespace wcsph
