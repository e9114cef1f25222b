// density_blocks.cuh — the density pass over blocks of cells (one neighbour
// cell in every direction, neighbour lists on).
//
// A unit of work is a Morton-aligned block of cells (2x2x2, 4x4x2 or 4x4x4:
// its particles are contiguous in sorted order) and one thread block of NT
// threads. The unit
//   1. looks up the cells of the block and of the layer around it (64, 144 or
//      216), one lane per cell; the block's own cells add up to its rows;
//   2. stages their particles (the candidates) in shared memory, cells in the
//      x, y, z nesting order, as x / y / z / particle-index arrays;
//   3. lets every lane take one row. The 27 cells around the row's cell are 9
//      runs of 3 cells that lie next to each other in the staged order, so
//      the row's candidates are 9 segments, in the reference's order. The lane
//      tests a segment four candidates at a time (three 128-bit shared loads,
//      packed FP32 in the rounding of dist2) and shifts the results into a
//      32-bit word: r2 <= h2 holds exactly when r2 - (the float after h2) is
//      negative, so a funnel shift collects the sign bits, without compares.
//      Words with hits are kept in shared memory (one column per thread), then
//      the lane walks their bits: it sums W and writes its list, slot t of
//      all lanes of a warp in one 128-byte store.
// Rows hold 25 to 45 neighbours, so the lanes of a warp finish together
// within a few hits, and no partial sums cross lanes: a row's sum runs over its
// neighbours in the reference's order whatever the block size.
//
// What bounds it (1 M particles, 4x4x4 cells, ten steps into a run): instruction
// issue (166 M warp instructions, 64 % of the cycles issue) and the shared-memory
// data pipe (76 % busy: a 128-bit load costs three wavefronts for a warp's four or
// five cells, a walked hit four loads of four). Of the lattice's 213 us, before
// the sums carried their errors, look-ups took 34 (latency; 9 less since warps
// that are done look up for the next unit), staging 14, the tests 85, the walk 57,
// the epilogue 23. The pass it replaced gave a warp the two cells of an x-pair (36
// looked-up cells and 18 staged candidates per row, where a row here pays for
// 3.4), split their hits over the lanes and wrote the lists one scattered word at
// a time: 349 M warp instructions, 460 us (4 M particles 2055 -> 830 us, 0.7 M
// settled 434 -> 258, 33 k with walls 51 -> 30).
#pragma once

namespace wcsph {
namespace {

// Threads per unit, candidate capacity and hit words per row. The capacity is
// 12 to 16 particles per cell (the 0.92-spaced, settled fluid holds 10.3);
// denser blocks are split into smaller ones. The thread counts fit the rows of
// a block into whole rounds: 4x4x4 cells hold 512 rows and a few (17 groups of
// 32), two rounds of 9 warps and three of 8 (4 M particles: 853 us against 930);
// 4x4x2 cells one round of 9 and two of 8 (393 k with walls 125 -> 119, 12
// scenes 0.285 -> 0.275 ms a step).
template <int LEVEL>
struct BlockCfg;
template <>
struct BlockCfg<3> {   // 2x2x2 cells
    static constexpr int nt = 96, cap = 1024, words = 12, min_blocks = 8;
};
template <>
struct BlockCfg<5> {   // 4x4x2 cells
    static constexpr int nt = 288, cap = 2048, words = 12, min_blocks = 3;
};
template <>
struct BlockCfg<6> {   // 4x4x4 cells
    static constexpr int nt = 288, cap = 2560, words = 12, min_blocks = 3;
};

// Thin units (up to thin_rows(level) particles) per thread block above which
// their rows are summed one lane each from global memory, 32 to a warp, instead
// of unit by unit. A unit costs a block's look-ups of 64 to 216 cells whatever it
// holds (some 5 us of one of 444 to 1184 resident blocks), a batch of rows one
// chain of 27 look-ups (about 30 us) that all blocks can share. Step time in us,
// units / rows (the pass before the blocks): 60 k scattered particles 318 / 110
// (188), 400 k 4123 / 300 (736), 1 M with 100 k of spray 1533 / 845 (1298); but
// 2 k scattered 50 / 72, and 20 k at 1.2 a cell (2 k thin units) 72 / 101.
constexpr u32 THIN_UNITS = 6;
constexpr int BLOCK_CELLS = 216;   // cells of the largest block with its surrounding layer

template <class C>
struct BlockSmem {
    float x[C::cap], y[C::cap], z[C::cap];
    u32 j[C::cap];
    u32 word[C::words * C::nt];
    unsigned short wbase[C::words * C::nt];
    // cells of the running unit and of the next one: first particle, and the
    // count, then exclusive prefix (+ total)
    u32 rstart[2][BLOCK_CELLS];
    u32 rpref[2][BLOCK_CELLS + 4];
    u32 start[2];      // first row of the unit
    u64 id[2];         // its block key
    u32 rows[2];       // its particles
    u32 next;          // the unit claimed next
    u32 chunk;         // look-up chunks handed out
    // work items: `thin` thin units (by_rows: batches of their rows), then the
    // others (here and not in registers, which the row loop needs)
    u32 items, thin, by_rows;
};

// Density of row i's boundary particles (cell size h cells, one lane): its
// cell's candidate run, tested 32 at a time, then the hits in run order. The
// first 128 results are the row's hit mask for the force pass.
template <bool BATCH>
__device__ __forceinline__ void density_boundary_row(const DevParams& P, const TravArgs& a, float4 xi, u32 scene,
                                                     u32 i, float* resb) {
    HomeData H;
    H.x = xi;
    if (a.bcell.table == nullptr) {
        boundary_row<PASS_DENSITY, BATCH>(P, a, H, scene, resb, i);
        return;
    }
    u32 t, e;
    boundary_run<BATCH>(a, boundary_cell_key<BATCH>(cell_of(xi, P.h), scene), t, e);
    u32 mk[4] = {0u, 0u, 0u, 0u};
    for (u32 w = 0; t + 32u * w < e; ++w) {
        const u32 b0 = t + 32u * w;
        const u32 len = min(32u, e - b0);
        u32 bits = 0;
        // four in flight, past the end the last one again (as an unrolled loop the
        // compiler kept them in flight or not by the code around it: 2 k particles
        // 62 against 66 us a step)
        for (u32 u = 0; u < len; u += 4u) {
            float4 xb[4];
#pragma unroll
            for (u32 v = 0; v < 4u; ++v) xb[v] = ro_ld(a.bcx + guard(a, b0 + min(u + v, len - 1u), a.bcx_n));
#pragma unroll
            for (u32 v = 0; v < 4u; ++v) bits |= (dist2(xi, xb[v]) <= P.h2 ? 1u : 0u) << (u + v);
        }
        bits &= FULL >> (32u - len);
#pragma unroll
        for (u32 q = 0; q < 4; ++q)
            if (w == q) mk[q] = bits;
        float4 xb = xi;
        if (bits) xb = ro_ld(a.bcx + guard(a, b0 + (__ffs(bits) - 1), a.bcx_n));
        while (bits) {   // the next hit is in flight while one is summed
            const float4 now = xb;
            bits &= bits - 1;
            if (bits) xb = ro_ld(a.bcx + guard(a, b0 + (__ffs(bits) - 1), a.bcx_n));
            boundary_pair_m<PASS_DENSITY>(resb, H, now.w, now, dist2(xi, now), P);
        }
    }
    if (a.bmask != nullptr) a.bmask[i] = make_uint4(mk[0], mk[1], mk[2], mk[3]);
}

// Sum of W over a row's pairs: 2 (1 - q)^3 - max(1 - 2 q, 0)^3 is the cubic
// spline over its factor for q <= 1; the two cubes are summed apart. The first
// sum is a single chain of 25 to 100 terms, so its rounding errors are carried
// along (Kahan); few pairs are within h / 2, so the second is short. RMS error of
// rho against 64 bits, of the lane-run sums this pass had before / plain chains
// with q from sqrt.approx / as it is: 0.7 M settled 7.8e-5 / 9.4e-5 / 6.3e-5,
// 1 M lattice 5.4e-5 / 6.3e-5 / 4.6e-5, 79 k 2.09e-4 / 2.33e-4 / 2.05e-4; it costs
// 1 M settled 737 -> 753 us a step and the persistent ensemble 3 %. The rounding
// is written out: every kernel that inlines this produces the same bits.
struct DensitySum {
    float t3 = 0.f, over = 0.f;   // sum of (1 - q)^3, and by how much it is over
    float u3 = 0.f;
    __device__ __forceinline__ void pair(float r2, const DevParams& P) {
        float rinv;
        const float q = q_of(r2, rinv, P);
        const float t = __fsub_rn(1.f, q);
        const float u = fmaxf(__fmaf_rn(-2.f, q, 1.f), 0.f);
        const float term = __fmaf_rn(__fmul_rn(t, t), t, -over);
        const float sum = __fadd_rn(t3, term);
        over = __fsub_rn(__fsub_rn(sum, t3), term);
        t3 = sum;
        u3 = __fmaf_rn(__fmul_rn(u, u), u, u3);
    }
    __device__ __forceinline__ float value() const { return __fmaf_rn(2.f, t3, -__fmaf_rn(2.f, over, u3)); }
};

// Row i without staged candidates (a thin block, or a single cell whose 27
// cells exceed the capacity): its cells from global memory, in the same order,
// three looked up at a time. Returns the neighbour count.
template <bool BATCH>
__device__ __forceinline__ u32 density_direct_row(const DevParams& P, const TravArgs& a, u32 i, u64 pk, float4 xi,
                                                  DensitySum& W) {
    u32 ux, uy, uz, scene;
    decode_cell<BATCH>(pk, ux, uy, uz, scene);
    u32 hits = 0;
    for (u32 q = 0; q < 9u; ++q) {
        const u32 x = ux + q / 3u - 1u, y = uy + q % 3u - 1u;
        u64 ck[3], seen[3];
        u32 slot[3], s[3], e[3];
#pragma unroll
        for (u32 u = 0; u < 3u; ++u) {
            if constexpr (BATCH) ck[u] = pack_cell_batch(scene, x, y, uz + u - 1u);
            else ck[u] = pack_cell(x, y, uz + u - 1u);
            slot[u] = static_cast<u32>(slot_hash<BATCH>(ck[u])) & a.fluid.tmask;
            seen[u] = ro_ld(a.fluid.table + slot[u]);
        }
#pragma unroll
        for (u32 u = 0; u < 3u; ++u) {
            if (seen[u] != ck[u])
                slot[u] = seen[u] == EMPTY_HASH ? EMPTY_CELL : find_slot<BATCH>(a.fluid.table, a.fluid.tmask, ck[u]);
            s[u] = e[u] = 0u;
            if (slot[u] != EMPTY_CELL) {
                s[u] = ro_ld(a.fluid.cstart + slot[u]);
                e[u] = ro_ld(a.fluid.cend + slot[u]);
            }
        }
#pragma unroll
        for (u32 u = 0; u < 3u; ++u) {
            // four in flight, past the end the last one again (one at a time 120
            // particles a cell took 2.26 ms a step, so 1.56)
            for (u32 j0 = s[u]; j0 < e[u]; j0 += 4u) {
                float r2[4];
#pragma unroll
                for (u32 v = 0; v < 4u; ++v)
                    r2[v] = dist2(xi, ro_ld(a.pos + guard(a, min(j0 + v, e[u] - 1u), a.n)));
#pragma unroll
                for (u32 v = 0; v < 4u; ++v) {
                    const u32 j = j0 + v;
                    if (!(r2[v] <= P.h2) || j == i || j >= e[u]) continue;
                    if (hits < a.nbr_width) a.nbr[hits * a.n + i] = j;
                    ++hits;
                    W.pair(r2[v], P);
                }
            }
        }
    }
    return hits;
}

// Neighbours of row i among the staged candidates. seg0: first cell of the
// row's 9 runs (the block's cell grid has Dy x Dz cells per x); selfm: the
// row's own candidate index. Returns the neighbour count.
template <class C>
__device__ __forceinline__ u32 density_staged_row(const DevParams& P, const TravArgs& a, BlockSmem<C>& S, u32 i,
                                                  float4 xi, const u32* rpref, u32 seg0, u32 Dy, u32 Dz, u32 selfm,
                                                  bool act, DensitySum& W) {
    const float2 nx = make_float2(-xi.x, -xi.x), ny = make_float2(-xi.y, -xi.y), nz = make_float2(-xi.z, -xi.z);
    const float lim = -__uint_as_float(__float_as_uint(P.h2) + 1u);   // minus the float after h2
    const float2 nlim = make_float2(lim, lim);
    u32* const word = S.word + threadIdx.x;
    unsigned short* const wbase = S.wbase + threadIdx.x;
    u32 hits = 0;
    u32 slot_idx = i;      // list slot of the next hit (u32: the host caps nbr_width * n below 2^32)
    u32 seg = act ? 0u : 9u;
    u32 b = 0, s0 = 0, e0 = 0;
    bool open = false;     // segment seg is partly tested: [b, e0) remains
    do {
        // phase 1: words with hits, until all segments are tested or the column is full
        u32 k = 0;
        while (seg < 9u && k < static_cast<u32>(C::words)) {
            if (!open) {
                const u32 c = seg0 + ((seg / 3u) * Dy + seg % 3u) * Dz;
                s0 = rpref[c];
                e0 = rpref[c + 3u];
                b = s0 & ~3u;
            }
            if (b < e0) {
                const u32 nq = min(8u, (e0 - b + 3u) >> 2);
                const float4* X = reinterpret_cast<const float4*>(S.x + b);
                const float4* Y = reinterpret_cast<const float4*>(S.y + b);
                const float4* Z = reinterpret_cast<const float4*>(S.z + b);
                u32 bits = 0;
#pragma unroll
                for (u32 q = 0; q < 8u; ++q) {
                    if (q >= nq) break;
                    const float4 cx = X[q], cy = Y[q], cz = Z[q];
                    // x_j - x_i: the square is that of x_i - x_j, bit for bit
                    const float2 dx0 = __fadd2_rn(make_float2(cx.x, cx.y), nx);
                    const float2 dx1 = __fadd2_rn(make_float2(cx.z, cx.w), nx);
                    const float2 dy0 = __fadd2_rn(make_float2(cy.x, cy.y), ny);
                    const float2 dy1 = __fadd2_rn(make_float2(cy.z, cy.w), ny);
                    const float2 dz0 = __fadd2_rn(make_float2(cz.x, cz.y), nz);
                    const float2 dz1 = __fadd2_rn(make_float2(cz.z, cz.w), nz);
                    const float2 r0 = __fadd2_rn(__ffma2_rn(dz0, dz0, __ffma2_rn(dx0, dx0, __fmul2_rn(dy0, dy0))), nlim);
                    const float2 r1 = __fadd2_rn(__ffma2_rn(dz1, dz1, __ffma2_rn(dx1, dx1, __fmul2_rn(dy1, dy1))), nlim);
                    bits = __funnelshift_l(__float_as_uint(r0.x), bits, 1);
                    bits = __funnelshift_l(__float_as_uint(r0.y), bits, 1);
                    bits = __funnelshift_l(__float_as_uint(r1.x), bits, 1);
                    bits = __funnelshift_l(__float_as_uint(r1.y), bits, 1);
                }
                bits <<= 32u - 4u * nq;          // candidate b + t at bit 31 - t
                if (b < s0) bits &= FULL >> (s0 - b);
                if (e0 - b < 32u) bits &= ~(FULL >> (e0 - b));
                const u32 me = selfm - b;
                if (me < 32u) bits &= ~(0x80000000u >> me);
                if (bits) {
                    hits += __popc(bits);
                    word[k * C::nt] = bits;
                    wbase[k * C::nt] = static_cast<unsigned short>(b);
                    ++k;
                }
                b += 32u;
            }
            open = b < e0;
            if (!open) ++seg;
        }
        // phase 2: the hits, in candidate order (two per turn, for independent
        // chains, cost more than they hid: 1 M particles 204 -> 219 us)
        const bool listed = hits <= a.nbr_width;   // else the row's list is not used
        if (k) {
            u32 t = 0;
            u32 w = word[0];
            u32 base = wbase[0];
            do {
                const u32 bit = static_cast<u32>(__clz(static_cast<int>(w)));
                const u32 m = guard(a, base + bit, C::cap);
                w ^= 0x80000000u >> bit;
                if (w == 0u && ++t < k) {
                    w = word[t * C::nt];
                    base = wbase[t * C::nt];
                }
                const float r2 = dist2(xi, make_float4(S.x[m], S.y[m], S.z[m], 0.f));
                if (listed) a.nbr[slot_idx] = S.j[m];
                slot_idx += a.n;
                W.pair(r2, P);
            } while (w);
        }
    } while (seg < 9u);
    return hits;
}

// A block of 2^level cells with its surrounding layer.
template <bool BATCH>
struct BlockGrid {
    u32 ox, oy, oz, scene;   // first cell of the layer
    u32 Dx, Dy, Dz;
    __device__ __forceinline__ BlockGrid(u64 id, u32 level) {
        u32 ux, uy, uz;
        decode_cell<BATCH>(id, ux, uy, uz, scene);
        ox = ux - 1u; oy = uy - 1u; oz = uz - 1u;
        Dx = (1u << ((level + 2u) / 3u)) + 2u;
        Dy = (1u << ((level + 1u) / 3u)) + 2u;
        Dz = (1u << (level / 3u)) + 2u;
    }
    __device__ __forceinline__ u32 cells() const { return Dx * Dy * Dz; }
};

// Looks up the cells of block `id` into buffer b, 32 at a time: warps take
// chunks from S.chunk (zeroed before, as S.rows[b]). The block's own cells
// add up to its rows.
template <class C, bool BATCH>
__device__ __forceinline__ void density_lookup(const TravArgs& a, BlockSmem<C>& S, u32 b, u64 id, u32 level) {
    const u32 lane = lane_id();
    const BlockGrid<BATCH> G(id, level);
    const u32 ncell = G.cells();
    for (;;) {
        u32 c = 0;
        if (lane == 0) c = atomicAdd(&S.chunk, 1u);
        c = __shfl_sync(FULL, c, 0);
        if (c * 32u >= ncell) break;
        const u32 q = c * 32u + lane;
        u32 mine = 0;
        if (q < ncell) {
            const u32 x = q / (G.Dy * G.Dz), y = (q / G.Dz) % G.Dy, z = q % G.Dz;
            u64 pk;
            if constexpr (BATCH) pk = pack_cell_batch(G.scene, G.ox + x, G.oy + y, G.oz + z);
            else pk = pack_cell(G.ox + x, G.oy + y, G.oz + z);
            const u32 slot = find_slot_wide<BATCH>(a.fluid.table, a.fluid.tmask, pk);
            u32 s = 0, cnt = 0;
            if (slot != EMPTY_CELL) {
                s = ro_ld(a.fluid.cstart + slot);
                const u32 e = ro_ld(a.fluid.cend + slot);
                cnt = e > s ? e - s : 0u;
            }
            S.rstart[b][q] = s;
            S.rpref[b][q] = cnt;
            if (x - 1u < G.Dx - 2u && y - 1u < G.Dy - 2u && z - 1u < G.Dz - 2u) mine = cnt;
        }
        mine = __reduce_add_sync(FULL, mine);
        if (lane == 0 && mine) atomicAdd(&S.rows[b], mine);
    }
}

// Units of the whole array, by thread blocks that claim them from a device
// counter (the list and both counters are rebuilt by the sort plan and the
// reorder of every step). Warps that have finished their rows of a unit look
// the next one's cells up while the others still work: their dependent
// loads (list, key, hash, range) took 34 of 208 us at 1 M particles (256 scenes
// per stage 3.12 -> 2.93 ms a step, 1 M 209 -> 203 us).
template <class C, bool BATCH>
__device__ __forceinline__ void density_units(const DevParams& P, const TravArgs& a, BlockSmem<C>& S) {
    const u32 tid = threadIdx.x;
    const u32 lane = tid & 31u;
    const u32 n = a.n;
    const volatile DevState& st = *a.st;
    if (tid == 0) {
        const u32 by_rows = st.thin_count > THIN_UNITS * gridDim.x ? 1u : 0u;
        S.by_rows = by_rows;
        S.thin = by_rows ? (st.thin_rows + C::nt - 1u) / C::nt : st.thin_count;
        S.items = S.thin + st.unit_count;
    }
    volatile BlockSmem<C>& V = S;
    const u64 unit_mask = block_mask<BATCH>(a.unit_level);
    auto lookup_unit = [&](u32 u, u32 b) {
        const u32 thin = V.thin;
        if (u < thin && V.by_rows) return;
        const u32 start = guard(a, a.units[u < thin ? n - 1u - u : u - thin], n);
        const u64 id = a.ckey[start] & unit_mask;
        if (tid == 0) {
            S.start[b] = start;
            S.id[b] = id;
        }
        density_lookup<C, BATCH>(a, S, b, id, a.unit_level);
    };
    if (tid == 0) {
        S.chunk = 0u;
        S.rows[0] = 0u;
    }
    __syncthreads();
    u32 item = blockIdx.x;   // the first claim of every block is its own index
    if (item < V.items) lookup_unit(item, 0u);
    for (u32 b = 0; item < V.items; b ^= 1u) {
        u32 claimed = 0;
        if (tid == 0) claimed = atomicAdd(&a.st->unit_next, 1u) + gridDim.x;
        __syncthreads();   // the unit's look-ups, and the last rows of the one before
        const bool listed = item < V.thin && V.by_rows;   // rows of thin units
        u32 level = a.unit_level;
        u32 i0 = listed ? item * C::nt : S.start[b];
        u64 id = S.id[b];
        for (;;) {
            const BlockGrid<BATCH> G(id, level);
            const u32 ncell = G.cells();
            // exclusive prefix of the counts
            if (tid < 32u) {
                u32 run = 0;
                for (u32 base = 0; base < ncell && !listed; base += 32u) {
                    const u32 q = base + lane;
                    const u32 c = q < ncell ? S.rpref[b][q] : 0u;
                    const u32 incl = warp_incl_scan(c);
                    if (q < ncell) S.rpref[b][q] = run + incl - c;
                    run += __shfl_sync(FULL, incl, 31);
                }
                if (lane == 0) {
                    S.rpref[b][ncell] = run;
                    S.next = claimed;
                    S.chunk = 0u;
                    S.rows[b ^ 1u] = 0u;
                }
            }
            __syncthreads();
            const u32 M = S.rpref[b][ncell];
            const u32 rows = listed ? min(static_cast<u32>(C::nt), st.thin_rows - i0) : min(S.rows[b], n - i0);
            const bool split = M > static_cast<u32>(C::cap) && level > 0u;   // too dense: smaller blocks
            const bool staged = M <= static_cast<u32>(C::cap) && !listed;
            if (staged) {
                // eight lanes per cell: a cell's particles are contiguous
                for (u32 q = tid >> 3; q < ncell; q += C::nt / 8) {
                    const u32 s = S.rstart[b][q], m0 = S.rpref[b][q], cnt = S.rpref[b][q + 1u] - m0;
                    for (u32 t = tid & 7u; t < cnt; t += 8u) {
                        const u32 j = guard(a, s + t, n);
                        const float4 p = ro_ld(a.pos + j);
                        const u32 m = guard(a, m0 + t, C::cap);
                        S.x[m] = p.x;
                        S.y[m] = p.y;
                        S.z[m] = p.z;
                        S.j[m] = j;
                    }
                }
            }
            __syncthreads();
            if (!split) {
                for (u32 r0 = tid & ~31u; r0 < rows; r0 += C::nt) {
                    const u32 r = r0 + lane;
                    const bool act = r < rows;
                    u32 i = i0 + (act ? r : 0u);
                    if (listed) i = guard(a, a.units[n + i], n);
                    const u64 pk = a.ckey[i];
                    u32 cx, cy, cz, scene;
                    decode_cell<BATCH>(pk, cx, cy, cz, scene);
                    const float4 xi = ro_ld(a.pos + guard(a, i, n));
                    DensitySum W;
                    u32 hits = 0;
                    if (staged) {
                        cx -= G.ox; cy -= G.oy; cz -= G.oz;   // 1 .. D - 2 per axis
                        const bool in = cx - 1u < G.Dx - 2u && cy - 1u < G.Dy - 2u && cz - 1u < G.Dz - 2u;
                        const u32 ring = (G.Dy + 1u) * G.Dz + 1u;   // from the first of the 27 cells to their middle
                        const u32 cell = in ? (cx * G.Dy + cy) * G.Dz + cz : ring;
                        const u32 s = S.rstart[b][cell], m0 = S.rpref[b][cell];
                        const u32 selfm = i - s < S.rpref[b][cell + 1u] - m0 ? m0 + (i - s) : 0xFFFF0000u;
                        hits = density_staged_row<C>(P, a, S, i, xi, S.rpref[b], cell - ring, G.Dy, G.Dz, selfm,
                                                     act && in, W);
                    } else if (act) {
                        hits = density_direct_row<BATCH>(P, a, i, pk, xi, W);
                    }
                    if (act) {
                        const float res[1] = {W.value()};
                        float resb[1] = {0.f};
                        if (a.nb > 0) density_boundary_row<BATCH>(P, a, xi, scene, i, resb);
                        float r_max = 0.f, r_s = 0.f, r_s2 = 0.f;
                        finish_row<PASS_DENSITY, BATCH>(P, a, i, res, resb, hits <= a.nbr_width ? hits : NBR_SPILL,
                                                        scene, 0.f, 0.f, r_max, r_s, r_s2);
                    }
                }
                if (listed || level == a.unit_level) break;
                i0 += rows;
                if (rows == 0u || i0 >= n || (a.ckey[i0] & unit_mask) != S.id[b]) break;   // the same for every thread
            } else {
                --level;
            }
            // the next part of a split unit
            id = a.ckey[i0] & block_mask<BATCH>(level);
            __syncthreads();
            if (tid == 0) {
                S.chunk = 0u;
                S.rows[b] = 0u;
            }
            __syncthreads();
            density_lookup<C, BATCH>(a, S, b, id, level);
            __syncthreads();
        }
        item = S.next;
        if (item < V.items) lookup_unit(item, b ^ 1u);
    }
}

}  // namespace
}  // namespace wcsph
