// One-pass fused RK4 step of a periodic level (FP32).
//
// The two sweeps of a step (rk4_level.cu) move 28 words per site: sweep A
// writes the stage increments (d3, d4, E, Q) to HBM and sweep B reads them
// back. This kernel keeps them on chip. A CTA owns a TX x TY tile of the xy
// plane over a chunk of z planes and marches in z. Per plane it
//   - runs sweep A on the tile plus a 2-cell halo (the A region) from a TMA
//     ring of (psi, Pi) planes with a 4-cell halo, and leaves d3, d4 and (on the
//     tile) E, Q in a window of planes in shared memory,
//   - runs sweep B two planes behind on the tile and writes psi, Pi of the
//     step's end to the other state buffer.
// level_pad_kernel then writes the periodic copies of that buffer's padding
// (8 columns, 2 rows and their corners): kept out of the step's loop, whose
// code the copy branches slowed by 8 % although few tiles take them.
// Reading one buffer and writing the other makes the tiles independent (no
// tile reads what another writes), so the CTAs need no synchronisation with
// each other; the level's work buffer serves as the second state buffer and
// steps alternate between the two. A step moves 8 words per site (psi, Pi in
// and out) plus the halo rows the L2 does not catch, against 28 for the two
// sweeps; in return sweep A runs on (TX+4)(TY+4) sites per TX*TY.
//
// Columns in registers. The march is bound by the shared-memory pipe, the FP32
// pipe and issue together (70 %, 62 % and 71 % busy at 256^3), not by HBM, so the work
// per plane is kept to arithmetic. A thread owns two neighbouring sites for the
// whole march and keeps their column, of (psi, Pi) for sweep A or (d3, d4) for
// sweep B, in registers as the differences the z taps are made of
// (FusedColumn): a plane takes 28 shared loads for a unit of sweep A and 36 for
// one of sweep B, where 13 taps a Laplacian from shared memory took 44 and 52,
// and two packed additions fewer a Laplacian. The march is unrolled by three,
// so that the columns rotate by renaming.
// Warps: 12 of sweep A (the tile's and the halo's units), 8 of sweep B, one
// that issues the TMA loads. They hand planes on through four sets of
// mbarriers (a ring slot has landed / was read, a window slot was stored / was
// read), so sweep A runs ahead of sweep B and no warp waits for the block. 24
// warps of 80 registers fill the register file (one CTA per SM); setmaxnreg
// moves the producer's to the others (88 for sweep A, 96 for sweep B: at 80
// both spilled and ran 40 % slower).
// Measured, this kernel alone at 512^3: 1.67 ms, against 2.57 ms with all taps
// from shared memory and a block barrier per plane; the same columns in 12
// warps that ran both sweeps took 2.34 ms (three warps a scheduler left the
// latencies of shared loads and additions open). Window slots: with 5 instead
// of 4 sweep A runs two planes ahead and the step takes 6 % longer.
//
// The per-site arithmetic is the two sweeps' own (lap_taps, stage_a,
// stage_b), so both paths give the same bits.
//
// Halo: the box is (TX+8) x (TY+8) x 1 plane x 4 components, starting 4
// columns and 4 rows before the tile. In x the level's padding columns hold
// the periodic copies. In y the padding holds 2 rows of the 4 a box needs:
// tiles in the first or last row of tiles load their planes as pieces that
// skip the padding (4 wrapped rows beside TY+4 rows; pieces of 4 rows alone
// where one row of tiles wraps at both ends). Pieces of 4 rows keep every
// destination 128-byte aligned. z wraps by plane index. Extents that are no
// multiple of the tile: in x the last tile column runs past the box and masks
// its stores (it reads up to 4 padding columns; sites further right feed only
// masked ones); in y the tile rows are spread evenly and overlap, so that
// every tile is whole and only the first and the last touch the box's edge
// (fused_tiles_ny). Sites that two tiles own are written twice with the same
// bits.
#pragma once

#include "rk4_ops.cuh"

namespace axs {

// Whether the fused step takes a box of ny rows, and its rows of tiles: one
// tile, or evenly spread tiles of which no inner one reaches within 2 rows of
// the padding's end (ny >= TY + 4 keeps two wrapped pieces apart).
__host__ __device__ constexpr bool fused_takes_ny(int ny, int ty) { return ny == ty || ny >= ty + 4; }
__host__ __device__ constexpr int fused_tiles_ny(int ny, int ty) { return (ny + ty - 1) / ty; }

template <int TX_, int TY_, bool COMP_ = false> struct LevelFusedShape {
    using T = float;
    static constexpr bool COMP = COMP_;  // the compensated FP32 step (stage_a in rk4_ops.cuh)
    static constexpr int V = 2, TX = TX_, TY = TY_;
    static constexpr int U = 4;                     // window slots
    static constexpr int NS = 8;                    // ring slots
    static constexpr int BX = TX + 8, BY = TY + 8;  // TMA box: the A region and its stencil halo
    static constexpr int AX = TX + 4, AY = TY + 4;  // A region
    static constexpr int RING = 4 * BX * BY, WIN = 4 * AX * AY, EQW = 4 * TX * TY;
    static constexpr int NT = TX * TY / V;          // units of the tile: threads of sweep B, and of sweep A
    static constexpr int NH = 4 * (AX / V) + 2 * TY;  // halo units: 4 whole rows and 2 a tile row
    static constexpr int WA = (NT + NH + 31) / 32, WB = NT / 32;     // warps of sweep A and of sweep B
    static constexpr int THREADS = 32 * (WA + WB + 4);               // and the producer's warpgroup
    static constexpr size_t SMEM = sizeof(T) * ((size_t)NS * RING + U * ((size_t)WIN + EQW));
    static constexpr uint32_t SLOT_BYTES = RING * sizeof(T);
    static_assert(THREADS <= 1024 && NT % 32 == 0, "whole warps of each kind");
    static_assert((4 * BX * sizeof(T)) % 128 == 0 && ((TY + 4) * BX * sizeof(T)) % 128 == 0,
                  "the pieces of a split box land 128-byte aligned");
    static_assert((RING * sizeof(T)) % 128 == 0 && (BX * BY * sizeof(T)) % 128 == 0, "ring slots and components");
    static_assert(TY % 4 == 0 && BX <= 256 && BY <= 256, "pieces of 4 rows; TMA box extent limit");
    static_assert(NS >= 5 + U - 2, "sweep A's five planes, up to U - 2 ahead of sweep B's");
    static_assert(SMEM + 1024 <= 227 * 1024, "shared memory");
    static_assert(WA == 12 && WB == 8, "whole warpgroups and the register split of the kernel");
};

// The three tensor maps over one state buffer: the whole box (inner tile
// rows), one component of TY + 4 rows, one component of 4 rows.
struct LevelFusedMaps {
    CUtensorMap full, mid, rows4;
};

// A work item of the fused step: a TX x TY tile over a chunk of z planes of
// one periodic box, with the box's geometry and the three tensor maps of the
// buffer the step reads.
struct FusedItem {
    int x0, y0, z0, len;
    int nx, ny, nz;
    int64_t js, ks, base;  // base: element offset of the box in every component plane
    const CUtensorMap *full, *mid, *rows4;
};

// A block's walk over its work items (the producer thread and the consumers
// each keep one).
struct FusedCursor {
    int64_t pos, end;
};

// First row of tile row t of `rows`: evenly spread from 0 to ny - TY.
template <int TY> __device__ __forceinline__ int fused_tile_y0(int t, int rows, int ny)
{
    return rows > 1 ? t * (ny - TY) / (rows - 1) : 0;
}

// Work-item sources of the fused step: begin / valid / item / next.
// One periodic level in (tile, z-chunk) items, taken by blocks in turn;
// geometry from the launch parameters.
struct FusedLevel {
    static constexpr bool kMapsInTable = false;  // maps by value in the launch parameters
    static constexpr bool kPatches = false;
    __device__ __forceinline__ static FusedCursor begin(const SweepArgs<float> &a) { return {blockIdx.x, a.n_items}; }
    __device__ __forceinline__ static bool valid(const FusedCursor &c) { return c.pos < c.end; }
    __device__ __forceinline__ static void next(FusedCursor &c, const SweepArgs<float> &) { c.pos += gridDim.x; }
    template <int TX, int TY>
    __device__ __forceinline__ static FusedItem item(const SweepArgs<float> &a, const LevelFusedMaps &m,
                                                     const FusedCursor &c)
    {
        const int tile = (int)(c.pos % a.ntiles);
        const int z0 = (int)(c.pos / a.ntiles) * a.zchunk;
        const int y0 = fused_tile_y0<TY>(tile / a.tiles_x, a.ntiles / a.tiles_x, a.ny);
        return FusedItem{(tile % a.tiles_x) * TX, y0, z0, min(a.zchunk, a.nz - z0), a.nx, a.ny, a.nz, a.js, a.ks, 0,
                         &m.full, &m.mid, &m.rows4};
    }
};
// The boxes of an ensemble: the item list and box descriptors of a box table,
// and per box six tensor maps in the table (full, mid, rows4 over each of the
// two state buffers; map_sel picks the buffer read).
struct FusedBoxes {
    static constexpr bool kMapsInTable = true;  // written by a host copy: acquired before use
    static constexpr bool kPatches = false;
    __device__ __forceinline__ static FusedCursor begin(const SweepArgs<float> &a) { return {blockIdx.x, a.n_items}; }
    __device__ __forceinline__ static bool valid(const FusedCursor &c) { return c.pos < c.end; }
    __device__ __forceinline__ static void next(FusedCursor &c, const SweepArgs<float> &) { c.pos += gridDim.x; }
    template <int TX, int TY>
    __device__ __forceinline__ static FusedItem item(const SweepArgs<float> &a, const LevelFusedMaps &,
                                                     const FusedCursor &c)
    {
        const uint32_t e = __ldg(a.items + c.pos);
        const EnsBoxDesc &d = a.boxes[e >> kEnsItemBits];
        const int local = (int)(e & ((1u << kEnsItemBits) - 1));
        const int tile = local % d.ntiles;
        const int z0 = (local / d.ntiles) * d.zchunk;
        const int y0 = fused_tile_y0<TY>(tile / d.tiles_x, d.ntiles / d.tiles_x, d.ny);
        const CUtensorMap *m = a.maps + 3 * (2 * d.map_box + a.map_sel);
        return FusedItem{(tile % d.tiles_x) * TX, y0, z0, min(d.zchunk, d.nz - z0), d.nx, d.ny, d.nz, d.js, d.ks,
                         d.base, m, m + 1, m + 2};
    }
};

// The refined patches of a level (amr.cu), stepped in place: npatches = n_items
// boxes of nx cells a side with explicit ghost rings (4 rows and planes, so no
// piece of a load and no plane index wraps), their tiles a thread-block cluster
// that takes patches in turn; cs holds the elements of a patch in a component
// plane, maps two tensor maps a patch (the second boxes the state). A plane is
// overwritten by sweep B once it has landed in every tile of its patch: a tile
// tells the others of every kTell planes (the kernel's peer barriers, one per kTell
// ring slots; sweep A is 4 planes ahead of sweep B, so 4 have landed before the first
// is to be stored). The telling releases and sweep B's wait acquires at cluster scope,
// which puts the stores after the other tiles' loads. 1638 patches of 32^3: 0.82 ms a
// step, against 1.13 with all taps from shared memory, one patch a cluster and a
// cluster barrier per plane; telling of every plane costs 1.10, and doing that without
// release and acquire, which no memory model orders, 0.86.
// A peer barrier counts ntiles arrivals a round, whoever they come from. It
// completes a round only when every tile has told of its planes, although one tile's
// word may arrive after another's of the next round: a tile tells of round r + 1 (the
// planes NS on) only after its own barrier has completed round r, since sweep B frees
// the slots after that. Suppose a barrier were the first of all to complete a round r
// that tile Z has not told of. Of the ntiles (r + 1) arrivals it has counted (rounds
// from 0), at most r are Z's, so more than r + 1 are another tile's: that one has told
// of round r + 1, and its own barrier completed round r earlier. And telling means
// having landed, whichever tile hears of it first.
struct FusedPatches {
    static constexpr bool kMapsInTable = true;
    static constexpr bool kPatches = true;
    static constexpr int kRows = 4, kPlanes = 4;  // ghost rows and planes below the valid cells
    static constexpr int kTell = 4;               // sides are multiples of 32: items of whole groups
    __device__ __forceinline__ static FusedCursor begin(const SweepArgs<float> &a)
    {
        return {(int)blockIdx.x / a.ntiles, a.n_items};
    }
    __device__ __forceinline__ static bool valid(const FusedCursor &c) { return c.pos < c.end; }
    __device__ __forceinline__ static void next(FusedCursor &c, const SweepArgs<float> &a) { c.pos += (int)gridDim.x / a.ntiles; }
    template <int TX, int TY>
    __device__ __forceinline__ static FusedItem item(const SweepArgs<float> &a, const LevelFusedMaps &,
                                                     const FusedCursor &c)
    {
        const int tile = (int)blockIdx.x % a.ntiles;
        const CUtensorMap *m = a.maps + 2 * c.pos + 1;
        return FusedItem{(tile % a.tiles_x) * TX, (tile / a.tiles_x) * TY, kPlanes, a.nx, a.nx, a.nx, a.nx + 2 * kPlanes,
                         a.js, a.ks, c.pos * a.cs, m, m, m};
    }
};

__device__ __forceinline__ float2 lds2(const unsigned char *p) { return *reinterpret_cast<const float2 *>(p); }

// A thread's column of four components through the march, as the differences
// the stencil is made of: f(z+1) - f(z) serves z and, negated, z+1; f(z+2) - f(z)
// serves z and z+2. Step: the plane z+2 comes in as `f[P + 2]`; the z sums of
// plane z are handed out and the column moves on. P, the step modulo 3, makes
// the indices constants.
struct FusedColumn {
    F2 f[3][4];   // planes z, z+1, z+2
    F2 u1[4];     // f(z) - f(z-1)
    F2 u2[3][4];  // f(z+1) - f(z-1), f(z) - f(z-2); the third: room for f(z+2) - f(z)
    template <int P> __device__ __forceinline__ const F2 &mid(int c) const { return f[P % 3][c]; }
    template <int P> __device__ __forceinline__ F2 &in(int c) { return f[(P + 2) % 3][c]; }
    template <int P> __device__ __forceinline__ void sums(int c, F2 &z1, F2 &z2)
    {
        const F2 d1 = f[(P + 1) % 3][c] - f[P % 3][c], d2 = f[(P + 2) % 3][c] - f[P % 3][c];
        z1 = d1 - u1[c];
        z2 = d2 - u2[P % 3][c];  // u2[P % 3]: f(z) - f(z-2), of the step before last
        u1[c] = d1;
        u2[(P + 2) % 3][c] = d2;
    }
};

// Laplacians of a thread's two sites of the four components: xy taps from a
// plane in shared memory (p: the first site, component 0; RB the row length and
// CB the component stride in bytes), centre and z sums from the column.
template <int P, int RB, int CB, bool COMP>
__device__ __forceinline__ void star4_column(const SweepArgs<float> &a, const unsigned char *p, FusedColumn &col,
                                             F2 (&lap)[4])
{
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const unsigned char *q = p + c * CB;
        F2 z1, z2;
        col.sums<P>(c, z1, z2);
        lap[c] = lap_taps<COMP>(a, lds2(q - 8), col.mid<P>(c).v, lds2(q + 8), lds2(q - RB), lds2(q + RB),
                                lds2(q - 2 * RB), lds2(q + 2 * RB), z1, z2);
    }
}

template <class S, class Src = FusedLevel>
__global__ void __launch_bounds__(S::THREADS, 1)
    level_fused_kernel(const __grid_constant__ LevelFusedMaps maps, const SweepArgs<float> a)
{
    constexpr int V = S::V, TX = S::TX, TY = S::TY, NS = S::NS, U = S::U, BX = S::BX, BY = S::BY, AX = S::AX,
                  AY = S::AY;
    constexpr int SLOT = (int)S::SLOT_BYTES, WSLOT = S::WIN * 4, ESLOT = S::EQW * 4;
    // row and component strides in a ring slot, a (d3, d4) window slot and an (E, Q) window slot, bytes
    constexpr int RB = BX * 4, RC = BX * BY * 4, WB = AX * 4, WC = AX * AY * 4, EC = TX * TY * 4;
    extern __shared__ __align__(128) unsigned char lf_smem[];
    unsigned char *const win = lf_smem + (size_t)NS * SLOT, *const eqw = win + (size_t)U * WSLOT;
    // ring slots: landed, and read (by sweep B, last); window slots: stored, and read;
    // of patches, groups of ring slots: landed in every tile of the patch
    constexpr int TELL = FusedPatches::kTell;
    static_assert(NS % TELL == 0, "whole groups");
    __shared__ uint64_t bars[2 * NS + 2 * U + NS / TELL];
    __shared__ int failed;
    const int tid = threadIdx.x, warp = tid >> 5;
    const bool lane0 = (tid & 31) == 0;
    constexpr int oy = Src::kPatches ? 4 : 2;  // padded row of y = 0

    if (tid == 0) {
        for (int k = 0; k < NS; ++k) {
            mbar_init(&bars[k], 1);
            mbar_init(&bars[NS + k], S::WB);
            if (Src::kPatches && k % TELL == 0) mbar_init(&bars[2 * NS + 2 * U + k / TELL], (uint32_t)a.ntiles);
        }
        for (int k = 0; k < U; ++k) {
            mbar_init(&bars[2 * NS + k], S::WA);
            mbar_init(&bars[2 * NS + U + k], S::WB);
        }
        fence_mbar_init();
        failed = 0;
    }
    __syncthreads();
    if constexpr (Src::kPatches) cluster_meet();  // the other tiles' barriers are set up

    // A wait is a test whose answer is looked at a step later, and a bounded wait
    // where it said no: the latency of a wait at its point of use would lie on the
    // warp's path. A warp whose wait expired leaves the march there and then: it hands
    // nothing on, so what waits for it expires as well (at once: the waits see
    // `failed`), and sweep B stores nothing that was made from data still to come.
    uint32_t bar0 = smem_addr(bars);
    asm volatile("" : "+r"(bar0));  // kept, not recomputed
    auto landed = [&](int k) { return bar0 + 8u * k; };
    auto ring_read = [&](int k) { return bar0 + 8u * (NS + k); };
    auto stored = [&](int k) { return bar0 + 8u * (2 * NS + k); };
    auto win_read = [&](int k) { return bar0 + 8u * (2 * NS + U + k); };
    auto peers = [&](int k) { return bar0 + 8u * (2 * NS + 2 * U + k / TELL); };
    auto slow_wait = [&](uint32_t bar, uint32_t phase, auto cluster) -> bool {
        for (uint32_t it = 0; it < a.wait_polls; ++it) {
            if (mbar_try_wait_at<decltype(cluster)::value>(bar, phase)) return true;
            if ((it & 63) == 63 && *(volatile int *)&failed) return false;
        }
        if (*(volatile int *)&failed) return false;
        atomicOr(a.status, kDevTimeout);
        *(volatile int *)&failed = 1;
        return false;
    };
    constexpr std::false_type here_only{};
    // the whole warp's wait (cluster: for what another block of the cluster has told)
    auto need = [&](bool ready, uint32_t bar, uint32_t phase, auto cluster) -> bool {
        if (__all_sync(0xffffffffu, ready)) return true;
        return __all_sync(0xffffffffu, slow_wait(bar, phase, cluster)) != 0;
    };

    // March of an item. Planes are numbered from z0 - 4. Step i = 0 .. len + 3: sweep A
    // at plane i + 2 = z0 - 2 + i, with plane i + 4 new in the column; sweep B at plane
    // i = z0 - 4 + i, from i = 4 on, with d3, d4 of step i new in its column.
    if (warp >= S::WA + S::WB) {
        // registers: 24 warps x 80 at launch = 12 x 88 + 8 x 96 + 4 x 24
        asm volatile("setmaxnreg.dec.sync.aligned.u32 24;");
        // ---- producer: planes z0 - 4 .. z0 + len + 3 of each item, one after the other
        if (tid == 32 * (S::WA + S::WB)) {
            if constexpr (!Src::kMapsInTable) {
                prefetch_tensormap(&maps.full);
                prefetch_tensormap(&maps.mid);
                prefetch_tensormap(&maps.rows4);
            }
            int slot = 0;
            int64_t sent = 0;
            uint32_t phase = 1;  // of ring_read: the first round of slots is free
            bool ok = true;
            for (FusedCursor cur = Src::begin(a); ok && Src::valid(cur); Src::next(cur, a)) {
                const FusedItem p = Src::template item<TX, TY>(a, maps, cur);
                if constexpr (Src::kMapsInTable) {
                    fence_tensormap_acquire(p.full);
                    fence_tensormap_acquire(p.mid);
                    fence_tensormap_acquire(p.rows4);
                }
                int zp = p.z0 - 4;  // nz may be smaller than 4
                while (zp < 0) zp += p.nz;
                const int xc = a.ox - 4 + p.x0;  // padded column of the box's first column (16-byte aligned)
                const bool lo = !Src::kPatches && p.y0 == 0, hi = !Src::kPatches && p.y0 + TY == p.ny;
                for (int k = 0; k < p.len + 8; ++k) {
                    if (!(ok = slow_wait(ring_read(slot), phase, here_only))) break;
                    unsigned char *dst = lf_smem + (size_t)slot * SLOT;
                    uint64_t *bar = &bars[slot];
                    mbar_arrive_expect_tx(bar, S::SLOT_BYTES);
                    ++sent;
                    if (!lo && !hi) {
                        tma_load_4d(dst, p.full, xc, p.y0 - 4 + oy, zp, 0, bar);
                    } else if (lo && hi) {
                        for (int c = 0; c < 4; ++c)
                            for (int r = 0; r < BY; r += 4)
                                tma_load_4d(dst + c * RC + r * RB, p.rows4, xc, (r + TY - 4) % TY + oy, zp, c, bar);
                    } else {
                        // rows y0 - 4 .. y0 + TY + 3 as 4 wrapped rows below the others (first tile row) or above them
                        const int r4 = lo ? 0 : TY + 4, y4 = lo ? p.ny - 4 : 0, rm = lo ? 4 : 0, ym = lo ? 0 : p.y0 - 4;
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            tma_load_4d(dst + c * RC + r4 * RB, p.rows4, xc, y4 + oy, zp, c, bar);
                            tma_load_4d(dst + c * RC + rm * RB, p.mid, xc, ym + oy, zp, c, bar);
                        }
                    }
                    if (++zp == p.nz) zp = 0;
                    if (++slot == NS) {
                        slot = 0;
                        phase ^= 1;
                    }
                }
            }
            // No bulk copy may still be landing in shared memory when the block ends
            // (after an expired wait; bounded as well).
            for (int64_t v = sent > NS ? sent - NS : 0; v < sent; ++v)
                mbar_wait_bounded(&bars[v % NS], (uint32_t)((v / NS) & 1), 1u << 20);
        } else if (Src::kPatches && warp == S::WA + S::WB + 1) {
            // ---- the warp that tells the patch's tiles, this one too, of the planes that
            // have landed here (lane: the tile told)
            int slot = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (FusedCursor cur = Src::begin(a); ok && Src::valid(cur); Src::next(cur, a))
                for (int k = 0; k < a.nx + 2 * 4; ++k) {
                    if (!(ok = need(false, landed(slot), phase, here_only))) break;
                    if (slot % TELL == TELL - 1 && (tid & 31) < a.ntiles) mbar_arrive_cluster(peers(slot), tid & 31);
                    if (++slot == NS) {
                        slot = 0;
                        phase ^= 1;
                    }
                }
        }
    } else
    if (warp < S::WA) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 88;");
        // ---- sweep A. Units: the tile's, 16 pairs to a row; 16 pairs of each of the
        // halo's four rows; then groups of 8, four rows' pairs at the left and right
        // end, and the rest of the four halo rows (idle lanes of the last warp repeat
        // that group and store nothing). Half a warp reads whole bank rows, and a
        // group's 8 pairs lie in different banks of a ring plane (rows 40 words
        // apart); halo units in row order took 180 more wavefronts of 1670 a plane.
        static_assert(TX == 32 && TY % 4 == 0, "16 pairs to a row, groups of four rows");
        const bool tile_site = tid < S::NT;
        const int h = tid - S::NT;
        const bool has_a = h < S::NH;
        int alx, aly;  // A-region-local first site
        if (tile_site) {
            alx = 2 + V * (tid % 16);
            aly = 2 + tid / 16;
        } else if (h < 64) {
            alx = V * (h % 16);
            aly = h / 16 < 2 ? h / 16 : TY + h / 16;
        } else {
            const int g = min((h - 64) / 8, TY / 4), row = h & 3, right = (h >> 2) & 1;
            alx = right ? AX - 2 : g < TY / 4 ? 0 : AX - 4;
            aly = g < TY / 4 ? 2 + 4 * g + row : row < 2 ? row : TY + row;
        }
        const int site = 4 * ((aly + 2) * BX + alx + 2);
        unsigned char *const wsite = win + 4 * (aly * AX + alx), *const esite = eqw + 8 * tid;
        int slot = 0, off_new = site, off_mid;  // ring slot of plane i + 4; this site in it and in plane i + 2's
        int ws = 0;                             // window slot of step i
        uint32_t landed_phase = 0, read_phase = 1;  // of slot's next landing; of win_read (the first round is free)
        auto next_off = [&](int &off) {
            off += SLOT;
            if (off >= NS * SLOT) off -= NS * SLOT;
        };
        auto take_plane = [&](bool ready) -> bool {
            if (!need(ready, landed(slot), landed_phase, here_only)) return false;
            if (++slot == NS) {
                slot = 0;
                landed_phase ^= 1;
            }
            return true;
        };
        FusedColumn col;
        auto march = [&]() {  // returns when it is done or a wait expired
            for (FusedCursor cur = Src::begin(a); Src::valid(cur); Src::next(cur, a)) {
                const int n = Src::template item<TX, TY>(a, maps, cur).len + 4;
                {
                    F2 first[4][4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        if (!take_plane(false)) return;
                        if (k == 2) off_mid = off_new;
#pragma unroll
                        for (int c = 0; c < 4; ++c) first[k][c] = F2(lds2(lf_smem + off_new + c * RC));
                        next_off(off_new);
                    }
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        col.f[0][c] = first[2][c];
                        col.f[1][c] = first[3][c];
                        col.u1[c] = first[2][c] - first[1][c];
                        col.u2[1][c] = first[3][c] - first[1][c];
                        col.u2[0][c] = first[2][c] - first[0][c];
                    }
                }
                bool ready = false;
                auto step = [&](auto ph) -> bool {
                    constexpr int P = decltype(ph)::value;
                    if (!take_plane(ready)) return false;
                    ready = mbar_test_at(landed(slot), landed_phase);
                    const bool free = mbar_test_at(win_read(ws), read_phase);
#pragma unroll
                    for (int c = 0; c < 4; ++c) col.in<P>(c) = F2(lds2(lf_smem + off_new + c * RC));
                    next_off(off_new);
                    F2 lap[4];
                    star4_column<P, RB, RC, S::COMP>(a, lf_smem + off_mid, col, lap);
                    next_off(off_mid);
                    const StageAPair sa = stage_a_pair<S::COMP>(a, col.mid<P>(0), col.mid<P>(1), col.mid<P>(2),
                                                                col.mid<P>(3), lap[0], lap[1], lap[2], lap[3]);
                    if (!need(free, win_read(ws), read_phase, here_only)) return false;
                    unsigned char *const wz = wsite + ws * WSLOT, *const ez = esite + ws * ESLOT;
                    if (has_a) {
#pragma unroll
                        for (int c = 0; c < 4; ++c) *reinterpret_cast<float2 *>(wz + c * WC) = sa.d[c].v;
                    }
                    if (tile_site) {
                        F2 eq[4];
                        stage_a_eq<S::COMP>(a, sa, lap[0], lap[1], eq);
#pragma unroll
                        for (int c = 0; c < 4; ++c) *reinterpret_cast<float2 *>(ez + c * EC) = eq[c].v;
                    }
                    __syncwarp();
                    if (lane0) mbar_arrive_at(stored(ws));
                    if (++ws == U) {
                        ws = 0;
                        read_phase ^= 1;
                    }
                    return true;
                };
                for (int i = 0;;) {
                    if (!step(std::integral_constant<int, 0>{})) return;
                    if (++i == n) break;
                    if (!step(std::integral_constant<int, 1>{})) return;
                    if (++i == n) break;
                    if (!step(std::integral_constant<int, 2>{})) return;
                    if (++i == n) break;
                }
            }
        };
        march();
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 96;");
        // ---- sweep B, a unit of the tile to a thread
        const int bt = tid - 32 * S::WA;
        const int bx = V * (bt % (TX / V)), by = bt / (TX / V);  // tile-local first site
        const unsigned char *const wsite = win + 4 * ((by + 2) * AX + bx + 2), *const esite = eqw + 8 * bt;
        int slot = 0, off_y = 4 * ((by + 4) * BX + bx + 4);  // ring slot of plane i, this site in it
        int ws = 0, wm = 0;                                  // window slots of steps i and i - 2
        uint32_t stored_phase = 0, landed_phase = 0;
        // at the first plane of a group: the group has landed in all tiles
        auto peers_landed = [&]() -> bool {
            if (slot % TELL != 0) return true;
            return need(mbar_test_at<true>(peers(slot), landed_phase), peers(slot), landed_phase, std::true_type{});
        };
        auto release_plane = [&]() {  // after the warp's reads of it
            if (lane0) mbar_arrive_at(ring_read(slot));
            off_y += SLOT;
            if (++slot == NS) {
                slot = 0;
                off_y -= NS * SLOT;
                landed_phase ^= 1;
            }
        };
        auto release_window = [&]() {
            if (lane0) mbar_arrive_at(win_read(wm));
            if (++wm == U) wm = 0;
        };
        FusedColumn col;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            for (int k = 0; k < 3; ++k) col.f[k][c] = col.u2[k][c] = F2(0.f);
            col.u1[c] = F2(0.f);
        }
        auto march = [&]() {  // returns when it is done or a wait expired
            for (FusedCursor cur = Src::begin(a); Src::valid(cur); Src::next(cur, a)) {
                const FusedItem w = Src::template item<TX, TY>(a, maps, cur);
                const bool in_box = w.x0 + bx < w.nx;
                int64_t off = w.base + (int64_t)(w.x0 + bx + a.ox) + (int64_t)(w.y0 + by + oy) * w.js + (int64_t)w.z0 * w.ks;
                const int n = w.len + 4;
                bool ready = false;
                auto step = [&](auto ph, int i) -> bool {
                    constexpr int P = decltype(ph)::value;
                    if (!need(ready, stored(ws), stored_phase, here_only)) return false;
                    const unsigned char *const wz = wsite + ws * WSLOT;
                    if (++ws == U) {
                        ws = 0;
                        stored_phase ^= 1;
                    }
                    ready = mbar_test_at(stored(ws), stored_phase);
                    const bool here = mbar_test_at(landed(slot), landed_phase);  // long since: sweep A has read the plane
                    // every group, stored or not: it keeps the rounds of `peers` apart
                    if constexpr (Src::kPatches)
                        if (!peers_landed()) return false;
#pragma unroll
                    for (int c = 0; c < 4; ++c) col.in<P>(c) = F2(lds2(wz + c * WC));
                    if (i >= 4) {
                        // (E, Q) of plane i with its d3, d4, stored at step i - 2, and its psi_n, Pi_n
                        if (!need(here, landed(slot), landed_phase, here_only)) return false;
                        F2 lap[4], e[4], y[4], o[4];
                        star4_column<P, WB, WC, S::COMP>(a, wsite + wm * WSLOT, col, lap);
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            e[c] = F2(lds2(esite + wm * ESLOT + c * EC));
                            y[c] = F2(lds2(lf_smem + off_y + c * RC));
                        }
                        stage_b_pair<S::COMP>(a, col.mid<P>(0), col.mid<P>(1), col.mid<P>(2), col.mid<P>(3), lap, e, y, o);
                        if (in_box) {
#pragma unroll
                            for (int c = 0; c < 4; ++c) *reinterpret_cast<float2 *>(a.out[c] + off) = o[c].v;
                        }
                        off += w.ks;
                    } else {
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            F2 z1, z2;
                            col.sums<P>(c, z1, z2);
                        }
                    }
                    __syncwarp();
                    release_plane();
                    if (i >= 2) release_window();
                    return true;
                };
                for (int i = 0;;) {
                    if (!step(std::integral_constant<int, 0>{}, i)) return;
                    if (++i == n) break;
                    if (!step(std::integral_constant<int, 1>{}, i)) return;
                    if (++i == n) break;
                    if (!step(std::integral_constant<int, 2>{}, i)) return;
                    if (++i == n) break;
                }
                // the item's last planes: sweep A is done with them, and nothing reads the last two window slots
                if constexpr (Src::kPatches)
                    if (!peers_landed()) return;
                for (int k = 0; k < 4; ++k) release_plane();
                release_window();
                release_window();
            }
        };
        march();
    }
    // no tile leaves while another may still tell it of a plane
    if constexpr (Src::kPatches) cluster_meet();
}

// The periodic padding of one level-layout buffer (4 components): columns
// x = -8 .. -1 and nx .. nx+7 of rows y = -2 .. ny+1, and rows y = -2, -1, ny,
// ny+1 of columns 0 .. nx-1, each a copy of the valid cell it wraps to. Grid
// rows are planes (z + nz c); within a plane, consecutive threads take
// consecutive quads of a padding row (nx and the layout's offsets are multiples
// of 4 cells), and each thread copies kPadUnroll quads a grid-row stride apart,
// all loads before the stores (sources are valid cells of `from`, destinations
// padding: no copy reads another's destination). Latency-bound: a cell at a
// time took 1.9 us more of a 128^3 step (48.1 -> 46.2 us; 64^3 17.5 -> 16.5 us).
constexpr int kPadUnroll = 4;
__host__ __device__ constexpr int pad_quads(int nx, int ny) { return 4 * (ny + 4) + nx; }  // of a plane
template <typename T>
__device__ __forceinline__ void pad_box(T *buf, const T *from, int nx, int ny, int nz, int64_t js, int64_t ks,
                                        int64_t cs, int ox, int oy)
{
    using V4 = typename VecN<T, 4>::type;
    const int xpad = 4 * (ny + 4), per_plane = pad_quads(nx, ny), quads = nx / 4;
    const int stride = gridDim.x * blockDim.x;
    for (int plane = blockIdx.y; plane < 4 * nz; plane += gridDim.y) {
        const int64_t at = (int64_t)(plane / nz) * cs + (int64_t)(plane % nz) * ks + ox + (int64_t)oy * js;
        T *p = buf + at;
        const T *s = from + at;
        for (int r0 = blockIdx.x * blockDim.x + threadIdx.x; r0 < per_plane; r0 += kPadUnroll * stride) {
            int64_t dst[kPadUnroll], src[kPadUnroll];
            bool on[kPadUnroll];
#pragma unroll
            for (int u = 0; u < kPadUnroll; ++u) {
                const int r = r0 + u * stride;
                int x, y;
                if (r < xpad) {  // x padding: 4 quads of every padded row
                    const int k = r & 3;
                    x = k < 2 ? 4 * k - 8 : nx + 4 * (k - 2);
                    y = (r >> 2) - 2;
                } else {  // y padding: 4 rows of the valid columns
                    const int rr = r - xpad, k = rr / quads;
                    x = 4 * (rr - k * quads);
                    y = k < 2 ? k - 2 : ny + (k - 2);
                }
                int xs = x < 0 ? x + nx : (x >= nx ? x - nx : x);
                xs = xs < 0 ? xs + nx : (xs >= nx ? xs - nx : xs);  // 8 columns may wrap twice: nx is at least 4
                const int ys = y < 0 ? y + ny : (y >= ny ? y - ny : y);
                on[u] = r < per_plane;
                dst[u] = x + (int64_t)y * js;
                src[u] = on[u] ? xs + (int64_t)ys * js : 0;
            }
            V4 v[kPadUnroll];
#pragma unroll
            for (int u = 0; u < kPadUnroll; ++u) v[u] = *reinterpret_cast<const V4 *>(s + src[u]);
#pragma unroll
            for (int u = 0; u < kPadUnroll; ++u)
                if (on[u]) *reinterpret_cast<V4 *>(p + dst[u]) = v[u];
        }
    }
}

template <typename T>
__global__ void level_pad_kernel(T *__restrict__ buf, int nx, int ny, int nz, int64_t js, int64_t ks, int64_t cs,
                                 int ox, int oy)
{
    pad_box(buf, buf, nx, ny, nz, js, ks, cs, ox, oy);
}

// The valid cells of a level-layout buffer with their periodic padding, from
// another buffer's valid cells: the end of a run of an odd number of fused
// steps, which leaves the result in the second buffer. Grid rows are planes;
// within a plane the first nx ny / 4 tasks copy four cells each, the others
// write the padding (pad_box, sources in src).
template <typename T>
__device__ __forceinline__ void copy_pad_box(T *__restrict__ dst, const T *__restrict__ src, int nx, int ny, int nz,
                                             int64_t js, int64_t ks, int64_t cs, int ox, int oy)
{
    using V4 = typename VecN<T, 4>::type;
    const int quads = nx / 4, units = quads * ny;
    for (int plane = blockIdx.y; plane < 4 * nz; plane += gridDim.y) {
        const int64_t at = (int64_t)(plane / nz) * cs + (int64_t)(plane % nz) * ks + ox + (int64_t)oy * js;
        const int stride = gridDim.x * blockDim.x;
        for (int r0 = blockIdx.x * blockDim.x + threadIdx.x; r0 < units; r0 += kPadUnroll * stride) {
            V4 v[kPadUnroll];
            int64_t o[kPadUnroll];
#pragma unroll
            for (int u = 0; u < kPadUnroll; ++u) {
                const int r = min(r0 + u * stride, units - 1), y = r / quads;
                o[u] = at + 4 * (r - y * quads) + (int64_t)y * js;
                v[u] = *reinterpret_cast<const V4 *>(src + o[u]);
            }
#pragma unroll
            for (int u = 0; u < kPadUnroll; ++u)
                if (r0 + u * stride < units) *reinterpret_cast<V4 *>(dst + o[u]) = v[u];
        }
    }
    pad_box(dst, src, nx, ny, nz, js, ks, cs, ox, oy);
}

template <typename T>
__global__ void level_copy_pad_kernel(T *__restrict__ dst, const T *__restrict__ src, int nx, int ny, int nz, int64_t js,
                                      int64_t ks, int64_t cs, int ox, int oy)
{
    copy_pad_box(dst, src, nx, ny, nz, js, ks, cs, ox, oy);
}

// The same for every box of an ensemble buffer, one box per blockIdx.z.
template <typename T>
__global__ void ens_pad_kernel(T *__restrict__ buf, const EnsBoxDesc *__restrict__ boxes, int64_t cs, int ox)
{
    const EnsBoxDesc &d = boxes[blockIdx.z];
    pad_box(buf + d.base, buf + d.base, d.nx, d.ny, d.nz, d.js, d.ks, cs, ox, d.oy);
}

template <typename T>
__global__ void ens_copy_pad_kernel(T *__restrict__ dst, const T *__restrict__ src,
                                    const EnsBoxDesc *__restrict__ boxes, int64_t cs, int ox)
{
    const EnsBoxDesc &d = boxes[blockIdx.z];
    copy_pad_box(dst + d.base, src + d.base, d.nx, d.ny, d.nz, d.js, d.ks, cs, ox, d.oy);
}

}  // namespace axs
