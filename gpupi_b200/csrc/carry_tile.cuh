// Block- and grid-level binary carry resolution shared by every kernel that
// ends in a carry pass (carry-chain ops, NTT CRT stage, schoolbook).
//
// Scheme for a row split into tiles of `span` limbs, one CTA per tile:
//   1. the CTA computes its tile assuming carry-in 0, resolving carries
//      between its threads with ballots (block_resolve), and publishes
//      flags = G | P << 1 where G = carry out and P = the tile result is all
//      ones (all zeros for subtraction);
//   2. a fix-up kernel resolves the flags of each row and adds the incoming
//      carry to the tiles that receive one (usually one limb each).
// No CTA ever waits for another, so there is no spin loop to bound.
#pragma once

#include "common.cuh"

namespace gpupi {

struct BlockCarry {
    uint32_t cin;   // carry into this thread's chunk
    uint32_t G;     // carry out of the tile
    uint32_t P;     // tile propagates a carry
};

// g/p: this thread's chunk generates / propagates.  Threads are ordered by
// threadIdx.x (low limbs first), cin enters at thread 0 (the tile's carry-in;
// 0 where that is resolved later).  NWARPS <= 32.  Uses 2*NWARPS shared words.
template <int NWARPS>
__device__ __forceinline__ BlockCarry block_resolve(bool g, bool p, uint32_t *sh_g, uint32_t *sh_p,
                                                    uint32_t cin = 0u) {
    const uint32_t lane = lane_id();
    const uint32_t w = threadIdx.x >> 5;
    const uint32_t gm = __ballot_sync(0xffffffffu, g);
    const uint32_t pm = __ballot_sync(0xffffffffu, p);
    const GroupCarry wc = resolve_group(gm, pm, 0u);
    if (lane == 0) {
        sh_g[w] = wc.carry_out;
        sh_p[w] = (pm == 0xffffffffu) ? 1u : 0u;
    }
    __syncthreads();
    uint32_t wg = 0u, wp = 0u;
#pragma unroll
    for (int k = 0; k < NWARPS; ++k) {
        wg |= sh_g[k] << k;
        wp |= sh_p[k] << k;
    }
    const GroupCarry bc = resolve_group_n(wg, wp, cin, NWARPS);
    const uint32_t cin_w = (bc.carry_in_mask >> w) & 1u;
    const GroupCarry wc2 = resolve_group(gm, pm, cin_w);
    BlockCarry r;
    r.cin = (wc2.carry_in_mask >> lane) & 1u;
    r.G = bc.carry_out;
    r.P = (wp == ((NWARPS == 32) ? 0xffffffffu : ((1u << NWARPS) - 1u))) ? 1u : 0u;
    return r;
}

// Row `row` of a batch of results: C + row * sC with Lc limbs, or in a ragged
// batch (rows non-null) its descriptor's place and its own La + Lb limbs.
struct ResultRow {
    uint32_t *p;
    uint32_t L;
};
__device__ __forceinline__ ResultRow result_row(const RaggedRow *rows, uint32_t *C, uint64_t sC, uint32_t Lc,
                                                uint32_t row) {
    if (!rows) return {C + row * sC, Lc};
    return {C + rows[row].offC, rows[row].La + rows[row].Lb};
}

// Limbs [start, end) of tile t of a row of L limbs at `out`: tiles are `span`
// limbs, or, with `aligned`, span limbs counted from the row's last 16-byte
// boundary at or below its first limb (carry_ops.cu), so tile 0 is up to three
// limbs short.
struct TileRange {
    uint64_t start, end;
};
__device__ __forceinline__ TileRange tile_range(const uint32_t *out, uint32_t t, uint32_t span, uint32_t L,
                                                bool aligned) {
    const uint64_t mis = aligned ? (((uintptr_t)out >> 2) & 3u) : 0u;
    TileRange r;
    r.start = (uint64_t)t * span;
    r.start = r.start > mis ? r.start - mis : 0u;
    r.end = (uint64_t)(t + 1u) * span - mis;
    if (r.end > L) r.end = L;
    return r;
}

// Adds a carry (subtracts a borrow) at the tile's first limb; returns true
// when it runs past that limb.
template <bool SUB>
__device__ __forceinline__ bool patch_first(uint32_t *out, TileRange r) {
    if (r.start >= r.end) return false;
    const uint32_t v = out[r.start];
    out[r.start] = SUB ? v - 1u : v + 1u;
    return v == (SUB ? 0u : 0xffffffffu);
}

// The rest of a carry that ran past the first limb, by a whole warp: a tile
// that lets carries through becomes all zeros (all ones), any other is
// searched for its first absorbing limb 128 limbs at a time.
template <bool SUB>
__device__ __forceinline__ void patch_rest(uint32_t *out, TileRange r, bool all) {
    const uint32_t lane = lane_id();
    const uint32_t ones = SUB ? 0u : 0xffffffffu;
    for (uint64_t base = r.start + 1u; base < r.end; base += 128u) {
        uint32_t v[4];
        uint32_t stop[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint64_t j = base + 32u * k + lane;
            v[k] = (!all && j < r.end) ? out[j] : ones;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) stop[k] = __ballot_sync(0xffffffffu, v[k] != ones);
        bool open = true;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint64_t j = base + 32u * k + lane;
            const uint32_t upto = stop[k] ? (uint32_t)(__ffs(stop[k]) - 1) : 31u;
            if (open && lane <= upto && j < r.end) out[j] = SUB ? v[k] - 1u : v[k] + 1u;
            open = open && stop[k] == 0u;
        }
        if (!open) break;
    }
}

// rows non-null: a ragged batch; Lc and tiles_per_row are its longest row's.  A
// shorter row's tiles end with the row (what follows is another product's, or
// not the caller's); those wholly above it receive no carry.
// Cross-tile carry fix-up for rows of at most 32 tiles: one warp per row, one
// lane per tile.
template <bool SUB>
__global__ void carry_fixup_kernel(uint32_t *C, uint64_t sC, uint32_t N, uint32_t Lc, uint32_t tiles_per_row,
                                   uint32_t span, bool aligned, const uint32_t *flags, const RaggedRow *rows) {
    const uint32_t lane = lane_id();
    const uint32_t gwarp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t row = gwarp; row < N; row += nwarps) {
        const ResultRow out = result_row(rows, C, sC, Lc, row);
        const uint32_t f = (lane < tiles_per_row) ? flags[(uint64_t)row * tiles_per_row + lane] : 0u;
        const uint32_t gm = __ballot_sync(0xffffffffu, (f & 1u) != 0u);
        const uint32_t pm = __ballot_sync(0xffffffffu, (f & 2u) != 0u);
        const GroupCarry gc = resolve_group(gm, pm, 0u);
        bool more = false;
        if (lane < tiles_per_row && ((gc.carry_in_mask >> lane) & 1u))
            more = patch_first<SUB>(out.p, tile_range(out.p, lane, span, out.L, aligned));
        for (uint32_t left = __ballot_sync(0xffffffffu, more); left; left &= left - 1u) {
            const uint32_t t = (uint32_t)(__ffs(left) - 1);
            patch_rest<SUB>(out.p, tile_range(out.p, t, span, out.L, aligned), (pm >> t) & 1u);
        }
    }
}

// The same for longer rows: each CTA resolves 1024 tiles, four per thread.
// The carry into them comes from looking back over the flags 1024 tiles at a
// time until a group that generates or absorbs (a random group of tiles never
// lets a carry through, so nearly always one step; a row of all ones looks
// back over the whole row, 1024 tiles per step).  Every CTA works for itself
// and none waits for another; only C is written, never the flags.  A single
// CTA walking the row instead took 276 us on the 262,144 tiles of 1024 limbs of
// a 2^28-limb product and 40 us on 16,385 tiles of 4096 limbs; this takes 3.8
// and 7.1 us.
constexpr uint32_t kFixThreads = 256;
constexpr uint32_t kFixTiles = 4u * kFixThreads;

template <bool SUB>
__global__ void __launch_bounds__(kFixThreads) carry_fixup_rows_kernel(uint32_t *C, uint64_t sC, uint32_t Lc,
                                                                       uint32_t tiles_per_row, uint32_t blocks_per_row,
                                                                       uint32_t span, bool aligned,
                                                                       const uint32_t *flags,
                                                                       const RaggedRow *rows) {
    __shared__ uint32_t sg[kFixThreads / 32], sp[kFixThreads / 32];
    const uint32_t row = blockIdx.x / blocks_per_row;
    const uint32_t blk = blockIdx.x - row * blocks_per_row;
    const uint32_t *fr = flags + (uint64_t)row * tiles_per_row;
    const ResultRow out = result_row(rows, C, sC, Lc, row);
    // generate / propagate bits of this thread's four tiles of group b
    auto load = [&](uint32_t b, uint32_t &g, uint32_t &p) {
        g = p = 0u;
#pragma unroll
        for (uint32_t k = 0; k < 4u; ++k) {
            const uint64_t t = (uint64_t)b * kFixTiles + 4u * threadIdx.x + k;
            const uint32_t f = (t < tiles_per_row) ? fr[t] : 0u;
            g |= (f & 1u) << k;
            p |= ((f >> 1) & 1u) << k;
        }
    };
    uint32_t cin = 0u;
    for (uint32_t b = blk; b-- > 0u;) {
        uint32_t g, p;
        load(b, g, p);
        const GroupCarry c = resolve_group_n(g, p, 0u, 4);
        const BlockCarry bc = block_resolve<kFixThreads / 32>(c.carry_out != 0u, p == 15u, sg, sp);
        __syncthreads();   // sg / sp are rewritten by the next step
        if (bc.G || !bc.P) {
            cin = bc.G;
            break;
        }
    }
    uint32_t g, p;
    load(blk, g, p);
    const GroupCarry c = resolve_group_n(g, p, 0u, 4);
    const BlockCarry bc = block_resolve<kFixThreads / 32>(c.carry_out != 0u, p == 15u, sg, sp, cin);
    const uint32_t into = resolve_group_n(g, p, bc.cin, 4).carry_in_mask;
    const uint32_t t0 = blk * kFixTiles + 4u * threadIdx.x;
#pragma unroll
    for (uint32_t k = 0; k < 4u; ++k) {
        const uint32_t t = t0 + k;
        bool more = false;
        if (t < tiles_per_row && ((into >> k) & 1u))
            more = patch_first<SUB>(out.p, tile_range(out.p, t, span, out.L, aligned));
        for (uint32_t left = __ballot_sync(0xffffffffu, more); left; left &= left - 1u) {
            const int l = __ffs(left) - 1;
            const uint32_t tl = __shfl_sync(0xffffffffu, t, l);
            const uint32_t pl = __shfl_sync(0xffffffffu, (p >> k) & 1u, l);
            patch_rest<SUB>(out.p, tile_range(out.p, tl, span, out.L, aligned), pl != 0u);
        }
    }
}

inline void launch_carry_fixup(bool sub, uint32_t *C, uint64_t sC, uint32_t N, uint32_t Lc, uint32_t tiles_per_row,
                               uint32_t span, bool aligned, const uint32_t *flags, cudaStream_t st,
                               const RaggedRow *rows = nullptr) {
    if (tiles_per_row > 32u) {
        const uint32_t bpr = (tiles_per_row + kFixTiles - 1u) / kFixTiles;
        if (sub)
            carry_fixup_rows_kernel<true><<<N * bpr, kFixThreads, 0, st>>>(C, sC, Lc, tiles_per_row, bpr, span, aligned,
                                                                         flags, rows);
        else
            carry_fixup_rows_kernel<false><<<N * bpr, kFixThreads, 0, st>>>(C, sC, Lc, tiles_per_row, bpr, span,
                                                                          aligned, flags, rows);
    } else {
        const unsigned grid = grid_for(N, 4, kNumSMs * 8);
        if (sub)
            carry_fixup_kernel<true><<<grid, 128, 0, st>>>(C, sC, N, Lc, tiles_per_row, span, aligned, flags, rows);
        else
            carry_fixup_kernel<false><<<grid, 128, 0, st>>>(C, sC, N, Lc, tiles_per_row, span, aligned, flags, rows);
    }
    count_launch();
}

// Chunk arithmetic for kernels whose per-position values are up to 96 bits
// (convolution coefficients, schoolbook column sums).
//   S = sum_v c[v] * 2^(32v)   (V+3 limbs)
template <int V>
__device__ __forceinline__ void chunk_sum3(const uint32_t (&c)[V][3], uint32_t (&S)[V + 3]) {
    uint64_t carry = 0;
#pragma unroll
    for (int k = 0; k < V + 3; ++k) {
        uint64_t s = carry;
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const int d = k - v;
            if (d >= 0 && d <= 2) s += c[v][d];
        }
        S[k] = (uint32_t)s;
        carry = s >> 32;
    }
}

// X = S[0..V) + H (3 limbs spilled from the previous chunk); returns carry out.
template <int V>
__device__ __forceinline__ uint32_t chunk_add_spill(const uint32_t (&S)[V + 3], const uint32_t (&H)[3],
                                                    uint32_t (&X)[V]) {
    uint64_t t = 0;
#pragma unroll
    for (int k = 0; k < V; ++k) {
        t += (uint64_t)S[k] + (k < 3 ? H[k] : 0u);
        X[k] = (uint32_t)t;
        t >>= 32;
    }
    static_assert(V >= 3, "the 3-limb spill must fit in one chunk");
    return (uint32_t)t;
}

template <int V>
__device__ __forceinline__ void chunk_increment(uint32_t (&X)[V], uint32_t cin) {
    uint32_t c = cin;
#pragma unroll
    for (int k = 0; k < V; ++k) {
        const uint32_t s = X[k] + c;
        c = (s < X[k]) ? 1u : 0u;
        X[k] = s;
    }
}

}  // namespace gpupi
