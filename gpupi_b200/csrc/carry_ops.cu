// Carry-chain family: add, sub, add_small, sub_small, mul_small, shift_add,
// shift_sub (gpupi batch_add.cu, batch_sub.cu, batch_add_small.cu,
// batch_sub_small.cu, batch_mul_small.cu, batch_shift_add.cu,
// batch_shift_sub.cu).
//
// Every one of these is "out_j = x_j +/- y_j +/- carry" over j < L_c with a
// carry of at most one bit, once the operands are written as two limb
// streams:
//   add/sub         x = A_j,                         y = B_j
//   add/sub_small   x = A_j,                         y = (j == 0) ? b : 0
//   mul_small       x = lo(A_j * b),                 y = hi(A_{j-1} * b)
//   shift_add/sub   x = (A << s)_j (two limbs of A), y = B_j
// so one engine serves them all.  Limbs past an operand's length read as 0,
// which gives the reference's "computed over max+1 limbs, truncated or
// zero-extended to L_c" semantics directly.
//
// Every thread handles four consecutive limbs whose first output word lies on
// a 16-byte boundary of the row (a row's first chunk starts up to three limbs
// below limb 0, where both streams read as 0), so C is written in 128-bit
// stores; operands are read in 128-bit loads too, whatever their alignment
// (read4).  Launch shapes (no inter-CTA waiting):
//   * lanes per row    - rows of up to 125 limbs: 4, 8, 16 or 32 lanes per
//                        row, one ballot pair;
//   * warp per row     - longer rows up to 4096 limbs (or very many rows):
//                        256 or 512 limbs per step, the carry kept warp-
//                        uniform; rows that fill little of that, one limb per
//                        lane;
//   * tiles + fix-up   - long rows: each CTA owns a 4096-limb tile, writes its
//                        result assuming carry-in 0 plus (generate, propagate)
//                        flags; a second kernel scans the flags of each row and
//                        adds the carry to the tiles that receive one (usually
//                        one limb).
// Traffic is the algorithmic minimum (read operands once, write C once)
// except for the few fix-up limbs.
#include "common.cuh"
#include "carry_tile.cuh"

#include "batch_add.h"
#include "batch_add_small.h"
#include "batch_mul_small.h"
#include "batch_shift_add.h"
#include "batch_shift_sub.h"
#include "batch_sub.h"
#include "batch_sub_small.h"

namespace gpupi {

// ---------------------------------------------------------------------------
// Operand generators: read() gives limbs j .. j + 3 of the two streams (j may
// be as low as -3; limbs below 0 are 0), limb() limb j.
// ---------------------------------------------------------------------------

// mul_small reads the source limb below its own, which in place (C is A) may be
// a result already: at the first limb of a warp's step or of a tile it is taken
// from here, read before those results were written.
struct Edge {
    int64_t at = INT64_MIN;   // limb index
    uint32_t below = 0u;      // source limb at - 1
};

// How a chunk is read: limb by limb; in 128-bit loads where the chunk's words
// lie inside the row; or where those of the whole warp (its lanes' chunks in
// sequence) do.  Inside one warp lanes that take different paths wait for one
// another's loads, which rows of a few hundred limbs, mostly ends, pay for
// (65,536 sums of 200 limbs 67 -> 53 us with kByWarp); in the long rows' tiles the
// ends are few, and the common decision costs more than it saves (2^26 limbs,
// five operations: 574 us with kByLane, 587 with kByWarp).
enum Read { kByLimb, kByLane, kByWarp };

// out[v] = r[j + v], 0 outside [0, len).  Inside the row: one 128-bit load
// when r + j is 16-byte aligned; otherwise the two aligned words that hold the
// four limbs, where both lie inside the row (the second is the neighbouring
// thread's first and comes from L1); limb by limb at the row's ends.  The
// misalignment is the same for all chunks of a row.
template <Read MODE>
__device__ __forceinline__ void read4(const uint32_t *r, uint32_t len, int64_t j, uint32_t (&o)[4]) {
    const uint32_t *p = r + j;
    bool within = j >= 0 && j + 4 <= (int64_t)len;   // the four limbs
    if (MODE == kByWarp) {   // and the words that hold those of the warp
        const int64_t first = j - 4 * (int64_t)lane_id();
        within = first >= 3 && first + 132 <= (int64_t)len;
    }
    if (MODE != kByLimb && within) {
        const uint32_t m = ((uintptr_t)p >> 2) & 3u;
        if (m == 0u) {
            const uint4 q = *reinterpret_cast<const uint4 *>(p);
            o[0] = q.x;
            o[1] = q.y;
            o[2] = q.z;
            o[3] = q.w;
            return;
        }
        if (MODE == kByWarp || (j >= (int64_t)m && j - m + 8 <= (int64_t)len)) {
            const uint4 a = *reinterpret_cast<const uint4 *>(p - m);
            const uint4 b = *reinterpret_cast<const uint4 *>(p - m + 4);
            o[0] = m == 1u ? a.y : (m == 2u ? a.z : a.w);
            o[1] = m == 1u ? a.z : (m == 2u ? a.w : b.x);
            o[2] = m == 1u ? a.w : (m == 2u ? b.x : b.y);
            o[3] = m == 1u ? b.x : (m == 2u ? b.y : b.z);
            return;
        }
    }
#pragma unroll
    for (int v = 0; v < 4; ++v) o[v] = ((uint64_t)(j + v) < (uint64_t)len) ? p[v] : 0u;   // j + v < 0 wraps
}

struct GenTwo {
    static constexpr int kStreams = 2;   // operands read from memory
    static constexpr bool kBelow = false;   // reads the limb below its own in place
    const uint32_t *A;
    const uint32_t *B;
    uint32_t La, Lb;
    uint64_t sA, sB;
    template <Read MODE>
    __device__ __forceinline__ void read(uint32_t row, int64_t j, uint32_t (&x)[4], uint32_t (&y)[4], Edge) const {
        read4<MODE>(A + row * sA, La, j, x);
        read4<MODE>(B + row * sB, Lb, j, y);
    }
    __device__ __forceinline__ void limb(uint32_t row, uint32_t j, uint32_t &x, uint32_t &y, Edge) const {
        x = (j < La) ? A[row * sA + j] : 0u;
        y = (j < Lb) ? B[row * sB + j] : 0u;
    }
    double read_limbs(uint32_t Lc) const { return (double)std::min(La, Lc) + std::min(Lb, Lc); }
};

struct GenSmall {
    static constexpr int kStreams = 1;   // operands read from memory
    static constexpr bool kBelow = false;   // reads the limb below its own in place
    const uint32_t *A;
    uint32_t b;
    uint32_t La;
    uint64_t sA;
    template <Read MODE>
    __device__ __forceinline__ void read(uint32_t row, int64_t j, uint32_t (&x)[4], uint32_t (&y)[4], Edge) const {
        read4<MODE>(A + row * sA, La, j, x);
#pragma unroll
        for (int v = 0; v < 4; ++v) y[v] = (j + v == 0) ? b : 0u;
    }
    __device__ __forceinline__ void limb(uint32_t row, uint32_t j, uint32_t &x, uint32_t &y, Edge) const {
        x = (j < La) ? A[row * sA + j] : 0u;
        y = (j == 0u) ? b : 0u;
    }
    double read_limbs(uint32_t Lc) const { return (double)std::min(La, Lc); }
};

// IN_PLACE: C is A (instantiations of their own: the tests at every chunk cost the
// others 10 to 30 %).
template <bool IN_PLACE>
struct GenMulSmall {
    static constexpr int kStreams = 1;   // operands read from memory
    static constexpr bool kBelow = IN_PLACE;
    const uint32_t *A;
    uint32_t b;
    uint32_t La;
    uint64_t sA;
    const uint32_t *edges;   // tiles in place: the limb below each tile, else null
    __device__ __forceinline__ uint32_t below(uint32_t row, int64_t j) const {
        return ((uint64_t)(j - 1) < (uint64_t)La) ? A[row * sA + j - 1] : 0u;
    }
    template <Read MODE>
    __device__ __forceinline__ void read(uint32_t row, int64_t j, uint32_t (&x)[4], uint32_t (&y)[4], Edge e) const {
        const uint32_t *r = A + row * sA;
        uint32_t a[4];
        read4<MODE>(r, La, j, a);
        uint32_t prev = ((uint64_t)(j - 1) < (uint64_t)La) ? r[j - 1] : 0u;
        if (IN_PLACE && j == e.at) prev = e.below;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            x[v] = a[v] * b;
            y[v] = __umulhi(v ? a[v - 1] : prev, b);
        }
    }
    __device__ __forceinline__ void limb(uint32_t row, uint32_t j, uint32_t &x, uint32_t &y, Edge e) const {
        const uint32_t *r = A + row * sA;
        x = (j < La) ? r[j] * b : 0u;
        uint32_t prev = (j >= 1u && j - 1u < La) ? r[j - 1u] : 0u;
        if (IN_PLACE && (int64_t)j == e.at) prev = e.below;
        y = __umulhi(prev, b);
    }
    double read_limbs(uint32_t Lc) const { return (double)std::min(La, Lc); }
};

struct GenShiftTwo {
    static constexpr int kStreams = 2;   // operands read from memory
    static constexpr bool kBelow = false;   // reads the limb below its own in place
    const uint32_t *A;
    const uint32_t *B;
    uint32_t La, Lb;
    uint64_t sA, sB;
    uint32_t word, bit;
    template <Read MODE>
    __device__ __forceinline__ void read(uint32_t row, int64_t j, uint32_t (&x)[4], uint32_t (&y)[4], Edge) const {
        const uint32_t *r = A + row * sA;
        const int64_t i = j - (int64_t)word;
        uint32_t a[4];
        read4<MODE>(r, La, i, a);
        const uint32_t prev = ((uint64_t)(i - 1) < (uint64_t)La) ? r[i - 1] : 0u;
#pragma unroll
        for (int v = 0; v < 4; ++v) x[v] = __funnelshift_l(v ? a[v - 1] : prev, a[v], bit);   // bit < 32
        read4<MODE>(B + row * sB, Lb, j, y);
    }
    __device__ __forceinline__ void limb(uint32_t row, uint32_t j, uint32_t &x, uint32_t &y, Edge) const {
        const uint32_t *r = A + row * sA;
        const uint32_t i = j - word;
        const uint32_t lo = (j >= word && i < La) ? r[i] : 0u;
        const uint32_t prev = (j > word && i - 1u < La) ? r[i - 1u] : 0u;
        x = __funnelshift_l(prev, lo, bit);   // bit < 32
        y = (j < Lb) ? B[row * sB + j] : 0u;
    }
    double read_limbs(uint32_t Lc) const { return (double)std::min(La, Lc) + std::min(Lb, Lc); }
};

// ---------------------------------------------------------------------------
// Four-limb chunks
// ---------------------------------------------------------------------------
// s = x +/- y with carry-in 0; g: carry out, p: a carry in would run through.
template <bool SUB>
__device__ __forceinline__ void chunk_raw(const uint32_t (&x)[4], const uint32_t (&y)[4], uint32_t (&s)[4], bool &g,
                                          bool &p) {
    uint32_t c;
    if (SUB)
        asm("sub.cc.u32 %0, %5, %9;\n\tsubc.cc.u32 %1, %6, %10;\n\tsubc.cc.u32 %2, %7, %11;\n\t"
            "subc.cc.u32 %3, %8, %12;\n\tsubc.u32 %4, 0, 0;"
            : "=&r"(s[0]), "=&r"(s[1]), "=&r"(s[2]), "=&r"(s[3]), "=r"(c)
            : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(y[0]), "r"(y[1]), "r"(y[2]), "r"(y[3]));
    else
        asm("add.cc.u32 %0, %5, %9;\n\taddc.cc.u32 %1, %6, %10;\n\taddc.cc.u32 %2, %7, %11;\n\t"
            "addc.cc.u32 %3, %8, %12;\n\taddc.u32 %4, 0, 0;"
            : "=&r"(s[0]), "=&r"(s[1]), "=&r"(s[2]), "=&r"(s[3]), "=r"(c)
            : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(y[0]), "r"(y[1]), "r"(y[2]), "r"(y[3]));
    g = c != 0u;
    p = SUB ? (s[0] | s[1] | s[2] | s[3]) == 0u : (s[0] & s[1] & s[2] & s[3]) == 0xffffffffu;
}

template <bool SUB>
__device__ __forceinline__ void chunk_carry(uint32_t (&s)[4], uint32_t cin) {
    if (SUB)
        asm("sub.cc.u32 %0, %0, %4;\n\tsubc.cc.u32 %1, %1, 0;\n\tsubc.cc.u32 %2, %2, 0;\n\tsubc.u32 %3, %3, 0;"
            : "+r"(s[0]), "+r"(s[1]), "+r"(s[2]), "+r"(s[3])
            : "r"(cin));
    else
        asm("add.cc.u32 %0, %0, %4;\n\taddc.cc.u32 %1, %1, 0;\n\taddc.cc.u32 %2, %2, 0;\n\taddc.u32 %3, %3, 0;"
            : "+r"(s[0]), "+r"(s[1]), "+r"(s[2]), "+r"(s[3])
            : "r"(cin));
}

// Limbs j .. j + 3 of a row; out + j is 16-byte aligned.
__device__ __forceinline__ void chunk_write(uint32_t *out, uint32_t Lc, int64_t j, const uint32_t (&s)[4]) {
    if (j >= 0 && j + 4 <= (int64_t)Lc) {
        *reinterpret_cast<uint4 *>(out + j) = make_uint4(s[0], s[1], s[2], s[3]);
    } else {
#pragma unroll
        for (int v = 0; v < 4; ++v)
            if ((uint64_t)(j + v) < (uint64_t)Lc) out[j + v] = s[v];
    }
}

// Limbs from the last 16-byte boundary at or below a row to the row.
__device__ __forceinline__ int64_t row_offset(const uint32_t *out) { return (int64_t)(((uintptr_t)out >> 2) & 3u); }

// ---------------------------------------------------------------------------
// Kernels
// ---------------------------------------------------------------------------
// G lanes per row (L_c + 3 <= 4 G), 32 / G rows per warp, ROWS such sets per
// step so that each lane has the loads of several rows in flight.  Rows this
// short are read limb by limb (from L1 after the first of a chunk's loads):
// most chunks of a row that is not 16-byte aligned touch one of its ends, and
// a warp that takes both of read4's paths is slower than the plain loads.
template <class Gen, bool SUB, int G, int ROWS>
__global__ void __launch_bounds__(256) carry_lane_rows(Gen gen, uint32_t *C, uint64_t sC, uint32_t N, uint32_t Lc) {
    constexpr uint32_t kMask = (G == 32) ? 0xffffffffu : ((1u << G) - 1u);
    constexpr int PW = 32 / G;
    const uint32_t lane = lane_id();
    const uint32_t grp = lane / G, gl = lane % G;
    const uint32_t warps_per_cta = blockDim.x >> 5;
    const uint64_t gwarp = (uint64_t)blockIdx.x * warps_per_cta + (threadIdx.x >> 5);
    const uint64_t nwarps = (uint64_t)gridDim.x * warps_per_cta;
    // the whole warp runs every iteration (ballots); rows past N do nothing
    for (uint64_t base = gwarp * (PW * ROWS); base < N; base += nwarps * (PW * ROWS)) {
        uint32_t s[ROWS][4];
        bool g[ROWS], p[ROWS];
#pragma unroll
        for (int u = 0; u < ROWS; ++u) {
            const uint64_t row = base + u * PW + grp;
            g[u] = p[u] = false;
            if (row < N) {
                uint32_t x[4], y[4];
                gen.template read<kByLimb>((uint32_t)row, 4 * (int64_t)gl - row_offset(C + row * sC), x, y, Edge{});
                chunk_raw<SUB>(x, y, s[u], g[u], p[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < ROWS; ++u) {
            const uint64_t row = base + u * PW + grp;
            const uint32_t gm = (__ballot_sync(0xffffffffu, g[u]) >> (grp * G)) & kMask;
            const uint32_t pm = (__ballot_sync(0xffffffffu, p[u]) >> (grp * G)) & kMask;
            const GroupCarry gc = resolve_group_n(gm, pm, 0u, G);
            if (row < N) {
                uint32_t *out = C + row * sC;
                chunk_carry<SUB>(s[u], (gc.carry_in_mask >> gl) & 1u);
                chunk_write(out, Lc, 4 * (int64_t)gl - row_offset(out), s[u]);
            }
        }
    }
}

// The limb below a warp's next step, before this step's results are written.
template <class Gen>
__device__ __forceinline__ void next_edge(const Gen &gen, uint32_t row, int64_t next, Edge &e) {
    if constexpr (Gen::kBelow) {
        e.at = next;
        e.below = gen.below(row, next);
        __syncwarp();
    }
}

// A warp per row, one limb per lane, four 32-limb groups per step: for rows
// whose last 128-limb group of carry_warp_rows would be mostly empty and whose
// chunks are mostly at an end of the row (see run_carry).
template <class Gen, bool SUB>
__global__ void __launch_bounds__(256) carry_limb_rows(Gen gen, uint32_t *C, uint64_t sC, uint32_t N, uint32_t Lc) {
    constexpr int kGroups = 4;
    const uint32_t lane = lane_id();
    const uint32_t warps_per_cta = blockDim.x >> 5;
    const uint32_t gwarp = blockIdx.x * warps_per_cta + (threadIdx.x >> 5);
    const uint32_t nwarps = gridDim.x * warps_per_cta;
    for (uint32_t row = gwarp; row < N; row += nwarps) {
        uint32_t *out = C + row * sC;
        uint32_t cin = 0u;
        Edge edge;
        for (uint32_t base = 0; base < Lc; base += 32u * kGroups) {
            uint32_t s[kGroups], gm[kGroups], pm[kGroups];
#pragma unroll
            for (int u = 0; u < kGroups; ++u) {
                const uint32_t j = base + u * 32u + lane;
                uint32_t x = 0u, y = 0u;
                if (j < Lc) gen.limb(row, j, x, y, edge);
                s[u] = SUB ? x - y : x + y;
                gm[u] = __ballot_sync(0xffffffffu, SUB ? x < y : s[u] < x);
                pm[u] = __ballot_sync(0xffffffffu, s[u] == (SUB ? 0u : 0xffffffffu));
            }
            next_edge(gen, row, (int64_t)base + 32 * kGroups, edge);
#pragma unroll
            for (int u = 0; u < kGroups; ++u) {
                const uint32_t j = base + u * 32u + lane;
                const GroupCarry gc = resolve_group(gm[u], pm[u], cin);
                cin = gc.carry_out;
                const uint32_t c = (gc.carry_in_mask >> lane) & 1u;
                if (j < Lc) out[j] = SUB ? s[u] - c : s[u] + c;
            }
        }
    }
}

// A warp per row, UNROLL groups of 128 limbs per step.  Two for batches: the
// registers of four (64 a thread) leave 32 warps per SM, which cost rows of 500
// to 1000 limbs a second wave (20,000 sums of 600 limbs 45 us with four, 37 with
// two; 65,536 of 1600 limbs 306 and 284).  Four, each lane reading by its own
// path, for long rows that run alone (one of 4000 limbs 18.5 us with four, 20.5
// with two; one of 1600 limbs times a limb 6.2 us by lane, 8.2 by warp).
template <class Gen, bool SUB, int UNROLL, Read MODE>
__global__ void __launch_bounds__(256) carry_warp_rows(Gen gen, uint32_t *C, uint64_t sC, uint32_t N, uint32_t Lc) {
    const uint32_t lane = lane_id();
    const uint32_t warps_per_cta = blockDim.x >> 5;
    const uint32_t gwarp = blockIdx.x * warps_per_cta + (threadIdx.x >> 5);
    const uint32_t nwarps = gridDim.x * warps_per_cta;
    for (uint32_t row = gwarp; row < N; row += nwarps) {
        uint32_t cin = 0u;
        Edge edge;
        uint32_t *out = C + row * sC;
        for (int64_t base = -row_offset(out); base < (int64_t)Lc; base += 128 * UNROLL) {
            uint32_t s[UNROLL][4], gm[UNROLL], pm[UNROLL];
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) {
                uint32_t x[4], y[4];
                bool g, p;
                gen.template read<MODE>(row, base + u * 128 + 4 * lane, x, y, edge);
                chunk_raw<SUB>(x, y, s[u], g, p);
                gm[u] = __ballot_sync(0xffffffffu, g);
                pm[u] = __ballot_sync(0xffffffffu, p);
            }
            next_edge(gen, row, base + 128 * UNROLL, edge);
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) {
                const GroupCarry gc = resolve_group(gm[u], pm[u], cin);
                cin = gc.carry_out;
                chunk_carry<SUB>(s[u], (gc.carry_in_mask >> lane) & 1u);
                chunk_write(out, Lc, base + u * 128 + 4 * lane, s[u]);
            }
        }
    }
}

constexpr int kTileWarps = 8;
constexpr int kTileSub = 4;                                   // 128-limb groups per warp
constexpr uint32_t kTileSpan = 128u * kTileWarps * kTileSub;   // 4096 limbs
static_assert(kTileWarps * kTileSub == 32, "one lane per 128-limb group of the tile");

// A row's tiles start at its last 16-byte boundary at or below limb 0.
static uint32_t carry_tile_count(uint32_t Lc) { return (uint32_t)(((uint64_t)Lc + 3u + kTileSpan - 1u) / kTileSpan); }

// One 4096-limb tile per CTA: group (u, w) = 128 limbs, u-th of warp w.  The
// 32 groups' carries are resolved by one warp-wide ballot.  Flags: bit 0 =
// generates a carry with carry-in 0, bit 1 = lets a carry through.
// Bound by HBM: shift_add of two 2^26-limb rows 489 -> 162 us (805 MB,
// 5.0 TB/s), sub 443 -> 151 us, mul_small 428 -> 96 us (537 MB, 5.6 TB/s)
// against one limb per lane and ballot, whose 16 ballot pairs and resolutions
// per 512 limbs kept the loads apart.
template <class Gen, bool SUB>
__global__ void __launch_bounds__(kTileWarps * 32)
carry_tiles(Gen gen, uint32_t *C, uint64_t sC, uint32_t Lc, uint32_t tiles_per_row, uint32_t *flags) {
    __shared__ uint32_t group_g[32], group_p[32];
    const uint32_t lane = lane_id();
    const uint32_t w = threadIdx.x >> 5;
    const uint32_t tile = blockIdx.x;
    const uint32_t row = tile / tiles_per_row;
    const uint32_t t = tile - row * tiles_per_row;
    uint32_t *out = C + row * sC;
    const int64_t base = (int64_t)t * kTileSpan - row_offset(out) + w * 128 + 4 * lane;
    uint32_t s[kTileSub][4], gm[kTileSub], pm[kTileSub];
    Edge edge;
    if constexpr (Gen::kBelow)
        if (gen.edges) edge = Edge{(int64_t)t * kTileSpan - row_offset(out), gen.edges[tile]};
#pragma unroll
    for (int u = 0; u < kTileSub; ++u) {
        uint32_t x[4], y[4];
        bool g, p;
        gen.template read<kByLane>(row, base + u * (128 * kTileWarps), x, y, edge);
        chunk_raw<SUB>(x, y, s[u], g, p);
        gm[u] = __ballot_sync(0xffffffffu, g);
        pm[u] = __ballot_sync(0xffffffffu, p);
        if (lane == 0) {
            group_g[u * kTileWarps + w] = resolve_group(gm[u], pm[u], 0u).carry_out;
            group_p[u * kTileWarps + w] = (pm[u] == 0xffffffffu) ? 1u : 0u;
        }
    }
    __syncthreads();
    const uint32_t tg = __ballot_sync(0xffffffffu, group_g[lane] != 0u);
    const uint32_t tp = __ballot_sync(0xffffffffu, group_p[lane] != 0u);
    const GroupCarry tc = resolve_group(tg, tp, 0u);
#pragma unroll
    for (int u = 0; u < kTileSub; ++u) {
        const uint32_t cin = (tc.carry_in_mask >> (u * kTileWarps + w)) & 1u;
        const GroupCarry gc = resolve_group(gm[u], pm[u], cin);
        chunk_carry<SUB>(s[u], (gc.carry_in_mask >> lane) & 1u);
        chunk_write(out, Lc, base + u * (128 * kTileWarps), s[u]);
    }
    // P: the tile's result is all ones (all zeros), which with carry-in 0 means
    // that every limb's raw sum is
    if (threadIdx.x == 0) flags[tile] = tc.carry_out | ((tp == 0xffffffffu) ? 2u : 0u);
}

// In-place mul_small of rows in tiles: each tile's limb below, before any
// tile's results are written.
__global__ void __launch_bounds__(256) tile_edges(GenMulSmall<true> gen, const uint32_t *C, uint64_t sC, uint64_t total,
                                                  uint32_t tiles_per_row, uint32_t *edges) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const uint32_t row = (uint32_t)(i / tiles_per_row);
    const int64_t t = (int64_t)(i - (uint64_t)row * tiles_per_row);
    edges[i] = gen.below(row, t * kTileSpan - row_offset(C + row * sC));
}

// ---------------------------------------------------------------------------
// Dispatch
// ---------------------------------------------------------------------------
enum class CarryPlan { Lanes, Warp, Tiles };

static CarryPlan plan_for(uint32_t N, uint32_t Lc) {
    if (Lc <= 125u) return CarryPlan::Lanes;   // with the 3 limbs below a row: 4 limbs x 32 lanes
    if (Lc <= kTileSpan || (uint64_t)N >= (uint64_t)kNumSMs * 64u) return CarryPlan::Warp;
    return CarryPlan::Tiles;
}

static size_t carry_workspace_bytes(uint32_t N, uint32_t Lc) {
    if (N == 0u || Lc == 0u || plan_for(N, Lc) != CarryPlan::Tiles) return 0;
    return (size_t)N * carry_tile_count(Lc) * sizeof(uint32_t);
}

template <class Gen, bool SUB, int G, int ROWS>
static void launch_lanes(const Gen &gen, uint32_t *C, uint32_t N, uint32_t Lc, uint32_t sC, cudaStream_t st) {
    carry_lane_rows<Gen, SUB, G, ROWS>
        <<<grid_for(N, 8 * (32 / G) * ROWS, kNumSMs * 32), 256, 0, st>>>(gen, C, sC, N, Lc);
}

template <class Gen, bool SUB>
static void run_carry(const Gen &gen, uint32_t *C, uint32_t N, uint32_t Lc, uint32_t sC,
                      uint32_t *workspace) {
    if (N == 0u || Lc == 0u) return;
    cudaStream_t st = current_stream();
    const CarryPlan plan = plan_for(N, Lc);
    KernelTimed kt("carry_chain", 4.0 * N * (gen.read_limbs(Lc) + (double)Lc));
    if (plan == CarryPlan::Lanes) {
        if (Lc <= 13u)
            launch_lanes<Gen, SUB, 4, 2>(gen, C, N, Lc, sC, st);
        else if (Lc <= 29u)
            launch_lanes<Gen, SUB, 8, 2>(gen, C, N, Lc, sC, st);
        else if (Lc <= 61u)
            launch_lanes<Gen, SUB, 16, 2>(gen, C, N, Lc, sC, st);
        else
            launch_lanes<Gen, SUB, 32, 2>(gen, C, N, Lc, sC, st);
        GPUPI_LAUNCH_CHECK();
    } else if (plan == CarryPlan::Warp) {
        const unsigned warps = 8, grid = grid_for(N, warps);
        // Measured, one limb per lane against four (us, 65,536 rows): sums of 126
        // limbs 20 / 29, 160 35 / 37, 200 42 / 40, 253 49 / 43, 300 60 / 64, 350
        // 67 / 68, 400 78 / 75; one operand times a limb 126 16 / 23, 160 27 / 23.
        const bool limbs = Gen::kStreams == 2 ? Lc <= 192u || (Lc > 253u && Lc <= 381u && N >= 4096u) : Lc <= 144u;
        if (limbs)
            carry_limb_rows<Gen, SUB><<<grid, warps * 32, 0, st>>>(gen, C, sC, N, Lc);
        else if (N <= (uint32_t)kNumSMs && Lc > 509u)   // with the 3 limbs below a row: more than one step
            carry_warp_rows<Gen, SUB, 4, kByLane><<<grid, warps * 32, 0, st>>>(gen, C, sC, N, Lc);
        else
            carry_warp_rows<Gen, SUB, 2, kByWarp><<<grid, warps * 32, 0, st>>>(gen, C, sC, N, Lc);
        GPUPI_LAUNCH_CHECK();
    } else {
        const uint32_t tiles = carry_tile_count(Lc);
        const uint64_t total = (uint64_t)tiles * N;
        carry_tiles<Gen, SUB><<<(unsigned)total, kTileWarps * 32, 0, st>>>(gen, C, sC, Lc, tiles,
                                                                         workspace);
        GPUPI_LAUNCH_CHECK();
        launch_carry_fixup(SUB, C, sC, N, Lc, tiles, kTileSpan, true, workspace, st);
    }
}

}  // namespace gpupi

using namespace gpupi;

// ---------------------------------------------------------------------------
// Reference-compatible entry points
// ---------------------------------------------------------------------------
void batch_add_simple(uint32_t *A, uint32_t *B, uint32_t *C, uint32_t *workspace, uint32_t N,
                      uint32_t L_a, uint32_t L_b, uint32_t L_c, uint32_t stride_A,
                      uint32_t stride_B, uint32_t stride_C) {
    GenTwo g{A, B, L_a, L_b, stride_A, stride_B};
    run_carry<GenTwo, false>(g, C, N, L_c, stride_C, workspace);
}

size_t batch_add_simple_workspace_size(uint32_t N, uint32_t L_a, uint32_t L_b, uint32_t L_c) {
    (void)L_a;
    (void)L_b;
    return carry_workspace_bytes(N, L_c);
}

void batch_sub_simple(uint32_t *A, uint32_t *B, uint32_t *C, uint32_t *workspace, uint32_t N,
                      uint32_t L_a, uint32_t L_b, uint32_t L_c, uint32_t stride_A,
                      uint32_t stride_B, uint32_t stride_C) {
    GenTwo g{A, B, L_a, L_b, stride_A, stride_B};
    run_carry<GenTwo, true>(g, C, N, L_c, stride_C, workspace);
}

size_t batch_sub_simple_workspace_size(uint32_t N, uint32_t L_a, uint32_t L_b, uint32_t L_c) {
    (void)L_a;
    (void)L_b;
    return carry_workspace_bytes(N, L_c);
}

void batch_add_small(const uint32_t *A, uint32_t B, uint32_t *C, uint32_t *workspace, uint32_t N,
                     uint32_t L_a, uint32_t L_c, uint32_t stride_A, uint32_t stride_C) {
    GenSmall g{A, B, L_a, stride_A};
    run_carry<GenSmall, false>(g, C, N, L_c, stride_C, workspace);
}

size_t batch_add_small_workspace_size(uint32_t N, uint32_t L_a, uint32_t L_c) {
    (void)L_a;
    return carry_workspace_bytes(N, L_c);
}

void batch_sub_small(const uint32_t *A, uint32_t B, uint32_t *C, uint32_t *workspace, uint32_t N,
                     uint32_t L_a, uint32_t L_c, uint32_t stride_A, uint32_t stride_C) {
    GenSmall g{A, B, L_a, stride_A};
    run_carry<GenSmall, true>(g, C, N, L_c, stride_C, workspace);
}

size_t batch_sub_small_workspace_size(uint32_t N, uint32_t L_a, uint32_t L_c) {
    (void)L_a;
    return carry_workspace_bytes(N, L_c);
}

void batch_mul_small(const uint32_t *A, uint32_t B, uint32_t *C, uint32_t *workspace, uint32_t N,
                     uint32_t L_a, uint32_t L_c, uint32_t stride_A, uint32_t stride_C) {
    if (A != C) {
        run_carry<GenMulSmall<false>, false>({A, B, L_a, stride_A, nullptr}, C, N, L_c, stride_C, workspace);
        return;
    }
    GenMulSmall<true> g{A, B, L_a, stride_A, nullptr};
    if (N && L_c && plan_for(N, L_c) == CarryPlan::Tiles) {
        const uint32_t tiles = carry_tile_count(L_c);
        const uint64_t total = (uint64_t)N * tiles;
        uint32_t *edges = workspace + total;   // behind the flags
        tile_edges<<<(unsigned)((total + 255u) / 256u), 256, 0, current_stream()>>>(g, C, stride_C, total, tiles,
                                                                                    edges);
        GPUPI_LAUNCH_CHECK();
        g.edges = edges;
    }
    run_carry<GenMulSmall<true>, false>(g, C, N, L_c, stride_C, workspace);
}

size_t batch_mul_small_workspace_size(uint32_t N, uint32_t L_a, uint32_t L_c) {
    (void)L_a;
    return 2u * carry_workspace_bytes(N, L_c);   // flags, and in place the tiles' edges
}

void batch_shift_add_simple(const uint32_t *A, const uint32_t *B, uint32_t *C, uint32_t *workspace,
                            uint32_t shift, uint32_t N, uint32_t L_a, uint32_t L_b, uint32_t L_c,
                            uint32_t stride_A, uint32_t stride_B, uint32_t stride_C) {
    GenShiftTwo g{A, B, L_a, L_b, stride_A, stride_B, shift >> 5, shift & 31u};
    run_carry<GenShiftTwo, false>(g, C, N, L_c, stride_C, workspace);
}

size_t batch_shift_add_simple_workspace_size(uint32_t N, uint32_t L_a, uint32_t L_b, uint32_t L_c,
                                             uint32_t shift) {
    (void)L_a;
    (void)L_b;
    (void)shift;
    return carry_workspace_bytes(N, L_c);
}

void batch_shift_sub_simple(const uint32_t *A, const uint32_t *B, uint32_t *C, uint32_t *workspace,
                            uint32_t shift, uint32_t N, uint32_t L_a, uint32_t L_b, uint32_t L_c,
                            uint32_t stride_A, uint32_t stride_B, uint32_t stride_C) {
    GenShiftTwo g{A, B, L_a, L_b, stride_A, stride_B, shift >> 5, shift & 31u};
    run_carry<GenShiftTwo, true>(g, C, N, L_c, stride_C, workspace);
}

size_t batch_shift_sub_simple_workspace_size(uint32_t N, uint32_t L_a, uint32_t L_b, uint32_t L_c,
                                             uint32_t shift) {
    (void)L_a;
    (void)L_b;
    (void)shift;
    return carry_workspace_bytes(N, L_c);
}

// ---------------------------------------------------------------------------
// Allocation-free batched addition (gpupi_mp_add_noalloc in gpupi_c.h).
//
// Some callers cannot allocate device memory at the moment they need an add:
// code that runs with all device memory already handed to another allocator
// (a pre-sized pool it must not grow), and latency-critical loops that must
// not call cudaMalloc/cudaFree because those calls can synchronise the whole
// device.  For them the per-tile carry flags of long rows live in the fixed
// array below, compiled into the library, instead of a context workspace.
//
// Limit: kNoAllocMaxTiles flag words (256 KiB), i.e. N * ceil(L_c / 4096) tiles
// for rows on the multi-tile path; larger requests are rejected.
// The array is shared by every call and keeps the previous call's flags; no
// word has to start at zero because each tile's CTA writes its flag before
// the fix-up kernel reads it.  Calls whose kernels overlap on the GPU (two
// streams, two host threads) would race on the array.
// ---------------------------------------------------------------------------
#include "gpupi_c.h"

#include <mutex>

namespace gpupi {

constexpr uint64_t kNoAllocMaxTiles = 65536;
// rows on the multi-tile path (fewer than 64 per SM) have one tile more than
// ceil(L_c / 4096) when their last tile has fewer than three limbs to spare
static __device__ __align__(256) uint32_t g_noalloc_flags[kNoAllocMaxTiles + (uint64_t)kNumSMs * 64u];

// Device address of g_noalloc_flags, looked up once per device (with that
// device current) on the first call that needs it.
static uint32_t *g_noalloc_addr[64];
static std::mutex g_noalloc_mu;

static cudaError_t noalloc_flags_address(uint32_t **out) {
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> g(g_noalloc_mu);
    if (g_noalloc_addr[dev] == nullptr) {
        void *p = nullptr;
        err = cudaGetSymbolAddress(&p, g_noalloc_flags);
        if (err != cudaSuccess) return err;
        g_noalloc_addr[dev] = static_cast<uint32_t *>(p);
    }
    *out = g_noalloc_addr[dev];
    return cudaSuccess;
}

static bool noalloc_view_ok(const uint32_t *d, uint32_t len, uint32_t n, uint32_t stride) {
    if (n == 0u) return len <= stride;
    if (d == nullptr) return false;
    return stride == 0u || len <= stride;
}

}  // namespace gpupi

extern "C" int gpupi_mp_add_noalloc(uint32_t N, const uint32_t *d_A, uint32_t L_a, uint32_t stride_A,
                                    const uint32_t *d_B, uint32_t L_b, uint32_t stride_B, uint32_t *d_C,
                                    uint32_t L_c, uint32_t stride_C) {
    using namespace gpupi;
    if (!noalloc_view_ok(d_A, L_a, N, stride_A) || !noalloc_view_ok(d_B, L_b, N, stride_B) ||
        !noalloc_view_ok(d_C, L_c, N, stride_C))
        return (int)cudaErrorInvalidValue;
    if (N == 0u || L_c == 0u) return 0;
    uint32_t *flags = nullptr;
    if (plan_for(N, L_c) == CarryPlan::Tiles) {
        const uint64_t tiles = N * (((uint64_t)L_c + kTileSpan - 1u) / kTileSpan);
        if (tiles > kNoAllocMaxTiles) return (int)cudaErrorInvalidValue;   // beyond the fixed array
        const cudaError_t err = noalloc_flags_address(&flags);
        if (err != cudaSuccess) return (int)err;
    }
    GenTwo g{d_A, d_B, L_a, L_b, stride_A, stride_B};
    run_carry<GenTwo, false>(g, d_C, N, L_c, stride_C, flags);
    return (int)cudaGetLastError();
}
