// Batched exact multiplication by three-prime NTT (gpupi batch_mul_ntt.cu;
// API batch_mul_ntt.h:24-40).
//
// Shape.  A product of L_c = L_a + L_b limbs is a cyclic convolution of
// M * K points, K = 2^k <= 2^25, M <= 20, M * K >= L_a + L_b - 1.  M = 1 for
// products up to 2^25 points.  Longer products are split into M cosets:
// with c_i = g^(iK) (g a generator, i < M) the residues
// C_i = A B mod (x^K - c_i) are K-point cyclic convolutions of the twisted
// inputs (A mod (x^K - c_i))(g^i x), and the M blocks of K coefficients of
// C = A B follow from C_i = sum_b C_b c_i^b by the inverse Vandermonde
// matrix of the nodes c_i.
// Where M has two bits set and its larger part fits one transform (M = 3, 5,
// 6, ... with K 2^floor(log2 M) <= 2^25), the M K points are split instead into
// a transform of K1 = K 2^floor(log2 M) points mod x^K1 - 1 and one of the
// remaining K2 points mod x^K2 - g^K2 (twisted by g^i): with C = C1 +
// (x^K1 - 1) T, deg T < K2, T = (C2 - C1) / (g^K1 - 1) mod x^K2 - g^K2.
//
// Workspace: F[vrow][q][K] residues (vrow = row * M + coset), one such array
// for A (FA) and one for B (FB; none when B is A, one row when B is
// broadcast), then the CRT tile flags.
//
// Passes (four-step decomposition K = R1 [* R2] * C, C = 4096):
//   k_fold            operands of cosets, and longer than K: fold and twist
//   k_cols_r<first>   load limbs (residues after k_fold), R1-point DIF down
//                     each column of a 4096-residue tile, twist by
//                     w_K^(col * bitrev(pos)), store
//   k_cols_r          same on each segment for R2 (sizes above 2^22)
//   k_rows            C-point DIF of the A and B segments, pointwise product,
//                     C-point inverse DIT, store (products / R)
//   k_cols_r<inv>     untwist + inverse DIT on columns, mirror order; the first
//                     multiplies by K^-1 R too
//   k_combine<M>      (M > 1) untwist the cosets, inverse Vandermonde
//   k_combine2        (two parts) T and C's lower coefficients
//   k_crt             Garner CRT to 96-bit coefficients, carry into limbs
//                     (+ carry_fixup_kernel when a row spans several tiles)
// Small products (K <= 4096) are one k_rows<limbs> (4096 points), k_rows_r or
// k_rows_small launch and k_crt.  Code is compiled per prime (immediate
// operands) and the prime is the slowest index, so an SM works on one prime's
// tables and code at a time: a CTA of most kernels handles one prime, one of
// the persistent row kernels a run of segments in that order.
#include "ntt_core.cuh"
#include "carry_tile.cuh"
#include "batch_mul_ntt.h"
#include "spectrum.h"

#include <stdio.h>
#include <stdlib.h>

#include <mutex>
#include <vector>

namespace gpupi {
namespace ntt {

static const uint32_t kP[kPrimes] = {Prime<0>::p, Prime<1>::p, Prime<2>::p};
static const uint32_t kGen[kPrimes] = {Prime<0>::g, Prime<1>::g, Prime<2>::g};

struct NttParams {
    Tables tab;
};

// Row `row` of an operand: X + row * sX with Lx limbs, or in a ragged batch
// the A (side 0) or B (side 1) of its descriptor.
struct LimbRow {
    const uint32_t *p;
    uint32_t L;
};
__device__ __forceinline__ LimbRow limb_row(const RaggedRow *rows, int side, const uint32_t *X, uint64_t sX,
                                            uint32_t Lx, uint64_t row) {
    if (!rows) return {X + row * sX, Lx};
    const RaggedRow &d = rows[row];
    return side ? LimbRow{X + d.offB, d.Lb} : LimbRow{X + d.offA, d.La};
}

// ---------------------------------------------------------------------------
// Host modular helpers (table construction, coset matrices)
// ---------------------------------------------------------------------------
static uint32_t h_mul(uint32_t a, uint32_t b, uint32_t p) { return (uint32_t)((uint64_t)a * b % p); }
static uint32_t h_pow(uint32_t a, uint64_t e, uint32_t p) {
    uint32_t r = 1u % p;
    a %= p;
    while (e) {
        if (e & 1u) r = h_mul(r, a, p);
        a = h_mul(a, a, p);
        e >>= 1;
    }
    return r;
}
static uint32_t h_inv(uint32_t a, uint32_t p) { return h_pow(a, p - 2u, p); }
static uint32_t h_mont(uint32_t x, uint32_t p) { return (uint32_t)(((uint64_t)x << 32) % p); }

static NttParams make_params(const NTTPrecomputedTables &t) {
    NttParams P{};
    const uint32_t *lv1 = reinterpret_cast<const uint32_t *>(t.roots_table_lv1);
    const uint32_t *lv2 = reinterpret_cast<const uint32_t *>(t.roots_table_lv2);
    P.tab.root_lo = reinterpret_cast<const uint2 *>(lv1);
    P.tab.root_hi = reinterpret_cast<const uint2 *>(lv1 + kRootLoWords);
    P.tab.level = reinterpret_cast<const uint2 *>(lv1 + kLevelOffset);
    P.tab.coset_lo = lv2;
    P.tab.coset_hi = lv2 + kCosetWords;
    P.tab.inv2n = reinterpret_cast<const uint32_t *>(t.inv2n_table);
    return P;
}

// ---------------------------------------------------------------------------
// Kernels
// ---------------------------------------------------------------------------
constexpr int kThreads = 256;
constexpr int kTile = 4096;                    // residues per register-stage CTA tile
constexpr int kTilePad = kTile + kTile / 32;   // padded shared-memory words

// Grid index -> (prime, index within that prime's third of the grid).
__device__ __forceinline__ int grid_prime(uint64_t &b) {
    const uint32_t per = gridDim.x / kPrimes;
    const int q = (int)(blockIdx.x / per);
    b = blockIdx.x - (uint32_t)q * per;
    return q;
}

struct ColsArgs {
    const uint32_t *X;   // limbs (first pass of operands that need no folding only)
    uint64_t sX;
    uint32_t Lx;
    uint32_t *F;         // workspace of this operand: F[vrow][q][K]
    int log_k, log_s;
    int scaled;          // inverse pass: times K^-1 R as well (the row pass leaves products x y R^-1)
    // second operand of a paired pass (same shape, same tile)
    const uint32_t *X2;
    uint64_t sX2;
    uint32_t Lx2;
    uint32_t *F2;
    const RaggedRow *rows;   // first pass of a ragged batch: per-row operands
    int side;                // of X; X2 is side 1
};

// Offset of element j from element 0 in a LO = 0 stage with 2^B-point groups
// (LOG_R >= 4): j = g 2^B + v sits at pos_0 + v + g 2^(LOG_R - 4 + B), bits
// disjoint from those of pos_0.
__host__ __device__ constexpr uint32_t stage_delta(int j, int B, int log_r) {
    return ((uint32_t)j & ((1u << B) - 1u)) + (((uint32_t)j >> B) << (log_r - 4 + B));
}

// Distance of residue j of a thread from its residue 0 in stage S, in limbs of
// a tile row pitch of 2^log_cols: positions and columns of j occupy bits that
// those of residue 0 leave free, so it is the same for every thread.
template <class S, int LOG_R>
__device__ __forceinline__ uint32_t elem_delta(int j, int log_cols) {
    constexpr int B = S::kB;
    const uint32_t v = (uint32_t)j & ((1u << B) - 1u), g = (uint32_t)j >> B;
    if constexpr (LOG_R >= 4)
        return ((v << S::kLO) + (g << (LOG_R - 4 + B))) << log_cols;
    else   // whole columns, 256 apart
        return (v << log_cols) + 256u * g;
}

// Word i of an array by a 32-bit byte offset from a base that is the same for
// the whole CTA: the offsets of a thread's residues differ by uniform amounts
// (elem_delta), one 32-bit add each, where 64-bit indexing cost a wide
// multiply-add (four cycles of the pipe that bounds these passes) per access.
// i < 2^30: an operand has at most 20 * 2^25 limbs, a transform 2^25 points.
__device__ __forceinline__ const uint32_t *word_at(const uint32_t *base, uint32_t i) {
    return reinterpret_cast<const uint32_t *>(reinterpret_cast<const char *>(base) + (uint64_t)(i * 4u));
}
__device__ __forceinline__ uint32_t *word_at(uint32_t *base, uint32_t i) {
    return reinterpret_cast<uint32_t *>(reinterpret_cast<char *>(base) + (uint64_t)(i * 4u));
}

// Twist the 16 residues of stage S (the LO = 0 stage: last forward, first
// inverse) by one * w_S^(col * bitrev(pos)) / R or with the inverse root (one =
// R for the plain twist, K^-1 R^2 where the product's scale is folded in),
// E = colsh * bitrev(pos) with colsh = col << shift; with PAIR the same factors
// twist y as well.
// For LOG_R >= 4 the column is the same for all 16 residues and
// bitrev(pos_j) = bitrev(pos_0) + sum over the set bits i of j of
// bitrev(delta_(2^i)), so the 16 factors are the subset products of w^(E_0)
// and four D_i = w^(colsh bitrev(delta_(2^i))).  bitrev(delta_(2^i)) is a power
// of two that doubles as i falls within a group's bits, so D_i = D_(i+1)^2
// there: two or three table lookups, the squares and fifteen products instead
// of sixteen scattered lookup pairs.
template <class S, int LOG_R, int Q, bool PAIR>
__device__ __forceinline__ void twist16(uint32_t (&x)[16], uint32_t (&y)[16], uint32_t t, uint32_t c0, int shift,
                                        const uint2 *lo, const uint2 *hi, uint32_t one, bool scaled) {
    if constexpr (LOG_R >= 4) {
        constexpr int B = S::kB;
        static_assert(S::kLO == 0, "twist stage");
        uint32_t pos0, c;
        S::elem(t, 0, pos0, c);
        const uint32_t colsh = (c0 + c) << shift;
        uint32_t D[4];
#pragma unroll
        for (int i = 3; i >= 0; --i) {
            const uint32_t r = crev(stage_delta(1 << i, B, LOG_R), LOG_R);
            const uint32_t above = i < 3 ? crev(stage_delta(2 << i, B, LOG_R), LOG_R) : 0u;
            D[i] = (i < 3 && r == 2u * above) ? norm<Q>(mont<Q>(D[i < 3 ? i + 1 : 3], D[i < 3 ? i + 1 : 3]))
                                              : root_m<Q>(lo, hi, colsh * r);
        }
        uint32_t F[16];
        F[0] = mul_root<Q>(one, lo, hi, colsh * bitrev(pos0, LOG_R));
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int k = 0; k < (1 << i); ++k) F[(1 << i) + k] = mont<Q>(F[k], D[i]);   // lazy, < 2p
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            x[j] = norm<Q>(mont<Q>(x[j], F[j]));
            if (PAIR) y[j] = norm<Q>(mont<Q>(y[j], F[j]));
        }
    } else {
        // short columns: R = 2, 4 or 8 positions of each of 16 / R columns 256
        // apart; a column's factors are the powers of w^(col << shift), and
        // consecutive columns differ by w^(256 << shift)
        static_assert(S::kB == LOG_R && S::kLO == 0, "whole columns in registers");
        uint32_t pos0, c;
        S::elem(t, 0, pos0, c);
        uint32_t A = root_m<Q>(lo, hi, (c0 + c) << shift);
        const uint32_t step = LOG_R < 4 ? root_m<Q>(lo, hi, 256u << shift) : 0u;
#pragma unroll
        for (int g = 0; g < (16 >> LOG_R); ++g) {
            if (g) A = norm<Q>(mont<Q>(A, step));
            uint32_t F[1 << LOG_R];
            F[0] = one;
            F[1] = scaled ? mont<Q>(one, A) : A;
#pragma unroll
            for (int k = 2; k < (1 << LOG_R); ++k) F[k] = mont<Q>(F[k - 1], A);   // lazy, < 2p
#pragma unroll
            for (int v = 0; v < (1 << LOG_R); ++v) {
                const uint32_t k = crev((uint32_t)v, LOG_R);
                const int j = (g << LOG_R) + v;
                if (k != 0u || scaled) {
                    x[j] = norm<Q>(mont<Q>(x[j], F[k]));
                    if (PAIR) y[j] = norm<Q>(mont<Q>(y[j], F[k]));
                }
            }
        }
    }
}

// How a first pass gets its limbs: in general (an operand of at most K limbs),
// from operands that fill at most the lower half of their K points (a balanced
// product at one power-of-two transform: half the loads, and the first level
// multiplies without adding), or through a ragged batch's descriptors (apart
// from the others: operand addresses that come from memory are not uniform to
// the compiler, and every access then needs 64-bit sums).  Operands that have
// to be folded or twisted go through k_fold first.
enum Load { kGeneral, kHalf, kRagged };

template <class First, int LOG_R, int Q, bool HALF>
__device__ __forceinline__ void load_limbs(uint32_t (&x)[16], const uint32_t *xr, uint32_t Lx, int log_cols,
                                           uint32_t i0) {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const uint32_t i = i0 + elem_delta<First, LOG_R>(j, log_cols);
        const bool upper = HALF && ((j >> (First::kB - 1)) & 1);   // positions R / 2 .. R - 1
        x[j] = (!upper && i < Lx) ? reduce_limb<Q>(__ldg(word_at(xr, i))) : 0u;
    }
}

// ---------------------------------------------------------------------------
// Residues of an operand X mod x^K - c_i, c_i = g^(iK), twisted by g^(ij), for
// the cosets i = coset0 .. coset0 + M - 1 of each row: F[vrow][q][K], which the
// column passes then transform in place.  A thread makes four consecutive
// positions of every coset for one prime:
//     residue (i, j + v) = g^(ij) sum_b X[j + v + b K] W[i][b][v],
//     W[i][b][v] = c_i^b g^(iv)  (in shared memory, the same for the CTA),
// so its limbs are loaded once for all cosets, g^(ij) is a chain over i, and a
// block costs one wide multiply-add and one reduction: the 64-bit sum is kept
// below 2^32 p by reducing its upper word only, and reduced once at the end.
// Inside the first column pass, where every coset's CTA loaded all blocks anew,
// the folding of eight cosets of four blocks (2^27 x 2^27 limbs) took 7.5 of
// the pass's 10.2 ms for both operands; here it takes 1.29 ms an operand and
// the pass on the residues 2.87 ms.
// ---------------------------------------------------------------------------
struct FoldArgs {
    const uint32_t *X;
    uint64_t sX;
    uint32_t Lx;
    uint32_t nb;   // K-limb blocks of the longest row
    uint32_t *F;
    int log_k;
    int M, coset0;
    const RaggedRow *rows;
    int side;
};
constexpr int kFoldV = 4;
constexpr int kFoldRegs = 4;   // blocks whose limbs a thread holds in registers

// limbs i .. i + 3 of a row, 0 past its end
__device__ __forceinline__ void limbs4(const LimbRow &X, uint32_t i, uint32_t (&v)[kFoldV]) {
    const uint32_t *p = X.p + i;
    if (i + kFoldV <= X.L && ((uintptr_t)p & 15u) == 0u) {
        const uint4 q = __ldg(reinterpret_cast<const uint4 *>(p));
        v[0] = q.x;
        v[1] = q.y;
        v[2] = q.z;
        v[3] = q.w;
        return;
    }
#pragma unroll
    for (int k = 0; k < kFoldV; ++k) v[k] = (i + k < X.L) ? __ldg(p + k) : 0u;
}

template <int Q, bool REGS>
__device__ __forceinline__ void fold_body(const NttParams &P, const FoldArgs &a, uint64_t b, uint32_t *W) {
    const uint32_t tiles = (1u << a.log_k) / (kThreads * kFoldV);
    const uint64_t row = b / tiles;
    const uint32_t j = ((uint32_t)(b - row * tiles) * kThreads + threadIdx.x) * kFoldV;
    const LimbRow X = limb_row(a.rows, a.side, a.X, a.sX, a.Lx, row);
    const uint32_t *clo = coset_lo_ptr(P.tab, 0, Q), *chi = coset_hi_ptr(P.tab, 0, Q);
    uint32_t v[REGS ? kFoldRegs : 1][kFoldV];
    if constexpr (REGS) {
#pragma unroll
        for (int k = 0; k < kFoldRegs; ++k)
            limbs4(X, j + ((uint32_t)k << a.log_k), v[k]);   // beyond the row's blocks: zeros
    }
    for (uint32_t e = threadIdx.x; e < (uint32_t)a.M * a.nb * kFoldV; e += kThreads) {
        const uint32_t u = e & (kFoldV - 1u), rest = e / kFoldV;
        const uint32_t i = (uint32_t)a.coset0 + rest / a.nb, blk = rest % a.nb;
        uint32_t w = mul_coset<Q, 0>(PrimeC<Q>::r1, clo, chi, i * u);
        const uint32_t c = mul_coset<Q, 0>(PrimeC<Q>::r1, clo, chi, i << a.log_k);
        for (uint32_t k = 0; k < blk; ++k) w = norm<Q>(mont<Q>(w, c));
        W[e] = w;
    }
    const uint32_t h = mul_coset<Q, 0>(PrimeC<Q>::r1, clo, chi, j);   // g^j
    uint32_t f = PrimeC<Q>::r1;                                         // g^(ij)
    if (a.coset0) f = h;
    __syncthreads();
    uint32_t *F = a.F + (((row * a.M * 3 + Q) << a.log_k) + j);
    const uint32_t nb = REGS ? a.nb : (X.L + (1u << a.log_k) - 1u) >> a.log_k;
    for (int i = 0; i < a.M; ++i) {
        uint32_t lo[kFoldV], hi[kFoldV];
#pragma unroll
        for (int k = 0; k < kFoldV; ++k) lo[k] = hi[k] = 0u;
        auto add = [&](const uint32_t (&x)[kFoldV], uint32_t blk) {
            const uint4 q = *reinterpret_cast<const uint4 *>(W + ((uint32_t)i * a.nb + blk) * kFoldV);
            const uint32_t w[kFoldV] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int k = 0; k < kFoldV; ++k) {
                const uint64_t s = (uint64_t)x[k] * w[k] + (((uint64_t)hi[k] << 32) | lo[k]);
                lo[k] = (uint32_t)s;
                hi[k] = norm<Q>((uint32_t)(s >> 32));   // < p again
            }
        };
        if constexpr (REGS) {
#pragma unroll
            for (uint32_t blk = 0; blk < (uint32_t)kFoldRegs; ++blk)
                if (blk < nb) add(v[blk], blk);
        } else {
            for (uint32_t blk = 0; blk < nb; ++blk) {
                uint32_t x[kFoldV];
                limbs4(X, j + (blk << a.log_k), x);
                add(x, blk);
            }
        }
        uint32_t r[kFoldV];
#pragma unroll
        for (int k = 0; k < kFoldV; ++k) r[k] = norm<Q>(mont<Q>(redc<Q>(lo[k], hi[k]), f));
        *reinterpret_cast<uint4 *>(F + ((uint64_t)(3 * i) << a.log_k)) = make_uint4(r[0], r[1], r[2], r[3]);
        f = norm<Q>(mont<Q>(f, h));
    }
}

template <bool REGS>
__global__ void __launch_bounds__(kThreads) k_fold(NttParams P, FoldArgs a) {
    __shared__ __align__(16) uint32_t W[kMaxCosets * kMaxCosets * kFoldV];
    uint64_t b;
    const int q = grid_prime(b);
    if (q == 0)
        fold_body<0, REGS>(P, a, b, W);
    else if (q == 1)
        fold_body<1, REGS>(P, a, b, W);
    else
        fold_body<2, REGS>(P, a, b, W);
}

// Column pass: R = 2^LOG_R (<= 1024) points per column, TC = 4096 / R columns
// per CTA; segment of S = 2^log_s points viewed as [R][S/R].  PAIR: the
// forward pass of A and B together (same tile, shared twiddles and twists).
template <int LOG_R, bool FROM_LIMBS, bool INVERSE, bool PAIR, Load LOAD, int Q>
__device__ __forceinline__ void cols_body(const NttParams &P, const ColsArgs &a, uint64_t b, uint32_t *Sm,
                                          uint32_t *Sm2, uint2 *tw) {
    constexpr bool HALF = LOAD == kHalf;
    constexpr int LOG_TC = 12 - LOG_R;
    constexpr int NS = StagePlan<LOG_R>::n;
    using First = typename ExecStage<LOG_R, LOG_TC, INVERSE, 0>::S;
    using Last = typename ExecStage<LOG_R, LOG_TC, INVERSE, NS - 1>::S;
    const int log_cols = a.log_s - LOG_R;
    const uint32_t ctiles = 1u << (log_cols - LOG_TC);
    const uint32_t nseg = 1u << (a.log_k - a.log_s);
    uint32_t ct, seg;
    uint64_t vrow;
    ct = (uint32_t)(b % ctiles);
    b /= ctiles;
    seg = (uint32_t)(b % nseg);
    vrow = b / nseg;
    const int dir = INVERSE ? 1 : 0;
    const uint64_t K = 1ull << a.log_k;
    const uint2 *twhi = root_hi_ptr(P.tab, dir, Q);
    const uint2 *twlo = root_lo_ptr(P.tab, dir, Q);
    const uint2 *lev = level_ptr(P.tab, dir, Q);
    for (uint32_t e = threadIdx.x; e < (1u << LOG_R) - 1u; e += kThreads) tw[e] = __ldg(lev + e);
    const uint64_t off = vrow * 3 * K + (uint64_t)Q * K + ((uint64_t)seg << a.log_s);
    uint32_t *F = a.F + off;
    uint32_t *F2 = PAIR ? a.F2 + off : nullptr;
    const uint32_t c0 = ct << LOG_TC;
    const int twist_shift = kMaxLog - a.log_s;
    const uint32_t t = threadIdx.x;
    uint32_t pos0, col0;
    First::elem(t, 0, pos0, col0);
    const uint32_t i0 = (pos0 << log_cols) + c0 + col0;   // this thread's first residue
    uint32_t x[16], y[16];
    if constexpr (FROM_LIMBS) {
        const RaggedRow *rows = LOAD == kRagged ? a.rows : nullptr;
        const LimbRow X = limb_row(rows, a.side, a.X, a.sX, a.Lx, vrow);
        load_limbs<First, LOG_R, Q, HALF>(x, X.p, X.L, log_cols, i0);
        if constexpr (PAIR) {
            const LimbRow Y = limb_row(rows, 1, a.X2, a.sX2, a.Lx2, vrow);
            load_limbs<First, LOG_R, Q, HALF>(y, Y.p, Y.L, log_cols, i0);
        }
    } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const uint32_t i = i0 + elem_delta<First, LOG_R>(j, log_cols);
            x[j] = *word_at(F, i);
            if constexpr (PAIR) y[j] = *word_at(F2, i);
        }
        if constexpr (INVERSE) {
            const uint32_t one = a.scaled ? __ldg(P.tab.inv2n + a.log_k * kPrimes + Q) : PrimeC<Q>::r1;
            twist16<First, LOG_R, Q, PAIR>(x, y, t, c0, twist_shift, twlo, twhi, one, a.scaled != 0);
        }
    }
    __syncthreads();   // twiddle table ready
    run_stages_pair<LOG_R, LOG_TC, INVERSE, Q, 0, PAIR, CtaSync, HALF>(x, y, Sm, Sm2, t, tw, CtaSync{});
    if constexpr (!INVERSE) twist16<Last, LOG_R, Q, PAIR>(x, y, t, c0, twist_shift, twlo, twhi, PrimeC<Q>::r1, false);
    uint32_t pos1, c1;
    Last::elem(t, 0, pos1, c1);
    const uint32_t i1 = (pos1 << log_cols) + c0 + c1;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const uint32_t i = i1 + elem_delta<Last, LOG_R>(j, log_cols);
        *word_at(F, i) = x[j];
        if constexpr (PAIR) *word_at(F2, i) = y[j];
    }
}

template <int LOG_R, bool PAIR>
constexpr size_t cols_smem_bytes() {   // one or two padded tiles + the twiddle levels
    return (size_t)(PAIR ? 2 : 1) * kTilePad * 4u + (size_t)((1 << LOG_R) - 1) * 8u;
}

// Four CTAs per SM for every pass (64 registers; of them all, two unpaired first
// passes spill 16 and 36 bytes): the extra resident warps hide more of the limb
// and tile latency (first pass of a 2^24 x 2^24-limb product 0.589 -> 0.541 ms
// against three CTAs per SM).
template <int LOG_R, bool FROM_LIMBS, bool INVERSE, bool PAIR, Load LOAD>
__global__ void __launch_bounds__(kThreads, 4) k_cols_r(NttParams P, ColsArgs a) {
    extern __shared__ uint4 cols_smem[];
    uint32_t *Sm = reinterpret_cast<uint32_t *>(cols_smem);
    uint32_t *Sm2 = PAIR ? Sm + kTilePad : Sm;
    uint2 *tw = reinterpret_cast<uint2 *>(Sm + (PAIR ? 2 : 1) * kTilePad);
    uint64_t b;
    const int q = grid_prime(b);
    if (q == 0)
        cols_body<LOG_R, FROM_LIMBS, INVERSE, PAIR, LOAD, 0>(P, a, b, Sm, Sm2, tw);
    else if (q == 1)
        cols_body<LOG_R, FROM_LIMBS, INVERSE, PAIR, LOAD, 1>(P, a, b, Sm, Sm2, tw);
    else
        cols_body<LOG_R, FROM_LIMBS, INVERSE, PAIR, LOAD, 2>(P, a, b, Sm, Sm2, tw);
}

__device__ __forceinline__ void swap16(uint32_t (&x)[16], uint32_t (&y)[16]) {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const uint32_t v = x[j];
        x[j] = y[j];
        y[j] = v;
    }
}

struct RowsArgs {
    const uint32_t *A;   // limbs (whole products of at most 4096 points)
    uint64_t sA;
    uint32_t La;
    const uint32_t *B;
    uint64_t sB;
    uint32_t Lb;
    uint32_t *FA;
    const uint32_t *FB;
    int log_k;
    int M;               // cosets per row
    int b_bcast;         // B row 0 serves every row
    int square;          // B is A
    const RaggedRow *rows;   // whole products of a ragged batch: per-row operands
    __device__ __forceinline__ LimbRow a_row(uint64_t row) const { return limb_row(rows, 0, A, sA, La, row); }
    __device__ __forceinline__ LimbRow b_row(uint64_t row) const {
        return limb_row(rows, 1, B, b_bcast ? 0u : sB, square ? 0u : Lb, row);
    }
};

// Whole product of C = 2^LOG_C points (512 .. 2048, T = C/16 threads) from
// limbs: forward stages of A then B (A stays in registers while B reuses the
// shared tile), pointwise product * C^-1, inverse stages.  The last forward
// and the first inverse stage share one thread mapping, so the product never
// leaves registers.  The forward twiddle levels are replaced by the inverse
// ones in the same shared buffer once the forward stages are done.
template <int LOG_C, int Q>
__device__ __forceinline__ void rows_body(const NttParams &P, const RowsArgs &a, uint64_t row, uint32_t *Sm,
                                          uint2 *tw) {
    constexpr int C = 1 << LOG_C;
    constexpr int T = C / 16;
    constexpr int NS = StagePlan<LOG_C>::n;
    using First = typename ExecStage<LOG_C, 0, false, 0>::S;
    using Out = typename ExecStage<LOG_C, 0, true, NS - 1>::S;
    const LimbRow A = a.a_row(row), B = a.b_row(row);   // B empty for squares
    const uint32_t scale = __ldg(P.tab.inv2n + LOG_C * kPrimes + Q);
    const uint2 *levf = level_ptr(P.tab, 0, Q);
    const uint2 *levi = level_ptr(P.tab, 1, Q);
    for (uint32_t e = threadIdx.x; e < C - 1; e += T) tw[e] = __ldg(levf + e);
    const uint32_t t = threadIdx.x;
    uint32_t xa[16], xb[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        uint32_t pos, c;
        First::elem(t, j, pos, c);
        xa[j] = (pos < A.L) ? reduce_limb<Q>(__ldg(A.p + pos)) : 0u;
        xb[j] = (pos < B.L) ? reduce_limb<Q>(__ldg(B.p + pos)) : 0u;
    }
    __syncthreads();
#pragma unroll 1
    for (int op = 0; op < (a.square ? 1 : 2); ++op) {
        if (op) {
            __syncthreads();   // A's last hand-off has been read
            swap16(xa, xb);
        }
        run_stages<LOG_C, 0, false, Q, 0>(xa, Sm, t, tw, CtaSync{});
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const uint32_t y = a.square ? xa[j] : xb[j];
        xa[j] = norm<Q>(mont<Q>(mont<Q>(xa[j], y), scale));   // x y C^-1
    }
    __syncthreads();   // forward twiddles no longer read
    for (uint32_t e = threadIdx.x; e < C - 1; e += T) tw[e] = __ldg(levi + e);
    __syncthreads();
    run_stages<LOG_C, 0, true, Q, 0>(xa, Sm, t, tw, CtaSync{});
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        uint32_t pos, c;
        Out::elem(t, j, pos, c);
        a.FA[(row * 3 + Q) * C + pos] = xa[j];
    }
}

template <int LOG_C>
constexpr size_t rows_smem_bytes() {   // the padded tile + the twiddle levels
    return (size_t)((1 << LOG_C) + (1 << LOG_C) / 32) * 4u + (size_t)((1 << LOG_C) - 1) * 8u;
}

template <int LOG_C>
__global__ void __launch_bounds__((1 << LOG_C) / 16) k_rows_r(NttParams P, RowsArgs a) {
    extern __shared__ uint4 rows_smem[];
    constexpr int C = 1 << LOG_C;
    uint32_t *Sm = reinterpret_cast<uint32_t *>(rows_smem);
    uint2 *tw = reinterpret_cast<uint2 *>(Sm + C + C / 32);
    uint64_t b;
    const int q = grid_prime(b);
    if (q == 0)
        rows_body<LOG_C, 0>(P, a, b, Sm, tw);
    else if (q == 1)
        rows_body<LOG_C, 1>(P, a, b, Sm, tw);
    else
        rows_body<LOG_C, 2>(P, a, b, Sm, tw);
}

// ---------------------------------------------------------------------------
// 4096-point row passes: persistent CTAs of two 256-thread groups.  A group
// has a tile and a named barrier of its own; the CTA's forward and inverse
// twiddle levels (2 x 32 KiB) stay in shared memory while its groups work
// through a contiguous run of segments (at most two or three runs: one per
// prime).  With one CTA per segment the tables were loaded afresh for every
// product, two to four times, each with two barriers: as much shared-memory
// traffic as the transforms' own hand-offs.
// ---------------------------------------------------------------------------
constexpr int kRowLog = 12;
constexpr int kRowPoints = 1 << kRowLog;
constexpr int kRowGroups = 2;
constexpr int kRowThreads = 256 * kRowGroups;
constexpr int kRowCtas = 2;   // per SM: 64 registers a thread, 2 x 97 KiB shared memory
static_assert(kRowPoints == 16 * 256, "a group holds one segment in registers");

constexpr size_t row_smem_bytes() { return (size_t)kRowGroups * kTilePad * 4u + 2u * kRowPoints * 8u; }
// CTAs for all primes' segments.  Up to one per SM a segment has a CTA of its
// own: two in one CTA would share an SM while others idle, and a CTA's share
// across two primes loads both primes' tables one after the other (the three
// segments of one 2047 x 2047-limb product in two CTAs: 22.6 us a product, in three
// 16.4).  Above that the groups of a CTA share the tables (297 segments: 26.7 us
// in 149 CTAs, 27.9 in 296).
constexpr unsigned row_grid(uint64_t segments) {
    return segments <= (uint64_t)kNumSMs ? (unsigned)segments
           : (segments + kRowGroups - 1) / kRowGroups < (uint64_t)kNumSMs * kRowCtas
               ? (unsigned)((segments + kRowGroups - 1) / kRowGroups)
               : (unsigned)(kNumSMs * kRowCtas);
}
static_assert(row_grid(3) == 3 && row_grid(148) == 148 && row_grid(297) == 149 &&
              row_grid(1 << 20) == kNumSMs * kRowCtas, "CTAs of the row kernels");

struct RowShared {
    uint32_t *tile;   // this group's
    uint2 *twf, *twi;
};

__device__ __forceinline__ RowShared row_shared(uint4 *smem) {
    uint32_t *w = reinterpret_cast<uint32_t *>(smem);
    RowShared s;
    s.twf = reinterpret_cast<uint2 *>(w);
    s.twi = s.twf + kRowPoints;
    s.tile = reinterpret_cast<uint32_t *>(s.twi + kRowPoints) + (threadIdx.x >> 8) * kTilePad;
    return s;
}

__device__ __forceinline__ void row_tables(const NttParams &P, int q, const RowShared &s) {
    __syncthreads();   // the previous prime's stages are done
    const uint2 *f = level_ptr(P.tab, 0, q), *i = level_ptr(P.tab, 1, q);
    for (uint32_t e = threadIdx.x; e < (uint32_t)kRowPoints - 1u; e += kRowThreads) {
        s.twf[e] = __ldg(f + e);
        s.twi[e] = __ldg(i + e);
    }
    __syncthreads();
}

// This CTA's share [first, last) of prime q's `segs` segments (2^30 segments
// would be 12 TB of residues).
__device__ __forceinline__ bool row_share(uint32_t segs, uint32_t q, uint32_t &first, uint32_t &last) {
    const uint64_t total = (uint64_t)segs * kPrimes;
    const uint32_t lo = (uint32_t)(total * blockIdx.x / gridDim.x), hi = (uint32_t)(total * (blockIdx.x + 1u) / gridDim.x);
    const uint32_t a = segs * q;
    first = max(lo, a) - a;
    last = min(hi, a + segs);
    if (last <= a + first) return false;
    last -= a;
    return true;
}

// 16 KiB segments are 16-byte aligned (K >= 4096 residues from the workspace's
// base): bulk prefetch to L2 by the copy engine.
__device__ __forceinline__ void prefetch_segment(const uint32_t *p) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"((uint32_t)kRowPoints * 4u) : "memory");
}

using RowFirst = typename ExecStage<kRowLog, 0, false, 0>::S;
using RowOut = typename ExecStage<kRowLog, 0, true, StagePlan<kRowLog>::n - 1>::S;
using RowLast = typename ExecStage<kRowLog, 0, false, StagePlan<kRowLog>::n - 1>::S;
static_assert(RowLast::kLO == 0 && RowLast::kB == 4, "last row stage holds 16 consecutive positions");

// Fused row pass of one product: forward stages of A then B through one copy
// of the code (a loop: smaller code for the instruction cache), pointwise
// product / R, inverse stages; the first inverse column pass multiplies by
// K^-1 R with its twist.  The loads between the transforms come from L2, where
// the group's next segment is sent while it transforms the one before.
// One 2^28-point product (196,608 segments): 6.88 -> 5.13 ms.
template <int Q>
__device__ __forceinline__ void rows_run(const RowsArgs &a, uint32_t first, uint32_t last, const RowShared &s) {
    const uint32_t t = threadIdx.x & 255u;
    const uint32_t grp = threadIdx.x >> 8;
    const GroupSync sync{1u + grp};
    const int log_seg = a.log_k - kRowLog;
    auto offset = [&](uint32_t vrow, uint32_t b) {
        return ((uint64_t)(((vrow * 3u + Q) << log_seg) + (b & ((1u << log_seg) - 1u)))) << kRowLog;
    };
    auto prefetch = [&](uint32_t b) {
        if (t < 2u && b < last) {
            const uint32_t v = b >> log_seg;
            if (t == 0u)
                prefetch_segment(a.FA + offset(v, b));
            else if (!a.square)
                prefetch_segment(a.FB + offset(a.b_bcast ? v % (uint32_t)a.M : v, b));
        }
    };
    prefetch(first + grp);
#pragma unroll 1
    for (uint32_t b = first + grp; b < last; b += kRowGroups) {
        const uint32_t vrow = b >> log_seg;
        const uint32_t brow = a.b_bcast ? (vrow % (uint32_t)a.M) : vrow;
        uint32_t *FA = a.FA + offset(vrow, b) + t;
        prefetch(b + kRowGroups);
        uint32_t k[16], x[16];   // the transform of A, the operand at hand
#pragma unroll 1
        for (int op = a.square ? 1 : 0; op < 2; ++op) {
            const uint32_t *X = op && !a.square ? a.FB + offset(brow, b) + t : FA;
#pragma unroll
            for (int j = 0; j < 16; ++j) x[j] = X[256u * j];
            if (op && !a.square) sync();   // A's last hand-off has been read
            run_stages<kRowLog, 0, false, Q, 0>(x, s.tile, t, s.twf, sync);
            if (!op || a.square) {
#pragma unroll
                for (int j = 0; j < 16; ++j) k[j] = x[j];
            }
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) x[j] = norm<Q>(mont<Q>(k[j], x[j]));
        run_stages<kRowLog, 0, true, Q, 0>(x, s.tile, t, s.twi, sync);
#pragma unroll
        for (int j = 0; j < 16; ++j) FA[256u * j] = x[j];
    }
}

// Whole products of 4096 points, from limbs: both operands' limbs are loaded
// at once (their HBM latency overlaps), the product is scaled by K^-1 here.
// 1024 products of 2001 x 1903 limbs: 125 -> 98 us.
template <bool HALF, int Q>
__device__ __forceinline__ void rows_limbs_run(const NttParams &P, const RowsArgs &a, uint32_t first, uint32_t last,
                                               const RowShared &s) {
    const uint32_t t = threadIdx.x & 255u;
    const uint32_t grp = threadIdx.x >> 8;
    const GroupSync sync{1u + grp};
#pragma unroll 1
    for (uint32_t row = first + grp; row < last; row += kRowGroups) {
        const LimbRow A = a.a_row(row), B = a.b_row(row);   // B empty for squares
        uint32_t xa[16], xb[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const uint32_t pos = t + 256u * j;
            const bool upper = HALF && j >= 8;
            xa[j] = (!upper && pos < A.L) ? reduce_limb<Q>(__ldg(A.p + pos)) : 0u;
            xb[j] = (!upper && pos < B.L) ? reduce_limb<Q>(__ldg(B.p + pos)) : 0u;
        }
#pragma unroll 1
        for (int op = 0; op < (a.square ? 1 : 2); ++op) {
            if (op) {
                sync();   // A's last hand-off has been read
                swap16(xa, xb);
            }
            run_stages<kRowLog, 0, false, Q, 0, HALF>(xa, s.tile, t, s.twf, sync);
        }
        const uint32_t scale = __ldg(P.tab.inv2n + kRowLog * kPrimes + Q);
#pragma unroll
        for (int j = 0; j < 16; ++j)
            xa[j] = norm<Q>(mont<Q>(mont<Q>(xa[j], a.square ? xa[j] : xb[j]), scale));
        run_stages<kRowLog, 0, true, Q, 0>(xa, s.tile, t, s.twi, sync);
        uint32_t *out = a.FA + (((uint64_t)row * 3u + Q) << kRowLog) + t;
#pragma unroll
        for (int j = 0; j < 16; ++j) out[256u * j] = xa[j];
    }
}

template <bool LIMBS, bool HALF, int Q>
__device__ __forceinline__ void rows_prime(const NttParams &P, const RowsArgs &a, uint32_t segs, const RowShared &s) {
    uint32_t first, last;
    if (!row_share(segs, Q, first, last)) return;
    row_tables(P, Q, s);
    if constexpr (LIMBS)
        rows_limbs_run<HALF, Q>(P, a, first, last, s);
    else
        rows_run<Q>(a, first, last, s);
}

// HALF (with LIMBS): operands of at most 2048 limbs
template <bool LIMBS, bool HALF>
__global__ void __launch_bounds__(kRowThreads, kRowCtas) k_rows(NttParams P, RowsArgs a, uint32_t segs) {
    extern __shared__ uint4 rows_smem[];
    const RowShared s = row_shared(rows_smem);
    rows_prime<LIMBS, HALF, 0>(P, a, segs, s);
    rows_prime<LIMBS, HALF, 1>(P, a, segs, s);
    rows_prime<LIMBS, HALF, 2>(P, a, segs, s);
}

// Whole product of K <= 2^8 points per CTA (one prime, one row), radix-2
// levels in shared memory.
constexpr int kSmallLog = 8;

template <int Q>
__device__ __forceinline__ void rows_small_body(const NttParams &P, const RowsArgs &a, uint64_t row,
                                                uint32_t *SA, uint32_t *SB, uint2 *twf, uint2 *twi) {
    const int log_k = a.log_k;
    const uint32_t K = 1u << log_k;
    const LimbRow A = a.a_row(row), B = a.b_row(row);
    const uint32_t scale = __ldg(P.tab.inv2n + log_k * kPrimes + Q);
    const uint2 *levf = level_ptr(P.tab, 0, Q) + (K / 2 - 1u);   // top level: w_K^e, e < K/2
    const uint2 *levi = level_ptr(P.tab, 1, Q) + (K / 2 - 1u);
    for (uint32_t e = threadIdx.x; e < K / 2; e += blockDim.x) {
        twf[e] = __ldg(levf + e);
        twi[e] = __ldg(levi + e);
    }
    for (uint32_t i = threadIdx.x; i < K; i += blockDim.x) {
        SA[i] = (i < A.L) ? reduce_limb<Q>(__ldg(A.p + i)) : 0u;
        SB[i] = (i < B.L) ? reduce_limb<Q>(__ldg(B.p + i)) : 0u;
    }
    __syncthreads();
    tile_transform<Q, false>(SA, log_k, 0, twf);
    if (!a.square) tile_transform<Q, false>(SB, log_k, 0, twf);
    for (uint32_t i = threadIdx.x; i < K; i += blockDim.x) {
        const uint32_t x = SA[i];
        const uint32_t y = a.square ? x : SB[i];
        SA[i] = norm<Q>(mont<Q>(mont<Q>(x, y), scale));
    }
    __syncthreads();
    tile_transform<Q, true>(SA, log_k, 0, twi);
    for (uint32_t i = threadIdx.x; i < K; i += blockDim.x) a.FA[row * 3 * K + (uint64_t)Q * K + i] = SA[i];
}

__global__ void __launch_bounds__(128) k_rows_small(NttParams P, RowsArgs a) {
    __shared__ uint32_t SA[1 << kSmallLog], SB[1 << kSmallLog];
    __shared__ uint2 twf[1 << (kSmallLog - 1)], twi[1 << (kSmallLog - 1)];
    uint64_t row;
    const int q = grid_prime(row);
    if (q == 0)
        rows_small_body<0>(P, a, row, SA, SB, twf, twi);
    else if (q == 1)
        rows_small_body<1>(P, a, row, SA, SB, twf, twi);
    else
        rows_small_body<2>(P, a, row, SA, SB, twf, twi);
}

// ---------------------------------------------------------------------------
// Split row passes for products that share forward transforms.
//
// k_rows_fwd finishes the forward transform of one or two operands whose
// column passes are done; the last stage's registers (thread t holds
// positions 16t .. 16t + 15) go through the shared tile to the first
// stage's order (thread t holds t + 256 j), so the spectrum is stored with
// coalesced 128-byte warp accesses.  k_rows_inv loads T pairs of spectra in
// that order, forms sum_t X_t Y_t / R (mod p), moves the result back to
// the last stage's order through the tile and runs the inverse stages,
// leaving the segment in the order the inverse column passes expect, as the
// fused k_rows does.  So a transform computed once serves every product
// it takes part in, and a sum of products costs one inverse transform.
// ---------------------------------------------------------------------------
constexpr int kSplitLogC = kRowLog;
using SplitLast = RowLast;

struct RowsFwdArgs {
    uint32_t *F0;   // spectra [vrow][q][K], column passes done
    uint32_t *F1;   // second operand of the same shape, or null
    int log_k;
};

template <int Q>
__device__ __forceinline__ void rows_fwd_body(const RowsFwdArgs &a, uint64_t b, uint32_t *Sm, uint2 *tw) {
    constexpr int C = 1 << kSplitLogC;
    constexpr int T = C / 16;
    using First = typename ExecStage<kSplitLogC, 0, false, 0>::S;
    const uint32_t nseg = 1u << (a.log_k - kSplitLogC);
    const uint64_t K = 1ull << a.log_k;
    const uint64_t off = (b / nseg) * 3 * K + (uint64_t)Q * K + ((uint64_t)(b % nseg) << kSplitLogC);
    const uint32_t t = threadIdx.x;
    for (int op = 0; op < (a.F1 ? 2 : 1); ++op) {
        uint32_t *F = (op == 0 ? a.F0 : a.F1) + off;
        uint32_t x[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            uint32_t pos, c;
            First::elem(t, j, pos, c);
            x[j] = F[pos];
        }
        __syncthreads();   // twiddles loaded; the previous operand has left the tile
        run_stages<kSplitLogC, 0, false, Q, 0>(x, Sm, t, tw, CtaSync{});
        SplitLast::store(Sm, x, t);   // every thread passed the last stage's tile loads
        __syncthreads();
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            uint32_t pos, c;
            First::elem(t, j, pos, c);
            F[pos] = Sm[First::addr(pos, c)];
        }
        __syncthreads();
    }
    (void)T;
}

__global__ void __launch_bounds__((1 << kSplitLogC) / 16, 4) k_rows_fwd(NttParams P, RowsFwdArgs a) {
    extern __shared__ uint4 rows_smem[];
    constexpr int C = 1 << kSplitLogC;
    uint32_t *Sm = reinterpret_cast<uint32_t *>(rows_smem);
    uint2 *tw = reinterpret_cast<uint2 *>(Sm + C + C / 32);
    uint64_t b;
    const int q = grid_prime(b);
    const uint2 *lev = level_ptr(P.tab, 0, q);
    for (uint32_t e = threadIdx.x; e < C - 1; e += C / 16) tw[e] = __ldg(lev + e);
    if (q == 0)
        rows_fwd_body<0>(a, b, Sm, tw);
    else if (q == 1)
        rows_fwd_body<1>(a, b, Sm, tw);
    else
        rows_fwd_body<2>(a, b, Sm, tw);
}

constexpr int kMaxTerms = 2;
struct RowsInvArgs {
    const uint32_t *X[kMaxTerms];
    const uint32_t *Y[kMaxTerms];
    uint32_t *Fout;   // may be one of the X or Y (each CTA reads its segment before writing it)
    int terms;
    int log_k;
};

template <int TERMS, int Q>
__device__ __forceinline__ void rows_inv_body(const NttParams &P, const RowsInvArgs &a, uint64_t b, uint32_t *Sm,
                                              uint2 *tw) {
    using Out = typename ExecStage<kSplitLogC, 0, true, StagePlan<kSplitLogC>::n - 1>::S;
    const uint32_t nseg = 1u << (a.log_k - kSplitLogC);
    const uint64_t K = 1ull << a.log_k;
    const uint64_t off = (b / nseg) * 3 * K + (uint64_t)Q * K + ((uint64_t)(b % nseg) << kSplitLogC);
    const uint32_t t = threadIdx.x;
    using First = typename ExecStage<kSplitLogC, 0, false, 0>::S;
    uint32_t x[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) x[j] = 0u;
#pragma unroll
    for (int term = 0; term < TERMS; ++term) {
        const uint32_t *X = a.X[term] + off, *Y = a.Y[term] + off;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            uint32_t pos, c;
            First::elem(t, j, pos, c);
            x[j] = add_n<Q>(x[j], norm<Q>(mont<Q>(__ldg(X + pos), __ldg(Y + pos))));
        }
    }
    First::store(Sm, x, t);
    __syncthreads();   // tile written, inverse twiddles loaded
    SplitLast::load(Sm, x, t);
    run_stages<kSplitLogC, 0, true, Q, 0>(x, Sm, t, tw, CtaSync{});
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        uint32_t pos, c;
        Out::elem(t, j, pos, c);
        a.Fout[off + pos] = x[j];
    }
}

template <int TERMS>
__global__ void __launch_bounds__((1 << kSplitLogC) / 16, 4) k_rows_inv(NttParams P, RowsInvArgs a) {
    extern __shared__ uint4 rows_smem[];
    constexpr int C = 1 << kSplitLogC;
    uint32_t *Sm = reinterpret_cast<uint32_t *>(rows_smem);
    uint2 *tw = reinterpret_cast<uint2 *>(Sm + C + C / 32);
    uint64_t b;
    const int q = grid_prime(b);
    const uint2 *lev = level_ptr(P.tab, 1, q);
    for (uint32_t e = threadIdx.x; e < C - 1; e += C / 16) tw[e] = __ldg(lev + e);
    // two segments per CTA (their count is even: K >= 8192) share the
    // twiddle table load
    for (uint64_t s = 2 * b; s < 2 * b + 2; ++s) {
        if (q == 0)
            rows_inv_body<TERMS, 0>(P, a, s, Sm, tw);
        else if (q == 1)
            rows_inv_body<TERMS, 1>(P, a, s, Sm, tw);
        else
            rows_inv_body<TERMS, 2>(P, a, s, Sm, tw);
        // the next segment's first store goes where this thread's last loads came from
    }
}

// One merge level's four row products in one pass (the tuned form's level):
// from the column-transformed segments of P_e, P_o, R_o, Q_o, Q_e, R_e a group
// forms P' = P_e P_o, R2 = P_e R_o, Q' = Q_e Q_o, R1 = R_e Q_o (each / R; the
// first inverse column pass scales them by K^-1 R) and runs their inverse row
// stages, writing them over P_o, R_o, Q_e and R_e: six forward and four
// inverse row transforms, the kept operand (P_e, then Q_o) and one product in
// registers, no spectrum stored.  With Fpo null (the tree's root) P' is not
// formed: five and three.
struct RowsLevelArgs {
    uint32_t *Fpe, *Fpo, *Fro, *Fqo, *Fqe, *Fre;
    int log_k;
};

template <int Q>
__device__ __forceinline__ void level_run(const RowsLevelArgs &a, uint32_t first, uint32_t last, const RowShared &s) {
    const uint32_t t = threadIdx.x & 255u;
    const uint32_t grp = threadIdx.x >> 8;
    const GroupSync sync{1u + grp};
    const int log_seg = a.log_k - kRowLog;
    auto offset = [&](uint32_t b) {
        return ((uint64_t)((((b >> log_seg) * 3u + Q) << log_seg) + (b & ((1u << log_seg) - 1u)))) << kRowLog;
    };
    // The next segment's six operand segments go to L2 while this one is
    // transformed, so the loads between its transforms find them there.
    auto prefetch = [&](uint32_t b) {
        if (t < 6u && b < last) {
            const uint32_t *F = t == 0u ? a.Fpe : t == 1u ? a.Fpo : t == 2u ? a.Fro : t == 3u ? a.Fqo
                                                                          : t == 4u ? a.Fqe : a.Fre;
            if (F) prefetch_segment(F + offset(b));
        }
    };
    prefetch(first + grp);
    // One copy of the forward and one of the inverse stages per prime, run
    // in loops (the ten transforms written out would not fit the instruction
    // cache).  Per half: the kept operand F_keep, then F0 (its product with
    // F_keep waits in F0's own segment: word j of thread t at j * 256 + t,
    // coalesced; every thread has loaded F0 before the next barrier and reads
    // back only its own words; the segment is rewritten by the product's
    // inverse anyway), then F1 (its product stays in registers); the inverse of
    // F_keep F1 goes to F1, that of the held product to F0.
    // F0 null (the tree's root, uniform over the grid): no P' product.
#pragma unroll 1
    for (uint32_t b = first + grp; b < last; b += kRowGroups) {
        const uint64_t off = offset(b) + t;
        prefetch(b + kRowGroups);
        uint32_t k[16], x[16];
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
            const uint32_t *Fk = h ? a.Fqo : a.Fpe;
            uint32_t *F0 = h ? a.Fqe : a.Fpo;
            uint32_t *F1 = h ? a.Fre : a.Fro;
#pragma unroll 1
            for (int step = 0; step < 3; ++step) {
                const uint32_t *src = step == 0 ? Fk : (step == 1 ? F0 : F1);
                if (!src) continue;
#pragma unroll
                for (int j = 0; j < 16; ++j) x[j] = __ldg(src + off + 256u * j);
                if (step) sync();   // the previous forward transform's last hand-off has been read
                run_stages<kRowLog, 0, false, Q, 0>(x, s.tile, t, s.twf, sync);
                if (step == 0) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) k[j] = x[j];
                } else if (step == 1) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) F0[off + 256u * j] = norm<Q>(mont<Q>(k[j], x[j]));
                } else {
#pragma unroll
                    for (int j = 0; j < 16; ++j) x[j] = norm<Q>(mont<Q>(k[j], x[j]));
                }
            }
#pragma unroll 1
            for (int step = 0; step < 2; ++step) {
                uint32_t *dst = step ? F0 : F1;
                if (step == 1) {
                    if (!F0) break;
                    sync();   // the previous inverse transform's last hand-off has been read
#pragma unroll
                    for (int j = 0; j < 16; ++j) x[j] = F0[off + 256u * j];
                }
                run_stages<kRowLog, 0, true, Q, 0>(x, s.tile, t, s.twi, sync);
#pragma unroll
                for (int j = 0; j < 16; ++j) dst[off + 256u * j] = x[j];
            }
        }
    }
}

// 64 registers a thread (two CTAs of 512): 64 bytes of spill stores.
__global__ void __launch_bounds__(kRowThreads, kRowCtas) k_rows_level(NttParams P, RowsLevelArgs a, uint32_t segs) {
    extern __shared__ uint4 rows_smem[];
    const RowShared s = row_shared(rows_smem);
    uint32_t first, last;
    if (row_share(segs, 0, first, last)) {
        row_tables(P, 0, s);
        level_run<0>(a, first, last, s);
    }
    if (row_share(segs, 1, first, last)) {
        row_tables(P, 1, s);
        level_run<1>(a, first, last, s);
    }
    if (row_share(segs, 2, first, last)) {
        row_tables(P, 2, s);
        level_run<2>(a, first, last, s);
    }
}

// Coset recombination.  Row r holds z_i[j] = C_i[j] g^(ij) for cosets i < M;
// C_i[j] = sum_b C_b[j] c_i^b, so C_b[j] = sum_i Vinv[b][i] C_i[j].  The M
// outputs of position j overwrite the M inputs of position j.
struct CombineArgs {
    uint32_t *F;
    int log_k;
    uint32_t vinv[kPrimes][kMaxCosets][kMaxCosets];   // Montgomery form, [q][b][i]
};

// The untwist factors of position j are the powers of g^-j (one table lookup);
// each output sums 64-bit products, reducing the upper word only after each
// (as the first pass's coset sums) and fully once.  Eight cosets of 2^25
// points: 3.22 -> 1.85 ms.
template <int M, int Q>
__device__ __forceinline__ void combine_body(const NttParams &P, const CombineArgs &a, uint64_t row, uint32_t j) {
    const uint64_t K = 1ull << a.log_k;
    uint32_t *F0 = a.F + row * M * 3 * K + (uint64_t)Q * K + j;
    const uint32_t h = mul_coset<Q, 1>(PrimeC<Q>::r1, coset_lo_ptr(P.tab, 1, Q), coset_hi_ptr(P.tab, 1, Q), j);
    uint32_t u[M];
#pragma unroll
    for (int i = 0; i < M; ++i) u[i] = F0[(uint64_t)i * 3 * K];
    uint32_t f = h;   // g^(-ij), < 2p
#pragma unroll
    for (int i = 1; i < M; ++i) {
        u[i] = norm<Q>(mont<Q>(u[i], f));
        if (i + 1 < M) f = mont<Q>(f, h);
    }
#pragma unroll
    for (int b = 0; b < M; ++b) {
        uint32_t lo = 0u, hi = 0u;   // hi < p after each term
#pragma unroll
        for (int i = 0; i < M; ++i) {
            const uint64_t s = (uint64_t)u[i] * a.vinv[Q][b][i] + (((uint64_t)hi << 32) | lo);
            lo = (uint32_t)s;
            hi = norm<Q>((uint32_t)(s >> 32));
        }
        F0[(uint64_t)b * 3 * K] = norm<Q>(redc<Q>(lo, hi));
    }
}

template <int M>
__global__ void __launch_bounds__(kThreads) k_combine(NttParams P, CombineArgs a) {
    uint64_t rest;
    const int q = grid_prime(rest);
    const uint32_t jblocks = (1u << a.log_k) / kThreads;
    const uint64_t row = rest / jblocks;
    const uint32_t j = (uint32_t)(rest - row * jblocks) * kThreads + threadIdx.x;
    if (q == 0)
        combine_body<M, 0>(P, a, row, j);
    else if (q == 1)
        combine_body<M, 1>(P, a, row, j);
    else
        combine_body<M, 2>(P, a, row, j);
}

// Two-part recombination: C1 mod x^K1 - 1 in F1[row][q][K1], z[j] = C2[j] g^j
// in F2[row][q][K2] -> T in F2 and C's coefficients below K2, C1 - T, in F1
// (those from K2 to K1 are C1's own).  C1 folds mod x^K2 - c, c = g^K2, as
// sum_b C1[j + b K2] c^b; w[q][b] holds -c^b / (g^K1 - 1) and w[q][parts] its
// reciprocal factor 1 / (g^K1 - 1), Montgomery form.  One read of both parts and
// one write of 2 K2 points: HBM-bound, against M^2 products per M points for
// equal cosets (five cosets of 2^13 points x 96 rows: 42 us, this 20 us).
constexpr int kMaxFold = 16;   // K1 / K2
struct Combine2Args {
    uint32_t *F1, *F2;
    int log_k1, log_k2;
    uint32_t w[kPrimes][kMaxFold + 1];
};

template <int Q>
__device__ __forceinline__ void combine2_body(const NttParams &P, const Combine2Args &a, uint64_t row, uint32_t j) {
    const uint64_t base = row * 3 + Q;
    uint32_t *F1 = a.F1 + (base << a.log_k1) + j;
    uint32_t *F2 = a.F2 + (base << a.log_k2) + j;
    const uint32_t parts = 1u << (a.log_k1 - a.log_k2);
    const uint32_t first = F1[0];
    const uint32_t h = mul_coset<Q, 1>(PrimeC<Q>::r1, coset_lo_ptr(P.tab, 1, Q), coset_hi_ptr(P.tab, 1, Q), j);
    uint64_t s = (uint64_t)norm<Q>(mont<Q>(F2[0], h)) * a.w[Q][parts];
    uint32_t lo = (uint32_t)s, hi = (uint32_t)(s >> 32);   // hi < p, after each term
    uint32_t v = first;
    for (uint32_t b = 0; b < parts; ++b) {
        const uint32_t next = b + 1u < parts ? F1[(uint64_t)(b + 1u) << a.log_k2] : 0u;
        s = (uint64_t)v * a.w[Q][b] + (((uint64_t)hi << 32) | lo);
        lo = (uint32_t)s;
        hi = norm<Q>((uint32_t)(s >> 32));
        v = next;
    }
    const uint32_t T = norm<Q>(redc<Q>(lo, hi));
    F2[0] = T;
    F1[0] = sub_n<Q>(first, T);
}

__global__ void __launch_bounds__(kThreads) k_combine2(NttParams P, Combine2Args a) {
    uint64_t rest;
    const int q = grid_prime(rest);
    const uint32_t jblocks = (1u << a.log_k2) / kThreads;
    const uint64_t row = rest / jblocks;
    const uint32_t j = (uint32_t)(rest - row * jblocks) * kThreads + threadIdx.x;
    if (q == 0)
        combine2_body<0>(P, a, row, j);
    else if (q == 1)
        combine2_body<1>(P, a, row, j);
    else
        combine2_body<2>(P, a, row, j);
}

// Garner: residues (r0, r1, r2) -> coefficient < p0 p1 p2 as 3 limbs.
//   t1 = (r1 - r0) / p0 mod p1,  t2 = ((r2 - r0) / p0 - t1) / p1 mod p2,
//   x  = r0 + p0 t1 + p0 p1 t2.
constexpr uint32_t kI01 = cinv(Prime<0>::p, Prime<1>::p);
constexpr uint32_t kI02 = cinv(Prime<0>::p, Prime<2>::p);
constexpr uint32_t kI12 = cinv(Prime<1>::p, Prime<2>::p);
constexpr uint32_t kI01q = shoup_of(kI01, Prime<1>::p);
constexpr uint32_t kI02q = shoup_of(kI02, Prime<2>::p);
constexpr uint32_t kI12q = shoup_of(kI12, Prime<2>::p);
constexpr uint64_t kP0P1 = (uint64_t)Prime<0>::p * Prime<1>::p;

// x = r0 + p0 t1 + p0 p1 t2 as three wide multiply-adds: none overflows
// 64 bits (p0 t1 + r0 < 2^62, its sum with lo(p0 p1) t2 < 2^64).
__device__ __forceinline__ void garner(uint32_t r0, uint32_t r1, uint32_t r2, uint32_t (&out)[3]) {
    const uint32_t t1 = norm<1>(shoup<1>(sub_n<1>(r1, r0), kI01, kI01q));   // r0 < p0 < p1
    const uint32_t u = norm<2>(shoup<2>(sub_n<2>(r2, r0), kI02, kI02q));
    const uint32_t t2 = norm<2>(shoup<2>(sub_n<2>(u, t1), kI12, kI12q));    // t1 < p1 < p2
    const uint64_t w = (uint64_t)t2 * (uint32_t)kP0P1 + ((uint64_t)t1 * Prime<0>::p + r0);
    const uint64_t v = (uint64_t)t2 * (uint32_t)(kP0P1 >> 32) + (w >> 32);
    out[0] = (uint32_t)w;
    out[1] = (uint32_t)v;
    out[2] = (uint32_t)(v >> 32);
}

// CRT and carry: each thread turns eight consecutive coefficients into eight
// limbs and two words that spill into the next thread's.  Thread 0 of a CTA
// repeats the last chunk of the previous tile for its spill, so a tile is 255
// chunks (repeating it in the tile's first thread after its own chunk kept the
// CTA waiting for a second round of loads).
constexpr int kCrtV = 8;
constexpr uint32_t kCrtSpan = (kThreads - 1) * kCrtV;   // 2040 limbs per tile

// x += h (two words), carries through the eight words; returns the carry out
__device__ __forceinline__ uint32_t add_words(uint32_t (&x)[kCrtV], uint32_t h0, uint32_t h1) {
    uint32_t c;
    asm("add.cc.u32 %0, %0, %9;\n\taddc.cc.u32 %1, %1, %10;\n\taddc.cc.u32 %2, %2, 0;\n\t"
        "addc.cc.u32 %3, %3, 0;\n\taddc.cc.u32 %4, %4, 0;\n\taddc.cc.u32 %5, %5, 0;\n\t"
        "addc.cc.u32 %6, %6, 0;\n\taddc.cc.u32 %7, %7, 0;\n\taddc.u32 %8, 0, 0;"
        : "+&r"(x[0]), "+r"(x[1]), "+r"(x[2]), "+r"(x[3]), "+r"(x[4]), "+r"(x[5]), "+r"(x[6]), "+r"(x[7]), "=r"(c)
        : "r"(h0), "r"(h1));
    return c;
}

// words += c (96 bits) where words = {a1, a2} is what lies above the words
// already given out: returns the next word, leaves the rest in {a1, a2}
__device__ __forceinline__ uint32_t next_word(const uint32_t (&c)[3], uint32_t &a1, uint32_t &a2) {
    uint32_t w, b1, b2;
    asm("add.cc.u32 %0, %3, %6;\n\taddc.cc.u32 %1, %4, %7;\n\taddc.u32 %2, %5, 0;"
        : "=&r"(w), "=&r"(b1), "=&r"(b2)
        : "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(a1), "r"(a2));
    a1 = b1;
    a2 = b2;
    return w;
}

struct CrtArgs {
    const uint32_t *F;
    int log_k;
    int M;
    const uint32_t *F2;   // coefficients from K on, of a two-part product, or null
    int log_k2;
    uint32_t *C;
    uint64_t sC;
    uint32_t Lc;
    uint32_t tiles;
    uint32_t *flags;
    uint32_t ncoef;      // coefficients of the product (L_a + L_b - 1)
    // optional addend: C = product + (D << dshift), D rows at D + row * sD,
    // Ld limbs; C's L_c limbs must hold the sum
    const uint32_t *D;
    uint64_t sD;
    uint32_t Ld;
    uint32_t dshift;
    const RaggedRow *rows;   // ragged batch: each row's output place and length
};

// Adds limbs base .. base + 7 of (D << dshift) to a chunk's words (a carry
// runs into its spill words, which stay far from overflowing).
__device__ __forceinline__ void crt_add_shifted(const CrtArgs &a, const uint32_t *Dr, int64_t base,
                                                uint32_t (&S)[kCrtV + 2]) {
    const int64_t i0 = base - (int64_t)(a.dshift >> 5);
    uint32_t prev = ((uint64_t)(i0 - 1) < (uint64_t)a.Ld) ? Dr[i0 - 1] : 0u;   // below 0 wraps
    uint64_t cy = 0;
#pragma unroll
    for (int v = 0; v < kCrtV + 2; ++v) {
        uint32_t d = 0u;
        if (v < kCrtV) {
            const uint32_t cur = ((uint64_t)(i0 + v) < (uint64_t)a.Ld) ? Dr[i0 + v] : 0u;
            d = __funnelshift_l(prev, cur, a.dshift & 31u);
            prev = cur;
        }
        const uint64_t t = (uint64_t)S[v] + d + cy;
        S[v] = (uint32_t)t;
        cy = t >> 32;
    }
}

// A row's coefficients: n < M K lives in block b = n / K at F[(b * 3 + q) * K +
// n mod K], those of a two-part product from K on at F2[q * K2 + n - K].  There
// are ncoef = L_c - 1 of them (the top limb only receives carries).
struct CrtRow {
    const uint32_t *F, *F2;
    int log_k, log_k2;
    uint32_t ncoef;
    // the word of prime 0 for coefficient n, and the distance to the next prime's
    __device__ __forceinline__ const uint32_t *at(uint64_t n, uint64_t &next) const {
        if (F2 && (n >> log_k)) {
            next = 1ull << log_k2;
            return F2 + (n - (1ull << log_k));
        }
        next = 1ull << log_k;
        return F + (((n >> log_k) * 3) << log_k) + (n & (next - 1ull));
    }
};

// S = sum_v c_(base + v) 2^(32 v): eight words and the spill
__device__ __forceinline__ void crt_chunk(const CrtRow &r, int64_t base, uint32_t (&S)[kCrtV + 2]) {
    uint64_t K;
    uint32_t a1 = 0u, a2 = 0u, c[3];
    if (base >= 0 && base + kCrtV <= (int64_t)r.ncoef && r.log_k >= 3) {
        // the chunk lies in one block: two 128-bit loads per prime (K and base are multiples of 8)
        const uint32_t *f = r.at((uint64_t)base, K);
        uint4 q[3][2];
#pragma unroll
        for (int p = 0; p < 3; ++p)
#pragma unroll
            for (int h = 0; h < 2; ++h) q[p][h] = *reinterpret_cast<const uint4 *>(f + p * K + 4 * h);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            garner(q[0][h].x, q[1][h].x, q[2][h].x, c);
            S[4 * h] = next_word(c, a1, a2);
            garner(q[0][h].y, q[1][h].y, q[2][h].y, c);
            S[4 * h + 1] = next_word(c, a1, a2);
            garner(q[0][h].z, q[1][h].z, q[2][h].z, c);
            S[4 * h + 2] = next_word(c, a1, a2);
            garner(q[0][h].w, q[1][h].w, q[2][h].w, c);
            S[4 * h + 3] = next_word(c, a1, a2);
        }
    } else {
#pragma unroll
        for (int v = 0; v < kCrtV; ++v) {
            const int64_t i = base + v;
            c[0] = c[1] = c[2] = 0u;
            if (i >= 0 && i < (int64_t)r.ncoef) {
                const uint32_t *f = r.at((uint64_t)i, K);
                garner(f[0], f[K], f[2 * K], c);
            }
            S[v] = next_word(c, a1, a2);
        }
    }
    S[kCrtV] = a1;
    S[kCrtV + 1] = a2;
}

// Bound by HBM (12 bytes read and 4 written per limb): 2^28 limbs 1.18 -> 0.70
// ms (4.3 GB, 6.1 TB/s); 111 instructions per limb before (four coefficients per thread, 64-bit
// sums of their words, scalar stores).
__global__ void __launch_bounds__(kThreads) k_crt(CrtArgs a) {
    __shared__ uint32_t sg[kThreads / 32], sp[kThreads / 32];
    __shared__ uint32_t spill[kThreads / 32][2];
    const uint32_t tile = blockIdx.x;
    const uint32_t row = tile / a.tiles;
    const uint32_t t = tile - row * a.tiles;
    const uint32_t Lc = a.rows ? a.rows[row].La + a.rows[row].Lb : a.Lc;
    const CrtRow cr{a.F + (((uint64_t)row * a.M * 3) << a.log_k),
                    a.F2 ? a.F2 + (((uint64_t)row * 3) << a.log_k2) : nullptr, a.log_k, a.log_k2,
                    a.rows ? Lc - 1u : a.ncoef};
    const int64_t base = (int64_t)t * kCrtSpan + ((int)threadIdx.x - 1) * kCrtV;
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    uint32_t S[kCrtV + 2];
    crt_chunk(cr, base, S);
    if (a.D) crt_add_shifted(a, a.D + row * a.sD, base, S);
    // words of the previous chunk's sum that land in this chunk
    uint32_t h0 = __shfl_up_sync(0xffffffffu, S[kCrtV], 1);
    uint32_t h1 = __shfl_up_sync(0xffffffffu, S[kCrtV + 1], 1);
    if (lane == 31) {
        spill[warp][0] = S[kCrtV];
        spill[warp][1] = S[kCrtV + 1];
    }
    __syncthreads();
    if (lane == 0 && warp > 0) {
        h0 = spill[warp - 1][0];
        h1 = spill[warp - 1][1];
    }
    uint32_t X[kCrtV];
#pragma unroll
    for (int v = 0; v < kCrtV; ++v) X[v] = S[v];
    bool g = add_words(X, h0, h1) != 0u, p = base + kCrtV <= (int64_t)Lc;
#pragma unroll
    for (int v = 0; v < kCrtV; ++v) p = p && (X[v] == 0xffffffffu);
    if (threadIdx.x == 0) {   // the previous tile's chunk: neither generates nor stops a carry
        g = false;
        p = true;
    }
    const BlockCarry bc = block_resolve<kThreads / 32>(g, p, sg, sp);
    add_words(X, bc.cin, 0u);
    uint32_t *out = a.C + (a.rows ? a.rows[row].offC : row * a.sC);
    if (threadIdx.x > 0) {
        if (base + kCrtV <= (int64_t)Lc && ((uintptr_t)(out + base) & 15u) == 0u) {
            *reinterpret_cast<uint4 *>(out + base) = make_uint4(X[0], X[1], X[2], X[3]);
            *reinterpret_cast<uint4 *>(out + base + 4) = make_uint4(X[4], X[5], X[6], X[7]);
        } else {
#pragma unroll
            for (int v = 0; v < kCrtV; ++v)
                if (base + v < (int64_t)Lc) out[base + v] = X[v];
        }
    }
    if (a.tiles > 1u && threadIdx.x == 0) a.flags[tile] = bc.G | (bc.P << 1);
}

// ---------------------------------------------------------------------------
// Host orchestration
// ---------------------------------------------------------------------------
static int ceil_log2(uint64_t x) {
    int k = 0;
    while ((1ull << k) < x) ++k;
    return k;
}

struct Shape {
    int log_k;   // K = 2^log_k points per coset
    int M;       // cosets
};

// Smallest shape with M * K >= L_a + L_b - 1: one power-of-two transform up to
// 2^25 points, above that M cosets of 2^25 points.
}  // namespace ntt
bool ntt_shape_override(uint64_t need, uint32_t N, int *log_k, int *M);   // tune.cu
uint32_t ntt_small_batch(uint64_t need);                                  // tune.cu
namespace ntt {

static Shape shape_for(uint32_t La, uint32_t Lb);

// The transform shape of a batch of N products: the tune table's, else the
// built-in rule (shape_for).  Used by the plain product and its workspace size;
// the tuned splitting tree's spectra keep the built-in rule.
static Shape shape_tuned(uint32_t N, uint32_t La, uint32_t Lb) {
    int lk = 0, M = 0;
    const uint64_t need = (uint64_t)La + Lb - 1u;
    if (ntt_shape_override(need, N, &lk, &M)) return Shape{lk, M};
    // just above one transform: 2^25 points and a second part instead of two
    // cosets of 2^25
    if (need > (1ull << kMaxLog) && need <= (5ull << (kMaxLog - 2))) return Shape{kMaxLog - 2, 5};
    if (need > (1ull << kMaxLog) && need <= (3ull << (kMaxLog - 1))) return Shape{kMaxLog - 1, 3};
    return shape_for(La, Lb);
}

static Shape shape_for(uint32_t La, uint32_t Lb) {
    const uint64_t need = (uint64_t)La + Lb - 1u;
    if (need <= (1ull << kMaxLog)) {
        const int k = ceil_log2(need < 2 ? 2 : need);
        return {k < 1 ? 1 : k, 1};
    }
    const uint64_t K = 1ull << kMaxLog;
    return {kMaxLog, (int)((need + K - 1) / K)};
}

// Paired passes exist for R >= 32 only: shorter columns, of small transforms and
// second parts, run operand by operand.
constexpr int kPairMinLogR = 5;
// Column lengths up to 1024 run as one pass (tiles of 4096 / R columns; for
// R = 1024 a row segment is half a 32-byte sector, whose other half the
// neighbouring tile reads at the same time from L2).  Longer columns are
// split in two passes: single passes of 2048 / 4096 points measured slower
// (K = 2^23: 0.82 against 0.72 ms) with their 4095-entry twiddle tables per
// CTA and 4- / 8-byte row segments; K = 2^22 runs 0.36 ms in one 1024-point
// pass against 0.41 ms in two.
constexpr int kOnePassMaxLog = 10;

template <int LOG_R, bool FL, bool INV, bool PAIR, Load LOAD>
static void cols_launch(unsigned blocks, const NttParams &P, const ColsArgs &a, cudaStream_t st) {
    constexpr size_t smem = cols_smem_bytes<LOG_R, PAIR>();
    static bool attr = false;
    if (!attr) {
        if (smem > 48 * 1024)
            cudaFuncSetAttribute(k_cols_r<LOG_R, FL, INV, PAIR, LOAD>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem);
        attr = true;
    }
    k_cols_r<LOG_R, FL, INV, PAIR, LOAD><<<blocks, kThreads, smem, st>>>(P, a);
}

template <bool FL, bool INV, bool PAIR, Load LOAD = kGeneral>
static void cols_r_dispatch(int log_r, unsigned blocks, const NttParams &P, const ColsArgs &a, cudaStream_t st) {
    if constexpr (!PAIR) {
        switch (log_r) {
            case 1: cols_launch<1, FL, INV, false, LOAD>(blocks, P, a, st); return;
            case 2: cols_launch<2, FL, INV, false, LOAD>(blocks, P, a, st); return;
            case 3: cols_launch<3, FL, INV, false, LOAD>(blocks, P, a, st); return;
            case 4: cols_launch<4, FL, INV, false, LOAD>(blocks, P, a, st); return;
            default: break;
        }
    }
    switch (log_r) {
        case 5: cols_launch<5, FL, INV, PAIR, LOAD>(blocks, P, a, st); break;
        case 6: cols_launch<6, FL, INV, PAIR, LOAD>(blocks, P, a, st); break;
        case 7: cols_launch<7, FL, INV, PAIR, LOAD>(blocks, P, a, st); break;
        case 8: cols_launch<8, FL, INV, PAIR, LOAD>(blocks, P, a, st); break;
        case 9: cols_launch<9, FL, INV, PAIR, LOAD>(blocks, P, a, st); break;
        default: cols_launch<10, FL, INV, PAIR, LOAD>(blocks, P, a, st); break;
    }
}

// One column pass over vrows virtual rows (pair: operands A and B together).
static void launch_cols_r(bool from_limbs, bool inverse, bool pair, int log_r, const NttParams &P,
                          const ColsArgs &a, uint64_t vrows, cudaStream_t st) {
    const uint64_t ctiles = 1ull << (a.log_s - 12);
    const uint64_t nseg = 1ull << (a.log_k - a.log_s);
    const unsigned blocks = (unsigned)(vrows * kPrimes * nseg * ctiles);
    // algorithmic bytes: 4 B per residue read and written (3 primes per
    // point); a first pass on limbs reads those instead
    const double K = (double)(1ull << a.log_k);
    const double limbs = (double)a.Lx + (pair ? (double)a.Lx2 : 0.0);
    const double ops = pair ? 2.0 : 1.0;
    const double bytes = from_limbs ? (4.0 * limbs * (double)vrows + 12.0 * K * (double)vrows * ops)
                                    : 24.0 * K * (double)vrows * ops;
    KernelTimed kt(from_limbs ? "ntt_cols_fwd_first" : (inverse ? "ntt_cols_inv" : "ntt_cols_fwd"), bytes);
    if (from_limbs) {
        const uint64_t half = 1ull << (a.log_k - 1);
        const bool lower = a.Lx <= half && (!pair || a.Lx2 <= half);
        if (a.rows) {
            if (pair)
                cols_r_dispatch<true, false, true, kRagged>(log_r, blocks, P, a, st);
            else
                cols_r_dispatch<true, false, false, kRagged>(log_r, blocks, P, a, st);
        } else if (lower) {
            if (pair)
                cols_r_dispatch<true, false, true, kHalf>(log_r, blocks, P, a, st);
            else
                cols_r_dispatch<true, false, false, kHalf>(log_r, blocks, P, a, st);
        } else {
            if (pair)
                cols_r_dispatch<true, false, true>(log_r, blocks, P, a, st);
            else
                cols_r_dispatch<true, false, false>(log_r, blocks, P, a, st);
        }
    } else if (!inverse) {
        if (pair)
            cols_r_dispatch<false, false, true>(log_r, blocks, P, a, st);
        else
            cols_r_dispatch<false, false, false>(log_r, blocks, P, a, st);
    } else if (pair) {
        cols_r_dispatch<false, true, true>(log_r, blocks, P, a, st);
    } else {
        cols_r_dispatch<false, true, false>(log_r, blocks, P, a, st);
    }
    count_launch();
}

template <int LOG_C>
static void rows_launch(unsigned blocks, const NttParams &P, const RowsArgs &r, cudaStream_t st) {
    constexpr size_t smem = rows_smem_bytes<LOG_C>();
    static_assert(smem <= 48 * 1024, "within the default limit");
    k_rows_r<LOG_C><<<blocks, (1 << LOG_C) / 16, smem, st>>>(P, r);
}

// Shared-memory limit of the 4096-point row kernels, set once per device.
static void row_attr() {
    static std::mutex mu;
    static uint64_t done = 0;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> l(mu);
    if ((done >> (dev & 63)) & 1u) return;
    cudaFuncSetAttribute(k_rows<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)row_smem_bytes());
    cudaFuncSetAttribute(k_rows<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)row_smem_bytes());
    cudaFuncSetAttribute(k_rows<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)row_smem_bytes());
    cudaFuncSetAttribute(k_rows_level, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)row_smem_bytes());
    done |= 1ull << (dev & 63);
}

// Row pass of `segs` segments per prime.
static void launch_rows(int log_k, bool limbs, uint32_t segs, const NttParams &P, const RowsArgs &r, cudaStream_t st) {
    switch (limbs ? log_k : kRowLog) {
        case 9: rows_launch<9>((unsigned)(segs * kPrimes), P, r, st); break;
        case 10: rows_launch<10>((unsigned)(segs * kPrimes), P, r, st); break;
        case 11: rows_launch<11>((unsigned)(segs * kPrimes), P, r, st); break;
        default:
            row_attr();
            if (limbs && !r.rows && r.La <= kRowPoints / 2 && r.Lb <= kRowPoints / 2)
                k_rows<true, true><<<row_grid((uint64_t)segs * kPrimes), kRowThreads, row_smem_bytes(), st>>>(P, r,
                                                                                                            segs);
            else if (limbs)
                k_rows<true, false><<<row_grid((uint64_t)segs * kPrimes), kRowThreads, row_smem_bytes(), st>>>(
                    P, r, segs);
            else
                k_rows<false, false><<<row_grid((uint64_t)segs * kPrimes), kRowThreads, row_smem_bytes(), st>>>(P, r, segs);
    }
    count_launch();
}

// Inverse of the Vandermonde matrix V[i][b] = c_i^b (c_i = g^(i 2^log_k)) mod
// p_q, Montgomery form, out[q][b][i].
static void coset_matrix(int M, int log_k, uint32_t (&out)[kPrimes][kMaxCosets][kMaxCosets]) {
    for (int q = 0; q < kPrimes; ++q) {
        const uint32_t p = kP[q];
        uint32_t V[kMaxCosets][2 * kMaxCosets] = {};
        for (int i = 0; i < M; ++i) {
            const uint32_t c = h_pow(kGen[q], (uint64_t)i << log_k, p);
            uint32_t x = 1u;
            for (int b = 0; b < M; ++b) {
                V[i][b] = x;
                x = h_mul(x, c, p);
            }
            V[i][M + i] = 1u;
        }
        for (int col = 0; col < M; ++col) {   // Gauss-Jordan; the nodes are distinct
            int piv = col;
            while (V[piv][col] == 0u) ++piv;
            if (piv != col)
                for (int k = 0; k < 2 * M; ++k) {
                    const uint32_t tmp = V[piv][k];
                    V[piv][k] = V[col][k];
                    V[col][k] = tmp;
                }
            const uint32_t inv = h_inv(V[col][col], p);
            for (int k = 0; k < 2 * M; ++k) V[col][k] = h_mul(V[col][k], inv, p);
            for (int r = 0; r < M; ++r) {
                if (r == col || V[r][col] == 0u) continue;
                const uint32_t f = V[r][col];
                for (int k = 0; k < 2 * M; ++k)
                    V[r][k] = (uint32_t)((V[r][k] + (uint64_t)(p - h_mul(f, V[col][k], p))) % p);
            }
        }
        for (int b = 0; b < kMaxCosets; ++b)
            for (int i = 0; i < kMaxCosets; ++i)
                out[q][b][i] = (b < M && i < M) ? h_mont(V[b][M + i], p) : 0u;
    }
}

// Column passes below the 4096-point rows: one for up to 2^10 points,
// else two; returns their count.
static int column_passes(int log_k, int (&passes)[2]) {
    const int rest = log_k - 12;
    if (rest <= kOnePassMaxLog) {
        passes[0] = rest;
        return 1;
    }
    passes[0] = (rest + 1) / 2;
    passes[1] = rest / 2;
    return 2;
}

// Every coefficient, at most min(L_a, L_b) (2^32 - 1)^2, is below p0 p1 p2
// (min(L_a, L_b) < 4.18e8).
static bool crt_fits(uint64_t min_len) {
    unsigned __int128 cap = 1;
    for (int q = 0; q < kPrimes; ++q) cap *= kP[q];
    return (unsigned __int128)min_len * 0xffffffffull * 0xffffffffull < cap;
}

static void launch_combine(int M, const NttParams &P, const CombineArgs &c, uint32_t N, cudaStream_t st) {
    const uint64_t K = 1ull << c.log_k;
    const unsigned blocks = (unsigned)((uint64_t)N * kPrimes * (K / kThreads));
    KernelTimed kt("ntt_coset_combine", 24.0 * (double)K * M * N);
    switch (M) {
        case 2: k_combine<2><<<blocks, kThreads, 0, st>>>(P, c); break;
        case 3: k_combine<3><<<blocks, kThreads, 0, st>>>(P, c); break;
        case 4: k_combine<4><<<blocks, kThreads, 0, st>>>(P, c); break;
        case 5: k_combine<5><<<blocks, kThreads, 0, st>>>(P, c); break;
        case 6: k_combine<6><<<blocks, kThreads, 0, st>>>(P, c); break;
        case 7: k_combine<7><<<blocks, kThreads, 0, st>>>(P, c); break;
        case 8: k_combine<8><<<blocks, kThreads, 0, st>>>(P, c); break;
        case 9: k_combine<9><<<blocks, kThreads, 0, st>>>(P, c); break;
        case 10: k_combine<10><<<blocks, kThreads, 0, st>>>(P, c); break;
        case 11: k_combine<11><<<blocks, kThreads, 0, st>>>(P, c); break;
        case 12: k_combine<12><<<blocks, kThreads, 0, st>>>(P, c); break;
        case 13: k_combine<13><<<blocks, kThreads, 0, st>>>(P, c); break;
        case 14: k_combine<14><<<blocks, kThreads, 0, st>>>(P, c); break;
        case 15: k_combine<15><<<blocks, kThreads, 0, st>>>(P, c); break;
        case 16: k_combine<16><<<blocks, kThreads, 0, st>>>(P, c); break;
        case 17: k_combine<17><<<blocks, kThreads, 0, st>>>(P, c); break;
        case 18: k_combine<18><<<blocks, kThreads, 0, st>>>(P, c); break;
        case 19: k_combine<19><<<blocks, kThreads, 0, st>>>(P, c); break;
        default: k_combine<20><<<blocks, kThreads, 0, st>>>(P, c); break;
    }
    count_launch();
}

size_t workspace_bytes(uint32_t N, uint32_t La, uint32_t Lb) {
    if (N == 0u || La == 0u || Lb == 0u) return 0;
    const Shape s = shape_tuned(N, La, Lb);
    const uint64_t Lc = (uint64_t)La + Lb;
    const uint64_t tiles = (Lc + kCrtSpan - 1) / kCrtSpan;
    // a smaller batch may take a shape of more points: this size holds it too
    const Shape f = shape_for(La, Lb);
    const uint64_t few = std::min<uint64_t>(N, ntt_small_batch(Lc - 1u) - 1u);
    const uint64_t points = std::max(((uint64_t)N * s.M) << s.log_k, (few * f.M) << f.log_k);
    return (size_t)(2ull * points * 3 * 4 + N * tiles * 4 + 256);
}

// The two-part split of a shape of M K points (M with two bits set, the larger
// part within one transform).
static bool two_parts(Shape s, int *log_k1, int *log_k2) {
    if (s.log_k <= 12 || __builtin_popcount((unsigned)s.M) != 2) return false;
    const int hi = 31 - __builtin_clz((unsigned)s.M), lo = __builtin_ctz((unsigned)s.M);
    if (s.log_k + hi > kMaxLog || (1 << (hi - lo)) > kMaxFold) return false;
    *log_k1 = s.log_k + hi;
    *log_k2 = s.log_k + lo;
    return true;
}

// One operand of a transform: rows of X, or one side of a ragged batch.
struct Operand {
    const uint32_t *X;
    uint64_t sX;
    uint32_t Lx;       // limbs of the longest row
    uint32_t *F;
    uint32_t N;        // rows
};

// Forward column passes of one operand, or of two of the same shape (Y.F
// non-null; in the same launches where the columns are long enough to pair).
// Operands longer than K and cosets are folded into residues first.
static void forward_columns(const NttParams &P, int log_k, int M, int coset0, const Operand &X, const Operand &Y,
                            const RaggedRow *rows, int side, cudaStream_t st) {
    const uint64_t K = 1ull << log_k;
    int passes[2];
    const int npass = column_passes(log_k, passes);
    const bool pair = Y.F && passes[0] >= kPairMinLogR && (npass == 1 || passes[1] >= kPairMinLogR);
    const bool fold = M > 1 || coset0 || X.Lx > K || (Y.F && Y.Lx > K);
    for (int op = 0; fold && op < (Y.F ? 2 : 1); ++op) {
        const Operand &o = op ? Y : X;
        FoldArgs a{o.X, o.sX, o.Lx, (uint32_t)((o.Lx + K - 1) >> log_k), o.F, log_k, M, coset0, rows, side + op};
        const unsigned blocks = (unsigned)((uint64_t)o.N * kPrimes * (K / (kThreads * kFoldV)));
        KernelTimed kt("ntt_fold", 4.0 * (double)o.Lx * o.N + 12.0 * (double)K * M * o.N);
        if (a.nb <= (uint32_t)kFoldRegs)
            k_fold<true><<<blocks, kThreads, 0, st>>>(P, a);
        else
            k_fold<false><<<blocks, kThreads, 0, st>>>(P, a);
        count_launch();
    }
    for (int op = 0; op < (Y.F && !pair ? 2 : 1); ++op) {
        const Operand &o = op ? Y : X;
        int log_s = log_k;
        for (int ps = 0; ps < npass; ++ps) {
            ColsArgs a{o.X, o.sX, o.Lx, o.F, log_k, log_s, 0, Y.X, Y.sX, Y.Lx, pair ? Y.F : nullptr, rows, side + op};
            launch_cols_r(ps == 0 && !fold, false, pair, passes[ps], P, a, (uint64_t)o.N * M, st);
            log_s -= passes[ps];
        }
    }
}

// Inverse column passes of vrows virtual rows of F, innermost first (the
// first one scales by K^-1 R); of F2 as well, in the same launches where the
// columns are long enough to pair.
static void inverse_columns(const NttParams &P, int log_k, uint64_t vrows, uint32_t *F, uint32_t *F2,
                            cudaStream_t st) {
    int passes[2];
    const int npass = column_passes(log_k, passes);
    const bool pair = F2 && passes[0] >= kPairMinLogR && (npass == 1 || passes[1] >= kPairMinLogR);
    for (int op = 0; op < (F2 && !pair ? 2 : 1); ++op) {
        int log_s = kRowLog;
        for (int ps = npass - 1; ps >= 0; --ps) {
            log_s += passes[ps];
            ColsArgs a{nullptr, 0, 0, op ? F2 : F, log_k, log_s, ps == npass - 1, nullptr, 0, 0,
                       pair ? F2 : nullptr, nullptr, 0};
            launch_cols_r(false, true, pair, passes[ps], P, a, vrows, st);
        }
    }
}

struct Operands {
    const uint32_t *A, *B;
    uint32_t N, La, Lb;   // of a ragged batch: the longest operand on each side
    uint64_t sA, sB;
    bool square, bcast;   // B is A / one row of B serves every row
    const RaggedRow *rows;
};

// Residues of the products mod x^K - g^(iK) twisted by g^(ij), for the cosets
// i = coset0 .. coset0 + M - 1 of each row, left in FA.
static void cyclic_product(const NttParams &P, const Operands &o, int log_k, int M, int coset0, uint32_t *FA,
                           uint32_t *FB, cudaStream_t st) {
    const uint64_t K = 1ull << log_k;
    const uint64_t VR = (uint64_t)o.N * M;   // virtual rows (row, coset)
    // forward column passes: A and B together unless B is A or a broadcast row
    const Operand a{o.A, o.sA, o.La, FA, o.N}, b{o.B, o.sB, o.Lb, FB, o.bcast ? 1u : o.N}, none{};
    forward_columns(P, log_k, M, coset0, a, o.square || o.bcast ? none : b, o.rows, 0, st);
    if (o.bcast) forward_columns(P, log_k, M, coset0, b, none, nullptr, 1, st);
    RowsArgs r{o.A, o.sA, o.La, o.B, o.sB, o.Lb, FA, FB, log_k, M, o.bcast ? 1 : 0, o.square ? 1 : 0, nullptr};
    {
        KernelTimed kt("ntt_rows_fused", 12.0 * (double)K * ((o.square ? 2.0 : 3.0) * (double)VR));
        launch_rows(log_k, false, (uint32_t)(VR * (K >> kRowLog)), P, r, st);
    }
    inverse_columns(P, log_k, VR, FA, nullptr, st);
}

static void launch_combine2(const NttParams &P, uint32_t *F1, int log_k1, uint32_t *F2, int log_k2, uint32_t N,
                            cudaStream_t st) {
    Combine2Args a{};
    a.F1 = F1;
    a.F2 = F2;
    a.log_k1 = log_k1;
    a.log_k2 = log_k2;
    const int parts = 1 << (log_k1 - log_k2);
    for (int q = 0; q < kPrimes; ++q) {
        const uint32_t p = kP[q];
        const uint32_t c = h_pow(kGen[q], 1ull << log_k2, p);
        const uint32_t d = h_inv((h_pow(c, (uint64_t)parts, p) + p - 1u) % p, p);   // g^K1 != 1: p - 1 is no power of 2
        uint32_t x = p - d;
        for (int b = 0; b < parts; ++b) {
            a.w[q][b] = h_mont(x, p);
            x = h_mul(x, c, p);
        }
        a.w[q][parts] = h_mont(d, p);
    }
    KernelTimed kt("ntt_coset_combine", 12.0 * N * ((double)(1ull << log_k1) + 3.0 * (double)(1ull << log_k2)));
    k_combine2<<<(unsigned)((uint64_t)N * kPrimes * ((1ull << log_k2) / kThreads)), kThreads, 0, st>>>(P, a);
    count_launch();
}

// rows (device) non-null: a ragged batch, each product's operands and output
// from its descriptor; L_a + L_b is then the largest product's length (the
// workspace's too) and the strides are unused.
static void mul(const NttParams &P, const uint32_t *A, const uint32_t *B, uint32_t *C, uint32_t *ws,
                uint32_t N, uint32_t La, uint32_t Lb, uint64_t sA, uint64_t sB, uint64_t sC,
                const RaggedRow *rows = nullptr, uint32_t longest_a = 0u, uint32_t longest_b = 0u) {
    cudaStream_t st = current_stream();
    const uint32_t Lc = La + Lb;
    if (N == 0u || Lc == 0u) return;
    if (La == 0u || Lb == 0u) {
        cudaMemset2DAsync(C, sC * 4, 0, (size_t)Lc * 4, N, st);
        return;
    }
    const Shape s = shape_tuned(N, La, Lb);
    if (s.M > kMaxCosets) {
        fprintf(stderr, "gpupi_b200: product of %u limbs exceeds the 20 * 2^25-point limit\n", Lc);
        return;
    }
    if (!crt_fits(La < Lb ? La : Lb)) {
        fprintf(stderr, "gpupi_b200: min(L_a, L_b) = %u exceeds the three-prime CRT capacity\n", La < Lb ? La : Lb);
        return;
    }
    const bool square = (!rows && A == B && La == Lb && sA == sB);
    const bool bcast = (!rows && !square && sB == 0u && N > 1u);
    const uint32_t oa = rows ? longest_a : La, ob = rows ? longest_b : Lb;
    const uint64_t points = (uint64_t)N * s.M * 3 << s.log_k;
    const uint64_t tiles = ((uint64_t)Lc + kCrtSpan - 1) / kCrtSpan;
    uint32_t *FA = ws;
    uint32_t *FB = square ? FA : ws + points;
    uint32_t *flags = ws + 2ull * points;
    CrtArgs c{FA, s.log_k, s.M, nullptr, 0, C, sC, Lc, (uint32_t)tiles, flags, Lc - 1u, nullptr, 0, 0, 0, rows};
    int log_k2 = 0;
    if (s.log_k <= 12) {
        RowsArgs r{A, sA, La, B, sB, Lb, FA, FB, s.log_k, 1, bcast ? 1 : 0, square ? 1 : 0, rows};
        KernelTimed kt("ntt_local", 4.0 * N * ((double)La + (square ? 0 : Lb)) + 12.0 * (double)(1ull << s.log_k) * N);
        if (s.log_k >= 9) {
            launch_rows(s.log_k, true, N, P, r, st);
        } else {
            k_rows_small<<<(unsigned)(N * kPrimes), 128, 0, st>>>(P, r);
            count_launch();
        }
    } else if (two_parts(s, &c.log_k, &log_k2)) {
        const uint64_t p1 = (uint64_t)N * 3 << c.log_k;
        c.M = 1;
        c.F2 = FA + p1;
        c.log_k2 = log_k2;
        const Operands o{A, B, N, oa, ob, sA, sB, square, bcast, rows};
        cyclic_product(P, o, c.log_k, 1, 0, FA, FB, st);
        cyclic_product(P, o, log_k2, 1, 1, FA + p1, square ? FA + p1 : FB + p1, st);
        launch_combine2(P, FA, c.log_k, FA + p1, log_k2, N, st);
    } else {
        cyclic_product(P, Operands{A, B, N, oa, ob, sA, sB, square, bcast, rows}, s.log_k, s.M, 0, FA, FB, st);
        if (s.M > 1) {
            CombineArgs m{};
            m.F = FA;
            m.log_k = s.log_k;
            coset_matrix(s.M, s.log_k, m.vinv);
            launch_combine(s.M, P, m, N, st);
        }
    }
    KernelTimed kt("ntt_crt_carry", 12.0 * (double)Lc * N + 4.0 * (double)Lc * N);
    k_crt<<<(unsigned)(N * tiles), kThreads, 0, st>>>(c);
    count_launch();
    if (tiles > 1) launch_carry_fixup(false, C, sC, N, Lc, (uint32_t)tiles, kCrtSpan, false, flags, st, rows);
}

// ---------------------------------------------------------------------------
// Shared-transform products: spectrum_forward computes the forward transform
// of one operand (or two of the same shape) into caller buffers;
// spectrum_inverse turns a sum of products of such spectra into limbs.
// ---------------------------------------------------------------------------
static void rows_split_attr() {
    static bool done = false;
    if (!done) {
        constexpr int smem = (int)rows_smem_bytes<kSplitLogC>();
        cudaFuncSetAttribute(k_rows_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        cudaFuncSetAttribute(k_rows_inv<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        cudaFuncSetAttribute(k_rows_inv<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        done = true;
    }
}

static void spectrum_forward(const NttParams &P, Shape s, uint32_t N, const uint32_t *X, uint64_t sX, uint32_t Lx,
                             uint32_t *FX, const uint32_t *Y, uint64_t sY, uint32_t Ly, uint32_t *FY,
                             cudaStream_t st, bool rows) {
    const int log_k = s.log_k, M = s.M;
    const uint64_t K = 1ull << log_k;
    const uint64_t VR = (uint64_t)N * M;
    forward_columns(P, log_k, M, 0, Operand{X, sX, Lx, FX, N}, Operand{Y, sY, Ly, FY, N}, nullptr, 0, st);
    if (!rows) return;
    rows_split_attr();
    RowsFwdArgs r{FX, Y ? FY : nullptr, log_k};
    const unsigned blocks = (unsigned)(VR * kPrimes * (K >> kSplitLogC));
    KernelTimed kt("ntt_rows_fwd", 8.0 * (double)K * (double)VR * (Y ? 2.0 : 1.0) * kPrimes);
    k_rows_fwd<<<blocks, (1 << kSplitLogC) / 16, rows_smem_bytes<kSplitLogC>(), st>>>(P, r);
    count_launch();
}

static void spectrum_inverse(const NttParams &P, Shape s, uint32_t N, int terms, const uint32_t *const *X,
                             const uint32_t *const *Y, uint32_t *Fout, uint32_t *C, uint64_t sC, uint32_t Lc,
                             uint32_t *flags, cudaStream_t st, bool rows, bool cols,
                             const SpectrumAddend *add) {
    const int log_k = s.log_k, M = s.M;
    const uint64_t K = 1ull << log_k;
    const uint64_t VR = (uint64_t)N * M;
    rows_split_attr();
    if (rows) {
    RowsInvArgs r{};
    for (int i = 0; i < terms; ++i) {
        r.X[i] = X[i];
        r.Y[i] = Y[i];
    }
    r.Fout = Fout;
    r.terms = terms;
    r.log_k = log_k;
    const unsigned blocks = (unsigned)(VR * kPrimes * (K >> kSplitLogC) / 2);   // two segments per CTA
    {
        KernelTimed kt("ntt_rows_inv", 4.0 * (double)K * (double)VR * kPrimes * (2.0 * terms + 1.0));
        if (terms == 1)
            k_rows_inv<1><<<blocks, (1 << kSplitLogC) / 16, rows_smem_bytes<kSplitLogC>(), st>>>(P, r);
        else
            k_rows_inv<2><<<blocks, (1 << kSplitLogC) / 16, rows_smem_bytes<kSplitLogC>(), st>>>(P, r);
        count_launch();
    }
    }
    if (cols) inverse_columns(P, log_k, VR, Fout, nullptr, st);
    if (M > 1) {
        CombineArgs c{};
        c.F = Fout;
        c.log_k = log_k;
        coset_matrix(M, log_k, c.vinv);
        launch_combine(M, P, c, N, st);
    }
    const uint64_t tiles = ((uint64_t)Lc + kCrtSpan - 1) / kCrtSpan;
    CrtArgs c{Fout, log_k, M, nullptr, 0, C, sC, Lc, (uint32_t)tiles, flags, Lc - 1u, nullptr, 0, 0, 0, nullptr};
    if (add) {
        c.ncoef = add->ncoef;
        c.D = add->D;
        c.sD = add->sD;
        c.Ld = add->Ld;
        c.dshift = add->shift;
    }
    KernelTimed kt("ntt_crt_carry", 12.0 * (double)c.ncoef * N + 4.0 * (double)Lc * N +
                                        (add ? 4.0 * (double)add->Ld * N : 0.0));
    k_crt<<<(unsigned)(N * tiles), kThreads, 0, st>>>(c);
    count_launch();
    if (tiles > 1) launch_carry_fixup(false, C, sC, N, Lc, (uint32_t)tiles, kCrtSpan, false, flags, st);
}

void build_tables(std::vector<uint32_t> &lv1, std::vector<uint32_t> &lv2, std::vector<uint32_t> &inv2n) {
    lv1.assign(65536u * 3u, 0u);
    lv2.assign(65536u * 3u, 0u);
    inv2n.assign(33u * 3u, 0u);
    for (int q = 0; q < kPrimes; ++q) {
        const uint32_t p = kP[q];
        const uint32_t g = kGen[q];
        const uint32_t w = h_pow(g, (p - 1u) >> kMaxLog, p);   // primitive 2^25-th root
        for (int dir = 0; dir < 2; ++dir) {
            const uint32_t base = dir ? h_inv(w, p) : w;
            uint32_t x = 1u;
            for (uint32_t e = 0; e < kLoSize; ++e) {
                const size_t o = ((size_t)(dir * kPrimes + q) * kLoSize + e) * 2u;
                lv1[o] = x;
                lv1[o + 1] = shoup_of(x, p);
                x = h_mul(x, base, p);
            }
            const uint32_t step = h_pow(base, kLoSize, p);
            x = 1u;
            for (uint32_t e = 0; e < kHiSize; ++e) {
                const size_t o = kRootLoWords + ((size_t)(dir * kPrimes + q) * kHiSize + e) * 2u;
                lv1[o] = x;
                lv1[o + 1] = shoup_of(x, p);
                x = h_mul(x, step, p);
            }
            for (int lh = 0; lh < kLevelLogMax; ++lh) {
                const uint32_t root = h_pow(base, 1ull << (kMaxLog - 1 - lh), p);   // w_(2h), h = 2^lh
                x = 1u;
                for (uint32_t m = 0; m < (1u << lh); ++m) {
                    const size_t o =
                        kLevelOffset + ((size_t)(dir * kPrimes + q) * kLevelSize + (1u << lh) - 1u + m) * 2u;
                    lv1[o] = x;
                    lv1[o + 1] = shoup_of(x, p);
                    x = h_mul(x, root, p);
                }
            }
            const uint32_t gb = dir ? h_inv(g, p) : g;
            x = 1u;
            for (uint32_t e = 0; e < kCosetSize; ++e) {
                lv2[(size_t)(dir * kPrimes + q) * kCosetSize + e] = h_mont(x, p);
                x = h_mul(x, gb, p);
            }
            const uint32_t gstep = h_pow(gb, kCosetSize, p);
            x = 1u;
            for (uint32_t e = 0; e < kCosetSize; ++e) {
                lv2[kCosetWords + (size_t)(dir * kPrimes + q) * kCosetSize + e] = h_mont(x, p);
                x = h_mul(x, gstep, p);
            }
        }
        const uint32_t r2 = h_mont(h_mont(1u, p), p);   // R^2 mod p
        for (int k = 0; k <= 32; ++k) {
            const uint32_t kinv = h_inv(h_pow(2u, (uint64_t)k, p), p);
            inv2n[(size_t)k * kPrimes + q] = h_mul(kinv, r2, p);
        }
    }
}

}  // namespace ntt
}  // namespace gpupi

void init_ntt_precomputed_tables(NTTPrecomputedTables *tables) {
    std::vector<uint32_t> lv1, lv2, inv2n;
    gpupi::ntt::build_tables(lv1, lv2, inv2n);
    cudaMemcpy(tables->roots_table_lv1, lv1.data(), lv1.size() * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(tables->roots_table_lv2, lv2.data(), lv2.size() * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(tables->inv2n_table, inv2n.data(), inv2n.size() * 4, cudaMemcpyHostToDevice);
}

void batch_mul_ntt(uint32_t *A, uint32_t *B, uint32_t *ret, uint32_t *workspace,
                   NTTPrecomputedTables tables, uint32_t N, uint32_t L_a, uint32_t L_b,
                   uint32_t stride_A, uint32_t stride_B, uint32_t stride_ret) {
    const gpupi::ntt::NttParams P = gpupi::ntt::make_params(tables);
    gpupi::ntt::mul(P, A, B, ret, workspace, N, L_a, L_b, stride_A, stride_B, stride_ret);
}

size_t batch_mul_ntt_workspace_size(uint32_t N, uint32_t L_a, uint32_t L_b) {
    return gpupi::ntt::workspace_bytes(N, L_a, L_b);
}

namespace gpupi {

// A ragged batch of products of at most Lc limbs in all at one transform
// shape, the largest product's (Lc >= 2), operands of at most longest_a and
// longest_b limbs; workspace: batch_mul_ntt_workspace_size(N,
// Lc - 1, 1).
void ntt_mul_ragged(const NTTPrecomputedTables &tables, uint32_t *ws, const uint32_t *A, const uint32_t *B,
                    uint32_t *C, uint32_t N, const RaggedRow *rows, uint32_t Lc, uint32_t longest_a,
                    uint32_t longest_b) {
    ntt::mul(ntt::make_params(tables), A, B, C, ws, N, Lc - 1u, 1u, 0, 0, 0, rows, longest_a, longest_b);
}

// Transform shape products of La x Lb limbs get (tune table or built-in rule) in
// a large batch.
void ntt_shape_of(uint32_t La, uint32_t Lb, int *log_k, int *M) {
    const ntt::Shape s = ntt::shape_tuned(UINT32_MAX, La, Lb);
    *log_k = s.log_k;
    *M = s.M;
}

SpectrumShape spectrum_shape(uint64_t ncoef) {
    if (ncoef < 2u || ncoef > ((uint64_t)ntt::kMaxCosets << ntt::kMaxLog)) return SpectrumShape{0, 0};
    const ntt::Shape s = ntt::shape_for((uint32_t)ncoef, 1u);
    if (s.log_k <= ntt::kSplitLogC) return SpectrumShape{0, 0};
    return SpectrumShape{s.log_k, s.M};
}

uint64_t spectrum_words(SpectrumShape s, uint32_t N) { return (uint64_t)N * s.M * ntt::kPrimes << s.log_k; }

uint64_t spectrum_flag_words(uint32_t N, uint32_t Lc) {
    return (uint64_t)N * (((uint64_t)Lc + ntt::kCrtSpan - 1) / ntt::kCrtSpan);
}

bool spectrum_sum_fits(const uint32_t *La, const uint32_t *Lb, int terms) {
    // every coefficient of sum_t A_t B_t is below sum_t min(La_t, Lb_t) (2^32 - 1)^2,
    // which must stay below p0 p1 p2 for the CRT to be exact
    unsigned __int128 bound = 0;
    for (int t = 0; t < terms; ++t) {
        const uint64_t m = La[t] < Lb[t] ? La[t] : Lb[t];
        bound += (unsigned __int128)m * 0xffffffffull * 0xffffffffull;
    }
    unsigned __int128 cap = 1;
    for (int q = 0; q < ntt::kPrimes; ++q) cap *= ntt::kP[q];
    return bound < cap;
}

void spectrum_forward(const NTTPrecomputedTables &tables, SpectrumShape s, uint32_t N, const uint32_t *X,
                      uint64_t sX, uint32_t Lx, uint32_t *FX, const uint32_t *Y, uint64_t sY, uint32_t Ly,
                      uint32_t *FY, bool rows) {
    const ntt::NttParams P = ntt::make_params(tables);
    ntt::spectrum_forward(P, ntt::Shape{s.log_k, s.M}, N, X, sX, Lx, FX, Y, sY, Ly, FY, current_stream(), rows);
}

void spectrum_inverse(const NTTPrecomputedTables &tables, SpectrumShape s, uint32_t N, int terms,
                      const uint32_t *const *X, const uint32_t *const *Y, uint32_t *Fout, uint32_t *C, uint64_t sC,
                      uint32_t Lc, uint32_t *flags, bool rows, bool cols, const SpectrumAddend *add) {
    const ntt::NttParams P = ntt::make_params(tables);
    ntt::spectrum_inverse(P, ntt::Shape{s.log_k, s.M}, N, terms, X, Y, Fout, C, sC, Lc, flags, current_stream(),
                          rows, cols, add);
}

void spectrum_inverse_columns(const NTTPrecomputedTables &tables, SpectrumShape s, uint32_t N, uint32_t *F0,
                              uint32_t *F1) {
    ntt::inverse_columns(ntt::make_params(tables), s.log_k, (uint64_t)N * s.M, F0, F1, current_stream());
}

void spectrum_level_rows(const NTTPrecomputedTables &tables, SpectrumShape s, uint32_t N, uint32_t *Fpe,
                         uint32_t *Fpo, uint32_t *Fro, uint32_t *Fqo, uint32_t *Fqe, uint32_t *Fre) {
    const ntt::NttParams P = ntt::make_params(tables);
    cudaStream_t st = current_stream();
    ntt::row_attr();
    const uint64_t VR = (uint64_t)N * s.M;
    const uint64_t segs = VR * ((1ull << s.log_k) >> ntt::kRowLog);
    ntt::RowsLevelArgs a{Fpe, Fpo, Fro, Fqo, Fqe, Fre, s.log_k};
    // six residues read and four written per point, or five and three
    KernelTimed kt("ntt_rows_level", (Fpo ? 40.0 : 32.0) * (double)(1ull << s.log_k) * (double)VR * ntt::kPrimes);
    ntt::k_rows_level<<<ntt::row_grid(segs * ntt::kPrimes), ntt::kRowThreads, ntt::row_smem_bytes(), st>>>(
        P, a, (uint32_t)segs);
    count_launch();
}

}  // namespace gpupi
