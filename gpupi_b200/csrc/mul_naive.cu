// Batched schoolbook multiplication (gpupi batch_mul_naive.cu:8-273).
//
// Three shapes:
//   * k_school_rows<MB>: one thread per product for operands of at most 16
//     limbs each (the bottom levels of the splitting tree: 3..16-limb rows in
//     batches of millions), staged through shared memory.
//   * k_school_seg<G>: G = 8, 16 or 32 lanes per product for
//     L_a + L_b <= 4 G (up to 128), carries resolved with one ballot pair.
//   * k_school_cols: one CTA per product, 64-256 threads x 4 consecutive output
//     columns.  Each column sum sum_i a_i b_(k-i) is accumulated exactly in a
//     3-word register with mad.lo.cc / madc.hi.cc / addc (3 instructions per
//     32x32 product), then the 96-bit column sums are carried into limbs with
//     the same chunk/ballot carry as the NTT's CRT stage.  L_a + L_b <= 1024.
// The latter two are IMAD-bound, the first by its staging; algorithmic work =
// L_a * L_b 32x32->64 products.
#include "common.cuh"
#include "carry_tile.cuh"
#include "batch_mul_naive.h"

namespace gpupi {

// d = c + a (b_0 + b_2 2^64 + b_4 2^128 + ...) over 2 P words, dtop = ctop +
// carry: one carry chain of P 64-bit multiply-adds.  c and d may not overlap.
template <int P>
struct MadChain;
template <>
struct MadChain<2> {
    static __device__ __forceinline__ void run(uint32_t a, const uint32_t *b, const uint32_t *c, uint32_t ctop,
                                               uint32_t *d, uint32_t &dtop) {
        asm("mad.lo.cc.u32 %0, %5, %6, %8;\n\t"
            "madc.hi.cc.u32 %1, %5, %6, %9;\n\t"
            "madc.lo.cc.u32 %2, %5, %7, %10;\n\t"
            "madc.hi.cc.u32 %3, %5, %7, %11;\n\t"
            "addc.u32 %4, %12, 0;"
            : "=&r"(d[0]), "=&r"(d[1]), "=&r"(d[2]), "=&r"(d[3]), "=&r"(dtop)
            : "r"(a), "r"(b[0]), "r"(b[2]), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]), "r"(ctop));
    }
};
template <>
struct MadChain<3> {
    static __device__ __forceinline__ void run(uint32_t a, const uint32_t *b, const uint32_t *c, uint32_t ctop,
                                               uint32_t *d, uint32_t &dtop) {
        asm("mad.lo.cc.u32 %0, %7, %8, %11;\n\t"
            "madc.hi.cc.u32 %1, %7, %8, %12;\n\t"
            "madc.lo.cc.u32 %2, %7, %9, %13;\n\t"
            "madc.hi.cc.u32 %3, %7, %9, %14;\n\t"
            "madc.lo.cc.u32 %4, %7, %10, %15;\n\t"
            "madc.hi.cc.u32 %5, %7, %10, %16;\n\t"
            "addc.u32 %6, %17, 0;"
            : "=&r"(d[0]), "=&r"(d[1]), "=&r"(d[2]), "=&r"(d[3]), "=&r"(d[4]), "=&r"(d[5]),
              "=&r"(dtop)
            : "r"(a), "r"(b[0]), "r"(b[2]), "r"(b[4]), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]),
              "r"(c[4]), "r"(c[5]), "r"(ctop));
    }
};
template <>
struct MadChain<4> {
    static __device__ __forceinline__ void run(uint32_t a, const uint32_t *b, const uint32_t *c, uint32_t ctop,
                                               uint32_t *d, uint32_t &dtop) {
        asm("mad.lo.cc.u32 %0, %9, %10, %14;\n\t"
            "madc.hi.cc.u32 %1, %9, %10, %15;\n\t"
            "madc.lo.cc.u32 %2, %9, %11, %16;\n\t"
            "madc.hi.cc.u32 %3, %9, %11, %17;\n\t"
            "madc.lo.cc.u32 %4, %9, %12, %18;\n\t"
            "madc.hi.cc.u32 %5, %9, %12, %19;\n\t"
            "madc.lo.cc.u32 %6, %9, %13, %20;\n\t"
            "madc.hi.cc.u32 %7, %9, %13, %21;\n\t"
            "addc.u32 %8, %22, 0;"
            : "=&r"(d[0]), "=&r"(d[1]), "=&r"(d[2]), "=&r"(d[3]), "=&r"(d[4]), "=&r"(d[5]),
              "=&r"(d[6]), "=&r"(d[7]), "=&r"(dtop)
            : "r"(a), "r"(b[0]), "r"(b[2]), "r"(b[4]), "r"(b[6]), "r"(c[0]), "r"(c[1]), "r"(c[2]),
              "r"(c[3]), "r"(c[4]), "r"(c[5]), "r"(c[6]), "r"(c[7]), "r"(ctop));
    }
};
template <>
struct MadChain<5> {
    static __device__ __forceinline__ void run(uint32_t a, const uint32_t *b, const uint32_t *c, uint32_t ctop,
                                               uint32_t *d, uint32_t &dtop) {
        asm("mad.lo.cc.u32 %0, %11, %12, %17;\n\t"
            "madc.hi.cc.u32 %1, %11, %12, %18;\n\t"
            "madc.lo.cc.u32 %2, %11, %13, %19;\n\t"
            "madc.hi.cc.u32 %3, %11, %13, %20;\n\t"
            "madc.lo.cc.u32 %4, %11, %14, %21;\n\t"
            "madc.hi.cc.u32 %5, %11, %14, %22;\n\t"
            "madc.lo.cc.u32 %6, %11, %15, %23;\n\t"
            "madc.hi.cc.u32 %7, %11, %15, %24;\n\t"
            "madc.lo.cc.u32 %8, %11, %16, %25;\n\t"
            "madc.hi.cc.u32 %9, %11, %16, %26;\n\t"
            "addc.u32 %10, %27, 0;"
            : "=&r"(d[0]), "=&r"(d[1]), "=&r"(d[2]), "=&r"(d[3]), "=&r"(d[4]), "=&r"(d[5]),
              "=&r"(d[6]), "=&r"(d[7]), "=&r"(d[8]), "=&r"(d[9]), "=&r"(dtop)
            : "r"(a), "r"(b[0]), "r"(b[2]), "r"(b[4]), "r"(b[6]), "r"(b[8]), "r"(c[0]), "r"(c[1]),
              "r"(c[2]), "r"(c[3]), "r"(c[4]), "r"(c[5]), "r"(c[6]), "r"(c[7]), "r"(c[8]), "r"(c[9]),
              "r"(ctop));
    }
};
template <>
struct MadChain<6> {
    static __device__ __forceinline__ void run(uint32_t a, const uint32_t *b, const uint32_t *c, uint32_t ctop,
                                               uint32_t *d, uint32_t &dtop) {
        asm("mad.lo.cc.u32 %0, %13, %14, %20;\n\t"
            "madc.hi.cc.u32 %1, %13, %14, %21;\n\t"
            "madc.lo.cc.u32 %2, %13, %15, %22;\n\t"
            "madc.hi.cc.u32 %3, %13, %15, %23;\n\t"
            "madc.lo.cc.u32 %4, %13, %16, %24;\n\t"
            "madc.hi.cc.u32 %5, %13, %16, %25;\n\t"
            "madc.lo.cc.u32 %6, %13, %17, %26;\n\t"
            "madc.hi.cc.u32 %7, %13, %17, %27;\n\t"
            "madc.lo.cc.u32 %8, %13, %18, %28;\n\t"
            "madc.hi.cc.u32 %9, %13, %18, %29;\n\t"
            "madc.lo.cc.u32 %10, %13, %19, %30;\n\t"
            "madc.hi.cc.u32 %11, %13, %19, %31;\n\t"
            "addc.u32 %12, %32, 0;"
            : "=&r"(d[0]), "=&r"(d[1]), "=&r"(d[2]), "=&r"(d[3]), "=&r"(d[4]), "=&r"(d[5]),
              "=&r"(d[6]), "=&r"(d[7]), "=&r"(d[8]), "=&r"(d[9]), "=&r"(d[10]), "=&r"(d[11]),
              "=&r"(dtop)
            : "r"(a), "r"(b[0]), "r"(b[2]), "r"(b[4]), "r"(b[6]), "r"(b[8]), "r"(b[10]), "r"(c[0]),
              "r"(c[1]), "r"(c[2]), "r"(c[3]), "r"(c[4]), "r"(c[5]), "r"(c[6]), "r"(c[7]), "r"(c[8]),
              "r"(c[9]), "r"(c[10]), "r"(c[11]), "r"(ctop));
    }
};
template <>
struct MadChain<7> {
    static __device__ __forceinline__ void run(uint32_t a, const uint32_t *b, const uint32_t *c, uint32_t ctop,
                                               uint32_t *d, uint32_t &dtop) {
        asm("mad.lo.cc.u32 %0, %15, %16, %23;\n\t"
            "madc.hi.cc.u32 %1, %15, %16, %24;\n\t"
            "madc.lo.cc.u32 %2, %15, %17, %25;\n\t"
            "madc.hi.cc.u32 %3, %15, %17, %26;\n\t"
            "madc.lo.cc.u32 %4, %15, %18, %27;\n\t"
            "madc.hi.cc.u32 %5, %15, %18, %28;\n\t"
            "madc.lo.cc.u32 %6, %15, %19, %29;\n\t"
            "madc.hi.cc.u32 %7, %15, %19, %30;\n\t"
            "madc.lo.cc.u32 %8, %15, %20, %31;\n\t"
            "madc.hi.cc.u32 %9, %15, %20, %32;\n\t"
            "madc.lo.cc.u32 %10, %15, %21, %33;\n\t"
            "madc.hi.cc.u32 %11, %15, %21, %34;\n\t"
            "madc.lo.cc.u32 %12, %15, %22, %35;\n\t"
            "madc.hi.cc.u32 %13, %15, %22, %36;\n\t"
            "addc.u32 %14, %37, 0;"
            : "=&r"(d[0]), "=&r"(d[1]), "=&r"(d[2]), "=&r"(d[3]), "=&r"(d[4]), "=&r"(d[5]),
              "=&r"(d[6]), "=&r"(d[7]), "=&r"(d[8]), "=&r"(d[9]), "=&r"(d[10]), "=&r"(d[11]),
              "=&r"(d[12]), "=&r"(d[13]), "=&r"(dtop)
            : "r"(a), "r"(b[0]), "r"(b[2]), "r"(b[4]), "r"(b[6]), "r"(b[8]), "r"(b[10]), "r"(b[12]),
              "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]), "r"(c[4]), "r"(c[5]), "r"(c[6]), "r"(c[7]),
              "r"(c[8]), "r"(c[9]), "r"(c[10]), "r"(c[11]), "r"(c[12]), "r"(c[13]), "r"(ctop));
    }
};
template <>
struct MadChain<8> {
    static __device__ __forceinline__ void run(uint32_t a, const uint32_t *b, const uint32_t *c, uint32_t ctop,
                                               uint32_t *d, uint32_t &dtop) {
        asm("mad.lo.cc.u32 %0, %17, %18, %26;\n\t"
            "madc.hi.cc.u32 %1, %17, %18, %27;\n\t"
            "madc.lo.cc.u32 %2, %17, %19, %28;\n\t"
            "madc.hi.cc.u32 %3, %17, %19, %29;\n\t"
            "madc.lo.cc.u32 %4, %17, %20, %30;\n\t"
            "madc.hi.cc.u32 %5, %17, %20, %31;\n\t"
            "madc.lo.cc.u32 %6, %17, %21, %32;\n\t"
            "madc.hi.cc.u32 %7, %17, %21, %33;\n\t"
            "madc.lo.cc.u32 %8, %17, %22, %34;\n\t"
            "madc.hi.cc.u32 %9, %17, %22, %35;\n\t"
            "madc.lo.cc.u32 %10, %17, %23, %36;\n\t"
            "madc.hi.cc.u32 %11, %17, %23, %37;\n\t"
            "madc.lo.cc.u32 %12, %17, %24, %38;\n\t"
            "madc.hi.cc.u32 %13, %17, %24, %39;\n\t"
            "madc.lo.cc.u32 %14, %17, %25, %40;\n\t"
            "madc.hi.cc.u32 %15, %17, %25, %41;\n\t"
            "addc.u32 %16, %42, 0;"
            : "=&r"(d[0]), "=&r"(d[1]), "=&r"(d[2]), "=&r"(d[3]), "=&r"(d[4]), "=&r"(d[5]),
              "=&r"(d[6]), "=&r"(d[7]), "=&r"(d[8]), "=&r"(d[9]), "=&r"(d[10]), "=&r"(d[11]),
              "=&r"(d[12]), "=&r"(d[13]), "=&r"(d[14]), "=&r"(d[15]), "=&r"(dtop)
            : "r"(a), "r"(b[0]), "r"(b[2]), "r"(b[4]), "r"(b[6]), "r"(b[8]), "r"(b[10]), "r"(b[12]),
              "r"(b[14]), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]), "r"(c[4]), "r"(c[5]), "r"(c[6]),
              "r"(c[7]), "r"(c[8]), "r"(c[9]), "r"(c[10]), "r"(c[11]), "r"(c[12]), "r"(c[13]),
              "r"(c[14]), "r"(c[15]), "r"(ctop));
    }
};

// One thread per product, L_a >= L_b, L_b <= MB (even), L_a <= 16.  The CTA's 128
// rows are staged in shared memory: operands read and products written as
// contiguous runs, each thread working on a row of its own (odd pitch: no bank
// conflicts).  A row holds A, then B; B moves to registers and the product
// replaces A and B from the bottom as A's limbs are used up.
//
// Two limbs of A per step, sums kept in two sets of 64-bit accumulators (E:
// pairs of words at even positions from the step's base, O: at odd ones), so
// that the 2 MB products of a step are four carry chains of 64-bit
// multiply-adds (one instruction each) with no other carry handling; the two
// lowest words are final after the step and the rest moves down by two words
// as the second limb's chains write their results.
// Bound by the staging (one 4-byte copy and one index division per limb, no
// overlap with the arithmetic inside a CTA): 262,144 products of 14 x 13 limbs
// 41.9 -> 26.6 us a call, of which the multiply-adds (half rate: 4 cycles per
// warp and scheduler) take about 5.5 (the previous kernel read and wrote one
// row per thread straight from memory and kept one serial carry chain per limb
// of A).
constexpr int kRowsCta = 128;
constexpr uint32_t kDivShift = 20;   // e / d = e * ceil(2^20 / d) >> 20 for e < 4096, d <= 32

__device__ __forceinline__ void copy_limb(uint32_t *shared, const uint32_t *global) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(shared)),
                 "l"(global)
                 : "memory");
}

template <int MB>
__global__ void __launch_bounds__(kRowsCta) k_school_rows(const uint32_t *__restrict__ A,
                                                          const uint32_t *__restrict__ B, uint32_t *__restrict__ C,
                                                          uint32_t N, uint32_t La, uint32_t Lb, uint64_t sA,
                                                          uint64_t sB, uint64_t sC, uint32_t divA, uint32_t divB,
                                                          uint32_t divC) {
    __shared__ uint32_t sh[kRowsCta * 33];
    const uint32_t Lc = La + Lb;
    const uint32_t pitch = Lc | 1u;
    const uint32_t t = threadIdx.x;
    for (uint64_t r0 = (uint64_t)blockIdx.x * kRowsCta; r0 < N; r0 += (uint64_t)gridDim.x * kRowsCta) {
        const uint32_t rows = (uint32_t)(N - r0 < kRowsCta ? N - r0 : kRowsCta);
        // asynchronous copies: all in flight at once, without registers
#pragma unroll 4
        for (uint32_t e = t; e < rows * La; e += kRowsCta) {
            const uint32_t r = (e * divA) >> kDivShift;
            const uint32_t i = e - r * La;
            copy_limb(sh + r * pitch + i, A + (r0 + r) * sA + i);
        }
#pragma unroll 4
        for (uint32_t e = t; e < rows * Lb; e += kRowsCta) {
            const uint32_t r = (e * divB) >> kDivShift;
            const uint32_t i = e - r * Lb;
            copy_limb(sh + r * pitch + La + i, B + (r0 + r) * sB + i);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        if (t < rows) {
            uint32_t *row = sh + t * pitch;
            uint32_t b[MB];
#pragma unroll
            for (int j = 0; j < MB; ++j) b[j] = (j < (int)Lb) ? row[La + j] : 0u;
            uint32_t e[MB], o[MB];   // o[k] sits at position k + 1
#pragma unroll
            for (int k = 0; k < MB; ++k) e[k] = o[k] = 0u;
            uint64_t cr = 0;
#pragma unroll 1
            for (uint32_t i = 0; i < La; i += 2) {
                const uint32_t a0 = row[i];
                const uint32_t a1 = (i + 1u < La) ? row[i + 1] : 0u;
                uint32_t e1[MB], o1[MB], ec, oc;
                MadChain<MB / 2>::run(a0, b, e, 0u, e1, ec);
                MadChain<MB / 2>::run(a0, b + 1, o, 0u, o1, oc);
                // a1: positions 1 + j; odd j on words 2 .. MB + 1 of E
                uint32_t x[MB], o2[MB], top;
#pragma unroll
                for (int k = 0; k < MB - 2; ++k) x[k] = e1[k + 2];
                x[MB - 2] = ec;
                x[MB - 1] = 0u;
                MadChain<MB / 2>::run(a1, b + 1, x, 0u, e, top);   // no carry out: the sum fits
                MadChain<MB / 2>::run(a1, b, o1, oc, o2, oc);
                uint64_t s = cr + e1[0];
                row[i] = (uint32_t)s;
                s = (s >> 32) + e1[1] + o2[0];
                if (i + 1u < Lc) row[i + 1] = (uint32_t)s;
                cr = (s >> 32) + o2[1];
#pragma unroll
                for (int k = 0; k < MB - 2; ++k) o[k] = o2[k + 2];
                o[MB - 2] = oc;
                o[MB - 1] = 0u;
            }
            const uint32_t base = (La + 1u) & ~1u;
#pragma unroll
            for (int k = 0; k < MB; ++k) {
                const uint64_t s = cr + e[k] + (k ? o[k ? k - 1 : 0] : 0u);
                if (base + k < Lc) row[base + k] = (uint32_t)s;
                cr = s >> 32;
            }
        }
        __syncthreads();
#pragma unroll 4
        for (uint32_t e = t; e < rows * Lc; e += kRowsCta) {
            const uint32_t r = (e * divC) >> kDivShift;
            const uint32_t i = e - r * Lc;
            C[(r0 + r) * sC + i] = sh[r * pitch + i];
        }
        __syncthreads();
    }
}

__device__ __forceinline__ void mac3(uint32_t &c0, uint32_t &c1, uint32_t &c2, uint32_t a, uint32_t b) {
    asm("mad.lo.cc.u32 %0, %3, %4, %0;\n\t"
        "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
        "addc.u32 %2, %2, 0;"
        : "+&r"(c0), "+&r"(c1), "+r"(c2)
        : "r"(a), "r"(b));
}

constexpr int kSchoolV = 4;
constexpr int kSchoolMaxL = 256 * kSchoolV;   // 1024 output limbs

// G lanes per product (G = 8, 16, 32; L_a + L_b <= 4 G): lane l of a group
// owns output columns 4l .. 4l+3, carries between the group's lanes are
// resolved with one ballot pair.  32 / G products per warp, so short
// products (the lower levels of the splitting tree) keep most lanes busy.
constexpr int kSegWarps = 8;   // warps per CTA

template <int G>
__global__ void __launch_bounds__(32 * kSegWarps) k_school_seg(const uint32_t *__restrict__ A,
                                                               const uint32_t *__restrict__ B,
                                                               uint32_t *__restrict__ C, uint32_t N,
                                                               uint32_t La, uint32_t Lb, uint64_t sA,
                                                               uint64_t sB, uint64_t sC) {
    constexpr int PW = 32 / G;                    // products per warp
    constexpr int NP = kSegWarps * PW;            // products per CTA
    // row pitches: 4G + 1 words for A (the groups' broadcast reads of a_i hit
    // different banks), 4G + 13 for B (the groups' windows start in
    // different banks modulo 4)
    __shared__ uint32_t sa[NP][4 * G + 1];
    __shared__ uint32_t sb[NP][4 * G + 13];
    const uint32_t lane = lane_id();
    const uint32_t w = threadIdx.x >> 5;
    const uint32_t grp = lane / G, gl = lane % G;   // group in the warp, lane in the group
    const uint32_t slot = w * PW + grp;
    const uint32_t kPad = La + 4;
    const uint32_t Lc = La + Lb;
    const uint32_t gmask = (G == 32) ? 0xffffffffu : ((1u << G) - 1u);
    // the whole warp runs every iteration (ballots), rows past N compute zeros
    for (uint64_t base = ((uint64_t)blockIdx.x * kSegWarps + w) * PW; base < N;
         base += (uint64_t)gridDim.x * NP) {
        const uint64_t row = base + grp;
        const bool valid = row < N;
        const uint32_t *ar = A + row * sA;
        const uint32_t *br = B + row * sB;
        for (uint32_t i = gl; i < La; i += G) sa[slot][i] = valid ? ar[i] : 0u;
        for (uint32_t j = gl; j < kPad + Lb + 8; j += G)
            sb[slot][j] = (valid && j >= kPad && j - kPad < Lb) ? br[j - kPad] : 0u;
        __syncwarp();
        const uint32_t k0 = gl * kSchoolV;
        uint32_t c[kSchoolV][3];
#pragma unroll
        for (int v = 0; v < kSchoolV; ++v) c[v][0] = c[v][1] = c[v][2] = 0u;
        if (k0 < Lc) {
            const int ilo = max(0, (int)k0 + 1 - (int)Lb);
            const int ihi = min((int)La - 1, (int)k0 + kSchoolV - 1);
            // window bw[v] = b_(k0 + v - i), slid down one word per step of i:
            // one shared-memory load per four products
            const uint32_t *bcol = &sb[slot][kPad + k0];
            uint32_t bw[kSchoolV];
#pragma unroll
            for (int v = 0; v < kSchoolV; ++v) bw[v] = bcol[v - ilo];
            for (int i = ilo; i <= ihi; ++i) {
                const uint32_t ai = sa[slot][i];
#pragma unroll
                for (int v = 0; v < kSchoolV; ++v) mac3(c[v][0], c[v][1], c[v][2], ai, bw[v]);
#pragma unroll
                for (int v = kSchoolV - 1; v > 0; --v) bw[v] = bw[v - 1];
                bw[0] = bcol[-i - 1];
            }
        }
        uint32_t S[kSchoolV + 3];
        chunk_sum3<kSchoolV>(c, S);
        uint32_t H[3];
        H[0] = __shfl_up_sync(0xffffffffu, S[kSchoolV], 1);
        H[1] = __shfl_up_sync(0xffffffffu, S[kSchoolV + 1], 1);
        H[2] = __shfl_up_sync(0xffffffffu, S[kSchoolV + 2], 1);
        if (gl == 0) H[0] = H[1] = H[2] = 0u;
        uint32_t X[kSchoolV];
        const uint32_t g = chunk_add_spill<kSchoolV>(S, H, X);
        bool pp = true;
#pragma unroll
        for (int v = 0; v < kSchoolV; ++v) pp = pp && (X[v] == 0xffffffffu);
        const uint32_t gb = (__ballot_sync(0xffffffffu, g != 0u) >> (grp * G)) & gmask;
        const uint32_t pb = (__ballot_sync(0xffffffffu, pp) >> (grp * G)) & gmask;
        const GroupCarry gc = resolve_group_n(gb, pb, 0u, G);
        chunk_increment<kSchoolV>(X, (gc.carry_in_mask >> gl) & 1u);
        if (valid) {
            uint32_t *cr = C + row * sC;
#pragma unroll
            for (int v = 0; v < kSchoolV; ++v)
                if (k0 + v < Lc) cr[k0 + v] = X[v];
        }
        __syncwarp();
    }
}

template <int G>
static void launch_seg(const uint32_t *A, const uint32_t *B, uint32_t *C, uint32_t N, uint32_t La, uint32_t Lb,
                       uint64_t sA, uint64_t sB, uint64_t sC, cudaStream_t st) {
    constexpr int NP = kSegWarps * (32 / G);
    k_school_seg<G><<<grid_for(N, NP, kNumSMs * 32), 32 * kSegWarps, 0, st>>>(A, B, C, N, La, Lb, sA, sB, sC);
    count_launch();
}

// RAGGED: per-product descriptors (rows) give each product's offsets and
// lengths; otherwise La_u, Lb_u and the strides apply to every row.
template <int kSchoolThreads, bool RAGGED>
__global__ void __launch_bounds__(kSchoolThreads) k_school_cols(const uint32_t *__restrict__ A,
                                                                const uint32_t *__restrict__ B,
                                                                uint32_t *__restrict__ C, uint32_t N,
                                                                uint32_t La_u, uint32_t Lb_u, uint64_t sA,
                                                                uint64_t sB, uint64_t sC,
                                                                const RaggedRow *__restrict__ rows) {
    // a[0..La), bpad[j + kPad] = b_j (zero outside [0, Lb))
    __shared__ uint32_t sa[kSchoolMaxL];
    __shared__ uint32_t sb[kSchoolMaxL + kSchoolMaxL + 8];
    __shared__ uint32_t sg[kSchoolThreads / 32], sp[kSchoolThreads / 32];
    for (uint32_t row = blockIdx.x; row < N; row += gridDim.x) {
        const RaggedRow d = RAGGED ? rows[row] : RaggedRow{row * sA, row * sB, row * sC, La_u, Lb_u};
        const uint32_t La = d.La, Lb = d.Lb;
        const uint32_t kPad = La + 4;
        const uint32_t Lc = La + Lb;
        const uint32_t *ar = A + d.offA;
        const uint32_t *br = B + d.offB;
        for (uint32_t i = threadIdx.x; i < La; i += blockDim.x) sa[i] = ar[i];
        for (uint32_t j = threadIdx.x; j < kPad + Lb + 8; j += blockDim.x)
            sb[j] = (j >= kPad && j - kPad < Lb) ? br[j - kPad] : 0u;
        __syncthreads();
        const uint32_t k0 = threadIdx.x * kSchoolV;
        uint32_t c[kSchoolV][3];
#pragma unroll
        for (int v = 0; v < kSchoolV; ++v) c[v][0] = c[v][1] = c[v][2] = 0u;
        if (k0 < Lc) {
            // terms a_i * b_(k-i) for k in [k0, k0+4): i in [max(0, k0+1-Lb), min(La-1, k0+3)]
            const int ilo = max(0, (int)k0 + 1 - (int)Lb);
            const int ihi = min((int)La - 1, (int)k0 + kSchoolV - 1);
            for (int i = ilo; i <= ihi; ++i) {
                const uint32_t ai = sa[i];
                const uint32_t *bw = sb + kPad + k0 - i;   // bw[v] = b_(k0+v-i)
#pragma unroll
                for (int v = 0; v < kSchoolV; ++v) mac3(c[v][0], c[v][1], c[v][2], ai, bw[v]);
            }
        }
        uint32_t S[kSchoolV + 3];
        chunk_sum3<kSchoolV>(c, S);
        uint32_t H[3];
        H[0] = __shfl_up_sync(0xffffffffu, S[kSchoolV], 1);
        H[1] = __shfl_up_sync(0xffffffffu, S[kSchoolV + 1], 1);
        H[2] = __shfl_up_sync(0xffffffffu, S[kSchoolV + 2], 1);
        __shared__ uint32_t spill[kSchoolThreads / 32][3];
        if (lane_id() == 31) {
            spill[threadIdx.x >> 5][0] = S[kSchoolV];
            spill[threadIdx.x >> 5][1] = S[kSchoolV + 1];
            spill[threadIdx.x >> 5][2] = S[kSchoolV + 2];
        }
        __syncthreads();
        if (lane_id() == 0) {
            const int w = threadIdx.x >> 5;
            H[0] = w ? spill[w - 1][0] : 0u;
            H[1] = w ? spill[w - 1][1] : 0u;
            H[2] = w ? spill[w - 1][2] : 0u;
        }
        uint32_t X[kSchoolV];
        const uint32_t g = chunk_add_spill<kSchoolV>(S, H, X);
        bool p = true;
#pragma unroll
        for (int v = 0; v < kSchoolV; ++v) p = p && (X[v] == 0xffffffffu);
        const BlockCarry bc = block_resolve<kSchoolThreads / 32>(g != 0u, p, sg, sp);
        chunk_increment<kSchoolV>(X, bc.cin);
        uint32_t *cr = C + d.offC;
#pragma unroll
        for (int v = 0; v < kSchoolV; ++v)
            if (k0 + v < Lc) cr[k0 + v] = X[v];
        __syncthreads();
    }
}

template <int MB>
static void launch_rows(const uint32_t *A, const uint32_t *B, uint32_t *C, uint32_t N, uint32_t La, uint32_t Lb,
                        uint64_t sA, uint64_t sB, uint64_t sC, cudaStream_t st) {
    auto div = [](uint32_t d) { return ((1u << kDivShift) + d - 1u) / d; };
    k_school_rows<MB><<<grid_for(N, kRowsCta, kNumSMs * 32), kRowsCta, 0, st>>>(A, B, C, N, La, Lb, sA, sB, sC,
                                                                              div(La), div(Lb), div(La + Lb));
    count_launch();
}

bool school_thread_fits(uint32_t La, uint32_t Lb) {
    return (La <= 16u && Lb <= 16u);
}

void school_mul(const uint32_t *A, const uint32_t *B, uint32_t *C, uint32_t N, uint32_t La,
                uint32_t Lb, uint64_t sA, uint64_t sB, uint64_t sC) {
    cudaStream_t st = current_stream();
    if (N == 0u || La + Lb == 0u) return;
    if (La == 0u || Lb == 0u) {
        cudaMemset2DAsync(C, sC * 4, 0, (size_t)(La + Lb) * 4, N, st);
        return;
    }
    KernelTimed kt("schoolbook", 4.0 * N * (2.0 * (La + Lb)));
    // keep the longer operand as A for the register kernels
    if (La < Lb) {
        std::swap(A, B);
        std::swap(La, Lb);
        std::swap(sA, sB);
    }
    if (La <= 16u) {   // one thread per product; B's registers in steps of two
        switch ((Lb + 1u) / 2u) {
            case 1:
            case 2: launch_rows<4>(A, B, C, N, La, Lb, sA, sB, sC, st); break;
            case 3: launch_rows<6>(A, B, C, N, La, Lb, sA, sB, sC, st); break;
            case 4: launch_rows<8>(A, B, C, N, La, Lb, sA, sB, sC, st); break;
            case 5: launch_rows<10>(A, B, C, N, La, Lb, sA, sB, sC, st); break;
            case 6: launch_rows<12>(A, B, C, N, La, Lb, sA, sB, sC, st); break;
            case 7: launch_rows<14>(A, B, C, N, La, Lb, sA, sB, sC, st); break;
            default: launch_rows<16>(A, B, C, N, La, Lb, sA, sB, sC, st); break;
        }
    } else if (La + Lb <= 32u) {
        launch_seg<8>(A, B, C, N, La, Lb, sA, sB, sC, st);
    } else if (La + Lb <= 64u) {
        launch_seg<16>(A, B, C, N, La, Lb, sA, sB, sC, st);
    } else if (La + Lb <= 128u) {
        launch_seg<32>(A, B, C, N, La, Lb, sA, sB, sC, st);
    } else {
        // one CTA per product, 4 output columns per thread
        const uint32_t g = grid_for(N, 1, kNumSMs * 16);
        if (La + Lb <= 256u)
            k_school_cols<64, false><<<g, 64, 0, st>>>(A, B, C, N, La, Lb, sA, sB, sC, nullptr);
        else if (La + Lb <= 512u)
            k_school_cols<128, false><<<g, 128, 0, st>>>(A, B, C, N, La, Lb, sA, sB, sC, nullptr);
        else
            k_school_cols<256, false><<<g, 256, 0, st>>>(A, B, C, N, La, Lb, sA, sB, sC, nullptr);
        count_launch();
    }
}

// Ragged batch: rows[i] gives the operands' offsets and lengths (L_a >= L_b,
// L_a + L_b <= 1024) and the output offset of product i (L_a + L_b limbs).
void school_mul_ragged(const uint32_t *A, const uint32_t *B, uint32_t *C, uint32_t N, const RaggedRow *rows,
                       uint64_t limb_products) {
    if (N == 0u) return;
    cudaStream_t st = current_stream();
    KernelTimed kt("schoolbook", 8.0 * (double)limb_products);
    k_school_cols<256, true><<<grid_for(N, 1, kNumSMs * 16), 256, 0, st>>>(A, B, C, N, 0u, 0u, 0u, 0u, 0u, rows);
    count_launch();
}

}  // namespace gpupi

void batch_mul_naive(uint32_t *A, uint32_t *B, uint32_t *ret, int N, int L_a, int L_b, int stride_A,
                     int stride_B, int stride_ret) {
    if (N <= 0 || L_a < 0 || L_b < 0 || L_a + L_b > BATCH_MUL_NAIVE_L_MAX) return;
    gpupi::school_mul(A, B, ret, (uint32_t)N, (uint32_t)L_a, (uint32_t)L_b, (uint32_t)stride_A,
                      (uint32_t)stride_B, (uint32_t)stride_ret);
}
