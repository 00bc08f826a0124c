// Ragged batched multiplication: N independent products with per-product
// lengths, one call (no counterpart in the reference, whose batches share one
// L_a / L_b; gpupi's callers with uneven pairs issue one call per pair).
//
// Products are bucketed on the host; every kernel reads its products' offsets
// and lengths from one descriptor array, so operands and products are read and
// written in place:
//   * L_a = 0 or L_b = 0: the L_a + L_b output limbs are zeroed;
//   * products the tune table gives to the CUDA-core schoolbook: one
//     k_school_cols launch; those it gives to the tensor-core schoolbook: one
//     k_mul_tc launch, those that need most shared memory first, so that the
//     last CTAs to finish hold short products.  (Launches of their own for
//     those of less than 112, 56 and 28 KiB, with more CTAs per SM, were faster
//     only for some batches of thousands (4096 products of 300..2000 limbs 214
//     against 222 us, of 100..1300 limbs equal) and slower for all smaller
//     ones, a launch's last wave each: 600 of 200..1400 limbs 42 against 29
//     us, 16 of 64..512 limbs 18.5 against 12.8.)
//   * otherwise by transform size (powers of two up to 2^13 points, quarters of
//     an octave above): one NTT batch per bucket at its largest product's shape.
// 4096 products of 8..4096 limbs per operand: gathering the NTT products into
// padded rows and scattering them back took 104 of 503 us and gave rows of
// 3073..4096 limbs transforms of twice the size.
// The descriptors' device memory comes from the stream's scratch arena.
#include "common.cuh"
#include "batch_arith.h"
#include "batch_mul_ntt.h"

#include <algorithm>
#include <vector>

namespace gpupi {

void school_mul_ragged(const uint32_t *A, const uint32_t *B, uint32_t *C, uint32_t N, const RaggedRow *rows,
                       uint64_t limb_products);
cudaError_t tc_mul_ragged(const uint32_t *A, const uint32_t *B, uint32_t *C, uint32_t n, const RaggedRow *rows,
                          uint32_t maxQ, uint32_t maxN, uint64_t limbs_moved);
void tc_shape(uint32_t La, uint32_t Lb, uint32_t *Q, uint32_t *N);
uint32_t tc_smem_bytes(uint32_t La, uint32_t Lb);
void mul_kinds(uint32_t n, const uint32_t *La, const uint32_t *Lb, uint8_t *kinds);
void ntt_mul_ragged(const NTTPrecomputedTables &tables, uint32_t *ws, const uint32_t *A, const uint32_t *B,
                    uint32_t *C, uint32_t N, const RaggedRow *rows, uint32_t Lc, uint32_t longest_a,
                    uint32_t longest_b);
const NTTPrecomputedTables &context_tables(const BatchMPContext *ctx);
const void *context_workspace(const BatchMPContext *ctx);

namespace {

__global__ void __launch_bounds__(256) k_zero_rows(uint32_t *__restrict__ C, const RaggedRow *__restrict__ rows,
                                                   uint32_t n) {
    for (uint32_t r = blockIdx.x; r < n; r += gridDim.x) {
        const RaggedRow d = rows[r];
        const uint64_t len = (uint64_t)d.La + d.Lb;
        for (uint64_t i = threadIdx.x; i < len; i += blockDim.x) C[d.offC + i] = 0u;
    }
}

unsigned grid_rows(uint32_t n) { return (unsigned)std::max<uint32_t>(1u, std::min<uint32_t>(n, kNumSMs * 16)); }

// Group numbers: zero products, schoolbook, tensor-core products by KiB of
// shared memory from the largest, NTT buckets.
constexpr uint32_t kZero = 0u, kSchoolGroup = 1u, kTensorGroup = 2u;
// Products that need half an SM's shared memory or more (sums above 2560 limbs)
// go to the NTT: one of them would leave the whole launch one CTA per SM.
constexpr uint32_t kTensorMax = 112u;
constexpr uint32_t kNttGroup = kTensorGroup + kTensorMax;
constexpr uint32_t kNttGroups = 4u * 32u;
constexpr uint32_t kGroups = kNttGroup + kNttGroups;

uint32_t ntt_bucket(uint64_t need) {   // 4 ceil(log2 need), less the quarter octaves below above 2^13
    uint32_t k = 0;
    while ((1ull << k) < need) ++k;
    if (k <= 13u) return 4u * k;
    const uint64_t q = 1ull << (k - 3u);   // an eighth of 2^k: quarters of its octave
    const uint32_t below = (uint32_t)(((1ull << k) - need) / q);   // 0 .. 3
    return 4u * k - below;
}

}  // namespace

cudaError_t mul_ragged(BatchMPContext *ctx, uint32_t N, const uint32_t *A, const uint64_t *offA, const uint32_t *La,
                       const uint32_t *B, const uint64_t *offB, const uint32_t *Lb, uint32_t *C,
                       const uint64_t *offC) {
    if (N == 0u) return cudaSuccess;
    if (!ctx || !A || !B || !C || !offA || !La || !offB || !Lb || !offC) return cudaErrorInvalidValue;
    cudaStream_t st = current_stream();
    // counting sort into groups
    std::vector<uint8_t> kind(N);
    mul_kinds(N, La, Lb, kind.data());
    std::vector<uint16_t> group(N);
    std::vector<uint32_t> start(kGroups + 1u, 0u);
    for (uint32_t i = 0; i < N; ++i) {
        const uint64_t Lc = (uint64_t)La[i] + Lb[i];
        if (Lc > (20ull << 25) || std::min(La[i], Lb[i]) > (1u << 28)) return cudaErrorInvalidValue;
        uint32_t g;
        if (La[i] == 0u || Lb[i] == 0u)
            g = kZero;
        else if (kind[i] == 0u)
            g = kSchoolGroup;
        else if (const uint32_t kib = tc_smem_bytes(La[i], Lb[i]) >> 10; kind[i] == 1u && kib < kTensorMax)
            g = kTensorGroup + (kTensorMax - 1u - kib);
        else
            g = kNttGroup + ntt_bucket(Lc - 1u);
        group[i] = (uint16_t)g;
        ++start[g + 1u];
    }
    for (uint32_t g = 0; g < kGroups; ++g) start[g + 1u] += start[g];
    std::vector<RaggedRow> rows(N);
    {
        std::vector<uint32_t> at(start.begin(), start.end() - 1);
        for (uint32_t i = 0; i < N; ++i) rows[at[group[i]]++] = RaggedRow{offA[i], offB[i], offC[i], La[i], Lb[i]};
    }
    // descriptors on the device: those of the schoolbooks first, so that their
    // kernels start while the host stages those of the NTT batches (pageable
    // memory; the device copies them after those kernels)
    auto upload = [&](uint32_t from, uint32_t to, RaggedRow **d) {
        const size_t bytes = (size_t)(to - from) * sizeof(RaggedRow);
        if (!bytes) return cudaSuccess;
        cudaError_t e = scratch_alloc((void **)d, bytes);
        if (e != cudaSuccess) return e;
        note_h2d(bytes);
        return cudaMemcpyAsync(*d, rows.data() + from, bytes, cudaMemcpyHostToDevice, st);
    };
    const uint32_t ntt0 = start[kNttGroup];   // the first NTT product
    RaggedRow *dr = nullptr, *dn = nullptr;
    cudaError_t err = upload(0u, ntt0, &dr);
    const uint32_t nz = start[1], ns = start[2] - start[1];
    if (err == cudaSuccess && nz) {
        k_zero_rows<<<grid_rows(nz), 256, 0, st>>>(C, dr, nz);
        count_launch();
    }
    if (err == cudaSuccess && ns) {
        uint64_t work = 0;
        for (uint32_t i = start[1]; i < start[2]; ++i) work += (uint64_t)rows[i].La * rows[i].Lb;
        school_mul_ragged(A, B, C, ns, dr + start[1], work);
    }
    const uint32_t tc0 = start[kTensorGroup];
    if (err == cudaSuccess && ntt0 > tc0) {
        uint32_t maxQ = 0, maxN = 0;
        uint64_t limbs = 0;
        for (uint32_t i = tc0; i < ntt0; ++i) {
            uint32_t q = 0, n = 0;
            tc_shape(rows[i].La, rows[i].Lb, &q, &n);
            maxQ = std::max(maxQ, q);
            maxN = std::max(maxN, n);
            limbs += 2ull * (rows[i].La + rows[i].Lb);
        }
        err = tc_mul_ragged(A, B, C, ntt0 - tc0, dr + tc0, maxQ, maxN, limbs);
    }
    if (err == cudaSuccess) err = upload(ntt0, N, &dn);
    for (uint32_t g = kNttGroup; err == cudaSuccess && g < kGroups; ++g) {
        const uint32_t n = start[g + 1u] - start[g];
        if (!n) continue;
        uint32_t most = 0, la = 0, lb = 0;
        for (uint32_t i = start[g]; i < start[g + 1u]; ++i) {
            most = std::max(most, rows[i].La + rows[i].Lb);
            la = std::max(la, rows[i].La);
            lb = std::max(lb, rows[i].Lb);
        }
        err = batch_mp_ensure_workspace(ctx, batch_mul_ntt_workspace_size(n, most - 1u, 1u));
        if (err == cudaSuccess)
            ntt_mul_ragged(context_tables(ctx), (uint32_t *)context_workspace(ctx), A, B, C, n, dn + (start[g] - ntt0), most,
                           la, lb);
    }
    if (err == cudaSuccess) err = cudaGetLastError();
    if (dr) scratch_free(dr);
    if (dn) scratch_free(dn);
    return err;
}

}  // namespace gpupi
