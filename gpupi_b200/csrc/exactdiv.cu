// In-place exact division by an odd 32-bit divisor, modulo 2^(32L)
// (gpupi batch_exactdiv_small.cu:15-141).
//
// Hensel (2-adic) division, least significant limb first:
//   t_i = a_i - c_i;  q_i = t_i * B^-1 mod 2^32;  c_{i+1} = hi(q_i * B) + [a_i < c_i]
// which yields the unique q with q*B == A mod 2^(32L) (the quotient when B | A).
// One thread per row; a warp's 32 rows are staged through shared memory 32
// limbs at a time so that global loads and stores stay coalesced.
#include "common.cuh"
#include "batch_exactdiv_small.h"

namespace gpupi {

constexpr uint32_t kDivRows = 32;   // rows per warp
constexpr uint32_t kDivWarps = 4;

// The next 32 limbs of every row are loaded (32 independent loads per thread)
// while the current ones go through their serial multiply chain.
// 65,536 rows of 102 limbs: 25.5 -> 14.9 us (2 x 26.7 MB), 500,000 rows 130 ->
// 84 us against the kernel below.
__global__ void __launch_bounds__(kDivRows * kDivWarps) exactdiv_kernel(uint32_t *A, uint32_t B,
                                                                      uint32_t Binv, uint32_t N,
                                                                      uint32_t L, uint64_t stride) {
    __shared__ uint32_t tile[kDivWarps][32][33];
    const uint32_t lane = lane_id();
    uint32_t (*tw)[33] = tile[threadIdx.x >> 5];
    for (uint64_t base = ((uint64_t)blockIdx.x * kDivWarps + (threadIdx.x >> 5)) * kDivRows; base < N;
         base += (uint64_t)gridDim.x * kDivWarps * kDivRows) {
        const uint32_t rows = (uint32_t)((N - base) < kDivRows ? (N - base) : kDivRows);
        uint32_t *a0 = A + base * stride + lane;   // lane = limb of the chunk
        uint32_t v[32];
#pragma unroll
        for (uint32_t r = 0; r < 32u; ++r) v[r] = (r < rows && lane < L) ? a0[r * stride] : 0u;
        uint32_t c = 0u;
        for (uint32_t l0 = 0; l0 < L; l0 += 32u) {
#pragma unroll
            for (uint32_t r = 0; r < 32u; ++r) tw[r][lane] = v[r];
            __syncwarp();
#pragma unroll
            for (uint32_t r = 0; r < 32u; ++r)
                v[r] = (r < rows && l0 + 32u + lane < L) ? a0[r * stride + l0 + 32u] : 0u;
            // eight limbs at a time up to the row's last; those past L are zeros
            // and never stored
#pragma unroll
            for (uint32_t k0 = 0; k0 < 32u; k0 += 8u) {
                if (l0 + k0 >= L) break;
#pragma unroll
                for (uint32_t k = k0; k < k0 + 8u; ++k) {
                    const uint32_t a = tw[lane][k];
                    const uint32_t q = (a - c) * Binv;
                    c = __umulhi(q, B) + (a < c ? 1u : 0u);
                    tw[lane][k] = q;
                }
            }
            __syncwarp();
            if (l0 + lane < L) {
#pragma unroll
                for (uint32_t r = 0; r < 32u; ++r)
                    if (r < rows) a0[r * stride + l0] = tw[r][lane];
            }
            __syncwarp();
        }
    }
}

// The same without loads ahead: work for the rows and limbs there are only, and
// registers for more warps per SM.
__global__ void __launch_bounds__(kDivRows * kDivWarps) exactdiv_plain_kernel(uint32_t *A, uint32_t B,
                                                                            uint32_t Binv, uint32_t N,
                                                                            uint32_t L, uint64_t stride) {
    __shared__ uint32_t tile[kDivWarps][32][33];
    const uint32_t lane = lane_id();
    const uint32_t w = threadIdx.x >> 5;
    for (uint64_t base = ((uint64_t)blockIdx.x * kDivWarps + w) * kDivRows; base < N;
         base += (uint64_t)gridDim.x * kDivWarps * kDivRows) {
        const uint32_t rows = (uint32_t)((N - base) < kDivRows ? (N - base) : kDivRows);
        uint32_t c = 0u;
        for (uint32_t l0 = 0; l0 < L; l0 += 32u) {
            const uint32_t len = min(32u, L - l0);
            for (uint32_t r = 0; r < rows; ++r)
                tile[w][r][lane] = (lane < len) ? A[(base + r) * stride + l0 + lane] : 0u;
            __syncwarp();
            if (lane < rows) {
                for (uint32_t k = 0; k < len; ++k) {
                    const uint32_t a = tile[w][lane][k];
                    const uint32_t q = (a - c) * Binv;
                    c = __umulhi(q, B) + (a < c ? 1u : 0u);
                    tile[w][lane][k] = q;
                }
            }
            __syncwarp();
            for (uint32_t r = 0; r < rows; ++r)
                if (lane < len) A[(base + r) * stride + l0 + lane] = tile[w][r][lane];
            __syncwarp();
        }
    }
}

static uint32_t inverse_mod_2_32(uint32_t b) {
    uint32_t x = b;  // correct to 3 bits for odd b
    for (int i = 0; i < 5; ++i) x *= 2u - b * x;
    return x;
}

}  // namespace gpupi

void batch_exactdiv_small(uint32_t *A, uint32_t B, uint32_t N, uint32_t L, uint32_t stride_A) {
    using namespace gpupi;
    if (N == 0u || L == 0u || (B & 1u) == 0u) return;
    const uint32_t binv = inverse_mod_2_32(B);
    const unsigned grid = grid_for(N, kDivRows * kDivWarps, kNumSMs * 8);
    // Measured, loads ahead against plain: one row of 64 limbs 5.1 / 4.1 us, of 128
    // 6.7 / 6.2; three rows of 64 limbs 4.6 / 6.2, of 128 6.7 / 8.2; 32 rows of 28
    // limbs 4.1 / 6.2, of 101 7.3 / 16.4; 500,000 rows of 1 to 28 limbs 18.7 to
    // 24.6 / 14.4 to 22.6, of 40 36.2 / 37.0.
    if (N == 1u || (L <= 32u && N >= (1u << 18)))
        exactdiv_plain_kernel<<<grid, kDivRows * kDivWarps, 0, current_stream()>>>(A, B, binv, N, L, stride_A);
    else
        exactdiv_kernel<<<grid, kDivRows * kDivWarps, 0, current_stream()>>>(A, B, binv, N, L, stride_A);
    GPUPI_LAUNCH_CHECK();
}
