#pragma once
// Masked grouped GEMM for groups of at most 128 rows (mixture-of-experts decode): D[g] = A[g][0..masked_m[g]) . B[g]^T.
//
// With few rows per group the weights are all the traffic, and the general kernel spends its time elsewhere: it multiplies
// and loads 128 activation rows per tile whatever the group holds, and its 256-wide tiles leave the last wave nearly empty
// (16 groups x 28 tiles = 3.03 waves).  Here the operands are swapped: 128 weight rows are the UMMA M side and the group's
// rows the N side, rounded up to 16 at run time (the instruction descriptor is built per tile), so that the loads and the
// arithmetic follow masked_m.
//   * persistent, one CTA per SM, tiles = (group, 128 weight columns of D), groups without rows take none;
//   * warp 0: the weights, 16 KB per k-block; warp 2: tensor memory, then the activations, 8 KB per 64 rows (one thread that
//     issued both spent 400 - 570 cycles per k-block on it); warp 1: MMA;
//   * warp 3: the scales.  A column's sA[row] is the same for all lanes of a promotion warp, so a k-block's scales go to shared
//     memory, copied asynchronously up to four k-blocks ahead by one warp; the copies complete the same barrier as the
//     products.  (Loads into registers, however far ahead, held every k-block up for an L2 round trip of 800 cycles: the
//     loads in flight share a few scoreboards, and waiting for the oldest waits for the newest.)
//   * warps 4-11: two promotion warpgroups that share a tile's 16-column chunks alternately; thread = weight row;
//   * output straight from registers: 32 lanes hold 32 consecutive columns of a row, 64 bytes per store instruction.
// What bounds it: HBM (M_max=128, 16 groups of 24 rows, N=7168 K=2048: 57.3 -> 45.0 us, 5.3 TB/s of weights; 24 groups of 8
// rows, N=2048 K=4096: 48.5 -> 38.7), a CTA alone streams at about 500 cycles per k-block of 16 KB.

#include <cstdint>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "fp8_gemm.cuh"

namespace yan {

namespace ptx {
// acc_i = fma(t_i, s_i * scale, acc_i) for two neighbours with two instructions, each rounded like its scalar form.
__device__ __forceinline__ void scaled_fma_f32x2(float& acc0, float& acc1, uint32_t t0, uint32_t t1, float s0, float s1, float scale) {
    asm("{\n\t"
        ".reg .b64 a, t, s, f;\n\t"
        "mov.b64 a, {%0, %1};\n\t"
        "mov.b64 t, {%2, %3};\n\t"
        "mov.b64 s, {%4, %5};\n\t"
        "mov.b64 f, {%6, %6};\n\t"
        "mul.rn.f32x2 s, s, f;\n\t"
        "fma.rn.f32x2 a, t, s, a;\n\t"
        "mov.b64 {%0, %1}, a;\n\t"
        "}\n"
        : "+f"(acc0), "+f"(acc1)
        : "r"(t0), "r"(t1), "f"(s0), "f"(s1), "f"(scale));
}
}  // namespace ptx

constexpr uint32_t kFewRowsThreads = 384;

template <uint32_t kMaxRows>
struct FewRowsSmemLayout {
    static constexpr uint32_t kNumStages = kMaxRows == 64 ? 8 : 6;
    static constexpr uint32_t kNumTmemBufs = 4;
    static constexpr uint32_t kTmemCols = kNumTmemBufs * kMaxRows;
    static constexpr uint32_t kBytesW = 128 * kBlockK, kBytesX = kMaxRows * kBlockK;
    static constexpr uint32_t kOffW = 0;
    static constexpr uint32_t kOffX = kOffW + kNumStages * kBytesW;
    // [kNumScaleSlots][kMaxRows + 4] floats: sA of the rows, then sB.  A slot is rewritten when the accumulator of kNumTmemBufs k-blocks before has been
    // read: every promotion warp is then past the multiply-adds of the k-block before that one.
    static constexpr uint32_t kNumScaleSlots = 2 * kNumTmemBufs, kScaleSlotBytes = (kMaxRows + 4) * 4;
    static constexpr uint32_t kOffScales = kOffX + kNumStages * kBytesX;
    static constexpr uint32_t kOffBarriers = kOffScales + kNumScaleSlots * kScaleSlotBytes;
    static constexpr uint32_t kOffTmemSlot = kOffBarriers + (2 * kNumStages + 2 * kNumTmemBufs) * 8;
    static constexpr uint32_t kOffAbort = kOffTmemSlot + 4;
    static constexpr uint32_t kSmemSize = kOffAbort + 4 + 1024;
    static_assert(kSmemSize <= 232448);
};

// The tiles of one CTA: every group with rows contributes one tile per 128 columns of D.
struct FewRowsWalk {
    const int* masked_m;
    uint32_t num_groups, m_max, tiles_per_group;
    uint32_t next, group = 0, first = 0;  // `first`: index of the first tile of `group`
    uint32_t rows = 0, n_block = 0;

    __device__ __forceinline__ FewRowsWalk(const GemmParams& p)
        : masked_m(p.grouped_layout), num_groups(p.num_groups), m_max(p.shape_m), tiles_per_group(ceil_div(p.shape_n, 128u)),
          next(blockIdx.x) {}

    // Advances to this CTA's next tile; false when there is none.
    __device__ __forceinline__ bool advance() {
        for (; group < num_groups; ++group) {
            // the count lives in device memory where the host cannot check it: clamped to [0, m_max]
            rows = static_cast<uint32_t>(min(max(ptx::ld_global(masked_m + group), 0), static_cast<int>(m_max)));
            const uint32_t tiles = rows == 0 ? 0 : tiles_per_group;
            if (next < first + tiles) {
                n_block = next - first;
                next += gridDim.x;
                return true;
            }
            first += tiles;
        }
        return false;
    }
};

template <uint32_t kMaxRows>
__global__ void __launch_bounds__(kFewRowsThreads, 1)
    fp8_gemm_masked_few_rows_kernel(const GemmParams p, const __grid_constant__ CUtensorMap tensor_map_w,
                                    const __grid_constant__ CUtensorMap tensor_map_x) {
#if defined(__CUDA_ARCH__) && (__CUDA_ARCH__ >= 1000)
    using L = FewRowsSmemLayout<kMaxRows>;
    constexpr uint32_t kNumStages = L::kNumStages, kNumTmemBufs = L::kNumTmemBufs;
    constexpr uint32_t kChunksPerWG = kMaxRows / 32;  // 16-column chunks of a tile: alternately one per warpgroup
    constexpr uint32_t kColsPerWG = kMaxRows / 2;
    const uint32_t num_sb_rows = ceil_div(p.shape_n, 128u);
    static_assert(kMaxRows == 64 || kMaxRows == 128);

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (ptx::smem_u32(smem_raw) & 1023u)) & 1023u);
    uint64_t* full_barriers = reinterpret_cast<uint64_t*>(smem + L::kOffBarriers);
    uint64_t* empty_barriers = full_barriers + kNumStages;
    uint64_t* tmem_full_barriers = empty_barriers + kNumStages;
    uint64_t* tmem_empty_barriers = tmem_full_barriers + kNumTmemBufs;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::kOffTmemSlot);
    volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + L::kOffAbort);

    const uint32_t warp_idx = __shfl_sync(0xffffffffu, threadIdx.x / 32, 0);
    const uint32_t lane_idx = ptx::lane_id();
    const uint32_t num_k_blocks = p.shape_k / kBlockK;

    if (warp_idx == 0 && lane_idx == 0) {
        ptx::tma_prefetch_desc(&tensor_map_w);
        ptx::tma_prefetch_desc(&tensor_map_x);
    }
    if (warp_idx == 1 && lane_idx == 0) {
#pragma unroll
        for (uint32_t i = 0; i < kNumStages; ++i) {
            ptx::mbar_init(full_barriers + i, 2);   // the two producers' arrive.expect_tx
            ptx::mbar_init(empty_barriers + i, 1);  // tcgen05.commit
        }
#pragma unroll
        for (uint32_t i = 0; i < kNumTmemBufs; ++i) {
            ptx::mbar_init(tmem_full_barriers + i, 33);  // tcgen05.commit and the lanes of the scale warp
            ptx::mbar_init(tmem_empty_barriers + i, 8);  // one arrival per promotion warp
        }
        *abort_flag = 0;
        ptx::fence_barrier_init();
        ptx::fence_proxy_async_smem();
    }
    ptx::grid_dependency_wait();  // up to here this kernel may run beside the one in front
    if (warp_idx == 2) {
        ptx::tmem_alloc(tmem_slot, L::kTmemCols);
        ptx::tmem_relinquish_alloc_permit();
    }
    ptx::tcgen05_fence_before_thread_sync();
    __syncthreads();
    ptx::tcgen05_fence_after_thread_sync();
    const uint32_t tmem_base = *tmem_slot;
    FewRowsWalk walk(p);

    if ((warp_idx == 0 || warp_idx == 2) && lane_idx == 0) {
        // ------------------------------ TMA producers: weights (warp 0), activations (warp 2) ------------------------------
        uint32_t stage = 0, phase = 0;
        bool alive = true;
        while (alive && walk.advance()) {
            const int32_t w_row = static_cast<int32_t>(walk.group * p.shape_n + walk.n_block * 128u);
            const int32_t x_row = static_cast<int32_t>(walk.group * p.shape_m);
            const bool two_boxes = kMaxRows == 128 && walk.rows > 64;
            for (uint32_t kb = 0; kb < num_k_blocks; ++kb) {
                if (!detail::bounded_wait(empty_barriers + stage, phase ^ 1, abort_flag, p, 1)) {
                    alive = false;
                    break;
                }
                if (warp_idx == 0) {
                    ptx::mbar_arrive_expect_tx(full_barriers + stage, L::kBytesW);
                    ptx::tma_load_2d(smem + L::kOffW + stage * L::kBytesW, &tensor_map_w, full_barriers + stage,
                                     static_cast<int32_t>(kb * kBlockK), w_row);
                } else {
                    uint8_t* dst = smem + L::kOffX + stage * L::kBytesX;
                    ptx::mbar_arrive_expect_tx(full_barriers + stage, (two_boxes ? 128u : 64u) * kBlockK);
                    ptx::tma_load_2d(dst, &tensor_map_x, full_barriers + stage, static_cast<int32_t>(kb * kBlockK), x_row);
                    if (two_boxes)
                        ptx::tma_load_2d(dst + 64u * kBlockK, &tensor_map_x, full_barriers + stage, static_cast<int32_t>(kb * kBlockK),
                                         x_row + 64);
                }
                if (++stage == kNumStages) {
                    stage = 0;
                    phase ^= 1;
                }
            }
        }
        if (!alive) detail::drain_copies();
    } else if (warp_idx == 1 && lane_idx == 0) {
        // ------------------------------ MMA issuer ------------------------------
        uint32_t stage = 0, phase = 0, buf = 0, buf_phase = 0;
        bool alive = true;
        while (alive && walk.advance()) {
            const uint32_t idesc = make_instr_desc_e4m3_f32(128, ceil_div(walk.rows, 16u) * 16u);
            for (uint32_t kb = 0; kb < num_k_blocks; ++kb) {
                if (!detail::bounded_wait(full_barriers + stage, phase, abort_flag, p, 2) ||
                    !detail::bounded_wait(tmem_empty_barriers + buf, buf_phase ^ 1, abort_flag, p, 3)) {
                    alive = false;
                    break;
                }
                ptx::tcgen05_fence_after_thread_sync();
                const uint64_t w_desc = make_smem_desc_k_major_sw128(ptx::smem_u32(smem + L::kOffW + stage * L::kBytesW));
                const uint64_t x_desc = make_smem_desc_k_major_sw128(ptx::smem_u32(smem + L::kOffX + stage * L::kBytesX));
#pragma unroll
                for (uint32_t k = 0; k < kBlockK / kUmmaK; ++k)
                    ptx::umma_f8f6f4_ss(tmem_base + buf * kMaxRows, w_desc + k * kDescKStep, x_desc + k * kDescKStep, idesc, k > 0);
                ptx::umma_commit(empty_barriers + stage);
                ptx::umma_commit(tmem_full_barriers + buf);
                if (++stage == kNumStages) {
                    stage = 0;
                    phase ^= 1;
                }
                if (++buf == kNumTmemBufs) {
                    buf = 0;
                    buf_phase ^= 1;
                }
            }
        }
    } else if (warp_idx == 3) {
        // ------------------------------ scales ------------------------------
        uint32_t buf = 0, buf_phase = 0, slot = 0;
        bool alive = true;
        const uint32_t s_addr = ptx::smem_u32(smem + L::kOffScales);
        while (alive && walk.advance()) {
            const float* sb_ptr = p.scales_b + (static_cast<size_t>(walk.group) * num_sb_rows + walk.n_block) * num_k_blocks;
            const float* sa_ptr = p.scales_a + static_cast<size_t>(walk.group) * p.shape_m + lane_idx;
            for (uint32_t kb = 0; kb < num_k_blocks; ++kb, ++sb_ptr, sa_ptr += p.sa_ld) {
                const bool ok = detail::bounded_wait(tmem_empty_barriers + buf, buf_phase ^ 1, abort_flag, p, 8);
                if (!__all_sync(0xffffffffu, ok)) {
                    alive = false;
                    break;
                }
                const uint32_t dst = s_addr + slot * L::kScaleSlotBytes;
#pragma unroll
                for (uint32_t i = 0; i < kMaxRows; i += 32u)
                    if (lane_idx + i < walk.rows) ptx::cp_async_4(dst + (lane_idx + i) * 4u, sa_ptr + i);
                if (lane_idx == 0) ptx::cp_async_4(dst + kMaxRows * 4u, sb_ptr);
                ptx::cp_async_mbar_arrive(tmem_full_barriers + buf);
                slot = slot + 1 == L::kNumScaleSlots ? 0 : slot + 1;
                if (++buf == kNumTmemBufs) {
                    buf = 0;
                    buf_phase ^= 1;
                }
            }
        }
        ptx::cp_async_wait_all();
    } else if (warp_idx >= 4) {
        // ------------------------------ promotion + output ------------------------------
        const uint32_t wg = (warp_idx - 4) / 4, quarter = warp_idx % 4;
        const uint32_t tmem_lane_base = tmem_base + ((quarter * 32u) << 16) + wg * 16u;
        const uint32_t s_addr = ptx::smem_u32(smem + L::kOffScales) + wg * 64u;
        uint32_t buf = 0, buf_phase = 0, slot = 0;
        bool alive = true;
        float acc[kColsPerWG];

        while (alive && walk.advance()) {
            const uint32_t rows = walk.rows, chunks = __shfl_sync(0xffffffffu, ceil_div(rows, 16u), 0);
#pragma unroll
            for (uint32_t j = 0; j < kColsPerWG; ++j) acc[j] = 0.0f;

            for (uint32_t kb = 0; kb < num_k_blocks; ++kb) {
                const bool ok = detail::bounded_wait(tmem_full_barriers + buf, buf_phase, abort_flag, p, 4);
                if (!__all_sync(0xffffffffu, ok)) {
                    alive = false;
                    break;
                }
                ptx::tcgen05_fence_after_thread_sync();
                const uint32_t taddr = tmem_lane_base + buf * kMaxRows, scales = s_addr + slot * L::kScaleSlotBytes;
                const float sb = ptx::ld_shared_f32(scales + kMaxRows * 4u - wg * 64u);
                uint32_t t[kChunksPerWG][16];
#pragma unroll
                for (uint32_t i = 0; i < kChunksPerWG; ++i)
                    if (2 * i + wg < chunks) ptx::tmem_ld_32x32b<16>(taddr + i * 32u, t[i]);
#pragma unroll
                for (uint32_t i = 0; i < kChunksPerWG; ++i) ptx::tmem_ld_wait<16>(t[i]);
                ptx::tcgen05_fence_before_thread_sync();
                __syncwarp();
                if (lane_idx == 0) ptx::mbar_arrive(tmem_empty_barriers + buf);
#pragma unroll
                for (uint32_t i = 0; i < kChunksPerWG; ++i) {
                    if (2 * i + wg < chunks) {
                        float4 sc[4];
#pragma unroll
                        for (uint32_t j = 0; j < 4; ++j) sc[j] = ptx::ld_shared_v4_f32(scales + i * 128u + j * 16u);
#pragma unroll
                        for (uint32_t j = 0; j < 4; ++j) {
                            float* a = acc + i * 16 + j * 4;
                            ptx::scaled_fma_f32x2(a[0], a[1], t[i][j * 4], t[i][j * 4 + 1], sc[j].x, sc[j].y, sb);
                            ptx::scaled_fma_f32x2(a[2], a[3], t[i][j * 4 + 2], t[i][j * 4 + 3], sc[j].z, sc[j].w, sb);
                        }
                    }
                }
                slot = slot + 1 == L::kNumScaleSlots ? 0 : slot + 1;
                if (++buf == kNumTmemBufs) {
                    buf = 0;
                    buf_phase ^= 1;
                }
            }
            const uint32_t n = walk.n_block * 128u + quarter * 32u + lane_idx;
            if (alive && n < p.shape_n) {
                __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.out) + static_cast<size_t>(walk.group) * p.shape_m * p.ldd + n;
#pragma unroll
                for (uint32_t i = 0; i < kChunksPerWG; ++i) {
                    const uint32_t row0 = (2 * i + wg) * 16u;
                    if (row0 < rows) {
                        __nv_bfloat16* dst = out + static_cast<size_t>(row0) * p.ldd;
#pragma unroll
                        for (uint32_t j = 0; j < 16; ++j) {
                            if (row0 + j < rows) *dst = __float2bfloat16_rn(acc[i * 16 + j]);
                            dst += p.ldd;
                        }
                    }
                }
            }
        }
    }
    __syncwarp();

    ptx::tcgen05_fence_before_thread_sync();
    __syncthreads();
    if (warp_idx == 2) {
        ptx::tcgen05_fence_after_thread_sync();
        ptx::tmem_dealloc(tmem_base, L::kTmemCols);
    }
#endif
}

template <uint32_t kMaxRows>
inline int launch_masked_few_rows(const GemmArgs& a, cudaStream_t stream) {
    using L = FewRowsSmemLayout<kMaxRows>;
    GemmParams p;
    int max_smem = 0;
    uint64_t a_rows = 0, b_rows = 0;
    const int rc = check_and_fill(a, GemmType::GroupedMasked, sizeof(__nv_bfloat16), L::kSmemSize, p, a_rows, b_rows, max_smem);
    if (rc != kOk) return rc;
    if (a.m > kMaxRows) return kBadArgument;
    bool ok = true;
    const CUtensorMap map_w = make_2d_tma_desc_u8_sw128(a.rhs, b_rows, a.k, a.k, 128, ok);
    const CUtensorMap map_x = make_2d_tma_desc_u8_sw128(a.lhs, a_rows, a.k, a.k, 64, ok);
    if (!ok) return kTensorMapFailed;
    auto kernel = fp8_gemm_masked_few_rows_kernel<kMaxRows>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kSmemSize) != cudaSuccess) {
        cudaGetLastError();
        return kSmemTooLarge;
    }
    // Every CTA the same number of tiles if no group is empty: the weights come as fast to 128 CTAs with 7 tiles each as to 148
    // of which 8 have a seventh, and nothing is left over (16 groups, N=7168).
    const uint64_t tiles = static_cast<uint64_t>(a.num_groups) * ceil_div(a.n, 128u), sms = static_cast<uint64_t>(a.num_sms);
    const uint32_t grid = static_cast<uint32_t>(ceil_div(tiles, ceil_div(tiles, sms)));
    return launch_kernel(kernel, grid, kFewRowsThreads, L::kSmemSize, stream, 1, true, p, map_w, map_x);
}

}  // namespace yan
