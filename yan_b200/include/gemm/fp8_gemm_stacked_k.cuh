#pragma once
// Weight-streaming FP8 GEMM for M <= 64 ("stacked K").
//
// The operands are swapped as in fp8_gemm_small_m.cuh (weight rows on the UMMA M side, activation rows on the N side),
// but a CTA owns only R = 128 / F weight rows (F = kStack = 4, 2 or 1).  The F lane groups of the 128-row MMA operand hold
// the same R weight rows at F different k-blocks, and the activation operand stacks the F matching activation tiles along
// N (here F = 4):
//
//        A operand (128 x 128 B)            B operand (4*M_PAD x 128 B)          D in TMEM (128 lanes x 4*M_PAD cols)
//   rows  0..31 : W[n0.., kb(0,s)]     rows 0..M_PAD-1     : X[.., kb(0,s)]      lanes  0..31, cols 0..M_PAD-1      useful
//   rows 32..63 : W[n0.., kb(1,s)]     rows M_PAD..2M_PAD-1: X[.., kb(1,s)]      lanes 32..63, cols M_PAD..2M_PAD-1 useful
//   ...                                                                           (the off-diagonal blocks are waste)
//
// (F - 1) / F of the MMA work is thrown away, which costs nothing here: the kernel is bound by memory latency and
// bandwidth, the tensor pipe idles.  What it buys is a choice of how many CTAs share the weights, with the k-parts of a
// weight row meeting in ONE CTA: the sum over them is a shared-memory exchange between its four promotion warps.
//
// K is cut into F * cluster parts of `steps` k-blocks (the last ones may be short or empty: their loads are out of bounds
// and read zeros).  A cluster of 2 or 4 CTAs shares the R weight rows when N / R CTAs alone would leave SMs idle; its
// CTAs send their M_PAD x R sums to the first one through distributed shared memory.
//
//   warps 0-3: promotion (thread = TMEM lane = (k-part, weight row)); warp 4: producer; warp 5: tensor memory and MMA.  One elected
//   lane issues all loads, another one all products.
// kSlots step slots of shared memory and kTmemSlots of tensor memory rotate: the loads of step s + kSlots go out as soon as
// the MMAs of step s are complete, the MMAs of step s + kTmemSlots wait until the promotion warps have read the accumulator
// of step s.
// Tensor memory goes back before a CTA waits for the others of its cluster: two CTAs of different clusters on an SM (another
// stream's launch, or this launch's next cluster) may need more columns than there are, and one that kept its own while it
// waited for a CTA that in turn waits for columns elsewhere would close a circle of waits that nothing bounds.
// In front of griddepcontrol.wait a CTA sets up its barriers and asks L2 for its first weights (a hint); it reads nothing, unless the
// caller has promised that weights are constant: then they are loaded there.  Waits are bounded.

#include <cstdint>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "fp8_gemm_small_m.cuh"
#include "stacked_k_plan.h"

namespace yan {

// What may still be running when a CTA of this launch starts (every launch has programmatic stream serialization).
// Tensor memory is taken after the wait for the kernel in front in either case: that kernel, or one that it waits for, may
// still have to take some, and a CTA that held columns while it waits for it would close a circle.
enum StackedOrder : uint32_t {
    kAfterAnyKernel = 0,   // nothing is known: barriers and prefetches, then wait, then everything else
    kConstantWeights = 1,  // any kernel, none of which writes weights (the caller's promise): they are loaded before the wait
};

// Steps whose weights every CTA asks L2 for before it waits (0 / 4, us in a graph over weights from HBM: M=1 N=4096 K=7168 7.6 / 7.0,
// M=16 N=7168 K=2048 5.0 / 4.6, M=64 N=7168 K=2048 6.1 / 5.8, behind a quantizer 6.2 / 5.8 and 7.3 / 6.9; several waves of CTAs:
// M=3 N=16384 K=2048 11.0 / 10.2, M=4 N=28672 K=8192 40.1 / 40.1; fp8_linear M=16 N=2048 K=7168 7.2 / 6.8).  More only fetch twice
// what the loads of a launch of several waves fetch anyway (8 / all: M=4 N=28672 K=8192 42.8 / 45.0).  Leaving it to the CTAs that
// start first gives nothing (fp8_linear M=4 N=28672 K=2048 16.3 against 15.9).
constexpr uint32_t kPrefetchSteps = 4;

// Adds kCols floats of shared memory; false where they come from a thread that gave up.
template <uint32_t kCols>
__device__ __forceinline__ bool add_row_piece(float (&v)[kCols], uint32_t smem_addr) {
    bool complete = true;
#pragma unroll
    for (uint32_t i = 0; i < kCols; i += 4) {
        const float4 t = ptx::ld_shared_v4_f32(smem_addr + i * 4u);
        if (i == 0) complete = detail::is_complete(t.x);
        v[i] += t.x, v[i + 1] += t.y, v[i + 2] += t.z, v[i + 3] += t.w;
    }
    return complete;
}

template <uint32_t M_PAD, uint32_t kStack, uint32_t kSlots, uint32_t kTmemSlots = stacked_k_tmem_slots(kSlots)>
__global__ void __launch_bounds__(kStackedThreads, kTmemSlots * kStack * M_PAD <= 256 ? 2 : 1)
    fp8_gemm_stacked_k_kernel(const GemmParams p, const __grid_constant__ CUtensorMap tensor_map_w,
                              const __grid_constant__ CUtensorMap tensor_map_x, const uint32_t cluster,
                              const uint32_t order) {
#if defined(__CUDA_ARCH__) && (__CUDA_ARCH__ >= 1000)
    constexpr uint32_t kRows = 128 / kStack;       // weight rows of this CTA
    constexpr uint32_t kMmaN = kStack * M_PAD;
    constexpr uint32_t kWarpsPerPart = 4 / kStack;  // promotion warps (of 32 weight rows each) that share a k-part
    constexpr uint32_t kStepBytes = 16384u + kMmaN * 128u;
    constexpr uint32_t kTmemCols = stacked_k_tmem_cols(M_PAD, kStack, kSlots);
    static_assert(M_PAD == 16 || M_PAD == 32 || M_PAD == 64, "activation rows are padded to 16, 32 or 64");
    static_assert(kStack == 1 || kStack == 2 || kStack == 4, "whole lane quarters of the 128-row operand");
    static_assert(kSlots <= 8 && kTmemSlots <= 8, "the issue loops are unrolled over both rings");
    static_assert(kTmemCols == kTmemSlots * kMmaN && kTmemCols <= 512 && (kTmemCols & (kTmemCols - 1)) == 0, "a power of two of at most 512 columns");
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (ptx::smem_u32(smem_raw) & 1023u)) & 1023u);

    const uint32_t warp_idx = __shfl_sync(0xffffffffu, threadIdx.x / 32, 0);
    const uint32_t lane_idx = ptx::lane_id();
    const uint32_t num_k_blocks = p.shape_k / kBlockK;
    const uint32_t steps = ceil_div(num_k_blocks, kStack * cluster);
    const StackedSmem L = stacked_k_smem_layout(M_PAD, kStack, steps, kSlots, cluster);
    uint64_t* full_barriers = reinterpret_cast<uint64_t*>(smem + L.off_barriers);
    // with as many accumulators as operand slots the two are recycled by the same commit
    constexpr bool kOneRing = kSlots == kTmemSlots;
    uint64_t* done_barriers = full_barriers + kSlots;
    uint64_t* empty_barriers = kOneRing ? done_barriers : done_barriers + 2 * kTmemSlots;
    uint64_t* tmem_empty_barriers = done_barriers + kTmemSlots;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L.off_tmem_slot);
    volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + L.off_abort);
    float* s_scales = reinterpret_cast<float*>(smem + L.off_scales);
    float* s_reduce = reinterpret_cast<float*>(smem + L.off_w);

    const uint32_t rank = blockIdx.x % cluster;  // = the CTA's rank in its (one-dimensional) cluster
    const uint32_t n0 = blockIdx.x / cluster * kRows;
    // k-block of (k-part q, step s): (part0 + q) * steps + s
    const uint32_t part0 = rank * kStack;

    if (cluster > 1) ptx::cluster_arrive();  // waited for in front of the exchange: by then every CTA of it has started
    if (order == kConstantWeights) ptx::grid_dependency_launch_dependents();
    if (warp_idx < 4 && order == kAfterAnyKernel) {
        // the first weights on their way to L2 while the kernel in front ends: thread = (k-part, row) of a step
        const uint32_t r = threadIdx.x % kRows, kb = (part0 + threadIdx.x / kRows) * steps;
        const uint8_t* w = p.weights + static_cast<size_t>(n0 + r) * p.shape_k + kb * kBlockK;
        if (n0 + r < p.shape_n)
            for (uint32_t s = 0; s < steps && s < kPrefetchSteps && kb + s < num_k_blocks; ++s) ptx::prefetch_l2(w + s * kBlockK);
    }
    if (warp_idx == 5) {
        // First thing: an SM does not start its second CTA before the first one has given up the permit to allocate
        // (CTAs 148.. of a 224-CTA grid started 2.0 us late when the allocation followed the activations' loads:
        // M=16 N=7168 K=2048 with its quantizer 8.1 -> 7.0 us).
        ptx::grid_dependency_wait();
        ptx::tmem_alloc(tmem_slot, kTmemCols);
        ptx::tmem_relinquish_alloc_permit();
        // the kernel behind this one may start: its own allocation cannot get in front of this grid's any more
        if (order != kConstantWeights) ptx::grid_dependency_launch_dependents();
    }
    // the operands of step s, slot by slot: a box per k-part
    auto load_weights = [&](const uint32_t slot, const uint32_t s) {
        ptx::mbar_arrive_expect_tx(full_barriers + slot, kStepBytes);
#pragma unroll
        for (uint32_t part = 0; part < kStack; ++part)
            ptx::tma_load_2d(smem + L.off_w + slot * 16384u + part * (kRows * 128u), &tensor_map_w, full_barriers + slot,
                             static_cast<int32_t>(((part0 + part) * steps + s) * kBlockK), static_cast<int32_t>(n0));
    };
    auto load_activations = [&](const uint32_t slot, const uint32_t s) {
#pragma unroll
        for (uint32_t part = 0; part < kStack; ++part)
            ptx::tma_load_2d(smem + L.off_x + slot * (kMmaN * 128u) + part * (M_PAD * 128u), &tensor_map_x, full_barriers + slot,
                             static_cast<int32_t>(((part0 + part) * steps + s) * kBlockK), 0);
    };
    if (warp_idx == 4) {
        if (lane_idx == 0) {
            ptx::tma_prefetch_desc(&tensor_map_w);
            ptx::tma_prefetch_desc(&tensor_map_x);
#pragma unroll
            for (uint32_t r = 0; r < kSlots; ++r) {
                ptx::mbar_init(full_barriers + r, 1);   // the producer's arrive.expect_tx
                if (!kOneRing) ptx::mbar_init(empty_barriers + r, 1);  // tcgen05.commit: the slot may be refilled
            }
#pragma unroll
            for (uint32_t b = 0; b < kTmemSlots; ++b) {
                ptx::mbar_init(done_barriers + b, 1);        // tcgen05.commit: the accumulator is complete
                ptx::mbar_init(tmem_empty_barriers + b, 4);  // one arrival per promotion warp
            }
            *abort_flag = 0;
            ptx::fence_barrier_init();
            ptx::fence_proxy_async_smem();
        }
        __syncwarp();
        if (order == kAfterAnyKernel) ptx::grid_dependency_wait();
        if (ptx::elect_one()) {
#pragma unroll
            for (uint32_t slot = 0; slot < kSlots; ++slot)
                if (slot < steps) load_weights(slot, slot);
        }
        __syncwarp();
    }
    ptx::tcgen05_fence_before_thread_sync();
    __syncthreads();  // barriers and the tensor memory address exist
    ptx::tcgen05_fence_after_thread_sync();
    const uint32_t tmem_base = *tmem_slot;

    if (warp_idx == 4) {
        ptx::grid_dependency_wait();
        if (ptx::elect_one()) {
#pragma unroll
            for (uint32_t slot = 0; slot < kSlots; ++slot)
                if (slot < steps) load_activations(slot, slot);
            // refills: the slot is free again when the MMAs of the step it held are complete
            uint32_t pos = 0, phase = 0, s = kSlots;
            if (steps > kSlots)
                ring_steps<kSlots>(pos, steps - kSlots, [&](const uint32_t slot) {
                    if (!detail::bounded_wait(empty_barriers + slot, phase, abort_flag, p, 7)) return false;
                    load_weights(slot, s);
                    load_activations(slot, s);
                    ++s;
                    if (slot + 1 == kSlots) phase ^= 1;
                    return true;
                });
        }
        __syncwarp();
    } else if (warp_idx == 5) {
        if (ptx::elect_one()) {
            constexpr uint32_t idesc = make_instr_desc_e4m3_f32(128, kMmaN);
            const uint32_t w_low = make_smem_desc_low(ptx::smem_u32(smem + L.off_w)), x_low = make_smem_desc_low(ptx::smem_u32(smem + L.off_x));
            uint32_t pos = 0, phase = 0, buf_phase = 0, left = steps;
            ring_steps<common_round(kSlots, kTmemSlots)>(pos, steps, [&](const uint32_t u) {
                const uint32_t r = u % kSlots, b = u % kTmemSlots;
                if (!detail::bounded_wait(full_barriers + r, phase, abort_flag, p, 5)) return false;
                if (!detail::bounded_wait(tmem_empty_barriers + b, buf_phase ^ 1, abort_flag, p, 8)) return false;
                ptx::tcgen05_fence_after_thread_sync();
                umma_k_block(tmem_base + b * kMmaN, w_low + r * (16384u >> 4), x_low + r * (kMmaN * 128u >> 4), idesc);
                ptx::umma_commit(done_barriers + b);
                if (!kOneRing && left > kSlots) ptx::umma_commit(empty_barriers + r);
                --left;
                if (r + 1 == kSlots) phase ^= 1;
                if (b + 1 == kTmemSlots) buf_phase ^= 1;
                return true;
            });
        }
        __syncwarp();
        // the promotion warps have read the last accumulator, or a role gave up: then loads and products may be in flight
        ptx::named_barrier_sync(2, 160);
        if (*abort_flag != 0) detail::drain_copies();
        ptx::tcgen05_fence_after_thread_sync();
        ptx::tmem_dealloc(tmem_base, kTmemCols);
    }

    // Promotion warps: TMEM lane 32 * warp + lane = (k-part q, weight row n0 + r)
    const uint32_t q = warp_idx / kWarpsPerPart, r_local = (warp_idx % kWarpsPerPart) * 32 + lane_idx;
    // The final sums: an item is kCols neighbouring columns of one activation row, so that a row leaves in whole pieces of 64
    // or 128 bytes (a thread that finished a column stored 2 bytes of every row: M=64 N=7168 K=2048 1.05 us for 64 x 64 values).
    constexpr uint32_t kCols = M_PAD == 16 ? 4 : 8, kItems = M_PAD * (kRows / kCols) / 128;
    const uint32_t m_first = threadIdx.x / (kRows / kCols), col = threadIdx.x % (kRows / kCols) * kCols;
    constexpr uint32_t kItemRows = 128 / (kRows / kCols);  // item j of a thread: activation row m_first + j * kItemRows
    float v[kItems][kCols];
    bool alive = true;
    if (warp_idx < 4) {
        // Fold both scale factors of every (k-part, step, row) while the weights stream in.
        const float* sb_ptr = p.scales_b + static_cast<size_t>(n0 / 128u) * num_k_blocks;
        ptx::grid_dependency_wait();
        // eight of each in flight: one after the other they took longer than the weights (M=1 N=4096 K=7168: 1.3 us behind them)
        const uint32_t num_scales = kStack * steps * M_PAD;
        for (uint32_t first = threadIdx.x; first < num_scales; first += 8 * 128) {
            float sa[8], sb[8];
#pragma unroll
            for (uint32_t j = 0; j < 8; ++j) {
                const uint32_t i = first + j * 128, m = i % M_PAD, kb = part0 * steps + i / M_PAD;
                const bool ok = i < num_scales && m < p.shape_m && kb < num_k_blocks;
                sa[j] = ok ? ptx::ld_global(p.scales_a + static_cast<size_t>(kb) * p.sa_ld + m) : 0.0f;
                sb[j] = ok ? ptx::ld_global(sb_ptr + kb) : 0.0f;
            }
#pragma unroll
            for (uint32_t j = 0; j < 8; ++j)
                if (first + j * 128 < num_scales) s_scales[first + j * 128] = sa[j] * sb[j];
        }
        ptx::named_barrier_sync(1, 128);
        // the useful columns of a step are [slot * kMmaN + q * M_PAD, +M_PAD)
        const uint32_t taddr = tmem_base + ((warp_idx * 32u) << 16) + q * M_PAD;
        constexpr uint32_t kChunk = M_PAD < 32 ? M_PAD : 32;
        float acc[M_PAD];
#pragma unroll
        for (uint32_t m = 0; m < M_PAD; ++m) acc[m] = 0.0f;
        for (uint32_t s = 0; s < steps && alive; ++s) {
            const uint32_t b = s % kTmemSlots;
            const bool ok = detail::bounded_wait(done_barriers + b, (s / kTmemSlots) & 1, abort_flag, p, 6);
            alive = __all_sync(0xffffffffu, ok);
            if (alive) {
                ptx::tcgen05_fence_after_thread_sync();
                const uint32_t sc = ptx::smem_u32(s_scales) + (q * steps + s) * (M_PAD * 4u);
#pragma unroll
                for (uint32_t c = 0; c < M_PAD / kChunk; ++c) {
                    uint32_t t[kChunk];
                    ptx::tmem_ld_32x32b<kChunk>(taddr + b * kMmaN + c * kChunk, t);
                    ptx::tmem_ld_wait<kChunk>(t);
                    if (c + 1 == M_PAD / kChunk) {
                        ptx::tcgen05_fence_before_thread_sync();
                        __syncwarp();
                        if (lane_idx == 0) ptx::mbar_arrive(tmem_empty_barriers + b);  // the accumulator slot may be overwritten
                    }
#pragma unroll
                    for (uint32_t m = 0; m < kChunk; m += 4) {
                        const float4 f = ptx::ld_shared_v4_f32(sc + (c * kChunk + m) * 4u);
                        float* a = acc + c * kChunk + m;
                        ptx::fma_f32x2(a[0], a[1], t[m], t[m + 1], f.x, f.y);
                        ptx::fma_f32x2(a[2], a[3], t[m + 2], t[m + 3], f.z, f.w);
                    }
                }
            }
        }
        ptx::tcgen05_fence_before_thread_sync();
        ptx::named_barrier_arrive(2, 160);
        // The k-parts of a weight row sit in different warps: exchange through shared memory, [q][m][r], in the weight slots,
        // which are dead once every warp has seen the last step's MMAs complete.
        ptx::named_barrier_sync(1, 128);
#pragma unroll
        for (uint32_t m = 0; m < M_PAD; ++m) s_reduce[(q * M_PAD + m) * kRows + r_local] = acc[m];
        ptx::named_barrier_sync(1, 128);
        if (rank == 0) {
            const uint32_t base = ptx::smem_u32(s_reduce) + (m_first * kRows + col) * 4u;
#pragma unroll
            for (uint32_t j = 0; j < kItems; ++j) {
#pragma unroll
                for (uint32_t i = 0; i < kCols; ++i) v[j][i] = 0.0f;
#pragma unroll
                for (uint32_t qq = 0; qq < kStack; ++qq)
                    add_row_piece(v[j], base + (qq * M_PAD + j * kItemRows) * (kRows * 4u));
            }
        }
    }
    if (cluster > 1) {
        __syncwarp();
        ptx::cluster_wait();
        if (warp_idx < 4 && rank != 0) {
            // a warp sends 128 contiguous bytes at a time (16 per lane were slower: M=32 N=2048 K=7168 7.85 us against 7.3)
            const bool gave_up = *abort_flag != 0;
            const uint32_t base = ptx::smem_u32(s_reduce) + threadIdx.x * 4u;
            const uint32_t remote = ptx::map_to_cta(ptx::smem_u32(smem + L.off_exchange) + (rank - 1) * (M_PAD * kRows * 4u), 0) + threadIdx.x * 4u;
#pragma unroll
            for (uint32_t j = 0; j < M_PAD * kRows / 128; ++j) {
                float sum = 0.0f;
#pragma unroll
                for (uint32_t qq = 0; qq < kStack; ++qq) sum += ptx::ld_shared_f32(base + (qq * M_PAD * kRows + j * 128u) * 4u);
                ptx::st_cluster_f32(remote + j * 512u, gave_up ? __uint_as_float(detail::kGaveUpSum) : sum);
            }
        }
        ptx::cluster_arrive();
        ptx::cluster_wait();
    }
    if (warp_idx < 4 && rank == 0 && alive && *abort_flag == 0) {
        const uint32_t exchange = ptx::smem_u32(smem + L.off_exchange) + (m_first * kRows + col) * 4u;
        for (uint32_t c = 0; c + 1 < cluster; ++c) {
#pragma unroll
            for (uint32_t j = 0; j < kItems; ++j)
                alive = add_row_piece(v[j], exchange + (c * M_PAD + j * kItemRows) * (kRows * 4u)) && alive;
        }
        if (alive && n0 + col < p.shape_n) {  // N % 16 == 0: a piece is inside or outside as a whole
            __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.out) + static_cast<size_t>(m_first) * p.ldd + n0 + col;
            const bool whole = reinterpret_cast<uintptr_t>(p.out) % 16 == 0 && p.ldd % 8 == 0;
#pragma unroll
            for (uint32_t j = 0; j < kItems; ++j, out += static_cast<size_t>(kItemRows) * p.ldd) {
                if (m_first + j * kItemRows >= p.shape_m) break;
                uint32_t w[kCols / 2];
#pragma unroll
                for (uint32_t i = 0; i < kCols / 2; ++i) {
                    const __nv_bfloat162 t = __floats2bfloat162_rn(v[j][2 * i], v[j][2 * i + 1]);
                    w[i] = *reinterpret_cast<const uint32_t*>(&t);
                }
                if (whole) {
                    if constexpr (kCols == 8) *reinterpret_cast<uint4*>(out) = make_uint4(w[0], w[1], w[2], w[3]);
                    else *reinterpret_cast<uint2*>(out) = make_uint2(w[0], w[1]);
                } else {  // an output that is only known to start on an element
#pragma unroll
                    for (uint32_t i = 0; i < kCols; ++i) out[i] = __float2bfloat16_rn(v[j][i]);
                }
            }
        }
    }
#endif
}

template <uint32_t M_PAD, uint32_t kStack, uint32_t kSlots>
inline int launch_stacked_k_instance(const GemmParams& p, const CUtensorMap& map_w, const CUtensorMap& map_x,
                                     uint32_t cluster, cudaStream_t stream, StackedOrder order) {
    auto kernel = fp8_gemm_stacked_k_kernel<M_PAD, kStack, kSlots>;
    const uint32_t smem_bytes = stacked_k_smem_layout(M_PAD, kStack, stacked_k_steps(p.shape_k, kStack, cluster), kSlots, cluster).total;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes) != cudaSuccess) {
        cudaGetLastError();
        return kSmemTooLarge;
    }
    return launch_kernel(kernel, ceil_div(p.shape_n, 128 / kStack) * cluster, kStackedThreads, smem_bytes, stream, cluster, true, p, map_w,
                         map_x, cluster, static_cast<uint32_t>(order));
}

// Host launcher.  Arguments as GemmLauncher::launch (Normal GEMM, bf16 output).
inline int launch_fp8_gemm_stacked_k(const GemmArgs& a, cudaStream_t stream, StackedOrder order) {
    if (a.lhs == nullptr || a.lhs_scales == nullptr || a.rhs == nullptr || a.rhs_scales == nullptr || a.out == nullptr)
        return kBadArgument;
    if (a.ldd < a.n || a.lhs_scales_ld < a.m || a.m > 64 || a.n % 16 != 0 || a.k % kBlockK != 0) return kBadArgument;
    if (!is_aligned(a.lhs, 16) || !is_aligned(a.rhs, 16) || !is_aligned(a.out, 2)) return kBadArgument;
    int device = 0, sm_count = 0, max_smem = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return kLaunchFailed;
    cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, device);
    cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    const StackedConfig c = choose_stacked_config(a.m, a.n, a.k, static_cast<uint32_t>(a.num_sms), static_cast<uint32_t>(sm_count),
                                                  static_cast<uint32_t>(max_smem));

    bool ok = true;
    const CUtensorMap map_w = make_2d_tma_desc_u8_sw128(a.rhs, a.n, a.k, a.k, 128 / c.stack, ok);
    const CUtensorMap map_x = make_2d_tma_desc_u8_sw128(a.lhs, a.m, a.k, a.k, c.m_pad, ok);
    if (!ok) return kTensorMapFailed;

    GemmParams p;
    p.scales_a = a.lhs_scales;
    p.scales_b = a.rhs_scales;
    p.grouped_layout = nullptr;
    p.weights = static_cast<const uint8_t*>(a.rhs);
    p.out = a.out;
    p.out_scales = nullptr;
    p.out_scales_ld = 0;
    p.sa_ld = a.lhs_scales_ld;
    p.ldd = a.ldd;
    p.shape_m = a.m;
    p.shape_n = a.n;
    p.shape_k = a.k;
    p.num_groups = 1;
    p.status = a.status;
    p.timeout_ns = a.timeout_ns;
    if (c.m_pad == 16) {
        if (c.slots == 8) return launch_stacked_k_instance<16, 4, 8>(p, map_w, map_x, c.cluster, stream, order);
        return launch_stacked_k_instance<16, 4, 4>(p, map_w, map_x, c.cluster, stream, order);
    }
    if (c.m_pad == 32) {
        if (c.slots == 8) return launch_stacked_k_instance<32, 2, 8>(p, map_w, map_x, c.cluster, stream, order);
        return launch_stacked_k_instance<32, 2, 4>(p, map_w, map_x, c.cluster, stream, order);
    }
    if (c.slots == 4) return launch_stacked_k_instance<64, 2, 4>(p, map_w, map_x, c.cluster, stream, order);
    return launch_stacked_k_instance<64, 2, 6>(p, map_w, map_x, c.cluster, stream, order);
}

}  // namespace yan
