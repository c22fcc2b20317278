#pragma once
// Host-side rules of the weight-streaming GEMM for M <= 64 (fp8_gemm_stacked_k.cuh): what a CTA needs, which CTAs share the
// work, where that kernel is the default.  Plain integer arithmetic, so that the rules can be walked without a GPU.

#include <cstdint>

#include "utils.cuh"

namespace yan {

constexpr uint32_t kStackedThreads = 192;

// Tensor memory of a CTA: one accumulator per slot, four where there are six operand slots.
__host__ __device__ constexpr uint32_t stacked_k_tmem_slots(uint32_t slots) { return slots == 6 ? 4 : slots; }
__host__ __device__ constexpr uint32_t stacked_k_tmem_cols(uint32_t m_pad, uint32_t stack, uint32_t slots) {
    return stacked_k_tmem_slots(slots) * stack * m_pad;
}

struct StackedSmem {
    uint32_t off_w, off_x, off_scales, off_exchange, off_barriers, off_tmem_slot, off_abort, total;
};

__host__ __device__ inline StackedSmem stacked_k_smem_layout(uint32_t m_pad, uint32_t stack, uint32_t steps, uint32_t slots,
                                                             uint32_t cluster) {
    StackedSmem s;
    const uint32_t used = steps < slots ? steps : slots;
    const uint32_t sums = 128u * m_pad * 4u;                          // [stack][m_pad][128 / stack] floats
    const uint32_t rings = used * (16384u + stack * m_pad * 128u);
    s.off_w = 0;                                                      // slots x [128 x 128 B]; at the end the sums
    s.off_x = s.off_w + used * 16384u;                                // slots x [stack*m_pad x 128 B]
    s.off_scales = s.off_w + (rings > sums ? rings : sums);           // [stack][steps][m_pad] floats: sA * sB
    s.off_exchange = s.off_scales + stack * steps * m_pad * 4u;       // [cluster - 1][m_pad][128 / stack] floats
    s.off_barriers = align_up(s.off_exchange + (cluster - 1) * m_pad * (128u / stack) * 4u, 8u);
    s.off_tmem_slot = s.off_barriers + 4 * 8u * 8u;  // full, empty, done, tmem_empty: at most 8 of each
    s.off_abort = s.off_tmem_slot + 4;
    s.total = s.off_abort + 4 + 1024;
    return s;
}

__host__ __device__ inline uint32_t stacked_k_steps(uint32_t k, uint32_t stack, uint32_t cluster) {
    return ceil_div(k / kBlockK, stack * cluster);
}

// What a caller may ask for by name (block_n = 2).
inline bool stacked_k_supported(uint32_t m, uint32_t n, uint32_t k) {
    return m >= 1 && m <= 32 && n % 32 == 0 && k % 512 == 0 && k / 512 <= 32;
}

struct StackedConfig {
    uint32_t m_pad, stack, slots, cluster;
};

// Which CTAs share the work (B200, graph of launches over weights that come from HBM, quantizer included, in us):
//   * 32 weight rows per CTA (stack 4) for M <= 16, 64 (stack 2) above: each CTA re-reads all activations.
//   * up to one CTA per SM: as many slots as tensor memory has (M=16 N=4096 K=7168 with 8 slots 11.0, with 4 12.4;
//     M=64 N=7168 K=4096 with 6 operand slots 13.4, with 4 14.8).  More row groups than SMs: 4 slots, two CTAs per SM
//     (M=16 N=7168 K=2048: 7.0; with 8 slots, one CTA per SM and two waves of them: 8.0).  At most four steps: 4 slots as
//     well, the others would never hold anything, and their columns are what a second CTA on the SM would wait for.
//   * a cluster along K where row groups leave SMs idle, as long as it saves every CTA four steps (at least two / four / six / nine
//     saved: M=64 N=1024 K=4096 4.8 / 4.9 / 5.4 / 6.7, M=16 N=1024 K=4096 3.5 / 3.3 / 3.8 / 3.8, M=64 N=2048 K=1024 4.1 / 3.3 / 3.3 /
//     3.3, M=16 N=1024 K=8192 4.4 / 4.4 / 4.7 / 5.4; clusters of eight: M=8 N=528 K=13440 9.2 against 7.4).
//   * clusters of four: as many as can be resident at once.  Where a CTA has an SM to itself that is 33 (132 CTAs: the SMs of a
//     processing cluster are no multiple of four); the others would start when the first have ended (M=64 K=7168: N=2112 8.5,
//     N=2176 14.1 against 10.6 with clusters of two, N=2368 14.4 against 10.7; M=32 N=2304 K=8192 12.8 against 9.3; M=16
//     N=1184 K=16384 12.3 against 9.2).  Where two CTAs fit an SM all of them start at once (M=16 N=1184 K=8192 5.9 against 6.7).
// `num_sms` below `sm_count` is a cap on the CTAs of a launch (the other SMs are somebody else's): M <= 16 then takes the
// twice as wide row groups of M <= 32 where those fit the cap and its own do not.
inline StackedConfig choose_stacked_config(uint32_t m, uint32_t n, uint32_t k, uint32_t num_sms, uint32_t sm_count,
                                           uint32_t max_smem) {
    StackedConfig c;
    c.m_pad = m <= 16 ? 16 : m <= 32 ? 32 : 64;
    if (num_sms > sm_count) num_sms = sm_count;
    if (c.m_pad == 16 && num_sms < sm_count && ceil_div(n, 32u) > num_sms && ceil_div(n, 64u) <= num_sms) c.m_pad = 32;
    c.stack = c.m_pad == 16 ? 4 : 2;
    const uint32_t groups = ceil_div(n, 128u / c.stack);
    for (c.cluster = 1; c.cluster < 4; c.cluster *= 2) {
        const uint32_t next = c.cluster * 2, next_steps = stacked_k_steps(k, c.stack, next);
        if (groups * next > num_sms || stacked_k_steps(k, c.stack, c.cluster) < next_steps + 4) break;
        const bool two_per_sm =
            next_steps <= 4 && 2 * (stacked_k_smem_layout(c.m_pad, c.stack, next_steps, 4, next).total + 1024) <= max_smem + 1024;
        if (next == 4 && groups * next > num_sms * 9 / 10 && !two_per_sm) break;
    }
    const uint32_t steps = stacked_k_steps(k, c.stack, c.cluster);
    c.slots = c.m_pad == 64 ? 6 : groups > num_sms || steps <= 4 ? 4 : 8;
    // the scale table grows with K, the exchange with M and the cluster: where they leave no room, four slots
    if (stacked_k_smem_layout(c.m_pad, c.stack, steps, c.slots, c.cluster).total > max_smem) c.slots = 4;
    return c;
}

// True where this kernel is the default: while all CTAs are resident at once (M=32 N=16384 K=2048 10.9 us against 18.4 with
// the pair kernel, but N=28672 K=1024 14.4 against 12.8 with 256-wide tiles of the general one; M=64 N=9216 K=2048 9.8
// against 12.4, but N=14336 K=1024 15.6 against 9.7), and for M <= 16, where several waves of CTAs hold up against the
// general kernel unless K is long too (N=28672: K=4096 28.0 against 31.0, K=8192 49.1 against 49.0, K=18432 104 against 92).
// Under a cap it is the default only with at most that many CTAs: its grid is not persistent and would spread over all SMs.
inline bool stacked_k_preferred(uint32_t m, uint32_t n, uint32_t k, uint32_t num_sms, uint32_t sm_count, uint32_t max_smem) {
    if (m > 64 || n % 16 != 0 || k % kBlockK != 0) return false;
    const StackedConfig c = choose_stacked_config(m, n, k, num_sms, sm_count, max_smem);
    const uint32_t groups = ceil_div(n, 128u / c.stack), steps = stacked_k_steps(k, c.stack, c.cluster);
    if (num_sms < sm_count ? groups * c.cluster > num_sms
                           : groups > sm_count * (c.m_pad == 64 ? 1 : 2) && (m > 16 || steps > 16))
        return false;
    return stacked_k_smem_layout(c.m_pad, c.stack, steps, c.slots, c.cluster).total <= max_smem;
}

}  // namespace yan
