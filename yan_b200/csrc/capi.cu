// C ABI of the FP8 fine-grained-scaled GEMM path (declarations and layouts: include/yan_b200.h).
// Every entry point validates on the host, enqueues on the caller's stream and reports through
// `return_code`; nothing allocates, frees or synchronises (except the explicit status read).

#include <cstdint>
#include <cstring>
#include <cuda.h>
#include <cuda_runtime.h>

#include "../../include/yan_b200.h"
#include "gemm_dispatch.h"
#include "launch_order.h"
#include "gemm/fp8_gemm_masked_few_rows.cuh"
#include "gemm/fp8_gemm_small_m.cuh"
#include "gemm/fp8_gemm_stacked_k.cuh"
#include "comm/peer_allreduce.cuh"
#include "quant/fp8_cast.cuh"

namespace {

// One status word per device image of this library; kernels report bounded-wait expiry here.
__device__ int g_status_word = 0;

unsigned long long g_timeout_ns = 2000000000ull;
// The waits between ranks have a bound of their own: ranks of one job drift apart by seconds for ordinary reasons
// (first-call module loading, a garbage collection, a stalled data loader), which no wait inside one kernel does.
unsigned long long g_collective_timeout_ns = 10000000000ull;
yan::ConstantWeights g_constant_weights;
long long* g_clock_probe = nullptr;

constexpr int kMaxDevices = 64;
int* g_status_ptr[kMaxDevices] = {};

int* status_word_of_current_device() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
    if (g_status_ptr[dev] == nullptr) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_status_word) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        g_status_ptr[dev] = static_cast<int*>(p);
    }
    return g_status_ptr[dev];
}

// Scratch of the allocation-free entry point: quantized activations followed by their scales.
// Every device that loads this library holds these bytes until the process exits.
constexpr size_t kStaticScratchQBytes = YAN_B200_STATIC_SCRATCH_MAX_ELEMENTS;  // one byte per element
constexpr size_t kStaticScratchScaleBytes = kStaticScratchQBytes / 128 * sizeof(float);
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchQBytes + kStaticScratchScaleBytes];

unsigned char* g_static_scratch_ptr[kMaxDevices] = {};

// In host code `g_static_scratch` is only a handle; the device address has to be asked for, once per
// device, with that device current.
unsigned char* static_scratch_of_current_device() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
    if (g_static_scratch_ptr[dev] == nullptr) {
        unsigned char* p = nullptr;
        if (cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_static_scratch) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        g_static_scratch_ptr[dev] = p;
    }
    return g_static_scratch_ptr[dev];
}

// Diagnostic kernel: one thread waits, with the same bounded wait the GEMMs use, on an mbarrier that nothing
// ever arrives on.  The wait runs out, the status word is written, the kernel returns.
__global__ void wait_probe_kernel(yan::GemmParams p) {
    __shared__ uint64_t bar;
    __shared__ uint32_t abort_flag;
    if (threadIdx.x == 0) {
        yan::ptx::mbar_init(&bar, 1);
        abort_flag = 0;
        yan::ptx::fence_barrier_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) yan::detail::bounded_wait(&bar, 0, &abort_flag, p, 15);
    __syncthreads();
}

yan::LaunchPlace launch_place(void* stream) {
    yan::LaunchPlace place;
    place.era = g_constant_weights.era();
    place.stream = stream;
    if (!yan::ConstantWeights::promised(place.era)) return place;
    cudaStreamCaptureStatus status;
    // the handle of the per-thread default stream is the same for every thread
    place.known = static_cast<cudaStream_t>(stream) != cudaStreamPerThread && cudaGetDevice(&place.device) == cudaSuccess &&
                  cudaStreamGetCaptureInfo_v2(static_cast<cudaStream_t>(stream), &status, &place.capture) == cudaSuccess;
    if (!place.known) cudaGetLastError();
    else if (status == cudaStreamCaptureStatusNone) place.capture = 0;
    return place;
}

inline void set_rc(int* rc, int v) {
    if (rc != nullptr) *rc = v;
}

// Picks BLOCK_N by a wave model: time = start + waves * (k-blocks * per_kb + epilogue), in us, fitted to graph timings on B200
// (37 tile rows, 1 to 5 full waves, K = 512 to 6144; within 6 %; 224 and 160 made slower, as they are in long runs).  A narrower
// tile is far from proportionally cheaper: the promotion of a k-block has a large fixed part, the widths without shared-memory
// room for the staged epilogue (224, 160, 96) or with a second B scale and a 16-column tail chunk pay for that; but with four
// accumulators instead of two its epilogue hides better.  Large problems therefore get 256; narrower tiles win when they fill
// the machine better or K is short.
// (The issue loop of the narrow tiles and the overlapped launches have since taken up to 0.03 us per k-block and a microsecond of the
// start off; over 57 random shapes of 65 to 4096 rows the choice is within 2 % of the best width.)
// `time_out`, when given, receives the winner's time.
int choose_block_n(int m, int n, int k, int num_sms, bool can_cut_tail, double* time_out = nullptr) {
    static const struct { int bn; double start, per_kb, epilogue; } candidates[8] = {
        {256, 3.15, 0.426, 2.02}, {224, 4.19, 0.470, 3.54}, {192, 3.14, 0.351, 1.66}, {160, 3.28, 0.330, 2.60},
        {128, 3.76, 0.254, 0.89}, {96, 3.80, 0.257, 1.49},  {64, 3.44, 0.215, 0.48},  {32, 3.29, 0.209, 0.41}};
    int best = 256;
    double best_time = -1.0;
    for (const auto& c : candidates) {
        if (c.bn > 32 && n < c.bn) continue;
        const long tiles = static_cast<long>((m + 127) / 128) * ((n + c.bn - 1) / c.bn);
        double waves = static_cast<double>((tiles + num_sms - 1) / num_sms);
        // with scratch for partial tiles the rest of a nearly empty last wave is cut along K (about a third of a wave)
        if (can_cut_tail && (c.bn == 256 || c.bn == 128 || c.bn == 64) &&
            yan::choose_tail_slices(static_cast<uint32_t>(tiles), static_cast<uint32_t>(num_sms), static_cast<uint32_t>(k / 128)) != 0)
            waves = static_cast<double>(tiles / num_sms) + 0.35;
        const double time = c.start + waves * (k / 128 * c.per_kb + c.epilogue);
        if (best_time < 0.0 || time < best_time * 0.98) {  // a narrower tile must win by 2 % to be taken
            best_time = time;
            best = c.bn;
        }
    }
    if (time_out != nullptr) *time_out = best_time;
    return best;
}

// CTAs per tile when K is cut over clusters (64-wide tiles), or 0 to leave tiles whole.  `whole` is the time of whole tiles by
// the model above, and 6.0 us + 0.215 per k-block of a slice that of a clustered launch: both were fitted before the issue loop and the
// overlapped launches of today, which took 0.7 us off a clustered launch and 2 to 3 off whole tiles.  Today, clustered against the best whole tiles: M=209
// N=480 K=12928, four slices, 11.0 us against 21.8; M=128 N=2048 K=7168 9.0 against 12.9; M=256 N=1024 K=8192, two slices, 9.6
// against 14.2; M=600 N=512 K=4096 7.9 against 8.5; left whole: M=128 N=1024 K=2048 5.6.  Clusters of four stop fitting the GPU at once
// between 132 and 136 CTAs, clusters of two at 148.
int choose_cluster_slices(int m, int n, int k, int num_sms, double whole) {
    const long tiles = static_cast<long>((m + 127) / 128) * ((n + 63) / 64);
    const int kb = k / 128;
    int best = 0;
    double best_time = 0.97 * whole;
    for (int slices = 2; slices <= 4; slices *= 2) {
        if (tiles * slices > (slices == 2 ? num_sms : num_sms * 7 / 8) || kb < 2 * slices) continue;
        const double t = 6.0 + 0.215 * ((kb + slices - 1) / slices);
        if (t < best_time) best = slices, best_time = t;
    }
    return best;
}

// Which kernel serves a bf16 product of ordinary operands.  M <= 64: the weight-streaming kernels.  block_n 1 asks for the
// pair-cluster kernel, 2 for the stacked-K kernel (M <= 32), 0 picks the stacked one where it is the fastest.
enum class BatchRoute { General, Stacked, Pair, Refused };

BatchRoute batch_route(const yan::GemmArgs& a, int block_n) {
    const bool want_auto = block_n == 0;
    if (!want_auto && block_n != 1 && block_n != 2) return BatchRoute::General;
    int dev = 0, max_smem = 0, sm_count = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev);
    const bool small_m_ok = yan::small_m_supported(a.m, a.n, a.k, max_smem);
    const bool stacked_ok = yan::stacked_k_supported(a.m, a.n, a.k);
    if (block_n == 2) return stacked_ok ? BatchRoute::Stacked : BatchRoute::Refused;
    if (block_n == 1) return small_m_ok ? BatchRoute::Pair : BatchRoute::Refused;
    // The general kernel stores 16 bytes at a time and checks num_sms; the weight-streaming kernels do neither.  A shape
    // that one of them serves whatever the output is keeps that; the others are held to the general kernel's terms.
    const bool general_ok = yan::is_aligned(a.out, 16) && a.ldd % 8 == 0 && a.num_sms <= sm_count;
    const bool any_output = small_m_ok || (stacked_ok && (a.m <= 16 || a.n / 32 <= static_cast<uint32_t>(sm_count)));
    if ((general_ok || any_output) &&
        yan::stacked_k_preferred(a.m, a.n, a.k, static_cast<uint32_t>(a.num_sms), static_cast<uint32_t>(sm_count),
                                 static_cast<uint32_t>(max_smem)))
        return BatchRoute::Stacked;
    // what the general kernel is the default for, with an output that it does not take
    if (!general_ok && any_output) return small_m_ok ? BatchRoute::Pair : BatchRoute::Stacked;
    return BatchRoute::General;
}

// after_own_quantizer: the kernel in front is this library's quantizer, which has let the pair kernel start only when whatever wrote
// its weights had completed.
int dispatch_gemm(yan::GemmType type, yan::OutKind out_kind, yan::GemmArgs& a, int block_n, void* stream, BatchRoute route,
                  bool constant_weights, bool after_own_quantizer) {
    if (a.m == 0 || a.n == 0 || a.k == 0) return yan::kBadArgument;
    if (a.num_sms <= 0) return yan::kBadArgument;
    const bool want_auto = (block_n == 0);
    double whole_tiles_time = 0.0;
    if (block_n == 0) {
        const int rows = (type == yan::GemmType::GroupedMasked) ? static_cast<int>(a.m * a.num_groups) : static_cast<int>(a.m);
        block_n = choose_block_n(rows, static_cast<int>(a.n), static_cast<int>(a.k), a.num_sms,
                                 type == yan::GemmType::Normal && out_kind == yan::OutKind::BF16 && a.tail_workspace != nullptr,
                                 &whole_tiles_time);
    }
    a.status = status_word_of_current_device();
    a.timeout_ns = g_timeout_ns;
    a.clock_probe = g_clock_probe;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (type == yan::GemmType::Normal && out_kind == yan::OutKind::BF16) {
        if (route == BatchRoute::Refused) return yan::kBadArgument;
        if (route == BatchRoute::Stacked)
            return yan::launch_fp8_gemm_stacked_k(a, s, constant_weights ? yan::kConstantWeights : yan::kAfterAnyKernel);
        if (route == BatchRoute::Pair) return yan::launch_fp8_gemm_small_m(a, s, constant_weights || after_own_quantizer);
    }
    if (type == yan::GemmType::Normal && want_auto && out_kind != yan::OutKind::E4M3 && a.scatter_world == 0) {
        const int slices = choose_cluster_slices(static_cast<int>(a.m), static_cast<int>(a.n), static_cast<int>(a.k), a.num_sms,
                                                 whole_tiles_time);
        if (slices != 0) return yan::launch_gemm_cluster_k(static_cast<uint32_t>(slices), out_kind, a, s);
    }
    // Groups of at most 128 rows: the kernel that follows masked_m, unless 32-wide tiles of the general one fit the GPU at once
    // (6 groups, N=768 K=4096: 14.9 us against 14.1; 8 groups, N=768 K=7168: 22.3 against 31.4).  Full groups of 128 rows lose up
    // to 15 % against 128-row tiles, groups of 64 gain 7 to 23 % (figures in jit_kernels/gemm.py); the counts are on the device, so
    // a caller who knows that groups are nearly full says so with a width.
    if (type == yan::GemmType::GroupedMasked && want_auto && a.m <= 128 &&
        static_cast<uint64_t>(a.num_groups) * ((a.n + 31) / 32) > static_cast<uint64_t>(a.num_sms))
        return a.m <= 64 ? yan::launch_masked_few_rows<64>(a, s) : yan::launch_masked_few_rows<128>(a, s);
    // e4m3 output: 128-wide tiles while every CTA has at most one of them (M=225 N=1152 K=8064, 10 wide tiles or 18)
    if (out_kind == yan::OutKind::E4M3 &&
        static_cast<uint64_t>((a.m + 127) / 128) * ((a.n + 127) / 128) <= static_cast<uint64_t>(a.num_sms))
        return yan::launch_gemm_e4m3_bn128(a, s);
    switch (block_n) {
        case 32: return yan::launch_gemm_bn32(type, out_kind, a, s);
        case 64: return yan::launch_gemm_bn64(type, out_kind, a, s);
        case 96: return yan::launch_gemm_bn96(type, out_kind, a, s);
        case 128: return yan::launch_gemm_bn128(type, out_kind, a, s);
        case 160: return yan::launch_gemm_bn160(type, out_kind, a, s);
        case 192: return yan::launch_gemm_bn192(type, out_kind, a, s);
        case 224: return yan::launch_gemm_bn224(type, out_kind, a, s);
        case 256: return yan::launch_gemm_bn256(type, out_kind, a, s);
        default: return yan::kBadArgument;
    }
}

// A GEMM as a call of its own.
int dispatch_gemm(yan::GemmType type, yan::OutKind out_kind, yan::GemmArgs& a, int block_n, void* stream) {
    const yan::LaunchPlace place = launch_place(stream);
    const bool batch = type == yan::GemmType::Normal && out_kind == yan::OutKind::BF16 && a.num_sms > 0;
    const BatchRoute route = batch ? batch_route(a, block_n) : BatchRoute::General;
    const int rc = dispatch_gemm(type, out_kind, a, block_n, stream, route, g_constant_weights.holds(place), false);
    if (rc == yan::kOk) g_constant_weights.settle(place);
    return rc;
}

bool positive(int a, int b, int c) { return a > 0 && b > 0 && c > 0; }

// Quantizer and GEMM, one behind the other in the stream.
int quantize_and_gemm(const void* x, uint8_t* q, float* scales, const void* rhs, const void* rhs_scales, void* out, int m, int n,
                      int k, int ldd, void* stream, int num_sms, int block_n) {
    const yan::LaunchPlace place = launch_place(stream);
    const bool constant_weights = g_constant_weights.holds(place);
    yan::GemmArgs a;
    a.lhs = q;
    a.lhs_scales = scales;
    a.lhs_scales_ld = static_cast<uint32_t>(m);
    a.rhs = rhs;
    a.rhs_scales = static_cast<const float*>(rhs_scales);
    a.out = out;
    a.ldd = static_cast<uint32_t>(ldd);
    a.m = m, a.n = n, a.k = k;
    a.num_sms = num_sms;
    if (ldd <= 0 || num_sms <= 0) return yan::kBadArgument;
    const BatchRoute route = batch_route(a, block_n);
    // The quantizer lets the GEMM start before it has waited for the kernel in front: every GEMM waits for the quantizer before it
    // reads anything, except the pair kernel, which loads its weights first: it has to start behind whatever wrote them, unless the
    // caller has promised that nothing did.  (Into an output that only that kernel takes, us in a graph, launched like this / when the
    // quantizer has ended: M=64 N=14336 K=1024 16.7 / 17.1, M=64 N=16384 K=2048 21.7 / 22.4, M=32 N=20480 K=1024 13.0 / 13.7.)
    int rc = yan::launch_per_token_cast_to_fp8(x, q, scales, m, k, k, m, static_cast<cudaStream_t>(stream),
                                               route != BatchRoute::Pair || constant_weights);
    if (rc != yan::kOk) return rc;
    rc = dispatch_gemm(yan::GemmType::Normal, yan::OutKind::BF16, a, block_n, stream, route, constant_weights, true);
    if (rc == yan::kOk) g_constant_weights.settle(place);
    return rc;
}

}  // namespace

extern "C" {

#define YAN_EXPORT __attribute__((visibility("default")))

YAN_EXPORT int yan_b200_abi_version(void) { return YAN_B200_ABI_VERSION; }

YAN_EXPORT const char* yan_b200_return_code_string(int code) {
    switch (code) {
        case YAN_B200_OK: return "ok";
        case YAN_B200_BAD_ARGUMENT: return "bad argument (null/misaligned pointer, size, stride or K % 128 != 0)";
        case YAN_B200_SMEM_TOO_LARGE: return "configuration needs more shared memory than the device offers";
        case YAN_B200_TENSOR_MAP_FAILED: return "cuTensorMapEncodeTiled failed";
        case YAN_B200_LAUNCH_FAILED: return "kernel launch or CUDA runtime call failed";
        case YAN_B200_COMM_FAILED: return "collective communication failed";
        case YAN_B200_DEVICE_TIMEOUT: return "a bounded device-side wait ran out";
        case YAN_B200_WORKSPACE_TOO_SMALL: return "workspace too small";
        default: return "unknown code";
    }
}

YAN_EXPORT void yan_b200_gemm_fp8_fp8_bf16_nt(const void* lhs, const void* lhs_scales, const void* rhs,
                                              const void* rhs_scales, void* out, int m, int n, int k, int ldd,
                                              void* stream, int num_sms, int block_n, int* return_code) {
    if (!positive(m, n, k) || ldd <= 0) return set_rc(return_code, yan::kBadArgument);
    yan::GemmArgs a;
    a.lhs = lhs;
    a.lhs_scales = static_cast<const float*>(lhs_scales);
    a.lhs_scales_ld = static_cast<uint32_t>(m);
    a.rhs = rhs;
    a.rhs_scales = static_cast<const float*>(rhs_scales);
    a.out = out;
    a.ldd = static_cast<uint32_t>(ldd);
    a.m = m, a.n = n, a.k = k;
    a.num_sms = num_sms;
    set_rc(return_code, dispatch_gemm(yan::GemmType::Normal, yan::OutKind::BF16, a, block_n, stream));
}

YAN_EXPORT size_t yan_b200_gemm_tail_workspace_bytes(int num_sms) {
    return num_sms > 0 ? yan::tail_workspace_bytes(static_cast<uint32_t>(num_sms), 256) : 0;
}

YAN_EXPORT void yan_b200_gemm_fp8_fp8_bf16_nt_tail(const void* lhs, const void* lhs_scales, const void* rhs,
                                                   const void* rhs_scales, void* out, int m, int n, int k, int ldd,
                                                   void* stream, int num_sms, int block_n, void* workspace,
                                                   size_t workspace_bytes, int* return_code) {
    if (!positive(m, n, k) || ldd <= 0) return set_rc(return_code, yan::kBadArgument);
    if (workspace != nullptr && reinterpret_cast<uintptr_t>(workspace) % 256 != 0)
        return set_rc(return_code, yan::kBadArgument);
    yan::GemmArgs a;
    a.lhs = lhs;
    a.lhs_scales = static_cast<const float*>(lhs_scales);
    a.lhs_scales_ld = static_cast<uint32_t>(m);
    a.rhs = rhs;
    a.rhs_scales = static_cast<const float*>(rhs_scales);
    a.out = out;
    a.ldd = static_cast<uint32_t>(ldd);
    a.m = m, a.n = n, a.k = k;
    a.num_sms = num_sms;
    a.tail_workspace = workspace;
    a.tail_workspace_bytes = workspace_bytes;
    set_rc(return_code, dispatch_gemm(yan::GemmType::Normal, yan::OutKind::BF16, a, block_n, stream));
}

YAN_EXPORT void yan_b200_gemm_fp8_fp8_f32_nt(const void* lhs, const void* lhs_scales, const void* rhs,
                                             const void* rhs_scales, void* out, int m, int n, int k, int ldd,
                                             void* stream, int num_sms, int block_n, int* return_code) {
    if (!positive(m, n, k) || ldd <= 0) return set_rc(return_code, yan::kBadArgument);
    yan::GemmArgs a;
    a.lhs = lhs;
    a.lhs_scales = static_cast<const float*>(lhs_scales);
    a.lhs_scales_ld = static_cast<uint32_t>(m);
    a.rhs = rhs;
    a.rhs_scales = static_cast<const float*>(rhs_scales);
    a.out = out;
    a.ldd = static_cast<uint32_t>(ldd);
    a.m = m, a.n = n, a.k = k;
    a.num_sms = num_sms;
    set_rc(return_code, dispatch_gemm(yan::GemmType::Normal, yan::OutKind::F32, a, block_n, stream));
}

YAN_EXPORT void yan_b200_gemm_fp8_fp8_e4m3_nt(const void* lhs, const void* lhs_scales, const void* rhs,
                                              const void* rhs_scales, void* out, void* out_scales, int m, int n, int k,
                                              int ldd, int out_scales_ld, void* stream, int num_sms,
                                              int* return_code) {
    if (!positive(m, n, k) || ldd <= 0 || out_scales_ld <= 0) return set_rc(return_code, yan::kBadArgument);
    yan::GemmArgs a;
    a.lhs = lhs;
    a.lhs_scales = static_cast<const float*>(lhs_scales);
    a.lhs_scales_ld = static_cast<uint32_t>(m);
    a.rhs = rhs;
    a.rhs_scales = static_cast<const float*>(rhs_scales);
    a.out = out;
    a.ldd = static_cast<uint32_t>(ldd);
    a.out_scales = static_cast<float*>(out_scales);
    a.out_scales_ld = static_cast<uint32_t>(out_scales_ld);
    a.m = m, a.n = n, a.k = k;
    a.num_sms = num_sms;
    // 256: a thread holds one whole 1 x 128 group; dispatch_gemm takes 128-wide tiles instead where every CTA has at most one
    set_rc(return_code, dispatch_gemm(yan::GemmType::Normal, yan::OutKind::E4M3, a, 256, stream));
}

YAN_EXPORT void yan_b200_m_grouped_gemm_fp8_fp8_bf16_nt_contiguous(const void* lhs, const void* lhs_scales,
                                                                   const void* rhs, const void* rhs_scales, void* out,
                                                                   const int* m_indices, int m, int n, int k,
                                                                   int num_groups, void* stream, int num_sms,
                                                                   int block_n, int* return_code) {
    if (!positive(m, n, k) || num_groups <= 0 || m % 128 != 0) return set_rc(return_code, yan::kBadArgument);
    yan::GemmArgs a;
    a.lhs = lhs;
    a.lhs_scales = static_cast<const float*>(lhs_scales);
    a.lhs_scales_ld = static_cast<uint32_t>(m);
    a.rhs = rhs;
    a.rhs_scales = static_cast<const float*>(rhs_scales);
    a.out = out;
    a.ldd = static_cast<uint32_t>(n);
    a.grouped_layout = m_indices;
    a.m = m, a.n = n, a.k = k;
    a.num_groups = static_cast<uint32_t>(num_groups);
    a.num_sms = num_sms;
    if (n % 128 != 0) return set_rc(return_code, yan::kBadArgument);
    set_rc(return_code, dispatch_gemm(yan::GemmType::GroupedContiguous, yan::OutKind::BF16, a, block_n, stream));
}

YAN_EXPORT void yan_b200_m_grouped_gemm_fp8_fp8_bf16_nt_masked(const void* lhs, const void* lhs_scales, const void* rhs,
                                                               const void* rhs_scales, void* out, const int* masked_m,
                                                               int m_max, int n, int k, int num_groups, void* stream,
                                                               int num_sms, int block_n, int* return_code) {
    if (!positive(m_max, n, k) || num_groups <= 0 || n % 128 != 0) return set_rc(return_code, yan::kBadArgument);
    yan::GemmArgs a;
    a.lhs = lhs;
    a.lhs_scales = static_cast<const float*>(lhs_scales);
    a.lhs_scales_ld = static_cast<uint32_t>(m_max) * static_cast<uint32_t>(num_groups);
    a.rhs = rhs;
    a.rhs_scales = static_cast<const float*>(rhs_scales);
    a.out = out;
    a.ldd = static_cast<uint32_t>(n);
    a.grouped_layout = masked_m;
    a.m = m_max, a.n = n, a.k = k;
    a.num_groups = static_cast<uint32_t>(num_groups);
    a.num_sms = num_sms;
    set_rc(return_code, dispatch_gemm(yan::GemmType::GroupedMasked, yan::OutKind::BF16, a, block_n, stream));
}

YAN_EXPORT void yan_b200_per_token_cast_to_fp8(const void* x, void* out, void* out_scales, int m, int k, int x_ld,
                                               int scales_ld, void* stream, int* return_code) {
    if (m <= 0 || k <= 0 || x_ld <= 0 || scales_ld <= 0) return set_rc(return_code, yan::kBadArgument);
    set_rc(return_code,
           yan::launch_per_token_cast_to_fp8(x, out, static_cast<float*>(out_scales), m, k, x_ld, scales_ld,
                                             static_cast<cudaStream_t>(stream),
                                             yan::cast_releases_early(m, yan::ConstantWeights::promised(g_constant_weights.era()))));
}

YAN_EXPORT void yan_b200_per_block_cast_to_fp8(const void* w, void* out, void* out_scales, int n, int k, void* stream,
                                               int* return_code) {
    if (n <= 0 || k <= 0) return set_rc(return_code, yan::kBadArgument);
    set_rc(return_code, yan::launch_per_block_cast_to_fp8(w, out, static_cast<float*>(out_scales), n, k,
                                                          static_cast<cudaStream_t>(stream)));
}

YAN_EXPORT size_t yan_b200_fp8_linear_workspace_bytes(int m, int k) {
    if (m <= 0 || k <= 0 || k % 128 != 0) return 0;
    const size_t q_bytes = yan::align_up(static_cast<size_t>(m) * k, static_cast<size_t>(256));
    const size_t s_bytes = yan::align_up(static_cast<size_t>(m) * (k / 128) * sizeof(float), static_cast<size_t>(256));
    return q_bytes + s_bytes;
}

YAN_EXPORT void yan_b200_fp8_linear_bf16(const void* a, const void* rhs, const void* rhs_scales, void* out,
                                         void* workspace, size_t workspace_bytes, int m, int n, int k, int ldd,
                                         void* stream, int num_sms, int block_n, int* return_code) {
    if (!positive(m, n, k) || k % 128 != 0 || workspace == nullptr) return set_rc(return_code, yan::kBadArgument);
    if (reinterpret_cast<uintptr_t>(workspace) % 256 != 0) return set_rc(return_code, yan::kBadArgument);
    if (workspace_bytes < yan_b200_fp8_linear_workspace_bytes(m, k))
        return set_rc(return_code, yan::kWorkspaceTooSmall);
    uint8_t* q = static_cast<uint8_t*>(workspace);
    float* scales = reinterpret_cast<float*>(q + yan::align_up(static_cast<size_t>(m) * k, static_cast<size_t>(256)));
    set_rc(return_code, quantize_and_gemm(a, q, scales, rhs, rhs_scales, out, m, n, k, ldd, stream, num_sms, block_n));
}

YAN_EXPORT void yan_b200_fp8_linear_bf16_static(const void* a, const void* rhs, const void* rhs_scales, void* out,
                                                int m, int n, int k, int ldd, void* stream, int num_sms, int block_n,
                                                int* return_code) {
    if (!positive(m, n, k) || k % 128 != 0) return set_rc(return_code, yan::kBadArgument);
    const size_t elements = static_cast<size_t>(m) * static_cast<size_t>(k);
    if (elements > kStaticScratchQBytes || elements / 128 * sizeof(float) > kStaticScratchScaleBytes)
        return set_rc(return_code, yan::kWorkspaceTooSmall);  // M * K exceeds the built-in scratch
    unsigned char* scratch = static_scratch_of_current_device();
    if (scratch == nullptr) return set_rc(return_code, yan::kLaunchFailed);
    uint8_t* q = scratch;
    float* scales = reinterpret_cast<float*>(scratch + kStaticScratchQBytes);
    set_rc(return_code, quantize_and_gemm(a, q, scales, rhs, rhs_scales, out, m, n, k, ldd, stream, num_sms, block_n));
}

YAN_EXPORT void yan_b200_read_device_status(int* status, int reset, int* return_code) {
    if (status == nullptr) return set_rc(return_code, yan::kBadArgument);
    int* word = status_word_of_current_device();
    if (word == nullptr) return set_rc(return_code, yan::kLaunchFailed);
    // cudaMemcpy alone only orders against the legacy default stream; kernels on non-blocking streams must finish too
    if (cudaDeviceSynchronize() != cudaSuccess) {
        cudaGetLastError();
        return set_rc(return_code, yan::kLaunchFailed);
    }
    if (cudaMemcpy(status, word, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) {
        cudaGetLastError();
        return set_rc(return_code, yan::kLaunchFailed);
    }
    if (reset != 0 && *status != 0) {
        const int zero = 0;
        if (cudaMemcpy(word, &zero, sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess) {
            cudaGetLastError();
            return set_rc(return_code, yan::kLaunchFailed);
        }
    }
    set_rc(return_code, yan::kOk);
}

YAN_EXPORT void yan_b200_wait_probe(unsigned long long timeout_ns, void* stream, int* return_code) {
    yan::GemmParams p = {};
    p.status = status_word_of_current_device();
    p.timeout_ns = timeout_ns == 0 ? 1 : timeout_ns;
    if (p.status == nullptr) return set_rc(return_code, yan::kLaunchFailed);
    if (p.timeout_ns > 1000000000ull) return set_rc(return_code, yan::kBadArgument);  // a probe waits at most 1 s
    wait_probe_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(p);
    set_rc(return_code, cudaGetLastError() == cudaSuccess ? yan::kOk : yan::kLaunchFailed);
}

// ---- peer-mapped memory and the two-shot allreduce of the K-split GEMM ----

YAN_EXPORT void yan_b200_ipc_export(const void* ptr, void* handle, unsigned long long* offset, int* return_code) {
    if (ptr == nullptr || handle == nullptr || offset == nullptr) return set_rc(return_code, yan::kBadArgument);
    static_assert(sizeof(cudaIpcMemHandle_t) == YAN_B200_IPC_HANDLE_BYTES, "handle size is part of the ABI");
    using RangeFn = CUresult (*)(CUdeviceptr*, size_t*, CUdeviceptr);
    static RangeFn range = []() -> RangeFn {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuMemGetAddressRange", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return nullptr;
        return reinterpret_cast<RangeFn>(p);
    }();
    CUdeviceptr base = 0;
    size_t size = 0;
    if (range == nullptr || range(&base, &size, reinterpret_cast<CUdeviceptr>(ptr)) != CUDA_SUCCESS)
        return set_rc(return_code, yan::kCommFailed);
    cudaIpcMemHandle_t h;
    if (cudaIpcGetMemHandle(&h, reinterpret_cast<void*>(base)) != cudaSuccess) {
        cudaGetLastError();
        return set_rc(return_code, yan::kCommFailed);
    }
    memcpy(handle, &h, sizeof(h));
    *offset = static_cast<unsigned long long>(reinterpret_cast<CUdeviceptr>(ptr) - base);
    set_rc(return_code, yan::kOk);
}

YAN_EXPORT void yan_b200_ipc_open(const void* handle, void** base, int* return_code) {
    if (handle == nullptr || base == nullptr) return set_rc(return_code, yan::kBadArgument);
    cudaIpcMemHandle_t h;
    memcpy(&h, handle, sizeof(h));
    void* p = nullptr;
    if (cudaIpcOpenMemHandle(&p, h, cudaIpcMemLazyEnablePeerAccess) != cudaSuccess) {
        cudaGetLastError();
        return set_rc(return_code, yan::kCommFailed);
    }
    *base = p;
    set_rc(return_code, yan::kOk);
}

YAN_EXPORT void yan_b200_ipc_close(void* base, int* return_code) {
    if (base == nullptr) return set_rc(return_code, yan::kBadArgument);
    if (cudaIpcCloseMemHandle(base) != cudaSuccess) {
        cudaGetLastError();
        return set_rc(return_code, yan::kCommFailed);
    }
    set_rc(return_code, yan::kOk);
}

YAN_EXPORT void yan_b200_allreduce_bf16_two_shot(void* const* data, void* const* signals, int world, int rank,
                                                 unsigned long long elem_begin, unsigned long long elem_count,
                                                 unsigned int epoch, unsigned int counter_target, int num_ctas,
                                                 int exclusive_sms, void* stream, int* return_code) {
    if (data == nullptr || world < 2 || world > yan::kMaxPeers || (epoch != 0 && signals == nullptr))
        return set_rc(return_code, yan::kBadArgument);
    yan::AllreduceArgs a;
    for (int r = 0; r < world; ++r) {
        a.data.p[r] = data[r];
        a.signals.p[r] = (epoch != 0) ? signals[r] : nullptr;
    }
    a.world = world;
    a.rank = rank;
    a.elem_begin = elem_begin;
    a.elem_count = elem_count;
    a.epoch = epoch;
    a.counter_target = counter_target;
    a.num_ctas = num_ctas;
    a.exclusive = exclusive_sms != 0;
    a.status = status_word_of_current_device();
    a.timeout_ns = g_collective_timeout_ns;
    set_rc(return_code, yan::launch_two_shot_allreduce_bf16(a, static_cast<cudaStream_t>(stream)));
}

YAN_EXPORT void yan_b200_allreduce_bf16_in_switch(void* multicast, void* const* signals, int world, int rank,
                                                  unsigned long long elem_begin, unsigned long long elem_count,
                                                  unsigned int epoch, unsigned int counter_target, int num_ctas,
                                                  int exclusive_sms, void* stream, int* return_code) {
    if (multicast == nullptr || world < 2 || world > yan::kMaxPeers || (epoch != 0 && signals == nullptr))
        return set_rc(return_code, yan::kBadArgument);
    yan::AllreduceArgs a;
    a.multicast = multicast;
    for (int r = 0; r < world; ++r) a.signals.p[r] = (epoch != 0) ? signals[r] : nullptr;
    a.world = world;
    a.rank = rank;
    a.elem_begin = elem_begin;
    a.elem_count = elem_count;
    a.epoch = epoch;
    a.counter_target = counter_target;
    a.num_ctas = num_ctas;
    a.exclusive = exclusive_sms != 0;
    a.status = status_word_of_current_device();
    a.timeout_ns = g_collective_timeout_ns;
    set_rc(return_code, yan::launch_two_shot_allreduce_bf16(a, static_cast<cudaStream_t>(stream)));
}

YAN_EXPORT void yan_b200_gemm_fp8_fp8_bf16_nt_scatter(const void* lhs, const void* lhs_scales, const void* rhs,
                                                      const void* rhs_scales, void* const* stage, int world, int rank,
                                                      int m, int n, int k, int ldd, void* stream, int num_sms, int block_n,
                                                      int* return_code) {
    if (!positive(m, n, k) || ldd <= 0 || stage == nullptr || world < 2 || world > yan::kMaxPeers || rank < 0 || rank >= world)
        return set_rc(return_code, yan::kBadArgument);
    if (block_n != 0 && block_n != 256 && block_n != 128) return set_rc(return_code, yan::kBadArgument);
    yan::GemmArgs a;
    a.lhs = lhs;
    a.lhs_scales = static_cast<const float*>(lhs_scales);
    a.lhs_scales_ld = static_cast<uint32_t>(m);
    a.rhs = rhs;
    a.rhs_scales = static_cast<const float*>(rhs_scales);
    a.out = stage[rank];  // every tile goes to a staging array; `out` only has to be a valid pointer
    a.ldd = static_cast<uint32_t>(ldd);
    a.m = m, a.n = n, a.k = k;
    a.num_sms = num_sms;
    for (int r = 0; r < world; ++r) a.scatter_base[r] = stage[r];
    a.scatter_world = static_cast<uint32_t>(world);
    a.scatter_rank = static_cast<uint32_t>(rank);
    // the staged epilogue exists for the 256- and 128-wide tiles; the general width choice may pick others
    set_rc(return_code, dispatch_gemm(yan::GemmType::Normal, yan::OutKind::BF16, a, block_n == 0 ? 256 : block_n, stream));
}

YAN_EXPORT void yan_b200_allreduce_bf16_gather_staged(const void* stage, void* const* data, void* const* signals,
                                                      int world, int rank, int rows, int ld, unsigned int epoch,
                                                      unsigned int counter_target, int num_ctas, void* stream,
                                                      int* return_code) {
    if (stage == nullptr || data == nullptr || signals == nullptr || world < 2 || world > yan::kMaxPeers || rows <= 0 || ld <= 0)
        return set_rc(return_code, yan::kBadArgument);
    yan::AllreduceArgs a;
    for (int r = 0; r < world; ++r) {
        a.data.p[r] = data[r];
        a.signals.p[r] = signals[r];
    }
    a.world = world;
    a.rank = rank;
    a.epoch = epoch;
    a.counter_target = counter_target;
    a.num_ctas = num_ctas;
    a.status = status_word_of_current_device();
    a.timeout_ns = g_collective_timeout_ns;
    a.stage = stage;
    a.rows = static_cast<uint32_t>(rows);
    a.ld = static_cast<uint32_t>(ld);
    set_rc(return_code, yan::launch_gather_staged_allreduce_bf16(a, static_cast<cudaStream_t>(stream)));
}

YAN_EXPORT void yan_b200_set_programmatic_dependent_launch(int enabled) { g_constant_weights.set(enabled != 0); }

YAN_EXPORT void yan_b200_set_clock_probe(void* device_buffer) { g_clock_probe = static_cast<long long*>(device_buffer); }

YAN_EXPORT void yan_b200_set_wait_timeout_ns(unsigned long long timeout_ns) {
    g_timeout_ns = timeout_ns == 0 ? 1 : timeout_ns;
}

YAN_EXPORT void yan_b200_set_collective_timeout_ns(unsigned long long timeout_ns) {
    g_collective_timeout_ns = timeout_ns == 0 ? 1 : timeout_ns;
}

}  // extern "C"
