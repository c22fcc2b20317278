"""The weight-streaming kernel of the small batches (M <= 64) at the edges of its tiles, k-parts, slots and clusters, against
the CPU oracle and the general kernel, and its ordering behind kernels that write its weights."""
import pytest
import torch

from oracle import ref

pytestmark = pytest.mark.gpu


def _device(lhs, rhs):
    return (lhs[0].cuda(), lhs[1].t().contiguous().cuda().t()), (rhs[0].cuda(), rhs[1].cuda())


def _operands(m, n, k, seed):
    """Both operands (a ragged N is cut out of whole 128-row scale blocks) and the oracle's result."""
    a, b = ref.make_inputs(m, (n + 127) // 128 * 128, k, seed=seed, outliers=True)
    lhs, (q, s) = ref.per_token_cast_to_fp8(a), ref.per_block_cast_to_fp8(b)
    return lhs, (q[:n].contiguous(), s), ref.ref_gemm(lhs, (q, s))[:, :n]


# M: both sides of every padding.  N: one CTA, widths no CTA divides (n % 32 == 16), clusters of 2 and 4, more row groups
# than SMs.  K: one k-block (all k-parts but one empty), short last parts, more steps than slots, the longest declared.
@pytest.mark.parametrize("m,n,k", [(1, 16, 128), (16, 48, 384), (17, 16, 128), (32, 80, 640), (33, 16, 128), (64, 144, 896),
                                   (8, 528, 13440), (16, 1040, 7168), (5, 2064, 7168), (16, 4784, 1152), (31, 1008, 7168),
                                   (32, 9488, 384), (40, 528, 7168), (64, 1040, 4224), (64, 9472, 256), (63, 272, 18432),
                                   (2, 256, 18432), (24, 272, 18432)])
def test_edges_match_oracle_and_general_kernel(cuda_lib, m, n, k):
    import yan_b200
    lhs, rhs, d_ref = _operands(m, n, k, seed=m + n + k)
    lhs_d, rhs_d = _device(lhs, rhs)
    full = torch.full((m, n + 32), 7.0, dtype=torch.bfloat16, device="cuda")
    yan_b200.gemm_fp8_fp8_bf16_nt(lhs_d, rhs_d, full[:, 16:16 + n])
    general = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
    yan_b200.gemm_fp8_fp8_bf16_nt(lhs_d, rhs_d, general, block_n=32)
    torch.cuda.synchronize()
    assert yan_b200.read_device_status() == 0
    out = full[:, 16:16 + n].cpu()
    bound = ref.bf16_ulp_at(float(d_ref.float().abs().max()))
    assert ref.rel_frobenius(out, d_ref) <= 1e-3 and ref.max_abs_err(out, d_ref) <= bound
    # both kernels sum in fp32, in another order: bf16 results differ by one rounding of few values
    assert ref.rel_frobenius(out, general.cpu()) <= 1e-3
    assert bool((full[:, :16] == 7.0).all()) and bool((full[:, 16 + n:] == 7.0).all()), "stored outside the slice"


@pytest.mark.parametrize("m", [16, 64])
def test_fp8_linear_sees_weights_written_just_before(cuda_lib, m):
    """Weights copied in, then fp8_linear on them, many times over the same buffers: none may read the weights of the round
    before."""
    import yan_b200
    n, k = 2048, 2048
    gen = torch.Generator().manual_seed(3)
    x = torch.randn(m, k, generator=gen).to(torch.bfloat16).cuda()
    q, s = torch.empty(n, k, dtype=torch.float8_e4m3fn, device="cuda"), torch.empty(n // 128, k // 128, device="cuda")
    ws = [(torch.randn(n, k, generator=gen) * 0.02 * (i + 1)).to(torch.bfloat16).cuda() for i in range(4)]
    pairs = [yan_b200.per_block_cast_to_fp8(w) for w in ws]
    want = [yan_b200.fp8_linear(x, p).clone() for p in pairs]
    torch.cuda.synchronize()
    got = []
    for i in list(range(4)) * 3:
        q.view(torch.uint8).copy_(pairs[i][0].view(torch.uint8))
        s.copy_(pairs[i][1])
        got.append(yan_b200.fp8_linear(x, (q, s)).clone())
    torch.cuda.synchronize()
    assert yan_b200.read_device_status() == 0
    assert all(torch.equal(g, want[i % 4]) for i, g in enumerate(got))


@pytest.mark.parametrize("m", [16, 64, 200])
def test_fp8_linear_waits_for_a_kernel_that_lets_it_start_early(cuda_lib, m):
    """The weight codes are written by the activation quantizer, a kernel that lets its successors start before it has finished,
    directly in front of fp8_linear: no copy between them that would separate them.  The quantizer of fp8_linear must not let its
    GEMM load weights before that kernel has completed, nor the next writer overwrite them before the GEMM has."""
    import yan_b200
    n, k = 7168, 2048
    gen = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(m, k, generator=gen, device="cuda").to(torch.bfloat16)
    ws = [torch.randn(n, k, generator=gen, device="cuda").to(torch.bfloat16) for _ in range(4)]
    codes = (torch.empty(n, k, dtype=torch.float8_e4m3fn, device="cuda"), torch.empty(k // 128, n, device="cuda").t())
    rhs = (codes[0], torch.full((n // 128, k // 128), 0.01, device="cuda"))
    workspace = torch.empty(yan_b200.fp8_linear_workspace_bytes(m, k), dtype=torch.uint8, device="cuda")
    outs = [torch.empty(m, n, dtype=torch.bfloat16, device="cuda") for _ in range(16)]
    yan_b200.get_num_sms()

    def run(sync):
        for i, out in enumerate(outs):
            yan_b200.per_token_cast_to_fp8(ws[i % 4], out=codes)
            if sync:
                torch.cuda.synchronize()
            yan_b200.fp8_linear(x, rhs, out, workspace)
            if sync:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return [out.clone() for out in outs]

    want = run(True)
    assert not torch.equal(want[0], want[1])
    for _ in range(3):
        assert all(torch.equal(g, w) for g, w in zip(run(False), want))
    assert yan_b200.read_device_status() == 0


def test_output_that_only_the_streaming_kernels_take(cuda_lib):
    """An output row stride that is no multiple of 8: still accepted where a weight-streaming kernel serves the shape, still
    refused where the general kernel does."""
    import ctypes
    from yan_b200 import _lib
    lhs, rhs, d_ref = _operands(16, 256, 512, seed=5)
    lhs_d, rhs_d = _device(lhs, rhs)
    out = torch.zeros(16, 257, dtype=torch.bfloat16, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    sms = torch.cuda.get_device_properties(0).multi_processor_count

    def call(n, k):
        return _lib.call_rc("yan_b200_gemm_fp8_fp8_bf16_nt", lhs_d[0].data_ptr(), lhs_d[1].data_ptr(), rhs_d[0].data_ptr(),
                            rhs_d[1].data_ptr(), out.data_ptr(), 16, n, k, 257, stream, sms, 0)

    assert call(256, 512) == 0
    torch.cuda.synchronize()
    assert ref.rel_frobenius(out[:, :256].cpu(), d_ref) <= 1e-3
    assert call(256, 384) == 1 and call(240, 512) == 1


def test_clusters_of_several_streams_share_the_gpu(cuda_lib):
    """Kernels whose CTAs wait for one another inside a cluster, side by side on three streams: every one gives its tensor
    memory back before it waits, so they finish, with the results they have alone."""
    import yan_b200
    # clusters of two and four of this kernel, the pair kernel, the general kernel's clusters
    cases = [(16, 2048, 4096, 0), (32, 4096, 2048, 0), (16, 1024, 8192, 0), (16, 4096, 2048, 1), (128, 2048, 7168, 0)]
    calls, want = [], []
    for m, n, k, block_n in cases:
        a, b = ref.make_inputs(m, n, k, seed=m + n + block_n)
        lhs, rhs = yan_b200.per_token_cast_to_fp8(a.cuda()), yan_b200.per_block_cast_to_fp8(b.cuda())
        calls.append((lhs, rhs, block_n))
        want.append(torch.empty(m, n, dtype=torch.bfloat16, device="cuda"))
        yan_b200.gemm_fp8_fp8_bf16_nt(lhs, rhs, want[-1], block_n=block_n)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(3)]
    outs = [[torch.empty_like(w) for w in want] for _ in streams]
    for i in range(60):
        for j, stream in enumerate(streams):
            lhs, rhs, block_n = calls[(i + 2 * j) % len(calls)]
            with torch.cuda.stream(stream):
                yan_b200.gemm_fp8_fp8_bf16_nt(lhs, rhs, outs[j][(i + 2 * j) % len(calls)], block_n=block_n)
    torch.cuda.synchronize()
    assert yan_b200.read_device_status() == 0
    assert all(torch.equal(o, w) for out in outs for o, w in zip(out, want))


def test_output_that_only_the_streaming_kernels_take_beyond_their_default(cuda_lib):
    """The same where the general kernel is the default for other outputs: M <= 16, more row groups than two per SM, long K."""
    import ctypes
    import yan_b200
    from yan_b200 import _lib
    m, n, k = 9, 9600, 8704
    gen = torch.Generator(device="cuda").manual_seed(6)
    lhs = yan_b200.per_token_cast_to_fp8(torch.randn(m, k, generator=gen, device="cuda").to(torch.bfloat16))
    rhs = yan_b200.per_block_cast_to_fp8((torch.randn(n, k, generator=gen, device="cuda") * 0.02).to(torch.bfloat16))
    out = torch.zeros(m, n + 1, dtype=torch.bfloat16, device="cuda")
    general = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    sms = torch.cuda.get_device_properties(0).multi_processor_count

    def call(n, k):
        return _lib.call_rc("yan_b200_gemm_fp8_fp8_bf16_nt", lhs[0].data_ptr(), lhs[1].data_ptr(), rhs[0].data_ptr(),
                            rhs[1].data_ptr(), out.data_ptr(), m, n, k, n + 1, stream, sms, 0)

    assert call(n, k) == 0
    yan_b200.gemm_fp8_fp8_bf16_nt(lhs, rhs, general, block_n=32)
    torch.cuda.synchronize()
    assert yan_b200.read_device_status() == 0
    # both kernels sum in fp32, in another order: bf16 results differ by one rounding of few values
    assert ref.rel_frobenius(out[:, :n].cpu(), general.cpu()) <= 1e-3 and not out[:, n].any()
    assert call(n, k - 128) == 1 and call(n - 16, k) == 1


def test_num_sms_caps_the_grid(cuda_lib, tmp_path):
    """set_num_sms leaves SMs to another stream: no GEMM of a small batch may have more CTAs than that, whichever kernel it
    goes to (row groups that fit, M <= 16 in wider ones, the general kernel)."""
    import json
    import yan_b200
    from torch.profiler import ProfilerActivity, profile
    shapes = [(16, 1024, 2048), (16, 4096, 2048), (9, 9600, 1024), (64, 7168, 2048), (40, 528, 7168), (32, 6400, 640)]
    calls = []
    for m, n, k in shapes:
        lhs, rhs, d_ref = _operands(m, n, k, seed=m + n + k)
        calls.append((*_device(lhs, rhs), torch.empty(m, n, dtype=torch.bfloat16, device="cuda"), d_ref))
    sms = yan_b200.get_num_sms()
    yan_b200.set_num_sms(100)
    try:
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            for lhs, rhs, out, _ in calls * 2:  # the profiler may miss the first launches
                yan_b200.gemm_fp8_fp8_bf16_nt(lhs, rhs, out)
                torch.cuda.synchronize()
    finally:
        yan_b200.set_num_sms(sms)
    assert yan_b200.read_device_status() == 0
    for _, _, out, d_ref in calls:
        assert ref.rel_frobenius(out.cpu(), d_ref) <= 1e-3
    prof.export_chrome_trace(str(tmp_path / "trace.json"))
    events = json.loads((tmp_path / "trace.json").read_text())["traceEvents"]
    grids = [e["args"]["grid"] for e in events if e.get("cat") == "kernel" and "yan::" in e.get("name", "")]
    assert len(grids) >= len(shapes) and all(x * y * z <= 100 for x, y, z in grids), grids
