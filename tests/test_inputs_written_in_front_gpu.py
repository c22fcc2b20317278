"""What the kernel in front writes (activations, weights, the group layout) is read by a kernel that starts beside it only when it is
there."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _bytes_through_the_quantizer(data):
    """bf16 rows whose e4m3 codes are the bytes of `data` (int32, a multiple of 32 of them), the last byte of each 128 apart: its
    value, the largest there is, makes the scale of its group 1."""
    codes = data.contiguous().view(torch.uint8).view(-1, 128).clone()
    codes[:, -1] = 0x7E
    return codes.view(torch.float8_e4m3fn).float().to(torch.bfloat16)


def _case(kind, m, n, k, gen):
    """(rows of the activations, rows of the weights, sources of the group layout, call(lhs, rhs, layout, out), output)"""
    import yan_b200
    one = torch.zeros(32, dtype=torch.int32, device="cuda")
    bf16 = {"dtype": torch.bfloat16, "device": "cuda"}
    if kind == "f32":
        return m, n, [one], lambda lhs, rhs, layout, out: yan_b200.gemm_fp8_fp8_f32_nt(lhs, rhs, out), torch.zeros(m, n, device="cuda")
    if kind == "e4m3":  # two of them, chained on codes and scales (N = K)
        def call(lhs, rhs, layout, out):
            yan_b200.gemm_fp8_fp8_bf16_nt(yan_b200.gemm_fp8_fp8_e4m3_nt(lhs, rhs), rhs, out)
        return m, n, [one], call, torch.zeros(m, n, **bf16)
    if kind in ("masked", "masked_wide"):
        counts = [torch.tensor(c + [0] * 30, dtype=torch.int32, device="cuda") for c in ([7, m], [m, 7], [0, m // 2], [m, m])]
        m_max = (m + 63) // 64 * 64

        def call(lhs, rhs, layout, out):
            groups = lhs[0].view(2, m_max, k), lhs[1].as_strided((2, m_max, k // 128), (m_max, 1, 2 * m_max))
            experts = rhs[0].view(2, n, k), rhs[1].view(2, n // 128, k // 128)
            yan_b200.m_grouped_gemm_fp8_fp8_bf16_nt_masked(groups, experts, out, layout[:2], block_n=256 if kind == "masked_wide" else 0)
        return 2 * m_max, 2 * n, counts, call, torch.zeros(2, m_max, n, **bf16)
    if kind == "contiguous":
        layouts = [torch.tensor([(i + t) % 2 if t < 2 else i // 2 for t in range(m // 128) for _ in range(128)], dtype=torch.int32,
                                device="cuda") for i in range(4)]

        def call(lhs, rhs, layout, out):
            experts = rhs[0].view(2, n, k), rhs[1].view(2, n // 128, k // 128)
            yan_b200.m_grouped_gemm_fp8_fp8_bf16_nt_contiguous(lhs, experts, out, layout)
        return m, 2 * n, layouts, call, torch.zeros(m, n, **bf16)
    block_n = {"pair": 1, "bf16_96": 96}.get(kind, 0)
    return (m, n, [one], lambda lhs, rhs, layout, out: yan_b200.gemm_fp8_fp8_bf16_nt(lhs, rhs, out, block_n=block_n),
            torch.zeros(m, n, **bf16))


# the small-batch kernel with and without clusters, the pair kernel, one wave and two of the general one, its scales in shared
# memory and in registers, K shared by clusters, the cut last wave, the quantizing epilogue, fp32, the grouped forms
SHAPES = [("bf16", 16, 2048, 7168), ("bf16", 64, 7168, 2048), ("pair", 16, 7168, 2048), ("bf16", 200, 1024, 1024),
          ("bf16_96", 200, 1024, 1024), ("bf16", 1111, 5120, 1024), ("bf16", 128, 2048, 7168), ("bf16", 1300, 4096, 12288),
          ("e4m3", 200, 1024, 1024), ("f32", 200, 1024, 1024), ("masked", 100, 9600, 512), ("masked_wide", 200, 1024, 512),
          ("contiguous", 512, 1024, 512)]


@pytest.mark.parametrize("kind,m,n,k,written", [(*shape, written) for shape in SHAPES for written in ("activations", "weights", "layout")
                                                if written != "layout" or shape[0].startswith(("masked", "contiguous"))])
def test_back_to_back_equals_one_at_a_time_whatever_is_written(cuda_lib, kind, m, n, k, written):
    """The quantizer writes what the call behind it reads (activations with their scales, weight codes, the group layout): it lets
    the next kernel start before it has written anything."""
    import yan_b200
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    lhs_rows, rhs_rows, layouts, call, out = _case(kind, m, n, k, gen)

    def randn(rows):
        return torch.randn(rows, k, generator=gen, device="cuda").to(torch.bfloat16)

    rows = {"activations": lhs_rows, "weights": rhs_rows}.get(written)
    sources = [randn(rows) for _ in range(4)] if rows else [_bytes_through_the_quantizer(t) for t in layouts]
    lhs, codes = yan_b200.per_token_cast_to_fp8(randn(lhs_rows)), yan_b200.per_token_cast_to_fp8(randn(rhs_rows))
    rhs = (codes[0], torch.full((rhs_rows // 128, k // 128), 0.01, device="cuda"))
    layout = yan_b200.per_token_cast_to_fp8(_bytes_through_the_quantizer(layouts[0]))
    target = {"activations": lhs, "weights": codes, "layout": layout}[written]
    outs = [torch.zeros_like(out) for _ in range(12)]

    def run(sync):
        for o in outs:
            o.zero_()
        torch.cuda.synchronize()
        for i, o in enumerate(outs):
            yan_b200.per_token_cast_to_fp8(sources[i % 4], out=target)
            if sync:
                torch.cuda.synchronize()
            call(lhs, rhs, layout[0].view(torch.uint8).view(-1).view(torch.int32), o)
            if sync:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return [o.clone() for o in outs]

    want = run(True)
    assert not any(torch.equal(want[i], want[j]) for i in range(4) for j in range(i))
    for _ in range(3):
        assert all(torch.equal(a, b) for a, b in zip(run(False), want))
    assert yan_b200.read_device_status() == 0


# the small-batch kernel and the pair kernel, both of which load weights before their wait under the promise
@pytest.mark.parametrize("m,block_n", [(16, 0), (64, 0), (16, 1), (64, 1)])
@pytest.mark.parametrize("switched", [False, True])
def test_a_cast_separates_constant_weights_from_their_writer(cuda_lib, m, block_n, switched):
    """With the promise that the call in front of a GEMM does not write its weights: the weight codes are written by a kernel that
    lets its successors start early, the activations are quantized by a call between the two, and the GEMM sees the new weights;
    also where the promise is made for the GEMM's call alone."""
    import yan_b200
    n, k = 7168, 2048
    gen = torch.Generator(device="cuda").manual_seed(m)
    x = torch.randn(m, k, generator=gen, device="cuda").to(torch.bfloat16)
    ws = [torch.randn(n, k, generator=gen, device="cuda").to(torch.bfloat16) for _ in range(4)]
    codes = (torch.empty(n, k, dtype=torch.float8_e4m3fn, device="cuda"), torch.empty(k // 128, n, device="cuda").t())
    rhs = (codes[0], torch.full((n // 128, k // 128), 0.01, device="cuda"))
    lhs = yan_b200.per_token_cast_to_fp8(x)
    outs = [torch.empty(m, n, dtype=torch.bfloat16, device="cuda") for _ in range(16)]

    def run(sync):
        for i, out in enumerate(outs):
            for j in range(3):
                yan_b200.set_programmatic_dependent_launch(j == 2 or not switched)
                if j < 2:
                    yan_b200.per_token_cast_to_fp8(*((ws[i % 4], codes) if j == 0 else (x, lhs)))
                else:
                    yan_b200.gemm_fp8_fp8_bf16_nt(lhs, rhs, out, block_n=block_n)
                if sync:
                    torch.cuda.synchronize()
        torch.cuda.synchronize()
        return [out.clone() for out in outs]

    try:
        want = run(True)
        assert not torch.equal(want[0], want[1])
        for _ in range(3):
            assert all(torch.equal(g, w) for g, w in zip(run(False), want))
    finally:
        yan_b200.set_programmatic_dependent_launch(False)
    assert yan_b200.read_device_status() == 0


# an output that only the weight-streaming kernels take, where the pair kernel is the one of them; the same kernel by name
@pytest.mark.parametrize("block_n,pad", [(0, 1), (1, 1), (1, 0)])
def test_fp8_linear_of_the_pair_kernel_sees_weights_written_directly_in_front(cuda_lib, block_n, pad):
    """The pair kernel loads weights before it waits for the quantizer of its call, which lets it start behind whatever wrote them."""
    import yan_b200
    m, n, k = 64, 14336, 1024
    gen = torch.Generator(device="cuda").manual_seed(8)
    x = torch.randn(m, k, generator=gen, device="cuda").to(torch.bfloat16)
    ws = [torch.randn(n, k, generator=gen, device="cuda").to(torch.bfloat16) for _ in range(4)]
    codes = yan_b200.per_token_cast_to_fp8(ws[0])
    rhs = (codes[0], torch.full((n // 128, k // 128), 0.01, device="cuda"))
    outs = [torch.zeros(m, n + pad, dtype=torch.bfloat16, device="cuda") for _ in range(8)]

    def run(sync):
        for i, out in enumerate(outs):
            yan_b200.per_token_cast_to_fp8(ws[i % 4], out=codes)
            if sync:
                torch.cuda.synchronize()
            yan_b200.fp8_linear(x, rhs, out[:, :n], block_n=block_n)
            if sync:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return [out.clone() for out in outs]

    want = run(True)
    assert not torch.equal(want[0], want[1])
    general = yan_b200.fp8_linear(x, rhs, block_n=64)
    # other order of the fp32 sums: bf16 results differ by one rounding of few values
    assert float((want[3][:, :n].float() - general.float()).norm() / general.float().norm()) <= 1e-3
    for _ in range(3):
        assert all(torch.equal(g, w) for g, w in zip(run(False), want))
    assert yan_b200.read_device_status() == 0


# e4m3 output on tiles of one wave, on both sides of the line up to which the launch overlaps the kernel in front
@pytest.mark.parametrize("k", [12288, 12416])
def test_e4m3_output_of_long_k_behind_its_quantizer(cuda_lib, k):
    import yan_b200
    m, n = 200, 384
    gen = torch.Generator(device="cuda").manual_seed(k)
    xs = [torch.randn(m, k, generator=gen, device="cuda").to(torch.bfloat16) for _ in range(4)]
    rhs = yan_b200.per_block_cast_to_fp8((torch.randn(n, k, generator=gen, device="cuda") * 0.02).to(torch.bfloat16))
    want = []
    for x in xs:
        out = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
        lhs = yan_b200.per_token_cast_to_fp8(x)
        torch.cuda.synchronize()
        yan_b200.gemm_fp8_fp8_bf16_nt(lhs, rhs, out, block_n=256)
        torch.cuda.synchronize()
        want.append(yan_b200.per_token_cast_to_fp8(out))
        torch.cuda.synchronize()
    lhs = yan_b200.per_token_cast_to_fp8(xs[0])
    got = []
    for i in range(12):
        yan_b200.per_token_cast_to_fp8(xs[i % 4], out=lhs)
        got.append(yan_b200.gemm_fp8_fp8_e4m3_nt(lhs, rhs))
    torch.cuda.synchronize()
    for i, (q, s) in enumerate(got):
        assert torch.equal(q.view(torch.uint8), want[i % 4][0].view(torch.uint8)) and torch.equal(s, want[i % 4][1])
    assert yan_b200.read_device_status() == 0
