"""Few tiles: the instance of the general kernel whose tiles share K over a cluster (bf16 and fp32 output), and the 128-wide
tiles of the quantizing epilogue, at the edges of their ranges."""
import pytest
import torch

from oracle import ref

pytestmark = pytest.mark.gpu


def _operands(m, n, k, seed):
    a, b = ref.make_inputs(m, (n + 127) // 128 * 128, k, seed=seed, outliers=True)
    lhs, (q, s) = ref.per_token_cast_to_fp8(a), ref.per_block_cast_to_fp8(b)
    lhs_d = (lhs[0].cuda(), lhs[1].t().contiguous().cuda().t())
    return lhs_d, (q[:n].contiguous().cuda(), s.cuda()), ref.ref_gemm_f32(lhs, (q, s))[:, :n]


# two and four slices, K that they do not divide, M and N on both sides of a tile edge, N % 64 != 0, the most tiles that still
# use clusters of four (32) and two (74)
@pytest.mark.parametrize("m,n,k", [(65, 256, 18432), (128, 2048, 7168), (129, 1024, 6016), (209, 480, 12928), (1000, 272, 8192),
                                   (100, 4736, 7040), (127, 4096, 7168), (600, 528, 4096)])
def test_clusters_share_k(cuda_lib, m, n, k):
    import yan_b200
    lhs, rhs, d_ref = _operands(m, n, k, seed=m + n)
    full = torch.full((m + 3, n + 64), 7.0, dtype=torch.bfloat16, device="cuda")
    f32 = torch.full((m + 3, n), 7.0, device="cuda")
    whole = torch.empty(m, n, device="cuda")
    for _ in range(2):
        yan_b200.gemm_fp8_fp8_bf16_nt(lhs, rhs, full[:m, 32:32 + n])
        yan_b200.gemm_fp8_fp8_f32_nt(lhs, rhs, f32[:m])
    yan_b200.gemm_fp8_fp8_f32_nt(lhs, rhs, whole, block_n=32)
    torch.cuda.synchronize()
    assert yan_b200.read_device_status() == 0
    # fp32 sums of K products in another order: a few units of 2^-24 times the number of k-blocks' roundings
    assert ref.rel_frobenius(f32[:m].cpu(), d_ref) <= 1e-5 and ref.rel_frobenius(f32[:m].cpu(), whole.cpu()) <= 1e-6
    d = full[:m, 32:32 + n].cpu()
    assert torch.equal(d, f32[:m].to(torch.bfloat16).cpu()), "both output types round the same sums"
    assert bool((full[m:] == 7.0).all()) and bool((full[:, :32] == 7.0).all()) and bool((full[:, 32 + n:] == 7.0).all())
    assert bool((f32[m:] == 7.0).all())


def test_whole_tiles_on_request(cuda_lib):
    import yan_b200
    lhs, rhs, _ = _operands(200, 512, 12800, seed=9)
    outs = [torch.empty(200, 512, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    yan_b200.set_tail_cut(False)
    try:
        yan_b200.gemm_fp8_fp8_bf16_nt(lhs, rhs, outs[0])
    finally:
        yan_b200.set_tail_cut(True)
    yan_b200.gemm_fp8_fp8_bf16_nt(lhs, rhs, outs[1], block_n=256)
    assert torch.equal(*outs)


# one tile, ragged rows, one k-block, the last grid of single tiles (148 of them) and the first beyond it
@pytest.mark.parametrize("m,n,k", [(1, 128, 128), (127, 256, 1024), (129, 384, 512), (128, 18944, 256), (128, 19072, 256)])
def test_e4m3_output_on_128_wide_tiles(cuda_lib, m, n, k):
    import yan_b200
    lhs, rhs, _ = _operands(m, n, k, seed=m + k)
    q = torch.zeros(m + 2, n, dtype=torch.uint8, device="cuda").view(torch.float8_e4m3fn)
    s = torch.full((n // 128, m + 2), 7.0, device="cuda").t()
    yan_b200.gemm_fp8_fp8_e4m3_nt(lhs, rhs, (q[:m], s[:m]))
    bf16 = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
    yan_b200.gemm_fp8_fp8_bf16_nt(lhs, rhs, bf16, block_n=256)
    q_ref, s_ref = yan_b200.per_token_cast_to_fp8(bf16)
    torch.cuda.synchronize()
    assert yan_b200.read_device_status() == 0
    assert torch.equal(q[:m].view(torch.uint8), q_ref.view(torch.uint8)) and torch.equal(s[:m], s_ref)
    assert not q[m:].view(torch.uint8).any() and bool((s[m:] == 7.0).all()), "stored behind the last row"


@pytest.mark.parametrize("op,m", [("f32", 200), ("f32", 33), ("linear", 200), ("linear", 65)])
def test_whole_tiles_on_request_of_the_other_operators(cuda_lib, op, m):
    """set_tail_cut(False) holds for fp32 output and fp8_linear too: bit for bit the result of an explicit width."""
    import yan_b200
    n, k = 512, 12800
    lhs, rhs, _ = _operands(m, n, k, seed=10)
    x = ref.make_inputs(m, n, k, seed=10, outliers=True)[0].cuda()
    outs = [torch.empty(m, n, dtype=torch.float32 if op == "f32" else torch.bfloat16, device="cuda") for _ in range(3)]
    run = (lambda out, **kw: yan_b200.gemm_fp8_fp8_f32_nt(lhs, rhs, out, **kw)) if op == "f32" else \
        (lambda out, **kw: yan_b200.fp8_linear(x, rhs, out, **kw))
    yan_b200.get_num_sms()
    yan_b200.set_tail_cut(False)
    try:
        run(outs[0])
    finally:
        yan_b200.set_tail_cut(True)
    run(outs[1], block_n=256)
    run(outs[2])
    torch.cuda.synchronize()
    assert yan_b200.read_device_status() == 0
    assert torch.equal(outs[0], outs[1])
    assert op != "f32" or not torch.equal(outs[0], outs[2]), "this shape is one whose K is cut by default"


# the two epilogues of fp32 output on 256-wide tiles: 128-byte box rows up to K = 3968, the ring of scales from K = 4096 on
@pytest.mark.parametrize("k", [128, 3968, 4096])
@pytest.mark.parametrize("m,n", [(129, 272), (300, 2304)])
def test_f32_output_on_256_wide_tiles(cuda_lib, m, n, k):
    import yan_b200
    lhs, rhs, d_ref = _operands(m, n, k, seed=m + k)
    outs = [torch.full((m + 1, n + 4), 7.0, device="cuda") for _ in range(2)]
    for out, block_n in zip(outs, (256, 128)):
        yan_b200.gemm_fp8_fp8_f32_nt(lhs, rhs, out[:m, :n], block_n=block_n)
    torch.cuda.synchronize()
    assert yan_b200.read_device_status() == 0
    assert torch.equal(*outs), "the same products in the same order"
    assert ref.rel_frobenius(outs[0][:m, :n].cpu(), d_ref) <= 1e-5
    assert bool((outs[0][m:] == 7.0).all()) and bool((outs[0][:, n:] == 7.0).all())
