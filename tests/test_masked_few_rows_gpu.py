"""Masked grouped GEMM with at most 128 rows per group: the kernel whose loads and arithmetic follow masked_m, against the CPU
oracle and the general kernel."""
import pytest
import torch

from oracle import ref

pytestmark = pytest.mark.gpu


# m_max on both sides of the two paddings, row counts on both sides of the 16-row and 32-row steps, empty groups, counts out of
# range, N that leaves part of the last tile, one k-block, more k-blocks than stages, more and fewer tiles than SMs
@pytest.mark.parametrize("g,m_max,n,k,masked", [
    (1, 1, 4864, 128, [1]), (13, 64, 384, 512, [64, 0, 1, 17] * 3 + [16]), (5, 64, 1024, 2048, [33, 500, -4, 0, 64]),
    (20, 128, 256, 1024, [128, 16, 0, 31, 32] * 4), (8, 100, 640, 384, [100, 65, 97, 48] * 2), (2, 65, 7168, 1280, [65, 64]),
    (24, 33, 1024, 256, [i * 33 // 23 for i in range(24)]), (38, 128, 128, 6784, [113, 5] * 19)])
def test_matches_oracle_and_general_kernel(cuda_lib, g, m_max, n, k, masked):
    import yan_b200
    gen = torch.Generator().manual_seed(g + n + k)
    a = torch.randn(g * m_max, k, generator=gen).to(torch.bfloat16)
    a[:, torch.randperm(k, generator=gen)[:max(1, k // 100)]] *= 20.0
    b = (torch.randn(g * n, k, generator=gen) * 0.02).to(torch.bfloat16)
    (qa, sa), (qb, sb) = ref.per_token_cast_to_fp8(a), ref.per_block_cast_to_fp8(b)
    lhs = (qa.cuda().view(g, m_max, k), sa.contiguous().cuda().view(g, m_max, k // 128))
    rhs = (qb.cuda().view(g, n, k), sb.cuda().view(g, n // 128, k // 128))
    counts = torch.tensor(masked, dtype=torch.int32, device="cuda")
    storage = torch.full((2, g + 1, m_max, n), 9.0, dtype=torch.bfloat16, device="cuda")
    yan_b200.m_grouped_gemm_fp8_fp8_bf16_nt_masked(lhs, rhs, storage[0, :g], counts)
    yan_b200.m_grouped_gemm_fp8_fp8_bf16_nt_masked(lhs, rhs, storage[1, :g], counts, block_n=256)
    torch.cuda.synchronize()
    assert yan_b200.read_device_status() == 0
    got = storage.cpu()
    assert bool((got[0, g] == 9.0).all()), "rows behind the last group were written"
    for i, count in enumerate(masked):
        rows = min(max(count, 0), m_max)
        assert bool((got[0, i, rows:] == 9.0).all()), f"group {i}: rows beyond masked_m must stay untouched"
        if rows:
            r = slice(i * m_max, i * m_max + rows)
            d_ref = ref.ref_gemm((qa[r], sa[r]), (qb[i * n:(i + 1) * n], sb[i * n // 128:(i + 1) * n // 128]))
            assert ref.rel_frobenius(got[0, i, :rows], d_ref) <= 1e-3, f"group {i}"
            # the same products in the same order, k-block by k-block
            assert torch.equal(got[0, i, :rows], got[1, i, :rows]), f"group {i}: differs from the general kernel"
