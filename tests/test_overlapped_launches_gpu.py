"""Kernels that are launched while the kernel in front still runs: none may read what that kernel writes before it has, nor
overwrite what it reads."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _call(kind, m, n, k, gen):
    """A function from quantized activations to the output of a call."""
    import yan_b200
    rhs = yan_b200.per_block_cast_to_fp8((torch.randn(n, k, generator=gen, device="cuda") * 0.02).to(torch.bfloat16))
    bf16 = {"dtype": torch.bfloat16, "device": "cuda"}
    if kind == "f32":
        def call(lhs):
            out = torch.empty(m, n, device="cuda")
            yan_b200.gemm_fp8_fp8_f32_nt(lhs, rhs, out)
            return out
    elif kind == "e4m3":  # two of them, chained on codes and scales (N = K)
        def call(lhs):
            out = torch.empty(m, n, **bf16)
            yan_b200.gemm_fp8_fp8_bf16_nt(yan_b200.gemm_fp8_fp8_e4m3_nt(lhs, rhs), rhs, out)
            return out
    elif kind == "masked":
        counts = torch.tensor([7, m], dtype=torch.int32, device="cuda")
        experts = torch.stack([rhs[0].view(torch.uint8)] * 2).view(torch.float8_e4m3fn), torch.stack([rhs[1]] * 2)

        def call(lhs):
            out = torch.zeros(2, 128, n, **bf16)
            groups = lhs[0].view(2, 128, k), lhs[1].as_strided((2, 128, k // 128), (128, 1, 256))
            yan_b200.m_grouped_gemm_fp8_fp8_bf16_nt_masked(groups, experts, out, counts)
            return out
    else:
        def call(lhs):
            out = torch.empty(m, n, **bf16)
            yan_b200.gemm_fp8_fp8_bf16_nt(lhs, rhs, out)
            return out
    return call


# the small-batch kernel with and without clusters, one wave and two of the general one, K shared by clusters, the cut last wave,
# the quantizing epilogue, fp32, masked groups
@pytest.mark.parametrize("kind,m,n,k", [("bf16", 16, 2048, 7168), ("bf16", 64, 7168, 2048), ("bf16", 200, 1024, 1024),
                                        ("bf16", 1111, 5120, 1024), ("bf16", 128, 2048, 7168), ("bf16", 1300, 4096, 12288),
                                        ("e4m3", 200, 1024, 1024), ("f32", 200, 1024, 1024), ("masked", 100, 9600, 512)])
def test_back_to_back_equals_one_at_a_time(cuda_lib, kind, m, n, k):
    import yan_b200
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    rows = 256 if kind == "masked" else m
    xs = [torch.randn(rows, k, generator=gen, device="cuda").to(torch.bfloat16) for _ in range(4)]
    call = _call(kind, m, n, k, gen)
    lhs = yan_b200.per_token_cast_to_fp8(xs[0])

    def run(sync):
        outs = []
        for i in range(12):
            yan_b200.per_token_cast_to_fp8(xs[i % 4], out=lhs)  # lets the next kernel start before it has written anything
            if sync:
                torch.cuda.synchronize()
            outs.append(call(lhs))
            if sync:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return outs

    want = run(True)
    assert not torch.equal(want[0], want[1])
    for _ in range(3):
        assert all(torch.equal(a, b) for a, b in zip(run(False), want))
    assert yan_b200.read_device_status() == 0
