"""The activation quantizer's wide and narrow accesses: rows that do or do not start on 32-byte boundaries, codes on 8-byte
boundaries, both row counts per CTA, k-groups that do not fill one; bit-exact against the CPU oracle."""
import ctypes

import pytest
import torch

from oracle import ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 9, 1023, 1024, 1057])
@pytest.mark.parametrize("k", [128, 640])
@pytest.mark.parametrize("x_offset,x_pad,q_offset", [(0, 0, 0), (8, 0, 0), (0, 8, 0), (0, 16, 8), (8, 24, 8)])
def test_every_alignment_is_bit_exact(cuda_lib, m, k, x_offset, x_pad, q_offset):
    from yan_b200 import _lib
    gen = torch.Generator().manual_seed(m + k)
    x = (torch.randn(m, k, generator=gen) * torch.logspace(-6, 3, m).view(-1, 1)).to(torch.bfloat16)
    x[m // 2, :128] = 0.0
    q_ref, s_ref = ref.per_token_cast_to_fp8(x)
    ld = k + x_pad
    storage = torch.full((x_offset + m * ld + 64,), 3.0, dtype=torch.bfloat16, device="cuda")
    view = storage[x_offset:x_offset + m * ld].view(m, ld)
    view[:, :k] = x.cuda()
    codes = torch.full((q_offset + m * k + 64,), 0x55, dtype=torch.uint8, device="cuda")
    scales = torch.full((k // 128, m + 3), 7.0, device="cuda")
    _lib.call("yan_b200_per_token_cast_to_fp8", view.data_ptr(), codes.data_ptr() + q_offset, scales.data_ptr(), m, k, ld, m + 3,
              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    got = codes.cpu()
    assert torch.equal(got[q_offset:q_offset + m * k].view(m, k), q_ref.view(torch.uint8))
    assert torch.equal(scales[:, :m].cpu(), s_ref.t()) and bool((scales[:, m:] == 7.0).all())
    assert bool((got[:q_offset] == 0x55).all()) and bool((got[q_offset + m * k:] == 0x55).all()), "stored outside the codes"
