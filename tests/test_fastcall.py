"""The native front of the operators: it takes exactly the ordinary calls, gives them the same result as the Python path,
and leaves everything else (copies, errors) to that path."""
import pytest
import torch

from oracle import ref


def test_leaves_unusual_arguments_to_python():
    from yan_b200 import _lib
    f = _lib.fast()
    t = torch.zeros(128, 128)
    assert f.gemm_bf16(t, t, t, t, t, 0, 148, True) == -1          # not on a CUDA device
    assert f.gemm_f32(1, None, "x", t, t, 0, 148, False) == -1     # not tensors
    assert f.gemm_bf16(t, t) == -1 and f.linear() == -1 and f.per_token_cast(t) == -1
    assert f.linear(t, t, t, t, None, {}, 0, 148) == -1
    with pytest.raises(TypeError):
        f.bind(1)


def test_a_missing_or_foreign_front_leaves_everything_to_python(monkeypatch, tmp_path):
    """Another torch's extension is not loaded, whatever the file times say; the operators then run without it."""
    from yan_b200 import _lib
    assert _lib.front_built_for(_lib.front_key())
    with open(_lib.FASTCALL_PATH, "rb") as f:
        built = f.read()
    foreign = tmp_path / "_fastcall.so"
    foreign.write_bytes(built.replace(b"yan_b200 front|torch ", b"yan_b200 front|torch 0"))
    for path in (str(tmp_path / "missing.so"), str(foreign)):
        monkeypatch.setattr(_lib, "FASTCALL_PATH", path)
        monkeypatch.setattr(_lib, "_fast", None)
        with pytest.warns(RuntimeWarning, match="python -m yan_b200.build"):
            assert _lib.fast().gemm_bf16(1, 2) == -1
        assert _lib.fast().per_token_cast() == -1


@pytest.mark.gpu
@pytest.mark.parametrize("m", [1, 7, 130])
@pytest.mark.parametrize("k", [128, 512])
def test_same_results_as_the_python_path(cuda_lib, m, k, monkeypatch):
    """Every scale layout, an output slice and both output types, with the native front and (where it did take the call)
    without it."""
    import yan_b200
    from yan_b200 import _lib
    a, b = ref.make_inputs(m, 256, k, seed=m + k)
    x, rhs = a.cuda(), tuple(t.cuda() for t in ref.per_block_cast_to_fp8(b))
    yan_b200.get_num_sms()

    class NotTaken:
        def __getattr__(self, name):
            return lambda *args: -1

    def run():
        q, s = yan_b200.per_token_cast_to_fp8(x)
        s_wide = torch.zeros(k // 128, m + 5, device="cuda").t()[:m]
        q2 = torch.empty_like(q)
        yan_b200.per_token_cast_to_fp8(x, out=(q2, s_wide))
        outs = [q2.view(torch.uint8), s_wide.clone()]
        for scales in (s, s.contiguous(), s_wide):
            full = torch.full((m, 512), 7.0, dtype=torch.bfloat16, device="cuda")
            yan_b200.gemm_fp8_fp8_bf16_nt((q, scales), rhs, full[:, 128:384])
            f32 = torch.empty(m, 256, device="cuda")
            yan_b200.gemm_fp8_fp8_f32_nt((q, scales), rhs, f32)
            outs += [full, f32]
        out = torch.empty(m, 256, dtype=torch.bfloat16, device="cuda")
        ws = torch.empty(yan_b200.fp8_linear_workspace_bytes(m, k), dtype=torch.uint8, device="cuda")
        outs += [yan_b200.fp8_linear(x, rhs), yan_b200.fp8_linear(x, rhs, out).clone(), yan_b200.fp8_linear(x, rhs, out, ws).clone()]
        torch.cuda.synchronize()
        return outs

    native = run()
    monkeypatch.setattr(_lib, "_fast", NotTaken())
    assert all(torch.equal(n, p) for n, p in zip(native, run()))


@pytest.mark.gpu
@pytest.mark.parametrize("m", [1, 16, 200])
def test_takes_the_ordinary_calls_and_no_others(cuda_lib, m):
    """Return codes of the native front itself: 0 where it made the call, -1 where it left it."""
    import yan_b200
    from yan_b200 import _lib
    f, n, k, sms = _lib.fast(), 256, 512, yan_b200.get_num_sms()
    a, b = ref.make_inputs(m, n, k, seed=m)
    x, (w, ws) = a.cuda(), (t.cuda() for t in ref.per_block_cast_to_fp8(b))
    q, s = yan_b200.per_token_cast_to_fp8(x)
    out, f32 = torch.empty(m, n, dtype=torch.bfloat16, device="cuda"), torch.empty(m, n, device="cuda")
    wide = torch.empty(m, 512, dtype=torch.bfloat16, device="cuda")[:, :n]
    scratch = torch.empty(yan_b200.fp8_linear_workspace_bytes(m, k), dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    kept = {(0, stream, scratch.numel()): scratch}

    assert f.per_token_cast(x, q, s) == 0
    assert f.gemm_bf16(q, s, w, ws, out, 0, sms, True) == 0 and f.gemm_bf16(q, s, w, ws, wide, 0, sms, True) == 0
    assert f.gemm_bf16(q, s, w, ws, out, 64, sms, False) == 0
    assert f.gemm_f32(q, s, w, ws, f32, 0, sms, True) == 0
    assert f.linear(x, w, ws, out, scratch, {}, 0, sms, True) == 0 and f.linear(x, w, ws, out, None, kept, 0, sms, True) == 0
    torch.cuda.synchronize()
    assert yan_b200.read_device_status() == 0
    assert f.gemm_bf16(q, s, w, ws, out, 48, sms, True) == 1, "the library's own refusal"

    row_major = torch.empty(m + 1, k // 128, device="cuda")[:m]
    assert f.per_token_cast(x, q, row_major) == -1 and f.per_token_cast(x.float(), q, s) == -1
    s_wide = torch.empty(k // 128, m + 3, device="cuda").t()[:m]
    for args in ((q, s_wide, w, ws, out), (q, s, w.t(), ws, out), (q, s, w, ws, f32), (q.cpu(), s, w, ws, out), (q, s, w, s, out)):
        assert f.gemm_bf16(*args, 0, sms, True) == -1
    assert f.gemm_f32(q, s, w, ws, out, 0, sms, True) == -1
    assert f.gemm_f32(q, s, w, ws, f32, 0, sms, False) == -1, "whole tiles on request"
    assert (f.gemm_bf16(q, s, w, ws, out, 0, sms, False) == -1) == (m > 64)
    assert (f.linear(x, w, ws, out, scratch, {}, 0, sms, False) == -1) == (m > 64)
    assert f.linear(x, w, ws, out, None, {}, 0, sms, True) == -1, "no scratch yet"
    assert f.linear(x, w, ws, out, scratch[1:], {}, 0, sms, True) == -1 and f.linear(x.float(), w, ws, out, scratch, {}, 0, sms, True) == -1
    torch.cuda.synchronize()


@pytest.mark.gpu
def test_errors_are_raised_as_before(cuda_lib):
    import yan_b200
    a, b = ref.make_inputs(16, 256, 512, seed=1)
    lhs = yan_b200.per_token_cast_to_fp8(a.cuda())
    rhs = tuple(t.cuda() for t in ref.per_block_cast_to_fp8(b))
    out = torch.empty(16, 256, dtype=torch.bfloat16, device="cuda")
    yan_b200.gemm_fp8_fp8_bf16_nt(lhs, rhs, out)
    for bad in (out.float(), out[:8], out.t(), out.cpu(), torch.empty(16, 257, dtype=torch.bfloat16, device="cuda")[:, :256]):
        with pytest.raises(AssertionError):
            yan_b200.gemm_fp8_fp8_bf16_nt(lhs, rhs, bad)
    with pytest.raises(AssertionError):
        yan_b200.gemm_fp8_fp8_f32_nt(lhs, rhs, out)
    with pytest.raises(AssertionError):
        yan_b200.per_token_cast_to_fp8(a.cuda(), out=(lhs[0], lhs[1].contiguous()))
    with pytest.raises(AssertionError):
        yan_b200.fp8_linear(a.cuda().float(), rhs, out)
    from yan_b200._lib import YanB200Error
    with pytest.raises(YanB200Error):
        yan_b200.gemm_fp8_fp8_bf16_nt(lhs, rhs, out, block_n=48)


@pytest.mark.gpu
@pytest.mark.parametrize("native", [True, False])
def test_default_workspace_of_fp8_linear_belongs_to_a_stream(cuda_lib, native, monkeypatch):
    """Calls of the same sizes on two streams, one right behind the other: neither may see the other's activations."""
    import yan_b200
    from yan_b200 import _lib
    from yan_b200.jit_kernels import gemm
    if not native:
        class NotTaken:
            def __getattr__(self, name):
                return lambda *args: -1
        monkeypatch.setattr(_lib, "_fast", NotTaken())
    monkeypatch.setattr(gemm, "_workspaces", {})
    m, n, k = 512, 4096, 2048
    gen = torch.Generator(device="cuda").manual_seed(4)
    rhs = yan_b200.per_block_cast_to_fp8((torch.randn(n, k, generator=gen, device="cuda") * 0.02).to(torch.bfloat16))
    xs = [torch.randn(m, k, generator=gen, device="cuda").to(torch.bfloat16) for _ in range(2)]
    want = [yan_b200.fp8_linear(x, rhs).clone() for x in xs]
    streams = [torch.cuda.Stream() for _ in range(2)]
    outs = [[torch.empty(m, n, dtype=torch.bfloat16, device="cuda") for _ in range(20)] for _ in streams]
    torch.cuda.synchronize()
    for i in range(20):
        for x, stream, out in zip(xs, streams, outs):
            with torch.cuda.stream(stream):
                yan_b200.fp8_linear(x, rhs, out[i])
    torch.cuda.synchronize()
    assert yan_b200.read_device_status() == 0
    assert len({ws.data_ptr() for ws in gemm._workspaces.values()}) == 3, "the default stream's and the two others'"
    assert all(torch.equal(o, w) for w, out in zip(want, outs) for o in out)


@pytest.mark.gpu
def test_quantizer_returns_a_tuple_whatever_holds_its_outputs(cuda_lib):
    import yan_b200
    x = torch.ones(8, 256, dtype=torch.bfloat16, device="cuda")
    q, s = yan_b200.per_token_cast_to_fp8(x)
    result = yan_b200.per_token_cast_to_fp8(x, out=[q, s])
    assert isinstance(result, tuple) and result[0] is q and result[1] is s
