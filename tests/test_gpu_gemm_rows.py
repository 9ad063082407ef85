"""The few-token form of the int4 products (csrc/gemm_w4_rows.cuh) against exact sums: token counts around its groups of 8, channel counts
around its tiles of 32 and around one tile per SM, k around its items of 256, and both sides of the rule that chooses it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from qspec_b200 import ops
    return ops


def _int4(w):
    low = (w << 4) >> 4
    return torch.stack((low, w >> 4), -1).reshape(w.shape[0], -1).double()


def _operands(M, N, K, dt, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = torch.randint(-128, 128, (N, K // 2), generator=g, dtype=torch.int8, device="cuda")
    sW = ((0.5 + torch.rand(N, generator=g, device="cuda")) * 2.0 ** -7).to(dt)
    bias = (torch.randn(N, generator=g, device="cuda") * 0.1).to(dt)
    sA = (0.01 + 0.1 * torch.rand(M, generator=g, device="cuda")).to(dt)
    q = torch.randint(-8, 8, (M, K), generator=g, dtype=torch.int8, device="cuda")
    x = torch.randn(M, K, generator=g, device="cuda").to(dt)
    return w, sW, bias, sA, q, x


SHAPES = [(1, 8, 128), (8, 32, 256), (9, 40, 384), (16, 136, 128), (4, 4096, 4096), (16, 4736, 640), (17, 4768, 384), (24, 9504, 256), (25, 776, 2176),
          (32, 14336, 512), (33, 1000, 1152), (48, 4800, 256), (49, 512, 3840), (64, 6144, 896), (16, 28672, 4096)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("with_bias", [False, True])
def test_rows_products_are_the_exact_sums(ops, monkeypatch, M, N, K, dt, with_bias):
    w, sW, bias, sA, q, x = _operands(M, N, K, dt, M * 131 + N + K)
    b = bias if with_bias else None
    packed = ((q[:, 0::2] & 15) | (q[:, 1::2] << 4)).contiguous()
    monkeypatch.setenv("QSPEC_GEMM_ROWS", "2")
    sums = q.double() @ _int4(w).T                                       # whole numbers: exact
    want = (sums.float() * sA.float()[:, None]) * sW.float()[None, :]
    want = (want + bias.float() if with_bias else want).to(dt)
    out = torch.full((M, N), float("nan"), dtype=dt, device="cuda")
    ops.rowwise_scaled_linear_cutlass_s4s4_unified(packed, sA, w, sW, b, out)
    assert torch.equal(out, want)
    assert torch.equal(ops.gemm_w4a4_acc_i32(packed, w), sums.int())
    if M <= 32:
        out.fill_(float("nan"))
        ops.rowwise_scaled_linear_cutlass_s8s4(q, sA, w, sW, b, out)
        assert torch.equal(out, want)
        out.fill_(float("nan"))
        ops.gemm_w4a16(x, w, sW, b, out)
        exact = x.double() @ _int4(w).T * sW.double()
        exact = exact + bias.double() if with_bias else exact
        # float32: the tensor cores cut the sum of 256 products (16 steps, 2^-23 each at most, of a partial sum's magnitude), the K / 256 sums and the
        # two epilogue operations round; partial sums stay below 6 standard deviations. Then one rounding to 8 or 11 bits.
        mag = (x.double().abs().square().sum(1, keepdim=True) * 21.5).sqrt() * 6 * sW.double()
        bound = mag * (16 + K / 256 + 2) * 2.0 ** -23 + exact.abs() * (2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -11) + 2.0 ** -24
        assert ((out.double() - exact).abs() <= bound).all()
    assert ops.attn_tile_timeouts() == 0


# twelve warps of a CTA alone (more than 16 items of 256 k, up to 8 tokens, W4A4 up to 16) and eight or four warps a CTA of W4A8 on more tiles than SMs
@pytest.mark.parametrize("M,N,K", [(1, 8, 4352), (8, 40, 6144), (9, 776, 6272), (16, 4736, 4352), (4, 4736, 14336), (4, 4744, 4096), (8, 9504, 256), (5, 4744, 4352)])
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
def test_more_warps_for_long_tiles(ops, monkeypatch, M, N, K, dt):
    test_rows_products_are_the_exact_sums(ops, monkeypatch, M, N, K, dt, True)


FORM = {"w4a4": 0, "w4a16": 1, "w4a8": 3}                    # the debug entries' modes


# the last token count that the few-token form takes, and the next group
@pytest.mark.parametrize("mode,M,N,K,few", [
    ("w4a4", 24, 28672, 4096, True), ("w4a4", 25, 28672, 4096, False), ("w4a4", 32, 12288, 4096, True), ("w4a4", 33, 12288, 4096, False), ("w4a4", 64, 8192, 8192, True),
    ("w4a4", 65, 8192, 8192, False), ("w4a4", 24, 32000, 1024, True), ("w4a4", 25, 32000, 1024, False), ("w4a8", 16, 28672, 4096, True), ("w4a8", 17, 28672, 4096, False),
    ("w4a8", 24, 11008, 4096, True), ("w4a8", 25, 11008, 4096, False), ("w4a8", 32, 4096, 14336, True), ("w4a8", 33, 4096, 14336, False), ("w4a16", 16, 28672, 4096, True),
    ("w4a16", 17, 28672, 4096, False), ("w4a16", 16, 12288, 4096, True), ("w4a16", 17, 12288, 4096, False), ("w4a16", 24, 8192, 8192, True), ("w4a16", 25, 8192, 8192, False),
    ("w4a16", 8, 5120, 27648, True), ("w4a16", 9, 5120, 27648, False)])
def test_both_sides_of_the_rule(ops, monkeypatch, mode, M, N, K, few):
    """The form that runs is the one expected (the deferred split of the few-token form is one slice), and both agree, run twice in a row on two inputs."""
    from qspec_b200 import _lib
    w, sW, _, sA, q, x = _operands(M, N, K, torch.float16, M + N)
    kind = {"w4a4": 0, "w4a16": 1, "w4a8": 2}[mode]
    packed = ((q[:, 0::2] & 15) | (q[:, 1::2] << 4)).contiguous()
    assert (_lib.load().qspec_debug_gemm_form(FORM[mode], M, N, K) == 1) == few

    def call(form, flip):
        monkeypatch.setenv("QSPEC_GEMM_ROWS", form)
        assert (_lib.load().qspec_debug_gemm_form(FORM[mode], M, N, K) == 1) == (few if form == "1" else form == "2")
        out = torch.empty(M, N, dtype=torch.float16, device="cuda")
        if mode == "w4a4":
            ops.rowwise_scaled_linear_cutlass_s4s4_unified(packed.flip(0).contiguous() if flip else packed, sA, w, sW, None, out)
        elif mode == "w4a8":
            ops.rowwise_scaled_linear_cutlass_s8s4(q.flip(0).contiguous() if flip else q, sA, w, sW, None, out)
        else:
            ops.gemm_w4a16(x.flip(0).contiguous() if flip else x, w, sW, None, out)
        return out

    if few:
        assert ops.gemm_split_factor(kind, M, N, K) == 1
    can = M <= (64 if mode == "w4a4" else 32)
    for flip in (False, True, False):
        a, b = call("0" if few or not can else "2", flip), call("1", flip)                 # the other form, and the rule's
        if mode == "w4a16":                                               # another order of float32 sums, then a rounding to 11 bits
            assert (a.float() - b.float()).norm() <= 1e-4 * b.float().norm()
        else:
            assert torch.equal(a, b)


@pytest.mark.parametrize("M,N,K", [(1, 8, 128), (4, 4096, 4096), (5, 776, 2176), (9, 40, 384), (16, 4736, 640), (17, 4768, 384), (32, 14336, 512)])
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
def test_few_tokens_through_the_tcgen05_form(ops, monkeypatch, M, N, K, dt):
    """What the rule leaves to the few-token form: the tcgen05 form takes it all the same, where it is asked to."""
    from qspec_b200 import _lib
    w, sW, bias, sA, q, x = _operands(M, N, K, dt, M * 131 + N + K)
    packed = ((q[:, 0::2] & 15) | (q[:, 1::2] << 4)).contiguous()
    monkeypatch.setenv("QSPEC_GEMM_ROWS", "0")
    assert all(_lib.load().qspec_debug_gemm_form(mode, M, N, K) != 1 for mode in range(4))
    sums = q.double() @ _int4(w).T
    want = ((sums.float() * sA.float()[:, None]) * sW.float()[None, :] + bias.float()).to(dt)
    for call, act in ((ops.rowwise_scaled_linear_cutlass_s4s4_unified, packed), (ops.rowwise_scaled_linear_cutlass_s8s4, q)):
        out = torch.full((M, N), float("nan"), dtype=dt, device="cuda")
        call(act, sA, w, sW, bias, out)
        assert torch.equal(out, want)
    assert torch.equal(ops.gemm_w4a4_acc_i32(packed, w), sums.int()) and torch.equal(ops.gemm_w4a8_acc_i32(q, w), sums.int())
    out = torch.full((M, N), float("nan"), dtype=dt, device="cuda")
    ops.gemm_w4a16(x, w, sW, bias, out)
    exact = x.double() @ _int4(w).T * sW.double() + bias.double()
    # float32: a partial sum of K products stays below 6 of its standard deviations; every 16 of them lose at most 2^-23 of it, as do the joins of a
    # tile's parts and the epilogue's two operations. Then one rounding to 8 or 11 bits.
    mag = (x.double().square().sum(1, keepdim=True) * 21.5).sqrt() * 6 * sW.double()
    tol = mag * (K / 16 + 8) * 2.0 ** -23 + (2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -11) * exact.abs() + 2.0 ** -24
    assert bool(((out.double() - exact).abs() <= tol).all())


def test_capture_and_two_streams(ops):
    """Captured calls replay; calls on two streams with weights of their own do not meet."""
    M, N, K = 4, 4096, 4096
    sets = [_operands(M, N, K, torch.float16, s) for s in (1, 2)]
    want = [ops.gemm_w4a16(s[5], s[0], s[1], None, torch.empty(M, N, dtype=torch.float16, device="cuda")) for s in sets]
    outs = [torch.zeros(M, N, dtype=torch.float16, device="cuda") for _ in sets]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for s, o in zip(sets, outs):
            ops.gemm_w4a16(s[5], s[0], s[1], None, o)
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(o, w) for o, w in zip(outs, want))
    streams = [torch.cuda.Stream() for _ in sets]
    for o in outs:
        o.zero_()
    torch.cuda.synchronize()
    for _ in range(20):
        for st, s, o in zip(streams, sets, outs):
            with torch.cuda.stream(st):
                ops.gemm_w4a16(s[5], s[0], s[1], None, o)
    torch.cuda.synchronize()
    assert all(torch.equal(o, w) for o, w in zip(outs, want))


def _outcome(call):
    try:
        return call().clone()
    except Exception as e:
        return type(e), str(e)


@pytest.mark.parametrize("kind", ["w4a4", "w4a8", "w4a16"])
def test_native_call_path_takes_and_refuses_what_the_python_path_does(ops, monkeypatch, kind):
    """Every form of call, with and without csrc/fast_call.cpp: the same values, the same errors."""
    if ops._fast is None:
        pytest.skip("csrc/fast_call.cpp is not built")
    M, N, K = 5, 96, 256
    w, sW, bias, sA, q, x = _operands(M, N, K, torch.float16, 3)
    packed = ((q[:, 0::2] & 15) | (q[:, 1::2] << 4)).contiguous()
    act = {"w4a4": packed, "w4a8": q, "w4a16": x}[kind]
    new = lambda *s, dtype=torch.float16: torch.zeros(*(s or (M, N)), dtype=dtype, device="cuda")  # noqa: E731

    def run(act=act, sA=sA, w=w, sW=sW, bias=bias, out=None):
        out = new() if out is None else out
        if kind == "w4a16":
            return ops.gemm_w4a16(act, w, sW, bias, out)
        return {"w4a4": ops.rowwise_scaled_linear_cutlass_s4s4_unified, "w4a8": ops.rowwise_scaled_linear_cutlass_s8s4}[kind](act, sA, w, sW, bias, out)

    wide = torch.cat([w, w], 1)
    forms = [
        {}, {"bias": None}, {"w": w.view(torch.uint8)}, {"sW": sW.view(-1, 1)}, {"act": act.view(1, M, -1)}, {"out": new(1, M, N)}, {"w": torch.nn.Parameter(w, requires_grad=False)},
        {"act": act.cpu()}, {"w": w.cpu()}, {"act": act.t().contiguous().t()}, {"w": wide[:, :K // 2]}, {"out": new(M, 2 * N)[:, :N]}, {"out": new(M + 1, N)},
        {"out": new(dtype=torch.float32)}, {"out": new(dtype=torch.bfloat16)}, {"sW": sW.float()}, {"sW": sW[:-1].contiguous()}, {"bias": bias[:-1].contiguous()},
        {"bias": bias.bfloat16()}, {"w": w.view(-1)}, {"w": wide}, {"act": act[:, :-128].contiguous()}, {"act": act[:0]}, {"act": act.float()}, {"w": w.int()},
        {"w": w[:N - 4].contiguous(), "sW": sW[:N - 4].contiguous(), "bias": None, "out": new(M, N - 4)}, {"act": None}, {"out": "no tensor"},
    ]
    if kind != "w4a16":
        forms += [{"sA": sA.view(-1, 1)}, {"sA": sA[:-1].contiguous()}, {"sA": sA.bfloat16()}, {"sA": None}, {"act": act.view(torch.uint8)}]
    fast = ops._fast
    for form in forms:
        got = _outcome(lambda: run(**form))
        monkeypatch.setattr(ops, "_fast", None)
        want = _outcome(lambda: run(**form))
        monkeypatch.setattr(ops, "_fast", fast)
        assert (torch.equal(got, want) if isinstance(want, torch.Tensor) and isinstance(got, torch.Tensor) else got == want), (form.keys(), got, want)
