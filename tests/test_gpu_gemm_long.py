"""The form of the tcgen05 int4 products whose CTAs have a tile's length or more to do each (csrc/gemm_w4_stream.cu, LONG): its 16-byte stores
and its shared tiles at remainders of tokens and channels, against exact sums and against the other form, which unaligned outputs take."""
import pytest
import torch

from test_gpu_gemm_rows import _int4, _operands

pytestmark = pytest.mark.gpu

# one token tile and two to four, channels that end 8 or 72 into a tile, tiles that end inside a range and ranges that end inside a tile
SHAPES = [(33, 18952, 256), (64, 28672, 384), (65, 19016, 1152), (128, 28672, 256), (129, 19016, 640), (200, 12296, 1024), (256, 28672, 128), (257, 9608, 384),
          (400, 10240, 1152), (700, 4104, 2048), (1000, 2056, 640)]


# of those, the shapes whose ranges are shorter than a tile: both outputs below then come from the other form
SHORT = {"w4a4": {(129, 19016, 640), (200, 12296, 1024), (257, 9608, 384), (700, 4104, 2048), (1000, 2056, 640)}, "w4a16": {(65, 19016, 1152)}, "w4a8": set()}


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("with_bias", [False, True])
def test_long_products(monkeypatch, M, N, K, dt, with_bias):
    from qspec_b200 import _lib, ops
    w, sW, bias, sA, q, x = _operands(M, N, K, dt, M * 131 + N + K)
    b = bias if with_bias else None
    packed = ((q[:, 0::2] & 15) | (q[:, 1::2] << 4)).contiguous()
    monkeypatch.setenv("QSPEC_GEMM_ROWS", "0")
    for name, mode in (("w4a4", 0), ("w4a16", 2 if dt == torch.bfloat16 else 1), ("w4a8", 3)):
        assert _lib.load().qspec_debug_gemm_form(mode, M, N, K) == (0 if (M, N, K) in SHORT[name] else 2), name
    sums = q.double() @ _int4(w).T                                       # whole numbers: exact
    want = (sums.float() * sA.float()[:, None]) * sW.float()[None, :]
    want = (want + bias.float() if with_bias else want).to(dt)
    room = torch.full((M * N + 16,), float("nan"), dtype=dt, device="cuda")
    got = []
    for shift in (0, 4):                                                 # 16-byte aligned, and 8 bytes off it: the other form
        out = room[shift:shift + M * N].view(M, N)
        for call, act in ((ops.rowwise_scaled_linear_cutlass_s4s4_unified, packed), (ops.rowwise_scaled_linear_cutlass_s8s4, q)):
            room.fill_(float("nan"))
            call(act, sA, w, sW, b, out)
            assert torch.equal(out, want)
            assert bool(room[:shift].isnan().all()) and bool(room[shift + M * N:].isnan().all())
        room.fill_(float("nan"))
        ops.gemm_w4a16(x, w, sW, b, out)
        assert bool(room[:shift].isnan().all()) and bool(room[shift + M * N:].isnan().all())
        got.append(out.clone())
    assert torch.equal(got[0], got[1])                                   # the same sums in the same order
    exact = x.double() @ _int4(w).T * sW.double()
    exact = exact + bias.double() if with_bias else exact
    # float32: a partial sum of K products stays below 6 of its standard deviations; every 16 of them lose at most 2^-23 of it, as do the joins of a
    # tile's parts and the epilogue's two operations. Then one rounding to 8 or 11 bits.
    mag = (x.double().square().sum(1, keepdim=True) * 21.5).sqrt() * 6 * sW.double()
    tol = mag * (K / 16 + 8) * 2.0 ** -23 + (2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -11) * exact.abs() + 2.0 ** -24
    assert bool(((got[0].double() - exact).abs() <= tol).all())
