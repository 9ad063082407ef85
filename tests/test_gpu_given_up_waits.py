"""Bounded waits that are given up (at once, while what they wait for is on its way): the result shows it, it is counted, nothing is left behind
and the next call is right. Each scenario runs in a process of its own, for the counts hold for the life of a process."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _product(mode, act, sA, w, sW, out, acc, give_up):
    import torch
    from qspec_b200 import _lib
    lib = _lib.load()
    M, N, K = act.shape[0], w.shape[0], 2 * w.shape[1]
    need = max(lib.qspec_gemm_w4a4_workspace_bytes(M, N, K), lib.qspec_gemm_w4a16_workspace_bytes(M, N, K), lib.qspec_gemm_w4a8_workspace_bytes(M, N, K))
    ws = _product.__dict__.setdefault("ws", torch.zeros(1 << 28, dtype=torch.uint8, device="cuda"))      # one for all calls: it has to stay clean
    assert ws.numel() >= need
    p = lambda t: None if t is None else t.data_ptr()  # noqa: E731
    _lib.check(lib.qspec_debug_gemm_give_up(mode, p(act), p(sA), p(w), p(sW), None, p(out), p(acc), M, N, K, int(mode == 2), p(ws), ws.numel(), give_up,
                                            torch.cuda.current_stream().cuda_stream), "qspec_debug_gemm_give_up")


def _products(shapes, modes):
    """Give the waits of a product up, then run it as ever: NaN or the lowest integer, and a count; then the exact sums."""
    import torch
    from qspec_b200 import ops
    for M, N, K in shapes:
        g = torch.Generator(device="cuda").manual_seed(M + N + K)
        w = torch.randint(-128, 128, (N, K // 2), generator=g, dtype=torch.int8, device="cuda")
        wide = torch.stack(((w << 4) >> 4, w >> 4), -1).reshape(N, K).double()
        q = torch.randint(-8, 8, (M, K), generator=g, dtype=torch.int8, device="cuda")
        packed = ((q[:, 0::2] & 15) | (q[:, 1::2] << 4)).contiguous()
        sums = q.double() @ wide.T
        for mode in modes:
            dt = torch.bfloat16 if mode == 2 else torch.float16
            one = torch.ones(max(M, N), dtype=dt, device="cuda")
            act = {0: packed, 3: q}.get(mode, q.to(dt))
            for raw in (False, True) if mode in (0, 3) else (False,):
                out = None if raw else torch.zeros(M, N, dtype=dt, device="cuda")
                acc = torch.zeros(M, N, dtype=torch.int32, device="cuda") if raw else None
                before = ops.attn_tile_timeouts()
                _product(mode, act, one, w, one, out, acc, 1)
                assert ops.attn_tile_timeouts() > before, (mode, M, N, K, raw)
                assert bool((acc == -2 ** 31).all() if raw else out.isnan().all()), (mode, M, N, K, raw)
                before = ops.attn_tile_timeouts()
                _product(mode, act, one, w, one, out, acc, 0)
                got = acc if raw else out
                assert torch.equal(got, sums.int() if raw else sums.float().to(dt)), (mode, M, N, K, raw)      # whole numbers below 2^24: exact in float32
                assert ops.attn_tile_timeouts() == before


def few_tokens():
    os.environ["QSPEC_GEMM_ROWS"] = "2"
    _products([(1, 8, 128), (9, 4736, 640), (17, 9504, 256), (32, 776, 2176), (4, 28672, 1024)], (0, 1, 2, 3))
    _products([(48, 4800, 256), (64, 9504, 512)], (0,))


def rotation():
    """Any CTAs of a row's cluster give up: the row's scale is NaN whichever they are, their outputs are NaN, and the row is counted once."""
    import math

    import torch
    from qspec_b200 import _lib, ops
    lib = _lib.load()
    for n, rows in [(256, 1), (256, 40), (512, 3), (512, 113), (1024, 2)]:
        x = torch.randn(rows, 28 * n, generator=torch.Generator(device="cuda").manual_seed(n + rows), device="cuda").half()
        scale = 1.0 / math.sqrt(28 * n)
        want_o, want_q, want_s = torch.empty_like(x), torch.empty(rows, 14 * n, dtype=torch.int8, device="cuda"), torch.empty(rows, dtype=torch.float16, device="cuda")
        ops.hadamard_k28(x, n, scale, out=want_o, out_q=want_q, scale_out=want_s)
        assert want_s.isfinite().all()

        def call(give_up, plain):
            o, q, s = torch.zeros_like(want_o), torch.zeros_like(want_q), torch.zeros_like(want_s)
            before = ops.attn_tile_timeouts()
            _lib.check(lib.qspec_debug_hadamard_k28_give_up(x.data_ptr(), o.data_ptr(), None if plain else q.data_ptr(), None if plain else s.data_ptr(), rows, n,
                                                            scale, give_up, torch.cuda.current_stream().cuda_stream), "qspec_debug_hadamard_k28_give_up")
            return o, q, s, ops.attn_tile_timeouts() - before
        for give_up in (1, 2, 8, 64, 127):
            for plain in (False, True):
                o, q, s, counted = call(give_up, plain)
                alone = plain and n == 256 and rows <= 32                                # each CTA counts itself
                assert counted == rows * (bin(give_up).count("1") if alone else 1)
                assert plain or s.isnan().all()
                for c in range(7):
                    part = slice(4 * c * n, 4 * (c + 1) * n)
                    if give_up >> c & 1:
                        assert o[:, part].isnan().all()
                    else:
                        assert torch.equal(o[:, part], want_o[:, part])
        o, q, s, counted = call(0, False)
        assert counted == 0 and torch.equal(o, want_o) and torch.equal(q, want_q) and torch.equal(s, want_s)


def experts():
    """Products that stop while every copy of a short k range has been issued, and an epilogue that leaves the products to themselves: the status
    word says so, and after it has been cleared the next call is right."""
    import torch
    from qspec_b200 import _lib, ops
    lib = _lib.load_seq()
    for T, top, E, W, F in [(5, 1, 1, 128, 128), (40, 2, 3, 256, 264), (700, 4, 8, 1024, 512), (3000, 2, 4, 384, 256)]:
        g = torch.Generator(device="cuda").manual_seed(T + W)
        h = torch.randn(T, W, generator=g, device="cuda").bfloat16()
        gate_up = (torch.randn(E, 2 * F, W, generator=g, device="cuda") * W ** -0.5).bfloat16()
        down = (torch.randn(E, W, F, generator=g, device="cuda") * F ** -0.5).bfloat16()
        idx = torch.randint(-1, E, (T, top), generator=g, device="cuda").int()
        want = torch.empty(T, top, W, dtype=torch.bfloat16, device="cuda")
        ops.moe_expert_grouped(h, gate_up, down, idx, want, E, F, 7.0, act="silu")
        assert ops.moe_grouped_status() == 0
        ws = torch.zeros(lib.qspec_moe_grouped_workspace_bytes(T, top, E, F), dtype=torch.uint8, device="cuda")
        out = torch.empty_like(want)
        for give_up in (1, 2, 3, 0):
            ws[:4].zero_()
            _lib.check(lib.qspec_debug_moe_grouped_give_up(h.data_ptr(), gate_up.data_ptr(), down.data_ptr(), idx.data_ptr(), out.data_ptr(), T, W, F, E, top, 7.0,
                                                           ops.EXPERT_ACTS["silu"], ws.data_ptr(), ws.numel(), give_up, torch.cuda.current_stream().cuda_stream),
                       "qspec_debug_moe_grouped_give_up")
            assert int(ws[:4].view(torch.int32).item()) == (give_up != 0)
            ops.moe_expert_grouped(h, gate_up, down, idx, out, E, F, 7.0, act="silu")
            assert torch.equal(out, want) and ops.moe_grouped_status() == 0


SCENARIOS = [few_tokens, rotation, experts]


@pytest.mark.gpu
@pytest.mark.parametrize("scenario", [s.__name__ for s in SCENARIOS])
def test_given_up_waits(scenario):
    run = subprocess.run([sys.executable, os.path.abspath(__file__), scenario], cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert run.returncode == 0, run.stdout[-2000:] + run.stderr[-4000:]


if __name__ == "__main__":
    sys.path.insert(0, ROOT)
    {s.__name__: s for s in SCENARIOS}[sys.argv[1]]()
