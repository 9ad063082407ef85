"""The gated recurrence of bfloat16 rows on the tensor cores, against float64, token by token: blocks of 16 tokens cut short, chunks, states carried in and
out, decays next to 0 and 1, values that are not finite, and the rule that takes it."""
import pytest
import torch

from test_gpu_recurrence_chunks import CASES, ops, table, walk  # noqa: F401

pytestmark = pytest.mark.gpu


def inputs(T, H, D, DV, slots, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    p = torch.randn(T, 2 * H * D + H * DV, generator=g, device="cuda").bfloat16()
    bias = torch.randn(H * D, generator=g, device="cuda") * 8                      # decays from e^-20 to 1
    lower = torch.rand(H * D, generator=g, device="cuda") * (torch.rand(H * D, generator=g, device="cuda") < 0.5)
    return p, bias, lower, torch.randn(DV, generator=g, device="cuda"), torch.randn(slots, H, D, DV, generator=g, device="cuda")


def want_of(p, bias, lower, norm, state, segments, H, D, DV):
    T, z, state = p.shape[0], p.double(), state.double()
    zq, zf, v = z[:, :H * D], z[:, H * D:2 * H * D], z[:, 2 * H * D:].view(T, H, DV)
    f = (lower.double() + (1 - lower.double()) * torch.sigmoid(zf + bias.double())).view(T, H, D)
    om = ((1 - lower.double()) * torch.sigmoid(-(zf + bias.double()))).view(T, H, D)
    o = walk((zq * torch.sigmoid(zq)).view(T, H, D), f, om, v, segments, state)
    return (o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-5) * norm.double()).view(T, H * DV), state


def taken(segments, T, H, D, DV):
    from qspec_b200 import _lib
    return _lib.load_seq().qspec_seq_hgrn2_chunk_bytes(len(segments), T, H, D, DV, _lib.DTYPE_BF16) > 0


@pytest.mark.parametrize("H,D,DV,segments", [
    (3, 128, 128, [(0, 0, 192)]),                                  # whole chunks of two blocks
    (2, 128, 128, [(1, 9, 193), (0, 0, 193)]),                     # a last chunk of one token, states carried in
    (40, 128, 128, [(0, 0, 1023)]),                                # chunks longer than the smallest, the last block cut short
    (5, 64, 128, [(2, 5, 300), (1, 0, 209)]),
    (4, 128, 64, [(0, 7, 250)]),
    (3, 64, 64, [(0, 0, 257), (2, 3, 1), (1, 8, 600)]),            # a segment of one token
])
def test_against_float64(ops, H, D, DV, segments):
    meta, starts = table(segments)
    T = meta.shape[1]
    assert taken(segments, T, H, D, DV)
    p, bias, lower, norm, state = inputs(T, H, D, DV, 3, D + DV + H)
    want, want_state = want_of(p, bias, lower, norm, state, segments, H, D, DV)
    out = torch.empty(T, H * DV, dtype=torch.bfloat16, device="cuda")
    ops.seq_hgrn2(p, bias, lower, norm, state, torch.empty(T * H * (DV + 3 * D), device="cuda"), out, meta, H, D, DV, 1e-5, seg_starts=starts)
    # half a unit in the last place of bfloat16; float32 sums whose terms' own rounding grows along the state's memory
    assert ((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2e-5 * want.abs().max()).all()
    for slot, _, _ in segments:
        assert (state[slot].double() - want_state[slot]).abs().max() <= 2e-5 * want_state[slot].abs().max()


def test_values_that_are_not_finite(ops):
    """An infinite value reaches its own column from there on, a gate that is not a number its row; other heads and earlier tokens see nothing of them."""
    H, D, DV, segments = 3, 128, 128, [(0, 4, 300)]
    meta, starts = table(segments)
    p, bias, lower, norm, state = inputs(300, H, D, DV, 1, 5)
    p[150, 2 * H * D + 7] = float("inf")
    p[200, H * D + 1 * D + 3] = float("nan")
    run = lambda s, form: ops.seq_hgrn2(p if form else p.float(), bias, lower, norm, s, torch.empty(300 * H * (DV + 3 * D), device="cuda"), form_out[form], meta, H, D, DV,
                                        1e-5, seg_starts=starts)
    form_out = [torch.empty(300, H * DV, device="cuda"), torch.empty(300, H * DV, dtype=torch.bfloat16, device="cuda")]
    states = [state.clone(), state.clone()]
    for form in (0, 1):                                            # float32 rows take the form without tensor cores
        run(states[form], form)
    a, b = form_out[0].double(), form_out[1].double()
    assert torch.equal(torch.isfinite(a), torch.isfinite(b))
    ok = torch.isfinite(a)
    assert ok[:150].all() and ok[:, 2 * DV:].all() and not ok[150:, 7].any() and not ok[200:, DV:2 * DV].any()
    assert ((a - b).abs()[ok] <= 2.0 ** -8 * a.abs()[ok] + 2e-5 * a[ok].abs().max()).all()
    assert torch.equal(torch.isfinite(states[0]), torch.isfinite(states[1]))
    fin = torch.isfinite(states[0])
    assert ((states[0] - states[1]).abs()[fin] <= 2e-5 * states[0][fin].abs().max()).all()


def test_rows_that_are_not_aligned_take_the_other_form(ops):
    H, D, DV, segments = 2, 128, 128, [(0, 0, 320)]
    meta, starts = table(segments)
    p, bias, lower, norm, state = inputs(320, H, D, DV, 1, 6)
    wide = torch.zeros(320 * (p.shape[1] + 3) + 1, dtype=torch.bfloat16, device="cuda")[1:].view(320, -1)   # 2-byte boundaries, rows of 771 elements
    wide[:, :p.shape[1]] = p
    want, want_state = want_of(p, bias, lower, norm, state, segments, H, D, DV)
    out = torch.empty(320, H * DV, dtype=torch.bfloat16, device="cuda")
    ops.seq_hgrn2(wide, bias, lower, norm, state, torch.empty(320 * H * (DV + 3 * D), device="cuda"), out, meta, H, D, DV, 1e-5, seg_starts=starts)
    assert ((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2e-5 * want.abs().max()).all()
    assert (state.double() - want_state).abs().max() <= 2e-5 * want_state.abs().max()


@pytest.mark.parametrize("H,D,DV,segments", CASES)
def test_rows_of_the_other_form_that_are_not_aligned(ops, H, D, DV, segments):
    meta, starts = table(segments)
    T = meta.shape[1]
    p, bias, lower, norm, state = inputs(T, H, D, DV, 3, 6)
    bias = bias * 3 / 8                                                         # decays from nearly 0 to nearly 1
    for slot, p0, _ in segments:
        if p0 == 0:
            state[slot] = float("nan")                                          # a slot's leftovers do not matter at position 0
    wide = torch.zeros(T * (p.shape[1] + 3) + 1, dtype=torch.bfloat16, device="cuda")[1:].view(T, -1)       # 2-byte boundaries, rows of an odd number of elements
    wide[:, :p.shape[1]] = p
    want, want_state = want_of(p, bias, lower, norm, state, segments, H, D, DV)
    out = torch.empty(T, H * DV, dtype=torch.bfloat16, device="cuda")
    ops.seq_hgrn2(wide, bias, lower, norm, state, torch.empty(T * H * (DV + 3 * D), device="cuda"), out, meta, H, D, DV, 1e-5, seg_starts=starts)
    assert ((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2e-5 * want.abs().max()).all()
    for slot, _, _ in segments:
        assert (state[slot].double() - want_state[slot]).abs().max() <= 2e-5 * want_state[slot].abs().max()


@pytest.mark.parametrize("H,D,DV,segments,mma", [
    (16, 128, 128, [(0, 0, 100)], False), (16, 128, 128, [(0, 0, 300)], True), (32, 128, 128, [(0, 0, 150)], False), (16, 96, 128, [(0, 0, 900)], False),
    (8, 64, 64, [(0, 0, 33), (1, 0, 33)], False), (16, 64, 64, [(0, 0, 300)], True)])
def test_both_sides_of_the_rule(ops, H, D, DV, segments, mma):
    meta, starts = table(segments)
    T = meta.shape[1]
    assert taken(segments, T, H, D, DV) == mma
    p, bias, lower, norm, state = inputs(T, H, D, DV, len(segments), 9)
    want, want_state = want_of(p, bias, lower, norm, state, segments, H, D, DV)
    out = torch.empty(T, H * DV, dtype=torch.bfloat16, device="cuda")
    ops.seq_hgrn2(p, bias, lower, norm, state, torch.empty(T * H * (DV + 3 * D), device="cuda"), out, meta, H, D, DV, 1e-5, seg_starts=starts)
    assert ((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2e-5 * want.abs().max()).all()
    assert (state.double() - want_state).abs().max() <= 2e-5 * want_state.abs().max()


def lengths(lens):
    return [(k, 0 if k % 2 else 70, n) for k, n in enumerate(lens)]             # every other segment starts from a state


@pytest.mark.parametrize("H,D,DV,lens", [
    (32, 128, 128, [4] * 64), (16, 128, 128, [1] * 64), (16, 128, 128, [1] * 512), (32, 128, 128, [1] * 256), (64, 128, 128, [5] * 16 + [9]),
    (32, 128, 128, [1] * 64 + [256]), (16, 128, 128, [17] * 64), (8, 64, 64, [5] * 400), (32, 64, 64, [8] * 256), (16, 64, 128, [16] * 128), (16, 128, 64, [100] * 24), (32, 128, 64, [150] * 5),
    (16, 128, 128, [33] * 4), (8, 64, 64, [40] * 24)])
def test_many_short_segments_keep_the_walk_and_no_workspace(ops, H, D, DV, lens):
    from qspec_b200 import _lib
    lib = _lib.load_seq()
    assert lib.qspec_seq_hgrn2_chunk_bytes(len(lens), sum(lens), H, D, DV, _lib.DTYPE_BF16) == lib.qspec_seq_recurrence_chunk_bytes(len(lens), sum(lens), H, D, DV) == 0


@pytest.mark.parametrize("H,D,DV,lens,nbytes", [
    (16, 128, 128, [24, 1, 300, 2, 16, 60], None),                              # one long, others shorter than a block
    (16, 128, 128, [1] * 32 + [1000], None),                                    # decoding sequences beside a prompt
    (16, 128, 128, [33] * 12, None),                                            # segments a little longer than the smallest chunk stay whole
    (200, 128, 128, [60], 16),                                                  # nothing is kept between chunks
    (4, 128, 64, [220, 200], None),
    (32, 64, 64, [1] * 16 + [512], None),
])
def test_segments_of_all_lengths(ops, H, D, DV, lens, nbytes):
    from qspec_b200 import _lib
    T = sum(lens)
    need = _lib.load_seq().qspec_seq_hgrn2_chunk_bytes(len(lens), T, H, D, DV, _lib.DTYPE_BF16)
    assert need == nbytes or nbytes is None and need > 16
    segments = lengths(lens)
    meta, starts = table(segments)
    p, bias, lower, norm, state = inputs(T, H, D, DV, len(lens), 17)
    bias = bias / 8 + 2                                                         # a memory of some ten tokens
    want, want_state = want_of(p, bias, lower, norm, state, segments, H, D, DV)
    out = torch.empty(T, H * DV, dtype=torch.bfloat16, device="cuda")
    ops.seq_hgrn2(p, bias, lower, norm, state, torch.empty(T * H * (DV + 3 * D), device="cuda"), out, meta, H, D, DV, 1e-5, seg_starts=starts)
    assert ((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2e-5 * want.abs().max()).all()
    for s in range(len(lens)):                                                  # float32 sums with such a memory: 1.2e-7 to 1.6e-7 of the state in every form
        assert (state[s].double() - want_state[s]).norm() <= 6e-7 * want_state[s].norm()


@pytest.mark.parametrize("H,D,DV,lens", [(16, 128, 128, [300]), (4, 64, 64, [257, 256]), (8, 128, 64, [600]), (32, 64, 128, [500, 300]), (16, 128, 128, [150] * 3), (200, 128, 128, [60])])
def test_every_workspace_size(ops, H, D, DV, lens):
    """The bytes of both queries, one less of each, and none: whichever form that leads to, the same results."""
    from qspec_b200 import _lib
    lib, T = _lib.load_seq(), sum(lens)
    segments = lengths(lens)
    meta, starts = table(segments)
    p, bias, lower, norm, start = inputs(T, H, D, DV, len(lens), 23)
    bias = bias / 8 + 2
    want, want_state = want_of(p, bias, lower, norm, start, segments, H, D, DV)
    old, new = lib.qspec_seq_recurrence_chunk_bytes(len(lens), T, H, D, DV), lib.qspec_seq_hgrn2_chunk_bytes(len(lens), T, H, D, DV, _lib.DTYPE_BF16)
    assert new >= old and new > 0                                               # (the larger of both forms': rows may be unaligned)
    scratch = torch.empty(T * H * (DV + 3 * D), device="cuda")
    for nbytes in sorted({0, max(0, old - 1), old, new - 1, new}):
        ws = torch.full((nbytes + 64,), 255, dtype=torch.uint8, device="cuda")
        state, out = start.clone(), torch.full((T, H * DV), float("nan"), dtype=torch.bfloat16, device="cuda")
        rc = lib.qspec_seq_hgrn2_chunked(p.data_ptr(), p.shape[1], bias.data_ptr(), lower.data_ptr(), norm.data_ptr(), state.data_ptr(), scratch.data_ptr(), out.data_ptr(),
                                         meta.data_ptr(), starts.data_ptr(), len(lens), T, H, D, DV, 1e-5, _lib.DTYPE_BF16, ws.data_ptr() if nbytes else None, nbytes,
                                         torch.cuda.current_stream().cuda_stream)
        assert rc == 0 and bool((ws[nbytes:] == 255).all())
        assert ((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2e-5 * want.abs().max()).all()
        for s in range(len(lens)):
            assert (state[s].double() - want_state[s]).norm() <= 6e-7 * want_state[s].norm()
