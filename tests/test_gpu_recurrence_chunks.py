"""The gated and the scalar-decay recurrence over long segments (chunks side by side) against float64, token by token."""
import pytest
import torch

pytestmark = pytest.mark.gpu
F64 = torch.float64


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from qspec_b200 import ops
    return ops


def table(segments):
    rows, starts, at = [], [], 0
    for slot, p0, n in segments:
        starts.append(at)
        rows += [(slot, p0 + k, at, at + n, 0) for k in range(n)]
        at += n
    return torch.tensor(rows, dtype=torch.int32).T.contiguous().cuda(), torch.tensor(starts, dtype=torch.int32).cuda()


def walk(q, f, k, v, segments, state):
    """S <- diag(f) S + k v^T, o = S^T q over every segment; `state` [slots, H, D, DV] is updated."""
    out = torch.zeros(q.shape[0], q.shape[1], v.shape[-1], dtype=F64, device="cuda")
    at = 0
    for slot, p0, n in segments:
        S = state[slot].clone() if p0 > 0 else torch.zeros_like(state[slot])
        for t in range(at, at + n):
            S = f[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
            out[t] = torch.einsum("hd,hdv->hv", q[t], S)
        state[slot] = S
        at += n
    return out


CASES = [
    # H, D, DV, segments (slot, first position, tokens)
    (2, 128, 128, [(0, 0, 256)]),                      # whole chunks of the smallest size
    (3, 64, 64, [(1, 7, 257)]),                        # a last chunk of one token; a state carried in
    (2, 128, 64, [(0, 0, 500), (2, 40, 129)]),         # blocks and chunks cut short, two segments
    (40, 64, 128, [(0, 0, 2000)]),                     # chunks longer than the smallest
    (1, 128, 128, [(2, 0, 900), (0, 3, 5), (1, 90, 33)]),   # a segment within one chunk beside a long one
]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,D,DV,segments", CASES)
def test_gated_recurrence(ops, H, D, DV, segments, dtype):
    from qspec_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(D + DV + H)
    meta, starts = table(segments)
    T = meta.shape[1]
    assert _lib.load_seq().qspec_seq_recurrence_chunk_bytes(len(segments), T, H, D, DV) > 0
    p = torch.randn(T, 2 * H * D + H * DV, generator=g, device="cuda").to(dtype)
    bias = torch.randn(H * D, generator=g, device="cuda") * 3          # decays from nearly 0 to nearly 1
    lower = torch.rand(H * D, generator=g, device="cuda") * (torch.rand(H * D, generator=g, device="cuda") < 0.5)
    norm = torch.randn(DV, generator=g, device="cuda")
    state = torch.randn(3, H, D, DV, generator=g, device="cuda")
    for slot, p0, _ in segments:
        if p0 == 0:
            state[slot] = float("nan")                                  # a slot's leftovers do not matter at position 0
    want_state = state.double()
    z = p.double()
    zq, zf, v = z[:, :H * D], z[:, H * D:2 * H * D], z[:, 2 * H * D:].view(T, H, DV)
    q = (zq * torch.sigmoid(zq)).view(T, H, D)
    f = (lower.double() + (1 - lower.double()) * torch.sigmoid(zf + bias.double())).view(T, H, D)
    o = walk(q, f, 1 - f, v, segments, want_state)
    want = o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-5) * norm.double()
    out = torch.empty(T, H * DV, dtype=dtype, device="cuda")
    ops.seq_hgrn2(p, bias, lower, norm, state, torch.empty(T * H * (DV + 3 * D), device="cuda"), out, meta, H, D, DV, 1e-5, seg_starts=starts)
    # float32 sums of D and of up to 2000 decayed terms; the gates' own rounding (2e-7) grows along the state's memory
    tol = 2e-5 if dtype == torch.float32 else 2 ** -8
    assert (out.double().view(T, H, DV) - want).abs().max() <= tol * want.abs().max()
    for slot, _, _ in segments:
        assert (state[slot].double() - want_state[slot]).abs().max() <= 2e-5 * want_state[slot].abs().max()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,D,DV,segments", CASES)
def test_scalar_decay_recurrence(ops, H, D, DV, segments, dtype):
    g = torch.Generator(device="cuda").manual_seed(D + DV + H + 1)
    meta, starts = table(segments)
    T = meta.shape[1]
    p = torch.randn(T, 2 * H * (D + DV), generator=g, device="cuda").to(dtype)
    decay = torch.rand(H, generator=g, device="cuda") * 0.5 + 0.5
    decay[0] = 0.97
    norm = torch.randn(H * DV, generator=g, device="cuda")
    state = torch.randn(3, H, D, DV, generator=g, device="cuda")
    want_state = state.double()
    z = p.double()
    s = z * torch.sigmoid(z)
    q, k, v = s[:, :H * D].view(T, H, D), s[:, H * D:2 * H * D].view(T, H, D), s[:, 2 * H * D:2 * H * D + H * DV].view(T, H, DV)
    o = walk(q, decay.double()[None, :, None].expand(T, H, D), k, v, segments, want_state).reshape(T, H * DV)
    want = o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-5) * norm.double() * torch.sigmoid(z[:, 2 * H * D + H * DV:])
    out = torch.empty(T, H * DV, dtype=dtype, device="cuda")
    ops.seq_lightning(p, decay, norm, state, torch.empty(T * H * (DV + 2 * D), device="cuda"), out, meta, H, D, DV, 1e-5, seg_starts=starts)
    tol = 2e-5 if dtype == torch.float32 else 2 ** -8
    assert (out.double() - want).abs().max() <= tol * want.abs().max()
    for slot, _, _ in segments:
        assert (state[slot].double() - want_state[slot]).abs().max() <= 2e-5 * want_state[slot].abs().max()


@pytest.mark.parametrize("H,D,DV,segments,gated,scalar", [
    (64, 64, 64, [(0, 0, 300), (1, 5, 300), (2, 0, 300), (3, 9, 300)], True, False),   # the scalar decay's walk is the faster one here
    (32, 128, 128, [(0, 0, 300)], False, False),                                       # and both are here
    (16, 128, 64, [(0, 3, 700)], True, True),
])
def test_both_sides_of_the_rule(ops, H, D, DV, segments, gated, scalar):
    """Which form is taken, and that the scalar decay gives the same on either side."""
    from qspec_b200 import _lib
    meta, starts = table(segments)
    T, lib = meta.shape[1], _lib.load_seq()
    assert (lib.qspec_seq_recurrence_chunk_bytes(len(segments), T, H, D, DV) > 0) == gated
    assert (lib.qspec_seq_lightning_chunk_bytes(len(segments), T, H, D, DV) > 0) == scalar
    g = torch.Generator(device="cuda").manual_seed(H)
    p = torch.randn(T, 2 * H * (D + DV), generator=g, device="cuda")
    decay, norm = torch.rand(H, generator=g, device="cuda") * 0.5 + 0.5, torch.randn(H * DV, generator=g, device="cuda")
    state = torch.randn(len(segments), H, D, DV, generator=g, device="cuda")
    want_state, z = state.double(), p.double()
    s = z * torch.sigmoid(z)
    q, k, v = s[:, :H * D].view(T, H, D), s[:, H * D:2 * H * D].view(T, H, D), s[:, 2 * H * D:2 * H * D + H * DV].view(T, H, DV)
    o = walk(q, decay.double()[None, :, None].expand(T, H, D), k, v, segments, want_state).reshape(T, H * DV)
    want = o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-5) * norm.double() * torch.sigmoid(z[:, 2 * H * D + H * DV:])
    out = torch.empty(T, H * DV, device="cuda")
    ops.seq_lightning(p, decay, norm, state, torch.empty(T * H * (DV + 2 * D), device="cuda"), out, meta, H, D, DV, 1e-5, seg_starts=starts)
    assert (out.double() - want).abs().max() <= 2e-5 * want.abs().max()
    assert (state.double() - want_state).abs().max() <= 2e-5 * want_state.abs().max()
