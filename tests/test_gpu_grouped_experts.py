"""The grouped expert feed-forward (tcgen05 form) at the edges of its tiles: rows of an expert around 128, around 256 and at multiples of 16, widths and
expert sizes that are not multiples of a tile or a k-step, pairs without an expert, experts without a pair, more pairs and experts than the grouping keeps in registers."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _expected(h, gate_up, down, idx, E, F, act, limit):
    """64 bits, with the bfloat16 roundings that the call makes: of the projections, and of the activation between the products."""
    T, top = idx.shape
    out = torch.empty(T, top, h.shape[1], dtype=torch.float64, device="cuda")
    for e in range(-1, E + 1):
        t, c = (idx == e).nonzero(as_tuple=True)
        if t.numel() == 0:
            continue
        if e < 0 or e >= E:
            out[t, c] = h[t].double()
            continue
        z = (h[t].double() @ gate_up[e].double().T).bfloat16().double()
        if act == "relu2":
            y = z.clamp_min(0).square()
        elif act == "silu":
            y = z[:, :F] * torch.sigmoid(z[:, :F]) * z[:, F:]
        else:
            g, u = z[:, :F].clamp_max(limit), z[:, F:].clamp(-limit, limit)
            y = g * torch.sigmoid(1.702 * g) * (u + 1)
        out[t, c] = y.bfloat16().double() @ down[e].double().T
    return out


@pytest.mark.parametrize("T,top,E,W,F", [(1, 1, 1, 8, 8), (127, 1, 1, 64, 40), (128, 1, 2, 72, 128), (129, 1, 1, 200, 136), (300, 2, 3, 256, 264), (64, 4, 16, 1024, 512),
                                         (513, 4, 8, 136, 248), (5000, 4, 5, 64, 64), (700, 3, 1500, 32, 16), (2048, 2, 4, 512, 384)])
@pytest.mark.parametrize("act", ["silu", "gated", "relu2"])
def test_grouped_experts_match_64_bits(T, top, E, W, F, act):
    from qspec_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(T + W + F)
    h = torch.randn(T, W, generator=g, device="cuda").bfloat16()
    rows = F if act == "relu2" else 2 * F
    gate_up = (torch.randn(E, rows, W, generator=g, device="cuda") * W ** -0.5).bfloat16()
    down = (torch.randn(E, W, F, generator=g, device="cuda") * F ** -0.5).bfloat16()
    idx = torch.randint(-1, E + 1, (T, top), generator=g, device="cuda").int()           # -1 and E: no expert
    if E > 1:
        idx[idx == 1] = 0                                                                 # an expert without a pair
    out = torch.full((T, top, W), float("nan"), dtype=torch.bfloat16, device="cuda")
    want = _expected(h, gate_up, down, idx, E, F, act, 7.0)
    for _ in range(2):
        ops.moe_expert_grouped(h, gate_up, down, idx, out, E, F, 7.0, act=act)
    none = ((idx < 0) | (idx >= E))
    assert torch.equal(out[none], h[:, None].expand(T, top, W)[none])
    # A projection that float32 and 64-bit sums put on two sides of a rounding edge moves by 2^-8 of itself: a share of about 2^-23 * sqrt(W) / 2^-9 of them,
    # each moving the result by at most 2^-7 (square) * sqrt(share); the rounding of the result is 2^-9 of its own value. 2^-8 covers both in the 2-norm.
    assert torch.isfinite(out).all()
    assert (out.double() - want).norm() <= 2.0 ** -8 * want.norm()
    assert ops.moe_grouped_status() == 0


@pytest.mark.parametrize("rows", [[255], [256], [257], [272, 16, 1], [512, 513, 15], [240, 0, 496, 17], [769]])
@pytest.mark.parametrize("act", ["silu", "relu2"])
def test_rows_of_an_expert_around_its_tiles(rows, act):
    """Experts with exactly these rows: tiles of up to 256 rows, evenly divided, in multiples of 16."""
    from qspec_b200 import ops
    E, W, F, T = len(rows), 264, 136, sum(rows)
    g = torch.Generator(device="cuda").manual_seed(T)
    h = torch.randn(T, W, generator=g, device="cuda").bfloat16()
    gate_up = (torch.randn(E, F if act == "relu2" else 2 * F, W, generator=g, device="cuda") * W ** -0.5).bfloat16()
    down = (torch.randn(E, W, F, generator=g, device="cuda") * F ** -0.5).bfloat16()
    idx = torch.repeat_interleave(torch.arange(E), torch.tensor(rows))[torch.randperm(T, generator=torch.Generator().manual_seed(T))].int().cuda()[:, None].contiguous()
    out = torch.full((T, 1, W), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.moe_expert_grouped(h, gate_up, down, idx, out, E, F, 7.0, act=act)
    want = _expected(h, gate_up, down, idx, E, F, act, 7.0)
    assert torch.isfinite(out).all()
    assert ((out.double() - want).norm(dim=2) <= 2.0 ** -6 * want.norm(dim=2)).all()     # each row by itself: a few projections beside a rounding edge in 136
    assert (out.double() - want).norm() <= 2.0 ** -8 * want.norm()                         # (the bound of the test above)
    assert ops.moe_grouped_status() == 0
