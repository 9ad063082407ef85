"""The cluster form of the 28 x n rotation (csrc/hadamard_kernels.cu) on both sides of the rule that gives a block one warp or two, and as part
of a larger batch: bit for bit the oracle, and the same row whatever stands around it."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [256, 512, 1024])
@pytest.mark.parametrize("rows", [1, 2, 112, 113, 300])
def test_rotation_is_the_oracle_and_batch_invariant(n, rows):
    from oracle import qspec_oracle as O
    from qspec_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(rows * 7 + n)
    x = torch.randn(rows, 28 * n, generator=g, device="cuda").half()
    x[rows - 1, 5] = 300.0                                               # a row maximum that one CTA of the seven holds
    scale = 0.00835418701171875

    def run(part):
        m = part.shape[0]
        o, q, s = torch.empty_like(part), torch.empty(m, 14 * n, dtype=torch.int8, device="cuda"), torch.empty(m, dtype=torch.float16, device="cuda")
        ops.hadamard_k28(part, n, scale, out=o, out_q=q, scale_out=s)
        plain = torch.empty_like(part)
        ops.hadamard_k28(part, n, scale, out=plain)
        assert torch.equal(o, plain)
        return o, q, s
    o, q, s = run(x)
    for i in sorted({0, rows - 1}):
        for a, b in zip((o, q, s), run(x[i:i + 1].contiguous())):
            assert torch.equal(a[i:i + 1], b)
        np.testing.assert_array_equal(o[i:i + 1].cpu().numpy(), O.hadamard_k28(x[i:i + 1].cpu().numpy(), n, scale))


@pytest.mark.parametrize("rows", [1, 7, 32, 33])
@pytest.mark.parametrize("gated", [False, True])
def test_256_wide_rows_by_stores_and_by_bulk_copies(rows, gated):
    """Both sides of the row count up to which the blocks of n = 256 leave as stores, with and without the quantiser: a row is the same in any batch."""
    from qspec_b200 import ops
    n, scale = 256, 0.0118
    x = torch.randn(300, (2 if gated else 1) * 28 * n, generator=torch.Generator(device="cuda").manual_seed(rows), device="cuda").half()

    def run(part, quant, plain):
        m = part.shape[0]
        o = torch.empty(m, 28 * n, dtype=torch.float16, device="cuda") if plain else None
        q = torch.empty(m, 14 * n, dtype=torch.int8, device="cuda") if quant else None
        s = torch.empty(m, dtype=torch.float16, device="cuda") if quant else None
        ops.hadamard_k28(None if gated else part, n, scale, gate_up=part if gated else None, out=o, out_q=q, scale_out=s)
        return [t for t in (o, q, s) if t is not None]
    for quant, plain in ((True, False), (False, True), (True, True)):
        for a, b in zip(run(x[:rows].contiguous(), quant, plain), run(x, quant, plain)):
            assert torch.equal(a, b[:rows])


@pytest.mark.parametrize("n", [256, 512, 1024])
def test_quantised_values_are_the_quotients(n):
    """Rows from subnormal scales to the largest, a row of zeros, rows with infinite values and NaN: every value is that of the rounded division."""
    from qspec_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(40, 28 * n, generator=g, device="cuda")
    x = (x * torch.logspace(-7.5, 2.5, 40, device="cuda")[:, None]).half()
    x[3] = 0.0
    x[5, 77] = float("inf")
    x[7, 99] = float("nan")
    out = torch.empty_like(x)
    q = torch.empty(40, 14 * n, dtype=torch.int8, device="cuda")
    s = torch.empty(40, dtype=torch.float16, device="cuda")
    ops.hadamard_k28(x, n, 0.0118, out=out, out_q=q, scale_out=s)
    quotient = (out.float() / s.float()[:, None]).half().float()                       # an IEEE division, rounded to float16
    want = torch.where(quotient.isnan(), 0.0, quotient.round().clamp(-8, 7)).to(torch.int8)
    got = torch.stack(((q << 4) >> 4, q >> 4), -1).view(40, -1)
    assert torch.equal(got, want)
