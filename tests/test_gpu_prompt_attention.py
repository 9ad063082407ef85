"""The int4 decoder's attention over prompt portions (tensor-core tiles inside seq_attention and decode_attention) against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from qspec_b200 import ops
    return ops


def reference(qkv, ck, cv, pos, seq, Hq, Hkv, scale):
    T, rep = len(pos), Hq // Hkv
    q = qkv[:, :Hq * 128].double().view(T, Hq, 128)
    out = torch.zeros(T, Hq, 128, dtype=torch.float64, device=qkv.device)
    for t in range(T):
        n = int(pos[t]) + 1
        k = ck[int(seq[t]), :n].double().repeat_interleave(rep, 1)
        v = cv[int(seq[t]), :n].double().repeat_interleave(rep, 1)
        p = torch.softmax(torch.einsum("hd,jhd->hj", q[t], k) * scale, 1)
        out[t] = torch.einsum("hj,jhd->hd", p, v)
    return out.view(T, Hq * 128)


def batch(segments, Hq, Hkv, S, nseq, seed=0):
    """segments: (sequence, first position, tokens) in batch order."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    pos = torch.cat([torch.arange(p, p + n) for _, p, n in segments]).to(torch.int32)
    seq = torch.cat([torch.full((n,), s) for s, _, n in segments]).to(torch.int32)
    qkv = torch.randn(len(pos), (Hq + 2 * Hkv) * 128, generator=g, device="cuda").half()
    ck = torch.randn(nseq, S, Hkv, 128, generator=g, device="cuda").half()
    cv = torch.randn(nseq, S, Hkv, 128, generator=g, device="cuda").half()
    return qkv, ck, cv, pos.cuda(), seq.cuda()


@pytest.fixture(autouse=True)
def no_wait_was_given_up(ops):
    yield
    assert ops.attn_tile_timeouts() == 0


def check(got, want, most=5.0):
    """Every (token, head) by itself: half a unit in the last place of float16 of its largest value, and 2^-16 of the largest value in the
    cache, `most`: scores of up to 2^7 (units of log2) carry an error of a few 2^-17 out of float32 sums, and so do their weights."""
    err = (got.double() - want).abs().view(-1, 128).amax(1)
    bound = 2 ** -11 * want.abs().view(-1, 128).amax(1) + 2 ** -16 * most
    assert (err <= bound).all(), (err / bound).max().item()


def check_bf16(got, want, most):
    """The same for bfloat16 outputs (seven bits behind the leading one: half a unit in the last place is up to 2^-8 of a value) and weights
    of two bfloat16 terms (2^-17 of each)."""
    err = (got.double() - want).abs().view(-1, 128).amax(1)
    bound = 2 ** -8 * want.abs().view(-1, 128).amax(1) + 2 ** -15 * most
    assert (err <= bound).all(), (err / bound).max().item()


CASES = [
    (32, 8, 300, [(0, 0, 64)]),                                   # the longest portion that is not tiled
    (32, 8, 300, [(0, 0, 65)]),                                   # the shortest that is: a last tile of one token
    (32, 8, 300, [(0, 0, 128)]),                                  # exactly one block of keys in the last tile
    (32, 8, 300, [(1, 0, 129)]),                                  # a block and one key; tokens of five CTAs
    (32, 8, 1100, [(0, 250, 800)]),                               # rows of a thousand keys: values of a hundredth of the first rows'
    (32, 8, 512, [(0, 200, 150)]),                                # starts inside the cache
    (8, 8, 400, [(0, 5, 257)]),                                   # one head per group: 128 tokens a tile
    (40, 8, 300, [(0, 1, 77)]),                                   # five heads: rows left over in every tile
    (64, 8, 600, [(0, 300, 45), (1, 77, 33)]),                    # eight heads; two runs in one CTA
    (16, 8, 700, [(0, 500, 15), (1, 0, 1), (2, 30, 16), (3, 9, 40), (4, 650, 4)]),   # short runs beside long ones
    (32, 8, 256, [(3, 100, 20), (0, 7, 1), (1, 8, 1), (2, 9, 1), (4, 255, 1), (5, 0, 256)]),
    (32, 8, 1000, [(k, 10 * k, 4) for k in range(12)]),           # no run at all
]


@pytest.mark.parametrize("Hq,Hkv,S,segments", CASES)
def test_prompt_runs_match_float64(ops, Hq, Hkv, S, segments):
    nseq = 1 + max(s for s, _, _ in segments)
    qkv, ck, cv, pos, seq = batch(segments, Hq, Hkv, S, nseq)
    out = torch.full((len(pos), Hq * 128), float("nan"), dtype=torch.float16, device="cuda")
    ops.seq_attention(qkv, ck, cv, pos, seq, out, Hq, Hkv, 128, 128 ** -0.5)
    check(out, reference(qkv, ck, cv, pos, seq, Hq, Hkv, 128 ** -0.5))


@pytest.mark.parametrize("Hq,Hkv", [(8, 8), (16, 8), (32, 8), (40, 8), (64, 8)])
@pytest.mark.parametrize("segments", [
    [(0, 100, 64)],                                               # one sequence: every chunk its own CTA
    [(5, 7, 63)],
    [(3, 40, 1)],
    [(1, 250, 33), (0, 0, 31)],                                   # the numbering passes from the first 32 tokens to the others
    [(k % 9, 20 * (k % 9) + k // 9, 1) for k in range(64)],       # a sequence's tokens all over the batch
    [(k, 299 - 3 * k, 1 + k % 3) for k in range(30)],
])
def test_passes_of_up_to_64_tokens_are_one_launch(ops, Hq, Hkv, segments):
    from qspec_b200 import _lib
    qkv, ck, cv, pos, seq = batch(segments, Hq, Hkv, 310, 1 + max(s for s, _, _ in segments) + 40, seed=9)
    out = torch.full((len(pos), Hq * 128), float("nan"), dtype=torch.float16, device="cuda")
    before = _lib.load().qspec_launch_count()
    ops.seq_attention(qkv, ck, cv, pos, seq, out, Hq, Hkv, 128, 128 ** -0.5)
    assert _lib.load().qspec_launch_count() - before == 1
    check(out, reference(qkv, ck, cv, pos, seq, Hq, Hkv, 128 ** -0.5))


@pytest.mark.parametrize("Hq,Hkv", [(24, 8), (48, 3), (32, 32)])
def test_decode_attention_takes_long_runs_too(ops, Hq, Hkv):
    """Head counts that the one-launch attention block does not take; positions that jump inside a sequence are no run."""
    qkv, ck, cv, pos, seq = batch([(0, 3, 90), (1, 120, 1), (1, 50, 20), (1, 90, 3)], Hq, Hkv, 128, 2, seed=1)
    out = torch.full((len(pos), Hq * 128), float("nan"), dtype=torch.float16, device="cuda")
    ops.decode_attention(qkv, ck, cv, pos, seq, out, Hq, Hkv, 128, 0.1)
    check(out, reference(qkv, ck, cv, pos, seq, Hq, Hkv, 0.1))


def test_decode_attention_over_1024_tokens(ops):
    """Portions longer than seq_attention takes, beside decoding sequences."""
    qkv, ck, cv, pos, seq = batch([(1, 500, 1), (2, 70, 1), (0, 33, 1090), (3, 1100, 3)], 32, 8, 1200, 4, seed=6)
    out = torch.full((len(pos), 32 * 128), float("nan"), dtype=torch.float16, device="cuda")
    ops.decode_attention(qkv, ck, cv, pos, seq, out, 32, 8, 128, 128 ** -0.5)
    check(out, reference(qkv, ck, cv, pos, seq, 32, 8, 128 ** -0.5))


def test_a_token_sees_nothing_but_its_own_keys(ops):
    """Infinite values and keys at a later position of the same portion, NaN past the portion's end: earlier tokens stay finite."""
    qkv, ck, cv, pos, seq = batch([(0, 0, 100)], 32, 8, 200, 1, seed=2)
    cv[0, 60, :, 5] = float("inf")
    ck[0, 60, :, 0] = float("nan")
    ck[0, 100:] = float("nan")
    cv[0, 100:] = float("nan")
    out = torch.empty(100, 32 * 128, dtype=torch.float16, device="cuda")
    ops.seq_attention(qkv, ck, cv, pos, seq, out, 32, 8, 128, 128 ** -0.5)
    want = reference(qkv[:60], ck, cv, pos[:60], seq[:60], 32, 8, 128 ** -0.5)
    check(out[:60], want)
    assert not torch.isfinite(out[60:].view(40, 32, 128)[..., 5]).any()


@pytest.mark.parametrize("Hq,Hkv", [(32, 8), (40, 8)])
def test_infinite_values_and_scores_without_a_number(ops, Hq, Hkv):
    """One infinite value that every later row sees, one NaN in a query, one in a key: what float64 makes of them, column by column."""
    qkv, ck, cv, pos, seq = batch([(0, 150, 200)], Hq, Hkv, 400, 1, seed=15)
    cv[0, 40, 0, 7] = float("inf")
    cv[0, 200, 0, 7] = float("-inf")
    cv[0, 170, 1, 64] = float("nan")
    qkv[30, 2 * 128 + 3] = float("nan")                           # head 2 of token 30
    ck[0, 300, 2, 9] = float("nan")                               # key/value head 2 from position 300 on
    out = torch.empty(200, Hq * 128, dtype=torch.float16, device="cuda")
    ops.seq_attention(qkv, ck, cv, pos, seq, out, Hq, Hkv, 128, 128 ** -0.5)
    want = reference(qkv, ck, cv, pos, seq, Hq, Hkv, 128 ** -0.5)
    assert torch.equal(out.isnan(), want.isnan())
    assert torch.equal(out.isinf(), want.isinf()) and torch.equal(out[out.isinf()].sign().double(), want[want.isinf()].sign())
    fine = want.isfinite()
    check(torch.where(fine, out, 0), torch.where(fine, want, 0))


def test_hidden_keys_leave_no_trace(ops):
    """The same tokens with other keys and values at later positions and in the sequence that shares their tile: bit for bit the same rows.
    Their own values are small, so that even a remainder of a hidden value of 6e4 times the smallest normal weight would show."""
    segments = [(0, 0, 100), (1, 0, 28)]
    qkv, ck, cv, pos, seq = batch(segments, 32, 8, 200, 2, seed=11)
    cv[0, :60] *= 1e-3
    outs = []
    for k, size in enumerate((1.0, 6e4)):
        g = torch.Generator(device="cuda").manual_seed(20 + k)
        for part in (ck[0, 60:100], ck[1], qkv[60:100], qkv[100:]):
            part.copy_(3 * torch.randn(part.shape, generator=g, device="cuda"))
        for part in (cv[0, 60:100], cv[1]):
            part.copy_(size * (2 * torch.rand(part.shape, generator=g, device="cuda") - 1))
        out = torch.empty(128, 32 * 128, dtype=torch.float16, device="cuda")
        ops.seq_attention(qkv, ck, cv, pos, seq, out, 32, 8, 128, 128 ** -0.5)
        outs.append(out[:60])
    check(outs[0], reference(qkv[:60], ck, cv, pos[:60], seq[:60], 32, 8, 128 ** -0.5), most=1e-3 * 5)
    assert torch.equal(*outs)


def signs_that_cancel(p):
    """p [heads, keys] weights of one row -> values +-1 [heads, keys, 128] whose weighted sums nearly vanish: what is left of the output is
    the error of the weights."""
    g = torch.Generator(device="cuda").manual_seed(5)
    v = torch.where(torch.rand(*p.shape, 128, generator=g, device="cuda") < 0.5, -1.0, 1.0).double()
    for _ in range(40):                                           # turn the key whose part is closest to half of what is left
        left = torch.einsum("hj,hjd->hd", p, v)
        j = (left[:, None, :] - 2 * p[:, :, None] * v).abs().argmin(1, keepdim=True)
        turned = v.scatter(1, j, -v.gather(1, j))
        better = torch.einsum("hj,hjd->hd", p, turned).abs() < left.abs()
        v = torch.where(better[:, None, :], turned, v)
    return v


def split_error(w, dtype):
    """w minus its two-term split with both terms rounded."""
    hi = w.to(dtype).double()
    return w - hi - (w - hi).to(dtype).double()


def test_weights_keep_both_terms(ops):
    """float16: 1000 keys of comparable weights whose values cancel. Without the second term of the weights (2^-12 of each) the outputs would
    be off by 2^-12 / sqrt(3000), 4e-6; with it by float32 sums (2^-24 a key at most) and the smallest float16 numbers (2^-25)."""
    H, n = 8, 1000
    qkv, ck, cv, pos, seq = batch([(0, n - 40, 40)], H, H, n, 1, seed=12)
    q = qkv[-1, :H * 128].double().view(H, 128)
    p = torch.softmax(torch.einsum("hd,jhd->hj", q, ck[0].double()) * 128 ** -0.5, 1)
    cv[0] = signs_that_cancel(p).permute(1, 0, 2).half()
    out = torch.empty(40, H * 128, dtype=torch.float16, device="cuda")
    ops.seq_attention(qkv, ck, cv, pos, seq, out, H, H, 128, 128 ** -0.5)
    want = torch.einsum("hj,jhd->hd", p, cv[0].double())
    assert (out[-1].double().view(H, 128) - want).abs().max() <= 2 ** -21


def test_long_sums_do_not_drift(ops):
    """3000 keys whose values cancel: every accumulation of a product loses up to the accumulator's last bit. The sums stay within 2^-25 of the
    values, which four partial sums in registers also do (2^-25.8); 375 accumulations in a row on one accumulator do not (2^-24.1)."""
    H, n = 8, 3000
    qkv, ck, cv, pos, seq = batch([(0, n - 100, 100)], H, H, n, 1, seed=16)
    q = qkv[-1, :H * 128].double().view(H, 128)
    p = torch.softmax(torch.einsum("hd,jhd->hj", q, ck[0].double()) * 128 ** -0.5, 1)
    cv[0] = (signs_that_cancel(p) * 1024).permute(1, 0, 2).half()
    out = torch.empty(100, H * 128, dtype=torch.float16, device="cuda")
    ops.seq_attention(qkv, ck, cv, pos, seq, out, H, H, 128, 128 ** -0.5)
    err = out[-1].double().view(H, 128) - torch.einsum("hj,jhd->hd", p, cv[0].double())
    assert err.pow(2).mean().sqrt() <= 2 ** -25 * 1024, (err.pow(2).mean().sqrt() / 1024).item()


def test_window_weights_are_rounded_twice(ops):
    """bfloat16: as above; the error is that of a split with both terms rounded and of float32 sums and exponentials (half as much again). A
    leading term that is cut instead leaves a remainder, and an error, of twice the size."""
    H, n = 32, 1000
    g = torch.Generator(device="cuda").manual_seed(13)
    q = torch.randn(40, H, 128, generator=g, device="cuda").bfloat16().float()
    ck = torch.randn(1, n, H, 128, generator=g, device="cuda").bfloat16()
    s = torch.einsum("hd,jhd->hj", q[-1].double(), ck[0].double()) * 128 ** -0.5
    p = torch.softmax(s, 1)
    cv = signs_that_cancel(p).permute(1, 0, 2)[None].bfloat16().contiguous()
    meta = torch.stack([torch.zeros(40), torch.arange(n - 40, n), torch.zeros(40), torch.full((40,), 40), torch.zeros(40)]).to(torch.int32).cuda()
    out = torch.empty(40, H, 128, dtype=torch.bfloat16, device="cuda")
    ops.seq_window_attention_mma(q, ck, None, cv, out, meta, 4096, 128 ** -0.5, True)
    err = out[-1].double() - torch.einsum("hj,jhd->hd", p, cv[0].double())
    w = torch.exp(s - s.amax(1, keepdim=True))
    expected = (split_error(w, torch.bfloat16).pow(2).sum(1).sqrt() / w.sum(1)).pow(2).mean().sqrt()
    assert err.pow(2).mean().sqrt() <= 1.5 * expected, (err.pow(2).mean().sqrt() / expected).item()


def test_values_that_arrive_late(ops):
    """Caches that no kernel has read yet and an L2 full of something else: the last blocks' values come from DRAM, after the weights they
    are multiplied with. The outputs wait for both of the products that can then still be under way."""
    Hq, Hkv, S, n = 32, 8, 1200, 160
    junk = torch.empty(300 << 20, dtype=torch.uint8, device="cuda")
    for i in range(48):
        qkv, ck, cv, pos, seq = batch([(0, 1000, n)], Hq, Hkv, S, 1, seed=i)
        junk.fill_(i)
        out = torch.empty(n, Hq * 128, dtype=torch.float16, device="cuda")
        ops.seq_attention(qkv, ck, cv, pos, seq, out, Hq, Hkv, 128, 128 ** -0.5)
        first = out.clone()
        ops.seq_attention(qkv, ck, cv, pos, seq, out, Hq, Hkv, 128, 128 ** -0.5)
        assert torch.equal(first, out), i


@pytest.mark.parametrize("Hq,Hkv,segments", [
    (32, 8, [(0, 1900, 96)]),                                     # 16 blocks, the maximum moves in each
    (32, 8, [(0, 1000, 16), (1, 1500, 16), (2, 700, 40)]),        # two runs in a tile: the second's rows start when the first's are done
    (8, 8, [(1, 1400, 129), (0, 900, 127)]),
])
def test_the_maximum_moves_in_every_block(ops, Hq, Hkv, segments):
    """Scores that rise by more than the rescale threshold (8 in units of log2) from block to block: the outputs so far are scaled before
    each product. A product that did not wait for every warp's part of that shows in the rows against float64, or between repetitions."""
    S, nseq, scale = 2048, 1 + max(s for s, _, _ in segments), 128 ** -0.5
    qkv, ck, cv, pos, seq = batch(segments, Hq, Hkv, S, nseq, seed=7)
    direction = torch.randn(128, generator=torch.Generator(device="cuda").manual_seed(8), device="cuda")
    direction /= direction.norm()
    score = (torch.arange(S, device="cuda") - S / 2) * (8.3 / 128)                     # 8.3 (12 in units of log2) a block
    qkv[:, :Hq * 128] = (qkv[:, :Hq * 128].view(-1, Hq, 128) * 0.3 + 40 * direction).half().view(-1, Hq * 128)
    ck.copy_((ck * 0.3 + (score / (40 * scale))[None, :, None, None] * direction).half())
    first = None
    for _ in range(300):
        out = torch.full((len(pos), Hq * 128), float("nan"), dtype=torch.float16, device="cuda")
        ops.seq_attention(qkv, ck, cv, pos, seq, out, Hq, Hkv, 128, scale)
        if first is None:
            first = out
        assert torch.equal(first, out)
    check(first, reference(qkv, ck, cv, pos, seq, Hq, Hkv, scale))


def test_rows_leave_through_shared_memory_the_same_every_time(ops):
    """Every lane stores pieces of rows that other lanes of its warp have finished, repaired ones among them: the same bits in every call."""
    Hq, Hkv = 32, 8
    qkv, ck, cv, pos, seq = batch([(0, 100, 200), (1, 3, 90)], Hq, Hkv, 320, 2, seed=16)
    cv[0, 30, :, 5] = float("inf")
    cv[0, 250:, 1, 64:] = float("nan")
    first = None
    for _ in range(100):
        out = torch.full((len(pos), Hq * 128), 7.0, dtype=torch.float16, device="cuda")
        ops.seq_attention(qkv, ck, cv, pos, seq, out, Hq, Hkv, 128, 0.1)
        if first is None:
            first = out
        assert torch.equal(first.view(torch.int16), out.view(torch.int16))
    assert torch.isinf(first[:200].view(200, Hq, 128)[..., 5]).sum() >= 150 * Hq
    check(first[200:], reference(qkv[200:], ck, cv, pos[200:], seq[200:], Hq, Hkv, 0.1))


def test_positions_outside_the_cache(ops):
    """seq_attention shows such a token every row of the cache (past its end) or none (before its start: zeros), decode_attention does
    not store it; neither reads outside."""
    Hq, Hkv, S = 24, 8, 64
    qkv, ck, cv, pos, seq = batch([(0, 50, 40), (1, -20, 30)], Hq, Hkv, S, 2, seed=4)
    out = torch.full((70, Hq * 128), 7.0, dtype=torch.float16, device="cuda")
    ops.decode_attention(qkv, ck, cv, pos, seq, out, Hq, Hkv, 128, 0.1)
    ok = (pos >= 0) & (pos < S)
    check(out[ok], reference(qkv[ok], ck, cv, pos[ok], seq[ok], Hq, Hkv, 0.1))
    assert (out[~ok] == 7.0).all()
    for segments in ([(0, 50, 40), (1, -20, 30)], [(0, 50, 30), (1, -15, 22)]):                   # tiles; a CTA per chunk
        qkv, ck, cv, pos, seq = batch(segments, 16, 8, S, 2, seed=5)
        out = torch.full((len(pos), 2048), 7.0, dtype=torch.float16, device="cuda")
        ops.seq_attention(qkv, ck, cv, pos, seq, out, 16, 8, 128, 0.1)
        seen = pos >= 0
        check(out[seen], reference(qkv[seen], ck, cv, pos[seen].clamp(max=S - 1), seq[seen], 16, 8, 0.1))
        assert (out[~seen] == 0).all()


@pytest.mark.parametrize("Hq", [16, 32])
@pytest.mark.parametrize("others", [[], [(1, 0, 150)]])
def test_tiles_without_a_key(ops, Hq, others):
    """Whole tiles whose tokens all stand before the cache's start, by themselves and beside tiles with keys: no query may be left in the rows that such a
    tile stores, however late a warp's queries come."""
    from qspec_b200 import _lib
    qkv, ck, cv, pos, seq = batch([(0, -200, 200)] + others, Hq, 8, 256, 2, seed=21)
    want = reference(qkv[200:], ck, cv, pos[200:], seq[200:], Hq, 8, 0.1)
    for _ in range(50):
        out = torch.full((len(pos), Hq * 128), 7.0, dtype=torch.float16, device="cuda")
        ops.seq_attention(qkv, ck, cv, pos, seq, out, Hq, 8, 128, 0.1)
        assert (out[:200] == 0).all()
        check(out[200:], want)
    # the window form: 0 / 0 without a sink, zeros with one, gated or not
    q = qkv[:, :Hq * 128].float().reshape(len(pos), Hq, 128)
    start = torch.tensor([0] * 200 + [200] * (len(pos) - 200), dtype=torch.int32, device="cuda")
    end = torch.tensor([200] * 200 + [len(pos)] * (len(pos) - 200), dtype=torch.int32, device="cuda")
    meta = torch.stack([seq, pos, start, end, 0 * pos]).contiguous()
    gate, sink = torch.randn(len(pos), Hq * 128, device="cuda").bfloat16(), torch.randn(Hq, device="cuda")
    for g, s in ((None, None), (gate, None), (None, sink), (gate, sink)):
        out = torch.full((len(pos), Hq, 128), 7.0, dtype=torch.bfloat16, device="cuda")
        before = _lib.load_seq().qspec_launch_count()
        ops.seq_window_attention_mma(q, ck.bfloat16(), None, cv.bfloat16(), out, meta, 1000, 0.1, True, sink=s, gate=g)
        assert _lib.load_seq().qspec_launch_count() - before == 2                       # tiles, and the kernel beside them
        assert torch.isnan(out[:200]).all() if s is None else (out[:200] == 0).all()
        assert torch.isfinite(out[200:]).all()


def test_far_apart_scores(ops):
    """Scores that grow along the sequence (the running maximum moves in every block) and a first key that outweighs all others."""
    qkv, ck, cv, pos, seq = batch([(0, 0, 300)], 8, 8, 300, 1, seed=3)
    qkv[:, :1024] = 1.0
    ramp = torch.linspace(-4, 4, 300, device="cuda").half()
    ck[0] = ramp[:, None, None].expand(300, 8, 128)
    ck[0, 0, 0] = 6.0
    out = torch.empty(300, 1024, dtype=torch.float16, device="cuda")
    ops.seq_attention(qkv, ck, cv, pos, seq, out, 8, 8, 128, 128 ** -0.5)
    check(out, reference(qkv, ck, cv, pos, seq, 8, 8, 128 ** -0.5))


@pytest.mark.parametrize("form", ["seq", "decode", "window", "sink"])
def test_rows_without_a_weight(ops, form):
    """Every score of the first 20 tokens is -inf: what softmax makes of it, 0 / 0, where the forms for few tokens say so (decode_attention,
    window attention without a sink), zeros where they say that."""
    T, S, dtype = 64, 100, torch.float16 if form in ("seq", "decode") else torch.bfloat16
    Hq, Hkv = (24, 8) if form == "decode" else (16, 8)
    qkv, ck, cv, pos, seq = batch([(0, 0, T)], Hq, Hkv, S, 1, seed=14)
    qkv[:, :Hq * 128:128] = 1.0
    ck, cv = ck.to(dtype), cv.to(dtype)
    ck[0, :20, :, 0] = float("-inf")
    if form in ("seq", "decode"):
        out = torch.full((T, Hq * 128), 7.0, dtype=dtype, device="cuda")
        (ops.seq_attention if form == "seq" else ops.decode_attention)(qkv, ck, cv, pos, seq, out, Hq, Hkv, 128, 0.1)
    else:
        out = torch.full((T, Hq, 128), 7.0, dtype=dtype, device="cuda")
        meta = torch.stack([seq, pos, 0 * pos, 0 * pos + T, 0 * pos]).contiguous()
        sink = torch.zeros(Hq, device="cuda") if form == "sink" else None
        ops.seq_window_attention_mma(qkv[:, :Hq * 128].float().reshape(T, Hq, 128), ck, None, cv, out, meta, 1000, 0.1, True, sink=sink)
    assert torch.isfinite(out[20:]).all()
    assert out[:20].isnan().all() if form in ("decode", "window") else (out[:20] == 0).all()


# ---- the same tiles in the sequence-mixer library: bfloat16, rings, window, sink, gates ---------------------------------------------
@pytest.mark.parametrize("H,G,window,cap,segments,gate,sink", [
    (16, 4, 40, 200, [(0, 150, 70)], "each", True),                    # the ring wraps inside a block, inside the portion
    (8, 8, 1000, 600, [(1, 0, 129), (0, 300, 5)], None, True),         # window longer than anything held; two sequences in one tile
    (12, 4, 16, 300, [(2, 1000, 33), (0, 3, 1), (1, 77, 64)], "head", False),   # three heads per group: rows left over
    (32, 2, 129, 400, [(0, 255, 17), (1, 256, 18)], "each", False),
])
def test_window_tiles_match_float64(ops, H, G, window, cap, segments, gate, sink):
    g = torch.Generator(device="cuda").manual_seed(H + window)
    slots = 1 + max(s for s, _, _ in segments)
    pos = torch.cat([torch.arange(p, p + n) for _, p, n in segments])
    slot = torch.cat([torch.full((n,), s) for s, _, n in segments])
    T = len(pos)
    begin = torch.cat([torch.full((n,), sum(m for _, _, m in segments[:i])) for i, (_, _, n) in enumerate(segments)])
    end = torch.cat([torch.full((n,), sum(m for _, _, m in segments[:i + 1])) for i, (_, _, n) in enumerate(segments)])
    meta = torch.stack([slot, pos, begin, end, torch.zeros(T, dtype=torch.int64)]).to(torch.int32).cuda()
    q = torch.randn(T, H, 128, generator=g, device="cuda")
    ck = torch.full((slots, cap, G, 128), float("nan"), dtype=torch.bfloat16, device="cuda")      # rows that nobody wrote must not matter
    cv = torch.full_like(ck, float("inf"))
    for s, p, n in segments:
        rows = torch.arange(max(0, p - window + 1), p + n) % cap
        ck[s, rows] = torch.randn(len(rows), G, 128, generator=g, device="cuda").bfloat16()
        cv[s, rows] = torch.randn(len(rows), G, 128, generator=g, device="cuda").bfloat16()
    gt = torch.randn(T, H if gate == "head" else H * 128, generator=g, device="cuda").bfloat16() if gate else None
    sk = torch.randn(H, generator=g, device="cuda") if sink else None
    wide = torch.zeros(T, H * 128 + 64, dtype=torch.bfloat16, device="cuda")                      # rows with a stride of their own
    out = wide[:, :H * 128].view(T, H, 128)
    ops.seq_window_attention_mma(q, ck, None, cv, out, meta, window, 0.07, True, sink=sk, gate=gt, gate_per_head=gate == "head", out_scale=0.5)
    want = torch.zeros(T, H, 128, dtype=torch.float64, device="cuda")
    for t in range(T):
        rows = torch.arange(max(0, int(pos[t]) - window + 1), int(pos[t]) + 1, device="cuda") % cap
        k = ck[int(slot[t]), rows].double().repeat_interleave(H // G, 1)
        v = cv[int(slot[t]), rows].double().repeat_interleave(H // G, 1)
        s = torch.einsum("hd,jhd->hj", q[t].bfloat16().double(), k) * 0.07                        # the product takes bfloat16 queries
        if sink:
            s = torch.cat([s, sk.double()[:, None]], 1)
        want[t] = torch.einsum("hj,jhd->hd", torch.softmax(s, 1)[:, :len(rows)], v) * 0.5
    if gate:
        z = torch.sigmoid(gt.double())
        want *= z[:, :, None] if gate == "head" else z.view(T, H, 128)
    check_bf16(out, want, most=0.5 * 5)
    assert float(wide[:, H * 128:].abs().max()) == 0.0


@pytest.mark.parametrize("segments", [
    [(k, 700 + 5 * k, 1) for k in range(37)] + [(40, 300, 170)],               # decoding sequences in front of a prompt
    [(0, 0, 15), (1, 900, 16), (2, 40, 17), (3, 1500, 3), (4, 7, 1)],           # both sides of the line
    [(0, 500, 4), (1, 0, 2)],                                                   # fewer tokens than a run
    [(k, 620 + 11 * k, 2 + k % 14) for k in range(30)],                         # pieces of every size, more than there are CTAs in a row
    [(0, 10, 20), (0, 30, 5), (1, 0, 16)],                                      # a segment that continues its neighbour
])
@pytest.mark.parametrize("H,G", [(16, 4), (12, 4), (16, 1), (32, 1)])            # 32 heads per group: no form with heads as rows
def test_window_of_mixed_steps(ops, H, G, segments):
    """Prompt portions beside decoding sequences: every token once, whichever form takes it."""
    g = torch.Generator(device="cuda").manual_seed(31)
    window, cap = 600, 900
    slots = 1 + max(s for s, _, _ in segments)
    meta, at = [], 0
    for s, p0, n in segments:
        meta += [(s, p0 + i, at, at + n, 0) for i in range(n)]
        at += n
    meta = torch.tensor(meta, dtype=torch.int32).T.contiguous().cuda()
    q = torch.randn(at, H, 128, generator=g, device="cuda")
    ck = torch.randn(slots, cap, G, 128, generator=g, device="cuda").bfloat16()
    cv = torch.randn(slots, cap, G, 128, generator=g, device="cuda").bfloat16()
    sink = torch.randn(H, generator=g, device="cuda")
    for rows in (1, 2) if min(n for _, _, n in segments) >= 16 else (1,):
        out = torch.full((at, H, 128), float("nan"), dtype=torch.bfloat16, device="cuda")
        ops.seq_window_attention_mma(q, ck, None, cv, out, meta, window, 0.09, rows, sink=sink)
        for t in range(at):
            slot, pos = int(meta[0, t]), int(meta[1, t])
            j = torch.arange(max(0, pos - window + 1), pos + 1, device="cuda") % cap
            s = torch.einsum("hd,jhd->hj", q[t].bfloat16().double(), ck[slot, j].double().repeat_interleave(H // G, 1)) * 0.09
            w = torch.softmax(torch.cat([s, sink.double()[:, None]], 1), 1)[:, :-1]
            check_bf16(out[t], torch.einsum("hj,jhd->hd", w, cv[slot, j].double().repeat_interleave(H // G, 1)), most=5.0)
