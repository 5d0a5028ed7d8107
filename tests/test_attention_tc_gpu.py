"""tcgen05 flash attention (forward, dQ, dK/dV) against the fp32 PyTorch attention of the oracle model."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def near(got, ref, chain=True):
    """(ok, worst error / allowance, rule) under the suite's comparison rule (tests/tolerances.py): attention
    results pass through 16-bit probabilities, so 16-bit outputs take the "chain" rule of their type; fp32 outputs
    (the log-sum-exp) take the fp32 rule."""
    from tolerances import kind_of, worst
    k = kind_of(got.dtype, chain)
    ok, w, _ = worst(got, ref, k, floor=1.0)     # operands are N(0, 1): a gradient that cancels to zero keeps that scale
    return ok, w, k


def rnd(*shape, seed=0, dtype=torch.float16):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, device="cuda", generator=g).to(dtype)


CASES = [
    # B, T, H, KV, hd, window, segments
    (1, 128, 2, 2, 64, 0, False),
    (2, 512, 12, 4, 64, 0, True),
    (1, 300, 4, 2, 64, 0, False),
    (2, 200, 4, 1, 64, 37, True),
    (1, 260, 2, 1, 128, 0, True),
    (1, 1, 2, 2, 64, 0, False),
    (1, 1024, 4, 4, 64, 0, False),
    (8, 512, 12, 4, 64, 0, True),       # more work items than resident CTAs: every CTA walks several
    (8, 384, 16, 4, 64, 100, True),
    (16, 512, 8, 4, 64, 0, True),       # more key-tile items than SMs too (the dK/dV kernel walks several per CTA)
]


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,T,H,KV,hd,window,use_seg", CASES)
def test_tc_attention_matches_oracle(dt, B, T, H, KV, hd, window, use_seg):
    from ghassan_b200.models import reference as R
    from ghassan_b200.ops import _lib, kernels as K
    n = B * T
    scale = hd ** -0.5
    qk = rnd(n, (H + KV) * hd, seed=1, dtype=dt)          # q and k share a buffer, v lives in a wider one
    qkv = rnd(n, (H + 2 * KV) * hd, seed=2, dtype=dt)
    q, k, v = qk[:, :H * hd], qk[:, H * hd:], qkv[:, (H + KV) * hd:]
    seg = None
    if use_seg:
        seg = (torch.arange(T, device="cuda") // 97).repeat(B).to(torch.int32)
    lo = torch.empty(n, dtype=torch.int32, device="cuda")
    o = torch.empty(n, H * hd, dtype=dt, device="cuda")
    lse = torch.empty(n, H, device="cuda")
    K.attn_tc_fwd(q, k, v, o, lse, seg, lo, B, T, H, KV, hd, window, scale)
    _lib.check_status(what="attn_tc_fwd")
    qf, kf, vf = (t.float().clone().requires_grad_(True) for t in (q, k, v))
    ref = R.attention(qf.view(n, H, hd), kf.view(n, KV, hd), vf.view(n, KV, hd), B, T, scale, window, seg)
    ok, err, atol = near(o, ref.detach())
    assert ok, ("o", err, atol)
    g = rnd(n, H * hd, seed=3, dtype=dt)
    (ref * g.float()).sum().backward()
    dqk = torch.zeros_like(qk)
    dqkv = torch.zeros_like(qkv)
    delta = torch.empty(n, H, device="cuda")
    K.attn_tc_bwd(q, k, v, o, lse, seg, lo, g, delta, dqk[:, :H * hd], dqk[:, H * hd:], dqkv[:, (H + KV) * hd:], B, T, H,
                  KV, hd, window, scale)
    _lib.check_status(what="attn_tc_bwd")
    for got, want, name in ((dqk[:, :H * hd], qf.grad, "dq"), (dqk[:, H * hd:], kf.grad, "dk"),
                            (dqkv[:, (H + KV) * hd:], vf.grad, "dv")):
        ok, err, atol = near(got, want)
        assert ok, (name, err, atol)


def test_tc_attention_agrees_with_cuda_core_kernels():
    from ghassan_b200.ops import kernels as K
    B, T, H, KV, hd = 2, 384, 6, 2, 64
    n = B * T
    q, k, v = rnd(n, H * hd, seed=4), rnd(n, KV * hd, seed=5), rnd(n, KV * hd, seed=6)
    o1, o2 = torch.empty_like(q), torch.empty_like(q)
    l1, l2 = torch.empty(n, H, device="cuda"), torch.empty(n, H, device="cuda")
    lo = torch.empty(n, dtype=torch.int32, device="cuda")
    K.attn_fwd(q, k, v, o1, l1, None, B, T, H, KV, hd, 0, 0.125)
    K.attn_tc_fwd(q, k, v, o2, l2, None, lo, B, T, H, KV, hd, 0, 0.125)
    assert near(o2, o1)[0]
    assert near(l2, l1)[0]
    # bitwise reproducible from run to run
    o3 = torch.empty_like(q)
    K.attn_tc_fwd(q, k, v, o3, l2, None, lo, B, T, H, KV, hd, 0, 0.125)
    assert torch.equal(o2, o3)


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("use_seg", [False, True])
def test_tc_attention_forward_rescales_when_the_row_maximum_jumps(dt, use_seg):
    """The forward kernel keeps the output in tensor memory and rescales it only when a row's maximum has grown by
    more than 2^8 since it was last taken.  Keys that grow in magnitude along the sequence force that path in every
    later tile (unit-variance inputs never do); a second case makes only some rows of a warp jump."""
    from ghassan_b200.models import reference as R
    from ghassan_b200.ops import _lib, kernels as K
    B, T, H, KV, hd = 2, 512, 4, 2, 64
    n = B * T
    scale = hd ** -0.5
    for variant in range(2):
        q, k, v = rnd(n, H * hd, seed=11, dtype=dt), rnd(n, KV * hd, seed=12, dtype=dt), rnd(n, KV * hd, seed=13, dtype=dt)
        pos = torch.arange(T, device="cuda").repeat(B)
        if variant == 0:
            k = (k.float() * (1.0 + 5.0 * (pos // 128).float())[:, None]).to(dt)          # every tile louder than the last
        else:
            q = (q.float() * torch.where(pos % 7 == 0, 8.0, 1.0)[:, None]).to(dt)         # a few rows of each warp jump
            k = (k.float() * torch.where(pos >= 256, 4.0, 1.0)[:, None]).to(dt)
        seg = (pos // 200).to(torch.int32) if use_seg else None
        lo = torch.empty(n, dtype=torch.int32, device="cuda")
        o = torch.empty(n, H * hd, dtype=dt, device="cuda")
        lse = torch.empty(n, H, device="cuda")
        K.attn_tc_fwd(q, k, v, o, lse, seg, lo, B, T, H, KV, hd, 0, scale)
        _lib.check_status(what="attn_tc_fwd")
        ref = R.attention(q.float().view(n, H, hd), k.float().view(n, KV, hd), v.float().view(n, KV, hd), B, T, scale, 0, seg)
        ok, err, rule = near(o, ref)
        assert ok, ("o", variant, err, rule)
        sc = torch.einsum("bihd,bjhd->bhij", q.float().view(B, T, H, hd),
                          k.float().view(B, T, KV, hd).repeat_interleave(H // KV, dim=2)) * scale
        vis = pos[:T][None, :] <= pos[:T][:, None]
        if use_seg:
            vis = vis & ((pos[:T] // 200)[None, :] == (pos[:T] // 200)[:, None])
        want = torch.logsumexp(sc.masked_fill(~vis, float("-inf")), dim=-1).permute(0, 2, 1).reshape(n, H)
        ok, err, rule = near(lse, want, chain=False)
        assert ok, ("lse", variant, err, rule)


def test_tc_attention_leading_negative_segment_ids():
    """Rows with a negative segment id at the head of a sequence see every earlier key (the oracle's rule); the documents
    after them see only themselves."""
    from ghassan_b200.models import reference as R
    from ghassan_b200.ops import _lib, kernels as K
    B, T, H, KV, hd = 2, 300, 4, 2, 64
    n = B * T
    dt = torch.float16
    scale = hd ** -0.5
    q, k, v = rnd(n, H * hd, seed=21, dtype=dt), rnd(n, KV * hd, seed=22, dtype=dt), rnd(n, KV * hd, seed=23, dtype=dt)
    one = torch.cat([torch.full((40,), -1, device="cuda"), torch.arange(T - 40, device="cuda") // 97])
    seg = one.repeat(B).to(torch.int32)
    lo = torch.empty(n, dtype=torch.int32, device="cuda")
    o = torch.empty(n, H * hd, dtype=dt, device="cuda")
    lse = torch.empty(n, H, device="cuda")
    K.attn_tc_fwd(q, k, v, o, lse, seg, lo, B, T, H, KV, hd, 0, scale)
    _lib.check_status(what="attn_tc_fwd")
    assert int(lo.view(B, T)[:, :40].max()) == 0 and int(lo.view(B, T)[0, 40]) == 40
    assert bool((lo.view(B, T)[:, 1:] >= lo.view(B, T)[:, :-1]).all())       # non-decreasing along a sequence
    ref = R.attention(q.float().view(n, H, hd), k.float().view(n, KV, hd), v.float().view(n, KV, hd), B, T, scale, 0, seg)
    ok, err, rule = near(o, ref)
    assert ok, ("o", err, rule)


# dK/dV: a cluster per item where there are no more items (key tiles x sequences x kv heads) than SMs, whole items beyond; query steps of
# 64 that end with the key tile's documents; one to eight query heads per kv head
ITEM_CASES = [
    (1, 1000, 8, 1, 64, 0, True),
    (1, 129, 3, 1, 64, 0, False),
    (37, 128, 12, 4, 64, 0, True),      # 148 items: the last of the clusters
    (30, 130, 12, 4, 64, 0, True),      # 240: whole, a key tile of two rows
    (7, 600, 12, 6, 64, 200, True),
    (2, 700, 6, 2, 128, 0, True),
]


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,T,H,KV,hd,window,use_seg", ITEM_CASES)
def test_tc_attention_at_item_edges(dt, B, T, H, KV, hd, window, use_seg):
    test_tc_attention_matches_oracle(dt, B, T, H, KV, hd, window, use_seg)


def _lse(q, k, B, T, H, KV, scale, vis):
    """Log-sum-exp [B * T, H] of the visible scores, in fp64, a sequence at a time; ``vis`` is [B, T, T]."""
    hd = q.shape[1] // H
    out = []
    for b in range(B):
        s = torch.einsum("ihd,jhd->hij", q.view(B, T, H, hd)[b].double(), k.view(B, T, KV, hd)[b].double().repeat_interleave(H // KV, dim=1)) * scale
        out.append(torch.logsumexp(s.masked_fill(~vis[b], float("-inf")), dim=-1).t())
    return torch.cat(out).contiguous()


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,T,H,KV,hd", [(24, 700, 12, 4, 64), (8, 520, 16, 4, 128)])
def test_tc_attention_forward_many_uneven_items_per_block(dt, B, T, H, KV, hd):
    """Every CTA walks many work items whose numbers of key tiles differ (documents of uneven lengths), so its warps are an item apart
    now and then: outputs and log-sum-exp equal the oracle's and, bit for bit, those of every other run."""
    from ghassan_b200.models import reference as R
    from ghassan_b200.ops import _lib, kernels as K
    n, scale = B * T, hd ** -0.5
    q, k, v = rnd(n, H * hd, seed=31, dtype=dt), rnd(n, KV * hd, seed=32, dtype=dt), rnd(n, KV * hd, seed=33, dtype=dt)
    g = torch.Generator().manual_seed(34)
    seg = (torch.rand(B, T, generator=g) < torch.tensor([0.0, 0.003, 0.01, 0.1])[torch.arange(B) % 4, None]).cumsum(1).to(torch.int32).cuda()
    lo = torch.empty(n, dtype=torch.int32, device="cuda")
    first = None
    for _ in range(20):
        o, lse = torch.empty(n, H * hd, dtype=dt, device="cuda"), torch.empty(n, H, device="cuda")
        K.attn_tc_fwd(q, k, v, o, lse, seg.view(-1), lo, B, T, H, KV, hd, 0, scale)
        _lib.check_status(what="attn_tc_fwd")
        if first is None:
            first = (o, lse)
            ref = R.attention(q.float().view(n, H, hd), k.float().view(n, KV, hd), v.float().view(n, KV, hd), B, T, scale, 0, seg.view(-1))
            ok, err, rule = near(o, ref)
            assert ok, ("o", err, rule)
            ar = torch.arange(T, device="cuda")
            vis = (ar[None, :] <= ar[:, None])[None] & (seg[:, None, :] == seg[:, :, None])
            ok, err, rule = near(lse, _lse(q, k, B, T, H, KV, scale, vis).float(), chain=False)
            assert ok, ("lse", err, rule)
        assert torch.equal(o, first[0]) and torch.equal(lse, first[1])


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("T,H,KV,hd,use_seg", [(100, 2, 2, 64, False), (700, 4, 2, 64, True), (96, 2, 1, 128, False), (520, 4, 2, 128, True)])
def test_tc_attention_scores_of_thousands(dt, T, H, KV, hd, use_seg):
    """Row maxima of about 3,000 to 9,000 in log2 units (nothing bounds scores without a norm on queries and keys): the largest
    probability of a row still has to be stored as about 1.  Allowances are sums of absolute values times eps: 16-bit probabilities, score gradients
    and outputs (2^-10, bf16 2^-7), and the exponent's fp32 roundings (scores, log-sum-exp, their difference: 8 x 2^-23 of the score's terms)."""
    from ghassan_b200.ops import _lib, kernels as K
    B, scale, rep = 2, hd ** -0.5, H // KV
    n = B * T
    for top in (3000.0, 9000.0):
        amp = (top / 1.4427 / 3.0) ** 0.5                   # scores are N(0, amp^4): a row's largest is about three deviations
        q, k = ((rnd(n, m * hd, seed=40 + m, dtype=torch.float32) * amp).to(dt) for m in (H, KV))
        v, g = rnd(n, KV * hd, seed=51, dtype=dt), rnd(n, H * hd, seed=52, dtype=dt)
        seg = (torch.arange(T, device="cuda") // 150).repeat(B).to(torch.int32) if use_seg else None
        lo = torch.empty(n, dtype=torch.int32, device="cuda")
        o, lse, delta = torch.empty_like(q), torch.empty(n, H, device="cuda"), torch.empty(n, H, device="cuda")
        dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
        K.attn_tc_fwd(q, k, v, o, lse, seg, lo, B, T, H, KV, hd, 0, scale)
        K.attn_tc_bwd(q, k, v, o, lse, seg, lo, g, delta, dq, dk, dv, B, T, H, KV, hd, 0, scale)
        _lib.check_status(what="attention")
        ar = torch.arange(T, device="cuda")
        vis = ar[None, :] <= ar[:, None]
        if use_seg:
            vis = vis & (ar[None, :] // 150 == ar[:, None] // 150)
        heads = lambda t, m: t.double().view(B, T, m, hd).transpose(1, 2)
        Q, G, Ov = heads(q, H), heads(g, H), heads(o, H)
        Kh, V = (heads(t, KV).repeat_interleave(rep, dim=1) for t in (k, v))
        S = (Q @ Kh.transpose(2, 3) * scale).masked_fill(~vis, float("-inf"))
        P = torch.softmax(S, dim=-1)
        terms = float((Q.abs() @ Kh.abs().transpose(2, 3) * scale * vis).max())
        eps = (2.0 ** -10 if dt == torch.float16 else 2.0 ** -7) + 8 * 2.0 ** -23 * terms
        want = P @ V
        dP = G @ V.transpose(2, 3)
        dS = P * (dP - (P * dP).sum(-1, keepdim=True))
        aS = P * (G.abs() @ V.abs().transpose(2, 3) + (G.abs() * want.abs()).sum(-1, keepdim=True))
        fold = lambda t: t.view(B, KV, rep, T, hd).sum(2)
        tiny = 2.0 ** -24 * T                               # probabilities and score gradients below fp16's smallest step
        for name, got, ref, room in (("o", Ov, want, P @ V.abs()), ("dq", heads(dq, H), dS @ Kh * scale, aS @ Kh.abs() * scale),
                                     ("dk", heads(dk, KV), fold(dS.transpose(2, 3) @ Q) * scale, fold(aS.transpose(2, 3) @ Q.abs()) * scale),
                                     ("dv", heads(dv, KV), fold(P.transpose(2, 3) @ G), fold(P.transpose(2, 3) @ G.abs()))):
            mag = {"o": V, "dq": Kh, "dk": Q, "dv": G}[name].abs().max()
            worst = float(((got - ref).abs() / (eps * room + tiny * mag)).max())
            assert worst <= 1.0, (name, top, worst)
        err = float((heads(lse.repeat_interleave(hd, dim=1), H)[..., 0] - torch.logsumexp(S, dim=-1)).abs().max())
        assert err <= 8 * 2.0 ** -23 * terms, ("lse", top, err)


# Two CTAs an item: from four key tiles on while every CTA has an SM (74 items; 385 is the shortest), from ten on up to 148 items; windows bound the tiles.
# Documents, short windows and many short items have one CTA each and are here for the other side of the line.
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,T,H,KV,window,use_seg", [(1, 385, 3, 1, 0, False), (1, 1501, 12, 4, 0, False), (2, 700, 8, 2, 0, True), (1, 1000, 8, 2, 129, True),
                                                     (3, 512, 12, 4, 1, False), (1, 2304, 8, 2, 0, False), (1, 2305, 8, 2, 0, False), (1, 384, 4, 2, 0, False),
                                                     (1, 1000, 8, 2, 385, False), (1, 700, 3, 1, 386, False), (1, 2304, 8, 2, 1153, False), (1, 2304, 8, 2, 1154, False),
                                                     (1, 1153, 12, 4, 0, False), (1, 1152, 12, 4, 0, False)])
def test_tc_forward_with_shared_items(dt, B, T, H, KV, window, use_seg):
    """Rows whose keys all lie in one CTA's tiles, documents that begin in the second half, windows shorter than a tile; log-sum-exp included."""
    from ghassan_b200.ops import kernels as K
    hd = 64
    n = B * T
    g = torch.Generator(device="cuda").manual_seed(T + H)
    q, k, v = (torch.randn(n, h * hd, device="cuda", generator=g).to(dt) * s for h, s in ((H, 2.0), (KV, 2.0), (KV, 1.0)))
    seg = torch.arange(T, device="cuda", dtype=torch.int32).div(317, rounding_mode="floor").to(torch.int32).repeat(B) if use_seg else None
    o, lse = torch.full((n, H * hd), 7.0, device="cuda", dtype=dt), torch.full((n, H), 7.0, device="cuda")
    lo = torch.zeros(n, dtype=torch.int32, device="cuda")
    K.attn_tc_fwd(q, k, v, o, lse, seg, lo, B, T, H, KV, hd, window, hd ** -0.5)
    i, j = torch.arange(T, device="cuda")[:, None], torch.arange(T, device="cuda")[None, :]
    see = j <= i
    if window:
        see = see & (j > i - window)
    if use_seg:
        see = see & (seg[:T, None] == seg[None, :T])
    for b in range(B):
        rows = slice(b * T, (b + 1) * T)
        for h in range(H):
            s = (q[rows, h * hd:(h + 1) * hd].float() @ k[rows, (h * KV // H) * hd:(h * KV // H + 1) * hd].float().t() * hd ** -0.5).masked_fill(~see, float("-inf"))
            want = torch.softmax(s, -1) @ v[rows, (h * KV // H) * hd:(h * KV // H + 1) * hd].float()
            ok, worst = near(o[rows, h * hd:(h + 1) * hd], want)[:2]
            assert ok, (b, h, worst)
            assert float((lse[rows, h] - torch.logsumexp(s, -1)).abs().max()) <= 2e-3          # fp32, fast exponentials, values up to about 30


@pytest.mark.parametrize("B,T,H,KV,window,doc", [(1, 1501, 12, 4, 256, 0), (1, 1000, 8, 2, 0, 100), (4, 512, 8, 2, 0, 0), (1, 1024, 12, 4, 0, 0)])
def test_tc_forward_of_short_items_does_not_depend_on_the_batch(B, T, H, KV, window, doc):
    """Items that two CTAs would not make faster are worked on as they are in a large batch: the same bits."""
    from ghassan_b200.ops import kernels as K
    hd, many = 64, 8
    g = torch.Generator(device="cuda").manual_seed(T)
    qkv = torch.randn(B * T, (H + 2 * KV) * hd, device="cuda", generator=g).half()
    outs = []
    for n in (B, B * many):
        x = qkv.repeat(n // B, 1)
        seg = torch.arange(T, device="cuda", dtype=torch.int32).div(doc, rounding_mode="floor").to(torch.int32).repeat(n) if doc else None
        o, lse, lo = torch.empty(n * T, H * hd, device="cuda", dtype=torch.float16), torch.empty(n * T, H, device="cuda"), torch.zeros(n * T, dtype=torch.int32, device="cuda")
        K.attn_tc_fwd(x[:, :H * hd], x[:, H * hd:(H + KV) * hd], x[:, (H + KV) * hd:], o, lse, seg, lo, n, T, H, KV, hd, window, hd ** -0.5)
        outs.append((o[:B * T], lse[:B * T]))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
