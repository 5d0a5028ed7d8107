"""All tokens of a small batch through all experts (``gemm_skinny_sm100.cu``) and the norm + router kernel ahead of it, against fp32."""
import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = [  # tokens, width, experts, picks, shared, expert width: tile edges of 8, 32 and 128 rows, 32 / 64 columns, clusters over K, more experts than warps
    (1, 64, 2, 2, False, 64), (7, 256, 4, 2, True, 64), (8, 512, 8, 2, True, 512), (31, 768, 8, 4, True, 192), (33, 776, 3, 1, False, 128),
    (64, 256, 12, 3, True, 64), (100, 1032, 40, 8, False, 64), (128, 768, 8, 2, True, 768)]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(str(int(x)) for x in c))
def test_experts_few(case, dtype):
    from ghassan_b200.ops import _lib, decode as D, gemm as G
    B, d, ne, top, shared, E = case
    g = torch.Generator(device="cuda").manual_seed(B * d)
    n = lambda *s: torch.randn(s, device="cuda", generator=g)
    x, norm_w, router, bias = n(B, d), 1.0 + 0.1 * n(d), n(ne, d) * d ** -0.5, 0.01 * n(ne)
    ne1 = ne + int(shared)
    gate, up, down = (n(ne1, E, d) * d ** -0.5).to(dtype), (n(ne1, E, d) * d ** -0.5).to(dtype), (n(ne1, d, E) * E ** -0.5).to(dtype)
    eps = torch.finfo(dtype).eps
    x16, weights = torch.empty(B, d, device="cuda", dtype=dtype), torch.full((B, ne1), 7.0, device="cuda")
    D.norm_route_few(x, norm_w, 1e-5, router, bias, top, shared, x16, weights)
    want16 = x * torch.rsqrt(x.pow(2).mean(1, keepdim=True) + 1e-5) * norm_w
    alone = torch.empty_like(x16)
    D.norm_few(x, norm_w, 1e-5, alone)
    assert torch.equal(alone, x16)
    assert float((x16.float() - want16).abs().max()) <= eps * float(want16.abs().max())          # half a unit in the last place, and the fp32 norm
    p = torch.softmax(x16.float() @ router.t(), 1)
    pick = (p + bias).topk(top, 1).indices
    want_w = torch.zeros(B, ne, device="cuda").scatter_(1, pick, p.gather(1, pick))
    want_w /= want_w.sum(1, keepdim=True)
    near = (p + bias).sort(1, descending=True).values
    clear = torch.ones(B, dtype=torch.bool, device="cuda") if top == ne else near[:, top - 1] - near[:, top] > 1e-4        # no tie in the last bits
    assert int(clear.sum()) >= B // 2
    assert float((weights[:, :ne] - want_w)[clear].abs().max()) <= 1e-5
    assert not shared or bool((weights[:, ne] == 1.0).all())
    act, out, resid = torch.full((B, ne1 * E), 3.0, device="cuda", dtype=dtype), torch.empty(B, d, device="cuda"), n(B, d)
    w_gu = G.interleave_gate_up(gate, up).reshape(ne1 * 2 * E, d)
    G.experts_few(x16, w_gu, down.reshape(ne1 * d, E), weights, act, out, resid)
    _lib.check_status(what="experts_few")
    h = x16.float()
    want_act = torch.stack([torch.nn.functional.silu(h @ gate[e].float().t()) * (h @ up[e].float().t()) * weights[:, e:e + 1] for e in range(ne1)], 1)
    assert float((act.float().view(B, ne1, E) - want_act).abs().max()) <= eps * float(want_act.abs().max())
    assert bool((act.view(B, ne1, E)[weights == 0] == 0).all())
    want = resid + torch.einsum("bek,edk->bd", act.float().view(B, ne1, E), down.float())
    assert float((out - want).abs().max()) <= 2e-5 * float(want.abs().max()) + 1e-6 * (ne1 * E) ** 0.5       # fp32 sums in another order


def test_unchosen_expert_does_not_matter():
    """The gate and up rows of an expert that no token has chosen may hold infinities."""
    from ghassan_b200.ops import gemm as G
    B, d, ne, E = 16, 256, 4, 64
    g = torch.Generator(device="cuda").manual_seed(5)
    h = torch.randn(B, d, device="cuda", generator=g).half()
    w_gu = (torch.randn(ne * 2 * E, d, device="cuda", generator=g) * 0.05).half()
    down = (torch.randn(ne * d, E, device="cuda", generator=g) * 0.1).half()
    w_gu[2 * E:4 * E] = float("inf")
    weights = torch.rand(B, ne, device="cuda", generator=g)
    weights[:, 1] = 0.0
    act, out = torch.empty(B, ne * E, device="cuda", dtype=torch.float16), torch.empty(B, d, device="cuda")
    G.experts_few(h, w_gu, down, weights, act, out, torch.zeros(B, d, device="cuda"))
    assert bool(torch.isfinite(out).all()) and bool((act[:, E:2 * E] == 0).all())


@pytest.mark.parametrize("M,N,K", [(1, 64, 64), (9, 256, 1024), (32, 2816, 1024), (33, 192, 200), (100, 2816, 1024), (128, 4736, 320)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_swiglu_of_few_rows(M, N, K, dtype):
    from ghassan_b200.ops import gemm as G
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a, gate, up = (torch.randn(*s, device="cuda", generator=g).mul(k).to(dtype) for s, k in (((M, K), 1.0), ((N, K), K ** -0.5), ((N, K), K ** -0.5)))
    out = torch.full((M, N), 3.0, device="cuda", dtype=dtype)
    assert G.swiglu_skinny_ok(M, 2 * N, out)
    G.gemm_swiglu(a, G.interleave_gate_up(gate, up), act_out=out)
    want = torch.nn.functional.silu(a.float() @ gate.float().t()) * (a.float() @ up.float().t())
    assert float((out.float() - want).abs().max()) <= torch.finfo(dtype).eps * float(want.abs().max())


@pytest.mark.parametrize("M,n1,n2,K", [(1, 8, 8, 64), (31, 136, 248, 512), (32, 1536, 2816, 1024), (64, 1824, 512, 328), (128, 64, 64, 1024)])
def test_two_outputs_of_few_rows(M, n1, n2, K):
    from ghassan_b200.ops import gemm as G
    g = torch.Generator(device="cuda").manual_seed(M + n1)
    a, w = torch.randn(M, K, device="cuda", generator=g).bfloat16(), (torch.randn(n1 + n2, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    out1, both = torch.full((M, n1), 3.0, device="cuda", dtype=torch.bfloat16), torch.full((M, 8 + n2), 3.0, device="cuda", dtype=torch.bfloat16)
    assert G.gemm_two(a, w, n1, out1, both[:, 8:])
    want = a.float() @ w.float().t()
    up = want[:, n1:].clamp(min=0) ** 2
    eps = torch.finfo(torch.bfloat16).eps
    assert float((out1.float() - want[:, :n1]).abs().max()) <= eps * float(want.abs().max())
    assert float((both[:, 8:].float() - up).abs().max()) <= eps * float(up.abs().max()) and bool((both[:, :8] == 3).all())


# a share of eight columns at 33 rows and more (one unit a row), shares of 16 to 64 on both sides of 32 rows, columns past the end, one CTA a tile
@pytest.mark.parametrize("M,N,K", [(32, 8, 1024), (33, 8, 1024), (33, 72, 4096), (128, 200, 2048), (64, 2560, 1000), (32, 4352, 1024), (40, 6912, 512), (127, 9472, 64), (1, 2568, 6912)])
@pytest.mark.parametrize("f32", [False, True])
def test_products_of_few_rows_share_by_share(M, N, K, f32):
    from ghassan_b200.ops import _lib, gemm as G
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a, w = torch.randn(M, K, device="cuda", generator=g).half(), (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).half()
    out = torch.full((M + 1, N), 3.0, device="cuda", dtype=torch.float32 if f32 else torch.float16)
    add = torch.randn(M, N, device="cuda", generator=g) if f32 else None
    assert G.skinny_ok(M, N, out, add)
    G.gemm(a, w, out=out[:M], addend=add, b_static=True)
    _lib.check_status(what="few rows")
    want = a.double() @ w.double().t() + (add if f32 else 0)
    # fp32 sums of products that are exact in fp32; half a unit in the last place where they are rounded
    tol = 1e-6 * K ** 0.5 if f32 else torch.finfo(torch.float16).eps * float(want.abs().max())
    assert float((out[:M].double() - want).abs().max()) <= tol and bool((out[M] == 3).all())


@pytest.mark.parametrize("window", [0, 40, 260])
@pytest.mark.parametrize("splits", [1, 4, 8])
def test_decode_attention_of_a_full_ring(splits, window):
    """A cluster's splits over a cache whose next slot lies inside the ring; windows that begin before it and behind it."""
    from ghassan_b200.ops import decode as D
    B, H, KV, hd, cap, pinned, seen = 2, 6, 2, 64, 300, 8, 1001                            # position 1000 has been appended and is not counted yet
    g = torch.Generator(device="cuda").manual_seed(splits)
    cK, cV = (torch.randn(B, cap, KV * hd, device="cuda", generator=g).half() for _ in range(2))
    q, out = torch.randn(B, H * hd, device="cuda", generator=g).half(), torch.zeros(B, H * hd, device="cuda", dtype=torch.float16)
    at, turn = torch.arange(cap, device="cuda"), cap - pinned
    slot_pos = torch.where(at < pinned, at, at + torch.div(seen - 1 - at, turn, rounding_mode="floor") * turn).int()
    state = torch.zeros(B, D.STATE_INTS, dtype=torch.int32, device="cuda")
    state[:, 0], state[:, 1], state[:, 2] = seen - 1, cap, (seen - 1 - cap) % turn
    assert int(slot_pos[pinned + int(state[0, 2])]) == seen - 1
    D.decode_attn(q, cK, cV, slot_pos.repeat(B, 1), state, out, torch.zeros(B * H * splits * (hd + 2), device="cuda"), splits, H, KV, hd, cap, window, hd ** -0.5)
    k, v = (c.float().view(B, cap, KV, hd).repeat_interleave(H // KV, 2) for c in (cK, cV))
    s = torch.einsum("bhd,blhd->bhl", q.float().view(B, H, hd), k) * hd ** -0.5
    if window:
        s = s.masked_fill(seen - 1 - slot_pos >= window, float("-inf"))
    want = torch.einsum("bhl,blhd->bhd", torch.softmax(s, -1), v)
    assert float((out.float().view(B, H, hd) - want).abs().max()) < 2e-3          # fp32 throughout, rounded once, values below 4
