"""MoE kernels (router top-k, route plan, grouped FP8 GEMM, combine) against PyTorch references."""

import pytest
import torch

from mfq_b200.ops import fp8_gemm, moe
from mfq_b200.ops import reference as ref
from mfq_b200.quantize.fp8_block import quantize_fp8_block_torch
from gpu_common import assert_close, check_status, require_gpu_lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t,h,e,k,sig,ng,tg", [(5, 256, 8, 2, False, 1, 1), (33, 2048, 512, 10, False, 1, 1),
                                               (17, 1024, 256, 8, True, 8, 4), (1, 512, 64, 6, True, 1, 1)])
def test_router_topk(t, h, e, k, sig, ng, tg):
    require_gpu_lib()
    g = torch.Generator(device="cuda").manual_seed(e)
    x = torch.randn((t, h), generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn((e, h), generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    bias = torch.randn(e, generator=g, device="cuda") * 0.1 if sig else None
    ids, wt, scores = moe.router_topk(x, w, k, bias=bias, sigmoid=sig, n_group=ng, topk_group=tg, scale=2.5 if sig else 1.0,
                                      want_scores=True)
    logits = x.float() @ w.float().T
    s = torch.sigmoid(logits) if sig else torch.softmax(logits, -1)
    assert_close(scores, s, rel=2e-3, what="scores")
    sel = scores + (bias if bias is not None else 0)  # selection on the kernel's own scores avoids near-tie flips
    if ng > 1:
        per = e // ng
        gs = sel.view(t, ng, per).topk(2, -1).values.sum(-1)
        keep = torch.zeros_like(gs, dtype=torch.bool).scatter_(1, gs.topk(tg, -1).indices, True)
        sel = sel.masked_fill(~keep.repeat_interleave(per, 1), float("-inf"))
    want_ids = sel.topk(k, -1).indices
    assert torch.equal(ids.long().sort(-1).values, want_ids.sort(-1).values)
    want_w = scores.gather(1, ids.long())
    want_w = want_w / want_w.sum(-1, keepdim=True) * (2.5 if sig else 1.0)
    assert_close(wt, want_w, rel=1e-4, what="weights")


@pytest.mark.parametrize("t,e,k,e_lo,e_hi", [(7, 8, 2, 0, 8), (300, 64, 6, 16, 32), (64, 256, 8, 224, 256)])
def test_moe_ffn_matches_reference(t, e, k, e_lo, e_hi):
    require_gpu_lib()
    h, inter = 512, 256
    g = torch.Generator(device="cuda").manual_seed(t)
    x = torch.randn((t, h), generator=g, device="cuda").to(torch.bfloat16)
    n_local = e_hi - e_lo
    gu_f = (torch.randn((n_local, 2 * inter, h), generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    dn_f = (torch.randn((n_local, h, inter), generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    gu_q, gu_s = zip(*[quantize_fp8_block_torch(m) for m in gu_f])
    dn_q, dn_s = zip(*[quantize_fp8_block_torch(m) for m in dn_f])
    gu_q, gu_s, dn_q, dn_s = torch.stack(gu_q), torch.stack(gu_s), torch.stack(dn_q), torch.stack(dn_s)
    ids = torch.stack([torch.randperm(e, generator=g, device="cuda")[:k] for _ in range(t)]).to(torch.int32)
    wt = torch.rand((t, k), generator=g, device="cuda")
    base = torch.randn((t, h), generator=g, device="cuda").to(torch.bfloat16)
    xq, xs = ref.quant_rows(x)
    got = moe.moe_ffn_fp8(xq, xs, ids, wt, gu_q, gu_s, dn_q, dn_s, e_lo=e_lo, base=base)
    check_status()
    want = base.float().clone()
    xd = xq.float() * xs[:, None]
    for le in range(n_local):
        tok, slot = (ids == e_lo + le).nonzero(as_tuple=True)
        if tok.numel() == 0:
            continue
        gu = (xd[tok] @ ref.dequant_block(gu_q[le], gu_s[le]).T).to(torch.bfloat16)
        hq, hs = ref.silu_mul_quant(gu)
        y = ((hq.float() * hs[:, None]) @ ref.dequant_block(dn_q[le], dn_s[le]).T).to(torch.bfloat16).float()
        want.index_add_(0, tok, y * wt[tok, slot][:, None])
    # the SwiGLU output is re-quantized to E4M3 between the two GEMMs: a bf16 ulp of difference there flips a code now
    # and then, which moves single outputs by more than the element-wise bound
    assert_close(got, want, rel=2e-2, what="moe ffn", outliers=5e-3)


@pytest.mark.parametrize("t,k,e,lo,hi", [(12288, 1, 512, 0, 512), (12289, 1, 64, 16, 48), (2500, 10, 512, 0, 512), (5000, 6, 64, 0, 1)])
def test_route_plan_of_many_routes(t, k, e, lo, hi):
    """Around the line from which a thread reads eight routes at a time, and several such rounds; routes to nobody and to other ranks."""
    require_gpu_lib()
    ids = torch.randint(-1, e, (t, k), generator=torch.Generator(device="cuda").manual_seed(t), device="cuda", dtype=torch.int32)
    plan = moe.plan_routes(ids, lo, hi, token_tile=32)
    flat, dest = ids.flatten().long().cpu(), plan.dest.flatten().long().cpu()
    mine = (flat >= lo) & (flat < hi)
    counts = torch.bincount(flat[mine] - lo, minlength=hi - lo)
    offsets = torch.cat([torch.zeros(1, dtype=torch.long), counts.cumsum(0)])
    assert torch.equal(plan.offsets.long().cpu(), offsets) and bool((dest[~mine] == -1).all())
    assert torch.equal(dest[mine].sort().values, torch.arange(int(mine.sum())))  # every row once ...
    at, expert = dest[mine], flat[mine] - lo
    assert bool(((at >= offsets[expert]) & (at < offsets[expert + 1])).all())  # ... among its expert's
    assert torch.equal(plan.src_token.long().cpu()[at], (torch.arange(t * k) // k)[mine])
    want = [(x, i) for x in range(hi - lo) for i in range(-(-int(counts[x]) // 32))]
    tiles = [tuple(r) for r in plan.tile_map.tolist()]
    assert tiles[: len(want)] == want and all(r[0] < 0 for r in tiles[len(want):])
    assert plan.totals.tolist() == [int(offsets[-1]), len(want)]


@pytest.mark.parametrize("t,k,e,lo,hi", [(250, 10, 512, 0, 512), (251, 10, 512, 0, 512), (2501, 1, 3, 0, 3), (8191, 5, 512, 100, 356)])
def test_route_plan_shared_by_a_cluster(t, k, e, lo, hi):
    """Around the number of routes from which eight CTAs share the plan, and shares that do not divide: the invariants of the test before."""
    test_route_plan_of_many_routes(t, k, e, lo, hi)


@pytest.mark.parametrize("e,k", [(1, 1), (5, 5), (128, 16), (129, 3), (256, 8), (300, 10), (512, 10)])
def test_selection_of_ties_and_values_that_cannot_be_chosen(e, k):
    """Largest first, the lowest index among equals; NaN and minus infinity never, and a token without enough others gets no more."""
    require_gpu_lib()
    g = torch.Generator(device="cuda").manual_seed(e)
    t, none = 37, 0x7FFFFFFF
    logits = (torch.randn((t, e), generator=g, device="cuda") * 4).round() / 4  # a quarter apart: equal or well apart after the exponential
    logits[3] = 1.5
    logits[4] = float("nan")
    bias = torch.zeros(e, device="cuda")
    bias[::3] = float("-inf")
    for b in (None, bias):
        for sig in (0, 1):
            ids = torch.full((t, k), -5, dtype=torch.int32, device="cuda")
            w, scores = torch.empty((t, k), device="cuda"), torch.empty((t, e), device="cuda")
            rc = moe._lib().mfq_moe_router_select(logits.data_ptr(), b.data_ptr() if b is not None else None, ids.data_ptr(), w.data_ptr(), scores.data_ptr(),
                                                  t, 64, e, k, sig, 0, 1.0, 1, 1, moe.stream_ptr())
            assert rc == 0
            for row in range(t):
                left = [i for i in range(e) if row != 4 and (b is None or i % 3)]
                want = sorted(left, key=lambda i: (-float(logits[row, i]), i))[:k] if row in (0, 3, 4, t - 1) else None
                if want is None:
                    continue
                assert ids[row].tolist() == want + [none] * (k - len(want)), (row, sig)
                assert torch.equal(w[row, : len(want)], scores[row, want]) and not w[row, len(want):].any()
    check_status()


@pytest.mark.parametrize("rows", [1, 1499, 1500, 1503])
@pytest.mark.parametrize("h", [16, 528, 2048])
def test_gathered_rows(rows, h):
    """Around the number of rows from which a warp takes four; the rows that no route fills stay as they are."""
    require_gpu_lib()
    xq, xs = torch.randint(0, 127, (97, h), device="cuda", dtype=torch.uint8).view(torch.float8_e4m3fn), torch.rand(97, device="cuda")
    token = torch.randint(0, 97, (rows,), device="cuda", dtype=torch.int32)
    live = rows - rows // 5
    plan = moe.RoutePlan(None, None, token, None, torch.tensor([live, 0], dtype=torch.int32, device="cuda"), 16, rows, 1)
    q, s = moe.gather_rows(xq, xs, plan)
    assert torch.equal(q.view(torch.uint8)[:live], xq.view(torch.uint8)[token[:live].long()]) and torch.equal(s[:live], xs[token[:live].long()])
    check_status()


@pytest.mark.parametrize("k", [1, 4, 5, 6, 10, 16])
def test_combined_rows(k):
    """Contributions in batches of five and what is left of one, some of other ranks: the sums in slot order, as fp32 gives them."""
    require_gpu_lib()
    t, h = 33, 264
    y, base = torch.randn(t * k, h, device="cuda").bfloat16(), torch.randn(t, h, device="cuda").bfloat16()
    dest = torch.randperm(t * k, device="cuda").int().view(t, k)
    dest[torch.rand(t, k, device="cuda") < 0.2] = -1
    w = torch.rand(t, k, device="cuda")
    plan = moe.RoutePlan(None, dest, None, None, None, 16, t * k, 1)
    want = base.double()
    for j in range(k):  # one rounding per addition, as a fused multiply-add has it
        want = (want + (w[:, j, None].double() * y[dest[:, j].clamp_min(0).long()].double()) * (dest[:, j, None] >= 0)).float().double()
    assert torch.equal(moe.combine(y, plan, w, base), want.bfloat16())
    check_status()


@pytest.mark.parametrize("sig,ng,tg,norm,scale", [(False, 1, 1, True, 1.0), (True, 1, 1, True, 2.5), (True, 8, 4, True, 2.5), (False, 1, 1, False, 1.0)])
def test_router_of_a_prompt_chooses_what_the_routers_own_kernels_do(sig, ng, tg, norm, scale, monkeypatch):
    """Beyond 64 tokens logits come from the dense product -- or, where its library is not there, from the router's own kernels."""
    require_gpu_lib()
    g = torch.Generator(device="cuda").manual_seed(ng)
    x, w = torch.randn((201, 1024), generator=g, device="cuda").to(torch.bfloat16), (torch.randn((256, 1024), generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    bias = torch.randn(256, generator=g, device="cuda") * 0.1 if sig else None
    how = dict(bias=bias, sigmoid=sig, n_group=ng, topk_group=tg, norm_topk=norm, scale=scale, want_scores=True)
    got = moe.router_topk(x, w, 8, **how)
    monkeypatch.setattr(moe, "dense_available", lambda: False)
    monkeypatch.setattr(moe, "DenseLinear", None)
    want = moe.router_topk(x, w, 8, **how)
    # fp32 sums of 1024 products in another order before an exponential: their absolute error, on either side
    slack = float((x.abs().float() @ w.abs().float().T).amax()) * 1032 * 2.0 ** -23
    assert bool(((got[2] - want[2]).abs() <= slack * want[2]).all())
    same = (got[0].sort(1).values == want[0].sort(1).values).all(1)
    assert same.float().mean() > 0.98  # near ties may fall either way
    assert bool(((got[1][same].sort(1).values - want[1][same].sort(1).values).abs() <= 2 * slack * scale).all())


@pytest.mark.parametrize("k", [128, 640, 4224])
@pytest.mark.parametrize("tile", [16, 32, 64, 128])
def test_grouped_product_over_several_tiles_per_cta(tile, k):
    """Empty experts, single rows, whole and ragged tiles; one, a few and more than 32 K blocks per tile: the bits of the product of each
    expert by itself."""
    require_gpu_lib()
    counts = [0, 1, 3 * tile + 5, tile, tile + 1, 0, 2 * tile - 1, 7] * 6 + [0]
    e, n, rows = len(counts), 1024, sum(counts)
    g = torch.Generator(device="cuda").manual_seed(k + tile)
    fp8 = lambda *s: (torch.randn(s, generator=g, device="cuda") * 60).clamp(-448, 448).to(torch.float8_e4m3fn)
    x, w = fp8(rows, k), fp8(e, n, k)
    xs, ws = torch.rand(rows, generator=g, device="cuda") + 0.1, torch.rand((e, n // 128, k // 128), generator=g, device="cuda") + 0.1
    ids = torch.repeat_interleave(torch.arange(e), torch.tensor(counts))[torch.randperm(rows, generator=torch.Generator().manual_seed(1))]
    plan = moe.plan_routes(ids.int()[:, None].cuda(), 0, e, token_tile=tile)
    assert int(plan.totals[1]) * (n // 128) > 3 * torch.cuda.get_device_properties(0).multi_processor_count
    assert not moe.grouped_gemv_ok(plan, n)
    got = moe.fp8_gemm_grouped(x, xs, w, ws, plan)
    check_status()
    at = 0
    for i, c in enumerate(counts):
        if c:
            rng = slice(at, at + c)
            assert torch.equal(got[rng], fp8_gemm(x[rng], xs[rng], w[i], ws[i], splits=1, token_tile=tile)), (i, c)
        at += c


@pytest.mark.parametrize("tile", [32, 64])
def test_grouped_product_into_an_unaligned_output(tile):
    """Results leave in 16-byte stores only where the output allows them."""
    require_gpu_lib()
    rows, k, n = 70, 256, 256
    fp8 = lambda *s: (torch.randn(s, device="cuda") * 60).clamp(-448, 448).to(torch.float8_e4m3fn)
    x, w, xs, ws = fp8(rows, k), fp8(2, n, k), torch.rand(rows, device="cuda"), torch.rand((2, n // 128, k // 128), device="cuda")
    plan = moe.plan_routes((torch.arange(rows, device="cuda") >= 41).int()[:, None], 0, 2, token_tile=tile)
    want = moe.fp8_gemm_grouped(x, xs, w, ws, plan)
    out = torch.zeros(rows * n + 2, device="cuda", dtype=torch.bfloat16)
    rc = moe._lib().mfq_fp8_gemm_grouped(w.data_ptr(), ws.data_ptr(), x.data_ptr(), xs.data_ptr(), out[1:].data_ptr(), moe.Workspace.get(x.device).status.data_ptr(),
                                         rows, n, k, 2, plan.tile_map.data_ptr(), plan.offsets.data_ptr(), plan.tile_map.shape[0], tile, moe.stream_ptr())
    assert rc == 0 and torch.equal(out[1:-1].view(rows, n), want) and not out[0] and not out[-1]
    check_status()
