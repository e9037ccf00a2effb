"""Each CUDA op against a plain PyTorch fp32 or fp64 reference of the same op. Results that are rounded to bf16 once are bounded
by that rounding; the absolute bounds are tighter than those of the reference's kernel smoke tests (LayerNorm out 0.08 / stats
0.05 / grads 0.12: dev/cuda/test_layernorm.cu:325-327; RMSNorm 0.04 / 0.01: test_rmsnorm.cu:229-230; RoPE 0.02:
test_rope.cu:150; attention fwd 0.08 / bwd 0.20: test_attention.cu:355-356)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def rnd(*shape, scale=1.0, dtype=BF):
    return (torch.randn(*shape, device="cuda", dtype=torch.float32) * scale).to(dtype)


def maxerr(a, b):
    return (a.float() - b.float()).abs().max().item()


def rounded(got, want, rest):
    """``got`` is ``want`` rounded to bf16 (at most 2^-9 of the value; 2^-8 leaves room for a result that lies on the other side
    of a rounding boundary) but for ``rest``, the error of the fp32 arithmetic in front of the rounding."""
    return ((got.double() - want.double()).abs() <= 2.0 ** -8 * want.double().abs() + rest).all().item()


@pytest.mark.parametrize("N,C", [(64, 768), (1000, 768), (3, 1024), (257, 2048), (128, 4096), (33, 1600)])
def test_layernorm_fwd_bwd(N, C):
    from llm_kittens_b200.ops import norm

    x, w, b = rnd(N, C), rnd(C, scale=0.5) + 1, rnd(C, scale=0.1)
    out, mean, rstd = norm.layernorm_fwd(x, w, b)
    xf = x.float().requires_grad_(True)
    wf, bf_ = w.float().requires_grad_(True), b.float().requires_grad_(True)
    ref = torch.nn.functional.layer_norm(xf, (C,), wf, bf_, 1e-5)
    assert rounded(out, ref, 1e-4)
    assert maxerr(mean, x.float().mean(-1)) < 1e-3
    assert maxerr(rstd, 1 / torch.sqrt(x.float().var(-1, unbiased=False) + 1e-5)) < 1e-2
    dout = rnd(N, C)
    ref.backward(dout.float())
    dinp0 = rnd(N, C)
    dinp = dinp0.clone()
    dw, db = torch.zeros(C, device="cuda", dtype=BF), torch.zeros(C, device="cuda", dtype=BF)
    norm.layernorm_bwd(dinp, dw, db, dout, x, w, mean, rstd, accumulate_dinp=True)
    assert rounded(dinp, xf.grad + dinp0.float(), 1e-3)
    assert maxerr(dw, wf.grad) < 0.02 * max(1.0, wf.grad.abs().max().item())
    assert maxerr(db, bf_.grad) < 0.02 * max(1.0, bf_.grad.abs().max().item())
    # deterministic
    dw2, db2, dinp2 = torch.zeros_like(dw), torch.zeros_like(db), dinp0.clone()
    norm.layernorm_bwd(dinp2, dw2, db2, dout, x, w, mean, rstd, accumulate_dinp=True)
    assert torch.equal(dw, dw2) and torch.equal(db, db2) and torch.equal(dinp, dinp2)


def test_residual_layernorm():
    from llm_kittens_b200.ops import norm

    N, C = 300, 768
    a, b, w, bias = rnd(N, C), rnd(N, C), rnd(C) + 1, rnd(C)
    res, out, mean, rstd = norm.residual_layernorm_fwd(a, b, w, bias)
    r = (a.float() + b.float()).to(BF)
    assert torch.equal(res, r)
    ref = torch.nn.functional.layer_norm(r.float(), (C,), w.float(), bias.float(), 1e-5)
    assert rounded(out, ref, 1e-4)     # (outputs above 16, one draw in ten, are rounded by up to 0.06)


@pytest.mark.parametrize("N,C", [(64, 2048), (100, 4096), (5, 768)])
def test_rmsnorm(N, C):
    from llm_kittens_b200.ops import norm

    x, w = rnd(N, C), rnd(C, scale=0.3) + 1
    out, rstd = norm.rmsnorm_fwd(x, w, 1e-5)
    xf, wf = x.float().requires_grad_(True), w.float().requires_grad_(True)
    ref = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-5) * wf
    assert rounded(out, ref, 1e-4)
    assert maxerr(rstd, torch.rsqrt(x.float().pow(2).mean(-1) + 1e-5)) < 0.01
    dout = rnd(N, C)
    ref.backward(dout.float())
    dinp = torch.zeros(N, C, device="cuda", dtype=BF)
    dw = torch.zeros(C, device="cuda", dtype=BF)
    norm.rmsnorm_bwd(dinp, dw, dout, x, w, rstd, accumulate_dinp=False)
    assert rounded(dinp, xf.grad, 1e-3)
    assert maxerr(dw, wf.grad) < 0.02 * max(1.0, wf.grad.abs().max().item())
    a, b = rnd(N, C), rnd(N, C)
    res, out2, _ = norm.residual_rmsnorm_fwd(a, b, w, 1e-5)
    assert torch.equal(res, (a.float() + b.float()).to(BF))


@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("N,C", [(1, 8), (5, 248), (9, 264), (700, 1600), (3, 1912), (300, 2040), (7, 2056), (5, 3200), (4, 6136),
                                 (512, 8), (4100, 128), (513, 248), (1024, 264), (2500, 384), (1023, 504), (1025, 776), (1030, 1272)])
def test_norms_of_widths_that_are_not_whole_vectors_per_lane(N, C, rms):
    """Row widths around the edges of the per-lane (256) and per-block (2048) vectors. Every tensor is followed by a row of
    NaNs that must be neither read into a result nor overwritten."""
    from llm_kittens_b200.ops import norm

    def padded(t):
        whole = torch.full((t.numel() + C,), float("nan"), device="cuda", dtype=t.dtype)
        whole[:t.numel()] = t.reshape(-1)
        return whole, whole[:t.numel()].view(t.shape)

    x, dout, dinp0 = rnd(N, C), rnd(N, C), rnd(N, C)
    w, b = rnd(C, scale=0.5) + 1, rnd(C, scale=0.1)
    xd, dd = x.double().requires_grad_(True), dout.double()
    wd, bd = w.double().requires_grad_(True), b.double().requires_grad_(True)
    if rms:
        rs = torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-5)
        ref, stats = xd * rs * wd, [None, rs.detach().view(-1).float()]
    else:
        ref = torch.nn.functional.layer_norm(xd, (C,), wd, bd, 1e-5)
        stats = [xd.detach().mean(-1).float(), torch.rsqrt(xd.detach().var(-1, unbiased=False) + 1e-5).float()]
    ref.backward(dd)
    (xw, xv), (ow, ov), (gw, gv), (ww, wv), (bw, bv), (dw_, dv) = (padded(t) for t in (x, torch.zeros_like(x), dinp0, w, b, dout))
    dw, db = torch.zeros(C, device="cuda", dtype=BF), torch.zeros(C, device="cuda", dtype=BF)
    if rms:
        _, rstd = norm.rmsnorm_fwd(xv, wv, out=ov)
        norm.rmsnorm_bwd(gv, dw, dv, xv, wv, stats[1], accumulate_dinp=True)
    else:
        _, mean, rstd = norm.layernorm_fwd(xv, wv, bv, out=ov)
        norm.layernorm_bwd(gv, dw, db, dv, xv, wv, stats[0], stats[1], accumulate_dinp=True)
        assert (mean - stats[0]).abs().max() < 1e-5
    # fp32 arithmetic, one rounding to bf16 (2^-9 of the value) and for the weight gradients one of the sum of N products
    ulp = 2.0 ** -8
    assert (rstd / stats[1] - 1).abs().max() < 1e-4
    assert ((ov.double() - ref).abs() <= ulp * ref.abs() + 1e-4).all()
    want = xd.grad + dinp0.double()
    assert ((gv.double() - want).abs() <= ulp * want.abs() + 1e-3).all()
    assert ((dw.double() - wd.grad).abs() <= ulp * wd.grad.abs() + 1e-3).all()
    if not rms:
        assert ((db.double() - bd.grad).abs() <= ulp * bd.grad.abs() + 1e-3).all()
    for whole, view in ((ow, ov), (gw, gv)):
        assert torch.isnan(whole[view.numel():]).all() and not torch.isnan(view).any()


@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("C", [256, 520, 768])
@pytest.mark.parametrize("extra", [0, 1])
def test_norm_backward_on_both_sides_of_two_rows_per_warp(C, extra, rms):
    """Every warp of every SM has two rows, and one of them a third."""
    from llm_kittens_b200.ops import norm

    N = 32 * torch.cuda.get_device_properties(0).multi_processor_count + extra
    x, dout, dinp0, w = rnd(N, C), rnd(N, C), rnd(N, C), rnd(C, scale=0.5) + 1
    xd, wd = x.double().requires_grad_(True), w.double().requires_grad_(True)
    bd = torch.zeros(C, device="cuda", dtype=torch.float64, requires_grad=True)
    mean = torch.zeros(N, device="cuda") if rms else x.double().mean(-1).float()
    rstd = torch.rsqrt((x.double() - mean.double()[:, None]).pow(2).mean(-1) + 1e-5).float()
    y = xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-5) * wd if rms else torch.nn.functional.layer_norm(xd, (C,), wd, bd, 1e-5)
    y.backward(dout.double())
    dinp, dw, db = dinp0.clone(), torch.zeros_like(w), torch.zeros_like(w)
    if rms:
        norm.rmsnorm_bwd(dinp, dw, dout, x, w, rstd, accumulate_dinp=True)
    else:
        norm.layernorm_bwd(dinp, dw, db, dout, x, w, mean, rstd, accumulate_dinp=True)
        assert rounded(db, bd.grad, 1e-3)
    assert rounded(dinp, xd.grad + dinp0.double(), 1e-3) and rounded(dw, wd.grad, 1e-3)   # as in the test above


@pytest.mark.parametrize("N,C", [(3, 1288), (2, 8200), (300, 16384)])
def test_norm_forward_of_wide_rows(N, C):
    from llm_kittens_b200.ops import norm

    a, b, w, bias = rnd(N, C), rnd(N, C), rnd(C, scale=0.5) + 1, rnd(C, scale=0.1)
    r = (a.float() + b.float()).to(BF)
    ulp = 2.0 ** -8     # one rounding to bf16
    res, out, _, _ = norm.residual_layernorm_fwd(a, b, w, bias)
    want = torch.nn.functional.layer_norm(r.double(), (C,), w.double(), bias.double(), 1e-5)
    assert torch.equal(res, r) and ((out.double() - want).abs() <= ulp * want.abs() + 1e-4).all()
    a2 = a.clone()
    res, out, _ = norm.residual_rmsnorm_fwd(a2, b, w, 1e-5, residual=a2)     # the sum overwrites an addend
    want = r.double() * torch.rsqrt(r.double().pow(2).mean(-1, keepdim=True) + 1e-5) * w.double()
    assert torch.equal(a2, r) and ((out.double() - want).abs() <= ulp * want.abs() + 1e-4).all()


@pytest.mark.parametrize("N,C", [(2048, 4104), (2049, 4104), (2049, 2056), (9, 8200), (2049, 8200), (700, 512), (4000, 392), (700, 1024), (1184, 1280),
                                 (1185, 1280), (2368, 768), (2369, 768)])
def test_norm_forward_where_the_arithmetic_changes(N, C):
    """Row counts and widths on both sides of packed arithmetic, of kept weights and of the register limits, with 148 SMs."""
    from llm_kittens_b200.ops import norm

    test_norm_forward_of_wide_rows(N, C)
    x, w, b = rnd(N, C), rnd(C, scale=0.5) + 1, rnd(C, scale=0.1)
    xd = x.double()
    out, mean, rstd = norm.layernorm_fwd(x, w, b)
    assert rounded(out, torch.nn.functional.layer_norm(xd, (C,), w.double(), b.double(), 1e-5), 1e-4)
    assert (mean - xd.mean(-1)).abs().max() < 1e-5 and (rstd * (xd.var(-1, unbiased=False) + 1e-5).sqrt() - 1).abs().max() < 1e-4
    out, rstd = norm.rmsnorm_fwd(x, w, 1e-5)
    rs = torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-5)
    assert rounded(out, xd * rs * w.double(), 1e-4) and (rstd / rs.view(-1) - 1).abs().max() < 1e-4


@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("N,C", [(1, 264), (444, 768), (445, 768), (592, 1280), (593, 1024), (591, 1024), (296, 504), (297, 512), (2, 2048),
                                 (295, 1600), (297, 1600), (1187, 1600), (5, 2048)])
def test_norms_of_few_rows(N, C, rms):
    """Row counts on both sides of where a block per row gives way to a warp per row, forward (three rows per SM up to 768
    columns, four beyond) and backward (four), with 148 SMs, and counts that are no multiple of the rows of a backward step."""
    test_norms_of_widths_that_are_not_whole_vectors_per_lane(N, C, rms)
    test_norm_forward_of_wide_rows(N, C)


@pytest.mark.parametrize("N,C", [(20001, 256), (19000, 512), (20001, 768), (19000, 1024), (19000, 1280), (8191, 1536), (8192, 1536),
                                 (20001, 1536)])
def test_norm_forward_of_more_rows_than_the_grid_has_warps(N, C):
    """Every variant of the warp-per-row and block-per-row kernels over several rows per warp, with and without a residual."""
    from llm_kittens_b200.ops import norm

    a, b, w, bias = rnd(N, C), rnd(N, C), rnd(C, scale=0.5) + 1, rnd(C, scale=0.1)
    ulp = 2.0 ** -8     # one rounding to bf16
    for x, ln, rms in ((a, norm.layernorm_fwd(a, w, bias), norm.rmsnorm_fwd(a, w, 1e-5)),
                       ((a.float() + b.float()).to(BF), norm.residual_layernorm_fwd(a, b, w, bias), norm.residual_rmsnorm_fwd(a, b, w, 1e-5))):
        if len(ln) == 4:
            assert torch.equal(ln[0], x) and torch.equal(rms[0], x)
            ln, rms = ln[1:], rms[1:]
        want = torch.nn.functional.layer_norm(x.double(), (C,), w.double(), bias.double(), 1e-5)
        assert ((ln[0].double() - want).abs() <= ulp * want.abs() + 1e-4).all()
        assert (ln[1] - x.double().mean(-1)).abs().max() < 1e-5
        rs = torch.rsqrt(x.double().pow(2).mean(-1) + 1e-5)
        want = x.double() * rs[:, None] * w.double()
        assert ((rms[0].double() - want).abs() <= ulp * want.abs() + 1e-4).all()
        assert (rms[1] / rs - 1).abs().max() < 1e-5


@pytest.mark.parametrize("n", [1, 7, 8, 9, 2047, 2048, 2049, 1000003])
def test_zeroing_ends_at_the_tensor(n):
    from llm_kittens_b200.ops import elementwise as ew

    for skip in (0, 1):       # 16-byte aligned or not
        whole = torch.full((n + 16,), 3.0, device="cuda", dtype=BF)
        ew.zero_(whole[skip:skip + n])
        assert (whole[skip:skip + n] == 0).all() and (whole[:skip] == 3).all() and (whole[skip + n:] == 3).all()


@pytest.mark.parametrize("rows,C,NH", [(64, 768, 12), (320, 2048, 32), (4096, 768, 12)])
def test_chains_of_kernels_keep_the_stream_order(rows, C, NH):
    """Chains in which every launch reads what the one before wrote and overwrites what the one before read, with work of
    another stream forked and joined in between: the same bits with a synchronisation after every call, without any, and
    replayed from a CUDA graph."""
    from llm_kittens_b200.ops import attention as attn, elementwise as ew, gemm, norm

    w1, w2, wq = rnd(C, C, scale=0.03), rnd(C, C, scale=0.03), rnd(3 * C, C, scale=0.03)
    nw, nb, x0 = rnd(C) + 1, rnd(C), rnd(rows, C)
    side = torch.cuda.Stream()
    x, y, z, qkv = x0.clone(), torch.empty_like(x0), torch.empty_like(x0), torch.empty(rows, 3 * C, device="cuda", dtype=BF)
    mean, rstd = (torch.empty(rows, device="cuda") for _ in range(2))
    lse, dvec = (torch.empty(1, NH, rows, device="cuda") for _ in range(2))
    dw, db, cs = torch.zeros(C, C, device="cuda", dtype=BF), torch.zeros(C, device="cuda", dtype=BF), torch.empty(C, device="cuda", dtype=BF)

    def chain(sync):
        step = torch.cuda.synchronize if sync else (lambda: None)
        x.copy_(x0), dw.zero_(), db.zero_()
        for _ in range(3):
            norm.layernorm_fwd(x, nw, nb, out=y, mean=mean, rstd=rstd), step()
            gemm.gemm_nt(y, wq, out=qkv), step()
            attn.attention_fwd(qkv, 1, rows, NH, NH, C // NH, out=y, lse=lse), step()
            gemm.gemm_nt(y, w1, add=x, out=x), step()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                ew.dbias(cs, x, accumulate=False), step()
            gemm.gemm_nn(x, w2, out=z), step()
            torch.cuda.current_stream().wait_stream(side)
            gemm.gemm_tn(z, x, out=dw, accumulate=True, dbias=db), step()
            ew.gelu_fwd(z, out=y), step()
            norm.layernorm_bwd(x, cs, db, y, z, nw, mean, rstd, accumulate_dinp=True), step()
            gemm.gemm_nt(x, dw, out=y), step()
        return [t.clone() for t in (x, y, z, qkv, dw, db, cs, lse)]

    want = chain(True)
    assert all(torch.isfinite(t).all() for t in want)
    for _ in range(3):
        assert all(torch.equal(a, b) for a, b in zip(want, chain(False)))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = chain(False)
    for _ in range(3):
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(want, got))


@pytest.mark.parametrize("N,C,E,K", [(1, 8, 1, 1), (7, 64, 3, 2), (1000, 264, 8, 2), (1025, 256, 5, 1), (4099, 1024, 16, 4), (5000, 72, 12, 3)])
def test_moe_routing_slots_and_density(N, C, E, K):
    """Router probabilities and choices, slots in token order up to the capacity, and expert densities, for expert counts that
    do not divide a warp or a block and token counts around the rounds of the slot assignment."""
    from llm_kittens_b200.ops import moe

    x, wr = rnd(N, C), rnd(E, C, scale=0.1)
    probs, idx, w = moe.router_fwd(x, wr, K)
    ref = (x.double() @ wr.double().T).softmax(-1)
    assert ((probs.double() - ref).abs() <= 1e-5).all()
    want = torch.sort(probs, dim=-1, descending=True, stable=True)       # equal probabilities: the lower expert first
    assert torch.equal(idx.long(), want.indices[:, :K])
    top = want.values[:, :K].double()
    assert ((w.double() - top / top.sum(-1, keepdim=True)).abs() <= 1e-6).all()
    cap = max(1, N * K // E)
    slot, counts = moe.assign_slots(idx, E, cap)
    flat, got = idx.view(-1), slot.view(-1)
    for e in range(E):
        mine = got[flat == e]
        ranks = torch.arange(mine.numel(), device="cuda", dtype=torch.int32)
        assert torch.equal(mine, torch.where(ranks < cap, ranks, torch.full_like(ranks, -1)))
        assert counts[e].item() == min(cap, mine.numel())
    dens, aux = moe.density(probs, 0.01)
    assert ((dens.double() - probs.double().mean(0)).abs() <= 1e-6).all()
    assert abs(aux.item() - 0.01 * E * probs.double().mean(0).pow(2).sum().item()) <= 1e-6


@pytest.mark.parametrize("N,C,E,K", [(1, 8, 1, 1), (9, 264, 3, 2), (4740, 1032, 5, 3), (9700, 1024, 8, 2), (5000, 2056, 16, 4), (40, 4096, 16, 2),
                                     (33, 520, 7, 5)])
def test_moe_rows_moved_and_summed(N, C, E, K):
    """Dispatch, its weighted form, combine and the routing weights' gradient with dropped assignments, for rows of less and
    more than a warp's vectors, tokens beyond one per resident warp, more experts per token than the router gives, and (40, 4096,
    16) a router too large for shared memory as fp32."""
    from llm_kittens_b200.ops import moe

    x, base, cap = rnd(N, C), rnd(N, C), max(1, N * K // (E + 1))
    if K <= 4:
        wr = rnd(E, C, scale=0.02)
        probs, idx, w = moe.router_fwd(x, wr, K)
        assert ((probs.double() - (x.double() @ wr.double().T).softmax(-1)).abs() <= 1e-5).all()
        assert torch.equal(idx.long(), torch.sort(probs, dim=-1, descending=True, stable=True).indices[:, :K])
    else:
        w, idx = (v.contiguous() for v in torch.rand(N, E, device="cuda").topk(K, dim=-1))
        idx = idx.int()
    slot, counts = moe.assign_slots(idx, E, cap)
    kept = slot >= 0
    assert N == 1 or not kept.all()
    at = (idx.long() * cap + slot.long())
    for scaled in (False, True):
        recv = torch.full((E * cap, C), float("nan"), device="cuda", dtype=BF)
        want = torch.zeros(E * cap, C, device="cuda", dtype=BF)
        for k in range(K):
            rows = (x.float() * w[:, k:k + 1]).to(BF) if scaled else x
            want[at[kept[:, k], k]] = rows[kept[:, k]]
        moe.dispatch(moe.ptr_table([recv]), x, idx, slot, w, counts, E, cap, scale_by_weight=scaled)
        assert torch.equal(recv, want)
    y, out = rnd(E * cap, C), torch.empty(N, C, device="cuda", dtype=BF)
    rows = y.double()[at.clamp(min=0)] * kept.unsqueeze(-1)              # [N, K, C], zero where dropped
    for add, weight in ((base, w), (None, None)):
        moe.combine(out, add, y, idx, slot, weight, cap)
        terms = rows if weight is None else rows * weight.double().unsqueeze(-1)
        ref = terms.sum(1) + (0 if add is None else add.double())
        size = terms.abs().sum(1) + (0 if add is None else add.double().abs())
        # one rounding to bf16 and one of fp32 per term
        assert ((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + (K + 1) * 2.0 ** -23 * size).all()
    dw = moe.combine_dweight(base, y, idx, slot, cap)
    terms = rows * base.double().unsqueeze(1)
    assert ((dw.double() - terms.sum(-1)).abs() <= (C / 32 + 6) * 2.0 ** -24 * terms.abs().sum(-1)).all()


@pytest.mark.parametrize("N,C,E,K", [(1024, 264, 4, 2), (1025, 264, 4, 2), (2048, 136, 6, 3), (2049, 136, 6, 3), (32768, 264, 3, 1), (32769, 264, 3, 1)])
def test_moe_rows_where_the_weight_gradient_changes_kernel(N, C, E, K):
    """Token counts on both sides of a warp per token and expert."""
    test_moe_rows_moved_and_summed(N, C, E, K)


@pytest.mark.parametrize("N,C,E,K", [(32767, 136, 3, 2), (32768, 136, 3, 2), (32769, 136, 2, 1)])
def test_moe_rows_where_the_unused_slots_are_zeroed_first(N, C, E, K):
    test_moe_rows_moved_and_summed(N, C, E, K)


def test_gelu_swiglu_add():
    from llm_kittens_b200.ops import elementwise as ew

    x = rnd(1000, 3072, scale=2.0)
    xf = x.float().requires_grad_(True)
    ref = torch.nn.functional.gelu(xf, approximate="tanh")
    assert maxerr(ew.gelu_fwd(x), ref) < 0.02
    d = rnd(1000, 3072)
    ref.backward(d.float())
    assert maxerr(ew.gelu_bwd_inplace(d.clone(), x), xf.grad) < 0.03
    g, u, do = rnd(512, 8192), rnd(512, 8192), rnd(512, 8192)
    gf, uf = g.float().requires_grad_(True), u.float().requires_grad_(True)
    r = torch.nn.functional.silu(gf) * uf
    assert maxerr(ew.swiglu_fwd(g, u), r) < 0.07  # |out| reaches ~16 where one bf16 ulp is 0.06
    r.backward(do.float())
    dg, du = ew.swiglu_bwd(do, g, u)
    assert maxerr(dg, gf.grad) < 0.1 and maxerr(du, uf.grad) < 0.1
    ug = torch.cat([u, g], dim=1).contiguous()
    assert torch.equal(ew.swiglu_fused_fwd(ug), ew.swiglu_fwd(g, u))
    dug = ew.swiglu_fused_bwd(do, ug)
    assert torch.equal(dug[:, :8192], du) and torch.equal(dug[:, 8192:], dg)
    a, b = rnd(777, 64), rnd(777, 64)
    assert torch.equal(ew.add(a, b), (a.float() + b.float()).to(BF))


@pytest.mark.parametrize("interleaved", [True, False])
def test_rope(interleaved):
    from llm_kittens_b200.ops import elementwise as ew

    B, T, NH, NKVH, HS = 2, 128, 8, 2, 64
    qkv = rnd(B, T, (NH + 2 * NKVH) * HS)
    freqs = ew.rope_tables(T, HS, 500000.0)
    out = ew.rope_qk_(qkv.clone(), freqs, B, T, NH, NKVH, HS, interleaved=interleaved)
    x = qkv.float().view(B, T, NH + 2 * NKVH, HS)
    cos, sin = freqs[..., 0][None, :, None, :], freqs[..., 1][None, :, None, :]
    ref = x.clone()
    rot = x[:, :, : NH + NKVH]
    if interleaved:
        x0, x1 = rot[..., 0::2], rot[..., 1::2]
        ref[:, :, : NH + NKVH, 0::2] = x0 * cos - x1 * sin
        ref[:, :, : NH + NKVH, 1::2] = x0 * sin + x1 * cos
    else:
        x0, x1 = rot[..., : HS // 2], rot[..., HS // 2:]
        ref[:, :, : NH + NKVH, : HS // 2] = x0 * cos - x1 * sin
        ref[:, :, : NH + NKVH, HS // 2:] = x0 * sin + x1 * cos
    assert maxerr(out, ref.view(B, T, -1)) < 0.02
    back = ew.rope_qk_(out.clone(), freqs, B, T, NH, NKVH, HS, interleaved=interleaved, inverse=True)
    assert maxerr(back, qkv) < 0.05


def test_dbias_and_encoder():
    from llm_kittens_b200.ops import elementwise as ew

    dout = rnd(1000, 2304)
    db0 = rnd(2304)
    db = db0.clone()
    ew.dbias(db, dout, accumulate=True)
    ref_db = db0.float() + dout.float().sum(0)
    assert ((db.float() - ref_db).abs() <= 0.01 * ref_db.abs() + 0.05).all()
    B, T, C, V = 4, 64, 768, 1000
    wte, wpe = rnd(V, C), rnd(T, C)
    tok = torch.randint(0, V, (B, T), device="cuda", dtype=torch.int32)
    tok[0, :10] = 7  # repeated token
    out = ew.encoder_fwd(tok, wte, wpe)
    assert rounded(out, wte.float()[tok.long()] + wpe.float()[None], 0.0)
    d = rnd(B, T, C)
    dwte, dwpe = torch.zeros_like(wte), torch.zeros_like(wpe)
    ew.encoder_bwd(dwte, dwpe, d, tok)
    ref_wte = torch.zeros(V, C, device="cuda").index_add_(0, tok.reshape(-1).long(), d.float().view(-1, C))
    assert rounded(dwte, ref_wte, 1e-5)
    assert rounded(dwpe, d.float().sum(0), 1e-5)
    dwte2, dwpe2 = torch.zeros_like(wte), torch.zeros_like(wpe)
    ew.encoder_bwd(dwte2, dwpe2, d, tok)
    assert torch.equal(dwte, dwte2)


@pytest.mark.parametrize("B,T,C,V,kind", [(1, 64, 768, 50, "same"), (3, 64, 64, 9, "few"), (2, 1024, 768, 50304, "zipf"),
                                          (1, 64, 2056, 1000, "distinct"), (33, 64, 768, 3, "few"), (9, 1024, 128, 1, "same"),
                                          (1, 8, 64, 50, "distinct"), (1, 7, 64, 3, "few"), (16, 64, 384, 50304, "zipf"),
                                          (1, 1025, 384, 700, "few"), (4, 1024, 384, 50304, "zipf"), (1, 4097, 256, 50304, "distinct"),
                                          (33, 1024, 256, 50304, "zipf"), (33, 1024, 64, 5, "few")])
def test_embedding_gradient_of_runs_that_cross_block_edges(B, T, C, V, kind):
    """Runs of one token that end at, cross, or cover whole blocks of sorted positions, against fp64 sums."""
    from llm_kittens_b200.ops import elementwise as ew

    if kind == "same":
        tok = torch.full((B, T), V - 1)
    elif kind == "distinct":
        tok = torch.randperm(V)[: B * T].view(B, T)
    elif kind == "few":
        tok = torch.randint(0, V, (B, T))
    else:
        tok = (torch.rand(B, T).pow(6) * V).long().clamp_(max=V - 1)
    tok = tok.to("cuda", torch.int32)
    d = rnd(B, T, C)
    dwte = rnd(V, C, scale=0.1)
    want = dwte.double().index_add_(0, tok.view(-1).long(), d.double().view(-1, C))
    ew.encoder_bwd(dwte, None, d, tok)
    # fp32 sums of at most B * T values of order 1, one rounding to bf16
    assert ((dwte.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6 * B * T).all()


@pytest.mark.parametrize("n,V", [(65536, 50304), (5000, 128256), (2048, 300), (33, 7), (131072, 50304)])
def test_bucket_sort_is_a_stable_sort_by_token(n, V):
    """The device radix sort that buckets positions by token id gives exactly the stable sort (token, position),
    for sizes that are not whole tiles and for vocabularies that need one, two and (hypothetically) more digit passes."""
    from llm_kittens_b200.ops import elementwise as ew

    g = torch.Generator(device="cuda").manual_seed(n)
    tok = torch.randint(0, V, (n,), generator=g, device="cuda", dtype=torch.int32)
    tok[: n // 3] = tok[0]                    # a heavy hitter, as natural text has
    st, sp = ew.bucket_sort(tok, V)
    ref_tok, ref_pos = torch.sort(tok, stable=True)
    assert torch.equal(st, ref_tok) and torch.equal(sp.long(), ref_pos)
    st2, sp2 = ew.bucket_sort(tok, 1 << 20)    # three passes
    assert torch.equal(st2, ref_tok) and torch.equal(sp2.long(), ref_pos)


@pytest.mark.parametrize("rows,V,Vp", [(64, 50257, 50304), (16, 1000, 1024), (8, 128256, 128256)])
def test_fused_classifier(rows, V, Vp):
    from llm_kittens_b200.ops import classifier

    logits = rnd(rows, Vp, scale=2.0)
    tg = torch.randint(0, V, (rows,), device="cuda", dtype=torch.int32)
    lf = logits.float()[:, :V].requires_grad_(True)
    ref_losses = torch.nn.functional.cross_entropy(lf, tg.long(), reduction="none")
    dloss = 1.0 / rows
    (ref_losses.sum() * dloss).backward()
    lg = logits.clone()
    losses = classifier.fused_classifier(lg, tg, V, dloss)
    assert maxerr(losses, ref_losses) < 2e-3
    assert maxerr(lg[:, :V], lf.grad) < 2e-3
    assert lg[:, V:].abs().max().item() == 0 if Vp > V else True
    lg2 = logits.clone()
    l2 = classifier.fused_classifier(lg2, tg, V, dloss, write_dlogits=False)
    assert torch.equal(lg2, logits) and torch.equal(l2, losses)
    tot = torch.zeros(1, device="cuda")
    classifier.sum_scaled(tot, losses, 1.0 / rows)
    assert abs(tot.item() - ref_losses.mean().item()) < 1e-3


@pytest.mark.parametrize("rows,V,Vp", [(1, 1, 8), (449, 50257, 50304), (450, 4999, 5000), (5, 56317, 56320), (149, 56325, 56328), (3, 84473, 84480),
                                       (7, 84481, 84488), (200, 128001, 128256), (3, 140801, 140808), (77, 225279, 225280), (2, 225281, 225288)])
def test_fused_classifier_over_blocks_and_clusters(rows, V, Vp):
    """Row widths on both sides of one, three, five and eight blocks per row, several rows per block, columns that are no whole
    vectors, rows with entries of -infinity, of the type's lowest value, and of a range whose exponentials leave the normal
    numbers."""
    from llm_kittens_b200.ops import classifier

    logits = rnd(rows, Vp, scale=3.0)
    logits[0, : V // 2] = float("-inf")
    logits[0, V - 1] = 1.0
    logits[rows // 2, V // 3 : V - 1] = torch.finfo(BF).min
    logits[rows - 1, ::3] -= 95.0
    logits[:, V:] = 60.0                                       # not real: neither maximum nor sum may see them
    tg = torch.randint(0, V, (rows,), device="cuda", dtype=torch.int32)
    tg[0], tg[rows // 2], tg[rows - 1] = V - 1, 0, V - 1
    dloss = 0.5
    lg, lg2 = logits.clone(), logits.clone()
    got = classifier.fused_classifier(lg, tg, V, dloss)
    assert torch.equal(classifier.fused_classifier(lg2, tg, V, dloss, write_dlogits=False), got) and torch.equal(lg2, logits)
    for r in range(rows):                                      # row by row: a double copy of all would not be small
        x = logits[r, :V].double()
        p = torch.softmax(x, -1)
        ref = torch.logsumexp(x, -1) - x[tg[r].long()]
        # fp32 sums of exponentials of 2 ulp, and a logarithm of 2 ulp
        assert abs(got[r].double() - ref) <= 1e-5 * (1 + ref.abs()), (r, got[r], ref)
        want = p.clone()
        want[tg[r].long()] -= 1
        want *= dloss
        # the exponential is rounded to bf16 and the gradient again (one of each where the row spans blocks), each 2^-9
        assert ((lg[r, :V].double() - want).abs() <= 2.0 ** -8 * (p.abs() * dloss + want.abs()) + 1e-6).all(), r
    assert (lg[:, V:] == 0).all()


@pytest.mark.parametrize("rows,V,Vp", [(1300, 6975, 6976), (700, 6977, 6984), (650, 14079, 14080), (300, 14081, 14088), (300, 28159, 28160),
                                       (150, 28161, 28168), (30, 168957, 168960), (3, 168961, 168968)])
def test_fused_classifier_at_the_edges_of_the_block_sizes(rows, V, Vp):
    """The widest row of a block size and the narrowest of the next, several rows per block where they are narrow."""
    test_fused_classifier_over_blocks_and_clusters(rows, V, Vp)


def _ref_attention(qkv, B, T, NH, NKVH, HS):
    x = qkv.float().view(B, T, NH + 2 * NKVH, HS)
    q = x[:, :, :NH].transpose(1, 2)
    k = x[:, :, NH:NH + NKVH].transpose(1, 2).repeat_interleave(NH // NKVH, dim=1)
    v = x[:, :, NH + NKVH:].transpose(1, 2).repeat_interleave(NH // NKVH, dim=1)
    s = q @ k.transpose(-1, -2) / math.sqrt(HS)
    mask = torch.ones(T, T, device=qkv.device, dtype=torch.bool).tril()
    s = s.masked_fill(~mask, float("-inf"))
    p = s.softmax(-1)
    o = (p @ v).transpose(1, 2).reshape(B, T, NH * HS)
    return o, torch.logsumexp(s, -1)


@pytest.mark.parametrize("B,T,NH,HS", [(200, 128, 12, 64), (40, 256, 20, 64), (25, 448, 12, 64), (60, 128, 8, 128), (37, 320, 12, 64), (8, 320, 16, 128)])
def test_attention_forward_of_many_short_tiles(B, T, NH, HS, monkeypatch):
    """Several query tiles per resident block, most of them with one or two key tiles: every tile's rows are written, to their
    own place, each of many times (a block takes its next tile while the last one's rows leave)."""
    from llm_kittens_b200.ops import _native, attention

    assert -(-T // 128) * B * NH > 2 * torch.cuda.get_device_properties(0).multi_processor_count
    entries, call = [], _native.call
    monkeypatch.setattr(_native, "call", lambda name, *a: (entries.append(name), call(name, *a))[1])
    qkv = rnd(B, T, 3 * NH * HS)
    q, k, v = (t.view(B, T, NH, HS).transpose(1, 2).float() for t in qkv.split(NH * HS, dim=-1))
    ref = torch.nn.functional.scaled_dot_product_attention(q, k, v, is_causal=True).transpose(1, 2).reshape(B, T, NH * HS)
    first = None
    for _ in range(60):
        out = torch.full((B, T, NH * HS), float("nan"), device="cuda", dtype=BF)
        lse = torch.full((B, NH, T), float("nan"), device="cuda", dtype=torch.float32)
        attention.attention_fwd(qkv, B, T, NH, NH, HS, out=out, lse=lse, impl="tc")
        if first is None:
            first = out, lse
            assert (out.float() - ref).abs().max() < 0.03
        assert torch.equal(out, first[0]) and torch.equal(lse, first[1])
    assert entries == ["llmk_attention_fwd_tc"] * 60


@pytest.mark.parametrize("B,T,NH,NKVH,HS", [(2, 128, 4, 4, 64), (1, 256, 12, 12, 64), (2, 192, 8, 2, 64), (1, 128, 4, 2, 128),
                                            (1, 1024, 2, 1, 128)])
def test_attention_fwd_bwd(B, T, NH, NKVH, HS):
    from llm_kittens_b200.ops import _native, attention

    qkv = rnd(B, T, (NH + 2 * NKVH) * HS)
    out_w, lse_w = attention.attention_fwd(qkv, B, T, NH, NKVH, HS, impl="warp")
    out, lse = attention.attention_fwd(qkv, B, T, NH, NKVH, HS, impl="tc")   # the tcgen05 kernels where they take the length
    _native.check_status()
    assert maxerr(out, out_w) < 0.03 and maxerr(lse, lse_w) < 0.02
    qf = qkv.float().requires_grad_(True)
    ref, ref_lse = _ref_attention(qf, B, T, NH, NKVH, HS)
    assert maxerr(out, ref) < 0.03
    assert maxerr(lse, ref_lse) < 0.02
    dout = rnd(B, T, NH * HS)
    ref.backward(dout.float())
    dqkv_w = attention.attention_bwd(dout, qkv, out, lse, B, T, NH, NKVH, HS, impl="warp")
    assert maxerr(dqkv_w, qf.grad) < 0.08
    dqkv = attention.attention_bwd(dout, qkv, out, lse, B, T, NH, NKVH, HS)
    _native.check_status()
    assert maxerr(dqkv, qf.grad) < 0.08
    dqkv2 = attention.attention_bwd(dout, qkv, out, lse, B, T, NH, NKVH, HS)
    assert torch.equal(dqkv, dqkv2)


@pytest.mark.parametrize("dkv,HS", [("1", 64), ("2", 64), ("1", 128)])
@pytest.mark.parametrize("T,bad", [(256, 0), (256, 70), (256, 200), (320, 291)])
def test_attention_backward_with_one_query_that_is_nan(T, bad, HS, dkv, monkeypatch):
    """One query's scores, output and log-sum-exp are NaN. The keys after it never saw it: their dV is that of the other queries,
    and so is every other row of dQ."""
    from llm_kittens_b200.ops import _native, attention as attn

    monkeypatch.setenv("LLMK_ATTN_BWD_DKV", dkv)
    B, NH, NKVH = 2, 4, 2
    W, C = (NH + 2 * NKVH) * HS, NH * HS
    qkv, dout = rnd(B, T, W), rnd(B, T, C)
    clean = qkv.double()
    qkv[0, bad, HS:2 * HS] = float("nan")                     # head 1 of sequence 0, which reads key head 0
    out, lse = attn.attention_fwd(qkv, B, T, NH, NKVH, HS, impl="tc")
    assert lse[0, 1, bad].isnan() and lse.isnan().sum() == 1
    dqkv = attn.attention_bwd(dout, qkv, out, lse, B, T, NH, NKVH, HS)
    _native.check_status()
    clean[0, bad, HS:2 * HS] = 0                               # (any finite query: it has no part in what is compared)
    leaf = clean.requires_grad_(True)
    x = leaf.view(B, T, NH + 2 * NKVH, HS).transpose(1, 2)
    q, k, v = x[:, :NH], x[:, NH:NH + NKVH].repeat_interleave(NH // NKVH, 1), x[:, NH + NKVH:].repeat_interleave(NH // NKVH, 1)
    s = (q @ k.transpose(-1, -2) / math.sqrt(HS)).masked_fill(torch.ones(T, T, device="cuda", dtype=torch.bool).triu(1), float("-inf"))
    ((s.softmax(-1) @ v).transpose(1, 2).reshape(B, T, C) * dout.double()).sum().backward()
    got, want = dqkv.double(), leaf.grad
    # as in the comparison of the gradients of ordinary inputs
    dv = slice((NH + NKVH) * HS, (NH + NKVH + 1) * HS)
    assert (got[0, bad + 1:, dv] - want[0, bad + 1:, dv]).abs().max() < 0.08
    others = [t for t in range(T) if t != bad]
    assert (got[0, others, :C] - want[0, others, :C]).abs().max() < 0.08
    assert (got[1] - want[1]).abs().max() < 0.08


@pytest.mark.parametrize("dkv,impl", [("1", "tc"), ("2", "tc"), ("2", None)])
@pytest.mark.parametrize("B,T,NH,NKVH,HS", [(2, 320, 4, 2, 64), (3, 448, 2, 2, 64), (2, 320, 4, 1, 128), (2, 576, 2, 2, 128),
                                            (1, 1088, 4, 1, 64), (73, 1088, 5, 5, 64)])
def test_attention_of_lengths_that_are_not_whole_tiles(B, T, NH, NKVH, HS, dkv, impl, monkeypatch):
    """A ragged last tile reads nothing of the next sequence (which is all infinities here) and writes nothing behind its
    own; output, log-sum-exp and gradients against fp64, with both dK / dV kernels (one query head per key head makes the
    number of sub-tiles odd), after the tcgen05 forward and after the one that the size of the call picks. The last case has
    more heads than one group of the tile order."""
    from llm_kittens_b200.ops import attention as attn

    monkeypatch.setenv("LLMK_ATTN_BWD_DKV", dkv)
    W, n = (NH + 2 * NKVH) * HS, B * T
    small = B < 10
    qkv, dout = rnd(n + 64, W), rnd(n + 64, NH * HS)
    qkv[n:], dout[n:] = float("inf"), float("nan")
    if small:
        qkv.view(-1)[T * W:2 * T * W] = float("inf")         # sequence 1
    out, dqkv = torch.full((n + 64, NH * HS), 7.0, device="cuda", dtype=BF), torch.full((n + 64, W), 7.0, device="cuda", dtype=BF)
    lse, dvec = torch.full((B * NH * T + 64,), 7.0, device="cuda"), torch.empty(B, NH, T, device="cuda")
    attn.attention_fwd(qkv[:n].view(B, T, W), B, T, NH, NKVH, HS, out=out[:n], lse=lse, impl=impl)
    attn.attention_bwd(dout[:n], qkv[:n], out[:n], lse, B, T, NH, NKVH, HS, dqkv=dqkv[:n], dvec=dvec)
    assert (out[n:] == 7).all() and (dqkv[n:] == 7).all() and (lse[B * NH * T:] == 7).all()
    for b in ([0] + list(range(2, B)) if small else [0, 36, 72]):
        x = qkv[b * T:(b + 1) * T].double().view(T, NH + 2 * NKVH, HS).requires_grad_(True)
        q, k, v = x[:, :NH], x[:, NH:NH + NKVH].repeat_interleave(NH // NKVH, 1), x[:, NH + NKVH:].repeat_interleave(NH // NKVH, 1)
        sc = torch.einsum("qhd,khd->hqk", q, k) / math.sqrt(HS)
        sc = sc.masked_fill(~torch.tril(torch.ones(T, T, dtype=torch.bool, device="cuda")), -math.inf)
        ref = torch.einsum("hqk,khd->qhd", sc.softmax(-1), v).reshape(T, NH * HS)
        ref.backward(dout[b * T:(b + 1) * T].double())
        rel = lambda got, want: ((got.double() - want).norm() / want.norm()).item()
        # P, O, dS and the gradients are each rounded to bf16 once (2^-9 / sqrt(3) in the norm); the log-sum-exp is fp32
        assert rel(out[b * T:(b + 1) * T], ref) < 3e-3
        assert rel(lse[b * NH * T:(b + 1) * NH * T].view(NH, T), torch.logsumexp(sc, -1)) < 1e-5
        assert rel(dqkv[b * T:(b + 1) * T], x.grad.reshape(T, W)) < 4e-3


@pytest.mark.parametrize("dkv", ["", "1", "2"])
@pytest.mark.parametrize("B,T,NH,NKVH,HS,scale", [(1, 1024, 8, 2, 64, 1.0), (1, 2048, 4, 1, 64, 1.0), (1, 2048, 12, 12, 64, 1.0),
                                                  (1, 4096, 32, 8, 128, 1.0), (1, 1024, 12, 12, 64, 3.0), (1, 2048, 8, 2, 128, 3.0)])
def test_attention_long_sequences(B, T, NH, NKVH, HS, scale, dkv, monkeypatch):
    """The sequence lengths of the training configurations: many key tiles per query tile (the K/V ring wraps
    around), grouped queries, the pipelined and the plain dK/dV kernel (by the launcher's own choice, and each of them
    through LLMK_ATTN_BWD_DKV), and inputs scaled so that logits reach +-30 and the row maximum
    jumps by more than 2^8 between key tiles (the lazy rescale of the output accumulator fires)."""
    from llm_kittens_b200.ops import _native, attention

    if dkv:
        monkeypatch.setenv("LLMK_ATTN_BWD_DKV", dkv)
    else:
        monkeypatch.delenv("LLMK_ATTN_BWD_DKV", raising=False)
    torch.manual_seed(T + NH + HS)
    qkv = rnd(B, T, (NH + 2 * NKVH) * HS, scale=scale)
    out, lse = attention.attention_fwd(qkv, B, T, NH, NKVH, HS)
    _native.check_status()
    qf = qkv.float().requires_grad_(True)
    ref, ref_lse = _ref_attention(qf, B, T, NH, NKVH, HS)
    assert maxerr(out, ref) < (0.03 if scale == 1.0 else 0.05 * scale)   # outputs reach |5| at scale 3: one bf16 ulp there is 0.03
    assert maxerr(lse, ref_lse) < 0.02 * max(1.0, scale * scale)
    dout = rnd(B, T, NH * HS)
    ref.backward(dout.float())
    dqkv = attention.attention_bwd(dout, qkv, out, lse, B, T, NH, NKVH, HS)
    _native.check_status()
    assert maxerr(dqkv, qf.grad) < 0.08 * max(1.0, scale * scale)
    dqkv2 = attention.attention_bwd(dout, qkv, out, lse, B, T, NH, NKVH, HS)
    assert torch.equal(dqkv, dqkv2)


def _rope_ref(x, table, B, T, heads, HS, inverse=False):
    """fp32 rotation of the first ``heads`` heads of a packed [B*T, W] tensor, interleaved pairs."""
    x = x.float().clone().view(B, T, -1)
    part = x[..., : heads * HS].reshape(B, T, heads, HS // 2, 2)
    cos, sin = table[..., 0][None, :, None, :], table[..., 1][None, :, None, :]
    if inverse:
        sin = -sin
    x0, x1 = part[..., 0], part[..., 1]
    rot = torch.stack([x0 * cos - x1 * sin, x0 * sin + x1 * cos], dim=-1)
    x[..., : heads * HS] = rot.reshape(B, T, heads * HS)
    return x.view(B * T, -1)


@pytest.mark.parametrize("B,T,NH,NKVH,HS,C", [(2, 128, 4, 2, 64, 256), (1, 256, 8, 2, 128, 512), (1, 1024, 8, 2, 64, 512)])
def test_rope_in_the_qkv_projection_and_in_the_attention_backward(B, T, NH, NKVH, HS, C):
    """RoPE folded into the QKV GEMM's epilogue equals projection followed by an fp32 rotation; the attention backward
    with the table returns dq / dk already rotated back, equal to the plain backward followed by the inverse rotation."""
    from llm_kittens_b200.ops import _native, attention, elementwise as ew, gemm

    torch.manual_seed(B * T + HS)
    W = (NH + 2 * NKVH) * HS
    x, w = rnd(B * T, C), rnd(W, C, scale=0.05)
    table = ew.rope_tables(T, HS, 500000.0, False)
    fused = gemm.gemm_qkv_rope(x, w, table, T, (NH + NKVH) * HS, HS)
    _native.check_status()
    ref = _rope_ref(x.float() @ w.float().T, table, B, T, NH + NKVH, HS)
    assert maxerr(fused, ref) < 0.03
    unfused = ew.rope_qk_(gemm.gemm_nt(x, w), table, B, T, NH, NKVH, HS, interleaved=True)
    assert maxerr(fused, unfused) < 0.05   # the unfused path rounds to bf16 twice
    # backward
    qkv = fused.view(B, T, W)
    out, lse = attention.attention_fwd(qkv, B, T, NH, NKVH, HS)
    dout = rnd(B, T, NH * HS)
    plain = attention.attention_bwd(dout, qkv, out, lse, B, T, NH, NKVH, HS)
    want = _rope_ref(plain.view(B * T, W), table, B, T, NH + NKVH, HS, inverse=True)
    got = attention.attention_bwd(dout, qkv, out, lse, B, T, NH, NKVH, HS, rope=table)
    _native.check_status()
    assert maxerr(got.view(B * T, W), want) < 0.02 * max(1.0, want.abs().max().item())
    assert torch.equal(got.view(B * T, W)[:, (NH + NKVH) * HS:], plain.view(B * T, W)[:, (NH + NKVH) * HS:])   # dv untouched


def test_adamw_and_norm():
    from llm_kittens_b200.ops import optim

    n = 100000
    p32 = torch.randn(n, device="cuda")
    params = p32.to(BF)
    grads = rnd(n, scale=0.1)
    m, v = torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    master = torch.empty(n, device="cuda")
    segs, max_len = optim.make_segments([(0, 0, 0, 60000, True), (60000, 60000, 60000, 40000, False)])
    n2 = optim.global_norm2(grads, segs, max_len)
    assert abs(n2.item() - grads.float().pow(2).sum().item()) / n2.item() < 1e-4
    scale, norm_, flag = torch.empty(1, device="cuda"), torch.empty(1, device="cuda"), torch.zeros(1, device="cuda", dtype=torch.int32)
    optim.clip_scale(n2, 1.0, scale, norm_, flag)
    nrm = math.sqrt(n2.item())
    assert abs(scale.item() - min(1.0, 1.0 / nrm)) < 1e-5 and flag.item() == 0
    optim.master_from_params(master, params, segs, max_len)
    assert torch.equal(master, params.float())
    lr, b1, b2, eps, wd = 1e-2, 0.9, 0.95, 1e-8, 0.1
    gs = scale.item()
    ref_p = params.float().clone()
    g = grads.float() * gs
    rm = (1 - b1) * g
    rv = (1 - b2) * g * g
    mh, vh = rm / (1 - b1), rv / (1 - b2)
    wdv = torch.cat([torch.full((60000,), wd), torch.zeros(40000)]).cuda()
    ref_p = ref_p - lr * (mh / (vh.sqrt() + eps) + wdv * ref_p)
    optim.adamw(params, master, grads, m, v, segs, max_len, lr, b1, b2, 1, eps, wd, grad_scale_ptr=scale, seed=1234)
    assert maxerr(master, ref_p) < 1e-5
    assert maxerr(m, rm) < 1e-6 and maxerr(v, rv) < 1e-6
    # stochastic rounding: within one bf16 ulp of the fp32 value and unbiased on average
    ulp = (master.abs() * 2 ** -7).clamp_min(1e-30)
    assert ((params.float() - master).abs() <= ulp).all()
    assert abs((params.float() - master).mean().item()) < 1e-4
    p2 = torch.empty_like(params)
    optim.params_from_master(p2, master, segs, max_len, 1234)
    assert torch.equal(p2, params)


def test_scratch_buffers_stay_inside_their_guard_regions():
    """The kernels that write scratch memory through raw pointers (split-K partials, column-sum partials) get
    exactly-sized buffers between canary pages; the canaries must be intact afterwards. The damaged case is made on
    the host (a tensor fill over the whole allocation), not by a kernel."""
    import pytest as _pytest

    from llm_kittens_b200.ops import _native, elementwise as ew, gemm, norm

    _native.set_guards(True)
    try:
        for M, Nn, K in [(768, 768, 4096), (2304, 768, 8192), (520, 264, 1000), (3072, 768, 2048)]:
            a, b = rnd(K, M, scale=0.1), rnd(K, Nn, scale=0.1)
            out = gemm.gemm_tn(a, b)
            assert maxerr(out, a.float().T @ b.float()) < 0.02 * K ** 0.5
        for rows, C in [(1000, 768), (4096, 1024), (777, 2048), (512, 4096)]:
            x, w, bb = rnd(rows, C), rnd(C, scale=0.5) + 1, rnd(C, scale=0.1)
            _, mean, rstd = norm.layernorm_fwd(x, w, bb)
            dinp = torch.zeros(rows, C, device="cuda", dtype=BF)
            dw, db = torch.zeros(C, device="cuda", dtype=BF), torch.zeros(C, device="cuda", dtype=BF)
            norm.layernorm_bwd(dinp, dw, db, rnd(rows, C), x, w, mean, rstd, accumulate_dinp=False)
            _, rstd2 = norm.rmsnorm_fwd(x, w, 1e-5)
            norm.rmsnorm_bwd(dinp, dw, rnd(rows, C), x, w, rstd2, accumulate_dinp=False)
            ew.dbias(db, rnd(rows, C), accumulate=False)
        assert _native.check_guards() >= 8
        _native.check_status()
        # host-made damage is reported
        name, whole, payload = _native._GUARDED[0]
        whole[-1:].fill_(0)
        with _pytest.raises(_native.NativeError, match="guard region"):
            _native.check_guards()
    finally:
        _native.set_guards(False)


def test_peer_flag_wait_runs_out_and_reports_status():
    """Failure detection inside a kernel, without any fault: a wait on a peer flag that nothing sets gives up after its
    limit (0.2 s here), records LLMK_ST_TIMEOUT_PEER with the silent peer's index in the status word and returns; the
    host reads the word and raises; the context stays usable."""
    import time

    import pytest as _pytest

    from llm_kittens_b200.ops import _native, gemm

    lib = _native.lib()
    ctrl = torch.zeros(int(lib.llmk_comm_ctrl_ints()), dtype=torch.int32, device="cuda")
    _native.check_status()
    # every flag of slot 0 already at the awaited epoch: returns at once, status stays clear
    ctrl[:8] = 1
    _native.call("llmk_comm_wait", ctrl, 0, 1, 2, int(2e8), _native.status_word())
    _native.check_status()
    # peer 1 never signals epoch 2
    ctrl[0] = 2
    torch.cuda.synchronize()
    t0 = time.time()
    _native.call("llmk_comm_wait", ctrl, 0, 2, 2, int(2e8), _native.status_word())
    with _pytest.raises(_native.NativeError, match="status 5") as info:
        _native.check_status()
    waited = time.time() - t0
    assert 0.15 < waited < 5.0, waited
    assert "thread=1" in str(info.value)              # the peer that stayed silent
    # the status word was reset by the check and the context still runs kernels
    a, b = rnd(256, 128), rnd(256, 128, scale=0.05)
    assert maxerr(gemm.gemm_nt(a, b), a.float() @ b.float().T) < 0.05
    _native.check_status()
