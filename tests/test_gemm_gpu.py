"""tcgen05 GEMM vs an fp32 PyTorch reference (tolerance of the reference's dev/cuda/test_matmul.cu:216
is max-abs 0.5; ours is far tighter because accumulation is fp32 in TMEM)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(*shape, scale=1.0):
    return (torch.randn(*shape, device="cuda", dtype=torch.float32) * scale).to(torch.bfloat16)


def _close(got, ref, tol):
    """Within ``tol``, or within one rounding to bf16 where a value is so large that this is more (2^-9 of it, and as much again
    for a result on the other side of a rounding boundary)."""
    err = (got.float() - ref.float()).abs()
    assert (err <= (2.0 ** -8 * ref.float().abs()).clamp_min(tol)).all(), err.max().item()


def _gelu(x):
    return torch.nn.functional.gelu(x, approximate="tanh")


SHAPES_NT = [(128, 256, 64), (256, 512, 128), (384, 768, 768), (200, 264, 72), (1024, 2304, 768), (512, 50304, 768)]


@pytest.mark.parametrize("M,N,K", SHAPES_NT)
def test_gemm_nt_plain_and_bias(M, N, K):
    from llm_kittens_b200.ops import gemm, _native

    a, b, bias = _rand(M, K), _rand(N, K, scale=0.05), _rand(N)
    ref = a.float() @ b.float().T
    _close(gemm.gemm_nt(a, b), ref, 0.05)
    _close(gemm.gemm_nt(a, b, bias=bias), ref + bias.float(), 0.06)
    _native.check_status()


@pytest.mark.parametrize("M,N,K", [(256, 512, 128), (1024, 3072, 768), (200, 264, 72)])
def test_gemm_nt_gelu_and_add(M, N, K):
    from llm_kittens_b200.ops import gemm, _native

    a, b, bias = _rand(M, K), _rand(N, K, scale=0.05), _rand(N)
    ref = a.float() @ b.float().T + bias.float()
    pre = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    out = gemm.gemm_nt(a, b, bias=bias, gelu_pre_out=pre)
    _close(pre, ref, 0.06)
    _close(out, _gelu(ref), 0.06)
    res = _rand(M, N)
    out2 = gemm.gemm_nt(a, b, bias=bias, add=res)
    _close(out2, ref + res.float(), 0.08)
    res2 = res.clone()
    gemm.gemm_nt(a, b, bias=bias, add=res2, out=res2)  # in-place residual add
    _close(res2, ref + res.float(), 0.08)
    _native.check_status()


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (256, 768, 2304), (1024, 768, 3072), (200, 264, 72), (512, 768, 50304)])
def test_gemm_nn(M, N, K):
    from llm_kittens_b200.ops import gemm, _native

    a, b = _rand(M, K), _rand(K, N, scale=0.05)
    ref = a.float() @ b.float()
    tol = 0.05 if K < 10000 else 0.3
    _close(gemm.gemm_nn(a, b), ref, tol)
    pre = _rand(M, N)
    xg = pre.float().requires_grad_(True)
    _gelu(xg).sum().backward()
    _close(gemm.gemm_nn(a, b, dgelu_of=pre), ref * xg.grad, tol)
    _native.check_status()


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (768, 768, 4096), (2304, 768, 8192), (200, 264, 136), (50304, 768, 1024)])
def test_gemm_tn(M, N, K):
    from llm_kittens_b200.ops import gemm, _native

    a, b = _rand(K, M, scale=0.1), _rand(K, N, scale=0.1)
    ref = a.float().T @ b.float()
    out = gemm.gemm_tn(a, b)
    _close(out, ref, 0.1)
    acc = _rand(M, N)
    acc0 = acc.clone()
    gemm.gemm_tn(a, b, out=acc, accumulate=True)
    _close(acc, ref + acc0.float(), 0.15)
    _native.check_status()


@pytest.mark.parametrize("M,N,K", [(768, 768, 4096), (3072, 768, 8192), (3072, 3072, 2048), (200, 136, 1000), (2304, 768, 640)])
def test_gemm_tn_with_bias_gradient_from_the_same_launch(M, N, K):
    """dW and dbias of a linear layer from one kernel: the column sums of dout are taken from the A tiles in shared
    memory. The shapes cover split K (partials finished by the reduction kernel), one split with two tiles per CTA
    pair (sums written by the GEMM kernel itself), a ragged tile and a K that is no multiple of the k-block."""
    from llm_kittens_b200.ops import gemm, _native

    if not gemm.fused_dbias_available():
        pytest.skip("needs the CTA-pair GEMM kernel")
    launches = _native.launch_count()
    a, b = _rand(K, M, scale=0.1), _rand(K, N, scale=0.1)
    ref, ref_db = a.float().T @ b.float(), a.float().sum(0)

    def close_db(got, want):                          # one bf16 rounding of a sum of K values: relative
        err = (got.float() - want).abs()
        bad = err > 0.005 * want.abs() + 0.02
        assert not bad.any(), f"{int(bad.sum())} columns off, worst {err.max().item()}"

    db = torch.full((M,), 7.0, device="cuda", dtype=torch.bfloat16)
    out = gemm.gemm_tn(a, b, dbias=db)
    assert _native.launch_count() == launches + 1     # no stand-alone column-sum kernel ran
    _close(out, ref, 0.1)
    close_db(db, ref_db)
    acc, db2 = _rand(M, N), _rand(M)
    acc0, db0 = acc.clone(), db2.clone()
    gemm.gemm_tn(a, b, out=acc, accumulate=True, dbias=db2)
    _close(acc, ref + acc0.float(), 0.15)
    close_db(db2, ref_db + db0.float())
    # run-to-run bit equality (fixed summation order), and the same bits as the GEMM without the column sums
    db3 = torch.empty_like(db)
    out3 = gemm.gemm_tn(a, b, dbias=db3)
    assert torch.equal(db3, db) and torch.equal(out3, out)
    assert torch.equal(gemm.gemm_tn(a, b), out)
    _native.check_status()


@pytest.mark.parametrize("G,M,N,K", [(4, 512, 512, 256), (2, 256, 1000, 192), (4, 768, 3072, 4096), (2, 200, 264, 128)])
def test_grouped_gemm_tn_with_bias_gradients_per_group(G, M, N, K):
    """The experts of a mixture-of-experts layer: dW [G, M, N] and dbias [G, M] from one grouped launch (the last shape
    has ragged tiles and takes the route of one GEMM per group plus the grouped column-sum kernel)."""
    from llm_kittens_b200.ops import gemm, _native

    if not gemm.fused_dbias_available():
        pytest.skip("needs the CTA-pair GEMM kernel")
    a, b = _rand(G * K, M, scale=0.1), _rand(G * K, N, scale=0.1)
    ref = torch.stack([a[g * K:(g + 1) * K].float().T @ b[g * K:(g + 1) * K].float() for g in range(G)])
    ref_db = torch.stack([a[g * K:(g + 1) * K].float().sum(0) for g in range(G)])
    acc, db = _rand(G, M, N), _rand(G, M)
    acc0, db0 = acc.clone(), db.clone()
    launches = _native.launch_count()
    gemm.gemm_tn(a, b, out=acc, accumulate=True, groups=G, dbias=db)
    if M % 256 == 0 and K % 64 == 0:
        assert _native.launch_count() == launches + 1
    _close(acc, ref + acc0.float(), 0.15)
    err = (db.float() - (ref_db + db0.float())).abs()
    assert not (err > 0.005 * ref_db.abs() + 0.03).any(), err.max().item()
    out, db2 = torch.empty(G, M, N, device="cuda", dtype=torch.bfloat16), torch.empty(G, M, device="cuda", dtype=torch.bfloat16)
    gemm.gemm_tn(a, b, out=out, groups=G, dbias=db2)
    _close(out, ref, 0.1)
    assert not ((db2.float() - ref_db).abs() > 0.005 * ref_db.abs() + 0.02).any()
    assert torch.equal(gemm.gemm_tn(a, b, groups=G).view(G, M, N), out)
    _native.check_status()


@pytest.mark.parametrize("B,T,NH,K", [(2, 256, 4, 256), (4, 1024, 12, 768), (1, 2048, 32, 2048), (3, 128, 3, 192)])
def test_gemm_nn_with_the_attention_backward_row_sums_in_its_epilogue(B, T, NH, K):
    """dO = dres @ W from the GEMM and D[b, h, t] = sum over head h of dO * O from its epilogue, against the stand-alone
    pre-pass of the attention backward and an fp32 formula; the GEMM's own output must not change by a bit."""
    from llm_kittens_b200.ops import attention, gemm, _native

    if not gemm.fused_drow_available(64):
        pytest.skip("entry point not built")
    M, N = B * T, NH * 64
    a, w, o = _rand(M, K), _rand(K, N, scale=0.05), _rand(M, N)
    plain = gemm.gemm_nn(a, w)
    dvec = torch.full((B, NH, T), 7.0, device="cuda", dtype=torch.float32)
    out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    assert gemm.gemm_nn(a, w, out=out, drow_of=(o, dvec, T)) is out
    assert torch.equal(out, plain)
    ref = (plain.float() * o.float()).view(B, T, NH, 64).sum(-1).permute(0, 2, 1)
    assert (dvec - ref).abs().max().item() <= 1e-3 * ref.abs().max().item() + 1e-4
    prep = torch.empty_like(dvec)
    assert attention.attention_bwd_prep(plain, o, prep, B, T, NH, 64)
    assert (dvec - prep).abs().max().item() <= 1e-3 * ref.abs().max().item() + 1e-4
    dvec2 = torch.empty_like(dvec)
    gemm.gemm_nn(a, w, out=out, drow_of=(o, dvec2, T))
    assert torch.equal(dvec2, dvec)
    _native.check_status()


def test_gemm_deterministic():
    from llm_kittens_b200.ops import gemm

    a, b = _rand(4096, 768), _rand(4096, 768)
    o1 = gemm.gemm_tn(a, b).clone()
    o2 = gemm.gemm_tn(a, b)
    assert torch.equal(o1, o2)


@pytest.mark.parametrize("G,M,N,K", [(4, 512, 512, 256), (3, 256, 1000, 192), (2, 200, 264, 128)])
def test_gemm_grouped_matches_per_group_reference(G, M, N, K):
    """One launch for G equal-shaped problems (MoE experts); the last shape has rows that are not a multiple of the
    tile height, which takes the one-launch-per-group path of the wrapper."""
    from llm_kittens_b200.ops import gemm, _native

    # NT with bias + GELU: a [G*M,K], w [G,N,K], bias [G,N]
    a, w, bias = _rand(G * M, K), _rand(G, N, K, scale=0.05), _rand(G, N)
    pre = torch.empty(G * M, N, device="cuda", dtype=torch.bfloat16)
    out = gemm.gemm_nt(a, w, bias=bias, gelu_pre_out=pre, groups=G)
    for g in range(G):
        ref = a[g * M:(g + 1) * M].float() @ w[g].float().T + bias[g].float()
        _close(pre[g * M:(g + 1) * M], ref, 0.06)
        _close(out[g * M:(g + 1) * M], _gelu(ref), 0.06)
    # NN: dy [G*M,N] @ w [G,N,K] -> [G*M,K], with the dGELU factor
    dy = _rand(G * M, N)
    pre2 = _rand(G * M, K)
    dx = gemm.gemm_nn(dy, w, dgelu_of=pre2, groups=G)
    x = pre2.float().requires_grad_(True)
    _gelu(x).sum().backward()
    for g in range(G):
        ref = (dy[g * M:(g + 1) * M].float() @ w[g].float()) * x.grad[g * M:(g + 1) * M]
        _close(dx[g * M:(g + 1) * M], ref, 0.15)
    # TN: per-group weight gradient dy_g^T @ a_g accumulated into [G,N,K]
    dyw = _rand(G * M, N, scale=0.1)
    gw = _rand(G, N, K)
    gw0 = gw.clone()
    gemm.gemm_tn(dyw, a, out=gw, accumulate=True, groups=G)
    for g in range(G):
        ref = gw0[g].float() + dyw[g * M:(g + 1) * M].float().T @ a[g * M:(g + 1) * M].float()
        _close(gw[g], ref, 0.12)
    _native.check_status()


def test_gemm_polls_readiness_flags_of_its_weight_operand():
    """The consumer half of the tile-granular parameter gather: a GEMM whose weight is registered with per-chunk
    flags gives the plain result when the flags carry the expected tick (NT and NN layouts, tiles that span chunk
    borders), and when one chunk's flag never arrives the bounded wait runs out after the given limit: status 5
    (peer flag timeout) is read by the host and the context stays usable."""
    from llm_kittens_b200.ops import _native, gemm

    torch.manual_seed(0)
    M, Nn, K = 512, 640, 256
    a = (torch.randn(M, K, device="cuda") * 0.1).to(torch.bfloat16)
    w = (torch.randn(Nn, K, device="cuda") * 0.1).to(torch.bfloat16)
    d = (torch.randn(M, Nn, device="cuda") * 0.1).to(torch.bfloat16)
    chunk = 10240                       # elements per flag: 40 rows of the weight, so tiles straddle chunks
    nflags = (Nn * K + chunk - 1) // chunk
    flags = torch.zeros(nflags + 3, dtype=torch.int32, device="cuda")
    entry = gemm.register_b_ready(w, flags, 3, chunk, int(0.2e9))
    try:
        plain_nt = gemm.gemm_nt(a, w.clone())
        plain_nn = gemm.gemm_nn(d, w.clone())
        entry[3] = 7
        flags.fill_(7)
        torch.cuda.synchronize()
        assert torch.equal(gemm.gemm_nt(a, w), plain_nt)
        assert torch.equal(gemm.gemm_nn(d, w), plain_nn)
        _native.check_status()
        # an older tick in one flag = a chunk that has not landed: nothing sets it, the wait must run out
        flags[3 + nflags // 2] = 6
        torch.cuda.synchronize()
        gemm.gemm_nt(a, w)
        torch.cuda.synchronize()
        with pytest.raises(_native.NativeError, match="peer flag"):
            _native.check_status()
        flags.fill_(7)
        assert torch.equal(gemm.gemm_nt(a, w), plain_nt)   # the context and the kernels still work
        _native.check_status()
    finally:
        gemm.unregister_b_ready(w)


@pytest.mark.parametrize("M,H,K", [(256, 128, 64), (512, 768, 256), (300, 1024, 200), (4096, 8192, 2048)])
def test_gemm_swiglu_epilogue(M, H, K):
    """up / gate projections with SwiGLU in the epilogue against fp32 references and, bit for bit, against two plain
    GEMMs followed by the stand-alone SwiGLU kernel (the activation is computed from the rounded up / gate)."""
    from llm_kittens_b200.ops import _native, elementwise as ew, gemm

    torch.manual_seed(M + H)
    a, wu, wg = _rand(M, K), _rand(H, K, scale=0.1), _rand(H, K, scale=0.1)
    act, up, gate = (torch.empty(M, H, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    if not gemm.gemm_swiglu(a, wu, wg, act, up, gate):
        pytest.skip("fused SwiGLU kernel not available for this shape / device")
    _native.check_status()
    ref_up, ref_gate = a.float() @ wu.float().T, a.float() @ wg.float().T
    _close(up, ref_up, 0.02 * max(1.0, ref_up.abs().max().item()))
    _close(gate, ref_gate, 0.02 * max(1.0, ref_gate.abs().max().item()))
    up2, gate2 = gemm.gemm_nt(a, wu), gemm.gemm_nt(a, wg)
    assert torch.equal(up, up2) and torch.equal(gate, gate2)
    assert torch.equal(act, ew.swiglu_fwd(gate2, up2))


@pytest.mark.parametrize("M,N,K", [(8, 8, 512), (1, 776, 64), (64, 768, 3072), (200, 264, 1000), (256, 768, 3072), (512, 768, 2056),
                                   (1024, 768, 768), (129, 2056, 1608), (64, 4096, 14336), (2048, 1024, 4096)])
def test_gemm_of_few_tiles(M, N, K):
    """Shapes that the small-tile kernels take: one and several CTAs per tile, both tile widths, tiles cut by the edges of
    every dimension; NT and NN with every epilogue against fp64, bit-equal on repetition."""
    from llm_kittens_b200.ops import gemm, _native

    a, bt, bias, add = _rand(M, K), _rand(N, K, scale=0.05), _rand(N), _rand(M, N)
    b = bt.T.contiguous()
    ref = a.double() @ bt.double().T

    def close(got, want):
        # fp32 sums of K products (of order 0.05), then one rounding to bf16
        assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5 * K ** 0.5 + 1e-6).all()

    pre, pre2 = (torch.empty(M, N, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    calls = [lambda: gemm.gemm_nt(a, bt), lambda: gemm.gemm_nt(a, bt, bias=bias), lambda: gemm.gemm_nt(a, bt, add=add),
             lambda: gemm.gemm_nt(a, bt, bias=bias, add=add), lambda: gemm.gemm_nn(a, b), lambda: gemm.gemm_nn(a, b, add=add)]
    wants = [ref, ref + bias.double(), ref + add.double(), ref + bias.double() + add.double(), ref, ref + add.double()]
    for call, want in zip(calls, wants):
        got = call()
        close(got, want)
        assert torch.equal(got, call())
    out = gemm.gemm_nt(a, bt, bias=bias, gelu_pre_out=pre)
    close(pre, wants[1])
    assert ((out.double() - _gelu(pre.double())).abs() <= 2.0 ** -8 * pre.double().abs() + 2e-3).all()   # tanh.approx: 5e-4 relative
    x = add.double().requires_grad_(True)
    _gelu(x).sum().backward()
    got = gemm.gemm_nn(a, b, dgelu_of=add)
    assert ((got.double() - ref * x.grad).abs() <= 2.0 ** -8 * (ref * x.grad).abs() + 3e-3 * ref.abs() + 1e-3).all()
    _native.check_status()


@pytest.mark.parametrize("M,N,K", [(8, 8, 64), (768, 768, 256), (264, 200, 1001), (768, 768, 3136), (1024, 1024, 2048), (128, 2304, 77)])
def test_weight_and_bias_gradients_of_few_tiles(M, N, K):
    """TN with the bias gradient from the tensor core, accumulating and overwriting, K (tokens) not whole k-blocks."""
    from llm_kittens_b200.ops import gemm, _native

    a, b = _rand(K, M, scale=0.1), _rand(K, N)
    ref, refb = a.double().T @ b.double(), a.double().sum(0)

    def close(got, want, bound):
        assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + bound).all()

    out0, db0 = _rand(M, N), _rand(M)
    out, db = out0.clone(), db0.clone()
    gemm.gemm_tn(a, b, out=out, accumulate=True, dbias=db)
    close(out, out0.double() + ref, 1e-5 * K ** 0.5)
    close(db, db0.double() + refb, 1e-5 * K ** 0.5)
    out2, db2 = out0.clone(), db0.clone()
    gemm.gemm_tn(a, b, out=out2, accumulate=True, dbias=db2)
    assert torch.equal(out, out2) and torch.equal(db, db2)
    gemm.gemm_tn(a, b, out=out, dbias=db)
    close(out, ref, 1e-5 * K ** 0.5)
    close(db, refb, 1e-5 * K ** 0.5)
    close(gemm.gemm_tn(a, b), ref, 1e-5 * K ** 0.5)
    _native.check_status()


@pytest.mark.parametrize("M,T,H,K", [(64, 64, 384, 512), (320, 320, 256, 2048)])
def test_fused_epilogues_of_few_tiles(M, T, H, K):
    """RoPE, SwiGLU and D = rowsum(dO * O) epilogues of the small-tile kernels against fp64."""
    from llm_kittens_b200.ops import elementwise as ew
    from llm_kittens_b200.ops import gemm, _native

    a = _rand(M, K)
    tol = lambda want: 2.0 ** -8 * want.abs() + 1e-5 * K ** 0.5
    for HS in (64, 128):
        w, tab = _rand(6 * HS, K, scale=0.05), ew.rope_tables(T, HS, 10000.0, False, device="cuda")
        x = (a.double() @ w.double().T).view(M, 6, HS // 2, 2)
        cs = tab.double().view(T, HS // 2, 2)[torch.arange(M, device="cuda") % T][:, None]
        rot = torch.stack([x[..., 0] * cs[..., 0] - x[..., 1] * cs[..., 1], x[..., 1] * cs[..., 0] + x[..., 0] * cs[..., 1]], -1)
        want = torch.cat([rot[:, :4], x[:, 4:]], 1).reshape(M, 6 * HS)
        got = gemm.gemm_qkv_rope(a, w, tab, T, 4 * HS, HS)
        assert ((got.double() - want).abs() <= tol(want)).all()
    wu, wg = _rand(H, K, scale=0.05), _rand(H, K, scale=0.05)
    act, up, gate = (torch.empty(M, H, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    assert gemm.gemm_swiglu(a, wu, wg, act, up, gate)
    for got, w in ((up, wu), (gate, wg)):
        want = a.double() @ w.double().T
        assert ((got.double() - want).abs() <= tol(want)).all()
    want = torch.nn.functional.silu(gate.double()) * up.double()
    assert ((act.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all()
    NH = H // 64
    b, o = _rand(K, H, scale=0.05), _rand(M, H)
    dvec, dout = torch.empty(M // T, NH, T, device="cuda"), torch.empty(M, H, device="cuda", dtype=torch.bfloat16)
    assert gemm.gemm_nn(a, b, out=dout, drow_of=(o, dvec, T)) is not False
    want = a.double() @ b.double()
    assert ((dout.double() - want).abs() <= tol(want)).all()
    want = (dout.double() * o.double()).view(M // T, T, NH, 64).sum(-1).transpose(1, 2)
    assert ((dvec.double() - want).abs() <= 1e-5 * 64).all()
    _native.check_status()


@pytest.mark.parametrize("max_ctas", [0, 2, 24, 100, 132, 146, 148])
@pytest.mark.parametrize("M,N,K", [(256, 4224, 38976), (768, 3072, 16384), (1024, 1024, 8200), (2304, 768, 4096)])
def test_split_products_get_the_workspace_of_their_split_count(M, N, K, max_ctas):
    """The split count depends on how many CTAs work on a product and does not change steadily with it; buffers here hold
    exactly what is asked for, whatever the limit."""
    from llm_kittens_b200.ops import gemm, _native

    a, b = _rand(K, M, scale=0.1), _rand(K, N)
    want = a.double().T @ b.double()
    _native.set_guards(True)
    gemm.set_max_ctas(max_ctas)
    try:
        db = torch.empty(M, device="cuda", dtype=torch.bfloat16)
        out = gemm.gemm_tn(a, b, dbias=db)
        assert _native.check_guards() >= 0
    finally:
        gemm.set_max_ctas(0)
        _native.set_guards(False)
    # an fp32 chain of K / 16 additions (the tensor core adds 16 products at a time, rounding the sum by at most 2^-23 of it,
    # and the running sums are of the size of the largest result), then one rounding to bf16
    chain = K / 16 * 2.0 ** -23 * want.abs().max()
    assert ((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + chain).all()
    assert ((db.double() - a.double().sum(0)).abs() <= 2.0 ** -8 * a.double().sum(0).abs() + 1e-5 * K ** 0.5).all()
    _native.check_status()


@pytest.mark.parametrize("M", [1, 5, 60, 130, 200])
def test_rows_of_few_tiles_dealt_out_unevenly_over_a_cluster(M):
    """The rows of a tile are summed by the CTAs of its cluster: row counts that are no multiple of the cluster size, fewer
    rows than CTAs, and the epilogues whose lanes work together (D = rowsum(dO * O), bias gradient) on such rows."""
    from llm_kittens_b200.ops import gemm, _native

    N, K, T = 768, 3072, 5 if M % 5 == 0 else 1
    a, w, bias, add = _rand(M, K), _rand(N, K, scale=0.05), _rand(N), _rand(M, N)
    want = a.double() @ w.double().T
    tol = lambda x: 2.0 ** -8 * x.abs() + 1e-5 * K ** 0.5   # fp32 sums of K products of order 0.05, one rounding to bf16
    got = gemm.gemm_nt(a, w, bias=bias, add=add)
    x = want + bias.double() + add.double()
    assert ((got.double() - x).abs() <= tol(x)).all()
    dvec, out = torch.empty(M // T, N // 64, T, device="cuda"), torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    assert gemm.gemm_nn(a, w.T.contiguous(), out=out, drow_of=(add, dvec, T)) is not False
    assert ((out.double() - want).abs() <= tol(want)).all()
    d = (out.double() * add.double()).view(M // T, T, N // 64, 64).sum(-1).transpose(1, 2)
    assert ((dvec.double() - d).abs() <= 1e-5 * 64).all()
    cols = 8 * M
    b, dout = _rand(3000, 256), _rand(3000, cols)
    dw, db = _rand(cols, 256), _rand(cols)
    dw0, db0 = dw.double(), db.double()
    gemm.gemm_tn(dout, b, out=dw, accumulate=True, dbias=db)
    for got, x in ((dw, dw0 + dout.double().T @ b.double()), (db, db0 + dout.double().sum(0))):
        assert ((got.double() - x).abs() <= 2.0 ** -8 * x.abs() + 1e-4 * 3000 ** 0.5).all()
    _native.check_status()


@pytest.mark.parametrize("M", [1, 33, 64, 200, 320, 400, 512])
@pytest.mark.parametrize("N,K", [(50312, 1032), (20008, 72)])
def test_gemm_of_few_rows_and_a_wide_output(M, N, K):
    """Rows on the N side of the MMA: counts that are no multiple of 32, one and two MMAs per weight tile, a last weight tile that
    is cut, K not whole k-blocks; nothing is written behind the rows and columns that exist."""
    from llm_kittens_b200.ops import gemm, _native

    a, w = _rand(M, K), _rand(N, K, scale=0.05)
    want = a.double() @ w.double().T
    whole = torch.full((M * N + 4096,), 7.0, device="cuda", dtype=torch.bfloat16)
    out = whole[:M * N].view(M, N)
    gemm.gemm_nt(a, w, out=out)
    # fp32 sums of K products of order 0.05, one rounding to bf16
    assert ((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5 * K ** 0.5).all()
    assert (whole[M * N:] == 7.0).all()
    assert torch.equal(out, gemm.gemm_nt(a, w))
    _native.check_status()


@pytest.mark.parametrize("M,H,K", [(320, 8192, 512), (257, 8320, 136), (64, 19072, 264), (512, 8192, 512)])
def test_swiglu_of_few_rows_and_a_wide_output(M, H, K):
    from llm_kittens_b200.ops import gemm, _native

    a, wu, wg = _rand(M, K), _rand(H, K, scale=0.05), _rand(H, K, scale=0.05)
    act, up, gate = (torch.empty(M, H, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    assert gemm.gemm_swiglu(a, wu, wg, act, up, gate)
    for got, w in ((up, wu), (gate, wg)):
        want = a.double() @ w.double().T
        assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5 * K ** 0.5).all()
    want = torch.nn.functional.silu(gate.double()) * up.double()
    assert ((act.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all()
    _native.check_status()


def _guarded(M, N):
    whole = torch.full((M * N + 4096,), 7.0, device="cuda", dtype=torch.bfloat16)
    return whole, whole[:M * N].view(M, N)


@pytest.mark.parametrize("M", [1, 33, 64, 200, 257, 320, 400, 512])
@pytest.mark.parametrize("N,K", [(264, 72), (8, 1032), (20008, 136), (40200, 520)])
@pytest.mark.parametrize("swiglu", [False, True])
def test_the_kernel_of_few_rows_itself(M, N, K, swiglu):
    """Asked for by name, whatever the rule picks: one and two MMAs per weight tile and one and two stretches of tokens, counts that are no
    multiple of 32, a last weight tile that is cut (or nearly empty), K not whole k-blocks, several units per pair of blocks; guards
    behind every output."""
    from llm_kittens_b200.ops import _native

    if swiglu and N > 30000:
        N = 20104                                              # (several units per pair of blocks too, at half the width)
    a, wu, wg = _rand(M, K), _rand(N, K, scale=0.05), _rand(N, K, scale=0.05)
    (cw, c), (uw, up), (gw, gate) = (_guarded(M, N) for _ in range(3))
    args = (wg, c, up, gate) if swiglu else (None, c, None, None)
    _native.call("llmk_gemm_few_rows", a, wu, *args, M, N, K, _native.status_word())
    _native.check_status()
    # fp32 sums of K products of order 0.05, one rounding to bf16
    within = lambda got, want: ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5 * K ** 0.5).all()
    u = a.double() @ wu.double().T
    if swiglu:
        assert within(up, u) and within(gate, a.double() @ wg.double().T)
        assert within(c, torch.nn.functional.silu(gate.double()) * up.double())
    else:
        assert within(c, u)
    first = c.clone()
    _native.call("llmk_gemm_few_rows", a, wu, *args, M, N, K, _native.status_word())
    assert torch.equal(c, first)
    for whole in (cw, uw, gw):
        assert (whole[M * N:] == 7.0).all()


@pytest.mark.parametrize("M,N,K,swiglu", [(320, 128256, 2048, 0), (448, 128256, 2048, 0), (320, 50304, 1600, 0), (64, 14336, 4096, 1), (320, 8192, 2048, 1),
                                          (257, 8192, 2048, 1), (320, 14336, 4096, 1)])
def test_products_that_take_the_kernel_of_few_rows(M, N, K, swiglu):
    """What the rule picks gives that kernel's bits; one row more than it can hold does not take it."""
    from llm_kittens_b200.ops import gemm, _native

    assert _native.lib().llmk_gemm_takes_few_rows(M, N, K, swiglu) == 1 and _native.lib().llmk_gemm_takes_few_rows(513, N, K, swiglu) == 0
    a, wu, wg = _rand(M, K), _rand(N, K, scale=0.05), _rand(N, K, scale=0.05)
    got, want = ([torch.empty(M, N, device="cuda", dtype=torch.bfloat16) for _ in range(3)] for _ in range(2))
    if swiglu:
        assert gemm.gemm_swiglu(a, wu, wg, *got)
        _native.call("llmk_gemm_few_rows", a, wu, wg, *want, M, N, K, _native.status_word())
    else:
        gemm.gemm_nt(a, wu, out=got[0])
        _native.call("llmk_gemm_few_rows", a, wu, None, want[0], None, None, M, N, K, _native.status_word())
    assert all(torch.equal(x, y) for x, y in list(zip(got, want))[: 3 if swiglu else 1])
    _native.check_status()


@pytest.mark.parametrize("M,N,K", [(200, 8192, 8192), (72, 2056, 32768), (768, 768, 16384), (264, 4104, 12288)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_weight_and_bias_gradient_from_split_partials(M, N, K, accumulate):
    """Column counts that are no multiple of the 64 of a finishing block, and more rows of partials than its 32 lanes."""
    from llm_kittens_b200.ops import gemm

    g = torch.Generator(device="cuda").manual_seed(M + N)
    a, b = (torch.randn(K, w, device="cuda", generator=g).to(torch.bfloat16) for w in (M, N))
    c0, d0 = torch.randn(M, N, device="cuda", generator=g).to(torch.bfloat16), torch.randn(M, device="cuda", generator=g).to(torch.bfloat16)
    out, db = c0.clone(), d0.clone()
    gemm.gemm_tn(a, b, out=out, accumulate=accumulate, dbias=db)
    ref, dref = a.double().T @ b.double(), a.double().sum(0)
    if accumulate:
        ref, dref = ref + c0.double(), dref + d0.double()
    # fp32 sums of K terms (3e-6 of their root sum of squares K^0.5), one rounding to bf16
    tol = K ** 0.5 * 1e-4
    assert ((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + tol).all()
    assert ((db.double() - dref).abs() <= 2.0 ** -8 * dref.abs() + tol).all()
    again, db2 = c0.clone(), d0.clone()
    gemm.gemm_tn(a, b, out=again, accumulate=accumulate, dbias=db2)
    assert torch.equal(again, out) and torch.equal(db2, db)
