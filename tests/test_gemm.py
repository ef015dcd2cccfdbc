"""tcgen05 GEMM and its fused epilogues against fp32 torch references of the same bf16 inputs (GPU).

Tolerance: the kernel accumulates in fp32 and rounds to bf16, so it agrees with the fp32 reference to one bf16 rounding
(2^-8 relative), twice where an epilogue rounds before a non-linearity and a tie falls the other way:
|got - want| <= 2^-6 * |want| + 2^-7 * rms(want)."""
import pytest
import torch

gpu = pytest.mark.gpu


def _check(got, want, what, mid=None):
    """``mid``: an intermediate the epilogue rounds to bf16 before adding something to it (the module output ahead of a
    residual add); one ulp of it is allowed on top, since it does not shrink when the sum cancels."""
    got, want = got.float(), want.float()
    tol = 2.0 ** -6 * want.abs() + 2.0 ** -7 * want.pow(2).mean().sqrt()
    if mid is not None:
        tol = tol + 2.0 ** -7 * mid.float().abs()
    bad = (got - want).abs() > tol
    assert not bad.any(), f"{what}: {int(bad.sum())} of {bad.numel()} outside tolerance, max err {(got - want).abs().max():.4g}"


def _rand(*shape, scale=1.0, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(torch.bfloat16)


@gpu
@pytest.mark.parametrize("m,n,k", [(128, 256, 64), (1, 256, 512), (64, 768, 768), (200, 256, 768), (1000, 2304, 768), (4096, 1024, 3072), (12544, 768, 3072)])
def test_gemm_plain(m, n, k):
    from ittai_b200 import ops
    a, w = _rand(m, k, seed=1), _rand(n, k, scale=0.05, seed=2)
    st = ops.new_status("cuda")
    out = ops.gemm(a, w, st)
    ops.check_status(st)
    _check(out, a.float() @ w.float().t(), f"gemm {m}x{n}x{k}")


@gpu
@pytest.mark.parametrize("n,k", [(1024, 2048), (768, 64), (256, 3072)])
def test_one_sm_and_two_sm_kernels_agree_bit_for_bit(n, k):
    """A row's value does not depend on how many rows share the launch: up to one round of 128 x 64 tiles on the SMs the one-SM
    kernel runs, above it the two-SM kernel (both sides of the line, and one row past a tile)."""
    from ittai_b200 import ops
    n_sms = torch.cuda.get_device_properties(0).multi_processor_count
    last = n_sms // (n // 64) * 128
    a, w, bias, res = _rand(last + 200, k, seed=51), _rand(n, k, scale=0.05, seed=52), _rand(n, seed=53).float(), _rand(last + 200, n, seed=54)
    st = ops.new_status("cuda")
    want = ops.gemm(a, w, st, bias=bias, residual=res)
    _check(want, res.float() + (a.float() @ w.float().t() + bias).to(torch.bfloat16).float(), "two-SM", mid=a.float() @ w.float().t() + bias)
    for m in (1, 128, 129, 300, last, last + 1):
        guard = torch.full((m + 1, n), 3.0, dtype=torch.bfloat16, device="cuda")
        got = ops.gemm(a[:m], w, st, bias=bias, residual=res[:m], out=guard[:m])
        assert torch.equal(got, want[:m]) and (guard[m] == 3.0).all(), m
    ops.check_status(st)


@gpu
@pytest.mark.parametrize("m", [2, 7, 8, 9, 16, 57, 120, 121, 127])
def test_short_tiles_load_only_their_rows(m):
    """The one-SM kernel's tile of fewer than 128 rows (boxes of A rounded up to eight rows), behind a launch that leaves NaNs in the stages: the
    bits of the same rows in a tile of 128, several times round the ring of stages, and no row past the last."""
    from ittai_b200 import ops
    a, w, res = _rand(128, 2048, seed=61), _rand(1024, 2048, scale=0.05, seed=62), _rand(128, 1024, seed=63)
    st = ops.new_status("cuda")
    want = ops.gemm(a, w, st, residual=res)
    ops.gemm(torch.full_like(a, float("nan")), w, st)
    guard = torch.full((m + 1, 1024), 3.0, dtype=torch.bfloat16, device="cuda")
    got = ops.gemm(a[:m], w, st, residual=res[:m], out=guard[:m])
    ops.check_status(st)
    assert torch.equal(got, want[:m]) and (guard[m] == 3.0).all()


@gpu
@pytest.mark.parametrize("n,k", [(4096, 2048), (4352, 2048), (256, 3072), (256, 3136), (16384, 512), (151808, 64)])
def test_weights_ahead_of_the_wait_and_not(n, k):
    """Both sides of the lines up to which the one-SM kernel brings W into L2 first (16 MiB, K 3072), behind a launch that writes nothing of it."""
    from ittai_b200 import ops
    a, w = _rand(70, k, seed=64), _rand(n, k, scale=0.05, seed=65)
    st = ops.new_status("cuda")
    for m in (70, 5):
        _check(ops.gemm(a[:m], w, st), a[:m].float() @ w.float().T, f"W {n} x {k}, {m} rows")
    ops.check_status(st)


@gpu
def test_a_weight_beyond_l2_streams_at_the_rate_of_memory():
    """537 MB of weights for 64 rows: 1.2 times as long as a copy that moves as many bytes.  (Requested as a whole ahead of its use, 1.5 times.)"""
    from ittai_b200 import ops
    a, w = _rand(64, 4096, seed=66), torch.zeros(65536, 4096, dtype=torch.bfloat16, device="cuda")
    half = w.numel() // 2
    src, dst = torch.zeros(2, half, dtype=torch.bfloat16, device="cuda")
    st, out = ops.new_status("cuda"), torch.empty(64, 65536, dtype=torch.bfloat16, device="cuda")

    def us(call):
        times = []
        for _ in range(9):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            for _ in range(5):
                call()
            e[1].record()
            torch.cuda.synchronize()
            times.append(e[0].elapsed_time(e[1]) * 200)
        return sorted(times)[4]

    copy = us(lambda: dst.copy_(src))
    assert us(lambda: ops.gemm(a, w, st, out=out)) < 1.38 * copy, copy
    ops.check_status(st)


@gpu
def test_gemm_row_identity():
    """A = rows of the identity picks out columns of W: catches a wrong swizzle or K-step in the operand descriptors."""
    from ittai_b200 import ops
    k, n = 256, 256
    a = torch.eye(k, device="cuda", dtype=torch.bfloat16)
    w = _rand(n, k, seed=3)
    st = ops.new_status("cuda")
    out = ops.gemm(a, w, st)
    ops.check_status(st)
    assert torch.equal(out, w.t().contiguous())


@gpu
def test_gemm_bias_gelu_residual_swiglu():
    from ittai_b200 import _C, ops
    m, n, k = 392, 3072, 768
    a, w = _rand(m, k, seed=4), _rand(n, k, scale=0.05, seed=5)
    bias = _rand(n, seed=7).float() * 0.1
    res = _rand(m, n, seed=6)
    st = ops.new_status("cuda")
    acc = a.float() @ w.float().t()
    rb = lambda x: x.to(torch.bfloat16).float()
    _check(ops.gemm(a, w, st, bias=bias), acc + bias, "bias")
    _check(ops.gemm(a, w, st, bias=bias, epi=_C.EPI_GELU),
           torch.nn.functional.gelu(rb(acc + bias), approximate="tanh"), "bias + gelu")
    _check(ops.gemm(a, w, st, bias=bias, residual=res), res.float() + rb(acc + bias), "bias + residual", mid=acc + bias)
    _check(ops.gemm(a, w, st, residual=res), res.float() + rb(acc), "residual", mid=acc)
    g, u = rb(acc[:, 0::2]), rb(acc[:, 1::2])
    _check(ops.gemm(a, w, st, epi=_C.EPI_SWIGLU), rb(torch.nn.functional.silu(g)) * u, "swiglu")
    ops.check_status(st)


@gpu
@pytest.mark.parametrize("m,n,k,epi", [(1000, 2304, 768, 0), (12544, 3072, 768, 1), (196, 1536, 768, 0)])
def test_gemm_folded_layernorm(m, n, k, epi):
    """Linear(LayerNorm(x)) with the LayerNorm folded into the GEMM (row statistics in the epilogue) against the unfused
    fp32 computation; rows carry a large common offset so that a wrong mean term would show."""
    import torch.nn.functional as F
    from ittai_b200 import _C, ops
    x = (_rand(m, k, seed=11).float() * 1.5 + 3.0).to(torch.bfloat16)
    w, bias = _rand(n, k, scale=0.05, seed=12), torch.randn(n, device="cuda")
    gain, beta = torch.rand(k, device="cuda") + 0.5, torch.randn(k, device="cuda") * 0.1
    st = ops.new_status("cuda")
    stats = ops.row_stats(x, 1e-6)
    xf = x.float()
    assert torch.allclose(stats[:, 0], xf.mean(-1), atol=1e-5, rtol=1e-5)
    assert torch.allclose(stats[:, 1], torch.rsqrt(xf.var(-1, unbiased=False) + 1e-6), rtol=1e-4)
    wp, bp, cs = ops.fold_layernorm(w, bias, gain, beta)
    out = ops.gemm(x, wp, st, bias=bp, epi=_C.EPI_GELU if epi else _C.EPI_NONE, row_stats=stats, col_sums=cs)
    ops.check_status(st)
    want = F.linear(F.layer_norm(xf, (k,), gain, beta, 1e-6), w.float(), bias)
    if epi:
        want = F.gelu(want.to(torch.bfloat16).float(), approximate="tanh")
    _check(out, want, f"folded LayerNorm gemm {m}x{n}x{k} epi={epi}")


@gpu
def test_gemm_statistics_from_the_producing_epilogue():
    """A GEMM writes (sum, sum of squares) of its output rows per 128-column slice; the next GEMM finishes mean / rstd
    from them and applies the folded LayerNorm: the pair must match LayerNorm + Linear on the stored bf16 rows."""
    import torch.nn.functional as F
    from ittai_b200 import ops
    m, d, n = 1000, 768, 2304
    a0, w0, r0 = _rand(m, d, seed=21), _rand(d, d, scale=0.05, seed=22), (_rand(m, d, seed=23).float() * 2 + 1).to(torch.bfloat16)
    st = ops.new_status("cuda")
    parts = torch.full((m, d // 128, 2), float("nan"), device="cuda")
    x = ops.gemm(a0, w0, st, residual=r0, stats_out=parts)
    xf = x.float().view(m, d // 128, 128)
    assert torch.allclose(parts[..., 0], xf.sum(-1), rtol=1e-5, atol=1e-3)
    assert torch.allclose(parts[..., 1], xf.pow(2).sum(-1), rtol=1e-5, atol=1e-3)
    w, bias = _rand(n, d, scale=0.05, seed=24), torch.randn(n, device="cuda")
    gain, beta = torch.rand(d, device="cuda") + 0.5, torch.randn(d, device="cuda") * 0.1
    wp, bp, cs = ops.fold_layernorm(w, bias, gain, beta)
    out = ops.gemm(x, wp, st, bias=bp, row_stats=parts, col_sums=cs, stats_eps=1e-6)
    ops.check_status(st)
    _check(out, F.linear(F.layer_norm(x.float(), (d,), gain, beta, 1e-6), w.float(), bias), "folded LayerNorm from epilogue statistics")


@gpu
def test_gemm_strided_views():
    """Operands and output as column slices of wider buffers (leading dimension > width)."""
    from ittai_b200 import ops
    big_a, big_w = _rand(256, 1024, seed=7), _rand(512, 1024, scale=0.05, seed=8)
    a, w = big_a[:, 256:768], big_w[:, 512:1024]
    out_big = torch.zeros(256, 1024, dtype=torch.bfloat16, device="cuda")  # columns 128..640 receive the product
    st = ops.new_status("cuda")
    ops.gemm(a, w, st, out=out_big[:, 128:640])
    ops.check_status(st)
    _check(out_big[:, 128:640], a.float() @ w.float().t(), "strided")
    assert (out_big[:, :128] == 0).all() and (out_big[:, 640:] == 0).all()


def test_gemm_argument_errors():
    import ctypes as C
    from ittai_b200 import _C
    g = _C.Gemm()
    assert _C.lib().ittai_gemm_bf16_launch(C.byref(g), None) == -1


@gpu
@pytest.mark.parametrize("m", [12544, 700])
def test_gemm_chain_equals_separate_launches(m):
    """Four dependent GEMMs of the SigLIP layer shapes (out-proj with an in-place residual and output statistics, fc1 with
    a folded LayerNorm and GELU, fc2 with an in-place residual, the next QKV projection with a folded LayerNorm) in one
    persistent launch: bit-identical to the same GEMMs launched one by one, on a second run over the same flag buffer
    (cleared in between) as well."""
    from ittai_b200 import _C, ops
    D, F = 768, 3072
    gen = torch.Generator(device="cuda").manual_seed(4)
    rnd = lambda *s, scale=1.0: (torch.randn(*s, generator=gen, device="cuda") * scale)
    attn, x0 = rnd(m, D).bfloat16(), rnd(m, D).bfloat16()
    wo, w1, w2, wq = rnd(D, D, scale=0.03).bfloat16(), rnd(F, D, scale=0.03).bfloat16(), rnd(D, F, scale=0.02).bfloat16(), rnd(3 * D, D, scale=0.03).bfloat16()
    bo, b1, b2, bq = rnd(D, scale=0.1), rnd(F, scale=0.1), rnd(D, scale=0.1), rnd(3 * D, scale=0.1)
    cs1, csq = w1.float().sum(1), wq.float().sum(1)
    st = ops.new_status(attn.device)

    def run(chained):
        x, h, qkv = x0.clone(), torch.empty(m, F, dtype=torch.bfloat16, device="cuda"), torch.empty(m, 3 * D, dtype=torch.bfloat16, device="cuda")
        sa, sm = (torch.zeros(m, D // 128, 2, device="cuda") for _ in range(2))
        args = [dict(a=attn, w=wo, bias=bo, residual=x, out=x, stats_out=sa),
                dict(a=x, w=w1, bias=b1, epi=_C.EPI_GELU, out=h, row_stats=sa, col_sums=cs1, stats_eps=1e-6),
                dict(a=h, w=w2, bias=b2, residual=x, out=x, stats_out=sm),
                dict(a=x, w=wq, bias=bq, out=qkv, row_stats=sm, col_sums=csq, stats_eps=1e-6)]
        if chained:
            flags = torch.zeros(4 * 2 * ((m + 255) // 256), dtype=torch.int32, device="cuda")
            for _ in range(2):
                x.copy_(x0)
                flags.zero_()
                ops.gemm_chain([ops.gemm_desc(k.pop("a"), k.pop("w"), st, **k)[0] for k in [dict(d) for d in args]], flags)
        else:
            for d in args:
                d = dict(d)
                ops.gemm(d.pop("a"), d.pop("w"), st, **d)
        ops.check_status(st)
        return x, h, qkv, sa, sm

    for got, want, name in zip(run(True), run(False), ("x", "h", "qkv", "stats_a", "stats_m")):
        assert torch.equal(got, want), f"{name}: chained GEMMs differ from separate launches ({(got.float() - want.float()).abs().max().item():.4g})"


@gpu
@pytest.mark.parametrize("k", [64, 128, 192])
def test_gemm_chain_with_a_short_first_gemm(k):
    """K of one to three k-blocks: the loads run up to seven tiles ahead of the epilogue, over eight tiles of the first GEMM for
    every pair of SMs.  The same bits as separate launches."""
    from ittai_b200 import _C, ops
    n = 512
    m = torch.cuda.get_device_properties(0).multi_processor_count // 2 * 1024
    a, w0, w1, b0, st = _rand(m, k, seed=91), _rand(n, k, scale=0.05, seed=92), _rand(n, n, scale=0.05, seed=93), _rand(n, seed=94).float(), ops.new_status("cuda")
    x, y = (torch.zeros(m, n, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    want_x = ops.gemm(a, w0, st, bias=b0, epi=_C.EPI_GELU)
    want_y = ops.gemm(want_x, w1, st)
    flags = torch.zeros(2 * 2 * ((m + 255) // 256), dtype=torch.int32, device="cuda")
    ops.gemm_chain([ops.gemm_desc(a, w0, st, bias=b0, epi=_C.EPI_GELU, out=x)[0], ops.gemm_desc(x, w1, st, out=y)[0]], flags)
    ops.check_status(st)
    assert torch.equal(x, want_x) and torch.equal(y, want_y)


@gpu
def test_gemm_chain_from_residual_to_plain_tiles():
    """As many tiles of a GEMM with a residual as make three for every pair of SMs, then one without: the warps go from one staging
    tile to three in rotation, on the first again.  Short main loops, so that the next accumulator is there before a tile is stored.  The
    second GEMM also reads the row statistics that all lanes of the first one's epilogue warps wrote with ordinary stores.  The same bits
    as separate launches, several times."""
    from ittai_b200 import ops
    n, k = 768, 256
    m = torch.cuda.get_device_properties(0).multi_processor_count // 2 * 256
    a, w0, w1, x0, st = _rand(m, k, seed=81), _rand(n, k, scale=0.05, seed=82), _rand(n, n, scale=0.05, seed=83), _rand(m, n, seed=84), ops.new_status("cuda")
    x, y, want_s, s = torch.empty_like(x0), torch.empty_like(x0), *(torch.empty(m, n // 128, 2, device="cuda") for _ in range(2))
    cs = w1.float().sum(1)
    want_x = ops.gemm(a, w0, st, residual=x0, stats_out=want_s)
    want_y = ops.gemm(want_x, w1, st, row_stats=want_s, col_sums=cs, stats_eps=1e-6)
    flags = torch.zeros(2 * 2 * ((m + 255) // 256), dtype=torch.int32, device="cuda")
    for _ in range(4):
        flags.zero_()
        s.fill_(float("nan"))
        ops.gemm_chain([ops.gemm_desc(a, w0, st, residual=x0, out=x, stats_out=s)[0], ops.gemm_desc(x, w1, st, out=y, row_stats=s, col_sums=cs, stats_eps=1e-6)[0]], flags)
        ops.check_status(st)
        assert torch.equal(x, want_x) and torch.equal(s, want_s) and torch.equal(y, want_y)


@gpu
@pytest.mark.parametrize("m", [129, 1300, 2500])
def test_consecutive_tiles_keep_to_their_rows(m):
    """GEMMs that fetch something per token give a pair of CTAs consecutive tiles: runs that begin and end inside a row block, and
    cross one (m 1300, 2500).  Rotary epilogue with a folded RMSNorm against the same GEMM and the row-wise pass (the same rounding
    steps; the head norm's sum is taken in another order, which flips a rounding now and then), and a folded LayerNorm with residual and
    output statistics against torch."""
    from ittai_b200 import _C, ops
    from ittai_b200.qwen3.decoder import rope_table
    g = torch.Generator(device="cuda").manual_seed(m)
    x, w, st = _rand(m, 1024, seed=61), _rand(4096, 1024, scale=0.05, seed=62), ops.new_status("cuda")
    cap = m + 7
    qn, kn = (torch.rand(128, generator=g, device="cuda") + 0.5).to(torch.bfloat16), (torch.rand(128, generator=g, device="cuda") + 0.5).to(torch.bfloat16)
    pos = torch.randint(0, 400, (m,), generator=g, device="cuda", dtype=torch.int32)
    seq, slot = torch.zeros(m, dtype=torch.int32, device="cuda"), torch.randperm(cap, generator=g, device="cuda")[:m].int()
    rope = rope_table(400, "cuda")
    xf = x.float().view(m, 8, 128)
    fold = dict(row_stats=torch.stack([xf.sum(-1), xf.pow(2).sum(-1)], -1).contiguous(), col_sums=torch.zeros(4096, device="cuda"), stats_eps=1e-6, stats_rms=True)
    kc, vc, kc2, vc2 = (torch.full((1, 8, cap, 128), 5.0, dtype=torch.bfloat16, device="cuda") for _ in range(4))
    want = ops.gemm(x, w, st, **fold)
    _C.check(_C.lib().ittai_qwen3_qk_rope_scatter(want.data_ptr(), qn.data_ptr(), kn.data_ptr(), rope.data_ptr(), pos.data_ptr(), seq.data_ptr(),
                                                  slot.data_ptr(), kc.data_ptr(), vc.data_ptr(), m, cap, 1e-6, ops._stream(x)))
    got = torch.zeros(m, 4096, dtype=torch.bfloat16, device="cuda")
    ops.gemm(x, w, st, out=got, epi=_C.EPI_QKROPE, qk_rope=dict(qn=qn, kn=kn, rope=rope, pos=pos, seq=seq, slot=slot, kcache=kc2, vcache=vc2, kv_cap=cap, eps=1e-6), **fold)
    ops.check_status(st)
    assert torch.equal(vc, vc2)
    for a, b in ((want[:, :2048], got[:, :2048]), (kc, kc2)):
        d = (a.float() - b.float()).abs()
        assert (d > 0).float().mean() < 1e-3 and d.max() <= 2.0 ** -6 * a.float().abs().max()
    # LayerNorm, residual, statistics
    n, d = 768, 768
    y, wl, res, gain, beta, bias = _rand(m, d, seed=63), _rand(n, d, scale=0.05, seed=64), _rand(m, n, seed=65), torch.rand(d, device="cuda") + 0.5, torch.randn(d, device="cuda") * 0.1, torch.randn(n, device="cuda")
    yf = y.float().view(m, 6, 128)
    wp, bp, cs = ops.fold_layernorm(wl, bias, gain, beta)
    parts = torch.full((m, n // 128, 2), float("nan"), device="cuda")
    out = ops.gemm(y, wp, st, bias=bp, residual=res, row_stats=torch.stack([yf.sum(-1), yf.pow(2).sum(-1)], -1).contiguous(), col_sums=cs, stats_eps=1e-6, stats_out=parts)
    ops.check_status(st)
    lin = torch.nn.functional.linear(torch.nn.functional.layer_norm(y.float(), (d,), gain, beta, 1e-6), wl.float(), bias)
    _check(out, res.float() + lin.to(torch.bfloat16).float(), "LayerNorm + residual", mid=lin)
    of = out.float().view(m, n // 128, 128)
    assert torch.allclose(parts[..., 0], of.sum(-1), rtol=1e-5, atol=1e-3) and torch.allclose(parts[..., 1], of.pow(2).sum(-1), rtol=1e-5, atol=1e-3)


def _qk_runs(m, n_sms):
    """Runs of consecutive QKV tiles (16 column tiles a row block) that the pairs of SMs walk."""
    tiles, pairs = (m + 255) // 256 * 16, min((m + 255) // 256 * 16, n_sms // 2)
    return [range(tiles * p // pairs, tiles * (p + 1) // pairs) for p in range(pairs)]


@gpu
@pytest.mark.parametrize("m", [2304, 16384])
def test_rotary_runs_equal_single_tiles_bit_for_bit(m):
    """A pair's run goes from the last q tile of a row block (column tile 7) to the first k tile (8) and on to the next row block; the
    warps' staging tiles change hands between bulk stores and ordinary ones there.  The same rows in launches that give every pair one
    tile: no order of sums depends on the rows, so q, k and v are the same bits."""
    from ittai_b200 import _C, ops
    from ittai_b200.qwen3.decoder import rope_table
    n_sms = torch.cuda.get_device_properties(0).multi_processor_count
    piece = n_sms // 2 // 16 * 256
    assert all(len(r) == 1 for r in _qk_runs(piece, n_sms))
    assert sum(7 in [t % 16 for t in r[:-1]] for r in _qk_runs(m, n_sms)) >= m // 512, "too few runs cross from q to k"
    g = torch.Generator(device="cuda").manual_seed(m)
    x, w, st = _rand(m, 1024, seed=71), _rand(4096, 1024, scale=0.05, seed=72), ops.new_status("cuda")
    qn, kn = (torch.rand(128, generator=g, device="cuda") + 0.5).to(torch.bfloat16), (torch.rand(128, generator=g, device="cuda") + 0.5).to(torch.bfloat16)
    pos, seq, slot = torch.randint(0, 400, (m,), generator=g, device="cuda", dtype=torch.int32), torch.zeros(m, dtype=torch.int32, device="cuda"), torch.randperm(m, generator=g, device="cuda").int()
    rope = rope_table(400, "cuda")

    def run(step):
        kc, vc = (torch.full((1, 8, m, 128), 5.0, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        out = torch.zeros(m, 4096, dtype=torch.bfloat16, device="cuda")
        for a in range(0, m, step):
            z = slice(a, a + step)
            ops.gemm(x[z], w, st, out=out[z], epi=_C.EPI_QKROPE, qk_rope=dict(qn=qn, kn=kn, rope=rope, pos=pos[z], seq=seq[z], slot=slot[z], kcache=kc, vcache=vc, kv_cap=m, eps=1e-6))
        return out[:, :2048], kc, vc

    want = run(piece)
    for _ in range(4):
        got = run(m)
        for a, b, name in zip(got, want, "qkv"):
            assert torch.equal(a, b), f"{name}: {int((a != b).sum())} values differ"
    ops.check_status(st)


@pytest.mark.parametrize("m", [2304, 16384])
def test_rotary_runs_cross_from_q_to_k(m):
    """The sizes above do what they are there for, and the runs share out every tile once (148 SMs)."""
    runs = _qk_runs(m, 148)
    assert [t for r in runs for t in r] == list(range((m + 255) // 256 * 16))
    assert sum(7 in [t % 16 for t in r[:-1]] for r in runs) >= m // 512


@gpu
@pytest.mark.parametrize("true,padded", [(1152, 1280), (1100, 1280), (64, 256)])
@pytest.mark.parametrize("m", [40, 300, 2600])
def test_zero_padded_columns_are_left_out(m, true, padded):
    """A folded LayerNorm over the true width of a zero-padded A (split-K, and above 128 rows pair tiles): the columns from the true width,
    rounded up to a k-block, on are not read (NaNs in W there do not show), and the bits are those of the GEMM whose K ends there."""
    import ctypes as C
    from ittai_b200 import _C, ops
    n, width = 768, -(-true // 64) * 64
    a = torch.zeros(m, padded, dtype=torch.bfloat16, device="cuda")
    w = torch.zeros(n, padded, dtype=torch.bfloat16, device="cuda")
    a[:, :true], w[:, :true] = _rand(m, true, seed=71), _rand(n, true, scale=0.05, seed=72)
    x = a.float().view(m, padded // 128, 128)
    parts = torch.stack([x.sum(-1), x.pow(2).sum(-1)], -1).contiguous()
    cols, st = w.float().sum(1).contiguous(), ops.new_status("cuda")
    mean = x.sum((1, 2)) / true
    rstd = torch.rsqrt(x.pow(2).sum((1, 2)) / true - mean * mean + 1e-6)
    acc = a.double() @ w.double().t()
    want = (rstd.double()[:, None] * (acc - mean.double()[:, None] * cols.double())).float()
    w[:, width:] = float("nan")
    for static_w in (True,) if m <= 128 else (True, False):
        kw = dict(row_stats=parts, col_sums=cols, stats_eps=1e-6, stats_k=true, static_w=static_w)
        got = ops.gemm(a, w, st, **kw)
        d, narrow = ops.gemm_desc(a, w, st, **kw)
        d.k = width
        _C.check(_C.lib().ittai_gemm_bf16_launch(C.byref(d), ops._stream(a)))
        ops.check_status(st)
        _check(got, want, f"{m}x{true} of {padded}")
        assert torch.equal(got, narrow)


def test_single_launches_of_a_run_are_queued_by_one_call(monkeypatch):
    """Single launches in place of a chain (four GEMMs a layer) go through the binding once, as the chain does."""
    from types import SimpleNamespace
    from ittai_b200 import _C, ops
    calls = []
    count = lambda name: lambda *a: calls.append((name, a)) or 0
    monkeypatch.setattr(_C, "lib", lambda: SimpleNamespace(ittai_gemm_each_launch=count("each"), ittai_gemm_bf16_launch=count("one")))
    monkeypatch.setattr(ops, "_stream", lambda t: None)
    descs = [_C.Gemm() for _ in range(4)]
    for i, d in enumerate(descs):
        d.m = 256 + i
    ops.gemm_each(descs, None)
    assert [name for name, _ in calls] == ["each"] and calls[0][1][1] == 4 and [d.m for d in calls[0][1][0]] == [256, 257, 258, 259]


@gpu
def test_a_run_of_single_launches(monkeypatch):
    """The bits of the calls one by one; a record that is refused ends the run with its message, those before it have run."""
    from ittai_b200 import _C, ops
    a, w, st = _rand(300, 768, seed=81), _rand(768, 768, scale=0.05, seed=82), ops.new_status("cuda")
    want = ops.gemm(ops.gemm(a, w, st), w, st, epi=_C.EPI_GELU)
    d0, x = ops.gemm_desc(a, w, st)
    d1, y = ops.gemm_desc(x, w, st, epi=_C.EPI_GELU)
    ops.gemm_each([d0, d1], a)
    assert torch.equal(y, want)
    x.zero_()
    d1.k = 100
    with pytest.raises(_C.IttaiError, match="multiple"):
        ops.gemm_each([d0, d1], a)
    ops.check_status(st)
    assert torch.equal(x, ops.gemm(a, w, st))
