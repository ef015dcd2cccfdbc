"""The split-K GEMM (few output tiles) and its epilogues against fp32 torch references of the same bf16 inputs (GPU).

Tolerance as for the other GEMMs: fp32 accumulation and one bf16 rounding (2^-8 relative), twice where an epilogue rounds
before a non-linearity and a tie falls the other way: |got - want| <= 2^-6 |want| + 2^-7 rms(want) (+ 2^-7 of the rounded
module output ahead of a residual add, which does not shrink when the sum cancels)."""
import pytest
import torch
import torch.nn.functional as F

from test_gemm import _check, _rand

gpu = pytest.mark.gpu
rb = lambda x: x.to(torch.bfloat16).float()


@gpu
@pytest.mark.parametrize("m", [1, 23, 127, 128, 129, 196, 385])
@pytest.mark.parametrize("n,k", [(1024, 64), (1024, 2048), (4096, 1024), (768, 3072), (256, 1088), (2304, 768)])
def test_split_k_plain_and_residual(m, n, k):
    """One k-block up to eight uneven splits, row remainders 1, 127 and 128; the residual is added in place."""
    from ittai_b200 import ops
    a, w, res, bias = _rand(m, k, seed=1), _rand(n, k, scale=0.05, seed=2), _rand(m, n, seed=3), _rand(n, seed=4).float() * 0.1
    st = ops.new_status("cuda")
    acc = a.float() @ w.float().t()
    guard = torch.full((m + 1, n), 7.0, dtype=torch.bfloat16, device="cuda")
    _check(ops.gemm(a, w, st, out=guard[:m], static_w=True), acc, f"{m}x{n}x{k}")
    assert (guard[m] == 7.0).all(), "a row past M was written"
    x = res.clone()
    ops.gemm(a, w, st, bias=bias, residual=x, out=x, static_w=True)
    ops.check_status(st)
    _check(x, res.float() + rb(acc + bias), "bias + residual", mid=acc + bias)


@gpu
@pytest.mark.parametrize("n,k", [(768, 768), (1024, 3072)])
@pytest.mark.parametrize("m", [31, 32, 33, 64, 65, 97, 640, 769])
def test_split_k_row_tiles(m, n, k):
    """Both sides of the lines between tiles of 32, 64 and 128 rows, uneven last tiles; K = 3072 at 640 rows takes 128."""
    from ittai_b200 import ops
    a, w, res = _rand(m, k, seed=41), _rand(n, k, scale=0.05, seed=42), _rand(m, n, seed=43)
    st = ops.new_status("cuda")
    acc = a.float() @ w.float().t()
    guard = torch.full((m + 1, n), 7.0, dtype=torch.bfloat16, device="cuda")
    parts = torch.full((m, n // 128, 2), float("nan"), device="cuda")
    got = ops.gemm(a, w, st, out=guard[:m], residual=res, stats_out=parts, static_w=True)
    ops.check_status(st)
    _check(got, res.float() + rb(acc), f"{m}x{n}x{k}", mid=acc)
    assert (guard[m] == 7.0).all(), "a row past M was written"
    xf = got.float().view(m, n // 128, 128)
    assert torch.allclose(parts[..., 0], xf.sum(-1), rtol=1e-5, atol=1e-3) and torch.allclose(parts[..., 1], xf.pow(2).sum(-1), rtol=1e-5, atol=1e-3)


@gpu
@pytest.mark.parametrize("m", [3, 196])
def test_split_k_activations(m):
    from ittai_b200 import _C, ops
    n, k = 3072, 768
    a, w, bias = _rand(m, k, seed=4), _rand(n, k, scale=0.05, seed=5), _rand(n, seed=7).float() * 0.1
    st = ops.new_status("cuda")
    acc = a.float() @ w.float().t()
    _check(ops.gemm(a, w, st, bias=bias, epi=_C.EPI_GELU, static_w=True), F.gelu(rb(acc + bias), approximate="tanh"), "bias + gelu")
    g, u = rb(acc[:, 0::2]), rb(acc[:, 1::2])
    _check(ops.gemm(a, w, st, epi=_C.EPI_SWIGLU, static_w=True), rb(F.silu(g)) * u, "swiglu")
    ops.check_status(st)


@gpu
@pytest.mark.parametrize("m", [40, 300])
def test_split_k_statistics_and_folded_norms(m):
    """stats_out of one GEMM feeds the folded LayerNorm (and RMSNorm) of the next, also below 128 rows."""
    from ittai_b200 import ops
    d, n = 768, 2304
    a0, w0, r0 = _rand(m, d, seed=21), _rand(d, d, scale=0.05, seed=22), (_rand(m, d, seed=23).float() * 2 + 1).to(torch.bfloat16)
    st = ops.new_status("cuda")
    parts = torch.full((m, d // 128, 2), float("nan"), device="cuda")
    x = ops.gemm(a0, w0, st, residual=r0, stats_out=parts, static_w=True)
    xf = x.float().view(m, d // 128, 128)
    assert torch.allclose(parts[..., 0], xf.sum(-1), rtol=1e-5, atol=1e-3)
    assert torch.allclose(parts[..., 1], xf.pow(2).sum(-1), rtol=1e-5, atol=1e-3)
    w, bias = _rand(n, d, scale=0.05, seed=24), torch.randn(n, device="cuda")
    gain, beta = torch.rand(d, device="cuda") + 0.5, torch.randn(d, device="cuda") * 0.1
    wp, bp, cs = ops.fold_layernorm(w, bias, gain, beta)
    got = ops.gemm(x, wp, st, bias=bp, row_stats=parts, col_sums=cs, stats_eps=1e-6, static_w=True)
    _check(got, F.linear(F.layer_norm(x.float(), (d,), gain, beta, 1e-6), w.float(), bias), "folded LayerNorm")
    got = ops.gemm(x, wp, st, bias=bp, row_stats=ops.row_stats(x, 1e-6), col_sums=cs, static_w=True)
    _check(got, F.linear(F.layer_norm(x.float(), (d,), gain, beta, 1e-6), w.float(), bias), "folded LayerNorm, finished statistics")
    wr = (w.float() * gain).to(torch.bfloat16)
    got = ops.gemm(x, wr, st, row_stats=parts, col_sums=torch.zeros(n, device="cuda"), stats_eps=1e-6, stats_rms=True, static_w=True)
    xn = x.float() * torch.rsqrt(x.float().pow(2).mean(-1, keepdim=True) + 1e-6)
    _check(got, F.linear(xn, wr.float()), "folded RMSNorm")
    ops.check_status(st)


@gpu
@pytest.mark.parametrize("T", [1, 37, 128, 200])
def test_split_k_rope_epilogue_matches_the_separate_pass(T):
    """QK-norm + RoPE + cache scatter in the epilogue against GEMM + row-wise pass: the same rounding steps on sums taken in
    another order, so values may differ by a bf16 step or two (2^-7 relative, and 2^-6 of the largest through the rotation)."""
    from ittai_b200 import _C, ops
    from ittai_b200.qwen3.decoder import rope_table
    cap, B = 256, 2
    x, w = _rand(T, 1024, seed=31), _rand(4096, 1024, scale=0.05, seed=32)
    qn, kn = (_rand(128, seed=33).float() * 0.2 + 1).to(torch.bfloat16), (_rand(128, seed=34).float() * 0.2 + 1).to(torch.bfloat16)
    rope = rope_table(cap, "cuda")
    seq = (torch.arange(T, device="cuda") % 2).int()
    slot = (torch.arange(T, device="cuda") // 2 + 5).int()
    pos = (slot * 2 % cap).int()
    st = ops.new_status("cuda")

    def run(fused):
        kc, vc = (torch.full((B, 8, cap, 128), 3.0, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        qkv = torch.zeros(T, 4096, dtype=torch.bfloat16, device="cuda")
        if fused:
            ops.gemm(x, w, st, out=qkv, epi=_C.EPI_QKROPE, static_w=True,
                     qk_rope=dict(qn=qn, kn=kn, rope=rope, pos=pos, seq=seq, slot=slot, kcache=kc, vcache=vc, kv_cap=cap, eps=1e-6))
        else:
            ops.gemm(x, w, st, out=qkv, static_w=True)
            _C.check(_C.lib().ittai_qwen3_qk_rope_scatter(qkv.data_ptr(), qn.data_ptr(), kn.data_ptr(), rope.data_ptr(), pos.data_ptr(),
                                                          seq.data_ptr(), slot.data_ptr(), kc.data_ptr(), vc.data_ptr(), T, cap, 1e-6, ops._stream(x)))
        ops.check_status(st)
        return qkv[:, :2048], kc, vc

    for got, want, name in zip(run(True), run(False), ("q", "k", "v")):
        assert ((got.float() - want.float()).abs() <= 2.0 ** -7 * want.float().abs() + 2.0 ** -6 * want.float().abs().max() / 8).all(), name
        assert torch.equal(got == 3.0, want == 3.0) or name == "q", f"{name}: other cache rows written"


def _early(stages, groups, n_kb=48):
    """k-blocks whose wait a group may leave a phase early: use u of a stage is waited for by the parity of u, which the end of use
    u - 2 satisfies as well, unless the group has seen use u - 1 end."""
    bad = []
    for g in range(groups):
        seen = {}
        for kb in range(g, n_kb, groups):
            s, u = kb % stages, kb // stages
            if u > seen.get(s, -1) + 1:
                bad.append(kb)
            seen[s] = u
    return bad


def test_normalising_groups_wait_for_every_use_of_a_stage():
    """As many groups as stages; six on four stages or two on three would be let through early."""
    assert not _early(4, 4) and not _early(3, 3)
    assert {4, 5, 6} <= set(_early(4, 6)) and 3 in _early(3, 2)


@gpu
@pytest.mark.parametrize("m,n,k", [(7, 256, 64), (32, 256, 2560), (23, 256, 4096), (32, 256, 8192), (31, 4096, 2048), (64, 4096, 1024), (40, 4096, 2048), (100, 4096, 3072),
                                   (640, 1024, 3072), (768, 1024, 6144)])
def test_normalisation_inside_the_gemm(m, n, k):
    """One to 24 k-blocks a CTA, up to eight uses of a stage, tiles of 32, 64 and 128 rows, against the same GEMM on rows normalised
    beforehand with the same roundings (the reciprocal root may differ by an ulp and tip one).  The gains tell the k-blocks apart."""
    import ctypes as C
    from ittai_b200 import _C, ops
    launch = getattr(_C.lib(), "_ZN5ittai18gemm_normed_launchEPK9IttaiGemmPKvP11CUstream_st")       # used by the prefill, not exported
    launch.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p]
    x, w, st = (_rand(m, k, seed=61).float() * 3).to(torch.bfloat16), _rand(n, k, scale=0.05, seed=62), ops.new_status("cuda")
    gain = ((torch.arange(k, device="cuda") // 64 % 7 + 1) * 0.25).to(torch.bfloat16)
    xf = x.float().view(m, -1, 64 if k < 128 else 128)
    parts = torch.stack([xf.sum(-1), xf.pow(2).sum(-1)], -1).contiguous()
    normed = rb(rb(x.float() * torch.rsqrt(xf.pow(2).sum((1, 2)) / k + 1e-6)[:, None]) * gain.float()).to(torch.bfloat16)
    want = ops.gemm(normed, w, st, static_w=True)
    g, out = ops.gemm_desc(x, w, st, static_w=True)
    zeros = torch.zeros(n, device="cuda")
    g.row_stats, g.col_sums, g.stats_parts, g.stats_eps, g.stats_rms = parts.data_ptr(), zeros.data_ptr(), parts.shape[1], 1e-6, 1
    for _ in range(3):
        out.zero_()
        _C.check(launch(C.addressof(g), gain.data_ptr(), ops._stream(x)))
        ops.check_status(st)
        _check(out, want, f"{m}x{n}x{k}")
    _check(out, normed.float() @ w.float().t(), f"{m}x{n}x{k} against fp32")


def test_limits_without_the_flag():
    """What needs more than 128 rows (or constant weights) is refused without the flag, and the flag is no epilogue of a chain."""
    import ctypes as C
    from ittai_b200 import _C
    g = _C.Gemm()
    g.m, g.n, g.k, g.epi = 64, 1024, 1024, _C.EPI_NONE
    g.a = g.w = g.out = g.status = g.stats_out = 4096
    assert _C.lib().ittai_gemm_bf16_launch(C.byref(g), None) == -1 and b"stats_out needs" in _C.lib().ittai_last_error()
    g.m, g.stats_out, g.epi = 512, None, _C.GEMM_STATIC_W
    assert _C.lib().ittai_gemm_chain_launch(C.byref(g), 1, 4096, None) == -1 and b"plain and GELU" in _C.lib().ittai_last_error()
    g.epi = _C.GEMM_STATIC_W | 9
    assert _C.lib().ittai_gemm_bf16_launch(C.byref(g), None) == -1 and b"unknown epilogue" in _C.lib().ittai_last_error()
