"""The decode chain (``csrc/qwen3_chain.cu``) against the CPU restatement at the cache lengths where its attention changes
shape: tile of 32 positions, ring of six tiles, a warp's 16 positions, and both sides of every line of the split rule (GPU).

Tolerance: that of the teacher-forced decode tests, max-abs 3e-2 and cosine 0.9995 on the logits; an appended key passes
five bf16 roundings in a row (projection, two of the norm, product and sum of the rotation), each of which may fall the other
way by one ulp, at most 2^-7 of the row's largest value."""
import pytest
import torch
import torch.nn.functional as F

from oracle import qwen3_ref as ref

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("batch,length", [(1, 0), (1, 1), (1, 31), (1, 48), (1, 49), (1, 1200), (1, 1201), (2, 17), (2, 400), (2, 401),
                                          (4, 64), (4, 1000), (8, 700), (8, 701), (8, 1219)])
def test_step_at_length(tiny_hf, batch, length):
    from ittai_b200.qwen3 import Qwen3Decoder
    model, dims = tiny_hf
    cap = 1220
    g = torch.Generator().manual_seed(length + batch)
    d = Qwen3Decoder(model, max_batch=batch, kv_capacity=cap)
    nan = torch.tensor(float("nan"), dtype=torch.bfloat16)
    kv = [(torch.randn(dims.n_layers, batch, dims.n_kv_heads, cap, dims.head_dim, generator=g) * s).to(torch.bfloat16) for s in (1.0, 0.5)]
    for c, t in zip((d.kcache, d.vcache), kv):
        t[:, :, :, length:] = nan                       # rows that were never written must not be read into the result
        c.copy_(t)
    ids = torch.randint(0, dims.vocab, (batch,), generator=g, dtype=torch.int32)
    d.rewind(length)
    d.next_id.copy_(ids)
    got = d.decode(1)[:, 0].tolist()
    assert d.pos.tolist() == [length + 1] * batch
    for b in sorted({0, batch - 1}):
        R = ref.Qwen3Ref(model.state_dict(), dims, cap)
        R.k, R.v, R.len = kv[0][:, b].float(), kv[1][:, b].float(), length
        want = R.forward(ids[b:b + 1].long())
        logits = d.logits[b].float().cpu()
        assert (logits - want).abs().max() <= 3e-2 and F.cosine_similarity(logits, want, dim=0) >= 0.9995, (batch, length, b)
        top = want.topk(2).values
        assert got[b] == int(want.argmax()) or top[0] - top[1] <= 0.0625
        for c, w in ((d.kcache, R.k), (d.vcache, R.v)):
            row, wrow = c[:, b, :, length].float().cpu(), w[:, :, length]
            assert (row - wrow).abs().max() <= 5 * 2.0 ** -7 * wrow.abs().max()
            assert torch.isnan(c[:, b, :, length + 1:]).all(), "a row beyond the new position was written"


@gpu
@pytest.mark.parametrize("batch,length", [(1, 400), (1, 401), (1, 700), (2, 48), (2, 49), (2, 111), (2, 1000)])
def test_step_at_pieces_that_are_no_power_of_two(tiny_hf, batch, length):
    """Caches cut in 12 and in 7, of which 8 and 4 merge: both sides of the lines, last pieces that are short or empty."""
    test_step_at_length(tiny_hf, batch, length)


@gpu
def test_a_captured_stream_gets_the_kernels(tiny_hf):
    """Inside a stream capture the chain enqueues its kernels instead of launching graphs of its own."""
    from ittai_b200.qwen3 import Qwen3Decoder
    model, dims = tiny_hf
    d = Qwen3Decoder(model, max_batch=1, kv_capacity=64)
    d.next_id.fill_(7)
    want = d.decode(3).cpu()
    d.reset()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = d.decode(3, check=False)
    d.reset()
    d.next_id.fill_(7)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out.cpu(), want) and d.pos.tolist() == [3]


def _chain_buffer(d, name):
    """bf16 ``[B, width]`` of the chain's scratch: a 256-byte state record, then these vectors, each from a 256-byte line on."""
    off = d._ws_ptr - d.workspace.data_ptr() + 256
    for nm, width in (("h", 1024), ("hmid", 1024), ("qkv", 4096), ("attn", 2048), ("act", 3072)):
        if nm == name:
            return d.workspace[off:off + d.B * width * 2].view(torch.bfloat16).view(d.B, width).clone()
        off += (d.B * width * 2 + 255) // 256 * 256


@gpu
@pytest.mark.parametrize("batch,length", [(1, 500), (2, 300), (8, 500)])
def test_attention_keeps_fp32_probabilities(tiny_hf, batch, length):
    """The last layer's attention output against 64-bit arithmetic on the same projections and cache: nearly every value is the
    exact one rounded once.  The share that is not is twice the error over the spacing of bf16.  Sums of fp32 products, a few 2^-24
    of values some ten times the result, leave 2e-4 (measured 0.6-3.6e-4 over all batches and lengths, the persistent kernel the
    same); probabilities of 16 bits left 1.5-3.3e-3.  A head whose query rounds the other way somewhere is not counted."""
    from ittai_b200.qwen3 import Qwen3Decoder
    model, dims = tiny_hf
    d = Qwen3Decoder(model, max_batch=batch, kv_capacity=512)
    g = torch.Generator(device="cuda").manual_seed(batch)
    d.kcache.normal_(0.0, 1.0, generator=g)
    d.vcache.normal_(0.0, 0.64, generator=g)
    f8, r = torch.float64, lambda x: x.to(torch.bfloat16).to(torch.float64)
    qn = d.w["qn"][-1].to(f8)
    cos, sin = d.rope[length, :64].to(f8), d.rope[length, 64:].to(f8)
    off = total = 0
    for _ in range(64 // batch):
        d.rewind(length)
        d.next_id.copy_(torch.randint(0, dims.vocab, (batch,), generator=g, device="cuda", dtype=torch.int32))
        d.decode(1)
        q = _chain_buffer(d, "qkv")[:, :2048].to(f8).view(batch, 16, 128)
        q = r(r(q / (q.pow(2).mean(-1, keepdim=True) + 1e-6).sqrt()) * qn)
        a, b = q[..., :64], q[..., 64:]
        q = torch.cat([r(r(a * cos) - r(b * sin)), r(r(b * cos) + r(a * sin))], -1)
        k, v = (c[-1, :, :, :length + 1].to(f8).repeat_interleave(2, 1) for c in (d.kcache, d.vcache))
        p = torch.softmax((k @ q[..., None])[..., 0] * 128 ** -0.5, -1)
        want = r((p[:, :, None] @ v)[:, :, 0])
        wrong = (_chain_buffer(d, "attn").to(f8).view(batch, 16, 128) != want).sum(-1)
        wrong = wrong[wrong <= 4]
        off, total = off + int(wrong.sum()), total + 128 * wrong.numel()
    assert total >= 0.9 * 64 * 2048 and off <= 8e-4 * total, off / total


@gpu
@pytest.mark.parametrize("batch,length", [(1, 5000), (2, 2500), (4, 1250), (8, 625)])
def test_tiles_held_by_gate_up_change_no_bit(tiny_hf, batch, length):
    """The last length at which gate/up holds two of its three tiles in registers: ids, logits and cache rows of the step are the same,
    bit for bit, where the bound on the positions that the caller gives (here one more) selects the kernel that holds none."""
    import ctypes as C
    from ittai_b200 import _C
    from ittai_b200.qwen3 import Qwen3Decoder
    model, dims = tiny_hf
    d = Qwen3Decoder(model, max_batch=batch, kv_capacity=length + 8)
    g = torch.Generator(device="cuda").manual_seed(3)
    d.kcache.normal_(0.0, 1.0, generator=g)
    d.vcache.normal_(0.0, 0.64, generator=g)
    got = []
    for bound in (length, length + 1):
        d.rewind(length)
        d.next_id.copy_(torch.arange(batch, dtype=torch.int32) + 5)
        d.logits.zero_()
        out = torch.full((1, batch), -7, dtype=torch.int32, device="cuda")
        p = d._params(1, 0, None, out, None)
        _C.check(d.lib.ittai_qwen3_chain_run(d._plan, C.byref(p), bound, d._stream()))
        d.check_status()
        got.append((out, d.logits.clone(), d.kcache[:, :, :, length].clone(), d.vcache[:, :, :, length].clone()))
    assert (got[0][0] >= 0).all() and got[0][1].abs().max() > 0 and all(torch.equal(a, b) for a, b in zip(*got))


@gpu
@pytest.mark.parametrize("length", [6000, 6001])
def test_step_at_clusters_of_eight_for_two_sequences(tiny_hf, length):
    """Caches of two sequences cut in 7 up to 6000 positions and in 8 beyond: against the CPU restatement, and the first sequence's bits
    beside a neighbour on either side of the line."""
    from ittai_b200.qwen3 import Qwen3Decoder
    model, dims = tiny_hf
    cap = 6100
    g = torch.Generator().manual_seed(length)
    d = Qwen3Decoder(model, max_batch=2, kv_capacity=cap)
    kv = [(torch.randn(dims.n_layers, 2, dims.n_kv_heads, cap, dims.head_dim, generator=g) * s).to(torch.bfloat16) for s in (1.0, 0.5)]
    ids = torch.randint(0, dims.vocab, (2,), generator=g, dtype=torch.int32)
    R = ref.Qwen3Ref(model.state_dict(), dims, cap)
    R.k, R.v, R.len = kv[0][:, 0].float(), kv[1][:, 0].float(), length
    want, first = R.forward(ids[:1].long()), None
    for other in (40, 5999, 6050):
        for c, t in zip((d.kcache, d.vcache), kv):
            c.copy_(t)
        d.set_length(0, length)
        d.set_length(1, other)
        d.next_id.copy_(ids)
        got = d.decode(1)[0].item()
        now = (got, d.logits[0].clone(), *(c[:, 0, :, length].clone() for c in (d.kcache, d.vcache)))
        first = first or now
        assert now[0] == first[0] and all(torch.equal(a, b) for a, b in zip(now[1:], first[1:])), other
    logits = first[1].float().cpu()
    assert (logits - want).abs().max() <= 3e-2 and F.cosine_similarity(logits, want, dim=0) >= 0.9995
