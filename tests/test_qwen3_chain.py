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
