"""Small embedding forwards, whose norms run inside the split-K GEMMs (GPU)."""
import pytest
import torch
import torch.nn.functional as F

from oracle import qwen3_hf as hf
from oracle import qwen3_ref as ref

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("lens", [[1], [23], [64, 63], [128], [129]])
def test_small_forwards_match_the_oracle(tiny_hf, lens):
    """Both sides of the 128-row limit, first as plain launches and then from a graph, which must agree bit for bit."""
    from ittai_b200.qwen3 import Engine
    model, dims = tiny_hf
    ids = [hf.prompt_ids(n, seed=50 + n, vocab=dims.vocab).tolist() for n in lens]
    eng = Engine(model.state_dict(), 256, 4)
    out = eng.forward(ids).clone()
    for _ in range(2):
        assert torch.equal(eng.forward(ids), out)
    eng.check()
    for i, s in enumerate(ids):
        R = ref.Qwen3Ref(model.state_dict(), dims, 256)
        R.forward(torch.tensor(s))
        assert F.cosine_similarity(out[i].cpu(), R.embed_pool(), dim=0) >= 0.9995, (i, lens)


@gpu
def test_a_failed_wait_of_any_new_shape_is_reported(tiny_hf):
    """A status word planted ahead of a forward: the first forward of every shape reads it, alone and inside ``embed``, and it is
    reported once."""
    from ittai_b200._C import IttaiError
    from ittai_b200.qwen3 import Qwen3Embedder
    model, dims = tiny_hf
    emb = Qwen3Embedder(model, max_tokens=256, max_seqs=4)
    ids = lambda n: list(range(1, n + 1))
    want = emb.embed([ids(7)]).clone()
    for call in (lambda: emb.engine.forward([ids(9)]), lambda: emb.embed([ids(11), ids(3)]), lambda: emb.embed([ids(40)] * 5)):
        emb.engine.core.status[0] = 5
        with pytest.raises(IttaiError, match="GEMM"):
            call()
        assert torch.equal(emb.embed([ids(7)]), want)
        emb.engine.check()


@gpu
def test_more_shapes_than_graphs(tiny_hf):
    """Queries of more lengths than the engine keeps graphs for, in turn: every length is captured at most once, and gives on plain
    launches and from a graph what it gave the first time."""
    from ittai_b200.qwen3 import Engine
    model, dims = tiny_hf
    eng = Engine(model, 128, 4)
    eng._graphs.limit = 3
    ids = lambda n: list(range(1, n + 1))
    want = {n: eng.forward([ids(n)]).clone() for n in range(2, 9)}
    for _ in range(4):
        for n, w in want.items():
            assert torch.equal(eng.forward([ids(n)]), w), n
        assert sorted(eng._graphs.graphs) == [(n, 1, n) for n in (2, 3, 4)]
    eng.check()


@gpu
@pytest.mark.parametrize("lens", [[2], [7], [8], [9], [15, 1], [17], [24], [25], [31], [32], [33], [40], [47], [48], [49], [5, 9, 1, 17], [1] * 32, [16, 1, 31]])
def test_short_forwards_match_the_split_gemms(tiny_hf, lens):
    """Forwards of up to 48 tokens (their own projections, tiles of 8 or of 48 tokens, a token per rank of four or eight) against the kernels of
    longer ones with the same rounding points (``fused_rope=False``): embeddings and the last layer's keys and values.  Bound: a bf16
    rounding is off by 1.1e-3 (rms), a layer has about eight in a row, so that two forwards of two layers whose roundings all fell
    differently would be sqrt(2 * 16) * 1.1e-3 = 6.2e-3 apart; half as much again for few tokens."""
    from ittai_b200.qwen3 import Engine
    model, dims = tiny_hf
    ids = [hf.prompt_ids(n, seed=90 + n + i, vocab=dims.vocab).tolist() for i, n in enumerate(lens)]
    T, outs = sum(lens), []
    for fused in (True, False):
        eng = Engine(model.state_dict(), 128, 32, fused_rope=fused)
        eng.kbuf.fill_(float("nan"))                      # rows behind the last token are not to be read
        eng.vbuf.fill_(float("nan"))
        out = eng.forward(ids).clone()
        eng.check()
        assert torch.equal(eng.forward(ids), out)
        outs.append((out, eng.kbuf[0, :, :T].float(), eng.vbuf[0, :, :T].float()))
        assert eng.kbuf[0, :, T:].isnan().all() and eng.vbuf[0, :, T:].isnan().all()
    for a, b in zip(*outs):
        assert torch.linalg.vector_norm(a - b) <= 9.3e-3 * torch.linalg.vector_norm(b), lens


@gpu
def test_a_short_text_does_not_depend_on_the_others(tiny_hf):
    """Up to 32 tokens: the order of every sum is the same whatever tile a token lies in, so a text's embedding is the same bits alone and
    packed with others (tiles of 8 to 32 tokens; attention of its own rows)."""
    from ittai_b200.qwen3 import Engine
    model, dims = tiny_hf
    eng = Engine(model.state_dict(), 128, 32)
    for lens in ([3, 5], [7, 9, 1], [8, 16], [9, 23], [31, 1], [2, 30], [1] * 32, [16, 15, 1]):
        ids = [hf.prompt_ids(n, seed=40 + n + i, vocab=dims.vocab).tolist() for i, n in enumerate(lens)]
        together = eng.forward(ids).clone()
        for i, text in enumerate(ids):
            assert torch.equal(eng.forward([text])[0], together[i]), (lens, i)
    eng.check()


@gpu
def test_a_short_prompt_behind_a_cached_one(tiny_hf):
    """The attention of few queries, one tile of 32 or two, with cached keys in front of them: a prompt appended in pieces against the prompt
    at once (keys and values of two layers: the bound above)."""
    from ittai_b200.qwen3 import Qwen3Decoder
    model, dims = tiny_hf
    ids = hf.prompt_ids(150, seed=4, vocab=dims.vocab)
    whole, pieces = (Qwen3Decoder(model, max_batch=1, kv_capacity=256) for _ in range(2))
    whole.prefill_cache(ids)
    for a, b in ((0, 64), (64, 97), (97, 98), (98, 128), (128, 150)):
        pieces.prefill_cache(ids[a:b])
    for a, b in ((whole.kcache, pieces.kcache), (whole.vcache, pieces.vcache)):
        a, b = a[..., :150, :].float(), b[..., :150, :].float()
        assert torch.linalg.vector_norm(a - b) <= 9.3e-3 * torch.linalg.vector_norm(b)


@pytest.mark.parametrize("tokens", [1, 32, 48])
def test_short_forwards_refuse_misaligned_rows(tokens):
    """Before anything is launched (CPU): an operand that the kernels read or write 16 bytes at a time lies eight bytes off."""
    import ctypes as C
    from ittai_b200 import _C
    names = ("wqkv", "wo", "wgu", "wd", "ln1", "ln2", "h", "xn", "qkv", "attn", "act")
    others = ("qn", "kn", "embed", "rope", "ids", "pos", "seq", "slot", "seqs", "kcache", "vcache", "stats", "zeros", "status")
    for off in names:
        p = _C.Qwen3Prefill()
        p.n_layers, p.vocab, p.tokens, p.n_seqs, p.max_q_len, p.kv_cap, p.fused_rope, p.split_k = 1, 8, tokens, 1, tokens, 64, 1, 1
        for i, name in enumerate(names + others):
            setattr(p, name, 4096 * (i + 1) + (8 if name == off else 0))
        assert _C.lib().ittai_qwen3_prefill_launch(C.byref(p), None) == -1, off
        with pytest.raises(_C.IttaiError, match="16-byte"):
            _C.check(-1)
