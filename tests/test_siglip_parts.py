"""Short batches and the position-row kernel of the vision engines (GPU)."""
import pytest
import torch

from oracle import siglip_hf as hf

gpu = pytest.mark.gpu
SHAPES = [(16, 16), (12, 20), (1, 1), (10, 25), (1, 256), (200, 1), (3, 5), (27, 9)]


@gpu
@pytest.mark.parametrize("side,width,ld", [(16, 768, 768), (27, 1152, 1280)])
def test_position_rows_match_the_torch_resize(side, width, ld):
    """Grids smaller and larger than the learned one, one row, one column, one patch.  Both sides sum at most some 60 products
    of a weight and an fp32 value: one bf16 rounding (2^-8 relative) and 1e-5 of the largest value for the sums."""
    from ittai_b200 import _C, ops
    from ittai_b200.siglip.kernel import resize_positions
    g = torch.Generator(device="cuda").manual_seed(side)
    grid = torch.randn(side, side, width, generator=g, device="cuda")
    n, rows = len(SHAPES), 256
    out = torch.full((n * rows + 1, ld), 9.0, dtype=torch.bfloat16, device="cuda")
    seqs, pool = (torch.full((n, 4), -1, dtype=torch.int32, device="cuda") for _ in range(2))
    shapes = torch.tensor(SHAPES, dtype=torch.int32, device="cuda")
    _C.check(_C.lib().ittai_siglip_positions(grid.data_ptr(), side, width, shapes.data_ptr(), n, rows, out.data_ptr(), ld, seqs.data_ptr(), pool.data_ptr(),
                                             ops._stream(out)))
    want = resize_positions(grid, SHAPES, rows).reshape(n * rows, width)
    got = out[:-1, :width].float()
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5 * want.abs().max()).all(), (got - want).abs().max()
    assert (out[-1] == 9.0).all() and (ld == width or (out[:, width:] == 9.0).all())
    area = torch.tensor([h * w for h, w in SHAPES], dtype=torch.int32, device="cuda")
    for t in (seqs, pool):
        assert torch.equal(t[:, 3], area) and (t[:, :3] == -1).all()


@gpu
@pytest.mark.parametrize("batch,images", [(8, 11), (8, 7), (2, 3), (16, 16)])
def test_a_short_batch_gives_what_the_full_batch_gives(batch, images):
    """The images behind the last whole batch run as a smaller forward: the same rows, bit for bit, as in a full batch, on the
    first pass (plain launches) and on repeated ones (a graph)."""
    from ittai_b200.siglip.kernel import Siglip2Embedder
    emb = Siglip2Embedder(hf.build_hf(seed=0, device="cuda"), batch_size=batch)
    g = torch.Generator().manual_seed(5)
    px = torch.randn(images, 3, 224, 224, generator=g)
    padded = torch.cat([px, px[-1:].expand(-images % batch, -1, -1, -1)])
    want = torch.cat(emb.embed_batches([padded[k:k + batch] for k in range(0, len(padded), batch)]))[:images]
    for _ in range(3):
        got = emb.embed(px)
        assert got.shape == want.shape
        cos = torch.nn.functional.cosine_similarity(got.float(), want.float(), dim=-1).min()
        assert torch.equal(got, want) if batch >= 6 else cos >= 0.9999, cos
    emb.engine.check()


@gpu
def test_a_short_naflex_batch():
    from ittai_b200.siglip.kernel import Siglip2Embedder
    shapes = [(16, 16), (9, 21), (3, 5), (12, 20), (1, 1), (10, 25), (16, 15)]
    emb = Siglip2Embedder(hf.build_hf_naflex(seed=2, device="cuda"), batch_size=5)
    inp = hf.naflex_inputs(shapes, seed=8)
    full = {k: torch.cat([v, v[:3]]) for k, v in inp.items()}
    want = emb.embed(full)[:7]
    for _ in range(2):
        assert torch.equal(emb.embed(inp), want)
    bad = dict(inp, spatial_shapes=torch.tensor([(17, 16)] + shapes[1:]))
    with pytest.raises(ValueError):
        emb.embed(bad)


@gpu
@pytest.mark.parametrize("lens", [[729, 729], [128, 65, 1, 200], [257]])
def test_packed_attention_with_80_columns_per_head(lens):
    """The key-loop kernel on heads 80 columns apart against fp32 softmax attention: P and the output are rounded to bf16 once
    each (2^-8 relative on P's unit row sums, 2^-9 on the result), with the scores exact to fp32: 2^-7 of the largest value."""
    from ittai_b200 import ops
    H, hd = 5, 80
    total = sum(lens)
    g = torch.Generator(device="cuda").manual_seed(total)
    qkv = torch.randn(total, 3 * H * hd, generator=g, device="cuda").to(torch.bfloat16)
    out = torch.full((total + 1, H * hd), 9.0, dtype=torch.bfloat16, device="cuda")
    first = [sum(lens[:i]) for i in range(len(lens))]
    seqs = torch.tensor([[f, n, f, n] for f, n in zip(first, lens)], dtype=torch.int32, device="cuda")
    st = ops.new_status("cuda")
    kw = dict(n_heads=H, group=1, head_dim=hd, causal=False, q_strides=(3 * H * hd, hd), k_strides=(3 * H * hd, hd, 0),
              v_strides=(3 * H * hd, hd, 0), o_strides=(H * hd, hd), q_rows_total=total, kv_rows_total=total, status=st)
    ops.attention(qkv, qkv[:, H * hd:], qkv[:, 2 * H * hd:], out, seqs, max_q_len=max(lens), **kw)
    ops.check_status(st)
    for f, n in zip(first, lens):
        q, k, v = (qkv[f:f + n, i * H * hd:(i + 1) * H * hd].float().view(n, H, hd).transpose(0, 1) for i in range(3))
        want = torch.softmax(q @ k.transpose(1, 2) / hd ** 0.5, -1) @ v
        got = out[f:f + n].float().view(n, H, hd).transpose(0, 1)
        assert (got - want).abs().max() <= 2.0 ** -7 * want.abs().max()
    assert (out[-1] == 9.0).all()
    from ittai_b200 import _C
    with pytest.raises(_C.IttaiError, match="head_dim 80"):
        ops.attention(qkv, qkv[:, H * hd:], qkv[:, 2 * H * hd:], out, seqs, max_q_len=64, **kw)


@gpu
@pytest.mark.parametrize("batch", [1, 3])
def test_key_counts_of_the_batch_before_are_not_seen(batch):
    """A padded variable-resolution tower on plain launches, the host far ahead: the key counts that the position kernel writes
    alternate from batch to batch, and the attention kernel, which may start before that kernel has ended, must see its own
    batch's.  Every batch gives, bit for bit, what it gives alone on an idle device."""
    from ittai_b200.siglip.kernel import Engine
    eng = Engine(hf.build_hf_so400m(True, n_layers=2, device="cuda"), batch, graph=False)
    assert eng.hde == 80 and not eng.chain
    inputs = []
    for i, shapes in enumerate([[(16, 16), (12, 20), (9, 21)], [(1, 1), (3, 5), (2, 2)], [(10, 25), (1, 200), (16, 9)]]):
        inp = hf.naflex_inputs(shapes[:batch], seed=20 + i)
        inputs.append(dict(inp, pixel_values=inp["pixel_values"].cuda()))
    want = []
    for inp in inputs:
        want.append(eng.forward(inp).clone())
        torch.cuda.synchronize()
    got = [eng.forward(inputs[i % 3]).clone() for i in range(48)]
    eng.check()
    for i, t in enumerate(got):
        assert torch.equal(t, want[i % 3]), i


@gpu
def test_a_failed_wait_of_any_new_size_is_reported():
    """A status word planted ahead of a forward: the first forward of every batch size reads it, and it is reported once."""
    from ittai_b200._C import IttaiError
    from ittai_b200.siglip.kernel import Siglip2Embedder
    emb = Siglip2Embedder(hf.build_hf(seed=0, device="cuda", n_layers=1), batch_size=4)
    px = hf.pixels(4, seed=3)
    want = emb.embed(px)
    for call in (lambda: emb.embed(px[:3]), lambda: emb.engine.forward_part({"pixel_values": px[:1]}), lambda: emb.embed(torch.cat([px, px[:2]]))):
        emb.engine.status[0] = 5
        with pytest.raises(IttaiError, match="GEMM"):
            call()
        assert torch.equal(emb.embed(px), want)
        emb.engine.check()


@gpu
def test_more_batch_sizes_than_graphs():
    """Short batches of more sizes than the engine keeps graphs for, in turn, with the full batch among them: each size is captured
    at most once, and every size gives what it gave the first time."""
    from ittai_b200.siglip.kernel import Siglip2Embedder
    emb = Siglip2Embedder(hf.build_hf(seed=0, device="cuda", n_layers=1), batch_size=5)
    eng = emb.engine
    eng._graphs.limit = 2
    px = hf.pixels(5, seed=3).cuda()
    want = {n: emb.embed(px[:n]) for n in (1, 2, 3, 4, 5)}
    for _ in range(4):
        for n, w in want.items():
            assert torch.equal(emb.embed(px[:n]), w), n
        assert sorted(eng._graphs.graphs) == [1, 2] and list(eng._full.graphs) == [5]
    eng.check()


@gpu
@pytest.mark.parametrize("slot", [0, 1])
def test_a_new_staging_buffer_waits_for_the_block_s_last_user(slot):
    """A batch larger than the ones before gets a new staging buffer.  The allocator may hand out a block that the caller has just
    freed and that queued work still reads: the copy on the side stream must not overtake that work."""
    from ittai_b200.siglip.kernel import Siglip2Embedder
    emb = Siglip2Embedder(hf.build_hf(seed=0, device="cuda", n_layers=1), batch_size=16)
    px = hf.pixels(32, seed=3).pin_memory()
    want = emb.embed(px.cuda())
    emb.embed(px[:1])                                      # a buffer of one image in the first slot
    if slot == 1:
        emb.embed(px[:16])                                 # the first slot has its full size, the second none
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    mine = torch.arange(16 * 3 * 224 * 224, dtype=torch.float32, device="cuda")
    torch.cuda._sleep(40_000_000)                          # some 20 ms
    seen = mine * 1.0
    ptr = mine.data_ptr()
    del mine
    got = emb.embed(px)
    assert any(b.data_ptr() == ptr for b in emb._staged), "the block was not reused: the test does not test"
    assert torch.equal(seen, torch.arange(seen.numel(), dtype=torch.float32, device="cuda")) and torch.equal(got, want)


@gpu
@pytest.mark.parametrize("kind,batch", [("vit", 6), ("vit", 25), ("naflex", 5), ("so400m", 2), ("so400m", 5)])
def test_chained_and_single_launches_give_the_same_bits(monkeypatch, kind, batch):
    """Which of the two a forward takes follows from its rows; with the choice forced either way, on plain launches and from a graph."""
    from ittai_b200.siglip import kernel
    build = {"vit": hf.build_hf, "naflex": hf.build_hf_naflex, "so400m": hf.build_hf_so400m}[kind]
    vm = build(n_layers=2, device="cuda")
    if kind == "naflex":
        inp = hf.naflex_inputs(SHAPES[:batch], seed=31)
    else:
        side = 224 if kind == "vit" else 384
        inp = {"pixel_values": torch.randn(batch, 3, side, side, generator=torch.Generator().manual_seed(31))}
    got, chains = {}, []
    real = kernel.ops.gemm_chain
    monkeypatch.setattr(kernel.ops, "gemm_chain", lambda *a: chains.append(1) or real(*a))
    for chained in (True, False):
        monkeypatch.setattr(kernel, "chain_pays", lambda *a: chained)
        eng = kernel.Engine(vm, batch)
        assert eng.chain
        before = len(chains)
        got[chained] = [eng.forward(inp).clone() for _ in range(3)]
        eng.check()
        assert (len(chains) > before) == chained
        assert all(torch.equal(g, got[chained][0]) for g in got[chained])
    assert torch.equal(got[True][0], got[False][0])
