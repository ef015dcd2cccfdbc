"""Properties of a call of the decode chain (``csrc/qwen3_chain.cu``): what a sequence sees of its neighbours, what is left behind by
a call that fails, calls on several streams (GPU)."""
import pytest
import torch

from oracle import qwen3_hf as hf

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("batch", [2, 4, 8])
@pytest.mark.parametrize("length", [0, 20, 47, 399, 450, 699])
def test_a_sequence_does_not_depend_on_its_neighbours(tiny_hf, batch, length):
    """Ids, logits and cache rows of a sequence are the same, bit for bit, whatever lengths the others have, on both sides of
    every line of the split rule; the four steps cross the lines."""
    from ittai_b200.qwen3 import Qwen3Decoder
    model, dims = tiny_hf
    g = torch.Generator().manual_seed(batch + length)
    d = Qwen3Decoder(model, max_batch=batch, kv_capacity=1200)
    kv = [(torch.randn(d.kcache.shape, generator=g) * s).to(torch.bfloat16) for s in (1.0, 0.5)]
    ids = torch.randint(0, dims.vocab, (batch,), generator=g, dtype=torch.int32)

    def run(other):
        for c, t in zip((d.kcache, d.vcache), kv):
            c.copy_(t)
        d.reset()
        for b in range(batch):
            d.set_length(b, length if b == 0 else other)
        d.next_id.copy_(ids)
        out = d.decode(4)[0].clone()
        return out, d.logits[0].clone(), *(c[:, 0, :, length:length + 4].clone() for c in (d.kcache, d.vcache))

    want = run(1)
    for other in (46, 399, 699, 1100):
        for got, ref in zip(run(other), want):
            assert torch.equal(got, ref), (other, (got.float() - ref.float()).abs().max())


@gpu
@pytest.mark.parametrize("slots", [2, 8])
def test_served_tokens_do_not_depend_on_the_other_requests(tiny_hf, slots):
    """Short requests beside ones past 400 and 700 positions give the tokens of their solo runs."""
    from ittai_b200.qwen3 import DecodeServer, Qwen3Decoder
    model, dims = tiny_hf
    d = Qwen3Decoder(model, max_batch=slots, kv_capacity=1024)
    prompts = [hf.prompt_ids(n, seed=170 + i, vocab=dims.vocab).tolist() for i, n in enumerate((20, 720, 45, 410, 33, 90, 12, 500))]
    budgets = [24, 9, 20, 12, 17, 8, 30, 6]
    srv = DecodeServer(d, chunk=4)
    rids = [srv.submit(p, m) for p, m in zip(prompts, budgets)]
    out = dict(srv.run())
    for rid, p, m in zip(rids, prompts, budgets):
        solo = DecodeServer(d, chunk=4)
        r = solo.submit(p, m)
        assert solo.run()[r] == out[rid], f"request {rid} (prompt {len(p)}, {m} tokens) depends on its neighbours"


@gpu
@pytest.mark.parametrize("batch", [1, 8])
def test_a_wait_that_runs_out_ends_the_call(tiny_hf, batch):
    """CTA 0 of every projection leaves its weights out and gives up after a shortened wait: the call reports it, stores no id,
    and leaves positions and the next input where they were; the next call goes on from there."""
    import ctypes as C
    from ittai_b200 import _C
    from ittai_b200.qwen3 import Qwen3Decoder
    model, dims = tiny_hf
    d = Qwen3Decoder(model, max_batch=batch, kv_capacity=64)
    d.next_id.fill_(7)
    want = d.decode(6).cpu()
    d.reset()
    d.next_id.fill_(7)
    assert torch.equal(d.decode(2).cpu(), want[:, :2])
    out = torch.full((3, batch), -7, dtype=torch.int32, device="cuda")
    p = d._params(3, 0, None, out, None)
    p.flags, p.spin_limit = _C.F_TEST_DROP_CTA, 64
    _C.check(d.lib.ittai_qwen3_chain_run(d._plan, C.byref(p), 2, d._stream()))
    with pytest.raises(_C.IttaiError, match="stream"):
        d.check_status()
    assert (out == -7).all() and d.pos.tolist() == d.lengths == [2] * batch
    assert torch.equal(d.decode(4).cpu(), want[:, 2:])


@gpu
@pytest.mark.parametrize("batch,length", [(1, 60), (1, 500), (2, 60), (4, 30)])
def test_a_wait_that_runs_out_beside_clusters(tiny_hf, batch, length):
    """The same where the attention runs in clusters (of 8, 12, 7 and 4): the call ends with a report, the next one goes on."""
    import ctypes as C
    from ittai_b200 import _C
    from ittai_b200.qwen3 import Qwen3Decoder
    model, dims = tiny_hf
    d = Qwen3Decoder(model, max_batch=batch, kv_capacity=600)
    g = torch.Generator(device="cuda").manual_seed(length)
    d.kcache.normal_(0.0, 1.0, generator=g)
    d.vcache.normal_(0.0, 0.5, generator=g)
    d.rewind(length)
    d.next_id.fill_(7)
    want = d.decode(3).cpu()
    d.rewind(length)
    d.next_id.fill_(7)
    out = torch.full((2, batch), -7, dtype=torch.int32, device="cuda")
    p = d._params(2, 0, None, out, None)
    p.flags, p.spin_limit = _C.F_TEST_DROP_CTA, 64
    _C.check(d.lib.ittai_qwen3_chain_run(d._plan, C.byref(p), length, d._stream()))
    with pytest.raises(_C.IttaiError, match="stream"):
        d.check_status()
    assert (out == -7).all() and d.pos.tolist() == d.lengths == [length] * batch
    assert torch.equal(d.decode(3).cpu(), want)


@gpu
def test_a_reported_failure_is_not_reported_again(tiny_hf):
    """After a failed decode, prefills that go well are accepted; so is what follows a second failure."""
    from ittai_b200._C import IttaiError
    from ittai_b200.qwen3 import Qwen3Decoder
    model, dims = tiny_hf
    d = Qwen3Decoder(model, max_batch=1, kv_capacity=256)
    for _ in range(2):
        d.next_id.fill_(10 ** 6)
        with pytest.raises(IttaiError, match="out of range"):
            d.decode(1)
        d.reset()
        d.prefill_cache(hf.prompt_ids(40, seed=1, vocab=dims.vocab))
        d.prefill_slots({0: [1, 2, 3]})
        d.prefill_slots({0: [4, 5]})
        d.check_status()
        assert d.lengths == d.pos.tolist() == [45]


@gpu
@pytest.mark.parametrize("batch", [1, 4])
def test_a_sum_of_squares_that_overflows(tiny_hf, batch):
    """Hidden values whose squares overflow fp32 normalise to zero, as 1 / sqrt(inf) has it: the ids and logits are the persistent
    kernel's (which an unused flag bit selects), not a row of NaNs."""
    from ittai_b200.qwen3 import Qwen3Decoder
    model, dims = tiny_hf
    sd = {k: v.clone() for k, v in model.state_dict().items()}
    sd["model.embed_tokens.weight"][5] = 3e19
    d = Qwen3Decoder(sd, max_batch=batch, kv_capacity=64)
    got = []
    for d.flags in (1 << 20, 0):
        d.reset()
        d.next_id.fill_(5)
        got.append((d.decode(1).clone(), d.logits.clone()))
    assert all(torch.equal(a, b) for a, b in zip(*got)) and not got[1][1].isnan().any()


@gpu
def test_calls_on_two_streams_follow_one_another(tiny_hf):
    """Calls of one decoder queued on two streams, nothing waited for in between: the second starts where the first ends."""
    from ittai_b200.qwen3 import Qwen3Decoder
    model, dims = tiny_hf
    d = Qwen3Decoder(model, max_batch=2, kv_capacity=256)
    d.next_id.fill_(9)
    want = d.decode(90).cpu()
    d.reset()
    d.next_id.fill_(9)
    torch.cuda.synchronize()
    streams, parts = [torch.cuda.Stream(), torch.cuda.Stream()], []
    for i, n in enumerate((40, 7, 1, 30, 12)):
        with torch.cuda.stream(streams[i % 2]):
            parts.append(d.decode(n, check=False))
    torch.cuda.synchronize()
    d.check_status()
    assert torch.equal(torch.cat([t.cpu() for t in parts], 1), want) and d.pos.tolist() == d.lengths == [90, 90]


@gpu
@pytest.mark.parametrize("batch,length,steps", [(1, 380, 45), (2, 20, 50), (4, 10, 21), (8, 600, 47)])
def test_several_tokens_a_graph_are_the_tokens_one_by_one(tiny_hf, batch, length, steps):
    """A long call queues several tokens as one graph from its 17th on, with single ones where the rest is shorter or a line of the rules
    (clusters: 400, 48 and 700 positions; tiles held: 625 of eight) falls among them: ids, logits and cache rows are those of calls of one
    step, in the first call and, with the graphs there, in the next."""
    from ittai_b200.qwen3 import Qwen3Decoder
    model, dims = tiny_hf
    g = torch.Generator().manual_seed(7 * batch)
    d = Qwen3Decoder(model, max_batch=batch, kv_capacity=1024)
    kv = [(torch.randn(d.kcache.shape, generator=g) * s).to(torch.bfloat16) for s in (1.0, 0.5)]
    ids = torch.randint(0, dims.vocab, (batch,), generator=g, dtype=torch.int32)

    def run(call):
        for c, t in zip((d.kcache, d.vcache), kv):
            c.copy_(t)
        d.rewind(length)
        d.next_id.copy_(ids)
        return torch.cat([d.decode(n).clone() for n in call], 1), d.logits.clone(), d.pos.clone(), d.kcache[:, :, :, :length + steps].clone(), d.vcache[:, :, :, :length + steps].clone()

    want = run([1] * steps)
    for call in ([steps], [steps], [17, steps - 17], [steps - 2, 2]):
        for got, ref in zip(run(call), want):
            assert torch.equal(got, ref), call


@gpu
@pytest.mark.parametrize("batch,length", [(1, 20), (8, 500)])
def test_the_graph_captured_behind_short_calls_is_the_tokens_one_by_one(tiny_hf, batch, length):
    """A request loop's calls of eight steps: single tokens until 64 of a kind are queued, then a graph of four, captured behind a call (the host
    side: test_qwen3_chain_host.py).  Ids, logits and cache rows are those of calls of one step."""
    from ittai_b200.qwen3 import Qwen3Decoder
    model, dims = tiny_hf
    g = torch.Generator().manual_seed(11 * batch)
    steps, kv, got = 96, None, []
    ids = torch.randint(0, dims.vocab, (batch,), generator=g, dtype=torch.int32)
    for call in (8, 1):
        d = Qwen3Decoder(model, max_batch=batch, kv_capacity=640)
        kv = kv or [(torch.randn(d.kcache.shape, generator=g) * s).to(torch.bfloat16) for s in (1.0, 0.5)]
        for c, t in zip((d.kcache, d.vcache), kv):
            c.copy_(t)
        d.rewind(length)
        d.next_id.copy_(ids)
        out = torch.cat([d.decode(call).clone() for _ in range(steps // call)], 1)
        got.append((out, d.logits.clone(), d.pos.clone(), d.kcache[:, :, :, :length + steps].clone(), d.vcache[:, :, :, :length + steps].clone()))
    for a, b in zip(*got):
        assert torch.equal(a, b)
