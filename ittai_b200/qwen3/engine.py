"""Qwen3-0.6B prefill on the tensor-core kernels, behind the reference's ``Engine`` surface
(reference ``src/ittai/qwen3/engine.py:13-187``).

``Engine.forward(input_ids)`` packs variable-length sequences into one activation matrix, runs 28 layers of
RMSNorm -> QKV GEMM -> QK-norm + RoPE -> causal GQA attention -> O-proj + residual -> RMSNorm -> gate/up GEMM with
SwiGLU -> down-proj + residual, and returns the L2-normalised final-norm of every sequence's last token, the
embedding head of the reference (``src/ittai/qwen3/base.py:131-145``).  ``PrefillCore`` is the layer loop itself; the
decoder reuses it to fill its KV cache from a prompt.
"""
from __future__ import annotations

import ctypes as C
import itertools

import numpy as np
import torch

from .. import _C, ops
from ..graphs import Graphs
from .config import BM, D, DGU, DQ, DQKV, EPS, FF, HD, NH, NKV, QB
from .decoder import _strip, pack_weights, rope_table
from .tasks import build_tasks


def rope_perm(n_heads):
    """Row order that puts the two halves of every RoPE pair side by side: within each 128-row head, rows
    0, 64, 1, 65, ... (reference ``src/ittai/qwen3/engine.py:13-14``).

    Kept for callers that import it; this build stores Q/K rows in the eager order and rotates (i, i + 64) directly."""
    within = np.stack([np.arange(HD // 2), np.arange(HD // 2) + HD // 2], axis=1).reshape(-1)
    return (np.arange(n_heads)[:, None] * HD + within[None, :]).reshape(-1)


def packing(seqlens):
    """Host description of one packed forward for the kernels: per-token positions, sequence ids and cache rows, and the
    per-sequence (first row, rows, first key row, key rows) records the attention kernel walks.
    Returns (pos, seq, slot, seqs, T) as int32 numpy arrays."""
    seqlens = [int(x) for x in seqlens]
    cu = np.concatenate([[0], np.cumsum(seqlens)]).astype(np.int64)
    T = int(cu[-1])
    pos = np.concatenate([np.arange(n) for n in seqlens]).astype(np.int32) if T else np.zeros(0, np.int32)
    seq = np.zeros(T, np.int32)                       # one packed key/value store: every token lives in "sequence 0"
    slot = np.arange(T, dtype=np.int32)
    seqs = np.array([[cu[s], seqlens[s], cu[s], seqlens[s]] for s in range(len(seqlens))], dtype=np.int32).reshape(-1, 4)
    return pos, seq, slot, seqs, T


def upload(arrays) -> torch.Tensor:
    """int32 arrays behind one another in one host tensor, to be copied to the device at once.  A large one is pinned (a
    pageable copy beyond the driver's staging size would wait for the stream); torch's host allocator keeps the block until
    the copy has run."""
    n = sum(a.size for a in arrays)
    t = torch.empty(n, dtype=torch.int32, pin_memory=n > 8192)
    np.concatenate([a.reshape(-1) for a in arrays], out=t.numpy())
    return t


class PrefillCore:
    """The 28-layer loop over a packed ``[T, 1024]`` activation matrix.  Owns the activation buffers (torch tensors, as
    the reference's Engine owns its buffers: ``src/ittai/qwen3/engine.py:123-134``); weights and the key/value store are
    borrowed."""

    def __init__(self, w: dict, n_layers: int, max_tokens: int, device, fused_rope: bool = True, fold_norm: bool = False, status=None):
        self.w, self.L, self.M, self.dev = w, n_layers, max_tokens, device
        self.fused_rope = fused_rope       # QK-norm + RoPE + cache scatter inside the QKV GEMM's epilogue
        # ``fold_norm``: the RMSNorms in front of the QKV and gate/up projections are folded into those GEMMs, as in the
        # reference's kernels (``src/ittai/qwen3/engine.py:107-114``: gain folded into the weights in fp32 and rounded once;
        # ``base.py:59-78``: the residual epilogue before leaves per-row partial sums of squares, the consuming epilogue
        # applies rstd): no norm kernel is left in a layer but the very first.  Off, every rounding point is the eager
        # module's (what the decoder's prefill uses: its cache feeds the decode loop).
        self.fold_norm = fold_norm
        if fold_norm:
            fold = lambda W, g: (W.float() * g.float()[:, None, :]).to(torch.bfloat16).contiguous()
            self.wqkv_f, self.wgu_f = fold(w["wqkv"], w["ln1"]), fold(w["wgu"], w["ln2"])
        self.stats = torch.empty(max_tokens, D // 128, 2, dtype=torch.float32, device=device)
        self.zeros = torch.zeros(DGU, dtype=torch.float32, device=device)
        z = lambda *s: torch.empty(*s, dtype=torch.bfloat16, device=device)
        self.h, self.xn, self.qkv, self.attn, self.act = z(max_tokens, D), z(max_tokens, D), z(max_tokens, DQKV), z(max_tokens, DQ), z(max_tokens, FF)
        self.status = ops.new_status(device) if status is None else status

    def run(self, T, tokens, pos, seq, slot, seqs, max_q_len, rope, kcache, vcache, kv_layer, kv_cap, k_strides,
            split_k=True):
        """``tokens/pos/seq/slot``: int32 device ``[T]``; ``seqs``: int32 device ``[n, 4]``; ``kcache`` / ``vcache``: the store
        of layer 0, laid out ``[B, 8, kv_cap, 128]``, each further layer ``kv_layer`` elements behind (0: one store for all);
        ``k_strides`` = (row, head, seq) in elements.  ``split_k=False``: sums over K in one order,
        whatever else is packed into the forward (see ``IttaiQwen3Prefill``).  Queues the whole stack on the current stream with one library call."""
        p, w = _C.Qwen3Prefill(), self.w
        p.n_layers, p.vocab, p.tokens, p.n_seqs, p.max_q_len, p.kv_cap = self.L, w["embed"].shape[0], T, seqs.shape[0], max_q_len, kv_cap
        p.fused_rope, p.split_k, p.eps = int(self.fused_rope), int(split_k), EPS
        for name in ("wqkv", "wo", "wgu", "wd", "ln1", "ln2", "qn", "kn", "embed"):
            setattr(p, name, w[name].data_ptr())
        if self.fold_norm:
            p.wqkv_f, p.wgu_f = self.wqkv_f.data_ptr(), self.wgu_f.data_ptr()
        p.rope, p.ids, p.pos, p.seq, p.slot, p.seqs = (t.data_ptr() for t in (rope, tokens, pos, seq, slot, seqs))
        p.kcache, p.vcache, p.kv_layer = kcache.data_ptr(), vcache.data_ptr(), kv_layer
        (p.k_row, p.k_head, p.k_seq), p.kv_rows_total = k_strides, (kv_layer or kcache.numel()) // HD
        p.h, p.xn, p.qkv, p.attn, p.act, p.stats, p.zeros, p.status = (
            t.data_ptr() for t in (self.h, self.xn, self.qkv, self.attn, self.act, self.stats, self.zeros, self.status))
        _C.check(_C.lib().ittai_qwen3_prefill_launch(C.byref(p), ops._stream(self.h)))
        return self.h[:T]


class Engine:
    """``Engine(sd, max_tokens, max_seqs, ...)`` with ``forward(input_ids: list[list[int]]) -> fp32 [B, 1024]``, a view of
    a persistent buffer (callers clone, as with the reference: ``src/ittai/qwen3/model.py:88``).  The tuning arguments
    of the reference (``arch, tile_n, stages, kv_block, group_m, warps``) are accepted and ignored."""

    @torch.no_grad()
    def __init__(self, sd, max_tokens, max_seqs, arch=None, tile_n=None, stages=None, kv_block=None, group_m=None, warps=8,
                 device="cuda", graph=True, fused_rope=True, fold_norm=True):
        sd = _strip(sd if isinstance(sd, dict) else sd.state_dict())
        self.dev = torch.device(device)
        self.M, self.Bmax = (max_tokens + BM - 1) // BM * BM, max_seqs
        self.L = 1 + max(int(k.split(".")[1]) for k in sd if k.startswith("layers."))
        self.w = pack_weights(sd, self.L, self.dev)
        self.embed, self.fin_w = self.w["embed"], self.w["fin_w"]
        self.rope = rope_table(self.M, self.dev)
        self.core = PrefillCore(self.w, self.L, self.M, self.dev, fused_rope=fused_rope, fold_norm=fold_norm)
        z = lambda *s, dt: torch.zeros(*s, dtype=dt, device=self.dev)
        # one packed key/value store reused by every layer: the embedding pass keeps no cache
        self.kbuf, self.vbuf = z(1, NKV, self.M, HD, dt=torch.bfloat16), z(1, NKV, self.M, HD, dt=torch.bfloat16)
        # the packing of a forward, written by one copy: seqs [B, 4], last [B], then tokens, pos, seq, slot [T] (see ``_views``)
        self.meta = z(5 * max_seqs + 4 * self.M, dt=torch.int32)
        self.out = z(max_seqs, D, dt=torch.float32)
        self._graphs, self._plain = Graphs(self.GRAPHS if graph else 0), Graphs(0)
        self._unread = False                 # a shape ran for the first time and its status words have not been read yet

    def _views(self, T, B):
        """The parts of ``meta`` for a forward of ``T`` tokens in ``B`` sequences; ``seqs`` first: it is read 16 bytes at a time."""
        m, o = self.meta, 5 * B
        return m[:4 * B].view(B, 4), m[4 * B:o], *(m[o + i * T:o + (i + 1) * T] for i in range(4))

    def _body(self, T, B, max_len):
        seqs, last, tokens, pos, seq, slot = self._views(T, B)
        h = self.core.run(T, tokens, pos, seq, slot, seqs, max_len, self.rope, self.kbuf, self.vbuf, 0, self.M, (HD, self.M * HD, 0))
        _C.check(_C.lib().ittai_qwen3_final_pool(h.data_ptr(), last.data_ptr(), self.fin_w.data_ptr(), self.out.data_ptr(), B, EPS,
                                                 ops._stream(h)))

    # Up to this many tokens a repeated shape is replayed from a CUDA graph; above, the GPU is busy for longer than the host
    # needs to queue the launches.
    GRAPH_TOKENS, GRAPHS = 1024, 16

    @torch.no_grad()
    def forward(self, input_ids, check=True):
        """Embeddings of the packed sequences.  The first forward of a shape is waited for and its status words are read; with
        ``check=False`` that is left to ``check_new``, for callers that queue several forwards."""
        seqlens = [len(x) for x in input_ids]
        T, B = sum(seqlens), len(seqlens)
        assert T <= self.M and B <= self.Bmax and min(seqlens) > 0
        pos, seq, slot, seqs, _ = packing(seqlens)
        flat = np.fromiter(itertools.chain.from_iterable(input_ids), np.int32, T)
        if int(flat.min()) < 0 or int(flat.max()) >= self.embed.shape[0]:
            raise ValueError(f"token id outside [0, {self.embed.shape[0]})")      # the gather kernel would clamp it silently
        meta = upload((seqs, seqs[:, 0] + seqs[:, 1] - 1, flat, pos, seq, slot))
        self.meta[:meta.numel()].copy_(meta, non_blocking=True)
        # the launches depend on these three numbers alone, the packing itself is read on the device
        key = (T, B, max(seqlens))
        new, graph, capture = (self._graphs if T <= self.GRAPH_TOKENS else self._plain).use(key)
        self._unread |= new
        if capture:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                self._body(*key)
            self._graphs.put(key, graph)
        if graph is not None:
            graph.replay()
        else:
            self._body(*key)
        if check:
            self.check_new()
        return self.out[:B]

    def check(self) -> None:
        """Wait for the queued forwards and raise if a bounded wait of theirs ran out."""
        self._unread = False
        ops.check_status(self.core.status)

    def check_new(self) -> None:
        """``check`` if a shape has run for the first time since the last one."""
        if self._unread:
            self.check()

    def task_list(self, seqlens, group_m=8):
        """The forward over ``seqlens`` as the reference's device queue would see it: ``(tasks, expect, T)`` of
        ``build_tasks`` for this engine's geometry (256-column GEMM tiles, one arrival per tile).  The launches this
        engine records into its CUDA graph realise the same dependencies by stream order, phase after phase; the list
        is what a single persistent kernel would walk instead."""
        return build_tasks(seqlens, self.M // BM, self.Bmax, self.L + 1, (DQKV // 256, D // 256, 2 * FF // 256, D // 256), 1, 128, group_m)
