"""SigLIP towers whose geometry the tensor-core kernels do not take as it is (so400m: width 1152, head_dim 72, MLP 4304,
patch 14): the same kernels on zero-padded weights.

The reference pads too (head_dim to a multiple of 16, the MLP width to a multiple of 128, the patch row to a multiple of
32, tokens per image to a multiple of 128: ``src/ittai/siglip/kernel.py:537-539,551-563``).  Here the widths go up to what
the kernels of this build take: model width and MLP width to multiples of 256 (the two-SM GEMM's tile), head_dim to 80
in the encoder and 128 in the pooling head (the attention kernels know 64, 80 and 128), the patch row to a multiple of 64.  Everything that is padding is zero and stays
zero: padded weight rows and bias entries are zero, so the padded columns of every activation are zero, so the padded
weight columns never contribute.  The softmax scale of the attention kernels is ``padded head_dim ** -0.5``; the q
projection is pre-scaled by ``sqrt(padded / true)`` so that the scores carry the true ``head_dim ** -0.5``.  LayerNorm runs
as its own pass over the true width (the statistics must not see the padding).  Tokens are packed, not padded.
"""
from __future__ import annotations

import ctypes as C
import math

import torch
import torch.nn.functional as F

from .. import _C, ops
from ..graphs import Graphs


def _up(n: int, m: int) -> int:
    return (n + m - 1) // m * m


class PaddedEngine:
    """Same surface as ``Engine``: ``forward(inputs) -> bf16 [B, D]`` view of a persistent buffer, ``check()``, ``flops()``."""

    PARTS = 8                # as in ``Engine``

    @torch.no_grad()
    def __init__(self, vm, B, graph=True, fold_ln=True, chain=True, **ignored):
        from .kernel import _vision_model
        vm = _vision_model(vm)
        cfg, emb = vm.config, vm.embeddings
        self.vm, self.B = vm, B
        self.conv = isinstance(emb.patch_embedding, torch.nn.Conv2d)
        D, Fm, H, p = cfg.hidden_size, cfg.intermediate_size, cfg.num_attention_heads, cfg.patch_size
        self.D, self.F, self.H, self.L, self.p, self.eps = D, Fm, H, cfg.num_hidden_layers, p, cfg.layer_norm_eps
        self.img = getattr(cfg, "image_size", 0)
        hd = D // H
        if hd > 128 or hd * H != D:
            raise NotImplementedError(f"head_dim {hd}: the attention kernels take at most 128")
        self.hd, self.hdp = hd, 64 if hd <= 64 else 128
        self.Dp, self.Fp, self.Kp0 = _up(D, 256), _up(Fm, 256), 3 * p * p
        self.Kp = _up(self.Kp0, 64)
        self.S0 = emb.num_patches
        dev = next(vm.parameters()).device
        self.dev = dev
        Dp, Fp, hdp, Hp = self.Dp, self.Fp, self.hdp, H * self.hdp
        self.M = M = B * self.S0
        f = lambda t: t.detach().to(dev, torch.float32)
        bf = lambda t: t.to(torch.bfloat16).contiguous()

        def pad2(w, rows, cols):                     # fp32 [r, c] -> fp32 [rows, cols], zero-filled
            return F.pad(f(w), (0, cols - w.shape[1], 0, rows - w.shape[0]))

        def heads_out(w, b, to, scale=1.0):          # a projection INTO head space: [H*hd, D], [H*hd] -> [H*to, Dp], [H*to]
            w = F.pad(f(w).view(H, hd, D) * scale, (0, Dp - D, 0, to - hd)).reshape(H * to, Dp)
            b = F.pad(f(b).view(H, hd) * scale, (0, to - hd)).reshape(H * to)
            return w, b

        def heads_in(w, to):                         # a projection OUT OF head space: [D, H*hd] -> [Dp, H*to]
            return F.pad(f(w).view(D, H, hd), (0, to - hd, 0, 0, 0, Dp - D)).reshape(Dp, H * to)

        # the encoder's heads go to 80 columns where the key-loop kernel's packed form covers them (so400m: 72), the one-query
        # pooling head keeps ``hdp``
        self.hde = 80 if 64 < hd <= 80 and self.S0 > 64 and 3 * H * 80 % 256 == 0 and H * 80 % 64 == 0 else hdp
        hde, He = self.hde, H * self.hde
        qs = math.sqrt(hde / hd)
        pe = emb.patch_embedding
        self.wpe, self.bpe = bf(pad2(pe.weight.reshape(D, -1), Dp, self.Kp)), F.pad(f(pe.bias), (0, Dp - D)).contiguous()
        self.layers = []
        for lyr in vm.encoder.layers:
            a, m = lyr.self_attn, lyr.mlp
            parts = [heads_out(a.q_proj.weight, a.q_proj.bias, hde, qs), heads_out(a.k_proj.weight, a.k_proj.bias, hde), heads_out(a.v_proj.weight, a.v_proj.bias, hde)]
            self.layers.append(dict(
                ln1=(f(lyr.layer_norm1.weight).contiguous(), f(lyr.layer_norm1.bias).contiguous()),
                ln2=(f(lyr.layer_norm2.weight).contiguous(), f(lyr.layer_norm2.bias).contiguous()),
                wqkv=bf(torch.cat([w for w, _ in parts])), bqkv=torch.cat([b for _, b in parts]).contiguous(),
                wo=bf(heads_in(a.out_proj.weight, hde)), bo=F.pad(f(a.out_proj.bias), (0, Dp - D)).contiguous(),
                w1=bf(pad2(m.fc1.weight, Fp, Dp)), b1=F.pad(f(m.fc1.bias), (0, Fp - Fm)).contiguous(),
                w2=bf(pad2(m.fc2.weight, Dp, Fp)), b2=F.pad(f(m.fc2.bias), (0, Dp - D)).contiguous()))
        self.post = (f(vm.post_layernorm.weight).contiguous(), f(vm.post_layernorm.bias).contiguous())
        h = vm.head
        inw, inb = h.attention.in_proj_weight, h.attention.in_proj_bias
        # the probe's query does not depend on the image: projected once, as the eager module would (bf16 Linear), then laid
        # out in padded head space with the score scale folded in
        q = F.linear(h.probe[0].to(dev, torch.bfloat16), inw[:D].to(dev, torch.bfloat16), inb[:D].to(dev, torch.bfloat16)).float()
        self.probe_q = bf(F.pad(q.view(H, hd) * math.sqrt(hdp / hd), (0, hdp - hd)).reshape(1, Hp))
        kv = [heads_out(inw[D:2 * D], inb[D:2 * D], hdp), heads_out(inw[2 * D:], inb[2 * D:], hdp)]
        self.wkv, self.bkv = bf(torch.cat([w for w, _ in kv])), torch.cat([b for _, b in kv]).contiguous()
        self.who, self.bho = bf(heads_in(h.attention.out_proj.weight, hdp)), F.pad(f(h.attention.out_proj.bias), (0, Dp - D)).contiguous()
        self.hln = (f(h.layernorm.weight).contiguous(), f(h.layernorm.bias).contiguous())
        self.hw1, self.hb1 = bf(pad2(h.mlp.fc1.weight, Fp, Dp)), F.pad(f(h.mlp.fc1.bias), (0, Fp - Fm)).contiguous()
        self.hw2, self.hb2 = bf(pad2(h.mlp.fc2.weight, Dp, Fp)), F.pad(f(h.mlp.fc2.bias), (0, Dp - D)).contiguous()
        # LayerNorm folded into the GEMM that follows it (as in ``Engine``): W' = W * gain along K (zero in the padding
        # columns), row sums of the rounded W', bias' = bias + W beta; the producing GEMM's epilogue writes the row sums
        # and the consuming epilogue finishes mean and rstd over the TRUE width (``stats_k``).
        self.fold_ln = bool(fold_ln) and M > 128
        self.chain = bool(chain) and self.fold_ln and M >= 1024
        self.n_sms = torch.cuda.get_device_properties(dev).multi_processor_count

        def folded(w_bf16, bias, ln):
            g, beta = (F.pad(t, (0, Dp - D)) for t in ln)
            wf = w_bf16.float()
            wp = (wf * g).to(torch.bfloat16).contiguous()
            return wp, (bias + wf @ beta).contiguous(), wp.float().sum(1).contiguous()

        if self.fold_ln:
            for w in self.layers:
                w["qkv_f"] = folded(w["wqkv"], w["bqkv"], w["ln1"])
                w["fc1_f"] = folded(w["w1"], w["b1"], w["ln2"])
            self.kv_f = folded(self.wkv, self.bkv, self.post)
            self.stats_a = torch.zeros(M, Dp // 128, 2, dtype=torch.float32, device=dev)
            self.stats_m = torch.zeros(M, Dp // 128, 2, dtype=torch.float32, device=dev)
            self.chain_flags = torch.zeros(len(self.layers) + 1, 4 * 2 * ((M + 255) // 256), dtype=torch.int32, device=dev)
        z = lambda *s: torch.zeros(*s, dtype=torch.bfloat16, device=dev)
        self.pos = z(M, Dp)
        if self.conv:
            self.pos[:, :D] = emb.position_embedding.weight.detach().to(dev, torch.bfloat16).repeat(B, 1)
            self.pixels = torch.empty(B, 3, self.img, self.img, dtype=torch.float32, device=dev)
        else:
            side = int(round(self.S0 ** 0.5))
            self.pos_grid = f(emb.position_embedding.weight).reshape(side, side, D)
        self.patches, self.x, self.y = z(M, self.Kp), z(M, Dp), z(M, Dp)
        self.qkv, self.attn, self.h = z(M, 3 * He), z(M, He), z(M, Fp)
        self.kv, self.pool_a, self.pool_r, self.pool_y, self.pool_h = z(M, 2 * Hp), z(B, Hp), z(B, Dp), z(B, Dp), z(B, Fp)
        self.embeds_p = z(B, Dp)
        S = self.S0
        self.seqs = torch.tensor([[b * S, S, b * S, S] for b in range(B)], dtype=torch.int32, device=dev)
        self.pool_seqs = torch.tensor([[b, 1, b * S, S] for b in range(B)], dtype=torch.int32, device=dev)
        self.status = ops.new_status(dev)
        self._full, self._graphs, self._unread = Graphs(1 if graph else 0), Graphs(self.PARTS if graph else 0), False

    def _chained(self, rows):
        from .kernel import chain_pays
        He, Dp, Fp = self.H * self.hde, self.Dp, self.Fp
        return self.chain and chain_pays(rows, ((3 * He, Dp), (Dp, He), (Fp, Dp), (Dp, Fp)), self.n_sms)

    def _body(self, B):
        """Queue the forward of the first ``B`` images of the buffers."""
        D, S, H, hdp, eps, st = self.D, self.S0, self.H, self.hdp, self.eps, self.status
        Hp, M = H * hdp, B * S
        patches, pos, x, y, h, qkv_b, attn, kv = (t[:M] for t in (self.patches, self.pos, self.x, self.y, self.h, self.qkv, self.attn, self.kv))
        if self.fold_ln:
            stats_a, stats_m = self.stats_a[:M], self.stats_m[:M]
        seqs, pool_seqs = self.seqs[:B], self.pool_seqs[:B]
        pool_a, pool_r, pool_y, pool_h, embeds = (t[:B] for t in (self.pool_a, self.pool_r, self.pool_y, self.pool_h, self.embeds_p))
        if self.conv:       # patch rows in (channel, row, column) order: what a Conv2d weight flattens to; the padding columns stay zero
            _C.check(_C.lib().ittai_siglip_im2col(self.pixels.data_ptr(), self.patches.data_ptr(), B, self.img, self.img, self.p, self.Kp,
                                                  ops._stream(self.pixels)))
        def attention():
            # row totals + status words: the tcgen05 key-loop kernel (keys and values packed like the queries)
            he, He = self.hde, H * self.hde
            ops.attention(qkv_b, qkv_b[:, He:], qkv_b[:, 2 * He:], attn, seqs, n_heads=H, group=1, head_dim=he, causal=False, max_q_len=S,
                          q_strides=(3 * He, he), k_strides=(3 * He, he, 0), v_strides=(3 * He, he, 0), o_strides=(He, he), max_kv_len=S,
                          q_rows_total=self.M, kv_rows_total=self.M, status=st, seqs_ready=self.conv)   # else the position kernel writes them

        if self.fold_ln:
            sw = dict(static_w=not self.chain)                  # a chained GEMM takes no such flag
            ln = dict(stats_eps=eps, stats_k=D, **sw)
            embed = ops.gemm_desc(patches, self.wpe, st, **sw, bias=self.bpe, residual=pos, out=x, stats_out=stats_m)[0]
            qkv = lambda w: ops.gemm_desc(x, w["qkv_f"][0], st, bias=w["qkv_f"][1], out=qkv_b, row_stats=stats_m,
                                          col_sums=w["qkv_f"][2], **ln)[0]
            chained = self._chained(M)
            run = ops.gemm_chain if chained else lambda descs, flags: ops.gemm_each(descs, x)
            if chained:
                self.chain_flags.zero_()
            run([embed, qkv(self.layers[0])], self.chain_flags[len(self.layers)])
            for i, w in enumerate(self.layers):
                attention()
                descs = [ops.gemm_desc(attn, w["wo"], st, **sw, bias=w["bo"], residual=x, out=x, stats_out=stats_a)[0],
                         ops.gemm_desc(x, w["fc1_f"][0], st, bias=w["fc1_f"][1], epi=_C.EPI_GELU, out=h, row_stats=stats_a,
                                       col_sums=w["fc1_f"][2], **ln)[0],
                         ops.gemm_desc(h, w["w2"], st, **sw, bias=w["b2"], residual=x, out=x, stats_out=stats_m)[0]]
                descs.append(qkv(self.layers[i + 1]) if i + 1 < len(self.layers) else
                             ops.gemm_desc(x, self.kv_f[0], st, bias=self.kv_f[1], out=kv, row_stats=stats_m, col_sums=self.kv_f[2], **ln)[0])
                run(descs, self.chain_flags[i])
        else:
            ops.gemm(patches, self.wpe, st, static_w=True, bias=self.bpe, residual=pos, out=x)
            for w in self.layers:
                ops.layernorm_rows(x[:, :D], *w["ln1"], eps, out=y[:, :D])
                ops.gemm(y, w["wqkv"], st, static_w=True, bias=w["bqkv"], out=qkv_b)
                attention()
                ops.gemm(attn, w["wo"], st, static_w=True, bias=w["bo"], residual=x, out=x)
                ops.layernorm_rows(x[:, :D], *w["ln2"], eps, out=y[:, :D])
                ops.gemm(y, w["w1"], st, static_w=True, bias=w["b1"], epi=_C.EPI_GELU, out=h)
                ops.gemm(h, w["w2"], st, static_w=True, bias=w["b2"], residual=x, out=x)
            # post-LayerNorm + MAP head: the probe attends over the image's tokens, then LayerNorm + MLP with a residual
            ops.layernorm_rows(x[:, :D], *self.post, eps, out=y[:, :D])
            ops.gemm(y, self.wkv, st, static_w=True, bias=self.bkv, out=kv)
        ops.attention(self.probe_q, kv, kv[:, Hp:], pool_a, pool_seqs, n_heads=H, group=1, head_dim=hdp, causal=False, max_q_len=1, q_strides=(0, hdp),
                      k_strides=(2 * Hp, hdp, 0), v_strides=(2 * Hp, hdp, 0), o_strides=(Hp, hdp))
        ops.gemm(pool_a, self.who, st, static_w=True, bias=self.bho, out=pool_r)
        ops.layernorm_rows(pool_r[:, :D], *self.hln, eps, out=pool_y[:, :D])
        ops.gemm(pool_y, self.hw1, st, static_w=True, bias=self.hb1, epi=_C.EPI_GELU, out=pool_h)
        ops.gemm(pool_h, self.hw2, st, static_w=True, bias=self.hb2, residual=pool_r, out=embeds)

    @torch.no_grad()
    def forward(self, inp):
        self._load(inp, self.B)
        self._run(self.B)
        self.check_new()
        return self.embeds_p[:, :self.D]

    @torch.no_grad()
    def forward_part(self, inp, check=True):
        from .kernel import part_size
        n = len(inp["pixel_values"])
        assert 1 <= n <= self.B, f"1 to {self.B} images, got {n}"
        self._load(inp, n)
        self._run(part_size(n, self.B, self.S0, self.chain))
        if check:
            self.check_new()
        return self.embeds_p[:n, :self.D]

    def _load(self, inp, n):
        from .kernel import checked_shapes
        px, S, K = inp["pixel_values"], self.S0, self.Kp0
        if self.conv:
            assert px.shape[0] == n and px.shape[1:] == self.pixels.shape[1:], f"expected {(n, *self.pixels.shape[1:])}, got {tuple(px.shape)}"
            self.pixels[:n].copy_(px, non_blocking=True)
            return
        assert tuple(px.shape) == (n, S, K), f"expected {(n, S, K)}, got {tuple(px.shape)}"
        shapes = checked_shapes(inp, n, S)
        self.patches[:n * S, :K].copy_(px.reshape(n * S, K), non_blocking=True)
        shapes_d = shapes.to(self.dev, non_blocking=True)
        _C.check(_C.lib().ittai_siglip_positions(self.pos_grid.data_ptr(), self.pos_grid.shape[0], self.D, shapes_d.data_ptr(), n, S, self.pos.data_ptr(),
                                                 self.pos.stride(0), self.seqs.data_ptr(), self.pool_seqs.data_ptr(), ops._stream(self.pos)))

    def _run(self, n):
        from .kernel import Engine
        Engine._run(self, n)

    def check(self) -> None:
        self._unread = False
        ops.check_status(self.status)

    def check_new(self) -> None:
        if self._unread:
            self.check()

    def launches_per_forward(self) -> int:
        """Kernels in one forward (all inside one CUDA graph)."""
        n_l = len(self.layers)
        encoder = (n_l + 1) + n_l if self._chained(self.M) else 1 + n_l * (5 if self.fold_ln else 7) + (1 if self.fold_ln else 2)
        return (1 if self.conv else 0) + encoder + 5

    def flops(self, formula: str = "reference") -> float:
        """FLOPs of one forward at the TRUE widths (the padding is overhead, not work); formulas as in ``Engine.flops``."""
        B, L, S, D, Fm = self.B, self.L, self.S0, self.D, self.F
        ref = B * L * (2 * S * D * (4 * D + 2 * Fm) + 4 * S * S * D)
        if formula == "reference":
            return float(ref)
        head = 2 * S * D * 2 * D + 4 * S * D + 2 * D * D + 4 * D * Fm
        return float(ref + B * (2 * S * D * self.Kp0 + head))
