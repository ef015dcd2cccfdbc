"""Performance cases: the work a program built on this package gives it, through the public entry points.

Language side (Qwen3-0.6B, 28 layers): greedy decode from a filled cache, prompt prefill, one chat turn from host memory,
the request loop, and text embedding from one query to a corpus.  Vision side: SigLIP ViT-B/16-224, the SigLIP2 NaFlex base
tower and the so400m-patch14-384 tower, from one image to a stack of batches.  Everything is bf16 with fp32 accumulation,
the one data type the package computes in.  Weights are random at the true geometry, made on the GPU from the seed.
"""
from __future__ import annotations

import math
import random
from types import SimpleNamespace

import torch
from torch import nn

from ittai_b200.qwen3 import (D, DGU, DKV, DQ, DQKV, FF, HD, L, NKV, DecodeServer, Qwen3Decoder, Qwen3Embedder,
                              decode_bytes_per_token)
from ittai_b200.siglip.kernel import Siglip2Embedder

VOCAB = 151936
DEV = "cuda"
# hidden, heads, mlp, layers, patch, image side (None: variable resolution), patches per image
TOWERS = {"vit": (768, 12, 3072, 12, 16, 224, 196), "naflex": (768, 12, 3072, 12, 16, None, 256),
          "so400m": (1152, 16, 4304, 27, 14, 384, 729)}


def listed():
    return [
        # a long chat, one user: 256 tokens generated behind 4096 cached ones (the repository's headline benchmark)
        dict(name="decode_1x4096", path="decode", batch=1, context=4096, steps=256),
        # a full server at the end of its cache: eight sequences near the capacity of 8192
        dict(name="decode_8x8160", path="decode", batch=8, context=8160, steps=32),
        # eight long prompts filled in together (the prefill half of the same server benchmark)
        dict(name="prefill_8x2048", path="prefill", batch=8, prompt=2048),
        # one short chat turn, ids in from the host and ids back: prefill, the first token and 31 more
        dict(name="generate_47", path="generate", prompt=47, steps=32),
        # the request loop: twelve requests of mixed prompt and answer lengths over four sequence slots
        dict(name="serve_4slots", path="serve", slots=4, requests=12, shortest=16, longest=512, answer=48),
        # one search query through the embedder: latency only
        dict(name="embed_query", path="embed", sequences=1, shortest=23, longest=23, max_tokens=8192),
        # the embedding benchmark: 64 texts of 512 tokens as one forward
        dict(name="embed_64x512", path="embed", sequences=64, shortest=512, longest=512, max_tokens=32768),
        # a corpus of texts of every length at the embedder's default limits: about a dozen forwards, no two packed alike
        dict(name="embed_corpus", path="embed", sequences=600, shortest=16, longest=512, max_tokens=8192),
        # one uploaded image, from host memory
        dict(name="image_1", path="images", tower="vit", images=1, batch=1, host=True),
        # an image set from pinned host memory at the default batch of 64; the last batch is a short one
        dict(name="images_200", path="images", tower="vit", images=200, batch=64, host=True),
        # processor outputs of photos with mixed aspect ratios for the variable-resolution tower
        dict(name="naflex_24", path="images", tower="naflex", images=24, batch=16, host=True),
        # the large tower on images that a GPU decoder left in device memory
        dict(name="so400m_8", path="images", tower="so400m", images=8, batch=8, host=False),
    ]


def _log(rng, lo, hi):
    """An integer of [lo, hi], spread evenly over its logarithm."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    path = rng.choice(["decode", "prefill", "generate", "serve", "embed", "embed", "images", "images"])
    if path == "decode":
        steps = _log(rng, 8, 256)
        return dict(path=path, batch=rng.choice([1, 2, 4, 8]), context=_log(rng, 8, 8192 - steps), steps=steps)
    if path == "prefill":
        batch = rng.choice([1, 2, 4, 8])
        return dict(path=path, batch=batch, prompt=_log(rng, 5, min(8000, 16384 // batch)))
    if path == "generate":
        return dict(path=path, prompt=_log(rng, 5, 2000), steps=_log(rng, 4, 128))
    if path == "serve":
        return dict(path=path, slots=rng.choice([2, 4, 8]), requests=rng.randint(4, 24), shortest=_log(rng, 2, 64),
                    longest=_log(rng, 65, 1024), answer=_log(rng, 8, 96))
    if path == "embed":
        shortest = _log(rng, 3, 512)
        longest = _log(rng, shortest, 2048)
        return dict(path=path, sequences=_log(rng, 1, max(1, min(600, 65536 // longest))), shortest=shortest, longest=longest,
                    max_tokens=rng.choice([8192, 32768]))
    tower = rng.choice(["vit", "vit", "naflex", "so400m"])
    batch = _log(rng, 1, 12 if tower == "so400m" else 64)
    images = _log(rng, batch, 12 if tower == "so400m" else 3 * batch)
    return dict(path=path, tower=tower, images=images, batch=batch, host=rng.random() < 0.5)


def _lengths(n, lo, hi):
    """``n`` text lengths spread evenly over the logarithm of [lo, hi], in an order of no pattern, the same for every seed."""
    spread = [round(lo * (hi / lo) ** ((i + 0.5) / n)) for i in range(n)]
    random.Random(n).shuffle(spread)
    return spread


def _grids(n):
    """Patch grids of ``n`` images with aspect ratios from 1:2 to 2:1, each filling the budget of 256 patches as the
    variable-resolution processor does."""
    out = []
    for i in range(n):
        ratio = 2.0 ** (2 * ((i * 0.6180339887) % 1.0) - 1)
        h = max(1, int(16 * math.sqrt(ratio)))
        out.append((h, 256 // h))
    return out


def _language_weights(g):
    """A state dict with the checkpoint's key names.  Linear weights N(0, 0.02); embedding rows N(0, 1) and a final gain of
    0.1, which put the logits where a trained model has them (3 wide, the chosen token some 20 above the next): the greedy
    choice is then decided by more than the rounding, and sequences stay comparable over many steps."""
    def rn(*shape, std=0.02, mean=0.0):
        return torch.empty(*shape, dtype=torch.bfloat16, device=DEV).normal_(mean, std, generator=g)
    sd = {"embed_tokens.weight": rn(VOCAB, D, std=1.0), "norm.weight": rn(D, std=0.01, mean=0.1)}
    for l in range(L):
        p = f"layers.{l}."
        for name, rows, cols in (("self_attn.q_proj", DQ, D), ("self_attn.k_proj", DKV, D), ("self_attn.v_proj", DKV, D),
                                 ("self_attn.o_proj", D, DQ), ("mlp.gate_proj", FF, D), ("mlp.up_proj", FF, D), ("mlp.down_proj", D, FF)):
            sd[p + name + ".weight"] = rn(rows, cols)
        for name, n in (("input_layernorm", D), ("post_attention_layernorm", D), ("self_attn.q_norm", HD), ("self_attn.k_norm", HD)):
            sd[p + name + ".weight"] = rn(n, std=0.1, mean=1.0)
    return sd


class _Tower(nn.Module):
    """The modules of a SigLIP vision tower under the names a checkpoint's module has, for its weights alone."""

    def __init__(self, kind):
        super().__init__()
        d, heads, mlp, layers, patch, side, patches = TOWERS[kind]
        group = lambda **kw: nn.ModuleDict(kw)
        self.config = SimpleNamespace(hidden_size=d, num_attention_heads=heads, intermediate_size=mlp, num_hidden_layers=layers,
                                      patch_size=patch, image_size=side, num_patches=patches, layer_norm_eps=1e-6)
        self.embeddings = nn.Module()
        self.embeddings.patch_embedding = nn.Conv2d(3, d, patch, patch) if side else nn.Linear(3 * patch * patch, d)
        self.embeddings.position_embedding = nn.Embedding(patches, d)
        self.embeddings.num_patches = patches
        self.encoder = nn.Module()
        self.encoder.layers = nn.ModuleList()
        for _ in range(layers):
            lyr = nn.Module()
            lyr.layer_norm1, lyr.layer_norm2 = nn.LayerNorm(d), nn.LayerNorm(d)
            lyr.self_attn, lyr.mlp = nn.Module(), nn.Module()
            for name in ("q_proj", "k_proj", "v_proj", "out_proj"):
                setattr(lyr.self_attn, name, nn.Linear(d, d))
            lyr.mlp.fc1, lyr.mlp.fc2 = nn.Linear(d, mlp), nn.Linear(mlp, d)
            self.encoder.layers.append(lyr)
        self.post_layernorm = nn.LayerNorm(d)
        self.head = nn.Module()
        self.head.probe = nn.Parameter(torch.empty(1, 1, d))
        self.head.attention = nn.MultiheadAttention(d, heads, batch_first=True)
        self.head.layernorm = nn.LayerNorm(d)
        self.head.mlp = nn.Module()
        self.head.mlp.fc1, self.head.mlp.fc2 = nn.Linear(d, mlp), nn.Linear(mlp, d)


@torch.no_grad()
def _vision_tower(kind, g):
    with torch.device(DEV):
        tower = _Tower(kind).to(torch.bfloat16)
    for name, p in tower.named_parameters():
        if name.endswith("bias"):
            p.normal_(0.0, 0.02, generator=g)
        elif "norm" in name:
            p.normal_(1.0, 0.1, generator=g)
        else:
            p.normal_(0.0, p[0].numel() ** -0.5, generator=g)
    return tower.eval()


@torch.no_grad()
def prepare(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    path = case["path"]
    if path == "images":
        embedder = Siglip2Embedder(_vision_tower(case["tower"], g), batch_size=case["batch"])
        n = case["images"]
        _, _, _, _, patch, side, patches = TOWERS[case["tower"]]
        place = (lambda t: t.cpu().pin_memory()) if case["host"] else (lambda t: t)
        if side:
            return SimpleNamespace(case=case, embedder=embedder, images=place(torch.randn(n, 3, side, side, generator=g, device=DEV)))
        shapes = _grids(n)
        pixels = torch.randn(n, patches, 3 * patch * patch, generator=g, device=DEV)
        mask = torch.zeros(n, patches, dtype=torch.int64)
        for i, (h, w) in enumerate(shapes):
            pixels[i, h * w:] = 0.0
            mask[i, :h * w] = 1
        # masks and grids stay in host memory, where the image processor makes them
        return SimpleNamespace(case=case, embedder=embedder, images={"pixel_values": place(pixels), "pixel_attention_mask": mask,
                                                                     "spatial_shapes": torch.tensor(shapes)})
    weights = _language_weights(g)
    ids = lambda *shape: torch.randint(0, VOCAB, shape, generator=g, device=DEV, dtype=torch.int32)
    if path == "embed":
        lengths = _lengths(case["sequences"], case["shortest"], case["longest"])
        texts = [t.tolist() for t in ids(sum(lengths)).cpu().split(lengths)]
        return SimpleNamespace(case=case, embedder=Qwen3Embedder(weights, max_tokens=case["max_tokens"]), texts=texts)
    if path == "serve":
        lengths = _lengths(case["requests"], case["shortest"], case["longest"])
        answers = _lengths(case["requests"] + 1, max(1, case["answer"] // 4), case["answer"])[1:]
        requests = [(t.tolist(), n) for t, n in zip(ids(sum(lengths)).cpu().split(lengths), answers)]
        return SimpleNamespace(case=case, decoder=Qwen3Decoder(weights, max_batch=case["slots"], kv_capacity=2048), requests=requests)
    if path == "generate":
        return SimpleNamespace(case=case, decoder=Qwen3Decoder(weights, kv_capacity=4096), prompt=ids(case["prompt"]).cpu())
    decoder = Qwen3Decoder(weights, max_batch=case["batch"], kv_capacity=8192)
    if path == "prefill":
        return SimpleNamespace(case=case, decoder=decoder, prompts=ids(case["batch"], case["prompt"]).cpu())
    # decode: keys as the head norm leaves them (unit variance), values as the value projection does
    for l in range(L):
        decoder.kcache[l, :, :, :case["context"]].normal_(0.0, 1.0, generator=g)
        decoder.vcache[l, :, :, :case["context"]].normal_(0.0, 0.64, generator=g)
    return SimpleNamespace(case=case, decoder=decoder, first=ids(case["batch"]))


def run(state):
    case = state.case
    path = case["path"]
    if path == "images":
        return state.embedder.embed(state.images)
    if path == "embed":
        return state.embedder.embed(state.texts)
    dec = state.decoder
    if path == "serve":
        server = DecodeServer(dec, chunk=8)
        for prompt, answer in state.requests:
            server.submit(prompt, answer)
        done = server.run()
        return torch.tensor([t for rid in sorted(done) for t in done[rid]])
    if path == "generate":
        out = dec.generate(state.prompt, case["steps"])
        rows = slice(0, case["prompt"] + case["steps"] - 1)
    elif path == "prefill":
        dec.reset()
        out = dec.prefill(state.prompts)
        rows = slice(0, case["prompt"])
    else:
        dec.rewind(case["context"])
        dec.next_id.copy_(state.first)
        out = dec.decode(case["steps"])
        rows = slice(case["context"], case["context"] + case["steps"])
    # the ids, the last logits, and the cache rows that the pass wrote
    return out, dec.logits, dec.kcache[:, :, :, rows], dec.vcache[:, :, :, rows]


_LAYER = D * (DQKV + DQ + DGU + FF)             # weights of one layer's four projections
_KV_ROW = L * 2 * DKV * 2                       # bytes of one position of the cache


def _language_flops(tokens, attended, heads):
    """``tokens`` through the layers, ``attended`` query-key pairs in all, ``heads`` rows through the language head."""
    return 2.0 * tokens * L * _LAYER + 4.0 * attended * DQ * L + 2.0 * heads * VOCAB * D


def _decode_work(batch, context, steps):
    weights = decode_bytes_per_token(0) - _KV_ROW - 2 * D
    attended = sum(context + s + 1 for s in range(steps))
    nbytes = steps * (weights + batch * (_KV_ROW + 2 * D)) + batch * (attended - steps) * _KV_ROW
    return nbytes, _language_flops(batch * steps, batch * attended, batch * steps)


def _causal(n):
    return n * (n + 1) // 2


def work(case):
    path = case["path"]
    layers = 2 * L * _LAYER
    if path == "images":
        d, _, mlp, n_layers, patch, side, patches = TOWERS[case["tower"]]
        counts = [patches] * case["images"] if side else [h * w for h, w in _grids(case["images"])]
        weights = n_layers * (4 * d * d + 2 * d * mlp) + 3 * patch * patch * d + 4 * d * d + 2 * d * mlp
        flops = sum(n_layers * (2 * s * d * (4 * d + 2 * mlp) + 4 * s * s * d) + 2 * s * d * (3 * patch * patch + 2 * d) + 4 * s * d
                    + 2 * d * d + 4 * d * mlp for s in counts)
        pixels = case["images"] * 3 * side * side if side else sum(counts) * 3 * patch * patch
        return {"bytes": 2 * weights + 4 * pixels + 2 * case["images"] * d, "flops": flops}
    if path == "embed":
        lengths = _lengths(case["sequences"], case["shortest"], case["longest"])
        return {"bytes": layers + sum(lengths) * 2 * D + len(lengths) * 4 * D,
                "flops": _language_flops(sum(lengths), sum(map(_causal, lengths)), 0)}
    if path == "decode":
        nbytes, flops = _decode_work(case["batch"], case["context"], case["steps"])
        return {"bytes": nbytes, "flops": flops}
    if path == "serve":
        lengths = _lengths(case["requests"], case["shortest"], case["longest"])
        answers = _lengths(case["requests"] + 1, max(1, case["answer"] // 4), case["answer"])[1:]
        # weights once for a prompt's rows, and once per step of the slots that decode together
        flops = _language_flops(sum(lengths) + sum(answers), sum(_causal(n + a) for n, a in zip(lengths, answers)), sum(answers))
        steps = max(max(answers), math.ceil(sum(answers) / case["slots"]))
        read = sum(a * n + _causal(a) for n, a in zip(lengths, answers)) * _KV_ROW
        return {"bytes": steps * (layers + 2 * VOCAB * D) + read + (sum(lengths) + sum(answers)) * (_KV_ROW + 2 * D), "flops": flops}
    batch, n = case.get("batch", 1), case["prompt"]
    nbytes = layers + 2 * VOCAB * D + batch * n * (_KV_ROW + 2 * D)
    flops = _language_flops(batch * n, batch * _causal(n), batch)
    if path == "generate" and case["steps"] > 1:
        more = _decode_work(1, n, case["steps"] - 1)
        nbytes, flops = nbytes + more[0], flops + more[1]
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """One bf16 rounding is off by up to 2^-9 and by 1.1e-3 on average (rms).  A layer of the language model has about eight
    of them in a row, each of the size of the residual stream or of a good part of it: over 28 layers sqrt(28 * 8) * 1.1e-3
    = 1.7e-2 for one order of rounding and sums, sqrt(2) times that between two of them (the package's own settings, norms
    folded into the projections or not, are 1.8e-2 apart).  The towers' pooled rows pass through a normalisation and a mean
    over the patches, which leaves the usual 1e-2.  Generated ids are the same but for ties."""
    return {"rel": 1e-2} if case["path"] == "images" else {"rel": 2.4e-2, "differ": 0.005}
