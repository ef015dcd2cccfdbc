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
