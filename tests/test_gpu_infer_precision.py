"""Precision of the sampling path: forward_infer keeps the residual stream's low half and returns fp32 accumulators."""
import math

import pytest
import torch

from helpers import make_config, single_world

pytestmark = pytest.mark.gpu


def _reference(eng, ids, layers, heads):
    """The model in fp64 on the weights as the GEMMs read them (matrices rounded to bf16)."""
    w = lambda k, gemm=False: eng.p32(k).to(torch.bfloat16).double() if gemm else eng.p32(k).double()
    B, T = ids.shape
    x = w("transformer.wte.weight")[ids] + w("transformer.wpe.weight")[:T]
    d = x.shape[-1]
    norm = lambda x, p: torch.nn.functional.layer_norm(x, (d,), w(p + ".weight"), w(p + ".bias"), 1e-5)
    lin = lambda x, p: x @ w(p + ".weight", True).T + w(p + ".bias")
    future = torch.ones(T, T, dtype=torch.bool, device=ids.device).triu(1)
    for l in range(layers):
        p = f"transformer.h.{l}."
        q, k, v = (t.view(B, T, heads, -1).transpose(1, 2) for t in lin(norm(x, p + "ln_1"), p + "attn.c_attn").split(d, dim=2))
        a = (q @ k.transpose(2, 3) / math.sqrt(d // heads)).masked_fill(future, -math.inf).softmax(-1) @ v
        x = x + lin(a.transpose(1, 2).reshape(B, T, d), p + "attn.c_proj")
        x = x + lin(torch.nn.functional.gelu(lin(norm(x, p + "ln_2"), p + "mlp.c_fc")), p + "mlp.c_proj")
    return norm(x, "transformer.ln_f") @ w("lm_head.weight", True).T


@pytest.mark.parametrize("B,T", [(5, 24), (8, 250)])               # the kernel for few rows, those for many
def test_the_residual_stream_is_not_rounded_to_bf16(B, T):
    """Rounding a bf16 residual stream at each of its 2 * layers additions alone costs 1.1e-3 of it a time (a uniform
    error of half a unit of the eighth bit), adding up in squares to sqrt(24) * 1.1e-3 = 5.4e-3 of the logits with 12
    layers, next to the roundings of everything else.  The whole error has to stay below that."""
    from diloco_swarm_b200.models.engine_b200 import B200Engine
    from diloco_swarm_b200.models.gpt2 import GPT2Config
    layers, heads = 12, 12
    shape = dict(n_layer=layers, n_head=heads, n_embd=768, vocab_size=512, block_size=256)
    eng = B200Engine(GPT2Config(**shape), single_world(), make_config(model=shape), torch.device("cuda", 0))
    gen = torch.Generator(device="cuda").manual_seed(7)
    ids = torch.randint(0, 500, (B, T), generator=gen, device="cuda")
    with torch.no_grad():
        ref = _reference(eng, ids, layers, heads)
        out = eng.forward_infer(ids, None).double()
    eng.check_status()
    assert ((out - ref).norm() / ref.norm()).item() < 1.1e-3 * math.sqrt(2 * layers)
