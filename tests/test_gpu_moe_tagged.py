"""The mixture-of-experts layer without grid barriers (rows, router logits, activations and the layer's sum travel as
tagged words; the activation sits in the gate/up linear's epilogue) against the same program with a barrier before
every op: the order of every sum is the same, so tokens and logits are bit-identical."""
import functools

import pytest
import torch

import fleet_chiplet_megakernel_b200 as mk
from fleet_chiplet_megakernel_b200 import qwen3_moe_graph
from oracle import qwen3_oracle as O

pytestmark = pytest.mark.gpu


def _generate(monkeypatch, g, w, prompts, n_new, debug_flags):
    geom = mk.Qwen3MoeGeometry(hidden=g.hidden, n_q=g.n_q, n_kv=g.n_kv, head_dim=g.head_dim, experts=g.experts, top_k=g.top_k,
                               moe_mlp=g.moe_mlp, layers=g.layers, vocab=g.vocab, rope_theta=g.rope_theta)
    with monkeypatch.context() as m:
        m.setattr(qwen3_moe_graph, "PersistentKernel", functools.partial(mk.PersistentKernel, debug_flags=debug_flags))
        dec = mk.Qwen3MoeDecoder(geom, {k: v.cuda() for k, v in w.items()}, max_seq_length=max(map(len, prompts)) + n_new,
                                 max_requests=len(prompts), page_size=16, keep_logits=True)
    dec.set_prompts(prompts)
    dec.run()
    out = [dec.generated(r).cpu() for r in range(len(prompts))], dec.logits.cpu(), dec.mpk.describe()
    dec.finalize()
    return out


# experts and slots: pairs of 8 units per CTA and more; expert widths that leave ragged chunks (200 = 25 units of 8) and a
# padded k (200 of 512); the last two keep their barriers: a router of 254 rows is not whole 8-row units, and two slots of
# 144 rows are fewer units than CTAs at one token
@pytest.mark.parametrize("experts,top_k,inter,requests,tagged", [
    (16, 4, 256, 1, True), (16, 4, 256, 2, True), (64, 8, 200, 1, True), (248, 3, 768, 2, True), (254, 3, 768, 1, False), (10, 2, 72, 2, False)])
def test_tagged_moe_layer_gives_the_bits_the_barriers_give(monkeypatch, experts, top_k, inter, requests, tagged):
    g = O.MoeGeometry(hidden=512, n_q=8, n_kv=2, experts=experts, top_k=top_k, moe_mlp=inter, layers=3, vocab=2048)
    w = O.make_moe_weights(g, 5, norm_jitter=0.1)
    prompts = [O.make_prompt(O.Geometry(vocab=g.vocab), 9 - 4 * r, r) for r in range(requests)]
    toks, logits, ops = _generate(monkeypatch, g, w, prompts, 14, 0)
    ref_toks, ref_logits, _ = _generate(monkeypatch, g, w, prompts, 14, 16)
    assert all(torch.equal(a, b) for a, b in zip(toks, ref_toks))
    assert torch.equal(logits, ref_logits)
    flags = [int(f.split("flags=")[1].split()[0], 16) for f in ops.strip().splitlines() if f.split()[1] == "moe_linear"]
    assert all(bool(f & (1 << 19)) == tagged for f in flags)  # input rows read from tagged words
