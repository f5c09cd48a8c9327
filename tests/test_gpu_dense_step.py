"""The one-launch decoding step against the step of the model's modules: the same tokens, states and positions, bit for bit."""

import threading

import pytest
import torch

from triune_b200.config import ModelConfig
from triune_b200.inference import GraphedGreedyDecoder
from triune_b200.models.factory import build_model
from triune_b200.runtime import dense_step
from triune_b200.utils import place_model

pytestmark = pytest.mark.gpu


def _model(dim, heads, head_dim, layers, hidden, vocab, mixer, ffn="swiglu", scale="none", seed=0):
    cfg = ModelConfig(family="universal", vocab_size=vocab, hidden_dim=dim, num_layers=layers, num_heads=heads, head_dim=head_dim, mixer=mixer,
                      ffn=ffn, dense_hidden=hidden, tie_embeddings=False, gla_scale=scale).validate()
    torch.manual_seed(seed)
    m = place_model(build_model(cfg), torch.device("cuda"), torch.bfloat16).eval()
    with torch.no_grad():
        for p in m.parameters():  # norms and biases that matter, logits without ties
            if p.dim() == 1:
                p.add_(torch.randn_like(p) * 0.1)
        m.embed_tokens.weight.normal_()
        m.lm_head.weight.normal_(0, 0.2)
    return m


def _both(m, batch, prompt, new, monkeypatch):
    ids = torch.randint(0, m.vocab_size, (batch, prompt), device="cuda", generator=torch.Generator("cuda").manual_seed(prompt))
    one = GraphedGreedyDecoder(m, batch_size=batch)
    got = one.generate(ids, new)
    with monkeypatch.context() as mp:
        mp.setattr(dense_step, "plan", lambda *a: None)
        captured = GraphedGreedyDecoder(m, batch_size=batch)
        want = captured.generate(ids, new)
    assert isinstance(captured.graph, torch.cuda.CUDAGraph)
    return one, got, captured, want


@pytest.mark.parametrize("mixer", ["gla", "gated_deltanet"])
@pytest.mark.parametrize("batch,dim,heads,head_dim,hidden,vocab", [
    (1, 128, 2, 64, 256, 64),        # fewer blocks than CTAs
    (3, 384, 6, 64, 1088, 1000),     # slices of different widths
    (8, 512, 8, 64, 1408, 4104),     # all rows of the matrix instruction
    (2, 1024, 8, 128, 2816, 5000),
    (5, 1536, 12, 128, 4224, 3208),  # whole heads per mixer unit
    (4, 2048, 16, 128, 5632, 32000),
    (1, 2048, 16, 128, 5632, 32000),
])
def test_step_gives_the_numbers_of_the_modules(mixer, batch, dim, heads, head_dim, hidden, vocab, monkeypatch):
    m = _model(dim, heads, head_dim, 2, hidden, vocab, mixer)
    one, got, captured, want = _both(m, batch, 9, 12, monkeypatch)
    assert isinstance(one.graph, dense_step.Step)
    assert torch.equal(got, want) and int(one.pos) == int(captured.pos) and torch.equal(one.token, captured.token)
    for a, b in zip(one.states, captured.states):
        assert torch.equal(a, b)
    assert int(one.graph.native.status) == 0


@pytest.mark.parametrize("batch,dim,heads,hidden,vocab", [(1, 128, 2, 128, 64), (4, 128, 2, 256, 300), (2, 256, 4, 128, 64)])
def test_ctas_without_blocks_leave_no_copies_behind(batch, dim, heads, hidden, vocab, monkeypatch):
    # 8 to 64 blocks a phase: which CTAs have one changes from phase to phase, and no norm's weights are like another's
    m = _model(dim, heads, 64, 6, hidden, vocab, "gated_deltanet")
    norms = [n for layer in m.layers for n in (layer.input_norm, layer.post_attn_norm)] + [m.norm]
    with torch.no_grad():
        for i, n in enumerate(norms):
            n.weight.copy_(torch.randn(dim, device="cuda") * 2.0 ** (i % 5 - 2))
    one, got, captured, want = _both(m, batch, 9, 24, monkeypatch)
    assert isinstance(one.graph, dense_step.Step) and torch.equal(got, want)
    for a, b in zip(one.states, captured.states):
        assert torch.equal(a, b)


@pytest.mark.parametrize("ffn,scale,vocab", [("gelu", "none", 512), ("gelu", "fla", 512), ("swiglu", "fla", 517)])
def test_step_with_biases_scales_and_ragged_vocabularies(ffn, scale, vocab, monkeypatch):
    m = _model(256, 4, 64, 3, 320, vocab, "gla", ffn, scale)
    one, got, captured, want = _both(m, 2, 21, 10, monkeypatch)
    assert isinstance(one.graph, dense_step.Step) and torch.equal(got, want)
    for a, b in zip(one.states, captured.states):
        assert torch.equal(a, b)


def test_second_request_longer_outputs_and_other_tables(monkeypatch):
    m = _model(128, 2, 64, 2, 256, 512, "gated_deltanet")
    one = GraphedGreedyDecoder(m)
    for prompt, new in ((5, 3), (7, 40), (70, 20)):
        ids = torch.randint(0, 512, (1, prompt), device="cuda")
        with monkeypatch.context() as mp:
            mp.setattr(dense_step, "plan", lambda *a: None)
            want = GraphedGreedyDecoder(m).generate(ids, new)
        assert torch.equal(one.generate(ids, new), want) and torch.equal(one.generate(ids, new), want)


@pytest.mark.parametrize("change", ["hook", "global hook", "forward", "bias", "nine rows", "float32"])
def test_other_models_keep_the_captured_step(change):
    m = _model(128, 2, 64, 2, 256, 512, "gla")
    batch, handle = 1, None
    if change == "hook":
        handle = m.layers[1].mlp.register_forward_hook(lambda mod, a, out: out * 0)
    elif change == "global hook":
        handle = torch.nn.modules.module.register_module_forward_hook(lambda mod, a, out: None)
    elif change == "forward":
        m.norm.forward = lambda x: x
    elif change == "bias":
        m.layers[0].attn.out_proj.bias = torch.nn.Parameter(torch.ones(128, device="cuda", dtype=torch.bfloat16))
    elif change == "nine rows":
        batch = 9
    elif change == "float32":
        m = m.float()
    try:
        dec = GraphedGreedyDecoder(m, batch_size=batch)
        dec.generate(torch.randint(0, 512, (batch, 5), device="cuda"), 3)
        assert isinstance(dec.graph, torch.cuda.CUDAGraph)
    finally:
        if handle is not None:
            handle.remove()


@pytest.mark.parametrize("how", ["status", "wait"])
def test_a_step_that_did_not_finish_raises_and_the_next_prompt_starts_over(how):
    m = _model(128, 2, 64, 2, 256, 512, "gla")
    ids = torch.randint(0, 512, (1, 9), device="cuda")
    dec = GraphedGreedyDecoder(m)
    want = dec.generate(ids, 6)
    first = dec.graph
    assert isinstance(first, dense_step.Step)
    if how == "status":
        first.status.fill_(4)
    else:  # nobody forms the first projection, so that the mixer's wait for it runs out after its second
        entry = first.native.program.view(torch.int32).view(-1, 40)[0]
        assert entry[16:19].tolist() == [0, 4 * 128, 128] and entry[26:29].tolist() == [32, 0, 32]
        entry[26:29] = 0
    with pytest.raises(RuntimeError, match="did not finish"):
        dec.generate(ids, 6)
    assert int(first.status) != 0
    with pytest.raises(RuntimeError, match="prefill"):
        dec.decode(3)
    assert torch.equal(dec.generate(ids, 6), want)
    assert dec.graph is not first and int(dec.graph.status) == 0


def test_steps_may_be_captured():
    m = _model(128, 2, 64, 2, 256, 512, "gla")
    ids = torch.randint(0, 512, (1, 9), device="cuda")
    dec = GraphedGreedyDecoder(m)
    want = dec.generate(ids, 6)[:, 9:]
    dec.prefill(ids)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = dec.decode(6)
    graph.replay()
    assert torch.equal(got, want)


def test_two_decoders_on_two_streams_take_turns():
    models = [_model(256, 4, 64, 3, 320, 512, "gla"), _model(384, 6, 64, 4, 1088, 1000, "gated_deltanet")]
    prompts = [torch.randint(0, 500, (b, 33), device="cuda") for b in (1, 2)]
    decoders = [GraphedGreedyDecoder(m, batch_size=p.shape[0]) for m, p in zip(models, prompts)]
    want = [d.generate(p, 40) for d, p in zip(decoders, prompts)]
    torch.cuda.synchronize()
    same = [[], []]

    def serve(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(8):
                same[i].append(torch.equal(decoders[i].generate(prompts[i], 40), want[i]))

    threads = [threading.Thread(target=serve, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert same == [[True] * 8] * 2
