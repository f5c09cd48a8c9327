"""Blocks in one native call against the same block module by module: the same kernels in the same order, so the same numbers, but for
gradients that join another one before they are rounded."""

import gc

import pytest
import torch

from triune_b200.models import TransformerBlock, native_block
from triune_b200.models.universal import UniversalBlock
from triune_b200.config import ModelConfig
from triune_b200.utils import place_model

pytestmark = pytest.mark.gpu


def _block(dim, heads, head_dim, delta, learn_beta=True, seed=0):
    torch.manual_seed(seed)
    m = TransformerBlock(dim, heads, 0, 1000, [], use_moe=False, head_dim=head_dim, use_delta_rule=delta, learn_beta=delta and learn_beta)
    m = place_model(m, torch.device("cuda"), torch.bfloat16)
    with torch.no_grad():
        for p in m.parameters():
            if p.dim() == 1:
                p.add_(torch.randn_like(p) * 0.1)
    return m


def _modules(monkeypatch, call):
    with monkeypatch.context() as mp:
        mp.setattr(native_block, "run", lambda *a: None)
        return call()


@pytest.mark.parametrize("delta,learn_beta", [(False, False), (True, True), (True, False)])
@pytest.mark.parametrize("batch,seq,dim,heads,head_dim", [(2, 2, 128, 2, 64), (3, 63, 256, 2, 128), (2, 64, 384, 6, 64), (1, 333, 512, 4, 128)])
def test_training_pass(batch, seq, dim, heads, head_dim, delta, learn_beta, monkeypatch):
    m = _block(dim, heads, head_dim, delta, learn_beta).train()
    x = torch.randn(batch, seq, dim, device="cuda").bfloat16().requires_grad_(True)
    dy = torch.randn_like(x)
    names, params = zip(*m.named_parameters())

    def step():
        y, _, cache = m(x)
        assert cache is None
        return y, torch.autograd.grad(y, (x, *params), dy)

    y, grads = step()
    assert type(y.grad_fn).__name__ == "_BlockFnBackward"
    want, want_grads = _modules(monkeypatch, step)
    assert torch.equal(y, want)
    for n, a, b in zip(("x", *names), grads, want_grads):
        assert a.dtype == b.dtype and a.shape == b.shape
        # gradients of x, and of what is read through the sum with the strengths' gradient, are rounded once less
        assert torch.equal(a, b) if n != "x" and not n.startswith("norm1") else (a - b).norm() <= 2 ** -7 * b.norm(), n


@pytest.mark.parametrize("delta", [False, True])
@pytest.mark.parametrize("frozen", ["", "x", "ffn", "norm1"])
def test_two_functions_give_the_numbers_of_one(delta, frozen, monkeypatch):
    m = _block(256, 4, 64, delta).train()
    x = torch.randn(2, 100, 256, device="cuda").bfloat16().requires_grad_(frozen != "x")
    dy = torch.randn_like(x)
    for n, p in m.named_parameters():
        p.requires_grad_(not frozen or not n.startswith(frozen))
    wanted = [t for t in (x, *m.parameters()) if t.requires_grad]
    y = m(x)[0]
    assert type(y.grad_fn).__name__ == "_BlockFnBackward"
    grads = torch.autograd.grad(y, wanted, dy)
    monkeypatch.setattr(native_block, "ONE_FUNCTION", 0)
    z = m(x)[0]
    assert type(z.grad_fn).__name__ == "_BlockRestFnBackward" and torch.equal(y, z)
    for a, b in zip(torch.autograd.grad(z, wanted, dy), grads):
        assert torch.equal(a, b) if not delta else (a - b).norm() <= 2 ** -7 * b.norm()  # strengths' gradients are summed up in any order


@pytest.mark.parametrize("delta", [False, True])
@pytest.mark.parametrize("train", [False, True])
def test_memory_is_that_of_the_modules(train, delta, monkeypatch):
    m = _block(512, 8, 64, delta).train(train)
    x = torch.randn(2, 4096, 512, device="cuda").bfloat16().requires_grad_(train)
    dy = torch.randn_like(x)

    def peak():
        def call():
            if train:
                return torch.autograd.grad(m(x)[0], (x, *m.parameters()), dy)
            with torch.no_grad():
                return m(x, cache=(None, 0))

        call()  # tables and workspaces that stay
        gc.collect()  # what other tests left is not given back meanwhile, and blocks' roundings do not count
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_stats()["requested_bytes.all.current"]
        gc.disable()
        call()
        gc.enable()
        return torch.cuda.memory_stats()["requested_bytes.all.peak"] - before

    native, modules = peak(), _modules(monkeypatch, peak)
    assert native <= 1.01 * modules


def test_a_block_s_output_may_be_written_into():
    m = _block(128, 2, 64, False).train()
    x = torch.randn(2, 70, 128, device="cuda").bfloat16().requires_grad_(True)
    y = m(x)[0]
    (plain,) = torch.autograd.grad((2 * y).float().sum(), x, retain_graph=True)
    y.mul_(2)
    (got,) = torch.autograd.grad(y.float().sum(), x)
    assert torch.equal(got, plain)


def test_gradients_added_into_buffers_and_frozen_parameters(monkeypatch):
    m = _block(256, 4, 64, True).train()
    x = torch.randn(2, 130, 256, device="cuda").bfloat16()
    frozen = {"norm2.weight", "ffn.0.weight", "attn.gla.out_proj.weight", "ffn.2.bias"}
    for n, p in m.named_parameters():
        p.requires_grad_(n not in frozen)

    def step():
        for n, p in m.named_parameters():
            p.grad = None
            if not n.endswith("beta_proj.weight") and n not in frozen:
                p.main_grad = torch.ones(p.shape, device="cuda")
        m(x)[0].float().square().mean().backward()
        return {n: (p.main_grad if hasattr(p, "main_grad") else p.grad) for n, p in m.named_parameters()}

    got, want = step(), _modules(monkeypatch, step)
    for n in want:
        assert (got[n] is None) == (want[n] is None) == (n in frozen), n
        if want[n] is not None:
            assert (got[n] - want[n]).norm() <= 2 ** -7 * (want[n] - (0 if n.endswith("beta_proj.weight") else 1)).norm() + 1e-5 * want[n].norm(), n


@pytest.mark.parametrize("delta", [False, True])
@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("batch,seq,fmt", [(1, 2, "tuple"), (2, 37, "dict"), (1, 200, "tensor"), (2, 64, "none"), (3, 16, "fresh")])
def test_prompt_with_and_without_a_state(batch, seq, fmt, gated, delta, monkeypatch):
    if gated:
        cfg = ModelConfig(family="universal", vocab_size=64, hidden_dim=256, num_layers=1, num_heads=2, head_dim=128, ffn="swiglu", dense_hidden=320,
                          mixer="gated_deltanet" if delta else "gla").validate()
        m = place_model(UniversalBlock(cfg, 0), torch.device("cuda"), torch.bfloat16).eval()
    else:
        m = _block(256, 2, 128, delta).eval()
    x, s0 = torch.randn(batch, seq, 256, device="cuda").bfloat16(), torch.randn(batch, 2, 128, 128, device="cuda")
    cache = {"tuple": (s0, 5), "dict": {"state": s0, "offset": 9}, "tensor": s0, "none": None, "fresh": (None, 0)}[fmt]
    kept, calls = s0.clone(), []
    inner = native_block.run

    def call():
        with torch.no_grad():
            out = m(x, cache=cache)
        return out[0], out[-1]

    monkeypatch.setattr(native_block, "run", lambda *a: calls.append(inner(*a) is not None) or inner(*a))
    y, after = call()
    assert calls == [True] and torch.equal(s0, kept)
    want, want_after = _modules(monkeypatch, call)
    assert torch.equal(y, want) and type(after) is type(want_after)
    state = {"tuple": lambda c: c[0], "fresh": lambda c: c[0], "dict": lambda c: c["state"], "tensor": lambda c: c, "none": lambda c: None}[fmt]
    if fmt != "none":
        assert torch.equal(state(after), state(want_after))
    if fmt == "tuple":
        assert after[1] == want_after[1] == 5 + seq
    if fmt == "dict":
        assert after["offset"] == want_after["offset"] == 9 + seq


@pytest.mark.parametrize("change", ["hook", "global hook", "backward hook", "forward", "bias", "module", "another module", "lora", "float32", "strided", "one token", "tangent"])
def test_other_blocks_run_module_by_module(change):
    m, handle = _block(128, 2, 64, False).eval(), None
    x = torch.randn(2, 8, 128, device="cuda").bfloat16()
    if change == "hook":
        m.ffn[1].register_forward_hook(lambda *a: None)
    elif change == "global hook":
        handle = torch.nn.modules.module.register_module_forward_hook(lambda *a: None)
    elif change == "backward hook":
        m.norm1.register_full_backward_hook(lambda *a: None)
    elif change == "forward":
        m.attn.gla.out_proj.forward = lambda t: t
    elif change == "bias":
        m.attn.gla.out_proj.bias = torch.nn.Parameter(torch.zeros(128, device="cuda", dtype=torch.bfloat16))
    elif change == "module":
        m.ffn[0] = torch.nn.Sequential(m.ffn[0])
    elif change == "another module":
        m.ffn.append(torch.nn.Identity())
    elif change == "lora":
        m.attn.gla.qkvg_lora = lambda t: t
    elif change == "float32":
        m, x = m.float(), x.float()
    elif change == "strided":
        x = x.transpose(0, 1)
    elif change == "one token":
        x = x[:, :1].contiguous()
    try:
        with torch.no_grad():
            if change == "tangent":
                with torch.autograd.forward_ad.dual_level():
                    got = native_block.run(m.norm1, m.attn, m.norm2, m.ffn, x, None)
            else:
                got = native_block.run(m.norm1, m.attn, m.norm2, m.ffn, x, None)
        assert got is None
    finally:
        if handle is not None:
            handle.remove()


@pytest.mark.parametrize("module,name", [(torch.jit, "is_tracing"), (torch.compiler, "is_compiling")])
def test_traced_and_compiled_calls_run_module_by_module(module, name, monkeypatch):
    m = _block(128, 2, 64, False).eval()
    x = torch.randn(2, 8, 128, device="cuda").bfloat16()
    with torch.no_grad():
        assert native_block.run(m.norm1, m.attn, m.norm2, m.ffn, x, None) is not None
        monkeypatch.setattr(module, name, lambda: True)
        assert native_block.run(m.norm1, m.attn, m.norm2, m.ffn, x, None) is None
