"""Kernels that a layer's forward, backward or decoding step takes at particular sizes, at the borders of those sizes."""

import pytest
import torch
import torch.nn.functional as F

from triune_b200.ops import gla_cuda
from triune_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm()).item()


def _gate_error(got, dg, q, k, dq, dk, end, slope):
    """Error of a gate gradient in units of what rounding gives: the gradient is the sum over the later tokens of q dq - k dk and of the
    final state's term, each formed with a relative error of about 2^-8, and independent errors add as their squares do."""
    terms = ((q * dq) ** 2 + (k * dk) ** 2).flip(1).cumsum(1).flip(1) + end.unsqueeze(1) ** 2
    return ((got.double() - dg).norm() / (2.0 ** -8 * (terms.sqrt() * slope).norm())).item()


def _mixer_inputs(B, T, H, D, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    q, k = (F.normalize(F.elu(rnd(B, T, H, D)) + 1, dim=-1).bfloat16() for _ in range(2))
    return q, k, rnd(B, T, H, D).bfloat16(), rnd(B, T, H, D).bfloat16(), rnd(B, H, D, D)


@pytest.mark.parametrize("B,T,H,D,beta_dims", [
    (1, 7, 2, 64, 1), (1, 8, 1, 64, 0), (2, 9, 3, 64, 1), (1, 15, 1, 128, 0), (2, 16, 2, 128, 2), (3, 65, 2, 64, 2), (1, 131, 2, 128, 1),
    (8, 500, 8, 128, 1),  # 64 heads: more tokens than one segment of records
    (1, 11, 2, 64, 1), (1, 12, 2, 64, 1), (2, 8, 8, 128, 1), (2, 8, 9, 128, 1), (4, 47, 96, 64, 1), (4, 48, 96, 64, 1),  # ends of the rule
    (7, 64, 64, 64, 0), (7, 64, 65, 64, 0), (2, 512, 256, 64, 1), (3, 512, 171, 64, 1),
])
def test_delta_rule_prompts_against_the_token_recurrence(B, T, H, D, beta_dims):
    q, k, v, g, s0 = _mixer_inputs(B, T, H, D)
    beta = None if beta_dims == 0 else torch.rand(B, T, H, *([D] if beta_dims == 2 else []), device="cuda")
    o, s = gla_cuda.gdn_recurrent(q, k, v, g, beta, s0, 0.7, True)
    gl = F.logsigmoid(g.double()).clamp(min=gla_cuda.GLA_MIN_LOG_DECAY)
    oo, ss = ref.gated_deltanet_recurrent(q.double(), k.double(), v.double(), gl, None if beta is None else beta.double(), s0.double(), 0.7)
    assert _rel(o, oo) < 2.0 ** -8   # outputs are rounded to bf16: at most 2^-9 each
    assert _rel(s, ss) < 1e-6        # the state is fp32 throughout


@pytest.mark.parametrize("B,T,H,D,beta_dims", [
    (1, 8, 16, 128, 1), (1, 17, 5, 128, 2), (1, 31, 3, 64, 0), (2, 33, 7, 64, 1),          # blocks of sixteen and their remainders
    (4, 12, 16, 64, 1), (4, 11, 16, 128, 1), (4, 12, 16, 128, 0), (8, 24, 16, 64, 1), (8, 23, 16, 128, 1), (8, 24, 16, 128, 2),
    (17, 31, 8, 64, 1), (17, 32, 8, 64, 1), (32, 32, 16, 128, 1), (27, 140, 19, 128, 1), (19, 140, 27, 64, 1),  # ends of the rule, segments
    (8, 25, 16, 128, 1), (8, 26, 16, 128, 1), (16, 32, 16, 64, 1), (385, 32, 1, 64, 1),
])
def test_rounds_of_sixteen_tokens_against_the_token_recurrence(B, T, H, D, beta_dims):
    test_delta_rule_prompts_against_the_token_recurrence(B, T, H, D, beta_dims)


@pytest.mark.parametrize("logits", [0.0, 4.0, 8.0, 10.0, 14.0])
@pytest.mark.parametrize("T,H,D", [(2048, 6, 64), (2048, 4, 128), (509, 3, 64)])
def test_delta_rule_prompts_lose_no_bits_of_a_long_memory(T, H, D, logits):
    """Gates near 1 keep thousands of tokens, so that an error to one side in each of them adds up. Pieces of four tokens take the kernel that
    goes token by token in fp32; a prompt's state may be off by as much as that one's, or by two roundings (2^-23)."""
    q, k, v, g, _ = _mixer_inputs(1, T, H, D)
    g = (g.float() + logits).bfloat16()
    beta = torch.sigmoid(torch.randn(1, T, H, device="cuda", generator=torch.Generator("cuda").manual_seed(T)))
    _, s = gla_cuda.gdn_recurrent(q, k, v, g, beta, None, 1.0, True)
    st = None
    for t in range(0, T, 4):
        _, st = gla_cuda.gdn_recurrent(*(x[:, t : t + 4] for x in (q, k, v, g, beta)), st, 1.0, True)
    gl = F.logsigmoid(g.double()).clamp(min=gla_cuda.GLA_MIN_LOG_DECAY)
    _, exact = ref.gated_deltanet_recurrent(q.double(), k.double(), v.double(), gl, beta.double(), torch.zeros(1, H, D, D, device="cuda").double(), 1.0)
    assert _rel(s, exact) < 1.5 * _rel(st, exact) + 2.0 ** -23


@pytest.mark.parametrize("E,K,N,D,skew", [(8, 2, 1, 64, 0.0), (8, 1, 257, 72, 4.0), (16, 2, 1000, 384, 0.0), (64, 4, 300, 128, 6.0), (8, 2, 4096, 1536, 3.0)])
def test_routing_statistics_in_one_kernel(E, K, N, D, skew, monkeypatch):
    from triune_b200.models import MoE_FFN

    def run(native):
        torch.manual_seed(E + N)
        m = MoE_FFN(D, num_experts=E, top_k=K, expert_hidden=64).cuda().bfloat16()
        for name in ("expert_bias", "expert_load_ratio", "last_centroids"):
            setattr(m, name, getattr(m, name).float())
        m.expert_bias[0] += skew  # tokens beyond the capacity are dropped
        m.train()
        out = []
        with monkeypatch.context() as mp:
            if not native:
                mp.setattr(MoE_FFN, "_stats_on_kernels", lambda *a: False)
            for step in range(3):  # no centroids yet, then running ones
                m._global_step.fill_(step * 700)
                with torch.no_grad():
                    m(torch.randn(1, N, D, device="cuda", generator=torch.Generator("cuda").manual_seed(step)).bfloat16())
                out.append([t.clone() for t in (m.last_counts, m.last_accepted_counts, m.last_dropped_counts, m._overflow_counter, m._pending_bias_update,
                                                m.expert_load_ratio, m.last_centroids)])
                m.step_bias()
        return out

    got, want = run(True), run(False)
    for g, w in zip(got, want):
        for n in range(4):
            assert g[n].dtype == w[n].dtype and g[n].shape == w[n].shape and torch.equal(g[n], w[n]), n
        for n in (4, 5, 6):  # fp32, a few operations in another order
            assert g[n].shape == w[n].shape and (g[n] - w[n]).abs().max() <= 2.0 ** -20 * max(1.0, float(w[n].abs().max())), n
    assert skew == 0.0 or int(want[-1][3]) > 0


@pytest.mark.parametrize("step", [0, 1, 12345, 10 ** 9])
def test_router_temperature_at_a_step(step):
    from triune_b200.models.moe import MOE_TEMPERATURE_STEPS
    from triune_b200 import _ext

    s = torch.tensor(step, device="cuda")
    want = (1.0 - s.float() / MOE_TEMPERATURE_STEPS).clamp(min=0.1)
    got = _ext.ext().moe_temperature(s, float(MOE_TEMPERATURE_STEPS), 0.1)
    assert got.shape == want.shape and abs(float(got) - float(want)) <= 2.0 ** -22


@pytest.mark.parametrize("chunks", [1, 2, 7, 8, 9, 15, 16, 17, 33])
@pytest.mark.parametrize("D", [64, 128])
def test_state_scan_over_batches_of_chunks(chunks, D):
    from triune_b200 import ops

    q, k, v, g, s0 = _mixer_inputs(1, 64 * chunks, 2, D)
    odd = torch.empty(s0.numel() + 1, device="cuda")[1:].view_as(s0).copy_(s0)  # a state that starts on any number
    x = [t.requires_grad_(True) for t in (q, k, v, g, odd)]
    o, s = ops.gla(*x[:4], initial_state=x[4], gate_logits=True)
    w, ws = torch.randn_like(o), torch.randn_like(s)
    grads = torch.autograd.grad((o * w).sum() + (s * ws).sum(), x)
    y = [t.detach().double().requires_grad_(True) for t in x]
    gl = F.logsigmoid(y[3]).clamp(min=gla_cuda.GLA_MIN_LOG_DECAY)
    S, rows = y[4], []
    for c in range(64 * chunks):
        S = S * gl[:, c].exp().unsqueeze(-1) + y[1][:, c].unsqueeze(-1) * y[2][:, c].unsqueeze(-2)
        rows.append((y[0][:, c].unsqueeze(-2) @ S).squeeze(-2))
    oo = torch.stack(rows, 1)
    want = torch.autograd.grad((oo * w.double()).sum() + (S * ws.double()).sum(), y)
    # states between chunks and chunk operands are bf16: a relative error of 2^-8 for each of a handful of roundings
    assert _rel(o, oo) < 2.0 ** -6 and _rel(s, S) < 2.0 ** -6
    # a gate's gradient is a sum of terms that nearly cancel: its bound follows from their sizes (_gate_error)
    z = [t.detach() for t in y]
    assert _gate_error(grads[3], want[3], z[0], z[1], want[0], want[1], (ws.double() * S.detach()).sum(-1), torch.sigmoid(-z[3])) < 1
    for n in (0, 1, 2, 4):
        assert _rel(grads[n], want[n]) < 2.0 ** -5, n


@pytest.mark.parametrize("B,T,H,D", [(1, 1, 1, 64), (2, 37, 3, 64), (1, 4736, 1, 64), (1, 4737, 2, 64), (3, 17, 5, 128), (1, 1579, 3, 128), (5, 1000, 7, 128)])
@pytest.mark.parametrize("rope", [False, True])
def test_feature_map_of_few_and_many_tokens(B, T, H, D, rope):
    from triune_b200 import ops

    qkvg = torch.randn(B * T, 4 * H * D, device="cuda", generator=torch.Generator("cuda").manual_seed(T)).bfloat16()
    cos, sin = ops.rope_tables(T, D, 10000.0, 0, "cuda") if rope else (None, None)
    got = ops.qk_feature_map(qkvg, cos, sin, B, T, H, D)
    for n, t in enumerate(got[:2]):
        f = F.normalize(F.elu(qkvg[:, n * H * D : (n + 1) * H * D].reshape(B, T, H, D).double()) + 1.0, dim=-1, eps=1e-6)
        if rope:
            f = ref.apply_rope(f, cos.double(), sin.double())
        assert (t.double() - f).abs().max() <= 2.0 ** -8 * f.abs().max()  # one rounding to bf16


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3.0e38])
@pytest.mark.parametrize("where", ["k", "q", "state"])
def test_rounds_of_sixteen_tokens_with_infinities_and_overflow(where, value):
    q, k, v, g, s0 = _mixer_inputs(1, 45, 2, 64)
    x = {"k": k.clone(), "q": q.clone(), "state": s0.clone()}
    x[where][(0, 1, 3, 5) if where == "state" else (0, 20, 1, 3)] = value
    o, s = gla_cuda.gdn_recurrent(x["q"], x["k"], v, g, None, x["state"], 1.0, True)
    # token by token: one call a token is the token kernel's
    rows, state = [], x["state"]
    for t in range(45):
        a, state = gla_cuda.gdn_recurrent(x["q"][:, t : t + 1], x["k"][:, t : t + 1], v[:, t : t + 1], g[:, t : t + 1], None, state, 1.0, True)
        rows.append(a)
    want = torch.cat(rows, 1)
    for a, b in ((o, want), (s, state)):
        assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.isinf(a), torch.isinf(b))
        ok = torch.isfinite(b)
        assert torch.equal(a[torch.isinf(a)], b[torch.isinf(b)]) and _rel(a[ok], b[ok]) < 2.0 ** -8


@pytest.mark.parametrize("T,at,D", [(8, 5, 64), (12, 5, 64), (19, 9, 128), (70, 33, 64)])
@pytest.mark.parametrize("where", ["v", "k", "q", "beta"])
def test_delta_rule_prompts_keep_what_is_no_number_from_earlier_tokens(T, at, D, where):
    q, k, v, g, s0 = _mixer_inputs(2, T, 2, D)
    beta = torch.rand(2, T, 2, device="cuda")
    clean, _ = gla_cuda.gdn_recurrent(q, k, v, g, beta, s0, 1.0, True)
    for value in (float("nan"), float("inf")):
        x = {"q": q.clone(), "k": k.clone(), "v": v.clone(), "beta": beta.clone()}
        x[where][(0, at, 1) if where == "beta" else (0, at, 1, 3)] = value
        o, s = gla_cuda.gdn_recurrent(x["q"], x["k"], x["v"], g, x["beta"], s0, 1.0, True)
        oo, ss = ref.gated_deltanet_recurrent(*(x[n].double() for n in "qkv"), F.logsigmoid(g.double()).clamp(min=gla_cuda.GLA_MIN_LOG_DECAY),
                                              x["beta"].double(), s0.double(), 1.0)
        assert torch.equal(o[:, :at], clean[:, :at])
        assert torch.equal(torch.isfinite(o), torch.isfinite(oo)) and torch.equal(torch.isfinite(s), torch.isfinite(ss))


def test_a_thread_without_a_context_of_its_own_runs_tensor_map_kernels():
    import threading

    from triune_b200 import ops

    x, w = torch.randn(256, 128, device="cuda").bfloat16(), torch.randn(64, 128, device="cuda").bfloat16()
    want = ops.linear(x, w)
    spare = torch.empty_like(want)
    del spare  # the thread's output comes from the allocator's cache: no CUDA call before the tensor map
    got = []
    t = threading.Thread(target=lambda: got.append(ops.linear(x, w)))
    t.start()
    t.join()
    assert got and torch.equal(got[0], want)


@pytest.mark.parametrize("M,N,K,a_mn,b_mn", [
    (1536, 384, 32768, True, True), (384, 1536, 4100, True, True), (384, 384, 1536, True, True), (8, 384, 32761, True, True),
    (37, 1536, 6144, False, False), (129, 72, 1544, False, False), (512, 512, 1472, False, True), (640, 1024, 8192, False, True),
    (600, 1536, 384, False, False),
])
@pytest.mark.parametrize("what", ["plain", "bias", "gelu", "dgelu", "f32"])
def test_products_of_few_tiles_against_fp32(M, N, K, a_mn, b_mn, what):
    from triune_b200 import ops

    if what in ("gelu", "dgelu") and a_mn:
        pytest.skip("activation epilogues follow row-major activations")
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    Mp = (M + 7) // 8 * 8
    a = rnd(K, Mp)[:, :M] if a_mn else rnd(M, K)
    b = rnd(K, N) if b_mn else rnd(N, K)
    bias = rnd(N) if what in ("bias", "gelu") else None
    alpha = K ** -0.5
    want = alpha * (a.float().t() if a_mn else a.float()) @ (b.float() if b_mn else b.float().t())
    if bias is not None:
        want = want + bias.float()
    # fp32 sums of K products in another order: relative error about sqrt(K) 2^-24 (4e-6 for the longest), before the rounding
    bf16 = 2.0 ** -8
    if what == "gelu":
        aux = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
        got = ops.gemm(a, b, a_mn=a_mn, b_mn=b_mn, bias=bias, alpha=alpha, gelu=True, aux_out=aux)
        x = want.clone().requires_grad_(True)
        y = F.gelu(x, approximate="tanh")
        (d,) = torch.autograd.grad(y.sum(), x)
        assert _rel(got, y.detach()) < bf16 and _rel(aux, d) < bf16
    elif what == "dgelu":
        aux = rnd(M, N)
        got = ops.gemm(a, b, a_mn=a_mn, b_mn=b_mn, alpha=alpha, dgelu_aux=aux)
        assert _rel(got, want * aux.float()) < bf16
    else:
        kw = {"out_dtype": torch.float32} if what == "f32" else {}
        got = ops.gemm(a, b, a_mn=a_mn, b_mn=b_mn, bias=bias, alpha=alpha, **kw)
        assert _rel(got, want) < (2e-5 if what == "f32" else bf16)
    assert torch.isfinite(got.float()).all()


@pytest.mark.parametrize("M,N,K", [
    (1, 8, 64), (31, 72, 384), (129, 264, 384), (300, 1536, 384), (9001, 1544, 384), (257, 520, 1016), (257, 520, 1024),
    (1000, 2056, 1536),
])
def test_products_with_saved_rows_at_ragged_edges(M, N, K):
    """Chunks of the second operand read ahead: tiles cut in both directions, several tiles a block, sixteen and eight warps."""
    from triune_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    a, b, aux, alpha = rnd(M, K), rnd(N, K), rnd(M, N), K ** -0.5
    want = alpha * a.float() @ b.float().t()
    x = aux.float()
    # one rounding to bf16 (2^-9 of the value) over fp32 sums: every element, with the sums' error of sqrt(K) 2^-24 of its size
    for got, ref in ((ops.gemm(a, b, alpha=alpha, dgelu_aux=aux), want * x),
                     (ops.gemm(a, b, alpha=alpha, add_aux=aux, beta=-0.75), want - 0.75 * x)):
        bound = 2.0 ** -8 * ref.abs() + 1e-5 * (1 + x.abs())
        assert ((got.float() - ref).abs() <= bound).all()


@pytest.mark.parametrize("M,N", [(0, 1536), (0, 72), (40, 0), (0, 0)])
@pytest.mark.parametrize("K", [1536, 8192])
def test_empty_products_of_long_reductions_do_nothing(M, N, K):
    from triune_b200 import ops

    empty = lambda *s: torch.empty(*s, device="cuda", dtype=torch.bfloat16)
    for b_mn in (False, True) if N else (False,):  # rows of no columns are no operand of the tensor maps
        a, b = empty(M, K), empty(K, N) if b_mn else empty(N, K)
        for dtype in (torch.bfloat16, torch.float32):
            assert ops.gemm(a, b, b_mn=b_mn, out_dtype=dtype).shape == (M, N)
        assert ops.gemm(a, b, b_mn=b_mn, gelu=True, aux_out=empty(M, N)).shape == (M, N)
        assert ops.gemm(a, b, b_mn=b_mn, dgelu_aux=empty(M, N)).shape == (M, N)


def test_layers_over_no_rows_train():
    from triune_b200 import ops

    w1, b1, w2, b2 = (torch.randn(*s, device="cuda").bfloat16().requires_grad_(True) for s in ((2048, 1536), (2048,), (1536, 2048), (1536,)))
    x = torch.empty(0, 1536, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    y = ops.mlp_gelu(x, w1, b1, w2, b2)
    assert y.shape == (0, 1536)
    frozen = ops.linear(x, w1.detach())
    (dx,) = torch.autograd.grad(frozen, x, torch.empty_like(frozen))
    assert dx.shape == x.shape


@pytest.mark.parametrize("M", [1, 7, 8, 9, 16, 17])
@pytest.mark.parametrize("N,K", [(8, 8), (24, 72), (200, 384), (4760, 264), (2048, 5632), (19008, 520)])
def test_products_of_a_few_rows_against_fp32(M, N, K):
    from triune_b200 import _ext, ops

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    wide = rnd(M, K + 16)
    a, b, bias = wide[:, 8 : K + 8], rnd(N, K), rnd(N)  # rows of a wider matrix
    want = K ** -0.5 * a.float() @ b.float().t() + bias.float()
    assert _rel(ops.gemm(a, b, bias=bias, alpha=K ** -0.5), want) < 2.0 ** -8
    assert _rel(ops.gemm(a, b, bias=bias, alpha=K ** -0.5, gelu=True), F.gelu(want, approximate="tanh")) < 2.0 ** -8
    if N % 64 == 0:  # gate rows, then up rows
        h = torch.empty(M, N // 2, device="cuda", dtype=torch.bfloat16)
        b = b * K ** -0.5
        _ext.serving().tc_gemm_swiglu(a, b, h, None)
        gate, up = (a.float() @ b.float().t()).chunk(2, dim=1)
        assert _rel(h, F.silu(gate) * up) < 2.0 ** -8


def test_kernels_without_an_autograd_function_refuse_tangents_and_survive_a_trace():
    import torch.autograd.forward_ad as fw

    from triune_b200 import ops
    from triune_b200.models.attention import VectorisedGLA

    rnd = lambda *s: torch.randn(*s, device="cuda").bfloat16()
    x, w13, w2, wide, b1, b2 = rnd(5, 128), rnd(512, 128), rnd(128, 256), rnd(128, 512), rnd(512), rnd(128)
    m = VectorisedGLA(128, 2, 64).cuda().bfloat16().eval()
    state = torch.randn(5, 2, 64, 64, device="cuda")
    calls = (lambda a: ops.swiglu_mlp(a, w13, w2), lambda a: ops.mlp_gelu(a, w13, b1, wide, b2),
             lambda a: m(a.unsqueeze(1), cache=(state.clone(), 3))[0])
    with torch.no_grad():
        for call in calls:
            want = call(x)
            with fw.dual_level():
                assert _rel(call(x), want) < 2.0 ** -7  # a single token takes its general path here
                with pytest.raises(NotImplementedError):
                    call(fw.make_dual(x, torch.ones_like(x)))
        for call in calls[:2]:
            traced = torch.jit.trace(call, (x,), check_trace=False)
            y = rnd(5, 128)
            assert torch.equal(traced(y), call(y))


@pytest.mark.parametrize("B,H,D,delta,learn_beta,rope,on_device", [
    (1, 1, 64, False, False, True, False), (3, 2, 64, False, False, False, True), (2, 3, 128, False, False, True, True),
    (1, 2, 128, True, True, True, False), (5, 1, 64, True, False, True, True), (2, 4, 64, True, True, False, False),
])
def test_mixer_step_against_a_64_bit_statement(B, H, D, delta, learn_beta, rope, on_device):
    from triune_b200.models.attention import VectorisedGLA

    torch.manual_seed(B * 100 + H * 10 + D)
    dim = H * D
    m = VectorisedGLA(dim, H, D, use_delta_rule=delta, use_rope=rope, learn_beta=learn_beta, rope_max_seq_len=64).cuda().bfloat16().eval()
    x = torch.randn(B, 1, dim, device="cuda").bfloat16()
    s0 = torch.randn(B, H, D, D, device="cuda")
    at = 77  # past the first size of the rotary tables
    if on_device and rope:
        m.rope(1, "cuda:0", offset=at)  # a position on the device relies on tables that cover it
    with torch.no_grad():
        y, (s1, after) = m(x, cache=(s0.clone(), torch.tensor([at], device="cuda") if on_device else at))
    assert int(after) == at + 1
    # from the projection rows as the model rounds them, so that only the step itself is compared
    from triune_b200 import ops

    with torch.no_grad():
        qkvg = ops.linear(x.reshape(B, dim), m.qkvg_weight).double()
    q, k, v, g = (t.reshape(B, H, D) for t in qkvg.chunk(4, dim=1))
    q, k = (F.normalize(F.elu(t) + 1, dim=-1) for t in (q, k))
    if rope:
        c, s = (t[at].double().cuda() for t in (m.rope._cos, m.rope._sin))
        q, k = (t * c + torch.cat((-t[..., D // 2:], t[..., : D // 2]), -1) * s for t in (q, k))
    u, st = v, s0.double()
    if delta:
        u = v - torch.einsum("bhk,bhkv->bhv", k, st)
        if learn_beta:
            u = u * torch.sigmoid(x.reshape(B, dim).double() @ m.beta_proj.weight.double().t()).unsqueeze(-1)
    st = st * torch.exp(F.logsigmoid(g)).unsqueeze(-1) + k.unsqueeze(-1) * u.unsqueeze(-2)
    o = torch.einsum("bhk,bhkv->bhv", q, st).reshape(B, dim)
    assert _rel(s1, st) < 2e-6                                              # fp32 throughout
    assert _rel(y.reshape(B, dim), o @ m.out_proj.weight.double().t()) < 2.0 ** -7  # two bf16 roundings


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("delta,learn_beta,on_device", [(False, False, True), (False, False, False), (True, False, True), (True, True, True)])
def test_verified_tokens_are_the_decoded_ones(D, delta, learn_beta, on_device):
    from triune_b200.models.attention import VectorisedGLA

    torch.manual_seed(D)
    B, T, H = 1, 4, 3
    m = VectorisedGLA(H * D, H, D, use_delta_rule=delta, learn_beta=learn_beta).cuda().bfloat16().eval()
    x, s0 = torch.randn(B, T, H * D, device="cuda").bfloat16(), torch.randn(B, H, D, D, device="cuda")
    at = lambda i: torch.tensor([i], device="cuda") if on_device else i
    with torch.no_grad():
        kept = s0.clone()
        y, states = m.forward_token_states(x, kept, at(11))
        assert torch.equal(kept, s0)
        state = s0.clone()
        for j in range(T):
            one, (state, _) = m(x[:, j : j + 1], cache=(state.clone(), at(11 + j)))
            # products of up to 16 rows add a row's terms in one order, whatever the number of rows
            assert torch.equal(states[j], state) and torch.equal(y[:, j : j + 1], one), j


@pytest.mark.parametrize("mixer", ["gla", "gated_deltanet"])
@pytest.mark.parametrize("head_dim", [64, 128])
def test_replayed_speculation_gives_the_tokens_of_plain_greedy_decoding(mixer, head_dim):
    from triune_b200.config import ModelConfig
    from triune_b200.inference import GraphedGreedyDecoder, GraphedSpeculativeDecoder
    from triune_b200.models import TriuneTransformer
    from triune_b200.utils import place_model

    torch.manual_seed(1)
    cfg = ModelConfig(vocab_size=256, hidden_dim=2 * head_dim, num_layers=5, num_heads=2, head_dim=head_dim, num_experts=4, top_k=1,
                      router_prefix_layers=1, reflex_exit_layer=2, limbic_exit_layer=3, expert_hidden=128, dense_hidden=128, mixer=mixer)
    m = place_model(TriuneTransformer.from_config(cfg), torch.device("cuda"), torch.bfloat16).eval()
    ids = torch.randint(0, 256, (1, 21), device="cuda")
    want = GraphedGreedyDecoder(m).generate(ids, 48)
    assert torch.equal(GraphedSpeculativeDecoder(m, k_draft=3).generate(ids, 48), want)


@pytest.mark.parametrize("T,grad", [(1, False), (5, False), (70, True)])
def test_a_write_strength_projection_with_hooks_or_a_bias_is_called(T, grad):
    from triune_b200.models.attention import VectorisedGLA

    torch.manual_seed(2)
    m = VectorisedGLA(256, 2, 128, use_delta_rule=True, learn_beta=True).cuda().bfloat16()
    x, cache = torch.randn(2, T, 256, device="cuda").bfloat16(), (torch.randn(2, 2, 128, 128, device="cuda"), 3)

    def run():
        with torch.set_grad_enabled(grad):
            return m(x, cache=(cache[0].clone(), 3))[0].detach()

    plain, seen = run(), []
    for register in (m.beta_proj.register_forward_hook, m.beta_proj.register_forward_pre_hook,
                     torch.nn.modules.module.register_module_forward_hook):
        handle = register(lambda mod, *a: seen.append(mod is m.beta_proj) and None)
        hooked = run()
        handle.remove()
        assert any(seen) and _rel(hooked, plain) < 0.01, register  # its own forward rounds the strength to bf16
        seen.clear()
    shut = m.beta_proj.register_forward_hook(lambda mod, a, out: out - 1e4)  # a strength of zero writes nothing
    nothing = run()
    shut.remove()
    m.beta_proj.bias = torch.nn.Parameter(torch.full((2,), -1e4, device="cuda", dtype=torch.bfloat16))
    assert torch.equal(run(), nothing) and _rel(nothing, plain) > 0.05
    m.beta_proj.bias = None
    m.beta_proj.forward = lambda a: torch.nn.functional.linear(a, m.beta_proj.weight) - 1e4
    assert torch.equal(run(), nothing)


@pytest.mark.parametrize("use_rope", [False, True])
@pytest.mark.parametrize("dtype,device", [(torch.int32, "cuda"), (torch.int16, "cuda"), (torch.float32, "cuda"), (torch.int64, "cuda"), (torch.int64, "cpu")])
def test_decoding_step_takes_positions_of_any_number_type(use_rope, dtype, device):
    from triune_b200.models.attention import VectorisedGLA

    if use_rope and device == "cpu":
        pytest.skip("rotary rows are gathered on the device")
    m = VectorisedGLA(128, 2, 64, use_rope=use_rope).cuda().bfloat16().eval()
    x, s0 = torch.randn(2, 1, 128, device="cuda").bfloat16(), torch.randn(2, 2, 64, 64, device="cuda")
    with torch.no_grad():
        want, (state, _) = m(x, cache=(s0.clone(), 9))
        got, (after, at) = m(x, cache=(s0.clone(), torch.tensor([9], dtype=dtype, device=device)))
    assert torch.equal(got, want) and torch.equal(after, state) and float(at) == 10


@pytest.mark.parametrize("position", [-1, 64, 10 ** 12])
def test_mixer_step_outside_the_rotary_table_is_nan(position):
    B, H, D = 2, 2, 64
    qkvg, state = torch.randn(B, 4 * H * D, device="cuda").bfloat16(), torch.randn(B, H, D, D, device="cuda")
    tables = tuple(torch.ones(64, D, device="cuda") for _ in range(2))
    with torch.no_grad():
        for where in (position, torch.tensor([position], device="cuda")):
            out, after = gla_cuda.mixer_step(qkvg, tables, where, state.clone(), False)
            assert torch.isnan(out).all() and torch.isnan(after).all()
        out, after = gla_cuda.mixer_step(qkvg, tables, 63, state.clone(), False)
        assert torch.isfinite(out).all() and torch.isfinite(after).all()


@pytest.mark.parametrize("mixer", ["gla", "gated_deltanet"])
def test_replayed_decoding_past_the_first_rotary_tables(mixer):
    from triune_b200.config import ModelConfig
    from triune_b200.inference import GraphedGreedyDecoder, GraphedSpeculativeDecoder, generate_tokens
    from triune_b200.models import TriuneTransformer
    from triune_b200.models.factory import build_model
    from triune_b200.utils import place_model

    V = 64
    cfg = ModelConfig(family="universal", vocab_size=V, hidden_dim=128, num_layers=2, num_heads=2, head_dim=64, mixer=mixer, ffn="swiglu",
                      dense_hidden=256, tie_embeddings=False, rope_max_seq_len=32).validate()
    torch.manual_seed(0)
    m = place_model(build_model(cfg), torch.device("cuda"), torch.bfloat16).eval()
    with torch.no_grad():  # a model that is sure of its next token, so that bf16 ties decide nothing
        emb = torch.randn(V, 128, device="cuda")
        m.embed_tokens.weight.copy_(emb)
        m.lm_head.weight.copy_(emb.roll(1, 0) * 0.25)
    dec = GraphedGreedyDecoder(m)
    for length, new in ((5, 40), (5, 20), (70, 100), (9, 3), (9, 1)):  # captures made before and after the tables grew
        ids = torch.randint(0, V, (1, length), device="cuda")
        want, cache, _ = generate_tokens(m, ids, new, temperature=0.0, repetition_penalty=1.0, count_penalty=0.0)
        assert dec.generate(ids, new)[0, length:].tolist() == want
        for a, b in zip(dec.states, cache):
            assert _rel(a, b[0]) < 1e-5
    tight = GraphedGreedyDecoder(m, max_positions=64)
    rows = dec.rotary[0]._cos.shape[0]
    with pytest.raises(ValueError, match="max_positions"):
        tight.generate(ids, rows)
    if mixer == "gla":
        t = place_model(TriuneTransformer.from_config(ModelConfig(vocab_size=256, hidden_dim=128, num_layers=5, num_heads=2, head_dim=64, num_experts=4,
                        top_k=1, router_prefix_layers=1, reflex_exit_layer=2, limbic_exit_layer=3, expert_hidden=128, dense_hidden=128)),
                        torch.device("cuda"), torch.bfloat16).eval()
        spec = GraphedSpeculativeDecoder(t, k_draft=3)
        spec.prefill(ids)
        for mod in spec.rotary:
            mod.max_seq_len, mod._cos, mod._sin = 16, None, None
        assert spec.generate(ids, 40).shape[1] == ids.shape[1] + 40


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("T", [2, 16, 17, 63, 64, 65, 191, 256])
def test_gated_attention_of_any_length_against_fp64(T, D):
    B, H = 2, 3
    q, k, v, g, s0 = (t.requires_grad_(True) for t in _mixer_inputs(B, T, H, D, seed=T))
    o, s = gla_cuda._GLAFn.apply(q, k, v, g, s0, True)
    wo, ws = torch.randn_like(o), torch.randn_like(s) * 0.1
    got = (o, s, *torch.autograd.grad((o.float() * wo).sum() + (s * ws).sum(), (q, k, v, g, s0)))
    x = [t.detach().double().requires_grad_(True) for t in (q, k, v, g, s0)]
    gl = F.logsigmoid(x[3])
    if T >= 64:
        gl = gl.clamp(min=gla_cuda.GLA_MIN_LOG_DECAY)
    oo, ss = ref.gla_chunk(*x[:3], gl, x[4])
    want = (oo, ss, *torch.autograd.grad((oo * wo.double()).sum() + (ss * ws.double()).sum(), x))
    # under 64 tokens everything is fp32 and bf16 results round by at most 2^-9; whole chunks have bf16 operands (states,
    # weighted keys and scores, 2^-9 each) in two products that follow one another
    rounding = 2.0 ** -8
    for n, a, b in zip(("o", "s", "dq", "dk", "dv", "dg", "ds0"), got, want):
        if n == "dg" and T >= 64:
            assert _gate_error(a, b, x[0].detach(), x[1].detach(), want[2], want[3], (ws.double() * ss.detach()).sum(-1), torch.sigmoid(-x[3]).detach()) < 1
            continue
        limit = (1e-5 if a.dtype == torch.float32 else rounding) if T < 64 else 2 * rounding
        assert _rel(a, b) < limit, (n, _rel(a, b))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("T,at", [(21, 7), (63, 40), (70, 66), (127, 64)])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), float("-inf")])
def test_gates_that_are_no_numbers_reach_what_depends_on_them(T, at, D, value):
    B, H = 2, 2
    q, k, v, g, s0 = _mixer_inputs(B, T, H, D, seed=T)
    g[0, at, 1, 5] = value
    ins = [t.requires_grad_(True) for t in (q, k, v, g, s0)]
    o, s = gla_cuda._GLAFn.apply(*ins, True)
    wo, ws = torch.randn_like(o), torch.randn_like(s)
    got = (o, s, *torch.autograd.grad((o.float() * wo).sum() + (s * ws).sum(), ins))
    x = [t.detach().double().requires_grad_(True) for t in ins]
    gl = F.logsigmoid(x[3])
    oo, ss = ref.gla_recurrent(*x[:3], gl if T < 64 else gl.clamp(min=gla_cuda.GLA_MIN_LOG_DECAY), x[4])
    want = (oo, ss, *torch.autograd.grad((oo * wo.double()).sum() + (ss * ws.double()).sum(), x))
    for n, a, b in zip(("o", "s", "dq", "dk", "dv", "dg", "ds0"), got, want):
        if T >= 64 and n not in ("o", "s", "dq"):  # whole chunks spread the state's gradient over all that its products touch
            a, b = a[:, 64:], b[:, 64:]
            if n == "ds0":
                continue
        assert torch.equal(torch.isnan(a), torch.isnan(b)), n


@pytest.mark.parametrize("D", [64, 128])
def test_wider_operands_are_not_rounded_after_the_last_chunk(D):
    from triune_b200 import ops

    B, T, H = 2, 100, 2
    gen = torch.Generator(device="cuda").manual_seed(D)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    q, k, v = F.normalize(rnd(B, T, H, D), dim=-1).bfloat16(), F.normalize(rnd(B, T, H, D), dim=-1), rnd(B, T, H, D)
    g = -0.05 * torch.rand(B, T, H, D, device="cuda", generator=gen)  # fp32 log decays, keys and values beside bf16 queries
    k, v, g = (t.requires_grad_(True) for t in (k, v, g))
    o, s = ops.gla(q, k, v, g)
    ds = torch.randn_like(s)
    got = (s, *(t[:, 64:] for t in torch.autograd.grad(s, (k, v, g), ds)))
    x = [t.detach().double() for t in (q, k, v, g)]
    with torch.no_grad():
        _, s64 = ops.gla(*(t[:, :64] for t in (q, k, v, g)))
    tail = [t[:, 64:].clone().requires_grad_(True) for t in x[1:]]
    oo, ss = ref.gla_recurrent(x[0][:, 64:], *tail, s64.double())
    want = (ss, *torch.autograd.grad(ss, tail, ds.double()))
    for n, a, b in zip(("s", "dk", "dv", "dg"), got, want):
        assert _rel(a, b) < 1e-5, (n, _rel(a, b))  # fp32 throughout: rounded operands are 2^-9 off
    assert _rel(o[:, 64:], oo) < 2.0 ** -8


@pytest.mark.parametrize("D", [64, 128])
def test_many_sequences_and_none(D):
    from triune_b200.models.attention import VectorisedGLA

    B, T, H = 65539, 2, 1
    gen = torch.Generator(device="cuda").manual_seed(D)
    x = torch.randn(B * T, 4 * H * D, device="cuda", generator=gen).bfloat16().requires_grad_(True)
    ends = torch.tensor([0, 1, 65534, 65535, 65536, 65538], device="cuda")  # past the largest grid dimension that is not x
    few = x.detach().view(B, T, -1)[ends].reshape(-1, 4 * H * D).requires_grad_(True)
    w = torch.randn(B * T, H * D, device="cuda", generator=gen).bfloat16()
    o, s = gla_cuda.gla_attention_core(x, None, None, None, B, T, H)
    (dx,) = torch.autograd.grad(o, x, w)
    oo, ss = gla_cuda.gla_attention_core(few, None, None, None, len(ends), T, H)
    (want,) = torch.autograd.grad(oo, few, w.view(B, T, -1)[ends].reshape(-1, H * D))
    pick = lambda t: t.view(B, T, -1)[ends].reshape(len(ends) * T, -1)
    assert torch.equal(pick(o), oo) and torch.equal(s[ends], ss) and torch.equal(pick(dx), want)
    with torch.no_grad():
        rows = x.detach()[:B]
        o, s = gla_cuda.mixer_step(rows, None, 0, s, False, keep_state=True)
        oo, ss = gla_cuda.mixer_step(rows[ends], None, 0, ss, False, keep_state=True)
        assert torch.equal(o[ends], oo) and torch.equal(s[ends], ss)
        m = VectorisedGLA(D, 1, D).cuda().bfloat16().eval()
        y, (state, at) = m(torch.empty(0, 5, D, device="cuda", dtype=torch.bfloat16), cache=(None, 0))
        assert y.shape == (0, 5, D) and state.shape == (0, 1, D, D) and at == 5


@pytest.mark.parametrize("T", [5, 64, 70])
@pytest.mark.parametrize("delta", [False, True])
def test_a_state_on_the_host_is_refused(T, delta):
    from triune_b200.models.attention import VectorisedGLA

    m = VectorisedGLA(128, 1, 128, use_delta_rule=delta, learn_beta=delta).cuda().bfloat16()
    x = torch.randn(2, T, 128, device="cuda").bfloat16()
    with pytest.raises(RuntimeError):  # before a kernel sees the pointer
        m(x, cache=(torch.zeros(2, 1, 128, 128), 0))
    y, (state, _) = m(x, cache=(torch.zeros(2, 1, 128, 128, device="cuda"), 0))
    assert torch.isfinite(y).all() and torch.isfinite(state).all()


@pytest.mark.parametrize("T,D", [(21, 128), (150, 64), (150, 128)])
def test_fused_projection_rows_match_separate_tensors(T, D):
    B, H = 2, 2
    gen = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(B * T, 4 * H * D, device="cuda", generator=gen).bfloat16().requires_grad_(True)
    s0 = torch.randn(1, H, D, D, device="cuda", generator=gen).requires_grad_(True)  # one state for every sequence
    w = torch.randn(B * T, H * D, device="cuda", generator=gen)
    o, s = gla_cuda.gla_attention_core(x, None, None, s0, B, T, H)
    got = torch.autograd.grad((o.float() * w).sum() + s.sum(), (x, s0))
    from triune_b200 import ops

    q, k, v, g = ops.qk_feature_map(x, None, None, B, T, H, D)
    oo, ss = gla_cuda._GLAFn.apply(q, k, v, g, s0.expand(B, H, D, D), True)
    want = torch.autograd.grad((oo.reshape(B * T, H * D).float() * w).sum() + ss.sum(), (x, s0))
    assert torch.equal(o, oo.reshape(B * T, H * D)) and torch.equal(s, ss)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


def _off_by_one(t):  # the same values, contiguous, four or two bytes past a 16-byte boundary
    flat = torch.empty(t.numel() + 1, device=t.device, dtype=t.dtype)
    return flat[1:].view(t.shape).copy_(t)


@pytest.mark.parametrize("T,D", [(1, 64), (9, 64), (9, 128)])
def test_rotary_tables_and_gradients_of_any_alignment(T, D):
    from triune_b200 import ops

    B, H = 2, 2
    x = torch.randn(B * T, 4 * H * D, device="cuda").bfloat16().requires_grad_(True)
    cos, sin = ops.rope_tables(T, D, 10000.0, 0, x.device)
    odd = torch.randn(T, D + 3, device="cuda")[:, :D].copy_(cos)  # rows of an odd pitch
    want = ops.qk_feature_map(x, cos, sin, B, T, H, D)
    for c, s in ((_off_by_one(cos), _off_by_one(sin)), (odd, sin), (cos[:, : D // 2].clone(), sin[:, : D // 2].clone())):
        assert all(torch.equal(a, b) for a, b in zip(ops.qk_feature_map(x, c, s, B, T, H, D), want))
    if T > 1:
        beta, d = torch.rand(B * T, H, device="cuda"), torch.randn(B * T, H * D, device="cuda").bfloat16()
        for core in (lambda: gla_cuda.gla_attention_core(x, cos, sin, None, B, T, H)[0],
                     lambda: gla_cuda.gdn_attention_core(x, cos, sin, beta, None, B, T, H)[0]):
            a, b = (torch.autograd.grad(core(), x, g)[0] for g in (d, _off_by_one(d)))
            assert torch.equal(a, b)


@pytest.mark.parametrize("rows,d", [(1, 8), (1, 2048), (7, 264), (37, 1536), (1185, 384), (1184, 776), (2375, 2040), (9480, 512), (5000, 1032),
                                    (2368, 776), (2369, 520), (2369, 768), (2400, 1024), (9473, 1024)])
@pytest.mark.parametrize("residual", [False, True])
def test_norm_rows_against_fp64(rows, d, residual):
    from triune_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(rows + d)
    x, r, dy, ds = (torch.randn(rows, d, device="cuda", generator=g).bfloat16().requires_grad_(i < 2) for i in range(4))
    w = (1 + 0.1 * torch.randn(d, device="cuda", generator=g)).bfloat16().requires_grad_(True)
    if residual:
        outs, seeds = ops.add_rmsnorm(x, r, w, 1e-6), (dy, ds)
    else:
        outs, seeds = (ops.rmsnorm(x, w, 1e-6),), (dy,)
    got = torch.autograd.grad(outs, (x, w), seeds)
    s = (x.detach() + r.detach() if residual else x.detach()).double().requires_grad_(True)
    w64 = w.detach().double().requires_grad_(True)
    y = s * torch.rsqrt(s.pow(2).mean(-1, keepdim=True) + 1e-6) * w64
    want = torch.autograd.grad((y, s * 1.0) if residual else (y,), (s, w64), tuple(t.double() for t in seeds))
    for a, b in zip((*outs, *got), (y, *((s,) if residual else ()), *want)):
        assert _rel(a, b) < 2.0 ** -8  # fp32 sums, results rounded to bf16: at most 2^-9 each


def test_weight_gradients_add_to_an_fp32_arena():
    from triune_b200 import ops

    x = torch.randn(700, 384, device="cuda").bfloat16().requires_grad_(True)
    w = torch.ones(384, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    plain, = torch.autograd.grad(ops.rmsnorm(x, w).float().square().sum(), w)
    w.main_grad = torch.full((384,), 3.0, device="cuda")
    ops.rmsnorm(x, w).float().square().sum().backward()
    assert w.grad is None and _rel(w.main_grad - 3.0, plain) < 2.0 ** -8


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("T", [2, 63, 64, 65, 130])
@pytest.mark.parametrize("with_beta", [False, True])
def test_delta_rule_training_of_any_length_against_fp64(T, D, with_beta):
    from triune_b200 import ops

    B, H = 2, 3
    q, k, v, g, s0 = _mixer_inputs(B, T, H, D, seed=T)
    ins = [q, k, v, g, s0] + ([torch.rand(B, T, H, device="cuda")] if with_beta else [])
    ins = [t.requires_grad_(True) for t in ins]
    o, s = ops.gated_deltanet(*ins[:4], beta=ins[5] if with_beta else None, initial_state=ins[4], gate_logits=True)
    wo, ws = torch.randn_like(o), torch.randn_like(s) * 0.1
    got = (o, s, *torch.autograd.grad((o.float() * wo).sum() + (s * ws).sum(), ins))
    x = [t.detach().double().requires_grad_(True) for t in ins]
    gl = F.logsigmoid(x[3]).clamp(min=gla_cuda.GLA_MIN_LOG_DECAY)
    oo, ss = ref.gated_deltanet_recurrent(*x[:3], gl, x[5] if with_beta else None, x[4])
    want = (oo, ss, *torch.autograd.grad((oo * wo.double()).sum() + (ss * ws.double()).sum(), x))
    # bf16 operands (2^-9 each) in the chunk's inverse, the effective values, states and scores: up to four products that follow
    # one another, twice that backward
    for n, a, b in zip(("o", "s", "dq", "dk", "dv", "dg", "ds0", "dbeta"), got, want):
        if n == "dg":
            assert _gate_error(a, b, x[0].detach(), x[1].detach(), want[2], want[3], (ws.double() * ss.detach()).sum(-1), torch.sigmoid(-x[3]).detach()) < 1
            continue
        assert _rel(a, b) < 2.0 ** -8 * (2 if n in ("o", "s") else 3), (n, _rel(a, b))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3.0e38])
def test_state_pass_of_the_delta_rule_keeps_infinite_states_infinite(D, value):
    """As fp32 arithmetic has it: in the column of an infinite element of the initial state the effective values are infinite with the
    other sign (equal keys, small strengths and open gates, so that every token reads it with one sign), and so are the rows that
    keys add them to; the element itself is no number then."""
    from triune_b200 import ops

    B, T, H = 1, 64, 2
    q, k, v, g, s0 = _mixer_inputs(B, T, H, D, seed=D)
    s0[0, 1, 7, 9] = value
    g.fill_(20.0)
    k.fill_(D ** -0.5)
    beta = torch.full((B, T, H), 0.01, device="cuda")
    o, s = ops.gated_deltanet(q.requires_grad_(True), k, v, g, beta=beta, initial_state=s0, gate_logits=True)
    clean = ops.gated_deltanet(q, k, v, g, beta=beta, initial_state=torch.where(torch.isfinite(s0) & (s0.abs() < 1e38), s0, 0.0), gate_logits=True)[1]
    touched = torch.zeros_like(s, dtype=torch.bool)
    touched[0, 1, :, 9] = True
    assert torch.equal(s[~touched], clean[~touched])
    column = s[0, 1, :, 9]
    others = torch.arange(D, device="cuda") != 7
    if value != value:
        assert torch.isnan(column).all()
    elif value == 3.0e38:
        assert not torch.isnan(column).any()
    else:
        assert torch.isinf(column[others]).all() and (torch.sign(column[others]) == -torch.sign(torch.tensor(value))).all()


@pytest.mark.parametrize("T,D", [(21, 128), (150, 64), (128, 128)])
def test_fused_delta_rule_rows_match_separate_tensors(T, D):
    from triune_b200 import ops

    B, H = 2, 2
    gen = torch.Generator(device="cuda").manual_seed(6)
    x = torch.randn(B * T, 4 * H * D, device="cuda", generator=gen).bfloat16().requires_grad_(True)
    beta = torch.rand(B * T, H, device="cuda", generator=gen).requires_grad_(True)
    s0 = torch.randn(B, H, D, D, device="cuda", generator=gen).requires_grad_(True)
    w = torch.randn(B * T, H * D, device="cuda", generator=gen)
    cos, sin = ops.rope_tables(T + 3, D, 10000.0, 0, x.device)
    cos, sin = cos[3:], sin[3:]
    o, s = gla_cuda.gdn_attention_core(x, cos, sin, beta, s0, B, T, H)
    got = torch.autograd.grad((o.float() * w).sum() + s.sum(), (x, beta, s0))
    q, k, v, g = ops.qk_feature_map(x, cos, sin, B, T, H, D)
    oo, ss = ops.gated_deltanet(q, k, v, g, beta=beta.view(B, T, H), initial_state=s0, gate_logits=True)
    want = torch.autograd.grad((oo.reshape(B * T, H * D).float() * w).sum() + ss.sum(), (x, beta, s0))
    assert torch.equal(o, oo.reshape(B * T, H * D)) and torch.equal(s, ss)
    # dbeta sums a row's parts with shared-memory atomics: the order of fp32 additions may differ between runs
    assert torch.equal(got[0], want[0]) and _rel(got[1], want[1]) < 1e-6 and torch.equal(got[2], want[2])


@pytest.mark.parametrize("H", [16, 17, 24])
def test_training_pass_of_any_number_of_heads(H, monkeypatch):
    from triune_b200 import ops
    from triune_b200.models.attention import VectorisedGLA

    torch.manual_seed(H)
    B, T, D, dim = 2, 70, 64, 256
    m = VectorisedGLA(dim, H, D, use_delta_rule=True, learn_beta=True, use_rope=False).cuda().bfloat16()
    x, w = torch.randn(B, T, dim, device="cuda").bfloat16().requires_grad_(True), torch.randn(B, T, dim, device="cuda").bfloat16()
    params = (x, m.qkvg_weight, m.beta_proj.weight, m.out_proj.weight)
    core, taken = gla_cuda.gdn_attention_core, []
    monkeypatch.setattr(gla_cuda, "gdn_attention_core", lambda *a: taken.append(1) or core(*a))
    y = m(x)[0]
    got = (y, *torch.autograd.grad(y, params, w))
    assert taken
    x2 = x.reshape(B * T, dim)
    q, k, v, g = ops.qk_feature_map(ops.linear(x2, m.qkvg_weight), None, None, B, T, H, D)
    beta = m._strengths(x, x2).view(B, T, H)
    o = ops.gated_deltanet(q, k, v, g, beta=beta, gate_logits=True)[0]
    y2 = ops.linear(o.reshape(B, T, H * D), m.out_proj.weight)
    want = (y2, *torch.autograd.grad(y2, params, w))
    # the same kernels on separate tensors; the strengths' gradients come from shared-memory atomics, whose order differs
    for i, (a, b) in enumerate(zip(got, want)):
        assert torch.equal(a, b) if i in (0, 2, 4) else _rel(a, b) < 2.0 ** -8, i


@pytest.mark.parametrize("rows,dim,H", [(1, 8, 1), (15, 264, 6), (16, 384, 8), (33, 520, 9), (600, 2048, 16), (9000, 1024, 8)])
def test_write_strengths_against_fp64(rows, dim, H):
    gen = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, dim, device="cuda", generator=gen).bfloat16().requires_grad_(True)
    w = (torch.randn(H, dim, device="cuda", generator=gen) * dim ** -0.5).bfloat16().requires_grad_(True)
    db = torch.randn(rows, H, device="cuda", generator=gen)
    beta = gla_cuda.write_strength(x, w)
    dx, dw = torch.autograd.grad(beta, (x, w), db)
    x64, w64 = (t.detach().double().requires_grad_(True) for t in (x, w))
    b64 = torch.sigmoid(x64 @ w64.t())
    dx64, dw64 = torch.autograd.grad(b64, (x64, w64), db.double())
    assert _rel(beta, b64) < 2e-6 and _rel(dx, dx64) < 2.0 ** -8 and _rel(dw, dw64) < 2.0 ** -8  # fp32 sums; bf16 gradients


@pytest.mark.parametrize("rows,V,offset", [(1, 1, 0), (3, 7, 0), (5, 256, 0), (5, 257, 0), (3, 263, 1), (2, 2048, 0), (2, 2049, 0), (2, 8191, 0),
                                         (4, 32000, 0), (2, 32001, 3)])
def test_largest_of_rows_as_torch_orders_them(rows, V, offset):
    from triune_b200 import ops

    x = torch.randn(rows, V + offset, device="cuda").bfloat16()[:, offset:]
    for change in ("none", "ties", "nan", "lowest", "zeros"):
        y = x.clone() if offset == 0 else x
        if change == "ties":
            y[:, V // 3:] = 9.0
        elif change == "nan":
            y[:, V // 2] = float("nan")
            y[:, V - 1] = float("nan")
        elif change == "lowest":
            y[:] = float("-inf")
        elif change == "zeros":
            y[:] = 0.0
            y[:, 0] = -0.0
        out = torch.full((rows, 1), -1, device="cuda")
        ops.argmax_into(y, out)
        assert torch.equal(out, y.float().cpu().argmax(-1, keepdim=True).cuda()), change
