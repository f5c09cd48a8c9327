"""Kernels that a layer's forward, backward or decoding step takes at particular sizes, at the borders of those sizes."""

import pytest
import torch
import torch.nn.functional as F

from triune_b200.ops import gla_cuda
from triune_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm()).item()


def _mixer_inputs(B, T, H, D, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    q, k = (F.normalize(F.elu(rnd(B, T, H, D)) + 1, dim=-1).bfloat16() for _ in range(2))
    return q, k, rnd(B, T, H, D).bfloat16(), rnd(B, T, H, D).bfloat16(), rnd(B, H, D, D)


@pytest.mark.parametrize("B,T,H,D,beta_dims", [
    (1, 7, 2, 64, 1), (1, 8, 1, 64, 0), (2, 9, 3, 64, 1), (1, 15, 1, 128, 0), (2, 16, 2, 128, 2), (3, 65, 2, 64, 2), (1, 131, 2, 128, 1),
    (8, 500, 8, 128, 1),  # 64 heads: more tokens than one segment of records
])
def test_delta_rule_prompts_against_the_token_recurrence(B, T, H, D, beta_dims):
    q, k, v, g, s0 = _mixer_inputs(B, T, H, D)
    beta = None if beta_dims == 0 else torch.rand(B, T, H, *([D] if beta_dims == 2 else []), device="cuda")
    o, s = gla_cuda.gdn_recurrent(q, k, v, g, beta, s0, 0.7, True)
    gl = F.logsigmoid(g.double()).clamp(min=gla_cuda.GLA_MIN_LOG_DECAY)
    oo, ss = ref.gated_deltanet_recurrent(q.double(), k.double(), v.double(), gl, None if beta is None else beta.double(), s0.double(), 0.7)
    assert _rel(o, oo) < 2.0 ** -8   # outputs are rounded to bf16: at most 2^-9 each
    assert _rel(s, ss) < 1e-6        # the state is fp32 throughout


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
