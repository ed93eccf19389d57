"""Attention over whole prompts where its kernels change their form: edges of query and key tiles, head sizes that fill
their 64-wide blocks in part, groups of heads.  Checked against the definition in fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def attention(q, k, v, causal):
    q, k, v = q.double(), k.double(), v.double()
    group, n, m = q.shape[1] // k.shape[1], q.shape[0], k.shape[0]
    s = torch.einsum("qhd,khd->hqk", q, k.repeat_interleave(group, 1)) * q.shape[2] ** -0.5
    if causal:  # row t sees the keys [0, min(t + 1, m))
        s.masked_fill_(torch.arange(m, device=q.device)[None, :] > torch.arange(n, device=q.device)[:, None], float("-inf"))
    return torch.einsum("hqk,khd->qhd", torch.softmax(s, -1), v.repeat_interleave(group, 1))


def tensors(sq, skv, hq, hkv, d, dtype, spread=1.0):
    g = torch.Generator(device="cuda").manual_seed(sq * 1000 + d)
    rnd = lambda n, h: torch.randn((n, h, d), generator=g, device="cuda")  # noqa: E731
    return (rnd(sq, hq) * spread).to(dtype), rnd(skv, hkv).to(dtype), rnd(skv, hkv).to(dtype)


@pytest.mark.parametrize("d", [8, 40, 64, 72, 96, 120])
@pytest.mark.parametrize("sq,skv", [(16, 16), (127, 129), (257, 256), (300, 511)])
def test_fp16_narrow_heads_on_tensor_cores(d, sq, skv):
    """Weights keep 22 bits and sums 32, so what is left is the rounding of the result: 2^-11 of its value, and 2^-20 for
    the sums."""
    from axono_b200 import ops

    for causal in (True, False):
        for hq, hkv, spread in ((4, 2, 1.0), (3, 3, 6.0)):
            q, k, v = tensors(sq, skv, hq, hkv, d, torch.float16, spread)
            out = ops.scaled_dot_product_attention(q, k, v, causal).double()
            ref = attention(q, k, v, causal)
            err = (out - ref).abs()
            assert (err <= ref.abs() * 2.0 ** -11 + ref.abs().max() * 2.0 ** -20).all(), (causal, hq, err.max())
    assert ops.last_error() == 0
