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


def without_scratch(q, k, v, causal):
    """The same through the kernels that a call without scratch takes: FMA kernel in fp32, whole blocks in fp16."""
    from axono_b200 import _capi

    lib, out = _capi.lib(), torch.empty_like(q)
    st = lib.axb200_sdpa(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), q.shape[0], q.shape[1], k.shape[1], q.shape[2],
                         k.shape[0], int(causal), _capi.FLOAT32 if q.dtype == torch.float32 else _capi.FLOAT16, None, 0, torch.cuda.current_stream().cuda_stream)
    assert st == 0
    return out


@pytest.mark.parametrize("d", [4, 20, 64, 68, 80, 128])
@pytest.mark.parametrize("sq,skv", [(16, 64), (16, 129), (128, 66), (127, 129), (129, 128), (300, 511), (1030, 1100)])
def test_fp32_on_tensor_cores(d, sq, skv):
    """A score is off by 2^-21 of the largest one (its sum of products and its exponent), which changes a weight by as much;
    sums over keys and the result by 2^-20."""
    from axono_b200 import ops

    for causal in (True, False):
        for hq, hkv, spread in ((4, 2, 1.0), (3, 3, 6.0)):
            q, k, v = tensors(sq, skv, hq, hkv, d, torch.float32, spread)
            out = ops.scaled_dot_product_attention(q, k, v, causal).double()
            ref = attention(q, k, v, causal)
            top = (torch.einsum("qhd,khd->hqk", q, k.repeat_interleave(hq // hkv, 1)).abs().max() * d ** -0.5).item()
            err = (out - ref).abs().max().item()
            assert err <= v.abs().max().item() * (2 * top * 2.0 ** -21 + 2.0 ** -20), (causal, hq, err)
    assert ops.last_error() == 0


@pytest.mark.parametrize("d", [64, 128])
def test_fp32_values_without_three_parts(d):
    """Infinities, NaN, the largest floats and subnormal ones: heads that hold them come out as from the FMA kernel."""
    from axono_b200 import ops

    for causal in (True, False):
        q, k, v = tensors(200, 260, 8, 4, d, torch.float32)
        k[70, 0, 3] = float("-inf")
        v[199, 1, 2] = 1e-39
        v[10, 2, 0] = float("nan")
        q[150, 7, 1] = 3.4e38  # a head of KV head 3
        out, ref = ops.scaled_dot_product_attention(q, k, v, causal), without_scratch(q, k, v, causal)
        assert torch.equal(torch.nan_to_num(out, 9e9, 8e9, 7e9), torch.nan_to_num(ref, 9e9, 8e9, 7e9))
    assert ops.last_error() == 0


@pytest.mark.parametrize("source", ["k", "v", "q"])
@pytest.mark.parametrize("sq,skv,hq,hkv", [(200, 260, 8, 4), (1536, 1536, 16, 8)])  # the second divides keys where nothing is masked
def test_fp32_only_the_flagged_head_is_done_over(source, sq, skv, hq, hkv):
    """One value without three parts, in one head's keys or values or in one query row of the last block: that KV head comes out
    as from the FMA kernel, the others bit for bit as from clean inputs."""
    from axono_b200 import ops

    for causal in (True, False):
        q, k, v = tensors(sq, skv, hq, hkv, 64, torch.float32)
        clean = ops.scaled_dot_product_attention(q, k, v, causal)
        {"k": k, "v": v, "q": q}[source][sq - 1 if source == "q" else 100, 2 if source == "q" else 1, 5] = 1e-33
        out, fma = ops.scaled_dot_product_attention(q, k, v, causal), without_scratch(q, k, v, causal)
        flagged = torch.arange(hq, device="cuda") // (hq // hkv) == 1
        assert torch.equal(out[:, flagged], fma[:, flagged]) and not torch.equal(fma[:, flagged], clean[:, flagged])
        assert torch.equal(out[:, ~flagged], clean[:, ~flagged])
    assert ops.last_error() == 0


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("qo,ko,vo", [(0, 2, 0), (2, 2, 0), (0, 0, 4), (2, 2, 4)])
def test_fp32_with_common_offsets(d, qo, ko, vo):
    """Where the sums' terms have one sign, truncation has too: the error stays below that of the FMA kernel, which rounds."""
    from axono_b200 import ops

    for sq, skv, causal in ((300, 300, True), (300, 2700, False), (1536, 1536, False)):
        q, k, v = tensors(sq, skv, 4, 2, d, torch.float32)
        q, k, v = q + qo, k + ko, v + vo
        ref = attention(q, k, v, causal)
        err = [(out.double() - ref).norm().item() for out in (ops.scaled_dot_product_attention(q, k, v, causal), without_scratch(q, k, v, causal))]
        assert err[0] <= err[1], (sq, skv, err)
    assert ops.last_error() == 0


def plain(q, k, v, causal, dtype, tol):
    out, ref = without_scratch(q, k, v, causal).double(), attention(q, k, v, causal)
    group = q.shape[1] // k.shape[1]
    top = (torch.einsum("qhd,khd->hqk", q.float(), k.float().repeat_interleave(group, 1)).abs().max() * q.shape[2] ** -0.5).item()
    bound = v.float().abs().max().item() * (2 * top * 2.0 ** -21 + 2.0 ** -20) + (ref.abs() * tol if tol else 0.0)
    assert ((out - ref).abs() <= bound).all()


@pytest.mark.parametrize("hq,hkv,d", [(16, 8, 128), (4, 4, 64), (6, 2, 80), (16, 2, 96), (3, 1, 8)])
@pytest.mark.parametrize("sq,skv", [(16, 16), (70, 300), (300, 70), (257, 257), (33, 2049)])
def test_fp32_without_scratch(hq, hkv, d, sq, skv):
    """The FMA kernel in fp32, which serves calls without scratch and the heads whose values have no three parts.  A score is off
    by 2^-21 of the largest one, sums and the result by 2^-20."""
    for causal in (True, False):
        plain(*tensors(sq, skv, hq, hkv, d, torch.float32), causal, torch.float32, 0.0)


@pytest.mark.parametrize("hq,hkv,d", [(4, 2, 12), (3, 3, 20), (8, 1, 68), (4, 2, 100), (4, 2, 64), (4, 2, 128)])
@pytest.mark.parametrize("sq,skv", [(16, 16), (70, 300), (257, 257), (33, 1025)])
def test_fp16_on_the_fma_kernel(hq, hkv, d, sq, skv):
    """fp16 head sizes off the multiples of 8, and (64 and 128) tensors one element off 16 bytes: the result's rounding is 2^-11 of
    it, the rest as in fp32."""
    for causal in (True, False):
        q, k, v = tensors(sq, skv, hq, hkv, d, torch.float16)
        if d % 8 == 0:
            q, k, v = (torch.cat([t.new_zeros(1), t.flatten()])[1:].view(t.shape) for t in (q, k, v))
            assert k.data_ptr() % 16
        plain(q, k, v, causal, torch.float16, 2.0 ** -11)


@pytest.mark.parametrize("d", [64, 80])
@pytest.mark.parametrize("offset", [0, 4])
def test_fp16_narrow_sums_do_not_drift(d, offset):
    """Sums over thousands of values: the tensor core's truncation pulls them towards zero with each of the 8 products of a tile of 64
    keys, by some 1e-5 over the 16 tiles after which a sum starts anew, which adds its square to that of the result's rounding
    (2.2e-4): a thousandth above the FMA kernel's error at most."""
    from axono_b200 import ops

    q, k, v = tensors(8192, 8192, 4, 2, d, torch.float16)
    v = v + offset
    off = [torch.cat([t.new_zeros(1), t.flatten()])[1:].view(t.shape) for t in (q, k, v)]  # off 16 bytes: the FMA kernel
    ref = attention(q, k, v, False)
    err = [(ops.scaled_dot_product_attention(*args, False).double() - ref).norm().item() for args in ((q, k, v), off)]
    assert err[0] <= 1.001 * err[1], err


@pytest.mark.parametrize("d", [8, 64, 128])
@pytest.mark.parametrize("sq,skv,hq,hkv", [(256, 4100, 2, 1), (300, 1500, 3, 3), (1300, 1300, 2, 2), (2700, 2700, 16, 8),
                                           (2305, 900, 16, 16), (3000, 3100, 4, 2)])
def test_fp16_keys_divided_among_blocks(d, sq, skv, hq, hkv):
    """Blocks of rows whose keys several CTAs share: the parts of a row are joined in fp32.  The result's rounding is 2^-11 of
    it; a weight is off by 2^-21 of the largest score (its sum of products and its exponent) and, for heads of 128, by its
    rounding to fp16, 2^-11; and a small weight, as multiples of 2^-24 of a sum that is at least one, by 2^-25.  The same
    bound for undivided blocks."""
    from axono_b200 import ops

    for causal in (True, False):
        q, k, v = tensors(sq, skv, hq, hkv, d, torch.float16, 3.0)
        ref, mass = attention(q, k, v, causal), attention(q, k, v.abs(), causal)
        top = (torch.einsum("qhd,khd->hqk", q.float(), k.float().repeat_interleave(hq // hkv, 1)).abs().max() * d ** -0.5).item()
        weight = 2 * top * 2.0 ** -21 + 2.0 ** -20 + (2.0 ** -11 if d == 128 else 0.0)
        for out in (ops.scaled_dot_product_attention(q, k, v, causal), without_scratch(q, k, v, causal)):
            err = (out.double() - ref).abs()
            small = 2.0 ** -25 * v.double().abs().sum(0).repeat_interleave(hq // hkv, 0)
            assert (err <= ref.abs() * 2.0 ** -11 + weight * mass + small + 2.0 ** -24).all(), (causal, err.max())
    assert ops.last_error() == 0


@pytest.mark.parametrize("sq,d", [(40000, 64), (60000, 128)])
def test_fp16_long_prompts_of_one_head(sq, d):
    """Plans of more than 448 blocks and parts: the last blocks, which are divided, and some others, within the bound above."""
    from axono_b200 import ops

    q, k, v = tensors(sq, sq, 1, 1, d, torch.float16)
    out = ops.scaled_dot_product_attention(q, k, v, False)
    weight = 2 * (q.float().norm(dim=-1).max() * k.float().norm(dim=-1).max() * d ** -0.5).item() * 2.0 ** -21 + 2.0 ** -20 + 2.0 ** -11
    small = 2.0 ** -25 * v.double().abs().sum(0)
    for at in (0, sq // 2, sq - 2000, sq - 1000):
        rows = slice(at, at + 1000)
        ref, mass = attention(q[rows], k, v, False), attention(q[rows], k, v.abs(), False)
        assert ((out[rows].double() - ref).abs() <= ref.abs() * 2.0 ** -11 + weight * mass + small + 2.0 ** -24).all()
    assert ops.last_error() == 0


@pytest.mark.parametrize("d", [8, 64, 72])
@pytest.mark.parametrize("sq,skv,hq,hkv", [(200, 260, 4, 2), (300, 4100, 2, 1), (1300, 1300, 2, 2)])  # the later two divide keys
def test_fp16_narrow_heads_with_infinities(d, sq, skv, hq, hkv):
    """Infinite and NaN values, keys and queries: rows that see them come out as the definition's, rows that the mask keeps
    from them as if they were not there."""
    from axono_b200 import ops

    inf, nan = float("inf"), float("nan")
    for causal in (True, False):
        q, k, v = tensors(sq, skv, hq, hkv, d, torch.float16)
        clean = ops.scaled_dot_product_attention(q, k, v, causal)
        at, group = {0: inf, 1: -inf, 2: nan}, hq // hkv
        for head in range(hkv):
            vb = v.clone()
            for c, x in at.items():
                vb[100, head, c] = x
            want = clean.clone()
            seen = torch.arange(sq, device="cuda") >= (100 if causal else 0)
            for c, x in at.items():
                for h in range(head * group, (head + 1) * group):
                    want[seen, h, c] = x
            out = ops.scaled_dot_product_attention(q, k, vb, causal)
            torch.testing.assert_close(out, want, rtol=2.0 ** -10, atol=1e-5, equal_nan=True)
        kb, qb = k.clone(), q.clone()
        kb[100, 0, 3], qb[150, hq - 1, 4] = nan, inf  # NaN scores; scores of +inf (and -inf: nothing)
        out = ops.scaled_dot_product_attention(qb, kb, v, causal)
        want = clean.clone()
        want[seen, 0:group] = nan
        want[150, hq - 1] = nan
        torch.testing.assert_close(out, want, rtol=2.0 ** -10, atol=1e-5, equal_nan=True)
    assert ops.last_error() == 0


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("d", [64, 128])
def test_plain_call_leaves_the_workspace_alone(dtype, d):
    """axb200_sdpa writes no workspace where it asks for none, so that calls on several streams may be given one buffer."""
    from axono_b200 import _capi

    lib, dt = _capi.lib(), _capi.FLOAT32 if dtype == torch.float32 else _capi.FLOAT16
    q, k, v = tensors(1300, 1300, 2, 2, d, dtype)
    buf, out = torch.full((64 << 20,), 77, dtype=torch.uint8, device="cuda"), torch.empty_like(q)
    assert lib.axb200_sdpa_workspace_bytes(1300, 2, 2, d, 1300, dt) == 0
    for causal in (0, 1):
        assert lib.axb200_sdpa(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), 1300, 2, 2, d, 1300, causal, dt, buf.data_ptr(),
                               buf.numel(), torch.cuda.current_stream().cuda_stream) == 0
        assert (buf == 77).all()


ROWS_THEN_DECODE = """
import torch
from axono_b200 import ops
from torch.profiler import ProfilerActivity, profile

rnd = lambda *s: torch.randn(s, device="cuda")
held = []
for i in range(80):  # ever other addresses are free
    q, k, v = rnd(4, 8, 64), rnd(4096, 8, 64), rnd(4096, 8, 64)
    held += [ops.scaled_dot_product_attention(q, k, v), torch.empty(4 << 20, dtype=torch.uint8, device="cuda")]
ops.workspace("cuda", 256 << 20)  # a buffer at an address not seen before
with profile(activities=[ProfilerActivity.CUDA]) as prof:
    ops.gqa_decode_attention(rnd(1, 8, 64), k, v)
    torch.cuda.synchronize()
names = [e.key for e in prof.key_averages()]
assert any("gqa_split" in n for n in names), names
assert not any("gqa_combine" in n for n in names), names
assert ops.last_error() == 0
"""


def test_row_by_row_calls_leave_counters_to_others():
    """A workspace's address takes one of 64 regions of counters for good: calls of a few rows, however many, take one in all,
    and a buffer first seen after them still gets its own (without one the merge is a launch of its own)."""
    import subprocess
    import sys

    from conftest import ROOT

    subprocess.run([sys.executable, "-c", ROWS_THEN_DECODE], cwd=ROOT, check=True, timeout=300)


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_prompts_where_memory_is_short(dtype, monkeypatch):
    """An allocation of scratch that fails: the call goes on without."""
    from axono_b200 import ops

    q, k, v = tensors(1300, 1300, 2, 2, 64, dtype)
    refused, empty = [], torch.empty

    def short(*size, **kw):
        if kw.get("dtype") is torch.uint8:
            refused.append(size)
            raise torch.OutOfMemoryError("no memory")
        return empty(*size, **kw)

    ops.workspace(q.device, 256)
    monkeypatch.setattr(torch, "empty", short)
    out = ops.scaled_dot_product_attention(q, k, v, True)
    assert refused and torch.equal(out, without_scratch(q, k, v, True)) and ops.last_error() == 0


@pytest.mark.parametrize("d", [16, 64, 80, 128])
@pytest.mark.parametrize("sq,skv", [(17, 63), (128, 64), (129, 65), (255, 1024), (256, 1025), (384, 1088), (40, 2113)])
def test_fp16_at_the_edges_of_key_tiles(d, sq, skv):
    """Tiles of 64 keys, of which the scores of two are ahead, and sums of narrow heads that start anew every sixteen: one tile, a
    tile and a key, one group of tiles and the next.  The bound of `test_fp16_keys_divided_among_blocks`."""
    from axono_b200 import ops

    for causal in (True, False):
        q, k, v = tensors(sq, skv, 2, 1, d, torch.float16, 2.0)
        ref, mass = attention(q, k, v, causal), attention(q, k, v.abs(), causal)
        top = (torch.einsum("qhd,khd->hqk", q.float(), k.float().repeat_interleave(2, 1)).abs().max() * d ** -0.5).item()
        weight = 2 * top * 2.0 ** -21 + 2.0 ** -20 + (2.0 ** -11 if d == 128 else 0.0)
        small = 2.0 ** -25 * v.double().abs().sum(0).repeat_interleave(2, 0)
        for out in (ops.scaled_dot_product_attention(q, k, v, causal), without_scratch(q, k, v, causal)):
            assert ((out.double() - ref).abs() <= ref.abs() * 2.0 ** -11 + weight * mass + small + 2.0 ** -24).all()
    assert ops.last_error() == 0
