"""fp32 decode attention at the edges of its tiles: head sizes that fill a 64- or 128-wide tile in part, groups of heads,
lengths around tiles and chunks, windows.  Checked against the definition in fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

LENGTHS = [1, 7, 63, 64, 65, 257, 1023, 1025, 4097]
# A weight's argument is a sum of up to 128 products (2^-24 of it at each step, about 2^-21 in all), the result a sum of
# thousands of weighted values in a few partial sums.
TOL = 2.0 ** -19


def reference(q, k, v):
    group = q.shape[0] // k.shape[1]
    s = torch.einsum("hd,nhd->hn", q.double(), k.double().repeat_interleave(group, 1)) * q.shape[1] ** -0.5
    return torch.einsum("hn,nhd->hd", torch.softmax(s, -1), v.double().repeat_interleave(group, 1))


def close(out, ref):
    assert (out.double() - ref).abs().max() <= TOL * ref.abs().max()


@pytest.mark.parametrize("d", [8, 32, 60, 64, 68, 96, 124, 128])
@pytest.mark.parametrize("hq,hkv", [(2, 2), (6, 3), (8, 2), (8, 1)])
def test_fp32_head_sizes(d, hq, hkv):
    from axono_b200 import ops
    from axono_b200.kv_cache import PagedKVCache

    g = torch.Generator(device="cuda").manual_seed(d)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    q, k, v = rnd(len(LENGTHS), hq, d), rnd(len(LENGTHS), max(LENGTHS), hkv, d), rnd(len(LENGTHS), max(LENGTHS), hkv, d)
    refs = [reference(q[i], k[i, :n], v[i, :n]) for i, n in enumerate(LENGTHS)]
    for i, n in enumerate(LENGTHS):
        close(ops.gqa_decode_attention(q[i:i + 1], k[i, :n], v[i, :n])[0], refs[i])
    cache = PagedKVCache(1, len(LENGTHS), hkv, d, max(LENGTHS), dtype=torch.float32)
    for pool in (*cache.k_pages, *cache.v_pages):
        pool.fill_(float("nan"))  # what lies behind a sequence's end takes no part
    cache.fill(0, k, v, LENGTHS)
    for i, n in enumerate(LENGTHS):  # the last page of each sequence behind its end
        at, slot = int(cache.block_table[i, (n - 1) // 64]), (n - 1) % 64 + 1
        cache.k_pages[0][at, :, slot:] = float("nan")
        cache.v_pages[0][at, :, slot:] = float("nan")
    out = cache.attend(0, q)
    for i in range(len(LENGTHS)):
        close(out[i], refs[i])
    out = cache.attend(0, q, window=70)
    for i, n in enumerate(LENGTHS):
        close(out[i], reference(q[i], k[i, max(0, n - 70):n], v[i, max(0, n - 70):n]))
    assert ops.last_error() == 0


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("hq,hkv", [(4, 2), (6, 2), (3, 3)])
def test_heads_of_four(dtype, hq, hkv):
    """The kernel for any head size at its smallest: two heads' merge of the chunks takes more shared memory than the tiles do.
    Tensors one element off 16 bytes, so that fp32 comes here too; fp16 rounds the result by 2^-11."""
    from axono_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(hq)

    def off(*s):
        n = s[0] * s[1] * s[2]
        return torch.randn(n + 1, generator=g, device="cuda").to(dtype)[1:].view(s)

    for n in (1, 64, 300, 1025, 4097):
        q, k, v = off(1, hq, 4), off(n, hkv, 4), off(n, hkv, 4)
        out, ref = ops.gqa_decode_attention(q, k, v)[0].double(), reference(q[0], k, v)
        assert ((out - ref).abs() <= TOL * ref.abs().max() + (ref.abs() * 2.0 ** -11 if dtype == torch.float16 else 0.0)).all()
    assert ops.last_error() == 0
