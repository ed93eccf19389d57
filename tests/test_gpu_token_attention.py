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
