"""`ops.row_chain`, the products and norms between two attention calls of a decode step in one launch, against the same in 64 bits
with the roundings of its stages to half precision, and the tower's step that is made of it."""
import pytest
import torch

from axono_b200 import ops
from axono_b200.decode import TextTower, TextTowerConfig

pytestmark = pytest.mark.gpu


def _inputs(rows, attn, width, ff, nxt, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)

    def rnd(*shape, gain=1.0):
        return (torch.randn(shape, generator=g, device="cuda") * gain).half()

    x, residual = rnd(rows, attn), rnd(rows, width)
    return x, {"w_o": rnd(width, attn, gain=attn ** -0.5), "residual": residual, "norm1": 1 + rnd(width, gain=0.1),
               "w_gate_up": rnd(2 * ff, width, gain=width ** -0.5), "w_down": rnd(width, ff, gain=ff ** -0.5),
               "norm2": 1 + rnd(width, gain=0.1), "w_next": rnd(nxt, width, gain=width ** -0.5)}


def _plain(x, w, eps):
    d = {k: v.double() for k, v in w.items()}

    def stored(t):
        return t.half().double()

    def normed(t, weight):
        return stored(t / torch.sqrt((t * t).mean(-1, keepdim=True) + eps) * weight)

    y = stored(x.double() @ d["w_o"].T + d["residual"])
    gate, up = (normed(y, d["norm1"]) @ d["w_gate_up"].T).chunk(2, -1)
    y = stored(stored(gate * torch.sigmoid(gate) * up) @ d["w_down"].T + y)
    return y, normed(y, d["norm2"]) @ d["w_next"].T


# widths below, at and above what 32 warps hold with a block of 64 each; more units of 32 rows than pairs of SMs (next 4864), fewer,
# a last unit of 8 rows and of 1
SIZES = [(1, 64, 64, 64, 8), (8, 2048, 2048, 6144, 4096), (2, 192, 320, 1088, 4864), (8, 4096, 2048, 512, 1), (7, 1024, 1984, 3008, 1000),
         (5, 2048, 4096, 12288, 64), (6, 128, 2112, 640, 264), (3, 8192, 4032, 256, 72)]


@pytest.mark.parametrize("rows,attn,width,ff,nxt", SIZES)
def test_row_chain(rows, attn, width, ff, nxt):
    assert ops.row_chain_supported(rows, attn, width, ff, nxt, torch.float16)
    x, w = _inputs(rows, attn, width, ff, nxt)
    for _ in range(2):  # the counter of the meetings is left ready for the next launch
        res, out = ops.row_chain(x, eps=1e-6, **w)
    want_res, want = _plain(x, w, 1e-6)
    # a rounding to half may fall the other way wherever the sums' order matters: half a unit at each of the roundings on the
    # way, values of about one to four
    unit = torch.finfo(torch.float16).eps
    assert (res.double() - want_res).norm() <= 2 * unit * want_res.norm()
    assert (out.double() - want).norm() <= 2 * unit * want.norm()
    assert (out.double() - want).abs().max() <= 16 * unit * want.abs().max()
    assert ops.last_error() == 0


@pytest.mark.parametrize("rows,attn,width,ff,nxt", [(0, 64, 64, 64, 8), (9, 64, 64, 64, 8), (8, 96, 64, 64, 8), (8, 64, 100, 64, 8),
                                                    (8, 64, 64, 72, 8), (8, 64, 4160, 64, 8), (1, 64, 64, 64, 0)])
def test_row_chain_sizes_it_does_not_take(rows, attn, width, ff, nxt):
    assert not ops.row_chain_supported(rows, attn, width, ff, nxt, torch.float16)
    assert not ops.row_chain_supported(8, 64, 64, 64, 8, torch.float32)


def test_row_chain_refuses_other_types_and_strides():
    x, w = _inputs(4, 64, 64, 64, 8)
    with pytest.raises(RuntimeError):
        ops.row_chain(x, eps=1e-6, **(w | {"residual": w["residual"].float()}))
    with pytest.raises(RuntimeError):
        ops.row_chain(x, eps=1e-6, **(w | {"w_down": w["w_down"].t().contiguous().t()}))
    with pytest.raises(RuntimeError):
        ops.row_chain(torch.randn(4, 96, device="cuda").half()[:, :64], eps=1e-6, **w)


def test_row_chain_in_a_graph_and_on_two_streams():
    x, w = _inputs(8, 2048, 2048, 6144, 4096)
    _, want = ops.row_chain(x, eps=1e-6, **w)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(3):
            _, out = ops.row_chain(x, eps=1e-6, **w)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        others = [ops.row_chain(x, eps=1e-6, **w)[1] for _ in range(20)]
    for _ in range(10):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want) and all(torch.equal(o, want) for o in others)
    assert ops.last_error() == 0


@pytest.mark.parametrize("made", ["w_o", "w_gate_up"])
def test_row_chain_waits_for_weights_that_the_launch_before_it_writes(made):
    """The launch in front of the chain makes one of its matrices (the rotated q of 4096 sequences), and lets dependents begin long
    before it is done."""
    from axono_b200.kv_cache import PagedKVCache

    batch, heads, d = 4096, 16, 128
    width, ff = (4096, 256) if made == "w_o" else (2048, 2048)
    x, w = _inputs(8, 2048, width, ff, 128)
    g = torch.Generator(device="cuda").manual_seed(5)
    qkv = [(torch.randn((batch, (heads + 2) * d), generator=g, device="cuda") * 2048 ** -0.5).half() for _ in range(4)]
    cache = PagedKVCache(1, batch, 1, d, 64)

    def step(t):
        cache.seq_lens.zero_()
        w[made] = cache.append_qkv(0, t, heads).view(batch, heads * d)
        return ops.row_chain(x, eps=1e-6, **w)

    outs = [step(t) for t in qkv * 3]
    for i, (_, out) in enumerate(outs):
        cache.seq_lens.zero_()
        w[made] = cache.append_qkv(0, qkv[i % 4], heads).view(batch, heads * d)
        torch.cuda.synchronize()
        assert torch.equal(out, ops.row_chain(x, eps=1e-6, weights_ready=True, **w)[1])
    assert ops.last_error() == 0


def test_row_chain_whose_waits_run_out_returns():
    """Two pairs of CTAs have 64 MB of the first product each, the others meet without them after 100 us: they go on, the call returns with
    the flag set, and the next one is as the one before."""
    from axono_b200 import _capi

    lib = _capi.lib()
    x, w = _inputs(8, 1 << 20, 64, 2048, 4864)
    _, want = ops.row_chain(x, eps=1e-6, **w)
    assert ops.last_error() == 0
    try:
        assert lib.axb200_set_wait_limit_ns(1) == 0
        ops.row_chain(x, eps=1e-6, **w)
        torch.cuda.synchronize()
        assert ops.last_error() == 1  # AXB200_ERR_WAIT_TIMEOUT
    finally:
        lib.axb200_set_wait_limit_ns(2_000_000_000)
    for _ in range(2):
        assert torch.equal(ops.row_chain(x, eps=1e-6, **w)[1], want)
    assert ops.last_error() == 0


def test_row_chain_on_streams_of_unequal_priority():
    """Each launch needs all SMs at once, with ordinary launches between them and other streams' in front."""
    x, w = _inputs(8, 2048, 2048, 6144, 4096)
    _, want = ops.row_chain(x, eps=1e-6, **w)
    square = torch.randn((2048, 2048), device="cuda").half()
    streams = [torch.cuda.Stream(priority=p) for p in (0, -1, -2)]
    outs = []
    for s in streams:
        s.wait_stream(torch.cuda.current_stream())
    for i in range(30):
        for j, s in enumerate(streams):
            with torch.cuda.stream(s):
                if (i + j) % 3 == 0:
                    ops.silu_mul_rows(square @ square, 1024)
                outs.append(ops.row_chain(x, eps=1e-6, weights_ready=bool(i & 1), **w)[1])
    torch.cuda.synchronize()
    assert all(torch.equal(o, want) for o in outs) and ops.last_error() == 0


@pytest.mark.parametrize("batch,vocab", [(1, 1000), (8, 1000), (9, 1000), (8, 40000)])
def test_tower_step_with_and_without_the_chain(batch, vocab):
    """The step with two launches per layer (and single operators for a narrow tower's many logits) against the step of single
    operators, from the same state."""
    cfg = TextTowerConfig(hidden=512, intermediate=1024, n_q_heads=8, n_kv_heads=4, head_dim=64, vocab=vocab, n_layers=3, mrope_section=(12, 10, 10))
    towers = [TextTower(cfg, batch, 192, seed=3, lt_gemm=lt) for lt in (True, False)]
    assert towers[0]._chains() == (batch <= 8) and not towers[1]._chains()
    assert towers[0]._chain_gains(vocab) == (batch <= 8 and vocab == 1000)
    lens = [64 + 5 * b % 64 for b in range(batch)]
    g = torch.Generator(device="cuda").manual_seed(4)
    kv = [[torch.randn((batch, 128, 4, 64), generator=g, device="cuda").half() for _ in range(2)] for _ in range(cfg.n_layers)]
    for tower in towers:
        for i, (k, v) in enumerate(kv):
            tower.cache.fill(i, k, v, lens)
        tower.set_state(list(range(batch)), lens)
    for _ in range(2):
        for tower in towers:
            tower.decode_step()
        a, b = (t.last_logits.double() for t in towers)
        # three layers of half precision whose roundings fall differently
        assert (a - b).norm() <= 8 * torch.finfo(torch.float16).eps * b.norm()
        towers[1].token_ids.copy_(towers[0].token_ids)
    assert torch.equal(towers[0].cache.seq_lens, towers[1].cache.seq_lens) and ops.last_error() == 0


def _strided(t):
    return torch.stack([t, t], dim=-1)[..., 0]


def _shifted(t):
    flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    return flat[1:].view(t.shape).copy_(t)


@pytest.mark.parametrize("name", ["input_ln", "qkv", "o", "post_ln", "gate_up", "down", "embed", "final_ln"])
@pytest.mark.parametrize("view", [_strided, _shifted])
def test_tower_with_weights_that_the_chain_does_not_take(name, view):
    """A program's own weights as views: the step runs as single operators, with the same results as with contiguous ones."""
    cfg = TextTowerConfig(hidden=256, intermediate=512, n_q_heads=4, n_kv_heads=2, head_dim=64, vocab=300, n_layers=2, mrope_section=(12, 10, 10))
    towers = [TextTower(cfg, 2, 64, seed=3, row_chain=chain) for chain in (True, False)]
    holder, key = (towers[0].layers[1], name) if name in towers[0].layers[1] else (vars(towers[0]), name)
    assert towers[0]._chains() and not towers[1]._chains()
    holder[key] = view(holder[key])
    assert not towers[0]._chains()
    for tower in towers:
        tower.set_state([1, 2], [0, 0])
        tower.decode_step()
    a, b = (t.last_logits.double() for t in towers)
    assert (a - b).norm() <= 4 * torch.finfo(torch.float16).eps * b.norm()  # a product's algorithm depends on its operands' alignment
    assert ops.last_error() == 0
