"""Float32 prompt portions in tiles against the general kernel (a block per row and head) and float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("heads,kv_heads,page", [(4, 2, 16), (3, 3, 8), (8, 1, 4)])
@pytest.mark.parametrize("window", [0, 1, 70])
@pytest.mark.parametrize("lengths,befores", [((64, 1, 65), (0, 90, 3)), ((2, 63), (127, 1)), ((200,), (64,))])
def test_tiles_are_the_general_kernel(hd, heads, kv_heads, page, window, lengths, befores):
    from tiny_llm_infer_b200 import ops
    from tiny_llm_infer_b200.engine.batch import StepContext
    g = torch.Generator(device=DEV).manual_seed(3)
    seg, tiles, dec, row = [], [], [], 0
    for s, (n, p0) in enumerate(zip(lengths, befores)):
        seg.append([s, row, n, p0])
        if n == 1:
            dec.append(row)
        else:
            tiles += [(s, off) for off in range(0, n, 64)]
        row += n

    def ints(v):
        return torch.tensor(v, dtype=torch.int32, device=DEV)
    longest = max(n + p for n, p in zip(lengths, befores))
    ctx = StepContext(tokens=row, token_ids=None, positions=ints([p0 + i for _, _, n, p0 in seg for i in range(n)]),
                      token_slot=ints([s for s, _, n, _ in seg for _ in range(n)]), want_rows=None, segments=[], seg_info=ints(seg),
                      dec_rows=ints(dec), n_dec=len(dec), pf_tiles=ints(tiles), n_tiles=len(tiles), max_context=longest, max_segment=max(lengths))
    pages = -(-longest // page)
    table = torch.randperm(len(lengths) * pages, generator=g, device=DEV).to(torch.int32).view(len(lengths), pages)
    if window == 1:
        table[0, 0] = -1 if befores[0] >= page else table[0, 0]     # a page that the window has passed
    cache = torch.randn(len(lengths) * pages, 2, kv_heads, page, hd, generator=g, device=DEV)
    q = torch.randn(row, heads * hd, generator=g, device=DEV) * 3
    out = []
    for c in (ctx, None):
        o, before = torch.empty_like(q), ops.launches
        ops.paged_attention(q, cache, ctx.positions, ctx.token_slot, table, page, heads, kv_heads, hd, window or None, hd ** -0.5, o, ctx=c)
        assert ops.launches - before == (1 if c is None or not dec else 2)
        out.append(o.double())
    want = torch.empty_like(out[0])
    for s, first, n, p0 in seg:
        k, v = (cache[table[s].long().clamp(min=0), i].permute(0, 2, 1, 3).reshape(-1, kv_heads, hd).double() for i in (0, 1))
        for i in range(n):
            lo = max(0, p0 + i + 1 - window) if window else 0
            kk, vv = (x[lo:p0 + i + 1].repeat_interleave(heads // kv_heads, 1) for x in (k, v))
            w = torch.softmax(torch.einsum("hd,jhd->hj", q[first + i].double().view(heads, hd), kk) * hd ** -0.5, 1)
            want[first + i] = torch.einsum("hj,jhd->hd", w, vv).flatten()
    tiled, general = ((o - want).norm() / want.norm() for o in out)
    # both sum in float32; the tiles may not be further off than the general kernel but for a few roundings of 2^-24
    assert tiled <= 1.5 * general + 2.0 ** -23, (float(tiled), float(general))
    # a token's key and value reach no row before it, whatever they are
    for s, first, n, p0 in seg:
        if n > 1:
            at = p0 + n - 1
            cache[table[s, at // page].long(), :, :, at % page] = float("nan") if s else float("inf")
    o = torch.empty_like(q)
    ops.paged_attention(q, cache, ctx.positions, ctx.token_slot, table, page, heads, kv_heads, hd, window or None, hd ** -0.5, o, ctx=ctx)
    last = torch.zeros(row, dtype=torch.bool, device=DEV)
    last[[first + n - 1 for _, first, n, _ in seg if n > 1]] = True
    assert torch.equal(o.double()[~last], out[0][~last])


@pytest.mark.parametrize("hd", [64, 128])
def test_portions_of_no_request_become_zero(hd):
    from tiny_llm_infer_b200 import ops
    from tiny_llm_infer_b200.engine.batch import StepContext
    lengths, slots, heads, kv_heads, page = (70, 40, 1), (-1, 0, -1), 4, 2, 16

    def ints(v):
        return torch.tensor(v, dtype=torch.int32, device=DEV)
    rows = sum(lengths)
    ctx = StepContext(tokens=rows, token_ids=None, positions=ints([i for n in lengths for i in range(n)]),
                      token_slot=ints([s for s, n in zip(slots, lengths) for _ in range(n)]), want_rows=None, segments=[],
                      seg_info=ints([[-1, 0, 70, 0], [0, 70, 40, 0], [-1, 110, 1, 0]]), dec_rows=ints([110]), n_dec=1,
                      pf_tiles=ints([(0, 0), (0, 64), (1, 0)]), n_tiles=3, max_context=70, max_segment=70)
    g = torch.Generator(device=DEV).manual_seed(8)
    table = ints([[2, 0, 1]])
    cache = torch.randn(3, 2, kv_heads, page, hd, generator=g, device=DEV)
    q = torch.randn(rows, heads * hd, generator=g, device=DEV)
    out = []
    for c in (ctx, None):
        o = torch.full_like(q, float("nan"))
        ops.paged_attention(q, cache, ctx.positions, ctx.token_slot, table, page, heads, kv_heads, hd, None, hd ** -0.5, o, ctx=c)
        out.append(o)
    for o in out:
        assert (o[:70] == 0).all() and (o[110:] == 0).all()
    assert torch.allclose(out[0][70:110], out[1][70:110], rtol=1e-5, atol=1e-5)
