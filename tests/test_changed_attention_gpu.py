"""Prompt portions through the tcgen05 kernel with a changed score or output, against the general kernel (one block per row
and head over all keys, float32 throughout), for every change alone and for mixtures of them."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV, D, PAGE = "cuda:0", 128, 16
FORMS = {
    "cap": dict(softcap=5.0), "slopes": dict(slopes=True), "chunk": dict(chunk=96), "chunk past a window": dict(chunk=256, window=70),
    "sink of one": dict(sink=True), "gate": dict(gate="elements"), "gate, rows of odd length": dict(gate="odd"),
    "gate per head": dict(gate="heads"), "cap, window, learned sink, gate per head": dict(softcap=2.0, window=150, sink=True, learned=True, gate="heads"),
    "cap, slopes, chunk, sink, gate": dict(softcap=9.0, slopes=True, chunk=200, sink=True, gate="elements"),
}


def context(lengths, befores):
    from tiny_llm_infer_b200.engine.batch import StepContext
    seg, tiles, row = [], [], 0
    for s, (n, p0) in enumerate(zip(lengths, befores)):
        seg.append([s, row, n, p0])
        tiles += [(s, off) for off in range(0, n, 64)]
        row += n
    tiles.sort(key=lambda t: (t[1] % 256 != 0, t[1] % 128 != 0))

    def ints(v):
        return torch.tensor(v, dtype=torch.int32, device=DEV)
    return StepContext(tokens=row, token_ids=None, positions=ints([p0 + i for _, _, n, p0 in seg for i in range(n)]),
                       token_slot=ints([s for s, _, n, _ in seg for _ in range(n)]), want_rows=None, segments=[], seg_info=ints(seg),
                       dec_rows=ints([]), n_dec=0, pf_tiles=ints(tiles), n_tiles=len(tiles),
                       n_tiles128=sum(t[1] % 128 == 0 for t in tiles), n_tiles256=sum(t[1] % 256 == 0 for t in tiles),
                       max_context=max(n + p for n, p in zip(lengths, befores)), max_segment=max(lengths))


@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("heads,kv_heads,lengths,befores", [
    (4, 2, (130, 2, 257), (0, 333, 61)),          # two heads of a group per block; a row past a tile, two rows, two tiles and one
    (3, 3, (300,), (17,)),                        # two blocks of positions per block
    (2, 1, (65,), (1500,)),                       # few rows and many keys: their keys cut into runs
])
def test_changes_of_the_score_and_the_output(form, heads, kv_heads, lengths, befores):
    from tiny_llm_infer_b200 import ops
    f = dict(FORMS[form])
    g = torch.Generator(device=DEV).manual_seed(5)

    def randn(*shape):
        return torch.randn(*shape, generator=g, device=DEV)
    ctx = context(lengths, befores)
    pages = -(-ctx.max_context // PAGE)
    order = torch.randperm(len(lengths) * pages, generator=g, device=DEV).to(torch.int32).view(len(lengths), pages)
    planes = [randn(len(lengths) * pages, kv_heads, PAGE, D).bfloat16() for _ in range(2)]
    q = randn(ctx.tokens, heads * D).bfloat16()
    gate = None
    if f.get("gate") == "heads":
        gate = randn(ctx.tokens, heads + 3).bfloat16()[:, 2:2 + heads]
    elif f.get("gate"):
        at = 2 if f["gate"] == "odd" else 8
        gate = randn(ctx.tokens, heads * D + (10 if f["gate"] == "odd" else 16)).bfloat16()[:, at:at + heads * D]
    kw = dict(softcap=f.get("softcap", 0.0), chunk=f.get("chunk", 0), window=f.get("window", 0), sink=f.get("sink", False),
              slopes=torch.rand(heads, generator=g, device=DEV) * 0.05 if f.get("slopes") else None, gate=gate,
              gate_per_head=f.get("gate") == "heads", sink_logits=randn(heads) if f.get("learned") else None)
    out = []
    for c in (ctx, None):
        o, before = torch.empty_like(q), ops.tcgen05_calls
        ops.attention_biased(q, *planes, ctx.positions, ctx.token_slot, order, PAGE, heads, kv_heads, D, D, D ** -0.5, o, ctx=c, **kw)
        assert (ops.tcgen05_calls > before) == (c is not None)
        out.append(o.double())
    ops.check_error_word(q.device)
    # weights rounded to bfloat16 (2^-8 each, of weights that sum to at most one) times values of at most |v|; both results
    # rounded to bfloat16 (2^-8 of values of at most |v| each)
    bound = 3 * 2.0 ** -8 * planes[1].abs().max().item()
    assert (out[0] - out[1]).abs().max().item() <= bound
    assert ((out[0] - out[1]).norm() / out[1].norm()).item() <= 2.0 ** -7       # roundings are not all of one sign


@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("heads,kv_heads,lengths,befores", [
    (4, 2, (130, 2, 257), (0, 333, 61)), (3, 3, (300,), (17,)), (2, 1, (65,), (1500,)),
])
def test_odd_values_reach_only_the_rows_that_see_them(form, heads, kv_heads, lengths, befores):
    """Infinities and NaN in values of a portion, in an old one, and in what another request left behind the last token: where
    results are finite and what they are is as in the general kernel, which looks at a row's own keys only."""
    from tiny_llm_infer_b200 import ops
    f = dict(FORMS[form])
    g = torch.Generator(device=DEV).manual_seed(6)

    def randn(*shape):
        return torch.randn(*shape, generator=g, device=DEV)
    ctx = context(lengths, befores)
    pages = -(-ctx.max_context // PAGE)
    order = torch.randperm(len(lengths) * pages, generator=g, device=DEV).to(torch.int32).view(len(lengths), pages)
    keys, values = (randn(len(lengths) * pages, kv_heads, PAGE, D).bfloat16() for _ in range(2))
    largest = values.abs().max().item()
    for s, (n, p0) in enumerate(zip(lengths, befores)):
        def value(pos):
            return values[order[s, pos // PAGE].long(), :, pos % PAGE]
        value(p0 + n // 2)[0, 5] = float("inf")
        value(p0 + n - 1)[:, 77] = float("nan")
        value(p0 // 3)[:, 9] = -float("inf")
        for pos in range(p0 + n, -(-(p0 + n) // PAGE) * PAGE):
            value(pos)[:] = float("nan")
            keys[order[s, pos // PAGE].long(), :, pos % PAGE] = float("nan")
    q = randn(ctx.tokens, heads * D).bfloat16()
    per_head = f.get("gate") == "heads"
    gate = randn(ctx.tokens, heads if per_head else heads * D).bfloat16() if f.get("gate") else None
    kw = dict(softcap=f.get("softcap", 0.0), chunk=f.get("chunk", 0), window=f.get("window", 0), sink=f.get("sink", False),
              slopes=torch.rand(heads, generator=g, device=DEV) * 0.05 if f.get("slopes") else None, gate=gate,
              gate_per_head=per_head, sink_logits=randn(heads) if f.get("learned") else None)
    out = []
    for c in (ctx, None):
        o, before = torch.empty_like(q), ops.tcgen05_calls
        ops.attention_biased(q, keys, values, ctx.positions, ctx.token_slot, order, PAGE, heads, kv_heads, D, D, D ** -0.5, o, ctx=c, **kw)
        assert (ops.tcgen05_calls > before) == (c is not None)
        out.append(o.double())
    ops.check_error_word(q.device)
    finite = torch.isfinite(out[1])
    assert finite.float().mean() > 0.9 and not finite.all()
    assert torch.equal(torch.isfinite(out[0]), finite)
    got, want = out[0][finite], out[1][finite]
    assert (got - want).abs().max().item() <= 3 * 2.0 ** -8 * largest          # as above
    assert ((got - want).norm() / want.norm()).item() <= 2.0 ** -7


@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("heads,kv_heads,lengths,befores", [(4, 2, (130, 2, 257), (0, 333, 61)), (3, 3, (301,), (17,)), (2, 1, (65,), (1500,))])
def test_what_lies_behind_the_last_token_changes_no_bit(form, heads, kv_heads, lengths, befores):
    """Keys and values that another request left in the last page, small beside the cap or far beyond it."""
    from tiny_llm_infer_b200 import ops
    f = dict(FORMS[form])
    g = torch.Generator(device=DEV).manual_seed(8)

    def randn(*shape):
        return torch.randn(*shape, generator=g, device=DEV)
    ctx = context(lengths, befores)
    pages = -(-ctx.max_context // PAGE)
    order = torch.randperm(len(lengths) * pages, generator=g, device=DEV).to(torch.int32).view(len(lengths), pages)
    keys, values = (randn(len(lengths) * pages, kv_heads, PAGE, D).bfloat16() for _ in range(2))
    q = (randn(ctx.tokens, heads * D) * 0.3).bfloat16()            # scores on either side of 0.4 of the cap of 2, within it of 9
    per_head = f.get("gate") == "heads"
    gate = randn(ctx.tokens, heads if per_head else heads * D).bfloat16() if f.get("gate") else None
    kw = dict(softcap=f.get("softcap", 0.0), chunk=f.get("chunk", 0), window=f.get("window", 0), sink=f.get("sink", False),
              slopes=torch.rand(heads, generator=g, device=DEV) * 0.05 if f.get("slopes") else None, gate=gate,
              gate_per_head=per_head, sink_logits=randn(heads) if f.get("learned") else None)
    out = []
    for left in (0.0, 1.0, 100.0):
        for s, (n, p0) in enumerate(zip(lengths, befores)):
            for pos in range(p0 + n, -(-(p0 + n) // PAGE) * PAGE):
                for plane in (keys, values):
                    plane[order[s, pos // PAGE].long(), :, pos % PAGE] = (randn(kv_heads, D) * left).bfloat16()
        o = torch.empty_like(q)
        ops.attention_biased(q, keys, values, ctx.positions, ctx.token_slot, order, PAGE, heads, kv_heads, D, D, D ** -0.5, o, ctx=ctx, **kw)
        out.append(o)
    ops.check_error_word(q.device)
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])


def test_maxima_and_sums_of_runs_may_lie_on_any_float():
    """The library's entry wants 16-byte boundaries of the partial results, not of their maxima and sums."""
    from tiny_llm_infer_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(9)
    heads, kv_heads, ctx = 2, 1, context((65,), (1500,))
    pages, splits = -(-ctx.max_context // PAGE), 4
    table = torch.randperm(pages, generator=g, device=DEV).to(torch.int32).view(1, pages)
    cache = torch.randn(pages, 2, kv_heads, PAGE, D, generator=g, device=DEV).bfloat16()
    q = torch.randn(ctx.tokens, heads * D, generator=g, device=DEV).bfloat16()
    part_o = torch.empty(ctx.tokens * heads * splits * D, device=DEV)
    room, out = torch.empty(ctx.tokens * heads * splits * 2 + 1, device=DEV), []
    for off in (0, 1):
        part_ml, o = room[off:], torch.empty_like(q)
        rc = ops.lib().tllm_paged_attention_prefill_tc(
            q.data_ptr(), ctx.tokens, cache.data_ptr(), pages, ctx.seg_info.data_ptr(), ctx.pf_tiles.data_ptr(), ctx.n_tiles128,
            table.data_ptr(), pages, PAGE, heads, kv_heads, D, 0, D ** -0.5, o.data_ptr(), splits, part_o.data_ptr(), part_ml.data_ptr(),
            ops.error_word(q.device).data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        out.append(o)
    ops.check_error_word(q.device)
    assert torch.equal(out[0], out[1]) and torch.isfinite(out[0]).all()
