"""One-token rows with at most eight query heads per block (the keys as the MMA's left operand; 24 heads on one go twelve to a block,
as the left operand themselves) against 64 bits: first and last keys of tiles and of runs of keys, pages that are no power of two,
every change of the score, places of the pages that nobody has written."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,dim,page", [(8, 8, 128, 16), (32, 8, 128, 16), (16, 2, 64, 48), (12, 4, 64, 32), (24, 1, 128, 16),
                                                        (21, 1, 128, 16), (50, 2, 64, 48)])       # three blocks of seven heads, five of five, per key/value head
@pytest.mark.parametrize("change", ["none", "cap window sink gate", "slopes chunk", "bias learned"])
@pytest.mark.parametrize("crowd", [0, 40])
def test_one_token_rows(heads, kv_heads, dim, page, change, crowd):
    from types import SimpleNamespace
    from tiny_llm_infer_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(heads + dim)

    def draw(*shape):
        return torch.randn(*shape, generator=g, device="cuda")
    positions = [0, 15, 16, 17, 63, 64, 700, 1023] + [5 + 3 * i for i in range(crowd)]       # a crowd takes one run of keys per row
    n, longest = len(positions), max(positions) + 1
    pages = -(-longest // page)
    table = torch.randperm(n * pages, generator=g, device="cuda").view(n, pages).to(torch.int32)
    k_plane, v_plane = (torch.full((n * pages, kv_heads, page, dim), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    q, keys, values = draw(n, heads * dim).bfloat16(), [], []
    for r, pos in enumerate(positions):
        k, v = draw(pos + 1, kv_heads, dim).bfloat16(), draw(pos + 1, kv_heads, dim).bfloat16()
        at = torch.arange(pos + 1, device="cuda")
        for plane, rows in ((k_plane, k), (v_plane, v)):
            plane[table[r].long()[at // page], :, at % page] = rows
        keys.append(k.double()), values.append(v.double())
    mods, gate = {}, None
    if "cap" in change:
        gate = draw(n, heads).bfloat16()
        mods = dict(softcap=20.0, window=333, sink=True, gate=gate, gate_per_head=True)
    if "slopes" in change:
        mods = dict(slopes=torch.rand(heads, generator=g, device="cuda") * 0.05, chunk=200)
    if "bias" in change:
        mods = dict(distance_bias=draw(heads, 50), sink=True, sink_logits=draw(heads))
    slot = torch.arange(n, dtype=torch.int32, device="cuda")
    slot[3] = -1
    ctx = SimpleNamespace(tokens=n, n_dec=n, dec_rows=None, n_tiles=0, pf_tiles=torch.zeros(0, 2, dtype=torch.int32, device="cuda"), max_context=longest)
    out = torch.full((n, heads * dim), float("nan"), dtype=torch.bfloat16, device="cuda")
    scale = dim ** -0.5
    ops.attention_biased(q, k_plane, v_plane, torch.tensor(positions, dtype=torch.int32, device="cuda"), slot, table, page, heads, kv_heads,
                         dim, dim, scale, out, ctx=ctx, **mods)
    for r, pos in enumerate(positions):
        if r == 3:
            assert (out[r] == 0).all()
            continue
        lo = 0
        if "chunk" in change:
            lo = pos // 200 * 200
        if "window" in change:
            lo = max(0, pos - 332)
        k, v = (t[lo:].repeat_interleave(heads // kv_heads, 1) for t in (keys[r], values[r]))
        s = torch.einsum("hd,jhd->hj", q[r].double().view(heads, dim), k) * scale
        back = pos - torch.arange(lo, pos + 1, device="cuda")
        if "cap" in change:
            s = 20.0 * torch.tanh(s / 20.0)
        if "slopes" in change:
            s = s - mods["slopes"].double()[:, None] * back
        if "bias" in change:
            s = s + mods["distance_bias"].double()[:, back.clamp(max=49)]
        if "sink" in change or "learned" in change:
            first = mods["sink_logits"].double() if "learned" in change else torch.zeros(heads, dtype=torch.float64, device="cuda")
            s = torch.cat([first[:, None], s], 1)
            p = torch.softmax(s, 1)[:, 1:]
        else:
            p = torch.softmax(s, 1)
        want = torch.einsum("hj,jhd->hd", p, v)
        if gate is not None:
            want = want * torch.sigmoid(gate[r].double())[:, None]
        got = out[r].double().view(heads, dim)
        # weights rounded to bfloat16 (2^-9 each, up to 1 in the sum of weights * values of size 1) and the result's own rounding
        assert ((got - want).abs() <= 2.0 ** -7 * (want.abs() + torch.einsum("hj,jhd->hd", p, v.abs()))).all(), (r, (got - want).abs().max())
