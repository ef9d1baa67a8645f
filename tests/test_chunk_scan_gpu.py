"""The recurrences by chunks of sixteen tokens against float64 and against the token-by-token scan: portions at the edges of a
chunk, portions in any order, rows of no request, every recurrence the chunks serve."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def lanes(dk):
    return 4 if dk <= 64 else 8


def pack(S):
    """[slots, heads, dk, dv] in the layout of a request's state."""
    n, heads, dk, dv = S.shape
    return S.reshape(n, heads, lanes(dk), dk // lanes(dk), dv).permute(0, 1, 3, 4, 2).reshape(n, -1).contiguous()


def unpack(flat, heads, dk, dv):
    return flat.reshape(-1, heads, dk // lanes(dk), dv, lanes(dk)).permute(0, 1, 4, 2, 3).reshape(-1, heads, dk, dv)


@pytest.mark.parametrize("mode", ["delta", "channel", "channel, no weights", "head", "fixed"])
# blocks of 16 columns, and of 32 (from 111 blocks of these on): of one decay per head in the form of one block per SM up to 148 of
# them (one portion of 32 x 128 or 64 x 64 columns), of two beyond
@pytest.mark.parametrize("heads,kv_heads,dk,dv", [(4, 2, 128, 128), (3, 3, 64, 48), (8, 8, 128, 16), (40, 40, 64, 64), (32, 8, 128, 128), (64, 16, 64, 64)])
@pytest.mark.parametrize("lengths", [(1, 15, 16, 17, 33), (200,), (64, 0, 31, 47)])
def test_chunks_are_the_recurrence(mode, heads, kv_heads, dk, dv, lengths, monkeypatch):
    from tiny_llm_infer_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(7)
    n = len(lengths)
    starts, row = [0] * n, 3                                       # rows of no portion before, between and after
    for s in reversed(range(n)):                                   # the portions' rows lie in the opposite order
        starts[s], row = row, row + lengths[s] + (2 if s == 1 else 0)
    tokens = row + 5
    slots = [n - s for s in range(n)]
    if n > 2:
        slots[2] = -1                                              # a portion of no request: left alone
    seg = torch.tensor([[slots[s], starts[s], lengths[s], 0] for s in range(n)], dtype=torch.int32, device=DEV)

    def randn(*shape):
        return torch.randn(*shape, generator=g, device=DEV)
    q, k = (torch.nn.functional.normalize(randn(tokens, kv_heads, dk), dim=-1) for _ in range(2))
    v = randn(tokens, heads, dv)
    decay = beta = fgate = None
    if mode in ("delta", "channel", "channel, no weights"):
        decay = torch.rand(tokens, heads, dk, generator=g, device=DEV) ** 0.2          # many near one, some near zero
        decay[::7, :, ::5] = 0.0
    if mode in ("delta", "channel"):
        beta = torch.rand(tokens, heads, generator=g, device=DEV)
    if mode == "head":
        beta, fgate = torch.rand(tokens, heads, generator=g, device=DEV) ** 0.3, torch.rand(tokens, heads, generator=g, device=DEV)
    if mode == "fixed":
        fgate = torch.rand(heads, generator=g, device=DEV) ** 0.1
    code = {"delta": ops.SCAN_DELTA, "head": ops.SCAN_HEAD_DECAY, "fixed": ops.SCAN_FIXED_DECAY}.get(mode, ops.SCAN_PLAIN)
    S0 = randn(n + 1, heads, dk, dv)

    want_o, want_S = torch.zeros(tokens, heads, dv, dtype=torch.float64, device=DEV), S0.double()
    rep = heads // kv_heads
    for s in range(n):
        if slots[s] < 0:
            continue
        S = want_S[slots[s]].clone()
        for t in range(starts[s], starts[s] + lengths[s]):
            kt, qt = (x[t].double().repeat_interleave(rep, 0) for x in (k, q))
            if mode == "head":
                S = S * beta[t].double()[:, None, None]
            elif mode == "fixed":
                S = S * fgate.double()[:, None, None]
            else:
                S = S * decay[t].double()[..., None]
            u = v[t].double()
            if mode == "delta":
                u = beta[t].double()[:, None] * (u - torch.einsum("hkv,hk->hv", S, kt))
            elif mode == "channel":
                u = beta[t].double()[:, None] * u
            elif mode == "head":
                u = fgate[t].double()[:, None] * u
            S = S + kt[..., None] * u[:, None]
            want_o[t] = torch.einsum("hkv,hk->hv", S, qt)
        want_S[slots[s]] = S

    def run(by_chunks):
        monkeypatch.setattr(ops, "CHUNK_TOKENS", 1 if by_chunks else 1 << 30)
        state, o = pack(S0), torch.zeros(tokens, heads, dv, device=DEV)
        before = ops.launches
        ops._scan(code, seg, tokens, None, q, k, v, decay, beta, state, heads, kv_heads, dk, dv, o, fgate=fgate)
        assert ops.launches - before == (2 if by_chunks else 1)
        return o, unpack(state, heads, dk, dv)

    (o, S), (o1, S1) = run(True), run(False)
    for got, token, want in ((o, o1, want_o), (S, S1, want_S)):
        error, token_error = ((x.double() - want).norm() / want.norm() for x in (got, token))
        # both sum in float32 (2^-24 a step); the chunks' sums may not be further off than a few more roundings
        assert error <= 1.5 * token_error + 2.0 ** -23, (float(error), float(token_error))
    idle = torch.ones(tokens, dtype=torch.bool, device=DEV)
    for s in range(n):
        if slots[s] >= 0:
            idle[starts[s]:starts[s] + lengths[s]] = False
    assert (o[idle] == 0).all()                                    # nothing is written for the others
    # a token reaches no read-out before it, whatever its values are
    last = [starts[s] + lengths[s] - 1 for s in range(n) if slots[s] >= 0 and lengths[s]]
    v[last[::2]], v[last[1::2]] = float("nan"), float("inf")
    o2, _ = run(True)
    kept = torch.ones(tokens, dtype=torch.bool, device=DEV)
    kept[last] = False
    assert torch.equal(o2[kept], o[kept])


@pytest.mark.parametrize("by_chunks", [True, False])
@pytest.mark.parametrize("mode,operands", [("delta", "q k v decay beta"), ("channel", "q k v decay beta"), ("channel, no weights", "q k v decay"),
                                           ("head", "q k v beta fgate"), ("fixed", "q k v")])
# blocks of 16 columns; of 32, more than 148 of them, at both widths of keys; of 32, at most 148
@pytest.mark.parametrize("heads,kv_heads,dk,dv", [(4, 2, 128, 128), (40, 40, 64, 64), (32, 8, 128, 128), (12, 4, 128, 128), (24, 8, 64, 64)])
@pytest.mark.parametrize("odd", [float("nan"), float("inf")])
def test_an_odd_token_reaches_no_read_out_before_it(by_chunks, mode, operands, heads, kv_heads, dk, dv, odd, monkeypatch):
    """One token of every portion has an infinity or a NaN in one operand; what is read out before it stays bit for bit."""
    from tiny_llm_infer_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(11)
    lengths, at = (50, 16, 37), (21, 15, 36)                       # inside a chunk, a chunk's last, a portion's last
    starts = [0, 50, 66]
    tokens = sum(lengths)
    seg = torch.tensor([[s, starts[s], lengths[s], 0] for s in range(3)], dtype=torch.int32, device=DEV)
    q, k = (torch.nn.functional.normalize(torch.randn(tokens, kv_heads, dk, generator=g, device=DEV), dim=-1) for _ in range(2))
    v, S0 = torch.randn(tokens, heads, dv, generator=g, device=DEV), torch.randn(3, heads, dk, dv, generator=g, device=DEV)
    rand = {n: torch.rand(*shape, generator=g, device=DEV) for n, shape in
            (("decay", (tokens, heads, dk)), ("beta", (tokens, heads)), ("fgate", (tokens, heads)), ("fixed", (heads,)))}
    clean = {"q": q, "k": k, "v": v, "decay": rand["decay"] if "decay" in operands else None,
             "beta": rand["beta"] if "beta" in operands else None, "fgate": rand["fixed"] if mode == "fixed" else rand["fgate"] if mode == "head" else None}
    code = {"delta": ops.SCAN_DELTA, "head": ops.SCAN_HEAD_DECAY, "fixed": ops.SCAN_FIXED_DECAY}.get(mode, ops.SCAN_PLAIN)
    monkeypatch.setattr(ops, "CHUNK_TOKENS", 1 if by_chunks else 1 << 30)

    def run(t):
        state, o, before = pack(S0), torch.zeros(tokens, heads, dv, device=DEV), ops.launches
        ops._scan(code, seg, tokens, None, t["q"], t["k"], t["v"], t["decay"], t["beta"], state, heads, kv_heads, dk, dv, o, fgate=t["fgate"])
        assert ops.launches - before == (2 if by_chunks else 1)
        return o
    want = run(clean)
    assert torch.isfinite(want).all()
    kept = torch.ones(tokens, dtype=torch.bool, device=DEV)
    for s in range(3):
        kept[starts[s] + at[s]:starts[s] + lengths[s]] = False
    for name in operands.split():
        spoilt = clean[name].clone()
        spoilt[[starts[s] + at[s] for s in range(3)]] = odd
        got = run({**clean, name: spoilt})
        assert torch.equal(got[kept], want[kept]), name
        assert not torch.isfinite(got[[starts[s] + at[s] for s in range(3)]]).all(), name


@pytest.mark.parametrize("mode", ["delta", "channel", "head", "fixed", "erase"])
@pytest.mark.parametrize("rows", [1, 5, 70])
@pytest.mark.parametrize("heads,kv_heads,dk,dv", [(4, 2, 128, 128), (3, 3, 64, 24), (2, 2, 128, 200), (6, 6, 64, 128)])
def test_rows_of_one_token(mode, rows, heads, kv_heads, dk, dv):
    """One step of the recurrence for requests that each bring one token, some rows of no request among them."""
    from tiny_llm_infer_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(9)
    if mode == "erase":
        kv_heads = heads

    def randn(*shape):
        return torch.randn(*shape, generator=g, device=DEV)

    def rand(*shape):
        return torch.rand(*shape, generator=g, device=DEV)
    slot = torch.randperm(rows, generator=g, device=DEV).to(torch.int32)
    slot[1::3] = -1
    q, k = (torch.nn.functional.normalize(randn(rows, kv_heads, dk), dim=-1) for _ in range(2))
    v, S0 = randn(rows, heads, dv), randn(rows, heads, dk, dv)
    decay = rand(rows, heads, dk) if mode in ("delta", "channel", "erase") else None
    beta = rand(rows, heads) if mode in ("delta", "channel", "head") else None
    fgate = rand(rows, heads) if mode == "head" else rand(heads) if mode == "fixed" else None
    erase = k * rand(rows, heads, dk) if mode == "erase" else None
    code = {"delta": ops.SCAN_DELTA, "channel": ops.SCAN_PLAIN, "head": ops.SCAN_HEAD_DECAY, "fixed": ops.SCAN_FIXED_DECAY, "erase": ops.SCAN_ERASE}[mode]
    state, o = pack(S0), torch.zeros(rows, heads, dv, device=DEV)
    ops._scan(code, None, rows, slot, q, k, v, decay, beta, state, heads, kv_heads, dk, dv, o, fgate=fgate, erase=erase)
    live = slot >= 0
    S, kt, qt = S0.double()[slot.clamp(min=0).long()], *(x.double().repeat_interleave(heads // kv_heads, 1) for x in (k, q))
    old = S
    if mode == "head":
        S = S * beta.double()[..., None, None]
    elif mode == "fixed":
        S = S * fgate.double()[:, None, None]
    else:
        S = S * decay.double()[..., None]
    u = v.double()
    if mode == "delta":
        u = beta.double()[..., None] * (u - torch.einsum("rhkv,rhk->rhv", S, kt))
    elif mode in ("channel", "head"):
        u = (beta if mode == "channel" else fgate).double()[..., None] * u
    elif mode == "erase":
        S = S - erase.double()[..., None] * torch.einsum("rhkv,rhk->rhv", old, kt)[:, :, None]
    S = S + kt[..., None] * u[:, :, None]
    want = torch.einsum("rhkv,rhk->rhv", S, qt)
    got = unpack(state, heads, dk, dv).double()
    assert (o[~live] == 0).all()
    untouched = torch.ones(rows, dtype=torch.bool, device=DEV)
    untouched[slot[live].long()] = False
    assert torch.equal(got[untouched], S0.double()[untouched])
    # sums of up to dk float32 products, a few roundings of 2^-24 each on average
    assert ((o.double() - want)[live].norm() / want[live].norm()) < 4e-7
    assert ((got[slot[live].long()] - S[live]).norm() / S[live].norm()) < 4e-7
