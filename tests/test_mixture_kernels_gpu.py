"""The kernels of a mixture of experts one by one, at the edges of their tiles, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
# rows per expert: none, one, the edges of sixteen, of a box of 64 and of a tile of 128, more than a tile
COUNTS = {"few": [0, 1, 0, 2, 1, 0, 0, 3], "edges": [15, 16, 17, 0, 63, 64, 65, 1], "tiles": [127, 128, 129, 0, 257, 5, 300, 2]}


def ids_of(counts):
    ids = torch.cat([torch.full((c,), e) for e, c in enumerate(counts)])
    g = torch.Generator().manual_seed(1)
    return ids[torch.randperm(len(ids), generator=g)].to(torch.int32).view(-1, 1).to(DEV)      # one choice per token


@pytest.mark.parametrize("counts", sorted(COUNTS))
@pytest.mark.parametrize("tile_rows", [64, 128])
@pytest.mark.parametrize("n,k", [(128, 64), (264, 200), (1040, 328)])        # weight rows: whole tiles, a rest of 8, one of 16
@pytest.mark.parametrize("form", ["plain", "float32", "gated", "relu2"])
def test_products_of_the_experts(counts, tile_rows, n, k, form):
    from tiny_llm_infer_b200 import ops
    ids = ids_of(COUNTS[counts])
    experts, rows = len(COUNTS[counts]), ids.numel()
    g = torch.Generator(device=DEV).manual_seed(2)
    x = torch.randn(rows, k, generator=g, device=DEV).bfloat16()
    w = (torch.randn(experts, 2 * n if form == "gated" else n, k, generator=g, device=DEV) * k ** -0.5).bfloat16()
    scale = torch.rand(rows, 1, generator=g, device=DEV)
    plan = ops.MoePlan(ids, experts, tile_rows, tensor_memory=True)
    if form == "gated":
        stored = torch.stack([ops.interleave_gate_up(e[:n], e[n:]) for e in w])
        got = ops.moe_grouped(x, stored, plan, 1, gated=True, gather=True, weights=scale, interleaved=True)
    else:
        got = ops.moe_grouped(x, w, plan, 1, gated=False, gather=True, weights=scale, unary=form == "relu2", act="relu2",
                              out_dtype=torch.float32 if form == "float32" else None)
    ops.check_error_word(x.device)
    assert got.dtype == (torch.float32 if form == "float32" else torch.bfloat16) and tuple(got.shape) == (rows, n)
    u = (x.float() * scale).bfloat16().double()                              # the scaled row is rounded before the product
    y = torch.einsum("rk,rnk->rn", u, w.double()[ids[:, 0].long()])
    if form == "gated":
        y = torch.nn.functional.silu(y[:, :n]) * y[:, n:]
    elif form == "relu2":
        y = y.clamp(min=0) ** 2
    back = got.double()[plan.row_of.long()]                                  # rows of the plan back in the tokens' order
    # float32: sums of k products in another order, k 2^-24 of the terms' size; bfloat16 (8 bits): half a unit in the last place, 2^-8
    tol = (k * 2.0 ** -24 if form == "float32" else 2.0 ** -8 + k * 2.0 ** -23) * y.abs().clamp(min=1.0)
    assert ((back - y).abs() <= tol).all(), ((back - y).abs() / tol).max()


@pytest.mark.parametrize("tokens,experts,real,top,tile_rows", [(1, 5, 5, 2, 64), (700, 64, 62, 4, 128), (333, 1500, 1500, 3, 64)])
def test_plan_sorts_by_expert_and_lists_the_tiles(tokens, experts, real, top, tile_rows):
    from tiny_llm_infer_b200 import ops
    g = torch.Generator().manual_seed(3)
    ids = torch.stack([torch.randperm(experts, generator=g)[:top] for _ in range(tokens)]).to(torch.int32)
    plan = ops.MoePlan(ids.to(DEV), experts, tile_rows, real=real, tensor_memory=True)
    flat = ids.flatten().long()
    count = torch.bincount(flat, minlength=experts)
    offsets = torch.cat([torch.zeros(1, dtype=torch.long), count.cumsum(0)])
    assert torch.equal(plan.offsets.cpu().long(), offsets)
    row_of, src_of = plan.row_of.cpu().long(), plan.src_of.cpu().long()
    assert torch.equal(row_of.sort().values, torch.arange(flat.numel())) and torch.equal(src_of[row_of], torch.arange(flat.numel()))
    assert torch.equal(plan.expert_of_row.cpu().long()[row_of], flat)
    tiles = [(e, int(offsets[e]) + r) for e in range(real) for r in range(0, int(count[e]), tile_rows)]
    n = int(plan.n_tiles)
    assert n == len(tiles) <= plan.max_tiles
    assert list(zip(plan.tile_expert[:n].tolist(), plan.tile_row0[:n].tolist())) == tiles


@pytest.mark.parametrize("width", [8, 264, 1001])                            # eight per access; one by one
@pytest.mark.parametrize("top", [1, 4, 6])
@pytest.mark.parametrize("y_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("identity", [False, True])
def test_combine_adds_the_choices(width, top, y_dtype, identity):
    from tiny_llm_infer_b200 import ops
    tokens, experts, real = 37, 9, 6 if identity else 9
    g = torch.Generator(device=DEV).manual_seed(4)
    ids = torch.stack([torch.randperm(experts, generator=g, device=DEV)[:top] for _ in range(tokens)]).to(torch.int32)
    plan = ops.MoePlan(ids, experts, real=real)
    y = torch.randn(tokens * top, width, generator=g, device=DEV).to(y_dtype)
    y[plan.expert_of_row >= real] = float("nan")                             # rows of experts without matrices are never written
    shared, x = (torch.randn(tokens, width, generator=g, device=DEV).bfloat16() for _ in range(2))
    weights, logit = torch.rand(tokens, top, generator=g, device=DEV), torch.randn(tokens, generator=g, device=DEV)
    got = ops.moe_combine(y, plan, top, shared, torch.bfloat16, weights=weights, identity_input=x if identity else None,
                          shared_gate=logit).double()
    own = y.double()[plan.row_of.long()].view(tokens, top, width)
    own = torch.where((ids >= real)[..., None], x.double()[:, None], own)
    want = shared.double() * torch.sigmoid(logit.double())[:, None] + (weights.double()[..., None] * own).sum(1)
    assert ((got - want).abs() <= (2.0 ** -8 + 1e-6) * want.abs() + 1e-5).all()


@pytest.mark.parametrize("rows", [9, 40])
def test_rows_off_the_16_byte_grid(rows):
    """The part takes rows that start anywhere (9 rows and more: fewer are refused by the router's product), on the kernels that
    look at the alignment; the lists' own product refuses them on the host."""
    from tiny_llm_infer_b200 import ops
    from tiny_llm_infer_b200.parts import lookup
    width, experts, top, inter = 64, 6, 2, 48
    g = torch.Generator(device=DEV).manual_seed(5)
    part = lookup("feed_forward", "moe")(width, experts, top, inter, torch.bfloat16, DEV)
    part.load({name: (torch.randn(*spec.shape, generator=g, device=DEV) * 0.2).bfloat16()
               for name, spec in part.param_specs(width, experts, top, inter).items()})
    x = torch.randn(rows, width, generator=g, device=DEV).bfloat16()
    off = torch.zeros(rows * width + 3, dtype=torch.bfloat16, device=DEV)[3:].view(rows, width)
    off.copy_(x)
    assert off.data_ptr() % 16 and off.is_contiguous()
    before = ops.tcgen05_calls
    got = part.forward(off, None).double()
    assert ops.tcgen05_calls == before
    want = part.forward(x, None).double()
    assert ops.tcgen05_calls == before + 2
    ops.check_error_word(torch.device(DEV))
    # both round the units' outputs and the result to bfloat16 (2^-9 of each, root mean square less)
    assert ((got - want).norm() / want.norm()).item() <= 2.0 ** -8
    plan = ops.MoePlan(torch.zeros(rows, 1, dtype=torch.int32, device=DEV), experts, 64, tensor_memory=True)
    with pytest.raises(ops.KernelError, match="aligned"):
        ops.moe_grouped(off, part.w_gate_up, plan, 1, gated=True, gather=True, interleaved=True)
    with pytest.raises(ops.KernelError, match="aligned"):
        ops.moe_grouped(off, part.w_gate_up, plan, 1, gated=True, gather=False, interleaved=True)
