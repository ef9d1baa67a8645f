"""Short portions taken row by row through captured graphs (``ModelRunner._rows_graphable``): the logits of the general way
for the same steps, in rounding.  One row short of a bucket, a whole one, one row more, the largest and one beyond it; behind
keys of earlier steps, beside decode rows, with places wanted inside the portion, with a window, with a late token."""
import pytest
import torch

from tiny import TINIES, make_folder, prompt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,dtype", [("B", "float32"), ("D", "bfloat16"), ("E", "bfloat16")])
def test_short_portions_row_by_row(tmp_path, name, dtype):
    from tiny_llm_infer_b200.cache import CacheManager
    from tiny_llm_infer_b200.engine import DTYPES, ModelRunner, StepEntry, load_model
    tiny = TINIES[name]
    model, cfg = load_model(str(make_folder(tiny, tmp_path / "m")), DTYPES[dtype], "cuda:0")
    runners = []
    for graphs in (True, False):
        cache = CacheManager(model.cache_needs(), tiny["page_size"], 160, 8, 512, DTYPES[dtype], "cuda:0")
        runners.append(ModelRunner(model, cache, max_batch_tokens=256, use_graphs=graphs))
    graph_runner, plain_runner = runners
    # two kernels' roundings of the same sums (the bounds of the batched against the whole prompt elsewhere)
    bound = 1e-4 if dtype == "float32" else 0.05

    def both(make, late=()):
        out = []
        for r in runners:
            p = r.prepare(make())
            keys.append(p.graph_key)
            out.append(r.run(p, late).clone())
        assert out[0].shape == out[1].shape and (out[0] - out[1]).abs().max() < bound
    for n in (2, 15, 16, 17, 128, 129):
        keys = []
        for turn in range(2):                            # the second time the bucket is captured
            toks = prompt(n + turn, n, cfg.vocab_size)
            more = prompt(900 + n + turn, 5, cfg.vocab_size)
            both(lambda: [StepEntry("a", toks, [n - 1, 0] if n > 2 else [n - 1])])
            both(lambda: [StepEntry("a", more[:3], [2]), StepEntry("b", more[3:], [])])       # behind keys, nothing wanted of b
            both(lambda: [StepEntry("a", [more[4]], [0]), StepEntry("b", [more[0], 0, more[1]], [2], late=1)], late=[more[2]])
            for r in runners:
                r.release("a"), r.release("b")
        assert (n == 129) == (keys[6] is None) and keys[8] is not None and all(k is None for k in keys[1::2])
    graph_runner.check_kernels()
    graph_runner.cache.audit()


@pytest.mark.parametrize("name,dtype", [("B", "float32"), ("D", "bfloat16"), ("E", "bfloat16")])
def test_the_same_step_again_gives_the_same_bits(tmp_path, name, dtype):
    """What a runner has done before decides nothing: the first step of a bucket, the one that captures its graph and those that
    replay it give the same logits, to the bit, whatever number of places is wanted."""
    from tiny_llm_infer_b200.cache import CacheManager
    from tiny_llm_infer_b200.engine import DTYPES, ModelRunner, StepEntry, load_model
    tiny = TINIES[name]
    model, cfg = load_model(str(make_folder(tiny, tmp_path / "m")), DTYPES[dtype], "cuda:0")
    cache = CacheManager(model.cache_needs(), tiny["page_size"], 160, 8, 512, DTYPES[dtype], "cuda:0")
    runner = ModelRunner(model, cache, max_batch_tokens=256)
    for n, want in ((2, [1]), (9, [8]), (16, []), (17, [0, 3, 16]), (100, [99]), (128, list(range(128)))):
        toks, more = prompt(40 + n, n, cfg.vocab_size), prompt(7, 5, cfg.vocab_size)
        keys, first = [], None
        for turn in range(4):
            got = []
            for entries in ([StepEntry("a", toks, want)], [StepEntry("a", more[:2], [1]), StepEntry("b", more[2:], [])]):
                prepared = runner.prepare(entries)
                keys.append(prepared.graph_key)
                got.append(runner.run(prepared).clone())
            runner.release("a"), runner.release("b")
            first = first or got
            assert got[0].shape == (len(want), cfg.vocab_size) and all(torch.equal(x, y) for x, y in zip(got, first)), (n, turn)
        assert keys[0] is None and all(keys[2:])             # the first was launched kernel by kernel, the others replayed
    runner.check_kernels()
    runner.cache.audit()
