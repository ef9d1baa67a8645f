"""Kernels with bounded waits report through a device word.  A step that replays such kernels from a CUDA graph (the
experts' products of every bfloat16 decode step of a mixture) has its report read as one that launches them: here the word
is written by hand, behind a step's kernels."""
import pytest
import torch

from tiny_panolorn import PANOLORNS, make_folder, prompt

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def test_a_replayed_decode_step_is_checked(tmp_path):
    from tiny_llm_infer_b200 import ops
    from tiny_llm_infer_b200.cache import CacheManager
    from tiny_llm_infer_b200.engine import ModelRunner, StepEntry, load_model
    model, _ = load_model(make_folder(PANOLORNS["P1"], tmp_path), torch.bfloat16, DEV)
    cache = CacheManager(model.cache_needs(), 16, 32, max_slots=2, max_seq_len=256, dtype=torch.bfloat16, device=DEV)
    runner = ModelRunner(model, cache, max_batch_tokens=64)
    runner.step([StepEntry("a", prompt(1, 20, 320), [19])])
    calls = []
    for token in (5, 6, 7):                                        # captured, then replayed
        before = ops.tcgen05_calls
        runner.step([StepEntry("a", [token], [0])])
        calls.append(ops.tcgen05_calls - before)
        runner.check_kernels()
    assert calls[1] == calls[2] == 2 and len(runner._graphs) == 1  # the two products of the one layer with experts
    runner.step([StepEntry("a", [8], [0])])
    ops.error_word(torch.device(DEV)).fill_(7)
    with pytest.raises(ops.KernelError, match="code 7"):
        runner.check_kernels()
    step = runner.prepare([StepEntry("a", [9], [0])])
    runner.run(step)
    ops.error_word(torch.device(DEV)).fill_(8)
    torch.cuda.synchronize()
    with pytest.raises(ops.KernelError, match="code 8"):
        runner.check_kernels(step)
    runner.step([StepEntry("a", [10], [0])])
    runner.check_kernels()                                         # the word was cleared


@pytest.mark.parametrize("overlap", [True, False])
@pytest.mark.parametrize("which", ["a prompt portion that samples nothing", "an early decode step", "the last decode step"])
def test_generation_stops_at_the_step_that_failed(tmp_path, monkeypatch, overlap, which):
    from tiny_llm_infer_b200 import LLM, SamplingParams, ops
    folder = make_folder(PANOLORNS["P1"], tmp_path)

    def generate(failing):
        llm = LLM(str(folder), dtype="bfloat16", max_model_len=128, num_kv_blocks=32, block_size=16, max_num_batched_tokens=32,
                  max_num_seqs=2, overlap_scheduling=overlap)
        launched, plain_run = [], llm.engine.runner.run

        def run(step, *args, **kwargs):
            logits = plain_run(step, *args, **kwargs)
            if len(launched) == failing:
                ops.error_word(torch.device(DEV)).fill_(5)
            launched.append(step.graph_key is not None)
            return logits
        monkeypatch.setattr(llm.engine.runner, "run", run)
        llm.generate([prompt(2, 40, 320)], SamplingParams(max_tokens=6, ignore_eos=True))
        return launched
    launched = generate(-1)
    assert launched == [False] * 2 + [True] * 5                    # 32 and 8 tokens of the prompt, then one token at a time
    failing = {"a prompt portion that samples nothing": 0, "an early decode step": 3, "the last decode step": 6}[which]
    with pytest.raises(ops.KernelError, match="code 5"):
        generate(failing)
    ops.check_error_word(torch.device(DEV))                        # read and cleared


def test_a_device_without_an_index_has_the_word_its_tensors_report_to():
    from tiny_llm_infer_b200 import ops
    x = torch.zeros(1, device="cuda")
    ops.error_word(x.device).fill_(9)
    with pytest.raises(ops.KernelError, match="code 9"):
        ops.check_error_word("cuda")
    ops.check_error_word(torch.device("cuda"))
    ops.check_error_word(x.device)
