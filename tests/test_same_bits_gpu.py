"""A decode step replayed on the same state gives the same bits, however its kernels overlap."""

import pytest
import torch

pytestmark = pytest.mark.gpu

CONFIG = {"architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", "hidden_size": 4096, "intermediate_size": 12288, "num_hidden_layers": 4,
          "num_attention_heads": 32, "num_key_value_heads": 8, "head_dim": 128, "rms_norm_eps": 1e-6, "rope_theta": 1000000.0, "vocab_size": 2048,
          "tie_word_embeddings": False, "max_position_embeddings": 8192}


@pytest.mark.parametrize("requests", [1, 8, 13])
def test_replays_of_a_decode_step_agree(requests):
    """Real widths and cold caches: a stage of the weight ring that is filled again before every warp has read it shows as other logits. With the kernels
    launched one behind the other the arithmetic is the same."""
    from oxr_inference_b200 import ops
    from oxr_inference_b200.engine.batch import StepEntry
    from oxr_inference_b200.engine.graphs import DecodeGraphs
    from oxr_inference_b200.engine.runtime import ModelRunner

    class Graphs(DecodeGraphs):
        def _forward(self, ctx):
            self.logits = self.runner.model.step(ctx, self.runner.cache)
            s = ctx.sampling
            return ops.sample(self.logits, s["temperature"], s["seed_lo"], s["seed_hi"], s["counter"])

    runner = ModelRunner.from_config(CONFIG, 1, dtype="bfloat16", page_size=16, num_pages=1200, max_requests=requests, max_positions=8192)
    entries = []
    for i in range(requests):
        request = runner.cache.open(i)
        length = 200 + 1600 * i // max(requests - 1, 1)
        assert runner.cache.reserve(request, length + 1)
        runner.step([StepEntry(request, [(7 * i + 31 * p) % 2048 for p in range(length)], [])])
        entries.append(StepEntry(request, [i], [0]))
    cold = torch.empty(64 << 20, device="cuda")
    libs = [ops._lib(), ops._attn_lib(128)]
    want = None
    try:
        for chained in (1, 0):
            for lib in libs:
                lib.oxr_set_chain(chained)
            graphs = Graphs(runner, max_batch=requests, max_positions=8192)
            for _ in range(40 if chained else 2):
                cold.fill_(1.0)
                torch.cuda.synchronize()
                graphs.run(entries)
                torch.cuda.synchronize()
                got = graphs.logits[:requests].clone()
                want = got if want is None else want
                assert torch.equal(got, want)
    finally:
        for lib in libs:
            lib.oxr_set_chain(int(ops.CHAIN_KERNELS))
    runner.check()
