"""The engine's allowance for a step's own tensors covers what the largest steps take, where the kernels' scratch is most of it:
many experts with few rows each (every run padded to whole tiles), wide heads on a narrow model by chunks of short requests."""
import json

import pytest
import torch

pytestmark = pytest.mark.gpu


def nomudra(width, mixer, mlp):
    return dict(architecture="Nomudra", vocab=256, width=width, norm=dict(eps=1e-6), dtype="bfloat16",
                layers=[dict(type="attention", mlp=mlp, mixer=mixer) if "kv_heads" in mixer else dict(type="mlstm", mlp=mlp, mixer=mixer)])


EXPERTS = nomudra(512, dict(heads=4, kv_heads=4, dim=64, vdim=64, scale=0.125, rot=dict(base=10000.0, dims=64)),
                  dict(kind="moe", router=dict(experts=640, top=8), expert=dict(ff=256, limit=7.0), shared=None))
CHUNKS = nomudra(256, dict(heads=64, dim=128, vdim=16, gate_cap=15.0), None)


@pytest.mark.parametrize("cfg,requests,tokens", [(EXPERTS, 1, 8192), (CHUNKS, 256, 32)], ids=["experts", "chunks"])
def test_the_allowance_covers_a_step(tmp_path, cfg, requests, tokens):
    from nanohybrid_vlm_b200 import LLM
    from nanohybrid_vlm_b200.engine import StepItem
    (tmp_path / "config.json").write_text(json.dumps(cfg))
    runner = LLM(str(tmp_path), random_weights_seed=1, kvcache_block_size=256, num_kvcache_blocks=requests * -(-tokens // 256) + 1,
                 max_model_len=tokens + 1, max_num_seqs=requests, max_num_batched_tokens=8192).model_runner
    items = []
    for r in range(requests):
        runner.cache.allocate(r, tokens)
        items.append(StepItem(r, [(7 * r + i) % 256 for i in range(tokens)], 0, [tokens - 1]))
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    runner.run(items, [(0.0, r, tokens) for r in range(requests)])
    took = torch.cuda.max_memory_allocated() - before
    assert took <= runner._activation_allowance(), (took >> 20, runner._activation_allowance() >> 20)
