"""What the attention parts plan on the host."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch


@pytest.mark.gpu  # (asks the kernel's library)
@pytest.mark.parametrize("head_dim,page_size,resident", [(128, 16, 2), (128, 8, 2), (128, 64, 2), (128, 4, 3), (128, 24, 3), (128, 128, 3),
                                                         (64, 16, 3), (64, 4, 3)])
def test_decode_splits_fill_one_wave_of_the_kernel_that_runs(monkeypatch, head_dim, page_size, resident):
    from torchlet_b200.parts import attention_bf16

    monkeypatch.setattr(attention_bf16, "_sm_count", lambda index: 148)
    splits = attention_bf16.decode_splits(8, 4, 100000, SimpleNamespace(index=0), head_dim, page_size)
    assert splits == resident * 148 // 32


@pytest.mark.parametrize("new,before,taken", [
    ([300], [0], True), ([2, 254], [0, 0], True), ([700, 257, 256, 40], [0] * 4, True),
    ([255], [0], False),  # fewer tokens than the per-head products take
    ([300, 1], [0, 0], False), ([300, 20], [0, 16], False)])  # a single token; a cached prefix
def test_tiles_of_whole_prompts_cover_every_request_longest_first(monkeypatch, new, before, taken):
    from torchlet_b200 import ops
    from torchlet_b200.parts.latent_attention import prompt_tiles

    monkeypatch.setattr(ops, "latent_prompt_tokens", lambda: 256)
    ctx = SimpleNamespace(plans={}, decode_only=False, num_tokens=sum(new), num_requests=len(new), upload=torch.from_numpy,
                          req_indptr_host=np.concatenate([[0], np.cumsum(new)]), kv_before_host=np.array(before))
    plan = prompt_tiles(ctx)
    assert prompt_tiles(ctx) is plan and (plan is not None) == taken
    if taken:
        req, row, count = plan
        pairs = list(zip(req.tolist(), row.tolist()))
        assert len(pairs) == count and sorted(pairs) == [(r, start) for r, n in enumerate(new) for start in range(0, n, 256)]
        seen = [min(start + 256, new[r]) for r, start in pairs]
        assert seen == sorted(seen, reverse=True)
