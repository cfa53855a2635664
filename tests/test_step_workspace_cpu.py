"""What a model's steps keep between kernels is left free beside the token caches."""

import pytest
import torch

from mllm_b200 import ops
from mllm_b200.configs import ServerConfig
from mllm_b200.executor import ModelRunner
from mllm_b200.executor import model_runner as runner
from mllm_b200.models.qwen3_5 import Qwen3_5ForCausalLM


def test_memory_profile_leaves_room_for_the_workspace(monkeypatch):
    mr = ModelRunner(ServerConfig(model_path="preset:qwen3-tiny", dtype="float32", max_running_requests=2, mem_fraction_static=0.8), device="cpu")
    mr.initialize()
    mr._pre_load_avail_gib = 100.0
    monkeypatch.setattr(runner, "get_available_gpu_memory", lambda *_a, **_k: 80.0)
    assert Qwen3_5ForCausalLM.step_workspace_bytes == ops.GDN_WORKSPACE_BYTES > 0
    mr.model.step_workspace_bytes = Qwen3_5ForCausalLM.step_workspace_bytes
    mr.device = torch.device("cuda", 0)
    assert mr._profile_max_num_tokens().rest_gib == pytest.approx(60.0 - ops.GDN_WORKSPACE_BYTES / 2 ** 30)
