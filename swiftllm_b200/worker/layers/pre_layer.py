"""Reference: swiftllm/worker/layers/pre_layer.py:6-20 (token embedding lookup)."""
import torch

from swiftllm_b200.worker.kernels.row_ops import embed_and_zero


class LlamaPreLayer:
    def __init__(self, model_config, weights):
        self.model_config = model_config
        self.weights = weights

    def forward(self, input_ids: torch.Tensor) -> torch.Tensor:
        return torch.embedding(self.weights.wte, input_ids, padding_idx=-1)

    def forward_with_residual(self, input_ids: torch.Tensor):
        """-> (embeddings, the zero residual stream that the first layer adds them to)"""
        return embed_and_zero(self.weights.wte, input_ids)
