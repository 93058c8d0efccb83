"""Grouped-query attention of the Llama layers under every choice of PyTorch's attention kernels."""
import pytest
import torch
from torch.nn.attention import SDPBackend, sdpa_kernel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("backend", ["FLASH_ATTENTION", "CUDNN_ATTENTION", "EFFICIENT_ATTENTION", "MATH"])
@pytest.mark.parametrize("d", [64, 128])
def test_every_attention_kernel_serves_grouped_queries(cuda, backend, d):
    """Same forward and backward within the rounding of bf16 probabilities and outputs (2^-8 of the largest value, in a sum of
    a few terms) whichever kernel a program has enabled."""
    from coccl_b200.models.gpt import GPTConfig, GPTStage
    cfg = GPTConfig(arch="llama", n_layer=1, hidden=4 * d, n_head=4, n_kv_head=2, ffn=256, seq_len=96, vocab=256, tie_embeddings=False)
    layer = GPTStage(cfg, cuda, seed=3).layers[0]
    qkv = torch.randn(2 * 96, 8 * d, device=cuda, generator=torch.Generator(cuda).manual_seed(1)).to(torch.bfloat16)
    dy = torch.randn(2 * 96, 4 * d, device=cuda, generator=torch.Generator(cuda).manual_seed(2)).to(torch.bfloat16)

    def run(x):
        x = x.clone().requires_grad_(True)
        o = layer.attention(x, 2, 96)
        o.backward(dy)
        return o.detach(), x.grad
    want = run(qkv)
    with sdpa_kernel(getattr(SDPBackend, backend)):
        got = run(qkv)
    for g, w in zip(got, want):
        assert (g.float() - w.float()).abs().max() <= 4 * 2.0 ** -8 * w.float().abs().max()
