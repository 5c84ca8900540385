"""Page copies queued on the executor's stream outlive the call that queued them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_page_copies_keep_their_index_tensors():
    from cubic_serve_b200.executor.gpu_executor import GpuExecutor
    from cubic_serve_b200.models.config import ModelConfig, QuantSpec
    from cubic_serve_b200.models.decoder import DecoderRunner, random_decoder_weights
    cfg = ModelConfig(name="copies", num_layers=2, hidden_size=512, num_q_heads=8, num_kv_heads=2, head_dim=128, intermediate_size=512, vocab_size=512,
                      rope_theta=1e6, quant=QuantSpec("none", 16, 0))
    n = 300
    ex = GpuExecutor(DecoderRunner(cfg, random_decoder_weights(cfg, "cuda", seed=0), num_pages=2 * n, max_tokens=64), max_rows=2, max_prefill_tokens=64, max_model_len=64)
    for kv in ex.runner.kv:
        kv[:n].random_(0, 255)
    torch.cuda.synchronize()
    with torch.cuda.stream(ex.stream):
        torch.cuda._sleep(20_000_000)                    # the copies wait behind other work of the stream
    ex.copy_pages([(i, n + i) for i in range(n)])
    later = [torch.full((n,), -1, dtype=torch.int32, device="cuda") for _ in range(4)]       # takes the memory of what was freed
    torch.cuda.synchronize()
    assert all((t == -1).all() for t in later)
    for kv in ex.runner.kv:
        assert torch.equal(kv[:n], kv[n:])
