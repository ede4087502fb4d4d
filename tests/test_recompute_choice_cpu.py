"""The choice of what a training step recomputes, by the memory that is free."""
import pytest


@pytest.mark.parametrize("tokens", [300, 2048, 4096, 16384])
@pytest.mark.parametrize("model", ["qwen2.5-0.5b", "qwen2.5-7b"])
def test_room_for_the_kept_logits(model, tokens):
    from art_b200.models.config import PRESETS
    from art_b200.models.native import activation_bytes_per_token, pick_recompute
    from art_b200.ops.logprob_loss import kept_rows

    cfg = PRESETS[model]
    logits = 4 * kept_rows(tokens) * cfg.vocab_size
    chosen = {pick_recompute(cfg, tokens, cfg.num_layers, free) for free in range(1 << 28, 160 << 30, 1 << 27)}
    assert chosen == {"none", "mlp", "full"}
    for free in range(1 << 28, 160 << 30, 1 << 27):
        mode = pick_recompute(cfg, tokens, cfg.num_layers, free)
        if mode != "full":
            assert tokens * cfg.num_layers * activation_bytes_per_token(cfg, mode) + logits < free


def test_rows_of_kept_logits():
    from art_b200.ops.logprob_loss import LOGIT_ROWS, kept_rows

    for M in (1, 255, 2047, 2048, 2049, 4095, 4097, 16384):
        assert kept_rows(M) <= min(M, max(LOGIT_ROWS, M // 2 + 256)) and -(-M // kept_rows(M)) <= 2
