"""Decode steps whose layers run on the projections of 9 to 64 rows (spsattn_decoder_blocks, and
spsattn_decoder_step from 9 rows on) against the step made of library GEMMs and single kernels."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant,batch,heads,hidden,inter,vocab,prompt,fused", [
    ("standard", 9, 1, 64, 64, 33, 9, True),            # one group of 64 columns, fewer outputs than a block holds
    ("reverse_sps", 5, 2, 128, 192, 200, 9, True),      # ten rows; three groups
    ("sps", 16, 5, 320, 576, 1001, 30, True),           # 32 rows; five and nine groups: a last stage that is not full
    ("standard", 17, 3, 192, 320, 200, 9, False),       # 17 rows, library head
    ("delayed_state", 17, 8, 512, 1024, 500, 140, False),   # 34 rows: three tiles of 16; ring counters left to c_proj
    ("standard", 33, 12, 768, 2048, 2048, 9, False),    # 33 rows
    ("sps", 32, 16, 1024, 2816, 2048, 20, False),       # 64 rows
    ("reverse_sps", 32, 16, 2048, 8192, 500, 9, False),
    ("standard", 64, 16, 2048, 8192, 500, 300, False),  # the tensor-core attention before c_proj
    ("sps", 9, 20, 2560, 4096, 500, 9, False),          # wider than the fused head takes
])
def test_step_by_row_tiles_matches_the_separate_kernels(variant, batch, heads, hidden, inter, vocab, prompt, fused):
    import sps_b200
    from sps_b200.generation import random_state_dict
    dims = sps_b200.SPSDims(block_size=prompt + 8, vocab_size=vocab, n_layer=2, n_head=heads, hidden_size=hidden,
                            intermediate_size=inter, eos_token_id=vocab - 3, pad_token_id=vocab - 1,
                            predict_token_id=vocab - 2, window_size=5)
    engine = sps_b200.SPSGenerator(random_state_dict(dims, seed=3), dims, variant=variant)
    g = torch.Generator().manual_seed(hidden + batch)
    ids = torch.randint(0, vocab - 3, (batch, prompt), generator=g)
    tokens = torch.randint(0, vocab - 3, (3, batch), generator=g)
    tokens[1, 0] = dims.eos_token_id                       # row 0 starts a new document in the third step
    active = torch.ones(batch, dtype=torch.bool)
    active[batch // 2] = False
    outs, states = [], []
    for by_rows in (True, False):
        state, _ = engine.prefill(ids, 8)
        engine._bind_step(state)
        s = engine._step
        assert (s.fused, s.blocks) == (fused, not fused)
        if not by_rows:
            s.fused = s.blocks = False
        outs.append([engine.decode_one_token(state, t, active).float() for t in tokens])
        states.append(state)
    sps_b200.check_device_status()
    for a, b in zip(*outs):
        # both round every projection to bf16; where their fp32 sums round differently at all, a value
        # moves by one unit of the last place (2^-8), and the logits by a fraction of their norm
        assert float((a - b).norm()) <= 2.0 ** -6 * float(b.norm())
        assert bool((a[~active] == 0).all())
    for name in ("br_len", "nw_len", "nw_pos", "processed_tokens", "next_doc_start"):
        assert torch.equal(getattr(states[0], name), getattr(states[1], name)), name
    for name in ("br_k", "br_v", "nw_k", "nw_v"):
        a, b = getattr(states[0], name).float(), getattr(states[1], name).float()
        # row by row: a row in a wrong place is as far off as its own norm
        assert bool(((a - b).norm(dim=-1) <= 2.0 ** -4 * b.norm(dim=-1)).all()), name
