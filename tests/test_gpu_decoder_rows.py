"""Decode steps whose layers run on the projections of 9 to 64 rows (spsattn_decoder_blocks, and
spsattn_decoder_step from 9 rows on) against the step made of library GEMMs and single kernels."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant,batch,heads,hidden,inter,vocab,prompt,fused", [
    ("standard", 9, 1, 64, 64, 33, 9, True),            # narrow, up to 16 rows: decoder_step.cuh, two tiles of rows
    ("reverse_sps", 5, 2, 128, 192, 200, 9, True),
    ("sps", 9, 1, 64, 64, 33, 9, True),                 # 18 rows; one group of 64 columns, fewer outputs than a block holds
    ("reverse_sps", 9, 2, 128, 192, 200, 9, True),      # three groups
    ("standard", 9, 6, 384, 192, 200, 9, True),         # the narrowest step of 9 rows that goes by row tiles
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


def test_layers_directly_behind_a_launch_that_writes_their_caches():
    """spsattn_decoder_blocks has no launch of its own before the first layer: what stands before it on the
    stream may have let its dependents go and still be writing the cache rows that the layer's attention reads."""
    import ctypes as C
    import sps_b200
    from sps_b200 import _lib
    from sps_b200.attention import _status
    from sps_b200.generation import random_state_dict
    prompt, batch, hidden, heads, window = 120, 6, 512, 8, 16
    dims = sps_b200.SPSDims(block_size=prompt + 8, vocab_size=500, n_layer=2, n_head=heads, hidden_size=hidden, intermediate_size=1024,
                            eos_token_id=497, pad_token_id=499, predict_token_id=498, window_size=window)
    engine = sps_b200.SPSGenerator(random_state_dict(dims, seed=3), dims, variant="reverse_sps")
    ids = torch.randint(0, 497, (batch, prompt), generator=torch.Generator().manual_seed(2))
    lib, status = engine.lib, _status(engine.device).data_ptr()
    stream = torch.cuda.current_stream().cuda_stream
    outs = []
    for wait in (True, False, False, False):
        state, _ = engine.prefill(ids, 8)                # rings full: a new row takes an old one's place, the length stays
        engine._bind_step(state)
        s = engine._step
        token, active = torch.full((batch,), 7, device="cuda"), torch.ones(batch, dtype=torch.bool, device="cuda")
        source = _lib.TokenSource()
        source.token_in, source.active_in = token.data_ptr(), active.data_ptr()
        _lib.check(lib.spsattn_decoder_start(C.byref(s.decoder), C.byref(source), status, stream), "start")
        g = torch.Generator(device="cuda").manual_seed(4)
        q = torch.randn(s.q.shape, generator=g, device="cuda").to(s.q.dtype)
        for buf in (s.k2, s.v2):
            buf.copy_(torch.randn(buf.shape, generator=g, device="cuda"))
        torch.cuda.synchronize()
        segs, n_seg, extras, append = s.layer_args[0]
        out = torch.empty_like(q)
        _lib.check(lib.spsattn_decode_step(q.data_ptr(), 2, out.data_ptr(), _lib.DTYPE_BF16, segs, n_seg, extras, 2, C.byref(append), batch,
                                           heads, hidden // heads, _lib.DTYPE_BF16, 0.125, s.ws.data_ptr(), s.ws_bytes, status, stream), "step")
        if wait:
            torch.cuda.synchronize()
        _lib.check(lib.spsattn_decoder_blocks(C.byref(s.decoder), s.xn.data_ptr(), status, stream), "blocks")
        sps_b200.check_device_status()
        outs.append([t.clone() for t in (out, s.xn, state.nw_k, state.nw_v, state.br_k, state.br_v, state.nw_pos, state.br_len)])
    assert state.nw_len.unique().tolist() == [window] and state.br_len[0].unique().tolist() == [prompt + 2]
    for other in outs[1:]:
        assert all(torch.equal(a, b) for a, b in zip(outs[0], other))


@pytest.mark.parametrize("batch,blocks", [(24, True), (25, False)])
def test_route_of_wide_steps(batch, blocks):
    import sps_b200
    from sps_b200.generation import random_state_dict
    dims = sps_b200.SPSDims(block_size=16, vocab_size=500, n_layer=1, n_head=20, hidden_size=2560, intermediate_size=10240, eos_token_id=497,
                            pad_token_id=499, predict_token_id=498, window_size=5)
    engine = sps_b200.SPSGenerator(random_state_dict(dims, seed=3), dims, variant="sps")
    engine._bind_step(engine.build_decode_state(batch, 8))
    assert not engine._step.fused and engine._step.blocks is blocks
