"""Decode steps whose layers run on the projections of 9 to 64 rows (spsattn_decoder_blocks, and
spsattn_decoder_step from 9 rows on) against the step made of library GEMMs and single kernels."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _engine(variant, layers, heads, hidden, inter, vocab, block, window=5, seed=3):
    """Norm weights are not the ones of a fresh model: each column has its own."""
    import sps_b200
    from sps_b200.generation import random_state_dict
    dims = sps_b200.SPSDims(block_size=block, vocab_size=vocab, n_layer=layers, n_head=heads, hidden_size=hidden,
                            intermediate_size=inter, eos_token_id=vocab - 3, pad_token_id=vocab - 1,
                            predict_token_id=vocab - 2, window_size=window)
    sd = random_state_dict(dims, seed=seed)
    g = torch.Generator(device="cuda").manual_seed(seed)
    for name, w in sd.items():
        if "norm" in name:
            w += (0.2 * torch.randn(w.shape, generator=g, device=w.device)).to(w.dtype)
    return sps_b200.SPSGenerator(sd, dims, variant=variant)


def _step64(engine, state, token, active):
    """Logits and new cache rows (k, v of every layer and slot) of one step on ``state`` as it is before it, in 64
    bits, rounded to bf16 where the step's tensors are bf16."""
    w, d, ns = engine.w, engine.dims, engine.n_slot
    b, h, hd, c = len(token), d.n_head, d.head_dim, d.hidden_size
    r = lambda t: t.to(torch.bfloat16).double()
    cpu = lambda t: t.detach().cpu().double()
    norm = lambda x, g: r(r(x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + d.norm_eps)) * cpu(g))
    ids = torch.stack([token] + [torch.full_like(token, d.predict_token_id)] * (ns - 1), dim=1)
    x = cpu(w.wte)[ids]                                                              # [B, ns, C]
    pos = torch.where(active, state.processed_tokens.cpu(), 0)
    cos, sin = cpu(engine.freqs)[pos][:, None, None].unbind(-1)                      # [B, 1, 1, hd / 2]
    new = []
    for layer in range(d.n_layer):
        qkv = r(norm(x, w.attn_norm[layer]) @ cpu(w.c_attn[layer]).T).view(b, ns, 3, h, hd)
        even, odd = qkv[:, :, :2, :, 0::2], qkv[:, :, :2, :, 1::2]
        rot = torch.empty_like(qkv[:, :, :2])
        rot[..., 0::2], rot[..., 1::2] = r(even * cos[:, None] - odd * sin[:, None]), r(even * sin[:, None] + odd * cos[:, None])
        q, k, v = rot[:, :, 0], rot[:, :, 1], qkv[:, :, 2]                           # [B, ns, H, hd]
        new.append((k, v))
        y = torch.empty(b, ns, h, hd, dtype=torch.double)
        ring, kept = [cpu(t[layer]) for t in (state.nw_k, state.nw_v)], [cpu(t[layer]) for t in (state.br_k, state.br_v)]
        for i in range(b):
            fresh = bool(state.next_doc_start[i]) and bool(active[i])               # forgets its caches
            n_ring = 0 if fresh or not engine.window_tokens else int(state.nw_len[layer, i])
            for j in range(h):
                n_kept = 0 if fresh else int(state.br_len[layer, i, j])
                keys = torch.cat([ring[0][i, j, :n_ring], kept[0][i, j, :n_kept], k[i, :, j]])
                vals = torch.cat([ring[1][i, j, :n_ring], kept[1][i, j, :n_kept], v[i, :, j]])
                scores = q[i, :, j] @ keys.T / math.sqrt(hd)
                if ns == 2:
                    scores[0, -1] = -math.inf                                       # the first row does not see the second
                y[i, :, j] = r(scores.softmax(-1) @ vals)
        x = r(x + r(y.reshape(b, ns, c) @ cpu(w.c_proj[layer]).T))
        gate, up = r(norm(x, w.mlp_norm[layer]) @ cpu(w.gate_up[layer]).T).chunk(2, dim=-1)
        x = r(x + r(r(r(torch.nn.functional.silu(gate)) * up) @ cpu(w.down[layer]).T))
    return r(norm(x[:, engine.pred_slot], w.out_norm) @ cpu(w.lm_head).T), new


@pytest.mark.parametrize("variant,batch,heads,hidden,inter,vocab,prompt,fused", [
    ("standard", 9, 1, 64, 64, 33, 9, True),            # narrow, up to 16 rows: decoder_step.cuh, two tiles of rows
    ("reverse_sps", 5, 2, 128, 192, 200, 9, True),
    ("sps", 9, 1, 64, 64, 33, 9, True),                 # 18 rows; one group of 64 columns, fewer outputs than a block holds
    ("reverse_sps", 9, 2, 128, 192, 200, 9, True),      # three groups
    ("standard", 9, 16, 1024, 2816, 200, 9, True),      # nine rows by row tiles
    ("reverse_sps", 7, 12, 768, 2048, 200, 9, True),    # fourteen, of 768 columns
    ("sps", 16, 5, 320, 576, 1001, 30, True),           # 32 rows; five and nine groups: a last stage that is not full
    ("standard", 17, 3, 192, 320, 200, 9, False),       # 17 rows, library head
    ("delayed_state", 17, 8, 512, 1024, 500, 140, False),   # 34 rows: three tiles of 16; ring counters left to c_proj
    ("standard", 33, 12, 768, 2048, 2048, 9, False),    # 33 rows
    ("sps", 32, 16, 1024, 2816, 2048, 20, False),       # 64 rows
    ("reverse_sps", 32, 16, 2048, 8192, 500, 9, False),
    ("standard", 64, 16, 2048, 8192, 500, 300, False),  # the tensor-core attention before c_proj
    ("sps", 9, 20, 2560, 4096, 500, 9, False),          # wider than the fused head takes
    ("standard", 1, 20, 2560, 4096, 500, 9, False),     # the same with one row,
    ("reverse_sps", 4, 20, 2560, 6912, 500, 9, False),  # and eight
    ("sps", 10, 8, 128, 320, 200, 30, True),            # heads of 16
    ("reverse_sps", 20, 24, 768, 1024, 500, 60, False), # heads of 32
])
def test_step_by_row_tiles_matches_the_separate_kernels(variant, batch, heads, hidden, inter, vocab, prompt, fused):
    import sps_b200
    engine = _engine(variant, 2, heads, hidden, inter, vocab, prompt + 8)
    dims = engine.dims
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
        # The same bits: both sum each output in one fp32 chain and round at the same places.  At a vocabulary of 1001 the
        # library's head splits its sums: a logit may round the other way, by a unit of the last place (2^-7 of it)
        assert torch.equal(a, b) or (vocab == 1001 and bool(((a - b).abs() <= 2.0 ** -7 * b.abs().amax(-1, keepdim=True)).all()))
        assert bool((a[~active] == 0).all())
    for name in ("br_len", "nw_len", "nw_pos", "processed_tokens", "next_doc_start"):
        assert torch.equal(getattr(states[0], name), getattr(states[1], name)), name
    for name in ("br_k", "br_v", "nw_k", "nw_v"):
        assert torch.equal(getattr(states[0], name), getattr(states[1], name)), name


@pytest.mark.parametrize("variant,batch,heads,hidden,inter,prompt", [
    ("sps", 9, 8, 128, 320, 30),                # heads of 16, row tiles of 18 rows
    ("reverse_sps", 5, 16, 1024, 2816, 140),    # ten rows
    ("standard", 17, 24, 768, 2048, 20),        # heads of 32, library head
    ("delayed_state", 20, 3, 192, 576, 12),     # 40 rows
    ("standard", 1, 10, 2560, 1024, 9),         # one row, heads of 256
])
def test_step_by_row_tiles_against_64_bits(variant, batch, heads, hidden, inter, prompt):
    """Every element.  fp32 sums instead of 64 bits move a value that is rounded to bf16 by a unit of its last place
    (2^-7 of it) at most; a rotated element is made of two of those and rounded again (1 + sqrt(2) units), and what
    such flips do to the sums behind them is below another unit of the row's largest: 4 units.  An element that is
    wrong is off by about its own size, a third of that largest."""
    import sps_b200
    close = lambda a, b: bool(((a - b).abs() <= 4 * 2.0 ** -7 * b.abs().amax(-1, keepdim=True)).all())
    engine = _engine(variant, 2, heads, hidden, inter, 500, prompt + 8)
    g = torch.Generator().manual_seed(hidden)
    ids = torch.randint(0, 497, (batch, prompt), generator=g)
    tokens = torch.randint(0, 497, (3, batch), generator=g)
    tokens[1, 0] = engine.dims.eos_token_id                # row 0 starts a new document in the third step
    active = torch.ones(batch, dtype=torch.bool)
    if batch > 1:
        active[batch // 2] = False
    state, _ = engine.prefill(ids, 8)
    for token in tokens:
        logits, new = _step64(engine, state, token, active)
        got = engine.decode_one_token(state, token, active).cpu().double()
        sps_b200.check_device_status()
        assert not engine._step.fused or batch * engine.n_slot > 8
        assert close(got[active], logits[active])
        for layer, (k, v) in enumerate(new):
            for cache, rows in ((state.br_k, k), (state.br_v, v)):
                for i in active.nonzero().flatten().tolist():
                    assert close(cache[layer, i, :, int(state.br_len[layer, i, 0]) - 1].cpu().double(), rows[i, engine.retained_slot])


@pytest.mark.parametrize("variant,batch,heads,hidden,inter", [("standard", 9, 6, 384, 192), ("reverse_sps", 7, 8, 512, 1024)])
def test_captured_steps_that_go_by_another_route(variant, batch, heads, hidden, inter):
    """Few rows of a light layer: row tiles in a graph, decoder_step.cuh launch by launch; the same bits."""
    engine = _engine(variant, 2, heads, hidden, inter, 500, 40)
    ids = torch.randint(0, 497, (batch, 20), generator=torch.Generator().manual_seed(2))
    outs = []
    for graph in (True, False):
        engine._session = None
        tokens = engine.generate(ids, 12, stop_on_eos=False, use_graph=graph)
        assert engine._step.fused
        st = engine._session.state
        outs.append([t.clone() for t in (tokens, engine._session.next_logits, st.br_k, st.br_v, st.br_len, st.nw_k, st.nw_v, st.nw_pos)])
    assert all(torch.equal(a, b) for a, b in zip(*outs))


def test_layers_directly_behind_a_launch_that_writes_their_caches():
    """spsattn_decoder_blocks has no launch of its own before the first layer: what stands before it on the
    stream may have let its dependents go and still be writing the cache rows that the layer's attention reads."""
    import ctypes as C
    import sps_b200
    from sps_b200 import _lib
    from sps_b200.attention import _status
    prompt, batch, hidden, heads, window = 120, 6, 512, 8, 16
    engine = _engine("reverse_sps", 2, heads, hidden, 1024, 500, prompt + 8, window)
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
    engine = _engine("sps", 1, 20, 2560, 10240, 500, 16)
    engine._bind_step(engine.build_decode_state(batch, 8))
    assert not engine._step.fused and engine._step.blocks is blocks
