"""The fused decode step (spsattn_decoder_step) against the step made of library GEMMs and single
kernels, at the edges of its tiles, stages and row counts; the greedy choice on the device."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _engine(variant, layers, heads, hidden, inter, vocab, seed=3, block=64, window=5):
    import sps_b200
    from sps_b200.generation import random_state_dict
    dims = sps_b200.SPSDims(block_size=block, vocab_size=vocab, n_layer=layers, n_head=heads, hidden_size=hidden,
                            intermediate_size=inter, eos_token_id=vocab - 3, pad_token_id=vocab - 1,
                            predict_token_id=vocab - 2, window_size=window)
    return sps_b200.SPSGenerator(random_state_dict(dims, seed=seed), dims, variant=variant), dims


@pytest.mark.parametrize("variant,batch,heads,hidden,inter,vocab", [
    ("standard", 1, 1, 64, 16, 33),           # one row, odd vocabulary, less than one stage
    ("sps", 4, 2, 128, 80, 200),              # remainder of four steps of 16 columns
    ("reverse_sps", 5, 3, 192, 1040, 1001),   # ten rows: two row tiles; a second stage of 16 columns
    ("delayed_state", 8, 16, 1024, 2816, 2048),
    ("standard", 16, 16, 2048, 8192, 50304),  # the widest rows, several rounds of the head
    ("sps", 8, 16, 2048, 8192, 9473),
    ("standard", 12, 125, 2000, 1040, 500),   # two row tiles of nearly the widest rows (no multiple of 64 columns), heads of 16
    ("reverse_sps", 8, 62, 1984, 2064, 500),  # an intermediate size that is no multiple of 64, heads of 32
])
def test_fused_step_matches_the_separate_kernels(variant, batch, heads, hidden, inter, vocab):
    import sps_b200
    engine, dims = _engine(variant, 2, heads, hidden, inter, vocab)
    g = torch.Generator().manual_seed(7)
    prompt = torch.randint(0, vocab - 3, (batch, 9), generator=g)
    tokens = torch.randint(0, vocab - 3, (3, batch), generator=g)
    tokens[1, 0] = dims.eos_token_id                       # row 0 starts a new document in the third step
    active = torch.ones(batch, dtype=torch.bool)
    active[batch // 2] = batch == 1
    outs, states = [], []
    for fused in (True, False):
        state, _ = engine.prefill(prompt, 8)
        engine._bind_step(state)
        assert engine._step.fused
        engine._step.fused = fused
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


@pytest.mark.parametrize("variant,batch,heads,hidden,prompt,window", [
    ("reverse_sps", 2, 3, 192, 250, 16),      # one block per pair: three chunks, three groups of threads
    ("sps", 1, 4, 256, 330, 32),              # the same, the last rows of its range
    ("standard", 3, 2, 256, 250, 5),          # no ring
    ("sps", 3, 4, 256, 600, 64),              # the split kernel, and it alone advances the ring
    ("standard", 16, 32, 2048, 300, 5),       # the tensor-core kernel
    ("sps", 8, 32, 2048, 300, 200),           # the same with a ring that it streams
])
def test_fused_step_on_long_caches(variant, batch, heads, hidden, prompt, window):
    """Each decode attention kernel inside the step's chain of launches, against the same kernel behind
    separate ones: ring full and wrapping, a row that leaves a long cache for a new document."""
    import sps_b200
    steps = 4
    engine, dims = _engine(variant, 2, heads, hidden, 256, 500, block=prompt + 8, window=window)
    g = torch.Generator().manual_seed(prompt)
    ids = torch.randint(0, 497, (batch, prompt), generator=g)
    tokens = torch.randint(0, 497, (steps, batch), generator=g)
    tokens[1, 0] = dims.eos_token_id                       # row 0 starts a new document in the third step
    active = torch.ones(batch, dtype=torch.bool)
    if batch > 2:
        active[2] = False
    outs, states = [], []
    for fused in (True, False):
        state, _ = engine.prefill(ids, 8)
        engine._bind_step(state)
        assert engine._step.fused
        engine._step.fused = fused
        outs.append([engine.decode_one_token(state, t, active).float() for t in tokens])
        states.append(state)
    sps_b200.check_device_status()
    for a, b in zip(*outs):
        assert float((a - b).norm()) <= 2.0 ** -6 * float(b.norm())          # as above
    for name in ("br_len", "nw_len", "nw_pos", "processed_tokens", "next_doc_start"):
        assert torch.equal(getattr(states[0], name), getattr(states[1], name)), name
    assert states[0].br_len[:, 0].unique().tolist() == [2]
    for name in ("br_k", "br_v"):
        a, b = getattr(states[0], name), getattr(states[1], name)
        written = torch.zeros(batch, a.shape[3], dtype=torch.bool)           # by the steps
        written[1:, prompt:prompt + steps] = True
        written[0, prompt:prompt + 2] = written[0, :2] = True
        written[~active] = False
        written = written.cuda()
        keep = lambda x, rows: x.transpose(2, 3)[:, rows]                    # [L, rows, H, D]
        assert torch.equal(keep(a, ~written), keep(b, ~written))
        a, b = keep(a, written).float(), keep(b, written).float()
        assert bool((b.norm(dim=-1) > 0).all())
        # row by row: a row in a wrong place is as far off as its own norm
        assert bool(((a - b).norm(dim=-1) <= 2.0 ** -4 * b.norm(dim=-1)).all())
    for name in ("nw_k", "nw_v"):
        a, b = getattr(states[0], name).float(), getattr(states[1], name).float()
        assert bool(((a - b).norm(dim=-1) <= 2.0 ** -4 * b.norm(dim=-1)).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_weights_at_any_element_of_a_flat_buffer(dtype):
    """Projections, embedding and head as views at odd elements: the step runs, by library projections."""
    import sps_b200
    from sps_b200.generation import random_state_dict
    _, dims = _engine("sps", 2, 2, 128, 80, 200)
    sd = random_state_dict(dims, seed=3, dtype=dtype)
    flat = torch.empty(1 + sum(w.numel() + 1 for w in sd.values()), device="cuda", dtype=dtype)
    views, at = {}, 1
    for name, w in sd.items():
        if "norm" in name:
            views[name] = w
            continue
        at += 1 - at % 2                                   # an odd element
        views[name] = flat[at:at + w.numel()].view(w.shape).copy_(w)
        at += w.numel()
    g = torch.Generator().manual_seed(7)
    prompt, tokens = torch.randint(0, 197, (3, 9), generator=g), torch.randint(0, 197, (2, 3), generator=g)
    outs = []
    for params in (sd, views):
        engine = sps_b200.SPSGenerator(params, dims, variant="sps", param_dtype=dtype)
        state, logits = engine.prefill(prompt, 4)
        engine._bind_step(state)
        assert engine._step.fused == (params is sd and dtype == torch.bfloat16)
        engine._step.fused = False
        outs.append([logits.float()] + [engine.decode_one_token(state, t, torch.ones(3, dtype=torch.bool)).float() for t in tokens])
    sps_b200.check_device_status()
    for a, b in zip(*outs):
        # the library may take another algorithm for such operands: bf16 projections, as above
        assert float((a - b).norm()) <= 2.0 ** -6 * float(b.norm())


def test_one_token_or_flag_for_all_rows():
    engine, _ = _engine("sps", 1, 2, 128, 80, 200)
    prompt = torch.randint(0, 197, (3, 9), generator=torch.Generator().manual_seed(5))
    full = lambda x: torch.full((3,), x)
    state, _ = engine.prefill(prompt, 8)
    want = engine.decode_one_token(state, full(11), full(True))
    for token, active in ((torch.tensor(11), torch.tensor(True)), (torch.tensor([11.0]), torch.tensor([1])),
                          (full(11).int(), torch.tensor(True, device="cuda"))):
        state, _ = engine.prefill(prompt, 8)
        assert torch.equal(engine.decode_one_token(state, token, active), want)
    for token in (torch.zeros(2, dtype=torch.long), torch.zeros(1, 3, dtype=torch.long), torch.zeros(3, 1, dtype=torch.long)):
        with pytest.raises(RuntimeError):
            engine.decode_one_token(state, token, full(True))


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("bad", [-1, 200, 1 << 40])
def test_a_token_outside_the_vocabulary_concerns_its_row_alone(fused, bad):
    """The row sits the step out as if it were inactive, the check raises, and an attention call before
    the check still gives its numbers (a tensor-core kernel asks the status word before it starts)."""
    import sps_b200
    from sps_b200 import _lib
    engine, dims = _engine("sps", 2, 2, 128, 80, 200)
    g = torch.Generator().manual_seed(17)
    prompt = torch.randint(0, 197, (4, 9), generator=g)
    good = torch.randint(0, 197, (4,), generator=g)
    q, k, v = (torch.randn(1, 2, 256, 64, generator=g).bfloat16().cuda() for _ in range(3))
    want = sps_b200.sps_sliding_attention(q, k, v, 0.125, 8)
    outs, states = [], []
    for given in (bad, None):
        state, _ = engine.prefill(prompt, 8)
        engine._bind_step(state)
        engine._step.fused = fused
        token, active = good.clone(), torch.ones(4, dtype=torch.bool)
        if given is None:
            active[1] = False
        else:
            token[1] = given
        logits = [engine.decode_one_token(state, token, active)]
        if given is not None:
            assert torch.equal(sps_b200.sps_sliding_attention(q, k, v, 0.125, 8), want)
            with pytest.raises(_lib.SpsAttnError, match="vocabulary"):
                sps_b200.check_device_status()
        active[1] = True
        logits.append(engine.decode_one_token(state, good, active))
        sps_b200.check_device_status()
        outs.append(logits)
        states.append(state)
    for a, b in zip(*outs):
        assert torch.equal(a, b)
    assert bool((outs[0][0][1] == 0).all())
    for name in ("br_k", "br_v", "br_len", "nw_k", "nw_v", "nw_len", "nw_pos", "processed_tokens", "next_doc_start"):
        assert torch.equal(getattr(states[0], name), getattr(states[1], name)), name


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("vocab", [7, 64, 1003, 50304])
def test_greedy_choice_is_the_first_unsuppressed_maximum(dtype, vocab):
    import ctypes as C
    from sps_b200 import _lib
    lib, dev, batch, new = _lib.load(), torch.device("cuda"), 6, 2
    g = torch.Generator().manual_seed(vocab)
    z = torch.randint(-3, 4, (batch, vocab), generator=g).to(dtype)              # many ties
    z[1] = float("-inf")
    z[2, vocab // 2] = float("nan")
    z[3] = 0.0
    z[3, 0] = -0.0
    hidden = torch.randperm(vocab, generator=g)[: vocab // 3]
    ref = z.float().clone()
    ref[:, hidden] = float("-inf")
    want = torch.stack([torch.argmax(r) for r in ref])
    want[5] = vocab - 1                                                           # finished: pad
    words = torch.zeros((vocab + 31) // 32, dtype=torch.long)
    words.index_add_(0, hidden >> 5, torch.ones_like(hidden) << (hidden & 31))
    words = torch.where(words >= 1 << 31, words - (1 << 32), words).to(torch.int32).to(dev)
    zd = z.to(dev)
    out = torch.full((batch, new), -1, dtype=torch.long, device=dev)
    step = torch.ones(batch, dtype=torch.long, device=dev)
    finished = torch.tensor([0, 0, 0, 0, 0, 1], dtype=torch.uint8, device=dev)
    d, s = _lib.Decoder(), _lib.TokenSource()
    d.batch, d.vocab, d.pad, d.eos = batch, vocab, vocab - 1, vocab - 2
    d.param_dtype = _lib.DTYPE_BF16 if dtype == torch.bfloat16 else _lib.DTYPE_FP32
    s.logits, s.suppressed, s.generated = zd.data_ptr(), words.data_ptr(), out.data_ptr()
    s.step, s.finished, s.max_new, s.stop_on_eos = step.data_ptr(), finished.data_ptr(), new, 1
    _lib.check(lib.spsattn_decoder_choose(C.byref(d), C.byref(s), torch.cuda.current_stream().cuda_stream), "choose")
    keep = [i for i in range(batch) if not (i == 2 and vocab // 2 in hidden)]     # a hidden NaN counts as hidden
    assert torch.equal(out[keep, 1].cpu(), want[keep])
    assert bool((out[:, 0] == -1).all())


@pytest.mark.parametrize("variant,batch,heads,hidden,vocab", [
    ("standard", 1, 1, 64, 33),           # one warp with one output past the end
    ("reverse_sps", 8, 2, 128, 9473),     # eight rows, several rounds, odd vocabulary
    ("standard", 13, 2, 128, 50304),      # two row tiles
])
def test_head_leaves_the_choice_of_the_next_token(variant, batch, heads, hidden, vocab):
    """The key that the head leaves is that of the first unsuppressed maximum of the logits it wrote;
    a finished row leaves none, and the start of the step takes the old ones away."""
    import sps_b200
    engine, dims = _engine(variant, 1, heads, hidden, 64, vocab)
    g = torch.Generator().manual_seed(11)
    prompt = torch.randint(0, vocab - 3, (batch, 5), generator=g)
    hidden_ids = torch.randperm(vocab - 3, generator=g)[: vocab // 2]
    engine.generate(prompt, 3, stop_on_eos=False, forbidden_token_ids=hidden_ids, use_graph=False)
    s = engine._session
    assert engine._step.fused
    s.finished[batch // 2] = batch > 1
    s.counters[0].zero_()
    engine._token_body(s)
    sps_b200.check_device_status()
    z = s.next_logits.float()
    z[:, hidden_ids.to(z.device)] = float("-inf")
    z[:, dims.pad_token_id] = float("-inf")
    if engine.n_slot == 2:
        z[:, dims.predict_token_id] = float("-inf")
    want = torch.stack([torch.argmax(r) for r in z])
    got = (~s.counters[1]) & 0xffffffff
    for r in range(batch):
        if batch > 1 and r == batch // 2:
            assert int(s.counters[1][r]) == 0
        else:
            assert int(got[r]) == int(want[r])
