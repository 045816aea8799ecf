"""The native host path: the ticket and record buffers that decode calls of different sizes share
on a stream, and differentiation of a prefill call twice."""

import math

import pytest
import torch

from oracle import sps_oracle as orc

pytestmark = pytest.mark.gpu


def test_decode_calls_of_different_sizes_share_their_buffers():
    """Large, small and large again, on two streams: tickets of one size must be zero for the next."""
    import sps_b200
    g = torch.Generator().manual_seed(3)
    bf = torch.bfloat16
    cases = []
    for s, h, d, cap in ((1, 3, 64, 40), (40, 12, 64, 700), (2, 1, 128, 3000), (30, 16, 128, 500), (1, 3, 64, 40)):
        q = torch.randn(s, h, d, generator=g).to(bf)
        k, v = (torch.randn(s, h, cap, d, generator=g).to(bf) for _ in range(2))
        lens = torch.randint(0, cap + 1, (s, h), generator=g)
        ref = orc.decode_attention(q.unsqueeze(1), [orc.Segment(k, v, lens)], [])[:, 0]
        cases.append(([x.cuda() for x in (q, k, v, lens)], ref))
    for stream in (torch.cuda.current_stream(), torch.cuda.Stream()):
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            for (q, k, v, lens), ref in cases * 2:
                out = sps_b200.masked_kv_attention(q, [sps_b200.KVSegment(k, v, lens)], attn_dtype=bf)
                # bf16 operands, probabilities rounded to bf16 at most: the tolerance of the decode tests
                assert float((out.cpu() - ref).abs().max()) <= 2e-2


def test_a_second_differentiation_is_refused():
    import sps_b200
    q, k, v = (torch.randn(1, 2, 64, 64, device="cuda", dtype=torch.bfloat16, requires_grad=True) for _ in range(3))
    o = sps_b200.sps_sliding_attention(q, k, v, 1 / math.sqrt(64), 8)
    d_o = torch.randn_like(o, requires_grad=True)
    (dq,) = torch.autograd.grad(o, q, d_o, create_graph=True)
    with pytest.raises(RuntimeError):
        dq.float().sum().backward()


def test_hooks_on_saved_tensors_see_the_operands_and_results_alone():
    """Hooks may give back other values than they were given; what the forward found out about the
    documents (row indices) is none of their business."""
    import sps_b200
    q, k, v = (torch.randn(1, 2, 64, 64, device="cuda", dtype=torch.bfloat16, requires_grad=True) for _ in range(3))
    docs = torch.arange(64, device="cuda").div(8, rounding_mode="floor").unsqueeze(0)
    packed, grads = [], []
    for hooked in (False, True):
        pack = lambda x: (packed.append(x.dtype), x)[1]
        with torch.autograd.graph.saved_tensors_hooks(pack if hooked else (lambda x: x), lambda x: x):
            o = sps_b200.sps_sliding_attention(q, k, v, 1 / math.sqrt(64), 8, documents_idx_BxT=docs)
            grads.append(torch.autograd.grad(o, (q, k, v), torch.ones_like(o)))
    assert packed == [torch.bfloat16] * 4 + [torch.float32]
    for a, b in zip(*grads):
        assert torch.equal(a, b)


@pytest.mark.parametrize("call", ["prefill", "backward", "decode", "kv_update", "engine"])
def test_other_threads_run_while_a_launch_waits_for_room_in_its_queue(call):
    """A launch blocks while its stream's queue is full.  What empties the queue may depend on another
    Python thread (a collective's other rank), so the interpreter lock must not be held meanwhile."""
    import threading
    import time
    import sps_b200
    from sps_b200.attention import prefill_attention_backward
    bf = torch.bfloat16
    rnd = lambda *s: torch.randn(s, device="cuda").to(bf)
    if call in ("prefill", "backward"):
        q, k, v = (rnd(1, 1, 64, 64).requires_grad_(call == "backward") for _ in range(3))
        with torch.no_grad():
            o, lse = sps_b200.prefill_attention(q, k, v, 0.125, persistent_parity=0, temporary_window=8, return_lse=True)
        run = ((lambda: sps_b200.sps_sliding_attention(q, k, v, 0.125, 8)) if call == "prefill" else
               (lambda: prefill_attention_backward(q.detach(), k.detach(), v.detach(), o, lse, o, 0.125,
                                                   persistent_parity=0, temporary_window=8)))
    elif call == "decode":
        q, seg = rnd(1, 1, 64), sps_b200.KVSegment(rnd(1, 1, 8, 64), rnd(1, 1, 8, 64), torch.tensor([8], device="cuda"))
        run = lambda: sps_b200.masked_kv_attention(q, [seg], attn_dtype=bf)
    elif call == "kv_update":
        k, v, row = rnd(1, 1, 8, 64), rnd(1, 1, 8, 64), rnd(1, 1, 64)
        length, active = torch.zeros(1, 1, dtype=torch.long, device="cuda"), torch.ones(1, dtype=torch.bool, device="cuda")
        run = lambda: sps_b200.fused_sps_kv_update(
            nw_k=None, nw_v=None, nw_len=None, nw_pos=None, br_k=k, br_v=v, br_len=length, k_window_BxHxD=None,
            v_window_BxHxD=None, k_retained_BxHxD=row, v_retained_BxHxD=row, active_mask_B=active, window_tokens=0)
    else:
        from sps_b200.generation import random_state_dict
        dims = sps_b200.SPSDims(block_size=64, vocab_size=200, n_layer=4, n_head=2, hidden_size=128, intermediate_size=80,
                                eos_token_id=197, pad_token_id=199, predict_token_id=198)
        engine = sps_b200.SPSGenerator(random_state_dict(dims), dims)
        ext, model = engine._native()
        ids = torch.randint(0, 197, (2, 16), device="cuda")
        pos = torch.arange(16, device="cuda").expand(2, -1)
        docs = torch.zeros(2, 16, dtype=torch.long, device="cuda")
        run = lambda: ext.engine_prefill(model, ids, pos, docs, None, None)
    run()
    torch.cuda.synchronize()
    gaps, done = [0.0], threading.Event()

    def tick():
        last = time.perf_counter()
        while not done.is_set():
            time.sleep(0.002)
            now = time.perf_counter()
            gaps[0] = max(gaps[0], now - last)
            last = now

    thread = threading.Thread(target=tick)
    thread.start()
    try:
        torch.cuda._sleep(int(2e9))                       # about a second of the GPU
        began = time.perf_counter()
        for _ in range(6000 if call != "engine" else 200):    # some thousands of launches: more than a queue holds
            run()
        blocked = time.perf_counter() - began
        torch.cuda.synchronize()
    finally:
        done.set()
        thread.join()
    assert blocked > 0.5                                   # the queue was full
    assert gaps[0] < 0.3


def test_running_out_of_memory_raises_torchs_error():
    """Programs that look for a batch that fits catch it by its type."""
    import sps_b200
    one = torch.zeros(1, 1, 1, 64, device="cuda", dtype=torch.bfloat16)
    q = one.expand(1, 1, 1 << 40, 64)                      # its copy would take 128 TB
    with pytest.raises(torch.OutOfMemoryError):
        sps_b200.full_attention(q, q, q, 0.125)
    seg = sps_b200.KVSegment(one, one, torch.tensor([1], device="cuda"))
    with pytest.raises(torch.OutOfMemoryError):
        sps_b200.masked_kv_attention(one[0].expand(1 << 40, 1, 64), [seg], attn_dtype=torch.bfloat16)
    with pytest.raises(TypeError):
        sps_b200.masked_kv_attention(one[0], 3, attn_dtype=torch.bfloat16)


def test_numbers_of_any_type_that_int_takes():
    import numpy as np
    import sps_b200
    bf = torch.bfloat16
    q, k, v = (torch.randn(1, 2, 96, 64, device="cuda").to(bf) for _ in range(3))
    call = lambda tw, pw, **kw: sps_b200.prefill_attention(q, k, v, 0.125, temporary_window=tw, persistent_window=pw,
                                                           **{"persistent_parity": 0, **kw})
    want = call(5, 9)
    for tw, pw in ((5.0, 9.7), (np.int32(5), np.float64(9)), (torch.tensor(5), torch.tensor(9.0, device="cuda"))):
        assert torch.equal(call(tw, pw, persistent_parity=np.float32(0), mask_flags=0.0), want)
    for long in (1 << 70, -(1 << 70)):
        assert torch.equal(call(long, long), call(200 if long > 0 else -1, 200 if long > 0 else -1))
    with pytest.raises((TypeError, ValueError)):
        call(5, "nine")
    # decode: query masks, the scan limit of a segment; cache update: ring size
    kc, vc = torch.randn(1, 2, 8, 64, device="cuda").to(bf), torch.randn(1, 2, 8, 64, device="cuda").to(bf)
    qd, e = torch.randn(1, 2, 2, 64, device="cuda").to(bf), torch.randn(1, 2, 64, device="cuda").to(bf)
    seg = lambda cap: sps_b200.KVSegment(kc, vc, torch.tensor([8], device="cuda"), max_len_cap=cap)
    want = sps_b200.decode_attention(qd, [seg(4)], [(e, e, 2)], segment_query_masks=[1])
    assert torch.equal(sps_b200.decode_attention(qd, [seg(4.0)], [(e, e, 2.0)], segment_query_masks=[np.float64(1)]), want)
    assert torch.equal(sps_b200.decode_attention(qd, [seg(1 << 70)], []), sps_b200.decode_attention(qd, [seg(None)], []))
    lens = []
    for window in (4, 4.0):
        ring = torch.zeros(1, dtype=torch.long, device="cuda")
        sps_b200.fused_sps_kv_update(
            nw_k=kc.clone(), nw_v=vc.clone(), nw_len=ring, nw_pos=torch.zeros_like(ring), br_k=kc.clone(), br_v=vc.clone(),
            br_len=torch.zeros(1, 2, dtype=torch.long, device="cuda"), k_window_BxHxD=e, v_window_BxHxD=e, k_retained_BxHxD=e,
            v_retained_BxHxD=e, active_mask_B=torch.ones(1, dtype=torch.bool, device="cuda"), window_tokens=window)
        lens.append(int(ring))
    assert lens == [1, 1]
