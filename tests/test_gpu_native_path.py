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
