"""One block per (sequence, head) against the split form: the same bits, at the borders of batches,
chunks and groups of threads."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def decode_path():
    from sps_b200 import _lib
    lib = _lib.load()
    yield lambda p: _lib.check(lib.spsattn_debug_decode_path(p), "decode_path")
    lib.spsattn_debug_decode_path(0)


@pytest.mark.parametrize("D,dtype", [(8, torch.bfloat16), (16, torch.bfloat16), (64, torch.bfloat16), (64, torch.float16), (128, torch.bfloat16)])
@pytest.mark.parametrize("nq", [1, 2])
@pytest.mark.parametrize("ring,cap", [(0, 1), (5, 129), (64, 448), (64, 960)])      # 1, 2, 4 and 8 chunks of 128
def test_pair_kernel_equals_the_split_kernel(decode_path, D, dtype, nq, ring, cap):
    import sps_b200
    g = torch.Generator(device="cuda").manual_seed(cap + D)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").to(dtype)
    S, H = 7, 3
    k, v = rnd(S, H, cap, D), rnd(S, H, cap, D)
    lens = torch.randint(0, cap + 1, (S, H), generator=g, device="cuda")
    lens[0], lens[1], lens[2] = cap, 0, min(cap, 64)
    lens[3], lens[4] = min(cap, 128 - ring), min(cap, 129 - ring)
    segs = [sps_b200.KVSegment(k, v, lens)]
    if ring:
        rl = torch.tensor([ring, 0, 1, ring, ring, 2, ring], device="cuda")
        segs.insert(0, sps_b200.KVSegment(rnd(S, H, ring, D), rnd(S, H, ring, D), rl))
    q = rnd(S, nq, H, D)
    extras = [(rnd(S, H, D), rnd(S, H, D), (1 << nq) - 1), (rnd(S, H, D), rnd(S, H, D), 2)][:nq]
    out = []
    for path in (1, 3):
        decode_path(path)
        out.append(sps_b200.decode_attention(q, segs, extras))
    assert torch.equal(out[0], out[1])
    decode_path(3)
    out = sps_b200.decode_attention(q, segs, [])                      # sequence 1 sees nothing in its cache
    decode_path(1)
    assert torch.equal(out, sps_b200.decode_attention(q, segs, []))


def test_pair_kernel_refuses_more_chunks_than_it_holds(decode_path):
    import sps_b200
    from sps_b200 import _lib
    k = torch.zeros(1, 1, 1100, 64, device="cuda", dtype=torch.bfloat16)
    seg = sps_b200.KVSegment(k, k, torch.tensor([3], device="cuda"))
    decode_path(3)
    with pytest.raises(_lib.SpsAttnError):
        sps_b200.masked_kv_attention(k[:, :, 0], [seg], attn_dtype=torch.bfloat16)
