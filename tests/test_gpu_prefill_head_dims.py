"""Head dims 16, 32 and 256 on the tensor-core kernel: tile edges, views, precision of the probabilities."""

import math

import pytest
import torch

from oracle import sps_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [16, 32, 256])
@pytest.mark.parametrize("n,parity,dtype", [(2, 0, torch.bfloat16), (130, 1, torch.bfloat16), (126, 0, torch.float16),
                                            (257, -1, torch.bfloat16), (640, 1, torch.float16)])
def test_other_head_dims_at_tile_edges(d, n, parity, dtype):
    import sps_b200
    g = torch.Generator().manual_seed(n + d)
    # token-major views with rows inside a wider buffer, as a fused projection gives them
    buf = torch.randn(2, n, 3, 3 * d, generator=g).to(dtype)
    q, k, v = (buf[:, :, :, i * d:(i + 1) * d].transpose(1, 2) for i in range(3))
    docs = (torch.arange(n) // 90).expand(2, n).contiguous() if n > 130 else None
    dev = buf.cuda()
    qd, kd, vd = (dev[:, :, :, i * d:(i + 1) * d].transpose(1, 2) for i in range(3))
    out, lse = sps_b200.prefill_attention(qd, kd, vd, 1 / math.sqrt(d), persistent_parity=parity, temporary_window=9,
                                          documents_idx=None if docs is None else docs.cuda(), return_lse=True)
    ref = orc.prefill_attention(q, k, v, 1 / math.sqrt(d), persistent_parity=parity, temporary_window=9, docs=docs)
    sps_b200.check_device_status()
    # probabilities keep about 16 bits, so what is left is the rounding of the result: half a unit of
    # the last place, and 16 bits of probability on values of up to 5
    # (bf16 stores 7 bits of mantissa, fp16 10: half a unit is at most 2^-8 and 2^-11 of the value)
    half_ulp = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    err = (out.float().cpu() - ref).abs()
    assert bool((err <= 1.01 * half_ulp * ref.abs() + 5 * 2.0 ** -14).all()), float(err.max())
    assert bool(torch.isfinite(lse).all())


@pytest.mark.parametrize("d,dtype", [(16, torch.bfloat16), (32, torch.float16), (256, torch.bfloat16)])
@pytest.mark.parametrize("parity,docs", [(-1, "ordered"), (0, None), (1, "mixed"), (0, "ordered")])
def test_a_value_that_is_not_finite_stays_with_the_rows_that_see_it(d, dtype, parity, docs):
    """Infinities and NaN in value rows reach the results of the rows that see them and no others,
    although a tile's products multiply the hidden ones too."""
    import sps_b200
    g = torch.Generator().manual_seed(d)
    n, scale = 260, 1 / math.sqrt(d)
    buf = torch.randn(2, n, 2, 3 * d, generator=g).to(dtype)
    q, k, v = (buf[:, :, :, i * d:(i + 1) * d].transpose(1, 2) for i in range(3))
    v[0, 0, 40, 3], v[0, 1, 200, d - 1], v[1, 0, 259] = float("inf"), float("-inf"), float("nan")
    v[1, 1, 100, 0], v[1, 1, 171, 0] = float("inf"), float("-inf")
    ids = None if docs is None else (torch.arange(n) // 90 if docs == "ordered" else torch.arange(n) // 2 % 3).expand(2, n).contiguous()
    dev = buf.cuda()
    qd, kd, vd = (dev[:, :, :, i * d:(i + 1) * d].transpose(1, 2) for i in range(3))
    vis = torch.from_numpy(orc.visible_mask(n, persistent_parity=parity, temporary_window=9,
                                            docs_row=None if ids is None else ids[0].numpy()))
    s = (q.float() @ k.float().transpose(-1, -2)) * scale
    p = torch.softmax(s.masked_fill(~vis, float("-inf")), dim=-1)
    ref = torch.stack([torch.stack([torch.where(vis[:, :, None], p[b, h][:, :, None] * v[b, h].float(), 0.0).sum(1)
                                    for h in range(2)]) for b in range(2)])
    for lse in (False, True):          # without it the blocks work the documents out themselves
        out = sps_b200.prefill_attention(qd, kd, vd, scale, persistent_parity=parity, temporary_window=9,
                                         documents_idx=None if ids is None else ids.cuda(), return_lse=lse)
        out = (out[0] if lse else out).float().cpu()
        assert torch.equal(torch.isnan(out), torch.isnan(ref)) and torch.equal(torch.isinf(out), torch.isinf(ref))
        assert torch.equal(out[torch.isinf(out)], ref[torch.isinf(ref)])
        fine = torch.isfinite(ref)
        half_ulp = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)          # as above
        assert bool(((out - ref).abs()[fine] <= 1.01 * half_ulp * ref.abs()[fine] + 5 * 2.0 ** -14).all())
    sps_b200.check_device_status()
