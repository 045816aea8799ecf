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
