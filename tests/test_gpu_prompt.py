"""The prompt scan against the host form of the same rules, across its columns per pass."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", [1, 2, 33, 1024, 1025, 2500])
@pytest.mark.parametrize("variant", ["sps", "standard"])
def test_prompt_scan_matches_the_host_rules(t, variant):
    import sps_b200
    from oracle import sps_oracle as orc
    from sps_b200.generation import left_padded_document_idx, left_padded_position_ids, random_state_dict
    dims = sps_b200.SPSDims(block_size=16, vocab_size=40, n_layer=1, n_head=1, hidden_size=64, intermediate_size=16,
                            eos_token_id=37, pad_token_id=39, predict_token_id=38)
    engine = sps_b200.SPSGenerator(random_state_dict(dims), dims, variant=variant)
    ns = engine.n_slot
    g = torch.Generator().manual_seed(t)
    idx = torch.randint(0, 38, (5, t), generator=g)
    idx[1, : t // 2] = 39
    idx[2, : t - 1] = 39
    idx[3, -1] = 37
    idx[4, t // 3] = 37
    ext, model = engine._native()
    ids2, pos2, runs, mask, real, ends, flags = [
        x.cpu() for x in ext.engine_scan(model, idx.cuda(), 37, 39, 38, variant == "standard")]
    docs = left_padded_document_idx(idx, 37, 39)
    want = (idx != 39) & (docs == docs[:, -1:])
    if variant == "standard":
        want &= idx[:, -1:] != 37
    assert torch.equal(mask.bool(), want)
    assert torch.equal(pos2, left_padded_position_ids(idx, 39).repeat_interleave(ns, dim=1))
    assert torch.equal(ids2[:, ::ns], idx) and (ns == 1 or bool((ids2[:, 1::2] == 38).all()))
    for row in range(5):
        starts = orc.run_starts(docs[row].repeat_interleave(ns).numpy())
        assert runs[row].tolist() == [int(x) for x in starts]
    assert torch.equal(real, (idx != 39).sum(1)) and torch.equal(ends.bool(), idx[:, -1] == 37)
    assert flags.tolist() == [0, 0, int(real.max()), 0]
    bad = idx.clone()
    bad[0, -1] = 39
    bad[1] = 39
    flags = ext.engine_scan(model, bad.cuda(), 37, 39, 38, False)[6].tolist()
    assert flags[:2] == [int(t > 1), 1]


@pytest.mark.parametrize("n,parity", [(2, 0), (128, 1), (130, -1), (1152, 0), (1154, 1)])
@pytest.mark.parametrize("mode", ["packed", "every_token", "arbitrary", "decreases_late"])
def test_document_scan_inside_the_attention_equals_the_pre_pass(n, parity, mode):
    import sps_b200
    g = torch.Generator().manual_seed(n)
    q, k, v = (torch.randn(2, 2, n, 64, generator=g).bfloat16().cuda() for _ in range(3))
    ids = torch.arange(n).expand(2, n) // (50 if mode == "packed" else 2)
    ids = ids.clone()
    if mode == "arbitrary":
        ids = torch.randint(0, 3, (2, n), generator=g)
    if mode == "decreases_late":
        ids[:, -1] = 0
        ids[0, n // 2:] -= 1
    wide = torch.zeros(2, n, 3, dtype=torch.int32)
    wide[:, :, 1] = ids
    for docs in (ids.cuda(), wide.cuda()[:, :, 1]):          # int64 dense, int32 strided
        call = lambda lse: sps_b200.prefill_attention(q, k, v, 0.125, persistent_parity=parity, temporary_window=7,
                                                      documents_idx=docs, return_lse=lse)
        assert torch.equal(call(False), call(True)[0])       # with lse the pre-pass runs
