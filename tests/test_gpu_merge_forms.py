"""The two forms in which the decode kernel merges split requests (shared by their CTAs, or by the last writer alone): both
against the oracle, and reproducible to the bit, whatever the number of partials and of units per merging CTA."""
import pytest
import torch

from oracle import mla_fp4_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens,heads,page_size,max_ctas", [
    ([1300], 64, 64, 2),            # two writers, one of them merges whole slots
    ([700, 129, 64, 2500], 40, 64, None),   # fewer tiles than CTAs: the writers are not consecutive CTAs
    ([9000, 1, 0, 600], 128, 32, None),     # two head groups, a request cut at both of a CTA's ends
    ([33000], 64, 128, None),       # every CTA a writer: several threads per unit of the merge
    ([5000] * 9, 16, 16, 31),       # partials at both ends of most CTAs
])
def test_both_merge_forms(lens, heads, page_size, max_ctas):
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    from flashinfer_mla_fp4_b200 import BatchMLADecodeCuteDSLFP4Wrapper, synth

    dev = torch.device("cuda:0")
    case = synth.build_case("merge", [max(n, 1) for n in lens], heads, page_size, seed=sum(lens), device=dev)
    case.seq_lens = torch.tensor(lens, dtype=torch.int32, device=dev)
    w = BatchMLADecodeCuteDSLFP4Wrapper(torch.empty(32 << 20, dtype=torch.int8, device=dev))
    w.plan(num_heads=heads, page_size=page_size, max_ctas=max_ctas)
    got = []
    for mask in (0, 4, 4, 0):  # twice in a row: the arrival counters are back to zero after a step
        w._phase_mask = mask
        got.append(w.run(case.q, case.kv_cache, case.block_tables, case.seq_lens, case.max_seq_len, case.softmax_scale,
                         kv_cache_sf=case.kv_cache_sf, return_lse=True))
        torch.cuda.synchronize()
        w.check_device_status()
    ref, ref_lse = O.mla_decode(case.q, case.kv_cache, case.kv_cache_sf, case.block_tables, case.seq_lens, case.softmax_scale)
    live = torch.isfinite(ref_lse)
    for out, lse in got:
        O.assert_parity(out, ref, "merge forms")
        torch.testing.assert_close(lse.cpu()[live], ref_lse[live], atol=2e-3, rtol=1e-4)
    for i, j in ((0, 3), (1, 2)):
        assert torch.equal(got[i][0], got[j][0]) and torch.equal(got[i][1], got[j][1])


@pytest.mark.parametrize("lens,heads", [
    ([16384], 64),       # 43 partials: several threads per unit, a different number of them in shares of 42 and of 43
    ([4500], 64),        # 22 or so
    ([115000], 40),      # every CTA
    ([2500, 6000, 900], 64),
])
def test_both_merge_forms_agree_to_the_bit(lens, heads):
    """Which form runs depends on what else holds the GPU at that moment: the result must not."""
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    from flashinfer_mla_fp4_b200 import BatchMLADecodeCuteDSLFP4Wrapper, synth

    dev = torch.device("cuda:0")
    case = synth.build_case("forms", lens, heads, 64, seed=lens[0], device=dev)
    w = BatchMLADecodeCuteDSLFP4Wrapper(torch.empty(32 << 20, dtype=torch.int8, device=dev))
    w.plan(num_heads=heads, page_size=64, out_dtype=torch.float32)
    got = []
    for mask in (0, 4):
        w._phase_mask = mask
        got.append(w.run(case.q, case.kv_cache, case.block_tables, case.seq_lens, case.max_seq_len, case.softmax_scale,
                         kv_cache_sf=case.kv_cache_sf, return_lse=True))
        torch.cuda.synchronize()
        w.check_device_status()
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


def test_a_step_that_gave_up_leaves_the_last_writer_form_consistent():
    """One block-table entry of a split request names a page outside the pool (the copy is never issued and a bounded wait runs out).
    The CTA that gives up counts itself into its requests all the same, so every arrival counter is back to zero: the next step on
    the same workspace, which nothing has initialised since, must not merge before the last partial is there."""
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    from flashinfer_mla_fp4_b200 import BatchMLADecodeCuteDSLFP4Wrapper, _cabi, synth

    dev = torch.device("cuda:0")
    case = synth.build_case("gave up", [3000, 5000], 64, 64, seed=21, device=dev)
    ws = torch.empty(32 << 20, dtype=torch.int8, device=dev)
    w = BatchMLADecodeCuteDSLFP4Wrapper(ws)
    w.plan(num_heads=64, page_size=64)
    w._phase_mask = 4
    head = _cabi.WORKSPACE_HEADER_BYTES
    tails = ws[head: head + 296 * 272].view(torch.int32).reshape(296, 68)  # 64 LSEs, scale, flag, arrival counter, flag of the LSEs

    def step(q, tables):
        out = w.run(q, case.kv_cache, tables, case.seq_lens, case.max_seq_len, case.softmax_scale, kv_cache_sf=case.kv_cache_sf)
        torch.cuda.synchronize()
        return out

    other = case.q.flip(2).contiguous()  # (the slots hold the partials of the step before: the queries have to differ)
    good = [step(q, case.block_tables) for q in (case.q, other)]
    w.check_device_status()
    bad = case.block_tables.clone()
    bad[1, 40] = case.kv_cache.shape[0] + 5
    w._wait_polls = 2000
    step(case.q, bad)
    assert w.device_status()[0] == _cabi.ERR_DEVICE_TIMEOUT
    assert int(tails[:, 66].abs().max()) == 0
    w._wait_polls = 0
    w._status.zero_()
    for q, want in ((case.q, good[0]), (other, good[1]), (case.q, good[0])):
        assert torch.equal(step(q, case.block_tables), want)
    assert w.device_status()[0] == 0
