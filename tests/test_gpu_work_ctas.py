"""The number of CTAs that share a step's work: on both sides of the rule's edges, against the oracle."""
import pytest
import torch

from oracle import mla_fp4_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens,heads,max_ctas", [
    ([513], 64, None),            # five tiles: the smallest request that is split, one CTA per tile
    ([1280, 1152], 64, 5),        # 25 tiles with the phantom ones on 5 CTAs: still by the rule
    ([1280, 1281], 64, 5),        # 27: the whole grid
    ([3000], 64, 1),              # a grid of one
    ([130, 0, 5000, 1, 700], 64, None),   # the walk that shares best is two tiles long; requests without work
    ([16000], 16, None),          # many more CTAs than the rule wants
    ([2500] * 30, 128, 7),        # partials at both ends of most CTAs
    ([130] * 131 + [700], 16, 2), # rounds of many segments: the partial in the first, none in the last, and the other way about
    ([700] + [130] * 131, 16, 2),
])
def test_any_number_of_working_ctas(lens, heads, max_ctas):
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    from flashinfer_mla_fp4_b200 import BatchMLADecodeCuteDSLFP4Wrapper, synth

    dev = torch.device("cuda:0")
    case = synth.build_case("ctas", [max(n, 1) for n in lens], heads, 64, seed=sum(lens), device=dev)
    case.seq_lens = torch.tensor(lens, dtype=torch.int32, device=dev)
    w = BatchMLADecodeCuteDSLFP4Wrapper(torch.empty(32 << 20, dtype=torch.int8, device=dev))
    w.plan(num_heads=heads, page_size=64, max_ctas=max_ctas)
    out, lse = w.run(case.q, case.kv_cache, case.block_tables, case.seq_lens, case.max_seq_len, case.softmax_scale,
                     kv_cache_sf=case.kv_cache_sf, return_lse=True)
    w.check_device_status()
    ref, ref_lse = O.mla_decode(case.q, case.kv_cache, case.kv_cache_sf, case.block_tables, case.seq_lens, case.softmax_scale)
    O.assert_parity(out, ref, "working CTAs")
    live = torch.isfinite(ref_lse)
    torch.testing.assert_close(lse.cpu()[live], ref_lse[live], atol=2e-3, rtol=1e-4)


@pytest.mark.parametrize("lens,heads,q_len,max_ctas", [
    ([513], 64, 1, None), ([16000], 64, 1, None), ([16000] + [0] * 32, 64, 1, None), ([4096] * 4, 64, 1, None), ([3000, 1500], 128, 2, None),
    ([130, 0, 5000, 1, 700], 40, 1, 31), ([2500] * 30, 128, 1, 7), ([512] * 6, 64, 1, None), ([60000], 8, 1, 100), ([9000, 100], 16, 3, 148),
    ([1280, 1152], 64, 1, 5), ([1280, 1281], 64, 1, 5),
])
def test_the_planner_describes_the_kernels_partition(lens, heads, q_len, max_ctas):
    """The partial slots that a step publishes are those of the host's partition over the host's number of working CTAs."""
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    from flashinfer_mla_fp4_b200 import BatchMLADecodeCuteDSLFP4Wrapper, _cabi, planner, synth

    dev = torch.device("cuda:0")
    case = synth.build_case("slots", [max(n, 1) for n in lens], heads, 64, q_len=q_len, seed=1, device=dev)
    case.seq_lens = torch.tensor(lens, dtype=torch.int32, device=dev)
    ws = torch.empty(32 << 20, dtype=torch.int8, device=dev)
    w = BatchMLADecodeCuteDSLFP4Wrapper(ws)
    w.plan(num_heads=heads, page_size=64, max_ctas=max_ctas)  # (zeroes the slots' flags)
    w.run(case.q, case.kv_cache, case.block_tables, case.seq_lens, case.max_seq_len, case.softmax_scale, kv_cache_sf=case.kv_cache_sf)
    w.check_device_status()
    head = _cabi.WORKSPACE_HEADER_BYTES
    published = ws[head: head + 296 * 272].view(torch.int32).reshape(296, 68)[:, 65].nonzero().flatten().tolist()
    n = planner.work_ctas(lens, q_len, heads, w._num_ctas)
    assert published == sorted(s.slot for s in planner.plan_partition(lens, q_len, heads, n) if s.slot >= 0)


@pytest.mark.parametrize("lens,heads,q_len,max_ctas,pair,grid", [
    ([2000] * 4, 128, 5, None, 1, 148),      # ten groups do not fill 148 CTAs evenly: the kernel with a group per CTA has them all
    ([1500, 700], 128, 3, None, 1, 144),     # six nearly do
    ([3000, 1500], 128, 2, None, 1, 148),
    ([9000] * 20, 128, 5, None, 2, 140),     # a pair of groups per cluster, on as many CTAs as ten groups share evenly
    ([30000, 500, 9000], 128, 3, None, 2, 144),
    ([5000, 700, 0, 1], 40, 2, 12, 2, 12),
])
def test_the_decode_plan_describes_the_step(lens, heads, q_len, max_ctas, pair, grid):
    """Which kernel, which grid, and the partial slots that the step publishes."""
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    from flashinfer_mla_fp4_b200 import BatchMLADecodeCuteDSLFP4Wrapper, _cabi, planner, synth

    dev = torch.device("cuda:0")
    case = synth.build_case("plan", [max(n, 1) for n in lens], heads, 64, q_len=q_len, seed=2, device=dev)
    case.seq_lens = torch.tensor(lens, dtype=torch.int32, device=dev)
    ws = torch.empty(32 << 20, dtype=torch.int8, device=dev)
    w = BatchMLADecodeCuteDSLFP4Wrapper(ws)
    w.plan(num_heads=heads, page_size=64, max_ctas=max_ctas)
    plan = planner.decode_plan(lens, q_len, heads, 64, case.block_tables.shape[1], w._num_ctas)
    assert (plan.groups_per_cluster, plan.grid) == (pair, grid)
    w.run(case.q, case.kv_cache, case.block_tables, case.seq_lens, case.max_seq_len, case.softmax_scale, kv_cache_sf=case.kv_cache_sf)
    w.check_device_status()
    head = _cabi.WORKSPACE_HEADER_BYTES
    published = ws[head: head + 296 * 272].view(torch.int32).reshape(296, 68)[:, 65].nonzero().flatten().tolist()
    assert published == sorted(s.slot for s in planner.plan_partition(lens, q_len, heads, plan.work_ctas) if s.slot >= 0)
