"""BF16 rows written straight from the accumulator, for head counts on both sides of the writer's forms, against the oracle."""
import pytest
import torch

from oracle import mla_fp4_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads", [1, 17, 32, 33, 96])
def test_rows_of_whole_requests(heads):
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    from flashinfer_mla_fp4_b200 import BatchMLADecodeCuteDSLFP4Wrapper, synth

    dev = torch.device("cuda:0")
    case = synth.build_case("rows", [300, 1, 512], heads, 64, q_len=2, seed=heads, device=dev)
    w = BatchMLADecodeCuteDSLFP4Wrapper(torch.empty(32 << 20, dtype=torch.int8, device=dev))
    w.plan(num_heads=heads, page_size=64)
    out = torch.full((3, 2, heads, 512), float("nan"), dtype=torch.bfloat16, device=dev)
    lse = w.run(case.q, case.kv_cache, case.block_tables, case.seq_lens, case.max_seq_len, case.softmax_scale,
                kv_cache_sf=case.kv_cache_sf, out=out, return_lse=True)[1]
    w.check_device_status()
    ref, ref_lse = O.mla_decode(case.q, case.kv_cache, case.kv_cache_sf, case.block_tables, case.seq_lens, case.softmax_scale)
    O.assert_parity(out, ref, "rows")
    torch.testing.assert_close(lse.cpu(), ref_lse, atol=2e-3, rtol=1e-4)
