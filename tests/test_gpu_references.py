"""The running softmax references of the decode kernel when scores keep outgrowing them: token scales that climb from tile to
tile (by little, or by more than FP32 exponentials could hold), fall, or vanish, against the oracle."""
import pytest
import torch

from oracle import mla_fp4_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("step", [0.4, 0.7, -1.0])
@pytest.mark.parametrize("heads,lens,max_ctas", [(64, [1500, 129], 1), (40, [2000], 3)])
def test_scores_that_outgrow_their_references(step, heads, lens, max_ctas):
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    from flashinfer_mla_fp4_b200 import BatchMLADecodeCuteDSLFP4Wrapper, synth

    dev = torch.device("cuda:0")
    case = synth.build_case("references", lens, heads, 64, seed=heads, device=dev)
    for b, n in enumerate(lens):  # page i of a request: scales times 2^(step * i); one page of vanishing scales
        for i in range(-(-n // 64)):
            page = int(case.block_tables[b, i])
            case.kv_cache_sf[page] *= 2.0 ** (step * i / 2) if i != 5 else 2.0 ** -90
    w = BatchMLADecodeCuteDSLFP4Wrapper(torch.empty(32 << 20, dtype=torch.int8, device=dev))
    w.plan(num_heads=heads, page_size=64, out_dtype=torch.float32, max_ctas=max_ctas)
    out, lse = w.run(case.q, case.kv_cache, case.block_tables, case.seq_lens, case.max_seq_len, case.softmax_scale,
                     kv_cache_sf=case.kv_cache_sf, return_lse=True)
    torch.cuda.synchronize()
    w.check_device_status()
    ref, ref_lse = O.mla_decode(case.q, case.kv_cache, case.kv_cache_sf, case.block_tables, case.seq_lens, case.softmax_scale)
    O.assert_parity(out, ref, "references")
    torch.testing.assert_close(lse.cpu(), ref_lse, atol=2e-3, rtol=1e-4)
