"""The running softmax references of the decode kernel when scores keep outgrowing them: token scales that climb from tile to
tile (by little, or by more than FP32 exponentials could hold), fall, or vanish, against the oracle."""
import math

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


@pytest.mark.parametrize("logit", [-90.0, -200.0, -2000.0, 200.0])
@pytest.mark.parametrize("lens,max_ctas,sink", [
    ([1], None, False),          # a tile of one token
    ([128, 257], None, True),    # a whole tile, and a first tile with two after it
    ([2000, 129], 3, False),     # first tiles of later segments of a split request
    ([2000], 3, True),
])
def test_scores_far_from_zero(logit, lens, max_ctas, sink):
    """A segment's first references lie as far from zero as its scores do.  All logits of the odd heads are moved by `logit`,
    all of the heads 2, 6, 10, ... by `logit` from token 600 on (a split request then has segments of no weight), none of the rest."""
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    from flashinfer_mla_fp4_b200 import AttentionWithSink, BatchMLADecodeCuteDSLFP4Wrapper, synth

    dev, heads = torch.device("cuda:0"), 40
    case = synth.build_case("far", lens, heads, 64, seed=len(lens), device=dev)
    # RoPE values 0..31 of every token are 8, values 32..63 are 8 from token 600 on and 0 before; the query selects one of them
    rows, tables = case.kv_cache.view(torch.float8_e4m3fn), case.block_tables.cpu()
    for b, n in enumerate(lens):
        for i in range(-(-n // 64)):
            late = torch.arange(64 * i, 64 * i + 64, device=dev) >= 600
            rows[int(tables[b, i]), :, 256:288] = torch.full((64, 32), 8.0, device=dev).to(torch.float8_e4m3fn)
            rows[int(tables[b, i]), :, 288:320] = (late.float() * 8.0).unsqueeze(1).expand(64, 32).to(torch.float8_e4m3fn)
    want = torch.tensor(logit / case.softmax_scale / (32 * 8.0), device=dev).to(torch.float8_e4m3fn)
    case.q[..., 512:] = torch.zeros((), device=dev).to(torch.float8_e4m3fn)
    case.q[:, :, 1::2, 512:544] = want
    case.q[:, :, 2::4, 544:] = want
    sinks = torch.linspace(-4.0, 4.0, heads, device=dev) + (float(want) * 32 * 8.0 * case.softmax_scale if logit < 0 else 0.0) if sink else None
    w = BatchMLADecodeCuteDSLFP4Wrapper(torch.empty(32 << 20, dtype=torch.int8, device=dev))
    w.plan(num_heads=heads, page_size=64, out_dtype=torch.float32, max_ctas=max_ctas, variant=AttentionWithSink(sinks) if sink else None)
    out, lse = w.run(case.q, case.kv_cache, case.block_tables, case.seq_lens, case.max_seq_len, case.softmax_scale,
                     kv_cache_sf=case.kv_cache_sf, return_lse=True)
    torch.cuda.synchronize()
    w.check_device_status()
    ref, ref_lse = O.mla_decode(case.q, case.kv_cache, case.kv_cache_sf, case.block_tables, case.seq_lens, case.softmax_scale, sink=sinks)
    O.assert_parity(out, ref, "far scores")
    torch.testing.assert_close(lse.cpu(), ref_lse, atol=2e-3, rtol=1e-4)


def test_heavy_tokens_keep_exact_weights():
    """Two tokens carry all the weight of every head: token 10 in the first tile, token 200 in the second, ahead of it by 0.3 to 8
    binades depending on the head.  The best token of a head has a weight of exactly 2^4 in its tile, so what is left of the error is
    that of FP32 exponents of up to a hundred (2^-24 * 100 * ln 2 = 4e-6) in a weight: 1e-4 of the output's RMS is far above it.
    With the references of the heads moved alone that the second token beats by more than the lazy threshold, the weights of the others
    are rounded to two E4M3 terms (2^-9 of a weight, a few 1e-4 of the output)."""
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    from flashinfer_mla_fp4_b200 import BatchMLADecodeCuteDSLFP4Wrapper, synth

    dev, heads, unit = torch.device("cuda:0"), 64, 1.1
    case = synth.build_case("heavy", [256], heads, 64, seed=5, device=dev)

    def e4m3(x):
        return torch.as_tensor(x, dtype=torch.float32, device=dev).to(torch.float8_e4m3fn)

    case.q[...] = e4m3(0.0)
    case.q[0, 0, :, 513] = e4m3(torch.linspace(0.3, 7.5, heads))
    case.q[0, 0, :, 514] = e4m3(-56.0)
    rows = case.kv_cache.view(torch.float8_e4m3fn)
    for i in range(4):
        page = int(case.block_tables[0, i])
        rows[page, :, 256:] = e4m3(0.0)
        rows[page, :, 258] = e4m3(8.0)
    for token, k in ((10, 256), (200, 257)):
        page = int(case.block_tables[0, token // 64])
        rows[page, token % 64, 258] = e4m3(0.0)
        rows[page, token % 64, k] = e4m3(8.0)
    scale = unit * math.log(2.0) / 8.0  # exponents of 1.1 times the query value
    w = BatchMLADecodeCuteDSLFP4Wrapper(torch.empty(32 << 20, dtype=torch.int8, device=dev))
    w.plan(num_heads=heads, page_size=64, out_dtype=torch.float32)
    out = w.run(case.q, case.kv_cache, case.block_tables, case.seq_lens, case.max_seq_len, scale, kv_cache_sf=case.kv_cache_sf)
    torch.cuda.synchronize()
    w.check_device_status()
    ref = O.mla_decode(case.q, case.kv_cache, case.kv_cache_sf, case.block_tables, case.seq_lens, scale)[0]
    assert O.parity_metrics(out, ref)["max_abs_over_rms"] <= 1e-4
