"""A plan made before the kernel ahead on the stream has ended must not outlive a change of the lengths by that kernel."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 32, 33, 130, 20481])  # lanes of one warp, one more, four rounds, more than are kept
def test_lengths_changed_by_the_kernel_ahead(batch):
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    from flashinfer_mla_fp4_b200 import BatchMLADecodeCuteDSLFP4Wrapper, synth

    dev = torch.device("cuda:0")
    n = min(batch, 130)
    case = synth.build_case("ahead", [700] * n, 16, 64, seed=batch, device=dev)
    rep = -(-batch // n)
    q = case.q.view(torch.uint8).repeat(rep, *([1] * (case.q.dim() - 1)))[:batch].contiguous().view(case.q.dtype)
    tables = case.block_tables.repeat(rep, 1)[:batch].contiguous()
    lens = [torch.full((batch,), v, dtype=torch.int32, device=dev) for v in (700, 65)]
    lens[1][-1] = 640  # (only the last one differs from the third step's)
    lens.append(lens[1].clone())
    lens[2][-1] = 1
    w = BatchMLADecodeCuteDSLFP4Wrapper(torch.empty(128 << 20, dtype=torch.int8, device=dev))
    w.plan(num_heads=16, page_size=64)

    def run(seq_lens):
        return w.run(q, case.kv_cache, tables, seq_lens, case.max_seq_len, case.softmax_scale, kv_cache_sf=case.kv_cache_sf).clone()

    want = []
    for x in lens:
        want.append(run(x))
        torch.cuda.synchronize()
    now = lens[0].clone()
    got = []
    for x in lens:
        now.copy_(x)
        got.append(run(now))
    for k in (1, 0):  # steps back to back, without a copy of the output between them
        now.copy_(lens[k])
        w.run(q, case.kv_cache, tables, lens[2], case.max_seq_len, case.softmax_scale, kv_cache_sf=case.kv_cache_sf)
        assert torch.equal(run(now), want[k])
    torch.cuda.synchronize()
    w.check_device_status()
    for a, b in zip(got, want):
        assert torch.equal(a, b)
