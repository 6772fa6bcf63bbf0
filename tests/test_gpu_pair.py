"""The decode kernel for an even number of head groups (two CTAs, two groups of the same tiles) where it can go wrong: edges of tiles,
half tiles and pages, many requests in one pair's walk, heads that fill no group, every output type and variant, both merge
forms, references that move, a wait that runs out, steps under capture and on two streams.  Against the oracle, and against the other
kernel (the two-kernel mode uses it).  The calls ask for this kernel (phase mask 8), whatever the rule between the two says of them."""
import pytest
import torch

from oracle import mla_fp4_oracle as O

pytestmark = pytest.mark.gpu
PAIRS = 8


def takes_pairs(w, q_len):
    """Whether a call of this wrapper can take the kernel under test: an even number of groups, and a grid that they nearly fill evenly."""
    groups = q_len * -(-w._num_heads // 64)
    assert groups % 2 == 0 and 8 * (w._num_ctas // groups * groups) >= 7 * w._num_ctas


def _run(lens, heads, page, q_len, max_ctas=None, out_dtype=None, variant=None, sharp=1.0, latent="normal", forms=(0, 4), **ref_kw):
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    from flashinfer_mla_fp4_b200 import BatchMLADecodeCuteDSLFP4Wrapper, _cabi, synth

    dev = torch.device("cuda:0")
    case = synth.build_case("pair", [max(n, 1) for n in lens], heads, page, q_len=q_len, seed=sum(lens) + heads, device=dev, latent_dist=latent)
    case.seq_lens = torch.tensor(lens, dtype=torch.int32, device=dev)
    w = BatchMLADecodeCuteDSLFP4Wrapper(torch.empty(32 << 20, dtype=torch.int8, device=dev))
    w.plan(num_heads=heads, page_size=page, max_ctas=max_ctas, out_dtype=out_dtype, variant=variant)
    scale, got = case.softmax_scale * sharp, []
    takes_pairs(w, q_len)
    for kernel, mask in [(_cabi.KERNEL_TCGEN05, PAIRS | f) for f in forms] + [(_cabi.KERNEL_TCGEN05_2PASS, 0)]:
        w._kernel, w._phase_mask = kernel, mask
        got.append(w.run(case.q, case.kv_cache, case.block_tables, case.seq_lens, case.max_seq_len, scale, kv_cache_sf=case.kv_cache_sf, return_lse=True))
        torch.cuda.synchronize()
        w.check_device_status()
    ref, ref_lse = O.mla_decode(case.q, case.kv_cache, case.kv_cache_sf, case.block_tables, case.seq_lens, scale, **ref_kw)
    return got, ref, ref_lse


@pytest.mark.parametrize("lens,heads,page,q_len,max_ctas", [
    ([1, 63, 64, 65, 127, 128, 129, 0, 512], 128, 64, 1, 2),   # half tiles with and without tokens
    ([1, 63, 64, 65, 127, 128, 129, 1025], 65, 128, 1, 2),            # one pair walks them all; pages copied by halves; one head in a group
    ([57, 120, 513, 1025], 100, 8, 2, 4),
    ([130] * 37 + [900], 128, 16, 1, 2),                          # more requests than a round holds
    ([640, 2304, 5000], 40, 32, 2, 8),                            # partials at both ends of a walk
    ([30000, 500, 9000], 128, 64, 3, None),                             # six groups: 144 of the 148 CTAs
    ([50000], 128, 64, 1, 36),
    ([300, 400, 500, 512, 100, 200, 300, 64, 65], 128, 64, 1, 36), # short requests, whole
])
@pytest.mark.parametrize("latent,sharp", [("normal", 1.0), ("student_t3", 8.0)])
def test_pairs_of_groups(lens, heads, page, q_len, max_ctas, latent, sharp):
    got, ref, ref_lse = _run(lens, heads, page, q_len, max_ctas, torch.float32, sharp=sharp, latent=latent)
    live = torch.isfinite(ref_lse)
    for out, lse in got:
        O.assert_parity(out, ref, "pairs")
        torch.testing.assert_close(lse.cpu()[live], ref_lse[live], atol=2e-3, rtol=1e-4)
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])  # both merge forms
    # P' has about eight bits on either side: the parity bar against the oracle, twice
    diff = (got[0][0] - got[2][0]).float().cpu()
    assert float(diff.abs().max()) <= 2 * O.MAXABS_OVER_RMS_BAR * float(ref.float().pow(2).mean(-1).sqrt().max())


@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32, torch.float8_e4m3fn])
@pytest.mark.parametrize("lens,max_ctas", [([90, 300], None), ([5000, 700], 16)])
def test_pairs_output_types_and_variants(out_dtype, lens, max_ctas):
    from flashinfer_mla_fp4_b200 import SoftCappingAttention

    sink = torch.linspace(-3.0, 3.0, 96)
    got, ref, ref_lse = _run(lens, 96, 64, 2, max_ctas, out_dtype, SoftCappingAttention(25.0, sink.cuda()), forms=(0,), sink=sink, logits_soft_cap=25.0)
    if out_dtype == torch.float8_e4m3fn:  # half a unit in the last place of E4M3 (2^-4 of the value, 2^-10 below its normal range) beside P'
        err = (got[0][0].float().cpu() - ref.float()).abs()
        assert bool((err <= ref.float().abs() * 0.0625 + 2.0 ** -10 + 2e-2 * ref.float().pow(2).mean(-1, keepdim=True).sqrt()).all())
    else:
        O.assert_parity(got[0][0], ref, "pairs, variants")
    torch.testing.assert_close(got[0][1].cpu(), ref_lse, atol=2e-3, rtol=1e-4)


def test_a_pair_that_gave_up_leaves_the_workspace_consistent():
    """A page id outside the pool: the copy is never issued (for CTA 0's or CTA 1's half of a tile), CTA 0's bounded wait runs out and takes
    the partner along; the next step on the same workspace is right."""
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    from flashinfer_mla_fp4_b200 import BatchMLADecodeCuteDSLFP4Wrapper, _cabi, synth

    dev = torch.device("cuda:0")
    case = synth.build_case("gave up", [3000, 5000], 128, 64, seed=21, device=dev)
    w = BatchMLADecodeCuteDSLFP4Wrapper(torch.empty(32 << 20, dtype=torch.int8, device=dev))
    w.plan(num_heads=128, page_size=64, max_ctas=8)
    w._phase_mask = PAIRS

    def step(tables):
        out = w.run(case.q, case.kv_cache, tables, case.seq_lens, case.max_seq_len, case.softmax_scale, kv_cache_sf=case.kv_cache_sf)
        torch.cuda.synchronize()
        return out

    good = step(case.block_tables)
    w.check_device_status()
    for page in (40, 41):
        bad = case.block_tables.clone()
        bad[1, page] = case.kv_cache.shape[0] + 5
        w._wait_polls = 2000
        step(bad)
        assert w.device_status()[0] == _cabi.ERR_DEVICE_TIMEOUT
        w._wait_polls = 0
        w._status.zero_()
        assert torch.equal(step(case.block_tables), good)
        assert w.device_status()[0] == 0


def test_a_small_poll_budget_is_a_budget_of_tiles():
    """CTA 1's QK^T warp has nothing to issue and waits for a whole segment at a time: a long correct step runs to its end with a budget
    that covers a tile."""
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    from flashinfer_mla_fp4_b200 import BatchMLADecodeCuteDSLFP4Wrapper, synth

    dev = torch.device("cuda:0")
    case = synth.build_case("polls", [200000, 200], 128, 64, seed=3, device=dev)  # one pair of CTAs: 1563 tiles, then two
    w = BatchMLADecodeCuteDSLFP4Wrapper(torch.empty(32 << 20, dtype=torch.int8, device=dev))
    w.plan(num_heads=128, page_size=64, max_ctas=2)
    w._phase_mask = PAIRS

    def step():
        out = w.run(case.q, case.kv_cache, case.block_tables, case.seq_lens, case.max_seq_len, case.softmax_scale, kv_cache_sf=case.kv_cache_sf)
        torch.cuda.synchronize()
        return out

    expect = step()
    w.check_device_status()
    w._wait_polls = 32
    got, status = step(), w.device_status()
    assert status[0] == 0, status
    assert torch.equal(got, expect)


def _pair_case(lens, heads, q_len, max_ctas, seed):
    from flashinfer_mla_fp4_b200 import BatchMLADecodeCuteDSLFP4Wrapper, synth

    dev = torch.device("cuda:0")
    case = synth.build_case("pair", lens, heads, 64, q_len=q_len, seed=seed, device=dev)
    w = BatchMLADecodeCuteDSLFP4Wrapper(torch.empty(32 << 20, dtype=torch.int8, device=dev))
    w.plan(num_heads=heads, page_size=64, max_ctas=max_ctas)
    takes_pairs(w, q_len)
    w._phase_mask = PAIRS
    return w, lambda seq_lens, out=None: w.run(case.q, case.kv_cache, case.block_tables, seq_lens, case.max_seq_len, case.softmax_scale, out=out,
                                               kv_cache_sf=case.kv_cache_sf), case


@pytest.mark.parametrize("batch", [1, 32, 33, 130])  # lanes of one warp, one more, several rounds of segments
def test_pairs_and_lengths_changed_by_the_kernel_ahead(batch):
    """Each CTA of a pair makes its own plan, before the kernel ahead has ended: both must see the lengths that it leaves."""
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    w, run, case = _pair_case([700] * batch, 128, 1, None, batch)
    lens = [torch.full((batch,), v, dtype=torch.int32, device="cuda:0") for v in (700, 65)]
    lens[1][-1] = 640  # (only the last one differs from the third step's)
    lens.append(lens[1].clone())
    lens[2][-1] = 1
    want = []
    for x in lens:
        want.append(run(x))
        torch.cuda.synchronize()
    now = lens[0].clone()
    for k in (0, 1, 2, 1, 0):  # steps back to back
        now.copy_(lens[k])
        run(lens[2])
        assert torch.equal(run(now), want[k])
    w.check_device_status()


def test_pairs_in_a_graph_and_on_two_streams():
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    both = [_pair_case([9000, 700, 3000], 128, 2, None, 4), _pair_case([300] * 40, 100, 1, None, 5)]
    want, graphs, streams = [], [], [torch.cuda.Stream() for _ in both]
    for w, run, case in both:
        shorter = case.seq_lens - 200
        want.append((run(case.seq_lens), run(shorter), shorter))
        now, out = case.seq_lens.clone(), torch.empty_like(want[-1][0])
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            run(now, out)
        graphs.append((graph, now, out))
    torch.cuda.synchronize()
    for lens in (0, 1, 0):  # one graph, other lengths
        for (graph, now, out), (a, b, shorter), (w, run, case) in zip(graphs, want, both):
            now.copy_(shorter if lens else case.seq_lens)
            graph.replay()
            assert torch.equal(out, b if lens else a)
    torch.cuda.synchronize()
    got = [[], []]
    for _ in range(20):  # steps of two workspaces side by side
        for i, (w, run, case) in enumerate(both):
            with torch.cuda.stream(streams[i]):
                got[i].append(run(case.seq_lens))
    torch.cuda.synchronize()
    for i, (w, run, case) in enumerate(both):
        w.check_device_status()
        assert all(torch.equal(x, want[i][0]) for x in got[i])


def test_a_backend_chooses_by_the_lengths_it_is_told():
    """A backend sized for a model's limit: the kernel of a step is chosen by the tables that prepare() was given, that of a graph by the
    length that capture() was told."""
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    from flashinfer_mla_fp4_b200 import FP4MLADecodeBackend, FP4MLAPagedCache, planner, synth

    dev, lens, limit = torch.device("cuda:0"), [4000, 200, 1500, 2000], 131072
    case = synth.build_case("backend", lens, 128, 64, seed=8, device=dev)
    backend = FP4MLADecodeBackend(128, 64, len(lens), limit, case.softmax_scale, dev)
    cache = FP4MLAPagedCache(case.kv_cache.shape[0], 64, dev)
    cache.kv_cache.copy_(case.kv_cache)
    cache.kv_cache_sf.copy_(case.kv_cache_sf)
    told, run = [], backend.wrapper.run
    backend.wrapper.run = lambda *a, **k: told.append(a[4]) or run(*a, **k)
    lat, rope = torch.randn(4, 512, device=dev), torch.randn(4, 64, device=dev)

    def eager():
        backend.prepare(case.block_tables, case.seq_lens)
        return backend.forward(case.q, lat, rope, cache).clone()

    def replayed(step):
        backend.prepare(case.block_tables, case.seq_lens)
        step.q.copy_(case.q), step.latent.copy_(lat), step.rope.copy_(rope)
        return step.replay().clone()

    width = case.block_tables.shape[1] * 64
    first = eager()
    assert told == [width] and planner.decode_plan(lens, 1, 128, 64, limit // 64, 148, width).groups_per_cluster == 1
    short = backend.capture(cache, in_dtype=torch.float32, expected_seq_len=4000)
    assert set(told[1:]) == {4000}
    del told[:]
    full = backend.capture(cache, in_dtype=torch.float32)
    assert set(told) == {limit} and planner.decode_plan(lens, 1, 128, 64, limit // 64, 148, limit).groups_per_cluster == 2
    assert torch.equal(replayed(short), first) and torch.equal(eager(), first)
    O.assert_parity(replayed(full), first.float().cpu(), "the other kernel")
    del told[:]
    graph = torch.cuda.CUDAGraph()  # a caller's own capture: for any later step, not for the one prepared last
    with torch.cuda.graph(graph):
        backend.forward(case.q, lat, rope, cache)
    assert told == [limit]
    with pytest.raises(ValueError, match="expected_seq_len"):
        backend.capture(cache, expected_seq_len=limit + 1)
    backend.wrapper.check_device_status()
