"""The native call path of the Python entry points: what it owes to other Python threads and to its callers."""
import ctypes
import subprocess
import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


def _dev():
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    return torch.device("cuda:0")


@pytest.mark.parametrize("call", ["decode", "write_tokens", "step_metadata"])
def test_other_python_threads_run_during_a_launch(call, tmp_path):
    """A launch that blocks (a full queue; here a stand-in of the library's function that sleeps) must not hold the interpreter."""
    from flashinfer_mla_fp4_b200 import BatchMLADecodeCuteDSLFP4Wrapper, FP4MLADecodeBackend, FP4MLAPagedCache, _cabi, synth
    from flashinfer_mla_fp4_b200.kvcache import write_tokens

    dev = _dev()
    (tmp_path / "slow.c").write_text("#include <unistd.h>\nint slow(void) { usleep(300000); return 0; }\n")
    subprocess.run(["cc", "-shared", "-fPIC", str(tmp_path / "slow.c"), "-o", str(tmp_path / "slow.so")], check=True)
    slow = ctypes.cast(ctypes.CDLL(str(tmp_path / "slow.so")).slow, ctypes.c_void_p).value
    names = ("mla_fp4_decode", "mla_fp4_workspace_bytes", "mla_fp4_cache_write", "mla_fp4_step_metadata", "mla_fp4_last_error")
    real = [ctypes.cast(getattr(_cabi.lib, n), ctypes.c_void_p).value for n in names]

    case = synth.build_case("gil", [100], 16, 64, device=dev)
    w = BatchMLADecodeCuteDSLFP4Wrapper(torch.empty(32 << 20, dtype=torch.int8, device=dev))
    w.plan(num_heads=16, page_size=64)
    cache = FP4MLAPagedCache(2, 64, dev)
    backend = FP4MLADecodeBackend(16, 64, 2, 128, 0.1, dev)
    lat, rope = torch.zeros(3, 512, dtype=torch.bfloat16, device=dev), torch.zeros(3, 64, dtype=torch.bfloat16, device=dev)
    calls = {
        "decode": lambda: w.run(case.q, case.kv_cache, case.block_tables, case.seq_lens, case.max_seq_len, case.softmax_scale,
                                kv_cache_sf=case.kv_cache_sf),
        "write_tokens": lambda: write_tokens(lat, rope, torch.arange(3, device=dev), cache.kv_cache, cache.kv_cache_sf),
        "step_metadata": lambda: backend.prepare(torch.zeros(1, 1, dtype=torch.int32).pin_memory(), torch.ones(1, dtype=torch.int32).pin_memory()),
    }
    calls[call]()
    torch.cuda.synchronize()
    ticks, stop = [], threading.Event()

    def tick():
        while not stop.is_set():
            ticks.append(time.monotonic())
            time.sleep(0.001)

    t = threading.Thread(target=tick)
    _cabi.native.bind(slow, real[1], slow, slow, real[4])
    try:
        t.start()
        begin = time.monotonic()
        calls[call]()
        end = time.monotonic()
    finally:
        stop.set()
        t.join()
        _cabi.native.bind(*real)
    assert end - begin > 0.25  # the stand-in was called
    assert sum(begin + 0.02 < x < end - 0.02 for x in ticks) > 20


def test_prepare_from_the_backends_own_buffers():
    """Rows of the persistent buffers as sources: refused where they lie across their places (a copy would), kept where they are the same."""
    from flashinfer_mla_fp4_b200 import FP4MLADecodeBackend

    dev = _dev()
    backend = FP4MLADecodeBackend(16, 16, 5, 1024, 0.1, dev)
    tables = torch.arange(4 * backend.max_pages, dtype=torch.int32, device=dev).reshape(4, -1)
    lens = torch.tensor([700, 1, 90, 1024], dtype=torch.int32, device=dev)
    backend.prepare(tables, lens)
    slots = backend.slot_mapping.clone()
    for bt, sl in ((backend.block_tables[1:4], lens[1:]), (tables[1:], backend.seq_lens[1:4])):
        with pytest.raises(RuntimeError, match="clone"):
            backend.prepare(bt, sl)
    backend.prepare(tables, lens)
    backend.prepare(backend.block_tables[:4], backend.seq_lens[:4])
    assert torch.equal(backend.block_tables[:4], tables) and torch.equal(backend.seq_lens[:4], lens) and torch.equal(backend.slot_mapping, slots)


def test_forward_reads_the_buffers_that_the_backend_has():
    """The rows kept from one forward() to the next belong to the buffers they were cut from: replaced buffers count at once."""
    from flashinfer_mla_fp4_b200 import FP4MLADecodeBackend, FP4MLAPagedCache, synth

    dev = _dev()
    case = synth.build_case("buffers", [300, 70], 16, 64, device=dev)
    lat, rope = torch.randn(2, 512, dtype=torch.bfloat16, device=dev), torch.randn(2, 64, dtype=torch.bfloat16, device=dev)

    def outputs(lens, replace):
        cache = FP4MLAPagedCache(case.kv_cache.shape[0], 64, dev)
        cache.kv_cache.copy_(case.kv_cache)
        cache.kv_cache_sf.copy_(case.kv_cache_sf)
        backend = FP4MLADecodeBackend(16, 64, 2, 320, case.softmax_scale, dev)
        backend.prepare(case.block_tables, case.seq_lens)
        backend.forward(case.q, lat, rope, cache)
        if replace:
            backend.block_tables, backend.seq_lens, backend.slot_mapping = (t.clone() for t in (backend.block_tables, backend.seq_lens, backend.slot_mapping))
        backend.prepare(case.block_tables, lens)
        return backend.forward(case.q, lat + 1, rope, cache), cache.kv_cache, cache.kv_cache_sf

    lens = torch.tensor([200, 64], dtype=torch.int32, device=dev)
    for a, b in zip(outputs(lens, False), outputs(lens, True)):
        assert torch.equal(a, b)


def test_prepare_into_buffers_of_another_form():
    """Replaced buffers that the one-kernel form was not made for: wider types and rows with a pitch are filled, too narrow ones refused."""
    from flashinfer_mla_fp4_b200 import FP4MLADecodeBackend

    dev = _dev()
    tables = torch.arange(12, dtype=torch.int32, device=dev).reshape(3, 4)
    lens = torch.tensor([60, 1, 33], dtype=torch.int32, device=dev)
    backend = FP4MLADecodeBackend(16, 16, 4, 64, 0.1, dev)
    backend.prepare(tables, lens)
    slots = backend.slot_mapping.clone()
    backend.seq_lens = torch.full((4,), -7, dtype=torch.int64, device=dev)
    backend.block_tables = torch.zeros(4, 9, dtype=torch.int32, device=dev)[:, :4]
    backend.prepare(tables, lens)
    assert backend.seq_lens.tolist() == [60, 1, 33, 0]
    assert torch.equal(backend.block_tables[:3], tables) and torch.equal(backend.slot_mapping, slots)
    backend.seq_lens = backend.seq_lens.int()
    backend.block_tables = torch.zeros(4, 3, dtype=torch.int32, device=dev)
    with pytest.raises(RuntimeError):
        backend.prepare(tables, lens)
