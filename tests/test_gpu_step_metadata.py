"""The step-metadata kernel against the torch form of the same refresh: row widths at the edges of a thread's share, lengths at
page and table edges, given and derived slots, device and pinned host sources."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [1, 127, 128, 513, 1400])
@pytest.mark.parametrize("host", [False, True])
def test_prepare_matches_the_torch_form(width, host):
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    from flashinfer_mla_fp4_b200 import FP4MLADecodeBackend
    from flashinfer_mla_fp4_b200.adapter import decode_slot_mapping

    dev = torch.device("cuda:0")
    g = torch.Generator().manual_seed(width)
    page, q_len, batch, max_batch = 16, 3, 7, 9
    backend = FP4MLADecodeBackend(16, page, max_batch, 1400 * page, 0.1, dev, q_len=q_len)
    bt = torch.randint(0, 1 << 20, (batch, width), generator=g, dtype=torch.int32)
    lens = torch.tensor([0, 1, q_len, page, min(page + 1, width * page), width * page, max(1, width * page // 2)], dtype=torch.int32)
    want = decode_slot_mapping(bt, lens, page, q_len)
    given = torch.randint(-1, 1 << 40, (batch * q_len,), generator=g)
    for dtype, slots in ((torch.int32, None), (torch.int64, given)):
        backend.block_tables.fill_(-5)
        src = [t.pin_memory() if host else t.to(dev) for t in (bt, lens.to(dtype))]
        assert backend.prepare(*src, slots if slots is None else (slots.pin_memory() if host else slots.to(dev))) == batch
        torch.cuda.synchronize()
        assert torch.equal(backend.block_tables[:batch, :width].cpu(), bt)
        assert (backend.block_tables[:, width:] == -5).all() and (backend.block_tables[batch:] == -5).all()
        assert backend.seq_lens.tolist() == lens.tolist() + [0] * (max_batch - batch)
        got = backend.slot_mapping.cpu()
        assert torch.equal(got[: batch * q_len], want if slots is None else slots) and (got[batch * q_len:] == -1).all()
