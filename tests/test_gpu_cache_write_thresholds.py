"""The CUDA cache writer where its division-free rounding can go wrong: values on and next to the rounding thresholds,
infinity, zeros of both signs, scales at the ends of the range, against the oracle's division and comparisons."""
import pytest
import torch

from oracle import mla_fp4_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("scales", ["amax", "given"])
def test_values_next_to_the_thresholds(dtype, scales):
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    from flashinfer_mla_fp4_b200.kvcache import write_tokens

    g = torch.Generator().manual_seed(17)
    T = 600
    latent = torch.randn(T, 512, generator=g) * torch.exp2(torch.randint(-6, 7, (T, 1), generator=g).float())
    given = torch.exp2(torch.randint(-5, 4, (T,), generator=g).float()) * torch.where(torch.rand(T, generator=g) < 0.5, 1.0, 1.37)
    s = given[:, None] if scales == "given" else O.amax_scale(latent.to(dtype).float())
    thr = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0])[torch.randint(0, 7, (T, 512), generator=g)]
    near = (thr * s).view(torch.int32) + torch.randint(-3, 4, (T, 512), generator=g, dtype=torch.int32)  # a few last places off
    near = near.view(torch.float32) * latent.sign()
    latent = torch.where(torch.arange(512) % 3 == 0, latent, near)
    latent[3:9, 1::2] = -0.0
    latent[10] = 0.0
    latent[11:14] *= 1e-30 if dtype != torch.float16 else 1e-5
    if scales == "given":
        latent[21, 7] = float("inf")
        given[30], given[31], given[32] = 2.0 ** -120, 2.0 ** 15, 2.0 ** 100
    latent = latent.to(dtype)
    rope = torch.randn(T, 64, generator=g).to(dtype)
    dev = torch.device("cuda:0")
    cache = torch.zeros(T, 1, 320, dtype=torch.uint8, device=dev)
    sf = torch.zeros(T, 1, 1, device=dev)
    write_tokens(latent.to(dev), rope.to(dev), None, cache, sf, token_scale=given.to(dev) if scales == "given" else None)
    want_s = given[:, None] if scales == "given" else O.amax_scale(latent.float())
    assert torch.equal(sf.cpu().view(-1), want_s.view(-1))
    assert torch.equal(cache.cpu().view(T, 320), O.pack_cache(latent.float(), rope, want_s))
