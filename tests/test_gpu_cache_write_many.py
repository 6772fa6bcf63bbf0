"""The cache writer's form for many 16-bit tokens (four to a warp) against its form for few, which the other tests hold against the
oracle: the same tokens written in one call and in pieces must give the same bytes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
MANY = {False: 24576, True: 65536}  # from here on in one call: the form under test (scales given or not)


def tokens_per_warp(dtype, n, given):
    import ctypes as C

    from flashinfer_mla_fp4_b200 import _cabi

    out = C.c_int32(0)
    _cabi.check(_cabi.lib.mla_fp4_cache_write_plan({torch.bfloat16: _cabi.IN_BF16, torch.float16: _cabi.IN_F16}[dtype], n, int(given), C.byref(out)))
    return out.value


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("extra", [0, 1, 6])
@pytest.mark.parametrize("form", ["plain", "strided", "given", "nans", "padding"])
def test_many_tokens_as_in_pieces(dtype, extra, form):
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    from flashinfer_mla_fp4_b200.kvcache import write_tokens

    dev, n, page = torch.device("cuda:0"), MANY[form == "given"] + extra, 16
    assert [tokens_per_warp(dtype, k, form == "given") for k in (n, MANY[form == "given"] - 1, 5000)] == [4, 1, 1]
    g = torch.Generator(device=dev).manual_seed(extra + 5)

    def rnd(*shape):
        return torch.randn(*shape, generator=g, device=dev)

    amax = (torch.rand(n, 1, generator=g, device=dev) * 3 + 0.1).to(dtype).float()
    thr = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0, 6.0], device=dev)[torch.randint(0, 8, (n, 512), generator=g, device=dev)]
    latent = torch.where(rnd(n, 512) > 0, rnd(n, 512).clamp(-1, 1) * amax, thr * amax / 6 * rnd(n, 512).sign())  # half on the thresholds
    latent[::7] *= 2.0 ** -10
    latent[11], latent[n - 1, 3] = 0.0, -0.0
    latent[17, 100], latent[18, 0], latent[23] = float("nan"), float("inf"), 1e-30  # (the last is zero in FP16)
    if form == "nans":  # one to four tokens of a warp; runs of them
        latent[rnd(n) > 0.5, 7] = float("nan")
        latent[1000:1064, 500] = float("nan")
    rope = rnd(n, 64) * 200
    stride = 520 if form == "strided" else 512
    lat = torch.empty(n, stride, dtype=dtype, device=dev)[:, :512].copy_(latent)
    rp = torch.empty(n, 66, dtype=dtype, device=dev)[:, 2:].copy_(rope) if form == "strided" else rope.to(dtype)
    scale = torch.exp2(torch.randint(-9, 3, (n,), generator=g, device=dev).float()) * 1.37 if form == "given" else None
    if scale is not None:
        scale[40], scale[41] = 2.0 ** -120, 2.0 ** 15
    pages = n // page + 40
    slots = torch.randperm(pages * page, generator=g, device=dev)[:n]
    slots[5], slots[n - 2], slots[300] = -1, pages * page, -7  # padding and out of the pool: nothing is written
    if form == "padding":  # whole warps and parts of them
        slots[rnd(n) > 0], slots[2000:3001] = -1, -1

    def written(step):
        cache = torch.full((pages, page, 320), 0xAB, dtype=torch.uint8, device=dev)
        sf = torch.full((pages, page, 1), -7.0, device=dev)
        for a in range(0, n, step):
            z = slice(a, a + step)
            write_tokens(lat[z], rp[z], slots[z], cache, sf, token_scale=None if scale is None else scale[z])
        return cache, sf.view(torch.int32)

    one, pieces = written(n), written(5000)
    assert torch.equal(one[0], pieces[0]) and torch.equal(one[1], pieces[1])
