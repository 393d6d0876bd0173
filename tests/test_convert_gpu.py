"""cfk_convert against torch's casts of the scaled fp32 values: whole vectors, remainders of every length, and addresses
that are aligned to the element only.  The conversion rounds once, to nearest even, so the bits must be equal."""
import pytest
import torch

pytestmark = pytest.mark.gpu

TORCH_DT = [torch.float16, torch.bfloat16, torch.float8_e4m3fn, torch.float32]
BITS = {1: torch.uint8, 2: torch.int16, 4: torch.int32}


@pytest.mark.parametrize("src", range(4))
@pytest.mark.parametrize("dst", range(4))
def test_convert_matches_the_casts_bit_for_bit(lib, cuda, src, dst):
    g = torch.Generator().manual_seed(10 * src + dst)
    for n, off_s, off_d in [(1, 0, 0), (3, 0, 0), (15, 0, 0), (16, 0, 0), (17, 0, 0), (2048, 0, 0), (2047 + 8192, 0, 0),
                            (4099, 1, 0), (4099, 0, 1), (5000, 3, 5), (5000, 16, 16), (300007, 0, 0),
                            (2047, 1, 0), (2048, 0, 1), (2049, 1, 1), (300007, 1, 3)]:
        x = torch.randn(n + off_s, generator=g) * 100
        for i, special in enumerate((0.0, -0.0, float("inf"), float("-inf"), float("nan"), 1e-7, 447.0, 1e6)):
            if n > 20:
                x[off_s + 11 * i % n] = special
        if TORCH_DT[src] == torch.float8_e4m3fn:       # torch's cast to e4m3 does not saturate
            x = x.clamp(-448, 448)
        x = x.to(TORCH_DT[src]).cuda()
        y = torch.zeros(n + off_d + 16, dtype=torch.float32, device="cuda").to(TORCH_DT[dst])
        lib.convert(x.data_ptr() + off_s * x.element_size(), src, y.data_ptr() + off_d * y.element_size(), dst, n, scale=0.75)
        torch.cuda.synchronize()
        f = x[off_s:].float() * 0.75
        want = (f.clamp(-448, 448) if dst == 2 else f).to(TORCH_DT[dst])
        got = y[off_d:off_d + n]
        bits = BITS[y.element_size()]
        nan = torch.isnan(f)
        same = got.view(bits)[~nan] == want.view(bits)[~nan]
        assert bool(same.all()), (n, off_s, off_d)
        assert bool(torch.isnan(got.float()[nan]).all()), (n, off_s, off_d)
        pad = torch.cat([y[:off_d].view(bits), y[off_d + n:].view(bits)])
        assert bool((pad == 0).all()), (n, off_s, off_d)       # nothing beyond the array was written
