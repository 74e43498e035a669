"""The convolution cache that the prompt form of the layer's front kernel leaves: the last three projection rows of the convolved
channels, whatever part of the last token group they fill."""
import pytest
import torch

from gdn2_tilelang_b200 import _cabi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [8, 9, 10, 11, 15, 16, 17, 26, 64])
@pytest.mark.parametrize("H,HK", [(2, 1), (3, 3)])
@pytest.mark.parametrize("old", [False, True])
def test_new_cache_is_the_last_three_rows(S, H, HK, old):
    D, K, B, dtype = 128, 4, 2, torch.bfloat16
    gen = torch.Generator("cuda").manual_seed(S)
    widths = [HK * D, HK * D, H * D, HK * D, H * D, HK * D, H * D]                   # q k v b w f o_gate
    offsets = [sum(widths[:i]) for i in range(7)]
    CC = 2 * HK * D + H * D

    def rand(*shape):
        return torch.randn(*shape, device="cuda", generator=gen).to(dtype)

    proj, state = rand(B, S, sum(widths)), rand(B, CC, K - 1) if old else None
    kernels = _cabi.kernels()
    before = kernels.launches
    *_, cache = kernels.layer_front(proj, offsets[:6], state, rand(CC, K), None, rand(HK), rand(HK, D), H, HK, D, D, K, 1.0, True)
    assert kernels.launches == before + 1
    assert torch.equal(cache, proj[:, S - 3:, :CC].transpose(1, 2))
