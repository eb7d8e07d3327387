"""Packing of 16-bit values, whose quotients are not divided out: the bytes are those of an IEEE division, ties included."""

import numpy as np
import pytest
import torch

import sageattention_b200.nvfp4 as nv
from oracle import nvfp4_oracle as O

pytestmark = pytest.mark.gpu


def _check(x):
    """x [groups, 16] on the GPU: packed bytes against the oracle's."""
    nib, sc = nv._quant_nvfp4(x[None])
    onib, osc = O.pack(x[None].float().cpu().numpy())
    assert np.array_equal(sc.view(torch.uint8).cpu().numpy(), osc)
    assert np.array_equal(nib.cpu().numpy(), onib)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_every_value_under_every_scale(dtype):
    bits = torch.arange(65536, dtype=torch.int32, device="cuda").to(torch.int16)
    every = bits.view(dtype)
    for first in range(1, 127, 21):
        rows = []
        for sb in range(first, min(first + 21, 127)):
            scale = torch.tensor([sb], dtype=torch.uint8, device="cuda").view(torch.float8_e4m3fn).float()
            amax = (6.0 * scale).to(dtype)                     # six significant bits: the scale byte is sb itself
            v = every[every.float().abs() <= amax.float()]     # drops the NaNs as well
            n = -(-v.numel() // 15) * 15
            v = torch.cat([v, v.new_zeros(n - v.numel())]).reshape(-1, 15)
            rows.append(torch.cat([amax.expand(v.shape[0], 1), v], dim=1))
        _check(torch.cat(rows))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_every_maximum(dtype):
    bits = torch.arange(65536, dtype=torch.int32, device="cuda").to(torch.int16)
    amax = bits.view(dtype)
    amax = amax[~torch.isnan(amax)]                            # both signs, zeros, subnormals and infinities
    x = torch.zeros(amax.numel(), 16, dtype=dtype, device="cuda")
    x[:, 5] = amax
    x[:, 9] = amax / 2
    x[:, 12] = -amax / 3
    _check(x)
