"""Forward masks at the edges of key tiles: biases that are zero in whole tiles and not in others, and samples of
packed rows that end at, before and behind tile and chunk boundaries, causal or not, with and without a bias."""

import numpy as np
import pytest
import torch

from gpu_util import cos, seeded_bf16
from oracle import nvfp4_oracle as O

pytestmark = pytest.mark.gpu

MAXABS = 2e-2


def _check(q, k, v, qf, kf, vf, h, hk, causal, bias=None, cu=None):
    import sageattention_b200.nvfp4 as nv
    from sageattention_b200 import _lib
    z, _, sq, d = q.shape
    skv = k.shape[2]
    packs = nv.nvfp4_flash_attention(q, k, v, d ** -0.5, num_key_value_groups=h // hk, return_packs=True)[1]
    out = nv.nvfp4_flash_attention_packed(
        *packs, z, h, hk, sq, skv, d, d ** -0.5, torch.float32, causal=causal,
        key_pad_bias=None if bias is None else torch.from_numpy(bias).cuda(),
        cu_seqlens=None if cu is None else torch.tensor(cu, dtype=torch.int32, device="cuda"))
    assert _lib.read_status("cuda") == 0
    ref, _ = O.attention_mode_b(qf, kf, vf, d ** -0.5, causal, h // hk, cu_seqlens=cu, key_pad_bias=bias)
    o = out.cpu().numpy()
    assert np.isfinite(o).all()
    assert cos(o, ref) >= 0.9999 and np.abs(o - ref).max() <= MAXABS, (cos(o, ref), np.abs(o - ref).max())


@pytest.mark.parametrize("d", [128, 256])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("keys", [(), (127,), (128,), (255, 256), range(256, 700), range(640, 700), (0, 699)])
def test_bias_in_some_tiles(d, causal, keys):
    z, h, hk, sq, skv = 2, 2, 1, 150, 700
    q, qf = seeded_bf16((z, h, sq, d), 51)
    k, kf = seeded_bf16((z, hk, skv, d), 52)
    v, vf = seeded_bf16((z, hk, skv, d), 53)
    bias = np.zeros((z, skv), np.float32)
    bias[1, list(keys)] = -np.inf                  # the other entry of the batch has no bias at all
    if len(keys) == 2:
        bias[1, keys[0]] = 2.5
    _check(q, k, v, qf, kf, vf, h, hk, causal, bias=bias)


@pytest.mark.parametrize("d", [128, 256])
@pytest.mark.parametrize("causal,biased", [(True, False), (True, True), (False, False), (False, True)])
@pytest.mark.parametrize("lens", [(128, 128, 128), (1, 127, 129, 31, 32, 33), (400, 3, 300), (63, 65, 1, 1, 254, 17)])
def test_packed_samples(d, causal, biased, lens):
    h, hk, s = 2, 1, sum(lens)
    q, qf = seeded_bf16((1, h, s, d), 61)
    k, kf = seeded_bf16((1, hk, s, d), 62)
    v, vf = seeded_bf16((1, hk, s, d), 63)
    bias = None
    if biased:
        bias = np.zeros((1, s), np.float32)
        bias[0, 1::7] = -3.0
    _check(q, k, v, qf, kf, vf, h, hk, causal, bias=bias, cu=np.cumsum((0,) + lens))


@pytest.mark.parametrize("d", [128, 256])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("visible", [0, 1, 127, 128, 129, 383, 384, 385, 443, 700])
def test_hidden_keys_at_the_end(d, causal, visible):
    """Tiles that the bias hides from every row are not walked, wherever the last visible key lies; one entry of the batch
    has its own number of keys, in another only the last one is visible."""
    z, h, hk, sq, skv = 3, 2, 1, 150, 700
    q, qf = seeded_bf16((z, h, sq, d), 55)
    k, kf = seeded_bf16((z, hk, skv, d), 56)
    v, vf = seeded_bf16((z, hk, skv, d), 57)
    bias = np.zeros((z, skv), np.float32)
    bias[1, visible:] = -np.inf
    bias[2, :skv - 1] = -np.inf
    import sageattention_b200.nvfp4 as nv
    from sageattention_b200 import _lib
    out, lse = nv.nvfp4_flash_attention(q.float(), k.float(), v.float(), d ** -0.5, causal=causal, num_key_value_groups=h // hk,
                                        key_pad_bias=torch.from_numpy(bias).cuda(), return_lse=True)
    assert _lib.read_status("cuda") == 0
    ref, ref_lse = O.attention_mode_b(qf, kf, vf, d ** -0.5, causal, h // hk, key_pad_bias=bias)
    o = out.cpu().numpy()
    assert np.isfinite(o).all() and np.abs(o - ref).max() <= MAXABS
    assert np.abs(lse.cpu().numpy().reshape(ref_lse.shape) - ref_lse).max() <= 2e-3


@pytest.mark.parametrize("d", [128, 256])
@pytest.mark.parametrize("tiles", [(1, 64), (64, 1), (33, 1, 1, 30), (2, 31, 32)])
def test_end_of_a_long_sample(d, tiles):
    """Non-causal packed rows whose samples go on for many tiles behind a query tile: samples of whole key tiles, so that each
    one is the same to the bit as alone."""
    import sageattention_b200.nvfp4 as nv
    h, hk, s = 2, 1, 128 * sum(tiles)
    q, _ = seeded_bf16((1, h, s, d), 64)
    k, _ = seeded_bf16((1, hk, s, d), 65)
    v, _ = seeded_bf16((1, hk, s, d), 66)
    cu = np.cumsum((0,) + tiles) * 128
    packs = nv.nvfp4_flash_attention(q, k, v, d ** -0.5, num_key_value_groups=h // hk, return_packs=True)[1]
    out = nv.nvfp4_flash_attention_packed(*packs, 1, h, hk, s, s, d, d ** -0.5, torch.bfloat16,
                                          cu_seqlens=torch.tensor(cu, dtype=torch.int32, device="cuda"))
    for a, b in zip(cu[:-1], cu[1:]):
        alone = nv.nvfp4_flash_attention(q[:, :, a:b], k[:, :, a:b], v[:, :, a:b], d ** -0.5, num_key_value_groups=h // hk)
        assert torch.equal(out[:, :, a:b], alone)
