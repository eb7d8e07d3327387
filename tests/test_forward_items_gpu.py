"""The forward's CTAs walk several query tiles: every tile of a launch with more tiles than SMs equals, to the bit, the
same tile in a launch of its head alone, for odd and even numbers of key tiles, tiles that see no key, packed rows and
output strides that leave through a tensor map or row by row."""

import numpy as np
import pytest
import torch

from gpu_util import seeded_bf16
from oracle import nvfp4_oracle as O

pytestmark = pytest.mark.gpu


def _packs(z, h, hk, sq, skv, d, seed):
    import sageattention_b200.nvfp4 as nv
    q = seeded_bf16((z, h, sq, d), seed)
    k = seeded_bf16((z, hk, skv, d), seed + 1)
    v = seeded_bf16((z, hk, skv, d), seed + 2)
    packs = nv.nvfp4_flash_attention(q[0], k[0], v[0], d ** -0.5, num_key_value_groups=h // hk, return_packs=True)[1]
    return packs, q[1], k[1], v[1]


def _run(packs, z, h, hk, sq, skv, d, dtype, **kw):
    from sageattention_b200 import _lib
    from sageattention_b200.nvfp4 import flash
    out, lse = flash._run_flash_packed(*packs, z, h, hk, sq, skv, d, d ** -0.5, dtype, return_lse=True, **kw)
    assert _lib.read_status("cuda") == 0
    return out, lse.view(z, h, sq)


@pytest.mark.parametrize("d,dtype", [(128, torch.bfloat16), (128, torch.float32), (256, torch.float16), (256, torch.float32)])
@pytest.mark.parametrize("z,h,hk,sq,skv,causal,cu", [
    (3, 64, 32, 257, 257, True, None),               # 1, 2 and 3 key tiles, an odd query tile
    (2, 96, 32, 300, 140, True, None),               # the first query tiles see no key
    (2, 96, 32, 129, 400, False, None),
    (1, 48, 16, 1000, 1000, True, (0, 1, 130, 300, 301, 640, 1000)),
    (1, 48, 16, 1000, 1000, False, (0, 1, 130, 300, 301, 640, 1000)),
])
def test_every_item_as_alone(d, dtype, z, h, hk, sq, skv, causal, cu):
    packs, qf, kf, vf = _packs(z, h, hk, sq, skv, d, 71)
    cus = None if cu is None else torch.tensor(cu, dtype=torch.int32, device="cuda")
    out, lse = _run(packs, z, h, hk, sq, skv, d, dtype, causal=causal, cu_seqlens=cus)
    g = h // hk
    for zi in range(z):
        for hi in {0, 1, g, h // 2 + 1, h - 1}:
            i, j = zi * h + hi, zi * hk + hi // g
            one = [p[i:i + 1].contiguous() for p in packs[:2]] + [p[j:j + 1].contiguous() for p in packs[2:]]
            o1, l1 = _run(one, 1, 1, 1, sq, skv, d, dtype, causal=causal, cu_seqlens=cus)
            assert torch.equal(out[zi, hi], o1[0, 0]) and torch.equal(lse[zi, hi], l1[0, 0]), (zi, hi)
    zi, hi = z - 1, h - 1
    ref, _ = O.attention_mode_b(qf[zi:, hi:], kf[zi:, hi // g:], vf[zi:, hi // g:], d ** -0.5, causal, 1,
                                cu_seqlens=None if cu is None else np.array(cu))
    o = out[zi, hi].float().cpu().numpy()
    assert np.abs(o - ref[0, 0]).max() <= 2e-2 + (0 if dtype == torch.float32 else 2.0 ** -7 * np.abs(ref).max())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_output_strides(dtype):
    """Heads and rows at any positive stride, padded rows untouched; a negative stride is stored row by row."""
    from sageattention_b200 import _lib
    z, h, hk, s, d = 2, 4, 2, 200, 128
    packs, *_ = _packs(z, h, hk, s, s, d, 81)
    want, _ = _run(packs, z, h, hk, s, s, d, dtype)
    pad = {torch.bfloat16: 8, torch.float32: 4}[dtype]
    for pitch, flip in ((d, False), (d + pad, False), (d, True)):
        buf = torch.full((z, h, s, pitch), 7.0, dtype=dtype, device="cuda")
        so_h, base = s * pitch, buf.data_ptr()
        if flip:                                     # heads from the last to the first
            base, so_h = buf[0, h - 1].data_ptr(), -so_h
        _lib.call("nvfp4_fwd", buf.device, *(p.data_ptr() for p in packs), None, None, None, base, _lib.dtype_code(dtype),
                  h * s * pitch, so_h, pitch, None, z, h, hk, s, s, (s + 127) // 128 * 128, d, d ** -0.5, 0,
                  _lib.status_word(buf.device).data_ptr(), _lib.stream_ptr(buf.device))
        got = buf.flip(1) if flip else buf
        assert _lib.read_status("cuda") == 0
        assert torch.equal(got[..., :d], want) and (got[..., d:] == 7.0).all()
