"""V^T and two-way packers over runs of key tiles: a block walks one, two or four tiles of 128 keys by the number of tiles in
the call, and the bytes do not depend on it.  Two-way packs of scaled operands against the oracle."""

import numpy as np
import pytest
import torch

import sageattention_b200.nvfp4 as nv
from gpu_util import np_u8
from oracle import nvfp4_oracle as O
from sageattention_b200.nvfp4 import flash

pytestmark = pytest.mark.gpu

# tiles of 128 keys x 64 columns: 9 a row, 2304 in all (runs of two); 10 a row, 4000 (four); 5 a row, 1800 at D 256 (two);
# 13 a row, 3640 (four); every last run is clipped
SHAPES = [(128, 1100, 128), (200, 1153, 128), (90, 513, 256), (140, 1601, 128)]
DTYPES = [torch.bfloat16, torch.float16, torch.float32]


def _operand(b, s, d, dtype, seed=5):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(b, s, d, device="cuda", generator=gen) * 1.3).to(dtype)


def _same(a, b):
    return torch.equal(a.contiguous().view(torch.uint8), b.contiguous().view(torch.uint8))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("b,s,d", SHAPES)
def test_runs_of_tiles(b, s, d, dtype):
    x = _operand(b, s, d, dtype)
    pad = -(-s // 128) * 128
    vn, vs = nv._quant_nvfp4(x, transpose=True, k_pad=pad)
    dn, ds, tn, ts = flash._quant_nvfp4_dual(x, pad)
    few = 16                                     # entries a call: a block takes one tile
    assert pad // 128 * (d // 64) * few < 1776
    for i in range(0, b, few):
        n, sc = nv._quant_nvfp4(x[i:i + few], transpose=True, k_pad=pad)
        rn, rs = nv._quant_nvfp4(x[i:i + few])
        for got, want in ((vn, n), (vs, sc), (tn, n), (ts, sc), (dn, rn), (ds, rs)):
            assert _same(got[i:i + few], want)
    for i in (0, b // 2, b - 1):
        n, sc = O.pack(x[i:i + 1].float().cpu().numpy(), transpose=True, k_pad=pad)
        assert np.array_equal(np_u8(vn[i:i + 1]), n) and np.array_equal(np_u8(vs[i:i + 1]), sc)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("b,s,d", SHAPES)
def test_runs_of_tiles_in_the_fused_packers(b, s, d, dtype):
    k, v = _operand(b, s, d, dtype, 6), _operand(b, s, d, dtype, 7)
    pad = -(-s // 128) * 128
    want = (*nv._quant_nvfp4(k), *nv._quant_nvfp4(v, transpose=True, k_pad=pad))       # held by the test above
    for got, ref in zip(flash._quant_qkv_fwd(k[:2], k, v, pad)[2:], want):
        assert _same(got, ref)
    cache = nv.NVFP4KVCache(2, b // 2, d, pad, "cuda", dtype)
    cache.prefill(k.view(2, b // 2, s, d), v.view(2, b // 2, s, d))
    groups = -(-s // 16)
    for got, ref in zip((cache.knv[..., :s, :], cache.ksc[..., :s, :], cache.vnv[..., :groups * 8], cache.vsc[..., :groups]),
                        (want[0], want[1], want[2][..., :groups * 8], want[3][..., :groups])):
        assert _same(got.reshape(ref.shape), ref)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("amax", [3e-3, 1.0, 1000.0])
def test_two_way_pack_of_scaled_values(amax, dtype):
    """Values that end on a rounding boundary under every scale byte, before them a division by a power of two."""
    pre = 2.0 ** np.ceil(np.log2(amax))
    ties = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0, 6.0])
    scales = torch.arange(1, 127, dtype=torch.uint8).view(torch.float8_e4m3fn).float()
    rows = torch.cat([ties, -ties])[None] * scales[:, None] * pre                       # 7 significant bits
    rows = rows[(rows.abs().amax(dim=1) <= torch.finfo(dtype).max) & (rows.abs().amin(dim=1) >= torch.finfo(dtype).tiny)]
    n = rows.shape[0] // 8 * 8
    ties_d = rows[:n].reshape(1, n // 8, 128)
    ties_s = rows[:n // 16 * 16].T.contiguous()[None]                                   # a group along S
    gen = torch.Generator().manual_seed(9)
    rand = torch.randn(3, 300, 128, generator=gen) * amax / 4
    t = torch.tensor([amax], device="cuda")
    for x in (ties_d, ties_s, rand):
        x = x.to(dtype)
        pad = -(-x.shape[1] // 128) * 128
        dn, ds, tn, ts = flash._quant_nvfp4_dual(x.cuda(), pad, t)
        scaled = (x.double() / pre).float().numpy()
        for (gn, gs), (wn, ws) in (((dn, ds), O.pack(scaled)), ((tn, ts), O.pack(scaled, transpose=True, k_pad=pad))):
            assert np.array_equal(np_u8(gs), ws) and np.array_equal(np_u8(gn), wn)
