"""Work split over CTAs: the dK / dV passes of the backward with the query steps of a key tile shared by a
cluster, the decode combine with many pieces per unit, and the tile widths of the V projection."""

import numpy as np
import pytest
import torch

from gpu_util import cos, seeded_bf16
from oracle import nvfp4_oracle as O

pytestmark = pytest.mark.gpu


def _status():
    from sageattention_b200 import _lib
    return _lib.read_status("cuda")


def _grads(q, k, v, do, g, causal, mode, cu=None):
    import sageattention_b200.nvfp4 as nv
    q, k, v = (t.clone().requires_grad_(True) for t in (q, k, v))
    out = nv.nvfp4_flash_attn_func(q, k, v, q.shape[-1] ** -0.5, causal=causal, num_key_value_groups=g, cu_seqlens=cu,
                                   backward_grad_dots=mode, stochastic_rounding=False)
    out.backward(do)
    torch.cuda.synchronize()
    assert _status() == 0
    return q.grad, k.grad, v.grad


# One batch entry alone leaves most SMs idle, so its key tiles are split where they have enough steps; among
# `copies` of itself there are enough tiles that they are not (or less).  CTAs of a cluster without a step; ragged
# ends; a head dim of two halves; keys that only the last rows see.
@pytest.mark.parametrize("mode", ["bf16", "fp4_rownorm", "fp8_rownorm"])
@pytest.mark.parametrize("d,h,hk,sq,skv,causal,copies", [
    (128, 1, 1, 129, 129, False, 160),
    (128, 8, 2, 65, 257, True, 64),
    (128, 8, 1, 1000, 1000, True, 40),
    (128, 4, 2, 700, 1300, False, 32),
    (256, 4, 1, 333, 333, True, 64),
    (256, 2, 2, 1, 140, True, 64),
    (128, 1, 1, 1900, 1900, True, 40),      # split by eight: the last tiles have fewer steps than CTAs
    (256, 1, 1, 880, 880, True, 40),
])
def test_split_key_tiles_match_whole_ones(d, h, hk, sq, skv, causal, copies, mode):
    q, _ = seeded_bf16((1, h, sq, d), 21)
    k, _ = seeded_bf16((1, hk, skv, d), 22)
    v, _ = seeded_bf16((1, hk, skv, d), 23)
    do, _ = seeded_bf16((1, h, sq, d), 24)
    alone = _grads(q, k, v, do, h // hk, causal, mode)
    many = _grads(*(t.repeat(copies, 1, 1, 1) for t in (q, k, v, do)), h // hk, causal, mode)
    for nm, a, b in zip(("dq", "dk", "dv"), alone, many):
        for i in (0, copies - 1):
            e = (a[0].float() - b[i].float()).norm() / b[i].float().norm().clamp_min(1e-20)
            assert float(e) <= 4e-3, (nm, i, float(e))      # sums in another order, rounded once to bf16


@pytest.mark.parametrize("mode,floor", [("bf16", 0.99), ("fp4_rownorm", 0.93)])
def test_split_packed_row_matches_exact_gradients(mode, floor):
    """Samples of a packed row end inside tiles: a CTA's share of a tile's steps may lie in one sample only."""
    h, hk, d, lens = 4, 2, 128, (3, 300, 129, 1, 500, 91)
    s = sum(lens)
    q, qn = seeded_bf16((1, h, s, d), 31)
    k, kn = seeded_bf16((1, hk, s, d), 32)
    v, vn = seeded_bf16((1, hk, s, d), 33)
    do, don = seeded_bf16((1, h, s, d), 34)
    cu = np.cumsum((0,) + lens)
    got = _grads(q, k, v, do, h // hk, True, mode, cu=torch.tensor(cu, dtype=torch.int32, device="cuda"))
    ref = O.attention_grads(qn, kn, vn, don, d ** -0.5, True, h // hk, cu_seqlens=cu)
    for nm, a, b in zip(("dq", "dk", "dv"), got, ref):
        a = a.float().cpu().numpy()
        assert np.isfinite(a).all()
        assert cos(a, b) >= floor, (nm, cos(a, b))


@pytest.mark.parametrize("d,s,split_kv", [(128, 128 * 514 + 5, 128), (128, 128 * 511 + 1, 128), (128, 1100, 128),
                                          (256, 1100, 384), (256, 4000, 0)])
def test_combine_of_many_pieces(d, s, split_kv):
    """Up to and beyond one round of the combine's table; a block of two, four and eight warps."""
    import sageattention_b200.nvfp4 as nv
    from sageattention_b200.nvfp4 import flash
    q, _ = seeded_bf16((1, 3, 1, d), 41)
    k, _ = seeded_bf16((1, 1, s, d), 42)
    v, _ = seeded_bf16((1, 1, s, d), 43)
    packed = nv.nvfp4_quant_kv_decode(k, v)
    out, lse = flash._decode_core(q.float(), packed, d ** -0.5, 3, True, split_kv=split_kv)
    whole, whole_lse = flash._decode_core(q.float(), packed, d ** -0.5, 3, True, split_kv=-(-s // 128) * 128)
    assert _status() == 0
    assert float((lse - whole_lse).abs().max()) <= 1e-3
    assert cos(out.cpu().numpy(), whole.cpu().numpy()) >= 0.99     # P is rounded against another running maximum


@pytest.mark.parametrize("s,hidden,hk,d", [(1000, 1000, 8, 128), (450, 1544, 8, 128), (130, 584, 3, 64), (17, 4096, 2, 256),
                                           (2430, 1000, 8, 128), (2500, 200, 16, 128)])
def test_projection_tiles_match_product(s, hidden, hk, d):
    """V projection in tiles of 32, 64 and 128 tokens, one and two CTAs per SM, hidden sizes that leave a remainder."""
    import sageattention_b200.nvfp4 as nv
    x, _ = seeded_bf16((1, s, hidden), 71)
    w, _ = seeded_bf16((hk * d, hidden), 72, scale=hidden ** -0.5)
    vnv, vsc, v = nv.vproj_quant_nvfp4(x, w, None, hk, d)
    assert _status() == 0
    ref = (x.float().double() @ w.double().T).view(1, s, hk, d).permute(0, 2, 1, 3)
    assert float((v.double() - ref).abs().max()) <= 2.0 ** -8 * max(1.0, float(ref.abs().max())) * 1.01
    n2, s2 = nv._quant_nvfp4(v.reshape(hk, s, d), transpose=True, k_pad=-(-s // 128) * 128)
    assert torch.equal(vnv, n2) and torch.equal(vsc.view(torch.uint8), s2.view(torch.uint8))
