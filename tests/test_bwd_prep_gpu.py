"""Backward pre-pass: delta, bf16 copy and maximum over rows of every layout that takes another path (32-byte, 16-byte
and unaligned rows, linear and not, both head dims, row counts around a block's share)."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("d", [128, 256])
@pytest.mark.parametrize("b1,b2,s", [(1, 1, 1), (2, 3, 63), (1, 5, 129), (3, 1, 65)])
@pytest.mark.parametrize("layout", ["zhsd", "zshd", "pad8", "pad1"])
def test_prep_layouts(dtype, d, b1, b2, s, layout):
    from sageattention_b200.nvfp4 import flash
    g = torch.Generator().manual_seed(d + s)
    x, y = (torch.randn(b1, b2, s, d, generator=g).to(dtype).cuda() for _ in range(2))
    if layout == "zshd":
        xs, ys = (t.transpose(1, 2).contiguous().transpose(1, 2) for t in (x, y))
    elif layout == "zhsd":
        xs, ys = x, y
    else:
        pad = int(layout[3:])
        xs, ys = (torch.nn.functional.pad(t, (0, pad))[..., :d] for t in (x, y))
    xc, delta, amax = flash._bwd_prep(xs, ys, want_copy=True, want_amax=True)
    assert torch.equal(xc, x.reshape(b1 * b2, s, d).to(torch.bfloat16))
    assert float(amax) == float(x.abs().max())
    ref = (x.double() * y.double()).sum(-1).reshape(b1 * b2, s)
    assert float((delta.double() - ref).abs().max()) <= 1e-4
    only, none = flash._bwd_prep(xs, None, want_copy=True)
    assert none is None and torch.equal(only, xc)


@pytest.mark.parametrize("d", [128, 256])
@pytest.mark.parametrize("z,h,hk,s", [(1, 2, 1, 1), (2, 4, 2, 63), (1, 8, 2, 129), (3, 2, 2, 200)])
@pytest.mark.parametrize("layout", ["zhsd", "zshd", "pad"])
def test_copies_of_fp16_operands(d, z, h, hk, s, layout):
    """Q, K, V copied to bf16 in one launch: the gradients are those of operands converted beforehand."""
    import sageattention_b200.nvfp4 as nv
    from sageattention_b200.nvfp4 import flash
    g = torch.Generator().manual_seed(d + s)

    def mk(heads):
        t = torch.randn(z, heads, s, d, generator=g).to(torch.float16).cuda()
        if layout == "zshd":
            return t.transpose(1, 2).contiguous().transpose(1, 2)
        return torch.nn.functional.pad(t, (0, 16))[..., :d] if layout == "pad" else t

    q, k, v, do = mk(h), mk(hk), mk(hk), mk(h)
    out, lse, packs = nv.nvfp4_flash_attention(q, k, v, d ** -0.5, num_key_value_groups=h // hk, return_lse=True,
                                               return_packs=True)
    res = [flash._run_bwd_hp(a, b, c, out, lse, do, d ** -0.5, False, h // hk, q_packs=packs[0:2], k_packs=packs[2:4])
           for a, b, c in ((q, k, v), tuple(t.to(torch.bfloat16).contiguous() for t in (q, k, v)))]
    for a, b in zip(*res):
        assert torch.equal(a, b)
