"""CTAs of the dQ kernel walk several query tiles: dQ of every head of a launch with more tiles than SMs equals, to the
bit, dQ of a launch of that head alone -- one and many steps a tile, ragged ends, samples of one token, a key bias."""

import pytest
import torch

from gpu_util import seeded_bf16

pytestmark = pytest.mark.gpu


def _dq(q, k, v, do, causal, cu, bias):
    import sageattention_b200.nvfp4 as nv
    from sageattention_b200 import _lib
    q = q.clone().requires_grad_(True)
    out = nv.nvfp4_flash_attn_func(q, k.clone().requires_grad_(True), v, q.shape[-1] ** -0.5, causal=causal,
                                   num_key_value_groups=q.shape[1] // k.shape[1], cu_seqlens=cu, key_pad_bias=bias)
    dq, = torch.autograd.grad(out, (q,), do)
    assert _lib.read_status("cuda") == 0 and torch.isfinite(dq).all()
    return dq


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("z,h,hk,sq,skv,causal,cu,biased", [
    (2, 64, 16, 257, 257, True, None, False),          # 1 to 5 steps, an odd query tile
    (2, 64, 16, 129, 333, False, None, True),
    (1, 160, 32, 60, 60, True, None, False),           # one step a tile
    (1, 48, 16, 1000, 1000, True, (0, 1, 130, 300, 301, 640, 1000), False),
])
def test_dq_of_every_item_as_alone(dtype, z, h, hk, sq, skv, causal, cu, biased):
    d, g = 128, h // hk
    q, k, v, do = (seeded_bf16((z, n, s, d), 91 + i)[0].to(dtype)
                   for i, (n, s) in enumerate(((h, sq), (hk, skv), (hk, skv), (h, sq))))
    cus = None if cu is None else torch.tensor(cu, dtype=torch.int32, device="cuda")
    bias = None
    if biased:
        bias = torch.zeros(z, skv, device="cuda")
        bias[:, 1::5] = -2.0
        bias[0, skv - 40:] = float("-inf")
    dq = _dq(q, k, v, do, causal, cus, bias)
    for zi in range(z):
        for hi in sorted({0, 1, g, h // 2 + 1, h - 1}):
            one = [t[zi:zi + 1, j:j + 1].contiguous() for t, j in ((q, hi), (k, hi // g), (v, hi // g), (do, hi))]
            assert torch.equal(dq[zi, hi], _dq(*one, causal, cus, None if bias is None else bias[zi:zi + 1])[0, 0]), (zi, hi)


@pytest.mark.parametrize("d", [128, 256])
@pytest.mark.parametrize("mode", ["fp4_rownorm", "fp8_rownorm"])
@pytest.mark.parametrize("shift", [4, 8])
def test_scales_at_any_four_byte_address(d, mode, shift):
    """Whole stages of 16-byte aligned scales are loaded a row at a time, others word by word: the same gradients."""
    import sageattention_b200.nvfp4 as nv
    z, h, hk, s = 1, 4, 2, 400
    q, k, v, do = (seeded_bf16((z, n, s, d), 191 + i)[0] for i, n in enumerate((h, hk, hk, h)))

    def grads(offset):
        packs = []
        for x in (q, k):
            nib, sc = nv._quant_nvfp4(x.reshape(-1, s, d))
            raw = sc.view(torch.uint8)
            buf = torch.zeros(raw.numel() + 64, dtype=torch.uint8, device="cuda")
            moved = buf[offset:offset + raw.numel()].view(raw.shape)
            moved.copy_(raw)
            packs.append((nib, moved.view(sc.dtype)))
        t = [x.clone().requires_grad_(True) for x in (q, k, v)]
        out = nv.nvfp4_flash_attn_func(*t, d ** -0.5, causal=True, num_key_value_groups=h // hk, backward_grad_dots=mode,
                                       q_packs=packs[0], k_packs=packs[1])
        assert packs[0][1].data_ptr() % 16 == offset
        return torch.autograd.grad(out, t, do)

    for a, b in zip(grads(0), grads(shift)):
        assert torch.equal(a, b)
