"""Operands whose extents do not fit one another are refused on the host: the kernels take their sizes from one
operand and would read past the end of another."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rn(*shape, dtype=torch.bfloat16):
    return torch.randn(*shape, device="cuda", dtype=dtype)


def _bad_kv(z, hk, s, d):
    """(key shape, value shape) that do not fit a query [z, 2 hk, s, d]."""
    ok = (z, hk, s, d)
    return [(ok, (z, hk, s // 2, d)), (ok, (z, hk // 2, s, d)), (ok, (1, hk, s, d)), (ok, (z, hk, s, d // 2)),
            ((1, hk, s, d), ok), ((z, hk, s, d // 2), ok), ((1, hk, s, d), (1, hk, s, d))]


@pytest.mark.parametrize("shapes", _bad_kv(2, 2, 256, 128))
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_attention_refuses_operands_of_other_extents(shapes, dtype):
    import sageattention_b200.nvfp4 as nv
    q, k, v = _rn(2, 4, 256, 128, dtype=dtype), _rn(*shapes[0], dtype=dtype), _rn(*shapes[1], dtype=dtype)
    for fn in (nv.nvfp4_flash_attention, nv.nvfp4_flash_attn_func):
        with pytest.raises((RuntimeError, AssertionError)):
            fn(q, k, v, 0.1, causal=True, num_key_value_groups=2)
    q.requires_grad_(True)
    with pytest.raises((RuntimeError, AssertionError)):
        nv.nvfp4_flash_attn_func(q, k, v, 0.1, causal=True, num_key_value_groups=2)


def test_value_of_another_shape_and_as_many_rows_is_taken():
    """[Z*Hk, S, D] rows and an already merged batch are the same values."""
    import sageattention_b200.nvfp4 as nv
    z, hk, s, d = 2, 2, 200, 128
    q, k, v = _rn(z, 4, s, d), _rn(z, hk, s, d), _rn(z, hk, s, d)
    ref = nv.nvfp4_flash_attention(q, k, v, 0.1, num_key_value_groups=2)
    for other in (v.view(z * hk, s, d), v.view(1, z * hk, s, d), v.view(z, hk, s, 2, d // 2)):
        assert torch.equal(ref, nv.nvfp4_flash_attention(q, k, other, 0.1, num_key_value_groups=2))


@pytest.mark.parametrize("which", ["k", "v", "v_rows", "out", "lse", "dout"])
def test_backward_refuses_operands_of_other_extents(which):
    from sageattention_b200.nvfp4 import flash
    z, h, hk, s, d = 2, 4, 2, 256, 128
    t = dict(q=_rn(z, h, s, d), k=_rn(z, hk, s, d), v=_rn(z, hk, s, d), out=_rn(z, h, s, d),
             lse=torch.zeros(z * h, s, device="cuda"), dout=_rn(z, h, s, d))
    name = which.split("_")[0]
    t[name] = t[name][:, :, : s // 2].contiguous() if which == "v_rows" else t[name][:1].contiguous()
    for run in (flash._run_bwd_hp, flash._run_bwd):
        with pytest.raises((RuntimeError, AssertionError)):
            run(t["q"], t["k"], t["v"], t["out"], t["lse"], t["dout"], 0.1, True, 2)


@pytest.mark.parametrize("call", ["quant", "dual", "mx8", "rope", "vproj", "attention", "train", "decode"])
@pytest.mark.parametrize("more", [False, True])
def test_operand_of_another_number_of_dimensions_is_a_value_error(call, more):
    import sageattention_b200.nvfp4 as nv
    from sageattention_b200.nvfp4 import flash
    x3 = torch.zeros(2, 16, 128, device="cuda", dtype=torch.bfloat16)
    x4 = torch.zeros(1, 2, 1, 128, device="cuda", dtype=torch.bfloat16)
    x = x3[None] if more else x3[0]                      # where three are wanted
    y = x4[None] if more else x4[0]                      # where four are wanted
    angle = torch.zeros(16, 64, device="cuda")
    packed = nv.nvfp4_quant_kv_decode(x4, x4)
    calls = dict(quant=lambda: nv._quant_nvfp4(x), dual=lambda: flash._quant_nvfp4_dual(x), mx8=lambda: flash._quant_mxfp8_t(x, 32),
                 rope=lambda: nv.rope_quant_nvfp4(x, angle, angle), vproj=lambda: nv.vproj_quant_nvfp4(x, x3[0, :, :], None, 1, 16),
                 attention=lambda: nv.nvfp4_flash_attention(y, x4, x4, 0.1),
                 train=lambda: nv.nvfp4_flash_attn_func(y, x4, x4, 0.1),
                 decode=lambda: nv.nvfp4_flash_decode_prequant(y, packed, 0.1))
    with pytest.raises(ValueError):
        calls[call]()
