"""Scale rows of Q and K that are aligned to words only: the loader's other path gives the same bits."""

import pytest
import torch

import sageattention_b200.nvfp4 as nv
from gpu_util import seeded_bf16
from sageattention_b200 import _lib

pytestmark = pytest.mark.gpu


def _shifted(t, by):
    """The same bytes at an address `by` bytes behind an allocation's start."""
    buf = torch.empty(t.numel() + by, dtype=torch.uint8, device=t.device)
    out = buf[by:].view(t.shape)
    out.copy_(t.view(torch.uint8))
    return out.view(t.dtype)


@pytest.mark.parametrize("d,sq,skv", [(128, 200, 200), (256, 129, 333), (128, 1, 127)])
def test_unaligned_scale_rows(d, sq, skv):
    z, h, hk = 1, 4, 2
    q, _ = seeded_bf16((z * h, sq, d), 81)
    k, _ = seeded_bf16((z * hk, skv, d), 82)
    v, _ = seeded_bf16((z * hk, skv, d), 83)
    qn, qs = nv._quant_nvfp4(q)
    kn, ks = nv._quant_nvfp4(k)
    vn, vs = nv._quant_nvfp4(v, transpose=True, k_pad=-(-skv // 128) * 128)
    run = lambda a, b: nv.nvfp4_flash_attention_packed(qn, a, kn, b, vn, vs, z, h, hk, sq, skv, d, d ** -0.5, torch.bfloat16,
                                                       causal=sq == skv)
    ref = run(qs, ks)
    for a, b in ((_shifted(qs, 4), ks), (qs, _shifted(ks, 4)), (_shifted(qs, 12), _shifted(ks, 4))):
        assert torch.equal(run(a, b), ref)
    assert _lib.read_status("cuda:0") == 0
