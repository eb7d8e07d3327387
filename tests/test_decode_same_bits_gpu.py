"""A unit's decode result does not depend on which kernel merges its pieces: the cluster that computed them, or, where not
all clusters are resident at once, the combine kernel."""

import pytest
import torch

import sageattention_b200.nvfp4 as nv
from gpu_util import seeded_bf16
from sageattention_b200 import _lib

pytestmark = pytest.mark.gpu

_UNTOUCHED = 0x5A


def _decode(q, packed, hk, g, s, nsplit, split):
    """(out, log-sum-exp, whether partials were written to the workspace) of the C entry."""
    z, d = q.shape[0], q.shape[-1]
    knv, ksc, vnv, vsc = (t.reshape(z * hk, *t.shape[-2:]) for t in packed[:4])
    out = torch.empty(z, hk * g, d, dtype=q.dtype, device="cuda")
    lse = torch.empty(z, hk * g, dtype=torch.float32, device="cuda")
    ws = torch.full((z * hk * nsplit * (16 * d + 32) * 4,), _UNTOUCHED, dtype=torch.uint8, device="cuda")
    _lib.check(_lib.lib().nvfp4_decode(
        q.data_ptr(), _lib.dtype_code(q.dtype), q.stride(0), q.stride(1), knv.data_ptr(), knv.stride(0), ksc.data_ptr(),
        ksc.stride(0), vnv.data_ptr(), vnv.stride(0), vnv.stride(1), vsc.data_ptr(), vsc.stride(0), vsc.stride(1), z, hk, g, d, s,
        d ** -0.5, out.data_ptr(), lse.data_ptr(), ws.data_ptr(), ws.numel(), nsplit, split, _lib.status_word(q.device).data_ptr(),
        _lib.stream_ptr(q.device)), "nvfp4_decode")
    assert _lib.read_status("cuda:0") == 0
    return out, lse, not bool((ws == _UNTOUCHED).all())


def _operands(z, hk, g, d, s, dtype):
    k, _ = seeded_bf16((z, hk, s, d), 71)
    v, _ = seeded_bf16((z, hk, s, d), 72)
    return seeded_bf16((z, hk * g, d), 73)[0].to(dtype), nv.nvfp4_quant_kv_decode(k, v)


# pieces a unit: all that a cluster can have; head counts of each of the kernel's three sizes; the last piece clipped
@pytest.mark.parametrize("nsplit", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("g,d,dtype", [(1, 128, torch.float16), (4, 128, torch.bfloat16), (8, 128, torch.float32),
                                       (16, 128, torch.float32), (3, 256, torch.float32), (16, 256, torch.bfloat16)])
def test_cluster_and_combine_kernel_agree(g, d, dtype, nsplit):
    hk, split = 2, 256
    s = split * nsplit - 77
    many = 148 // (hk * nsplit) + 1                       # more items than SMs
    q, packed = _operands(many, hk, g, d, s, dtype)
    all_out, all_lse, wrote = _decode(q, packed, hk, g, s, nsplit, split)
    assert wrote
    for z in (0, many - 1):
        one = tuple(t.reshape(many, hk, *t.shape[-2:])[z].contiguous() for t in packed[:4])
        out, lse, wrote = _decode(q[z:z + 1].contiguous(), one, hk, g, s, nsplit, split)
        assert not wrote                                  # merged by the cluster
        assert torch.equal(out[0], all_out[z]) and torch.equal(lse[0], all_lse[z])


# queries at an address, or with a stride, that is a multiple of their elements' size only
@pytest.mark.parametrize("d,dtype", [(128, torch.bfloat16), (256, torch.float16), (128, torch.float32)])
def test_queries_without_alignment(d, dtype):
    hk, g, s = 2, 4, 700
    q, packed = _operands(2, hk, g, d, s, dtype)
    ref = _decode(q, packed, hk, g, s, 2, 512)
    shifted = torch.empty(q.numel() + 1, dtype=dtype, device="cuda")[1:].view(q.shape)
    strided = torch.empty(2, hk * g, d + 1, dtype=dtype, device="cuda")[..., :d]
    for other in (shifted, strided):
        other.copy_(q)
        got = _decode(other, packed, hk, g, s, 2, 512)
        assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])
