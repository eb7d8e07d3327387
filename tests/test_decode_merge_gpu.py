"""Partials of a unit merged by the cluster that computed them, against the pieces one by one."""

import pytest
import torch

import sageattention_b200.nvfp4 as nv
from gpu_util import seeded_bf16
from sageattention_b200 import _lib
from sageattention_b200.nvfp4 import flash

pytestmark = pytest.mark.gpu


# items a unit: odd, even, the most a cluster has, one more (combine kernel); units that fill the GPU and that do not fit it
@pytest.mark.parametrize("z,hk,g,d,nsplit,dtype", [
    (1, 3, 4, 128, 2, torch.bfloat16), (2, 2, 1, 128, 3, torch.float16), (1, 5, 5, 128, 5, torch.float32),
    (1, 2, 16, 256, 7, torch.bfloat16), (3, 5, 8, 128, 8, torch.bfloat16), (2, 8, 3, 128, 8, torch.bfloat16),
    (1, 4, 4, 256, 9, torch.float16), (37, 4, 2, 128, 1, torch.bfloat16), (20, 8, 2, 128, 1, torch.float32)])
def test_cluster_merge_equals_pieces(z, hk, g, d, nsplit, dtype):
    split = 256
    s = split * nsplit - 77
    k, _ = seeded_bf16((z, hk, s, d), 51)
    v, _ = seeded_bf16((z, hk, s, d), 52)
    q = seeded_bf16((z, hk * g, 1, d), 53)[0].to(dtype)
    packed = nv.nvfp4_quant_kv_decode(k, v)
    out, lse = flash._decode_core(q, packed, d ** -0.5, g, True, split_kv=split)
    pieces = []
    for j in range(nsplit):
        n = min(split, s - j * split)
        one = nv.nvfp4_quant_kv_decode(k[:, :, j * split:j * split + n], v[:, :, j * split:j * split + n])
        o, w = flash._decode_core(q.float(), one, d ** -0.5, g, True, split_kv=split)
        pieces.append((o.double().reshape(z, hk * g, d), w.double().reshape(z, hk * g)))
    w = torch.stack([p[1] for p in pieces])
    total = torch.logsumexp(w, dim=0)
    ref = sum(torch.exp(p[1] - total)[..., None] * p[0] for p in pieces)
    assert _lib.read_status("cuda:0") == 0
    # fp32 sums in another order, and the output's own rounding
    assert float((lse.double().reshape(z, hk * g) - total).abs().max()) <= 1e-5
    eps = torch.finfo(dtype).eps if dtype != torch.float32 else 1e-5
    assert float((out.double().reshape(z, hk * g, d) - ref).abs().max()) <= eps * max(1.0, float(ref.abs().max()))


def test_result_without_alignment():
    """The C entry takes a result that is aligned to its elements only."""
    z, hk, g, d, s = 1, 2, 4, 128, 700
    k, _ = seeded_bf16((z, hk, s, d), 61)
    v, _ = seeded_bf16((z, hk, s, d), 62)
    q, _ = seeded_bf16((z, hk * g, 1, d), 63)
    knv, ksc, vnv, vsc = nv.nvfp4_quant_kv_decode(k, v)[:4]
    ref, _ = flash._decode_core(q, nv.nvfp4_quant_kv_decode(k, v), d ** -0.5, g, True, split_kv=512)
    buf = torch.zeros(z * hk * g * d + 1, dtype=torch.bfloat16, device="cuda")
    ws = torch.empty(1 << 20, dtype=torch.uint8, device="cuda")
    knv, ksc, vnv, vsc = (t.reshape(z * hk, *t.shape[-2:]) for t in (knv, ksc, vnv, vsc))
    stream = torch.cuda.current_stream().cuda_stream
    _lib.check(_lib.lib().nvfp4_decode(
        q.data_ptr(), 0, q.stride(0), q.stride(1), knv.data_ptr(), knv.stride(0), ksc.data_ptr(), ksc.stride(0), vnv.data_ptr(),
        vnv.stride(0), vnv.stride(1), vsc.data_ptr(), vsc.stride(0), vsc.stride(1), z, hk, g, d, s, d ** -0.5,
        buf[1:].data_ptr(), None, ws.data_ptr(), ws.numel(), 2, 512, None, stream), "nvfp4_decode")
    assert torch.equal(buf[1:].view(z, hk * g, 1, d), ref.view(z, hk * g, 1, d)) and float(buf[0]) == 0.0
