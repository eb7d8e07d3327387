"""The allocation-free decode entry where partials really go through its scratch: units of more pieces than a cluster
merges, and the balanced decomposition."""

import pytest
import torch

import sageattention_b200.nvfp4 as nv
from gpu_util import seeded_bf16
from sageattention_b200 import _lib

pytestmark = pytest.mark.gpu

_UNTOUCHED = 0x5A


@pytest.mark.parametrize("d,s,nsplit,split", [(128, 2300, 9, 256), (128, 1500, 12, 128), (256, 1400, 11, 128), (128, 3000, 0, 0),
                                              (256, 2000, 0, 0)])
def test_static_scratch_equals_a_workspace(d, s, nsplit, split):
    z, hk, g = 2, 2, 4
    L, status, stream = _lib.lib(), _lib.status_word("cuda:0"), _lib.stream_ptr("cuda:0")
    results = []
    for seed in (91, 95):                               # the array keeps what the call before it left
        k, _ = seeded_bf16((z, hk, s, d), seed)
        v, _ = seeded_bf16((z, hk, s, d), seed + 1)
        q, _ = seeded_bf16((z, hk * g, d), seed + 2)
        knv, ksc, vnv, vsc = nv.nvfp4_quant_kv_decode(k, v)[:4]
        common = (q.data_ptr(), _lib.dtype_code(q.dtype), q.stride(0), q.stride(1), knv.data_ptr(), knv.stride(0),
                  ksc.data_ptr(), ksc.stride(0), vnv.data_ptr(), vnv.stride(0), vnv.stride(1), vsc.data_ptr(), vsc.stride(0),
                  vsc.stride(1), z, hk, g, d, s, d ** -0.5)
        outs = []
        for static in (False, True, True):
            out, lse = torch.empty_like(q), torch.empty(z, hk * g, device="cuda")
            if static:
                _lib.check(L.nvfp4_decode_static(*common, out.data_ptr(), lse.data_ptr(), nsplit, split, status.data_ptr(),
                                                 stream), "nvfp4_decode_static")
            else:
                ws = torch.full((1 << 24,), _UNTOUCHED, dtype=torch.uint8, device="cuda")
                _lib.check(L.nvfp4_decode(*common, out.data_ptr(), lse.data_ptr(), ws.data_ptr(), ws.numel(), nsplit, split,
                                          status.data_ptr(), stream), "nvfp4_decode")
                assert bool((ws != _UNTOUCHED).any())      # the partials were here
            outs.append((out, lse))
        assert _lib.read_status("cuda:0") == 0
        for out, lse in outs[1:]:
            assert torch.equal(out, outs[0][0]) and torch.equal(lse, outs[0][1])
        results.append(outs[0][0])
    assert not torch.equal(*results)
