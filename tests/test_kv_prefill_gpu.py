"""The one-launch cache prefill against the general path (separate packs and copies), byte for byte."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("s", [1, 15, 16, 17, 127, 128, 129, 513, 700])
@pytest.mark.parametrize("d,window", [(128, 0), (128, 128), (256, 40)])
def test_prefill_equals_general_path(s, d, window, dtype):
    import sageattention_b200.nvfp4 as nv
    z, hk = 2, 3
    gen = torch.Generator(device="cuda").manual_seed(s)
    rn = lambda *sh: torch.randn(*sh, device="cuda", dtype=dtype, generator=gen)
    for k, v in ((rn(z, hk, s, d), rn(z, hk, s, d)),
                 (rn(z, s, hk, d).transpose(1, 2), rn(z, s, hk, d).transpose(1, 2)),      # unit axes do not collapse
                 (rn(z, hk, s, d + 4)[..., 4:], rn(z, hk, s, d + 4)[..., 4:])):            # unaligned rows
        a, b = (nv.NVFP4KVCache(z, hk, d, 768, "cuda", dtype, recent_window=window) for _ in range(2))
        for c in (a, b):                      # a longer prompt first: what it left must not show
            c.prefill(rn(z, hk, 720, d) * 0 + 1.0, rn(z, hk, 720, d) * 0 + 2.0)
        a.prefill(k, v)
        b._prefill_converting(k, v)
        assert (a.length, a.partial_len) == (s, s % 16)
        names = ["knv", "ksc", "vnv", "vsc", "v_partial_bf16"] + (["rk", "rv"] if window else [])
        for n in names:
            x, y = getattr(a, n), getattr(b, n)
            assert torch.equal(x.contiguous().view(torch.uint8), y.contiguous().view(torch.uint8)), n


def test_prefill_takes_values_of_another_shape():
    """A value of as many elements is taken as [Z*Hk, S, D] rows, any other is refused."""
    import sageattention_b200.nvfp4 as nv
    z, hk, s, d = 2, 3, 70, 128
    k, v = (torch.randn(z, hk, s, d, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    caches = []
    for other in (v, v.view(z * hk, s, d), v.view(1, z * hk, s, d), v.view(-1, d), v.view(z, hk, s, 2, d // 2)):
        caches.append(nv.NVFP4KVCache(z, hk, d, 128, "cuda"))
        caches[-1].prefill(k, other)
    for c in caches[1:]:
        assert torch.equal(caches[0].vnv, c.vnv) and torch.equal(caches[0].v_partial_bf16, c.v_partial_bf16)
    for other in (v[:, :, 1:], v[:1], v[..., :64]):
        with pytest.raises((RuntimeError, AssertionError)):
            caches[0].prefill(k, other)


@pytest.mark.parametrize("s", [20, 400])         # inside the window, and behind it
def test_hybrid_decode_refuses_other_head_counts(s):
    import sageattention_b200.nvfp4 as nv
    c = nv.NVFP4KVCache(2, 2, 128, 512, "cuda", recent_window=128)
    c.prefill(*(torch.randn(2, 2, s, 128, device="cuda", dtype=torch.bfloat16) for _ in range(2)))
    assert c.hybrid_decode(torch.randn(2, 4, 1, 128, device="cuda"), 0.1, 2).shape == (2, 4, 1, 128)
    for shape, g in (((2, 4, 1, 128), 4), ((1, 4, 1, 128), 2), ((2, 4, 1, 64), 2)):
        with pytest.raises((RuntimeError, AssertionError)):
            c.hybrid_decode(torch.randn(*shape, device="cuda"), 0.1, g)
