"""The native paths under saved-tensor hooks, activation checkpointing and CUDA graph capture: the same results to the bit."""

import pytest
import torch

pytestmark = pytest.mark.gpu

Z, H, HK, S = 1, 4, 2, 200


def _inputs(d=128):
    g = torch.Generator(device="cuda").manual_seed(5)
    return [torch.randn(Z, n, S, d, device="cuda", dtype=torch.bfloat16, generator=g) for n in (H, HK, HK, H)]


def _attend(q, k, v, mode):
    import sageattention_b200.nvfp4 as nv
    return nv.nvfp4_flash_attn_func(q, k, v, q.shape[-1] ** -0.5, causal=True, num_key_value_groups=H // HK,
                                    backward_grad_dots=mode)


def _grads(mode, d=128):
    q, k, v, do = _inputs(d)
    ops = [t.requires_grad_(True) for t in (q, k, v)]
    out = _attend(*ops, mode)
    return (out.detach(), *torch.autograd.grad(out, ops, do))


def _same(a, b):
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert torch.equal(x, y)


@pytest.mark.parametrize("mode", ["bf16", "fp4_rownorm"])
def test_saved_tensor_hooks(mode):
    kept = []

    def pack(t):
        kept.append(t.shape)
        return t.cpu()

    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.cuda()):
        got = _grads(mode)
    assert len(kept) >= 9                 # q, k, v, out, lse and the packs of q and k
    _same(got, _grads(mode))


@pytest.mark.parametrize("reentrant", [False, True])
def test_activation_checkpoint(reentrant):
    from torch.utils.checkpoint import checkpoint
    q, k, v, do = _inputs()
    ops = [t.requires_grad_(True) for t in (q, k, v)]
    out = checkpoint(lambda *a: _attend(*a, "bf16"), *ops, use_reentrant=reentrant)
    out.backward(do)
    _same((out.detach(), *(t.grad for t in ops)), _grads("bf16"))


def test_compiled_autograd_is_refused():
    from torch._dynamo import compiled_autograd
    q, k, v, do = _inputs()
    out = _attend(q.requires_grad_(True), k, v, "bf16")
    with pytest.raises((RuntimeError, NotImplementedError)):
        with compiled_autograd._enable(lambda graph: graph):
            out.backward(do)


def _captured(step):
    """Results of `step` run by a graph, on inputs that it holds."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step()
    for t in out:
        t.view(torch.uint8).zero_()
    graph.replay()
    torch.cuda.synchronize()
    res = [t.clone() for t in out]
    del graph
    return res


def _captured_training(mode, d):
    q, k, v, do = _inputs(d)
    ops = [t.requires_grad_(True) for t in (q, k, v)]

    def step():
        out = _attend(*ops, mode)
        return (out.detach(), *torch.autograd.grad(out, ops, do))

    return _captured(step)


@pytest.mark.parametrize("d", [128, 256])
@pytest.mark.parametrize("mode", ["bf16", "fp4_rownorm"])
def test_training_step_in_a_graph(mode, d):
    _same(_captured_training(mode, d), _grads(mode, d=d))


@pytest.mark.parametrize("d", [128, 256])
def test_prompt_and_decode_in_a_graph(d):
    import sageattention_b200.nvfp4 as nv
    q, k, v, _ = _inputs(d)
    scaling, g = d ** -0.5, H // HK

    def run(wrap):
        cache = nv.NVFP4KVCache(Z, HK, d, 256, "cuda", recent_window=64)

        def prompt():
            out = nv.nvfp4_flash_attention(q, k, v, scaling, causal=True, num_key_value_groups=g)
            cache.prefill(k, v)
            return (out,)

        def token():
            cache.length, cache.partial_len = S, S % 16
            cache.append(k[:, :, :1], v[:, :, :1])
            return (nv.nvfp4_flash_decode_prequant(q[:, :, :1], cache.get_packed(), scaling, g),
                    cache.hybrid_decode(q[:, :, :1], scaling, g))

        return (*wrap(prompt), *wrap(token), cache.knv, cache.vnv, cache.rk)

    _same(run(_captured), run(lambda f: f()))
