"""Host side of the B200 NVFP4 flash-attention path.

Mirrors the operator surface of the reference module ``sageattention/nvfp4/flash.py`` (same
names, argument order, defaults and error behaviour) so callers and tests written against the
reference run unchanged; each function cites the reference lines it stands in for.  All compute
is in ``libnvfp4_b200.so`` (hand-written sm_100a CUDA behind the C ABI of
``include/nvfp4_b200.h``); torch is used for allocation, streams and autograd plumbing only.
Argument checks, allocation and launches of an operator are one native call
(``csrc/host/native.cpp``); the functions here fix names, defaults and return arity.
There is no Triton and no CPU fallback: CPU tensors are rejected.

Tile arguments (``block_m``, ``block_n``, ``num_warps``, ``num_stages``) are accepted for
signature compatibility.  The sm_100a kernels always walk 128-key tiles (the reference's own
D=128 default), so ``block_n`` only has to be 128 where it fixes a visible padding
(``nvfp4_quant_kv_decode``); other tile hints are ignored.
"""

from __future__ import annotations

import ctypes
import functools

import torch

from .. import _lib

# --------------------------------------------------------------------------- constants
# (names kept importable: tests and scripts of the reference read them, flash.py:260-273,
#  :993-1037)
_BWD_GRAD_DOTS_MODES = ("bf16", "fp4_rownorm", "fp8_rownorm", "fp4_legacy")
_BWD_AUTO_FP4_MIN_SEQ = 4096
_BWD_RN_DO_ZSHD = True
_FWD_TILE = {256: (128, 128, 8, 2), 128: (128, 128, 8, 2)}
_FWD_TILE_DEFAULT = (64, 128, 8, 3)
_FWD_TILE_VARLEN = {256: (128, 128, 8, 2), 128: (128, 128, 8, 2)}
_FWD_FUSED_QUANT_MAX_SEQ = 3072
_FWD_VARLEN_DENSE_MIN_MEAN = 4096
_KEY_TILE = 128


def _next_mult(n: int, m: int) -> int:
    return ((n + m - 1) // m) * m


def _resolve_fwd_tiles(d, block_m, block_n, num_warps, num_stages, varlen=False, mean_len=None):
    """Tile policy hook of the reference (flash.py:1040-1056).

    Explicit tiles are echoed back, generic defaults resolve to the one tile shape the sm_100a
    forward kernel implements (128 query rows x 128 keys).
    """
    if (block_m, block_n, num_warps, num_stages) == _FWD_TILE_DEFAULT:
        return (_FWD_TILE_VARLEN if varlen else _FWD_TILE).get(d, _FWD_TILE_DEFAULT)
    return block_m, block_n, num_warps, num_stages


def _resolve_backward_grad_dots(mode, eff_seq, save_backward_packs, num_key_value_groups) -> str:
    """Backward-mode resolver, same table as the reference (flash.py:276-302).

    ``None`` = AUTO: "bf16" (high-precision gradient GEMMs) below ``_BWD_AUTO_FP4_MIN_SEQ``
    effective sequence, else "fp4_rownorm"; "bf16" silently downgrades to "fp4_rownorm" when only
    packs are saved or the GQA group exceeds 8.
    """
    if mode is None:
        mode = "bf16" if eff_seq < _BWD_AUTO_FP4_MIN_SEQ else "fp4_rownorm"
    if mode not in _BWD_GRAD_DOTS_MODES:
        raise ValueError(
            f"backward_grad_dots must be one of {_BWD_GRAD_DOTS_MODES} or None (auto), got {mode!r}")
    if mode == "bf16" and (save_backward_packs or num_key_value_groups > 8):
        mode = "fp4_rownorm"
    return mode


# --------------------------------------------------------------------------- packer
def _pack_into(x, nib, sc, transpose=False, k_pad=None):
    """Pack ``x`` ([B,R,K], or [B,K,R] with ``transpose``) into existing (possibly strided) views.

    ``nib`` [B,R,Kp/2] uint8 and ``sc`` [B,R,Kp/16] (uint8 or float8_e4m3fn) must have unit
    stride along their last axis; this is how the KV cache packs straight into its buffers.
    """
    _lib.native().pack_into(x, nib, sc, transpose, k_pad)


def _quant_nvfp4(x: torch.Tensor, transpose: bool = False, k_pad: int | None = None):
    """NVFP4-pack along the contraction axis; stands in for flash.py:363-419.

    ``x`` is ``[B, R, K]`` (quantised along K) or, with ``transpose=True``, ``[B, K, R]`` read
    through its strides to produce the V^T layout.  ``k_pad`` zero-pads the contraction axis
    (padded groups get the floor scale and zero nibbles).  Returns
    ``(uint8 [B, R, Kp/2], float8_e4m3fn [B, R, Kp/16])``.
    """
    return _lib.native().quant(x, transpose, k_pad)


def rope_quant_nvfp4(x: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, positions=None, pos0: int = 0):
    """Rotary embedding fused into the NVFP4 packer (the producer the reference asks callers to
    fuse before `q_packs` / `k_packs`, flash.py:10-13, 2812-2821).

    ``x`` ``[B, R, D]`` (row r at position ``positions[r]`` or ``pos0 + r``), ``cos`` / ``sin``
    ``[P, D/2]`` fp32, half-split ("rotate_half") convention.  The rotated values are rounded once to
    ``x.dtype`` and packed along D: bit-identical to ``_quant_nvfp4(rope(x).to(x.dtype))`` with the
    rotation in fp32, without writing the rotated tensor.  Returns ``(uint8 [B,R,D/2],
    float8_e4m3fn [B,R,D/16])``, directly usable as ``q_packs`` / ``k_packs``.
    """
    return _lib.native().rope_quant(x, cos, sin, positions, pos0)


def _quant_mxfp8_t(x: torch.Tensor, s_pad: int, _prescale_amax: torch.Tensor | None = None):
    """MXFP8 pack of ``x`` [B, S, D] along S: e4m3 bytes [B, D, s_pad] and e8m0 scale bytes
    [B, D, s_pad/32] (one power-of-two scale per 32 tokens); stands in for ``_pack_mxfp8_along_k`` of
    the transposed operand (flash.py:243-257, 1255-1394).  The gradient operands dO^T, Q^T, K^T of the
    ``fp8_rownorm`` backward."""
    return _lib.native().quant_mxfp8_t(x, s_pad, _prescale_amax)


def vproj_quant_nvfp4(x: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor | None, num_kv_heads: int,
                      head_dim: int, s_pad: int | None = None, return_value: bool = True):
    """V projection with the NVFP4 pack as its epilogue (the producer the reference asks callers to
    fuse for V, flash.py:10-13, 2812-2821): ``V = x @ weight.T (+ bias)`` on the tensor cores, written
    directly as the V^T pack along the keys, so V is never re-read for quantisation.

    ``x`` ``[Z, S, hidden]`` and ``weight`` ``[Hk*D, hidden]`` in bf16 or fp16.  Returns ``(vnv uint8
    [Z*Hk, D, s_pad/2], vsc float8_e4m3fn [Z*Hk, D, s_pad/16], value)`` where ``value`` is the
    projected tensor as a ``[Z, Hk, S, D]`` view (``None`` with ``return_value=False``); the packs are
    bit-identical to ``_quant_nvfp4(value, transpose=True, k_pad=s_pad)`` and feed
    ``nvfp4_flash_attention_packed`` / ``nvfp4_flash_decode_prequant`` as they are.
    """
    return _lib.native().vproj_quant(x, weight, bias, num_kv_heads, head_dim, s_pad, return_value)


def _quant_nvfp4_dual(x: torch.Tensor, s_pad: int | None = None, _prescale_amax: torch.Tensor | None = None,
                      _sr: tuple = (False, False), _seed: int = 0):
    """Both layouts of ``x`` [B, S, D] from one read: along D and along S (padded to ``s_pad``).

    Stands in for flash.py:514-561 (one kernel, one pass over ``x``); bytes equal two
    ``_quant_nvfp4`` calls.  Returns ``(nib_d, sc_d, nib_s, sc_s)``.  ``_prescale_amax`` (a device
    float holding max|x|) first divides ``x`` by the smallest power of two >= that value (the global
    normalisation of dO in the all-FP4 backward).  ``_sr`` = (along D, along S): round that pack's
    e2m1 codes stochastically from ``_seed`` (the dO packs of the ``fp4_legacy`` backward).
    """
    return _lib.native().quant_dual(x, s_pad, _prescale_amax, _sr[0], _sr[1], int(_seed))


def _quant_qkv_fwd(q2, k2, v2, s_kv_pad):
    """Q, K along D and V along keys (padded to ``s_kv_pad``) in one launch; stands in for
    flash.py:682-732.  ``q2`` [ZH, Sq, D], ``k2`` / ``v2`` [ZHk, Skv, D].  Operands that are not
    unit-stride along D (or differ in dtype) fall back to one ``_quant_nvfp4`` launch each."""
    return _lib.native().quant_qkv(q2, k2, v2, s_kv_pad)


def convert_fp32_to_fp4_packed(x_pairs):
    """Pairs of fp32 tensors -> one byte per pair (first in the low nibble), e2m1 RTNE.

    The reference exposes this as a Triton device function (_fp4_pack.py:15-56); here it is a
    host-callable helper over the same hardware convert: values are packed with unit scale.
    """
    lo, hi = x_pairs
    x = torch.stack([lo.float(), hi.float()], dim=-1).reshape(1, -1, 2)
    n = x.shape[1]
    # unit scale: pad every pair to a group whose amax is exactly 6 so the group scale is 1
    grp = torch.zeros(1, n, 16, dtype=torch.float32, device=x.device)
    grp[:, :, 0:2] = x.clamp(-6.0, 6.0)
    grp[:, :, 2] = 6.0
    nib, _ = _quant_nvfp4(grp)
    return nib[0, :, 0].reshape(lo.shape)


# --------------------------------------------------------------------------- varlen
def _varlen_seq_arrays(cu_seqlens: torch.Tensor, s: int, device):
    """``cu_seqlens`` [n+1] -> int32 ``[s]`` arrays (seq_id, seq_start, seq_end) on ``device``.

    Same contract and validation messages as flash.py:940-984, including the cache on the
    tensor keyed by (s, device, version) so one host copy serves every layer of a step.
    """
    assert cu_seqlens.ndim == 1 and cu_seqlens.numel() >= 2, (
        f"cu_seqlens must be a 1-D [nseq+1] tensor, got shape {tuple(cu_seqlens.shape)}")
    key = (int(s), str(device), cu_seqlens._version)
    cached = getattr(cu_seqlens, "_nvfp4_seq_arrays", None)
    if cached is not None and cached[0] == key:
        return cached[1]
    cu = cu_seqlens.detach().to("cpu", torch.int64)
    assert int(cu[0]) == 0, f"cu_seqlens[0] must be 0, got {int(cu[0])}"
    assert int(cu[-1]) == s, f"cu_seqlens[-1] ({int(cu[-1])}) must equal the packed seqlen ({s})"
    assert bool((cu[1:] >= cu[:-1]).all()), "cu_seqlens must be nondecreasing"
    lens = (cu[1:] - cu[:-1])
    ids = torch.repeat_interleave(torch.arange(lens.numel(), dtype=torch.int64), lens)
    seq_id = ids.to(torch.int32)
    seq_start = cu[ids].to(torch.int32)
    seq_end = cu[ids + 1].to(torch.int32)
    arrays = tuple(t.to(device).contiguous() for t in (seq_id, seq_start, seq_end))
    try:
        cu_seqlens._nvfp4_seq_arrays = (key, arrays)
    except (AttributeError, RuntimeError):
        pass
    return arrays


# --------------------------------------------------------------------------- decode
def nvfp4_quant_kv_decode(key: torch.Tensor, value: torch.Tensor, block_n: int = 128) -> tuple:
    """One-shot NVFP4 pack of a GQA KV cache (stands in for flash.py:3211-3241).

    ``key``/``value``: ``[Z, Hk, Skv, D]``.  Returns ``(knv, ksc, vnv, vsc, s_kv, s_kv_pad)`` with K
    packed along D and V packed along keys as V^T, the key axis padded to ``block_n``.
    """
    z, hk, s_kv, d = key.shape
    assert d % 16 == 0 and d in (128, 256)
    s_kv_pad = _next_mult(s_kv, block_n)
    knv, ksc = _quant_nvfp4(key.reshape(z * hk, s_kv, d))
    vnv, vsc = _quant_nvfp4(value.reshape(z * hk, s_kv, d), transpose=True, k_pad=s_kv_pad)
    return knv, ksc, vnv, vsc, s_kv, s_kv_pad


@functools.lru_cache(maxsize=64)
def _sm_count_cached(index: int) -> int:
    return torch.cuda.get_device_properties(index).multi_processor_count


def _sm_count(device) -> int:
    dev = device if isinstance(device, torch.device) else torch.device(device)
    return _sm_count_cached(torch.cuda.current_device() if dev.index is None else dev.index)


@functools.lru_cache(maxsize=4096)
def _decode_plan_cached(s_kv: int, zhk: int, d: int, sms: int):
    ns, sk, wb = ctypes.c_int(), ctypes.c_int64(), ctypes.c_size_t()
    _lib.check(_lib.lib().nvfp4_decode_plan(s_kv, zhk, d, sms, ctypes.byref(ns), ctypes.byref(sk), ctypes.byref(wb)),
               "nvfp4_decode_plan")   # host only
    return ns.value, sk.value, wb.value


def _decode_plan(s_kv: int, zhk: int, d: int, device):
    return _decode_plan_cached(int(s_kv), int(zhk), int(d), _sm_count(device))


def _decode_core(query, kv_packed, scaling, g, want_lse, split_kv=None):
    """Shared body of the decode entry points; ``split_kv`` forces the decomposition (keys per split,
    0 = the balanced one) instead of the planned one.  Returns ``(out, lse | None)``."""
    knv, ksc, vnv, vsc, s_kv, _ = kv_packed
    return _lib.native().decode(query, knv, ksc, vnv, vsc, s_kv, scaling, g, want_lse, split_kv)


def nvfp4_flash_decode_prequant(query, kv_packed, scaling, num_key_value_groups=1, block_n=128,
                                num_warps=4, num_stages=3, target_programs=256):
    """Decode one query token per head against a pre-packed NVFP4 cache (HBM-bound fast path).

    Stands in for flash.py:3296-3342.  ``query`` ``[Z, H, 1, D]``; ``kv_packed`` is the tuple from
    ``nvfp4_quant_kv_decode`` or ``NVFP4KVCache.get_packed()`` (strided views are read in place).
    The split count follows the device's SM count; ``target_programs`` is accepted and ignored.
    Returns ``[Z, H, 1, D]`` in ``query.dtype``.
    """
    assert block_n == 128, "the B200 decode kernel walks 128-key tiles"
    return _decode_core(query, kv_packed, scaling, num_key_value_groups, False)[0]


def _decode_prequant_with_lse(query, kv_packed, scaling, g, block_n=128, num_warps=4,
                              num_stages=3, target_programs=256):
    """Decode that also returns the per-head log-sum-exp (kv_cache.py:32-97): ``(out, lse[Z,H])``."""
    return _decode_core(query, kv_packed, scaling, g, want_lse=True)


def nvfp4_flash_decode(query, key, value, scaling, num_key_value_groups=1, block_n=128,
                       num_warps=4, num_stages=3, target_programs=256):
    """Convenience decode that packs K/V from high precision on every call (flash.py:3345-3400)."""
    z, h, s_q, d = query.shape
    _, hk, s_kv, _ = key.shape
    assert s_q == 1, "nvfp4_flash_decode is for seqlen_q == 1 (decode)"
    assert h % hk == 0 and h // hk == num_key_value_groups
    assert d % 16 == 0 and d in (128, 256)
    assert num_key_value_groups <= 16, f"GQA group {num_key_value_groups} must be <= 16"
    packed = nvfp4_quant_kv_decode(key, value, block_n)
    return nvfp4_flash_decode_prequant(query, packed, scaling, num_key_value_groups, block_n)


# --------------------------------------------------------------------------- forward
def _run_flash_packed(qnv, qsc, knv, ksc, vnv, vsc, z, h, hk, s_q, s_kv, d, scaling, out_dtype,
                      causal=False, key_pad_bias=None, cu_seqlens=None, block_m=64, block_n=128,
                      num_warps=8, num_stages=3, out_layout="zhsd", return_lse=False,
                      _varlen_arrays=None):
    """Launch the forward kernel over packed operands (stands in for flash.py:2560-2652)."""
    if out_layout not in ("zhsd", "zshd"):
        raise ValueError(f"out_layout must be 'zhsd' or 'zshd', got {out_layout!r}")
    seq_id = seq_start = None
    if cu_seqlens is not None or _varlen_arrays is not None:
        assert z == 1, "cu_seqlens varlen requires Z must be 1 (one packed row)"
        assert s_q == s_kv, "cu_seqlens varlen requires Sq == Skv"
        arrays = _varlen_arrays if _varlen_arrays is not None else _varlen_seq_arrays(cu_seqlens, s_q, qnv.device)
        seq_id, seq_start = arrays[0], arrays[1]
    out, lse = _lib.native().flash_packed(qnv, qsc, knv, ksc, vnv, vsc, z, h, hk, s_q, s_kv, d, scaling, out_dtype, causal,
                                          key_pad_bias, seq_id, seq_start, out_layout == "zshd", return_lse)
    return (out, lse) if return_lse else out


def nvfp4_flash_attention_packed(qnv, qsc, knv, ksc, vnv, vsc, z, h, hk, s_q, s_kv, d, scaling,
                                 out_dtype, causal=False, key_pad_bias=None, cu_seqlens=None,
                                 block_m=64, block_n=128, num_warps=8, num_stages=3,
                                 out_layout="zhsd", _varlen_arrays=None):
    """Forward over operands the caller already packed (stands in for flash.py:2655-2766)."""
    return _run_flash_packed(qnv, qsc, knv, ksc, vnv, vsc, z, h, hk, s_q, s_kv, d, scaling,
                             out_dtype, causal, key_pad_bias, cu_seqlens, block_m, block_n,
                             num_warps, num_stages, out_layout, False, _varlen_arrays)


def nvfp4_flash_attention(query, key, value, scaling, causal=False, num_key_value_groups=1,
                          key_pad_bias=None, cu_seqlens=None, block_m=64, block_n=128, num_warps=8,
                          num_stages=3, return_lse=False, return_packs=False, out_layout="zhsd",
                          q_packs=None, k_packs=None, _varlen_arrays=None):
    """NVFP4 flash-attention forward (no autograd); stands in for flash.py:2769-3015.

    ``query`` ``[Z, H, Sq, D]``, ``key``/``value`` ``[Z, Hk, Skv, D]`` (bf16 / fp16 / fp32),
    ``D`` in {128, 256}.  Q and K are packed along D, V along keys, then the block-scaled FP4
    kernel runs.  Causal masking is bottom-right aligned.  Return arity follows the two flags
    exactly as in the reference: ``out`` | ``(out, lse)`` | ``(out, packs)`` |
    ``(out, lse, packs)`` with ``packs = (qnv, qsc, knv, ksc, vnv, vsc)``.
    """
    if out_layout not in ("zhsd", "zshd"):
        raise ValueError(f"out_layout must be 'zhsd' or 'zshd', got {out_layout!r}")
    seq_id = seq_start = None
    if cu_seqlens is not None or _varlen_arrays is not None:
        s_q = query.shape[2]
        if cu_seqlens is not None:
            assert query.shape[0] == 1, "cu_seqlens varlen requires Z must be 1 (one packed row)"
            assert s_q == key.shape[2], "cu_seqlens varlen requires Sq == Skv"
            assert causal, "cu_seqlens varlen is block-diagonal causal: pass causal=True"
        arrays = _varlen_arrays if _varlen_arrays is not None else _varlen_seq_arrays(cu_seqlens, s_q, query.device)
        seq_id, seq_start = arrays[0], arrays[1]
    qnv, qsc = q_packs if q_packs is not None else (None, None)
    knv, ksc = k_packs if k_packs is not None else (None, None)
    out, lse, packs = _lib.native().flash_attention(
        query, key, value, scaling, causal, num_key_value_groups, key_pad_bias, cu_seqlens is not None, seq_id, seq_start,
        out_layout == "zshd", return_lse, return_packs, qnv, qsc, knv, ksc)
    if return_packs:
        return (out, lse, tuple(packs)) if return_lse else (out, tuple(packs))
    return (out, lse) if return_lse else out


# --------------------------------------------------------------------------- backward
def _bwd_prep(x, y=None, want_copy=False, want_amax=False):
    """C-ABI pre-pass on a ``[B1, B2, S, D]`` tensor with unit stride along D (any other strides):
    returns ``(xc [B1*B2, S, D] bf16 | None, delta [B1*B2, S] = rowsum(x*y) | None)``, and with
    ``want_amax`` a third element: a device float holding max|x|."""
    xc, delta, amax = _lib.native().bwd_prep(x, y, want_copy, want_amax)
    return (xc, delta, amax) if want_amax else (xc, delta)


def _as_bf16_rows(x):
    """``[B1, B2, S, D]`` -> contiguous bf16 ``[B1*B2, S, D]``; no copy when it already is one."""
    return _lib.native().bf16_rows(x)


def _run_bwd_hp(q, k, v, out, lse, dout, scaling, causal, g, varlen_arrays=None, out_layout="zhsd",
                q_packs=None, k_packs=None, key_pad_bias=None):
    """High-precision-grad-dots backward (stands in for flash.py:3459-3805).

    ``q`` ``[Z,H,Sq,D]``, ``k``/``v`` ``[Z,Hk,Skv,D]`` (v may be a strided view), ``out``/``dout`` in
    ``out_layout``, ``lse`` ``[Z*H, Sq]``.  Returns ``(dq, dk, dv)`` shaped like q, k, v in
    ``dout.dtype``.  One pre-pass launch for delta (plus a bf16 copy per operand that is not already
    contiguous bf16), then the dK/dV kernel (GQA reduced in-kernel) and the dQ kernel.
    """
    qnv, qsc = q_packs if q_packs is not None else (None, None)
    knv, ksc = k_packs if k_packs is not None else (None, None)
    seq_start, seq_end = (varlen_arrays[1], varlen_arrays[2]) if varlen_arrays is not None else (None, None)
    return _lib.native().bwd_hp(q, k, v, out, lse, dout, scaling, causal, seq_start, seq_end, out_layout == "zshd", qnv, qsc,
                                knv, ksc, key_pad_bias)


def _run_bwd(q, k, v, out, lse, dout, scaling, causal, g, varlen_arrays=None, out_layout="zhsd",
             mode="fp4_rownorm", q_packs=None, k_packs=None, key_pad_bias=None, sr=False, sr_p_dv=None,
             sr_dot_dv=None, sr_ds_dq=None, seed=None, qt_packs=None, kt_packs=None, vd_packs=None, **_unused):
    """Block-scaled backward for the ``fp4_rownorm`` / ``fp4_legacy`` / ``fp8_rownorm`` modes (stands
    in for flash.py:3811-4265): every GEMM of the backward is a block-scaled tensor-core product.

    Pre-pass (five launches and a zeroed word): delta = rowsum(dO o O) and max|dO|; dO / 2^e packed along D
    and along the tokens from one read; Q^T and K^T packed along the tokens; V packed along D.  Then the
    dK/dV kernel (GQA reduced in tensor memory; at D = 256 a dV and a dK kernel) and the dQ kernel.  In ``fp8_rownorm`` the operands
    of the three gradient GEMMs (dO^T, Q^T, K^T from the pre-pass; P^T, dS^T, dS packed in the
    kernels) are MXFP8 -- e4m3 with an e8m0 scale per 32 -- while S and dP stay NVFP4 products.

    Stochastic rounding (flash.py:3897-3915): only ``fp4_legacy`` honours the knobs; ``sr`` rounds
    the dO pack along D and the dS^T pack stochastically, ``sr_p_dv`` / ``sr_dot_dv`` / ``sr_ds_dq``
    (default: ``sr``) the P^T pack, the dO^T pack and the dS pack of the dQ kernel.  ``seed`` is drawn
    on the host when not given.

    ``qt_packs`` / ``kt_packs`` / ``vd_packs``: the transposed packs of Q and K (padded to 128
    tokens) and the along-D pack of V saved by the forward under ``save_backward_packs``; given,
    the pre-pass skips those launches (and the re-read of Q, K and V).
    """
    if mode != "fp4_legacy":         # the normalised modes round to nearest only
        sr = sr_p_dv = sr_dot_dv = sr_ds_dq = False
    sr = bool(sr)
    sr_p_dv = sr if sr_p_dv is None else bool(sr_p_dv)
    sr_dot_dv = sr if sr_dot_dv is None else bool(sr_dot_dv)
    sr_ds_dq = sr if sr_ds_dq is None else bool(sr_ds_dq)
    if seed is None:
        any_sr = sr or sr_p_dv or sr_dot_dv or sr_ds_dq
        seed = int(torch.randint(0, 2 ** 31 - 1, (1,), device="cpu").item()) if any_sr else 0
    two = lambda t: t if t is not None else (None, None)
    seq_start, seq_end = (varlen_arrays[1], varlen_arrays[2]) if varlen_arrays is not None else (None, None)
    return _lib.native().bwd_fp4(q, k, v, out, lse, dout, scaling, causal, seq_start, seq_end, out_layout == "zshd",
                                 mode == "fp8_rownorm", *two(q_packs), *two(k_packs), *two(qt_packs), *two(kt_packs),
                                 *two(vd_packs), key_pad_bias, sr, sr_p_dv, sr_dot_dv, sr_ds_dq, int(seed))


def _gqa_reduce_cast_dkdv(dk_planes: torch.Tensor, dv_planes: torch.Tensor, z: int, hk: int, g: int,
                          out_dtype=None):
    """Sum per-query-head dK/dV planes ``[Z*H, S, D]`` over each GQA group -> ``[Z, Hk, S, D]``.

    Kept for API parity with flash.py:2525-2557; the B200 kernels reduce inside the dK/dV kernel
    and never materialise the planes."""
    zh, s, d = dk_planes.shape
    dt = out_dtype or dk_planes.dtype
    dk = dk_planes.reshape(z, hk, g, s, d).float().sum(dim=2).to(dt)
    dv = dv_planes.reshape(z, hk, g, s, d).float().sum(dim=2).to(dt)
    return dk, dv


class _NVFP4FlashAttn(torch.autograd.Function):
    """Autograd wrapper of the NVFP4 attention (stands in for flash.py:4268-4545).

    ``apply`` takes the reference's 26 positional arguments in the same order (query, key, value,
    scaling, causal, num_key_value_groups, key_pad_bias, sr, save_backward_packs, the three
    backward stochastic-rounding knobs, dkdv_scratch_bf16, backward_grad_dots (resolved mode),
    out_zshd, four tile hints, seq_id / seq_start / seq_end, and the optional Q / K packs) and
    returns gradients for the first three.
    """

    @staticmethod
    def forward(ctx, query, key, value, scaling, causal, num_key_value_groups, key_pad_bias, sr,
                save_backward_packs, backward_p_dv_sr, backward_dot_dv_sr, backward_ds_dq_sr,
                dkdv_scratch_bf16, backward_grad_dots, out_zshd, block_m, block_n, num_warps, num_stages,
                seq_id, seq_start, seq_end, qnv_in, qsc_in, knv_in, ksc_in):
        varlen = (seq_id, seq_start, seq_end) if seq_id is not None else None
        if varlen is not None:
            assert not save_backward_packs, "varlen (cu_seqlens) is incompatible with save_backward_packs"
        # direct callers of the Function may pass None (AUTO on s_kv) or a raw mode
        backward_grad_dots = _resolve_backward_grad_dots(backward_grad_dots, key.shape[2], save_backward_packs,
                                                         num_key_value_groups)
        if backward_grad_dots == "fp8_rownorm":
            assert not save_backward_packs, (
                "backward_grad_dots='fp8_rownorm' is incompatible with the saved forward FP4 "
                "transposed packs (save_backward_packs)")
        if qnv_in is not None or knv_in is not None:
            assert not save_backward_packs, (
                "q_packs/k_packs are incompatible with save_backward_packs "
                "(the saved pack set must come from the same fused HP read)")
        out_layout = "zshd" if out_zshd else "zhsd"
        q_in = (qnv_in, qsc_in) if qnv_in is not None else None
        k_in = (knv_in, ksc_in) if knv_in is not None else None
        extra = ()
        if save_backward_packs and backward_grad_dots in ("fp4_rownorm", "fp4_legacy"):
            # flash.py:4330-4385: everything the all-FP4 backward needs of Q, K and V is packed here,
            # from the one read of each operand (along D for the forward, transposed for the backward)
            z, h, s_q, d = query.shape
            hk, s_kv = key.shape[1], key.shape[2]
            qd = _quant_nvfp4_dual(query.reshape(z * h, s_q, d), _next_mult(s_q, _KEY_TILE))
            kd = _quant_nvfp4_dual(key.reshape(z * hk, s_kv, d), _next_mult(s_kv, _KEY_TILE))
            q_in, k_in = (qd[0], qd[1]), (kd[0], kd[1])
            extra = (qd[2], qd[3], kd[2], kd[3], *_quant_nvfp4(value.reshape(z * hk, s_kv, d)))
        out, lse, packs = nvfp4_flash_attention(
            query, key, value, scaling, causal=causal, num_key_value_groups=num_key_value_groups,
            key_pad_bias=key_pad_bias, return_lse=True, return_packs=True, out_layout=out_layout,
            q_packs=q_in, k_packs=k_in, _varlen_arrays=varlen)
        ctx.save_for_backward(query, key, value, out, lse, packs[0], packs[1], packs[2], packs[3], key_pad_bias, *extra)
        ctx.meta = (float(scaling), bool(causal), int(num_key_value_groups), varlen, out_layout,
                    backward_grad_dots, (bool(sr), backward_p_dv_sr, backward_dot_dv_sr, backward_ds_dq_sr))
        return out

    @staticmethod
    def backward(ctx, grad_out):
        query, key, value, out, lse, qnv, qsc, knv, ksc, bias, *extra = ctx.saved_tensors
        scaling, causal, g, varlen, out_layout, mode, srk = ctx.meta
        if mode == "bf16":
            grads = _run_bwd_hp(query, key, value, out, lse, grad_out, scaling, causal, g, varlen,
                                     out_layout, q_packs=(qnv, qsc), k_packs=(knv, ksc), key_pad_bias=bias)
        else:
            grads = _run_bwd(query, key, value, out, lse, grad_out, scaling, causal, g, varlen,
                                  out_layout, mode=mode, q_packs=(qnv, qsc), k_packs=(knv, ksc),
                                  key_pad_bias=bias, sr=srk[0], sr_p_dv=srk[1], sr_dot_dv=srk[2],
                                  sr_ds_dq=srk[3], qt_packs=tuple(extra[0:2]) if extra else None,
                                  kt_packs=tuple(extra[2:4]) if extra else None,
                                  vd_packs=tuple(extra[4:6]) if extra else None)
        return (*grads,) + (None,) * 23


def _attention_backward(query, key, value, out, lse, grad_out, scaling, causal, g, seq_id, seq_start, seq_end, zshd, mode,
                        qnv, qsc, knv, ksc, bias, sr, sr_p_dv, sr_dot_dv, sr_ds_dq):
    """Block-scaled modes of the native graph node of ``nvfp4_flash_attn_func``: ``(dq, dk, dv)``.  (The node runs
    the "bf16" mode without coming here.)"""
    varlen = (seq_id, seq_start, seq_end) if seq_id is not None else None
    layout = "zshd" if zshd else "zhsd"
    return _run_bwd(query, key, value, out, lse, grad_out, scaling, causal, g, varlen, layout, mode=mode, q_packs=(qnv, qsc),
                    k_packs=(knv, ksc), key_pad_bias=bias, sr=sr, sr_p_dv=sr_p_dv, sr_dot_dv=sr_dot_dv, sr_ds_dq=sr_ds_dq)


def nvfp4_flash_attn_func(query, key, value, scaling, causal=False, num_key_value_groups=1,
                          key_pad_bias=None, cu_seqlens=None, stochastic_rounding=True,
                          save_backward_packs=False, backward_p_dv_stochastic_rounding=None,
                          backward_dot_dv_stochastic_rounding=None,
                          backward_ds_dq_stochastic_rounding=None, dkdv_scratch_bf16=None,
                          backward_grad_dots=None, backward_bf16_grad_dots=None, out_layout="zhsd",
                          block_m=64, block_n=128, num_warps=8, num_stages=3, q_packs=None, k_packs=None):
    """Differentiable NVFP4 flash attention (training entry; stands in for flash.py:4548-4703).

    Same signature as the reference.  ``backward_grad_dots`` in {None (auto), "bf16",
    "fp4_rownorm", "fp8_rownorm", "fp4_legacy"}; ``backward_bf16_grad_dots`` is the legacy boolean
    spelling of "bf16" (not both).  The stochastic-rounding knobs act on the "fp4_legacy" backward
    only (as in the reference, the normalised modes round to nearest); tile hints are accepted and
    ignored.
    """
    z, h, s_q, d = query.shape
    hk, s_kv = key.shape[1], key.shape[2]
    assert h % hk == 0 and h // hk == num_key_value_groups, "H must equal Hk * num_key_value_groups"
    assert d in (128, 256), "head dim must be 128 or 256"
    if out_layout not in ("zhsd", "zshd"):
        raise ValueError(f"out_layout must be 'zhsd' or 'zshd', got {out_layout!r}")
    if backward_bf16_grad_dots is not None:
        assert backward_grad_dots is None, (
            "pass either backward_grad_dots or the deprecated backward_bf16_grad_dots, not both")
        backward_grad_dots = "bf16" if backward_bf16_grad_dots else "fp4_legacy"
    if backward_grad_dots is None:
        # AUTO on the effective sequence: s_kv, or the mean sample length of a packed row
        eff = s_kv if cu_seqlens is None else s_q / max(1, cu_seqlens.numel() - 1)
        backward_grad_dots = _resolve_backward_grad_dots(None, eff, save_backward_packs, num_key_value_groups)
    else:
        backward_grad_dots = _resolve_backward_grad_dots(backward_grad_dots, s_kv, save_backward_packs, num_key_value_groups)
    seq_id = seq_start = seq_end = None
    if cu_seqlens is not None:
        assert causal, "varlen (cu_seqlens) implements block-diagonal causal attention; pass causal=True"
        assert z == 1, f"varlen packs all samples into one flattened row: Z must be 1, got Z={z}"
        assert s_q == s_kv, f"varlen requires packed self-attention (Sq == Skv), got {s_q} vs {s_kv}"
        seq_id, seq_start, seq_end = _varlen_seq_arrays(cu_seqlens, s_q, query.device)
    if q_packs is not None or k_packs is not None:
        assert not save_backward_packs, (
            "q_packs/k_packs are incompatible with save_backward_packs "
            "(the saved pack set must come from the same fused HP read)")
    qnv_in, qsc_in = q_packs if q_packs is not None else (None, None)
    knv_in, ksc_in = k_packs if k_packs is not None else (None, None)
    if not save_backward_packs:
        optional = lambda x: None if x is None else bool(x)
        return _lib.native().attention(
            query, key, value, scaling, causal, num_key_value_groups, key_pad_bias, seq_id, seq_start, seq_end,
            out_layout == "zshd", qnv_in, qsc_in, knv_in, ksc_in, backward_grad_dots, bool(stochastic_rounding),
            optional(backward_p_dv_stochastic_rounding), optional(backward_dot_dv_stochastic_rounding),
            optional(backward_ds_dq_stochastic_rounding))
    return _NVFP4FlashAttn.apply(
        query, key, value, scaling, causal, num_key_value_groups, key_pad_bias, stochastic_rounding,
        save_backward_packs, backward_p_dv_stochastic_rounding, backward_dot_dv_stochastic_rounding,
        backward_ds_dq_stochastic_rounding, dkdv_scratch_bf16, backward_grad_dots, out_layout == "zshd", block_m,
        block_n, num_warps, num_stages, seq_id, seq_start, seq_end, qnv_in, qsc_in, knv_in, ksc_in)
