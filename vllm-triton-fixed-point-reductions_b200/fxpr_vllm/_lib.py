"""``torch.ops.fxpr.*`` schemas and their CUDA implementations.

The six schema strings are those of ``fxpr_vllm/_lib.py:15-33`` in the
reference, so vLLM-side code written against the reference keeps working.
Implementations (``csrc/torch_ops.cpp``) are registered for the CUDA dispatch key
only (CPU tensors get the dispatcher's ``NotImplementedError``, as with the
reference) and hand raw pointers plus the current stream to the C ABI in
``libfxpr_b200.so``; this module keeps the selection knobs, the policies and the
functions around the operators that need no device code.

Three ops are additions with no counterpart in the reference:
``log_softmax_fxp`` (order-free sampler log-softmax), ``gemm_fxp_int`` and
``gemm_fxp_epilogue`` (integer accumulators out / back in, for the
tensor-parallel integer all-reduce).
"""
from __future__ import annotations

import contextlib
import threading

import torch

from . import _native as nat

_lib = torch.library.Library("fxpr", "DEF")

_lib.define("float_to_fixed(Tensor x, int int_bits, int fxp_frac_bits) -> Tensor")
_lib.define("fixed_to_float(Tensor x, int float_bits, int fxp_frac_bits) -> Tensor")
_lib.define("rms_norm_fxp(Tensor x, Tensor weight_fp32, float eps) -> Tensor")
_lib.define(
    "rms_norm_fxp_residual(Tensor x, Tensor(a!) residual, Tensor weight_fp32, "
    "float eps) -> Tensor"
)
_lib.define(
    "gemm_fxp(Tensor a, Tensor b, Tensor? bias, int fxp_int_bits, "
    "int fxp_frac_bits) -> Tensor"
)
_lib.define(
    "unified_attention_fxp(Tensor q, Tensor kv_cache, Tensor(a!) o, "
    "Tensor query_start_loc, Tensor seq_lens, Tensor block_table, "
    "int max_query_len, Tensor? alibi_slopes, bool is_causal, "
    "float? softmax_scale, int fxp_int_bits, int fxp_frac_bits, "
    "float logit_softcap, int window_size, int num_kv_splits) -> ()"
)
# additions
_lib.define("log_softmax_fxp(Tensor x, int fxp_frac_bits) -> Tensor")
_lib.define("rms_norm_fxp_from_int(Tensor acc, Tensor(a!) residual, Tensor weight, Tensor? bias, float eps, "
            "int gemm_frac_bits) -> Tensor")
_lib.define("gemm_fxp_int(Tensor a, Tensor b, int fxp_int_bits, int fxp_frac_bits) -> Tensor")
_lib.define(
    "gemm_fxp_epilogue(Tensor c_int, Tensor? bias, ScalarType out_dtype, "
    "int fxp_frac_bits) -> Tensor"
)

_INT_DTYPE = {16: torch.int16, 32: torch.int32, 64: torch.int64}


class _NativeOps:
    """``torch.ops.fxpr_b200``, loaded at the first use (which raises if the library is not built)."""

    def __getattr__(self, name):
        nat.load_ops()
        op = getattr(torch.ops.fxpr_b200, name)
        setattr(self, name, op)
        return op


_native_ops = _NativeOps()


def _report_missing_library() -> None:
    """CUDA implementations that raise nat.load_ops()'s error, which names the build command, instead of
    the dispatcher's "no kernel for CUDA".  Built after the import, the library's own take their place."""
    def stand_in(name):
        def op(*args):
            nat.load_ops()
            return getattr(torch.ops.fxpr, name)(*args)
        return op

    for name in ("float_to_fixed", "fixed_to_float", "rms_norm_fxp", "rms_norm_fxp_residual", "rms_norm_fxp_from_int",
                 "log_softmax_fxp", "gemm_fxp", "gemm_fxp_int", "gemm_fxp_epilogue", "unified_attention_fxp"):
        _lib.impl(name, stand_in(name), "CUDA")


class _KTileTable(dict):
    """The library's default K-tile (determinism granularity, gemm.py:26-30 of the reference) of each io
    dtype; tests read it the way the reference's test reads ``_BLOCK_K_BY_DTYPE``."""

    def __missing__(self, dtype):
        if dtype not in (torch.float16, torch.bfloat16, torch.float32):
            raise KeyError(dtype)
        self[dtype] = nat.load().fxpr_gemm_default_k_tile(nat.DTYPE_CODE[dtype])
        return self[dtype]


BLOCK_K_BY_DTYPE = _KTileTable()

if nat.load_ops(required=False) is None:
    _report_missing_library()
else:
    for _dt in (torch.float16, torch.bfloat16, torch.float32):
        BLOCK_K_BY_DTYPE[_dt]


@contextlib.contextmanager
def _on_device(t: torch.Tensor):
    """Make ``t``'s device current for the duration of a C call."""
    if t.device.index is not None and t.device.index != torch.cuda.current_device():
        with torch.cuda.device(t.device):
            yield
    else:
        yield


# --------------------------------------------------------------------------
# test / tuning overrides (the public schemas carry no such arguments)
# --------------------------------------------------------------------------

class _Overrides(threading.local):
    gemm_k_tile: int | None = None
    gemm_split_k: int | None = None
    gemm_portable: bool = False
    attn_portable: bool = False
    gemm_partials: bool = False
    gemm_flags: int = 0
    attn_flags: int = 0

    @property
    def last_partials(self) -> torch.Tensor:
        """fp32 K-tile partials of the last GEMM under ``gemm_partials`` (this thread)."""
        return _native_ops.last_partials()


_ovr = _Overrides()


def _push_overrides() -> None:
    o = _ovr
    nat.load_ops().fxpr_torch_set_overrides(
        -1 if o.gemm_k_tile is None else o.gemm_k_tile, -1 if o.gemm_split_k is None else o.gemm_split_k,
        o.gemm_portable, o.attn_portable, o.gemm_partials, o.gemm_flags, o.attn_flags)


class overrides:
    """Temporarily pin kernel-selection knobs (K-tile, split-K, portable route) in this thread."""

    def __init__(self, *, gemm_k_tile=None, gemm_split_k=None, gemm_portable=None,
                 attn_portable=None, gemm_partials=None, gemm_flags=None, attn_flags=None):
        self._set = {k: v for k, v in locals().items() if k != "self" and v is not None}
        self._old = []

    def __enter__(self):
        self._old.append({k: getattr(_ovr, k) for k in self._set})
        _ovr.__dict__.update(self._set)
        _push_overrides()
        return _ovr

    def __exit__(self, *exc):
        _ovr.__dict__.update(self._old.pop())
        _push_overrides()


def static_weights():
    """Inside this block every GEMM's ``b`` operand is a model weight: complete long before the
    launch and not written by any kernel in flight.  The decode-shape GEMM then requests its
    first weight tiles before it waits for the previous kernel of the stream
    (``FXPR_GEMM_WEIGHTS_STATIC``).  Results do not change."""
    return overrides(gemm_flags=_ovr.gemm_flags | nat.GEMM_WEIGHTS_STATIC)


# --------------------------------------------------------------------------
# decoder-layer element-wise steps (no reference counterpart: vLLM ops there)
# --------------------------------------------------------------------------

def rope_kv_write(qkv, cos, sin, positions, seq_ids, block_table, kv_cache, q_heads, kv_heads):
    """Split ``qkv`` [T, (q_heads + 2 kv_heads) * d], rotate Q and K, return Q [T, q_heads, d]
    and write K, V into the paged ``kv_cache`` (num_blocks, 2, page, kv_heads, d)."""
    return _native_ops.rope_kv_write(qkv, cos, sin, positions, seq_ids, block_table, kv_cache, q_heads, kv_heads)


def silu_mul(gate_up):
    """``silu(gate) * up`` of a fused [rows, 2 f] activation."""
    return _native_ops.silu_mul(gate_up, False)


def silu_mul_pairs(gate_up):
    """``silu(gate_up[:, 0::2]) * gate_up[:, 1::2]`` for an activation whose columns are
    (gate_j, up_j) pairs (the layout ``gemm_silu_mul`` keeps its weights in)."""
    return _native_ops.silu_mul(gate_up, True)


# --------------------------------------------------------------------------
# GEMM
# --------------------------------------------------------------------------

def _get_gemm_scratch(device: torch.device, nbytes: int) -> torch.Tensor:
    """The current stream's persistent zero-initialised split-K scratch, grown on demand (the
    kernel re-zeroes what it used; gemm.py:86-107 of the reference keeps one such buffer per device),
    and with it the one of the device's CUDA graphs: ``warmup_gemm`` sizes both before capture."""
    nat.load_ops()
    return _native_ops.gemm_scratch(_device_index(device), nbytes)


def gemm_scratch_policy_bytes(num_sms: int, int_bits: int = 64) -> int:
    """Largest scratch a split of the automatic policy (``pick_split_k``) can need,
    whatever M, N and K.  Splits that a cluster merges need none.  The others double only while
    ``tiles * split * 2 <= num_sms``, so at most ``num_sms`` integer partial tiles of 128 x 128 exist, and
    one more a split (16 at most) where the columns are padded to 256; rows padded to 256 can double
    that.  In front of them the fixed 256 KiB counter region."""
    planes = (num_sms + 16) * 128 * 256 * (8 if int_bits == 64 else 4)
    return 256 * 1024 + -(-planes // 256) * 256


def _device_index(device) -> int:
    idx = torch.device(device).index
    return idx if idx is not None else torch.cuda.current_device()


def _status_word(device: torch.device) -> torch.Tensor:
    """Per-device int32 the kernels set when a bounded device-side wait gives up."""
    nat.load_ops()
    return _native_ops.status_word(_device_index(device))


def check_device_status(device=None) -> None:
    """Synchronise and raise if any kernel reported a timed-out wait since the
    last check (not on the hot path: tests, benchmarks and debugging call it)."""
    nat.load_ops()
    for t in _native_ops.status_words():
        if device is not None and torch.device(device).index not in (None, t.device.index):
            continue
        v = int(t.item())
        if v != 0:
            t.zero_()
            nat.check(v, f"device status word on {t.device}")


def _sm_count(device: torch.device) -> int:
    return torch.cuda.get_device_properties(_device_index(device)).multi_processor_count


def pick_split_k(M: int, N: int, K: int, k_tile: int, int_bits: int, num_sms: int) -> int:
    """The GEMM's automatic K-split (host shapes only: every split gives the same bits, so this
    is a speed decision; the reference times it at warm-up instead, gemm.py:780-836)."""
    return nat.load().fxpr_pick_gemm_split_k(M, N, K, k_tile, int_bits, num_sms)


def interleave_gate_up(w_gate, w_up):
    """``(K, f)`` gate and up weights -> ``(K, 2f)`` with columns (gate_0, up_0, gate_1, ...)."""
    return torch.stack([w_gate, w_up], dim=2).reshape(w_gate.shape[0], -1).contiguous()


def gemm_silu_mul(a, b_pairs, int_bits, fxp_frac_bits):
    """``silu(a @ gate) * (a @ up)`` with the gate and up columns of ``b_pairs`` interleaved
    (``interleave_gate_up``).  For at most 64 rows the decode-shape GEMM combines the column pairs
    in its epilogue; otherwise the GEMM and ``silu_mul_pairs`` run one after the other.  Same bits
    either way (and as ``gemm_fxp`` + ``silu_mul`` on the plain layout)."""
    return _native_ops.gemm_silu_mul(a, b_pairs, int_bits, fxp_frac_bits)


def gemm_fxp_argmax(a, b, bias, int_bits, fxp_frac_bits, n_offset: int = 0):
    """``gemm_fxp`` for at most 64 rows that also returns, per row, the arg-max key of the
    outputs (``int64 [M]``, see ``argmax_from_keys``): greedy sampling straight from the lm_head
    GEMM, with no pass over the ``[M, vocab]`` logits.  Keys of vocab shards (``n_offset`` = first
    column of the shard) combine with ``combine_argmax_keys``.  Shapes the fused kernel does not
    take fall back to ``gemm_fxp`` + a key built from ``torch.max``: same result."""
    c, keys = _native_ops.gemm_argmax(a, b, bias, int_bits, fxp_frac_bits, int(n_offset))
    if keys.numel() != a.shape[0]:
        keys = argmax_keys_of(c, n_offset)
    return c, keys


def argmax_keys_of(logits, n_offset: int = 0):
    """The key ``fxpr_gemm_argmax`` leaves for each row of ``logits`` (16-bit io dtypes)."""
    v, idx = logits.max(dim=-1)                     # first maximal column, as torch.argmax
    bits = v.float().view(torch.int32).to(torch.int64) & 0xFFFFFFFF
    ordv = torch.where(bits >= 0x80000000, (~bits) & 0xFFFFFFFF, bits | 0x80000000)
    return ((ordv << 32) | (0xFFFFFFFF - (idx.to(torch.int64) + int(n_offset)))) ^ torch.iinfo(torch.int64).min ^ torch.iinfo(torch.int64).min


def combine_argmax_keys(keys_list):
    """Keys of several vocab shards -> keys of the whole row (unsigned 64-bit maximum)."""
    flip = torch.iinfo(torch.int64).min
    stacked = torch.stack([k ^ flip for k in keys_list], dim=0)     # signed order == unsigned order
    return stacked.max(dim=0).values ^ flip


def argmax_from_keys(keys):
    """Winning column per row: the largest output, the smallest column among equals."""
    return 0xFFFFFFFF - (keys & 0xFFFFFFFF)


def gemm_fxp_int_into(a, b, out, int_bits, fxp_frac_bits):
    """``gemm_fxp_int`` into a caller-owned accumulator tensor (for example a peer-mapped
    buffer that other ranks read)."""
    _native_ops.gemm_fxp_int_into(a, b, out, int_bits, fxp_frac_bits)
    return out


# --------------------------------------------------------------------------
# attention
# --------------------------------------------------------------------------

def pick_num_splits(requested, num_requests, num_q_blocks, num_heads, num_kv_tiles, num_sms):
    """attention.py:664-689 of the reference: an explicit request wins; otherwise
    split only long contexts on an under-filled GPU, power of two, at most 8."""
    return nat.load().fxpr_pick_attention_splits(requested, num_requests, num_q_blocks, num_heads, num_kv_tiles,
                                                 num_sms)


def pick_num_splits_b200(requested, num_requests, max_query_len, num_heads, num_kv_heads,
                         max_keys, num_sms):
    """Split policy of the tensor-core route, where splits are cluster ranks: results do
    not depend on it, so it only balances the GPU.  Host shapes only, so it is fixed under a
    CUDA graph."""
    return nat.load().fxpr_pick_attention_ranks(requested, num_requests, max_query_len, num_heads, num_kv_heads,
                                                max_keys, num_sms)
