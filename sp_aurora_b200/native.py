"""One-rank attention through the C++ autograd node of `_native-*.so` (csrc/native_path.cpp).

Every function answers (out, lse), or None where the call has to go the general way: several
ranks, per-kernel timing, or arguments that the node does not take (the general way also words
the errors)."""
from __future__ import annotations

import ctypes as C
import importlib.util

import torch.distributed as dist

from . import _lib, build, local_attn


def _load(build_failure):
    """The node built for this torch. One that is older than its sources is taken only where there
    is no compiler to say whether it still fits: after a failed compilation it may read the
    argument blocks of include/spa.h differently from the library."""
    path = build.native_path()
    outdated = path.exists() and build_failure is not None and \
        not isinstance(build_failure, build.CannotBuild) and build._stale(path, build.NATIVE_DEPS)
    if not path.exists() or outdated:
        raise ImportError(f"{path} is {'older than its sources' if outdated else 'missing'}: build it with "
                          "`python sp_aurora_b200/build.py` (this package has no fallback path)" +
                          (f"\nlast build attempt:\n{build_failure}" if build_failure else ""))
    spec = importlib.util.spec_from_file_location(f"{__package__}._native", path)
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    return module


_native = _load(_lib.build_failure)
_native.set_api([C.cast(getattr(_lib.lib, name), C.c_void_p).value for name in (
    "spa_attn_fwd", "spa_attn_fwd_workspace", "spa_attn_fwd_ws", "spa_attn_bwd", "spa_attn_varlen_fwd",
    "spa_attn_varlen_bwd", "spa_bwd_delta", "spa_check_status", "spa_last_error", "spa_rope_rows")], _lib.SpaError)


def _general(group) -> bool:
    return local_attn.KERNEL_TIMERS is not None or (
        dist.is_available() and dist.is_initialized() and dist.get_world_size(group) != 1)


def _scale(s):
    return None if s is None else float(s)


def attention(q, k, v, softmax_scale, causal, deterministic=False, group=None):
    """q, k, v [B,S,H,D]."""
    if _general(group):
        return None
    return _native.attention(q, k, v, _scale(softmax_scale), bool(causal), bool(deterministic), False)


def attention_local(q, k, v, softmax_scale, causal):
    """The same on this rank alone, whatever the groups; lse is marked as non-differentiable."""
    if local_attn.KERNEL_TIMERS is not None:
        return None
    return _native.attention(q, k, v, _scale(softmax_scale), bool(causal), False, True)


def attention_kvpacked(q, kv, softmax_scale, causal, deterministic=False, group=None):
    """kv [B,S,2,H,D]; its gradient is written in that layout."""
    if _general(group):
        return None
    return _native.attention_kvpacked(q, kv, _scale(softmax_scale), bool(causal), bool(deterministic))


def attention_qkvpacked(qkv, softmax_scale, causal, deterministic=False, group=None):
    """qkv [B,S,3,H,D]; its gradient is written in that layout."""
    if _general(group):
        return None
    return _native.attention_qkvpacked(qkv, _scale(softmax_scale), bool(causal), bool(deterministic))


def attention_heads_packed(x, hq, hkv, cos, sin, causal, group=None):
    """x [B,S,hq+2*hkv,D]: q, k and v side by side, as one projection writes them; with cos and
    sin (see rope_tables) q and k are rotated, positions from 0. The gradient is written in
    that layout."""
    if _general(group):
        return None
    return _native.attention_heads_packed(x, hq, hkv, cos, sin, bool(causal))


def attention_packed(q, k, v, seqs, softmax_scale, causal, deterministic=False, group=None):
    """Packed sequences, q, k, v [tokens,H,D]; `seqs` as in local_attn.attn_fwd_step."""
    if _general(group):
        return None
    return _native.attention_packed(q, k, v, seqs, _scale(softmax_scale), bool(causal), bool(deterministic))
