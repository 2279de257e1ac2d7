"""The forward's key split and head pairing (short blocks of queries over long contexts)."""
import ctypes as C

import pytest
import torch

from oracle import attention_oracle as orc

pytestmark = pytest.mark.gpu


def _args(q, k, v, out, lse, causal):
    from sp_aurora_b200 import _lib
    from sp_aurora_b200.local_attn import _fill_qkv
    a = _lib.FwdArgs()
    _fill_qkv(a, q, k, v)
    a.out, a.lse = out.data_ptr(), lse.data_ptr()
    a.o_sb, a.o_ss, a.o_sh = out.stride()[:3]
    a.B, a.Sq, a.Hq, a.D = q.shape
    a.Sk, a.Hkv, a.dtype, a.causal = k.shape[1], k.shape[2], _lib.DTYPE_CODE[q.dtype], int(causal)
    a.scale = q.shape[-1] ** -0.5
    return a


def _needed(q, k, v, causal):
    """Workspace bytes the planner asks for."""
    from sp_aurora_b200 import _lib
    return _lib.lib.spa_attn_fwd_workspace(C.byref(_args(q, k, v, q, q, causal)))


@pytest.mark.parametrize("B,Sq,Sk,Hq,Hkv,D,dtype,causal,split", [
    # one query tile per CTA (a CTA per tile fits the chip)
    (1, 1, 2049, 4, 2, 128, torch.bfloat16, False, True),       # one row, a ragged last key tile
    (2, 128, 4096, 8, 2, 128, torch.bfloat16, False, True),
    (1, 129, 2500, 8, 8, 64, torch.float16, False, True),       # one row in the second query tile
    (1, 300, 3000, 4, 2, 64, torch.bfloat16, False, True),
    (1, 3000, 3000, 4, 2, 128, torch.bfloat16, True, True),     # two tiles per CTA; early slices of early rows are empty
    (1, 640, 640, 4, 2, 128, torch.float16, True, False),       # too few keys to split
    (3, 130, 900, 6, 2, 64, torch.float16, False, False),
    # odd tile counts: heads paired
    (3, 300, 2100, 16, 8, 64, torch.bfloat16, False, True),     # and the keys split
    (2, 100, 1500, 32, 8, 128, torch.float16, False, True),
    (16, 640, 640, 4, 2, 128, torch.bfloat16, True, False),
    (26, 300, 300, 6, 2, 64, torch.float16, False, False),      # odd group: no pairing
])
def test_short_grids_match_the_oracle(B, Sq, Sk, Hq, Hkv, D, dtype, causal, split):
    import sp_aurora_b200 as spa
    g = torch.Generator().manual_seed(11)
    q = torch.randn(B, Sq, Hq, D, generator=g).to(dtype)
    kv = torch.randn(B, Sk, 2, Hkv, D, generator=g).to(dtype)
    k, v = kv[:, :, 0], kv[:, :, 1]
    qc, kvc = q.cuda(), kv.cuda()
    kc, vc = kvc[:, :, 0], kvc[:, :, 1]
    assert (_needed(qc, kc, vc, causal) > 0) == split
    out, lse = spa.flash_attn_forward(qc, kc, vc, None, causal)
    spa.check_status()
    ro, rl = orc.attention_ref(q, k, v, None, causal)
    assert (out.cpu().double() - ro).abs().max() <= 2e-2
    assert (lse.cpu().double() - rl).abs().max() <= 1e-3
    assert (out.cpu().double() - ro).norm() <= (4e-3 if dtype == torch.bfloat16 else 6e-4) * ro.norm()


def test_split_keeps_nan_and_inf():
    """A NaN key reaches every row that sees it, whatever slice it is in; an infinite value too."""
    import sp_aurora_b200 as spa
    q = torch.randn(1, 64, 4, 64, device="cuda", dtype=torch.bfloat16)
    kv = torch.randn(1, 4000, 2, 2, 64, device="cuda", dtype=torch.bfloat16)
    kv[0, 3900, 0, 0] = float("nan")
    kv[0, 100, 1, 1, 5] = float("inf")
    k, v = kv[:, :, 0], kv[:, :, 1]
    assert _needed(q, k, v, False) > 0
    out, lse = spa.flash_attn_forward(q, k, v)
    spa.check_status()
    assert out[:, :, :2].isnan().all()
    assert torch.isposinf(out[:, :, 2:, 5]).all() and torch.isfinite(out[:, :, 2:, :5]).all()


def test_workspace_size_is_checked():
    """Too small: refused. None: the unsplit kernel. Each of the two rounds its probabilities (scaled
    by its own running maximum) and its output to 8 bits: 2 * (2^-9 + 2^-9) of the largest value."""
    from sp_aurora_b200 import _lib
    q = torch.randn(1, 64, 4, 64, device="cuda", dtype=torch.bfloat16)
    k = torch.randn(1, 4000, 2, 64, device="cuda", dtype=torch.bfloat16)
    out, lse, out2, lse2 = (torch.empty(s, device="cuda", dtype=t) for s, t in (
        (q.shape, q.dtype), ((1, 4, 64), torch.float32)) * 2)
    need = _needed(q, k, k, False)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    a, a2 = _args(q, k, k, out, lse, False), _args(q, k, k, out2, lse2, False)
    assert _lib.lib.spa_attn_fwd_ws(C.byref(a), ws.data_ptr(), need - 4) == -1
    assert _lib.lib.spa_attn_fwd_ws(C.byref(a), ws.data_ptr(), need) == 0
    assert _lib.lib.spa_attn_fwd(C.byref(a2)) == 0
    torch.cuda.synchronize()
    assert (lse - lse2).abs().max() < 1e-5
    assert (out.float() - out2.float()).abs().max() <= 2 ** -7 * out.float().abs().max()


@pytest.mark.parametrize("Sq,D,causal,off", [(300, 128, True, 40), (257, 64, False, 0), (640, 64, True, -200)])
def test_head_pairs_merge_into_a_running_result(Sq, D, causal, off):
    """A ring step's form (fp32 result and lse in and out) on grids whose CTAs take one query tile
    of two heads: bitwise the calls on one head, which has no partner (odd tile counts, 2 query
    heads per kv head, more tiles than SMs, so neither the split nor single tiles apply)."""
    import sp_aurora_b200 as spa
    from sp_aurora_b200 import local_attn as la
    B, Sk, Hq, Hkv = 25, 500, 4, 2
    g = torch.Generator(device="cuda").manual_seed(17)
    q = torch.randn(B, Sq, Hq, D, device="cuda", generator=g).bfloat16()
    k, v = (torch.randn(B, Sk, Hkv, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    acc0, lse0 = torch.randn(B, Sq, Hq, D, device="cuda"), torch.randn(B, Hq, Sq, device="cuda")

    def call(hq, hk):
        acc, lse = acc0[:, :, hq].clone(), lse0[:, hq].clone()
        out = torch.empty_like(q[:, :, hq])
        la.attn_fwd_step(q[:, :, hq], k[:, :, hk], v[:, :, hk], D ** -0.5, causal, lse, out=out, out_acc=acc,
                         merge_prev=True, causal_off=off)
        return acc, lse, out
    acc, lse, out = call(slice(0, Hq), slice(0, Hkv))
    for h in range(Hq):
        a, l, o = call(slice(h, h + 1), slice(h // 2, h // 2 + 1))
        assert torch.equal(acc[:, :, h:h + 1], a) and torch.equal(lse[:, h:h + 1], l), h
        assert torch.equal(out[:, :, h:h + 1], o), h
    spa.check_status()
