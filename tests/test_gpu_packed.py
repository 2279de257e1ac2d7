"""One launch over packed sequences (spa_attn_varlen_fwd / _bwd) against one call per sequence."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _table(lengths_q, lengths_k, gap=0):
    seqs, q0, k0 = [], 0, 0
    for n, m, off in zip(lengths_q, lengths_k, range(len(lengths_q))):
        seqs.append((q0, n, k0, m, (m - n) if off % 2 else 0))
        q0, k0 = q0 + n, k0 + m + gap
    return seqs, q0, k0


@pytest.mark.parametrize("lengths_q,lengths_k,gap", [
    ([1], [1], 0),
    ([128, 256, 129, 127], [128, 256, 129, 127], 0),
    ([300, 1, 515, 208], [300, 700, 600, 208], 5),
    ([1 + (37 * i) % 290 for i in range(40)], [1 + (53 * i) % 310 for i in range(40)], 0),   # two launches
])
@pytest.mark.parametrize("D,dtype,causal", [(128, torch.bfloat16, True), (64, torch.float16, False),
                                            (64, torch.bfloat16, True), (32, torch.float32, True)])
def test_packed_equals_one_call_per_sequence(lengths_q, lengths_k, gap, D, dtype, causal):
    """Bitwise: a sequence goes through the same tiles in the same order either way. Every other
    sequence holds Inf / NaN rows, which must stay in it."""
    import sp_aurora_b200 as spa
    from sp_aurora_b200 import local_attn as la
    Hq, Hkv = 4, 2
    seqs, Tq, Tk = _table(lengths_q, lengths_k, gap)
    g = torch.Generator(device="cuda").manual_seed(7)
    q, do = (torch.randn(Tq, Hq, D, device="cuda", generator=g).to(dtype) for _ in range(2))
    kv = torch.randn(Tk, 2, Hkv, D, device="cuda", generator=g).to(dtype)
    for i, (q0, n, k0, m, _) in enumerate(seqs):
        if i % 2:
            kv[k0] = float("inf")
            do[q0] = float("nan")
            q[q0, :, 1] = float("inf")
    k, v = kv[:, 0], kv[:, 1]
    scale = D ** -0.5
    out, lse = la.packed_forward(q, k, v, seqs, scale, causal)
    dq, dk, dv = la.packed_backward(do, q, k, v, out, lse, seqs, scale, causal)
    spa.check_status()
    used = torch.zeros(Tk, dtype=torch.bool)
    for i, (q0, n, k0, m, off) in enumerate(seqs):
        qs, ks = slice(q0, q0 + n), slice(k0, k0 + m)
        used[ks] = True
        o = torch.empty(1, n, Hq, D, device="cuda", dtype=dtype)
        l = torch.empty(1, Hq, n, device="cuda")
        la.attn_fwd_step(q[None, qs], k[None, ks], v[None, ks], scale, causal, l, out=o, causal_off=off)
        d = la.bwd_delta(o, do[None, qs].contiguous())
        gq = torch.empty_like(o)
        gk, gv = (torch.empty(1, m, Hkv, D, device="cuda", dtype=dtype) for _ in range(2))
        la.attn_bwd_step(q[None, qs], k[None, ks], v[None, ks], do[None, qs].contiguous(), l, d, scale, causal,
                         None, gk, gv, causal_off=off, dq=gq, dq_overwrite=True)
        for name, a, b in (("out", out[qs], o[0]), ("lse", lse[:, qs], l[0]), ("dq", dq[qs], gq[0]),
                           ("dk", dk[ks], gk[0]), ("dv", dv[ks], gv[0])):
            assert torch.equal(a.nan_to_num(1e4), b.nan_to_num(1e4)), (i, name)
            assert i % 2 or torch.isfinite(a[..., :]).all() or name == "lse", (i, name)
    assert (dk[~used] == 0).all() and (dv[~used] == 0).all()


def test_packed_table_is_validated():
    import sp_aurora_b200 as spa
    from sp_aurora_b200 import local_attn as la
    q = torch.randn(64, 2, 64, device="cuda", dtype=torch.float16)
    for bad in ([(0, 65, 0, 64, 0)], [(0, 32, 0, 32, 0), (31, 32, 32, 32, 0)], [(0, 32, 0, 0, 0)],
                [(0, 32, 32, 32, 0), (32, 32, 0, 32, 0)], [(-1, 8, 0, 8, 0)]):
        with pytest.raises(spa.SpaError):
            la.packed_forward(q, q, q, bad, 0.125, True)
