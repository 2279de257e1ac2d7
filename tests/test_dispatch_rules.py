"""Dispatch rules of the CUDA library against their definition (host code, no GPU needed)."""
import ctypes as C
import random

from sp_aurora_b200 import _lib


def _rule():
    fn = _lib.lib._ZN3spa8dq_loopsEPK12spa_bwd_argsPK7spa_seqi      # spa::dq_loops
    fn.restype, fn.argtypes = C.c_bool, [C.POINTER(_lib.BwdArgs), C.POINTER(_lib.Seq), C.c_int]
    return fn


def _walk(sq, sk, causal, off):
    """(query tiles, K/V tiles they go through) for tiles of 128 by 128."""
    blocks, n = -(-sq // 128), -(-sk // 128)
    seen = [min(n, max(0, (i * 128 + 127 + off) // 128 + 1)) if causal else n for i in range(blocks)]
    return blocks, sum(seen)


def test_dq_loops_follow_the_mean_walk():
    """Query tiles loop where there are 3 per SM and a walk takes 24.5 K/V tiles at most, counting
    the tiles that the mask and its offset leave."""
    rule, r, taken = _rule(), random.Random(3), [0, 0]
    for i in range(4000):
        n_seq = r.choice([0, 0, 1, 5])
        a = _lib.BwdArgs()
        a.B, a.Hq, a.D, a.causal = 1 if n_seq else r.choice([1, 2, 8]), r.choice([8, 32]), r.choice([64, 128]), r.random() < .7
        rows = [(r.randint(1, 9000), r.randint(1, 9000), r.choice([0, 0, -1, 1, -128, 128, r.randint(-9000, 9000)]))
                for _ in range(max(n_seq, 1))]
        a.Sq, a.Sk, a.causal_off = rows[0]
        seqs = (_lib.Seq * len(rows))(*((0, sq, 0, sk, off) for sq, sk, off in rows))
        walks = [_walk(sq, sk, a.causal, off) for sq, sk, off in rows]
        items, walk = (sum(w[j] for w in walks) for j in (0, 1))
        want = items * a.Hq * a.B >= 3 * 148 and 2 * walk <= 49 * items
        assert rule(C.byref(a), seqs, n_seq) == want, (rows, n_seq, a.causal, a.B, a.Hq)
        taken[want] += 1
    assert min(taken) > 500
    a.D = 32
    assert not rule(C.byref(a), seqs, n_seq)
