"""The packed 16-bit SSW kernel against the oracle's ssw.c restatement (scores, spans,
CIGARs; integers, so for equality) where it can go wrong: query lengths on both sides of
every piece and row count (multiples of 8 and 16, up to the 511 it takes and beyond), with
few tasks (eight threads each) and many (four threads each), mixed lengths in one warp,
windows shorter than the query and of rescue size, Ns and lower case, blocks replaced by an
insertion next to a deletion (which the library's E can miss in one direction only), and
scores at the limits of its rule and outside it."""
import numpy as np
import pytest

from oracle_lib import aligner_oracle

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", np.uint8)


def _pair(rng, L, kind):
    pad = int(rng.integers(0, 60)) if kind % 4 else int(rng.integers(200, 600))
    w = ACGT[rng.integers(0, 4, L + 2 * pad + 12)]
    o = int(rng.integers(0, 2 * pad + 8)) if pad else 0
    q = w[o:o + L].copy()
    sub = rng.random(L) < (0.01, 0.05, 0.2)[kind % 3]
    q[sub] = ACGT[rng.integers(0, 4, int(sub.sum()))]
    if kind % 5 == 1 and L > 12:
        # one indel
        c, d = int(rng.integers(4, L - 4)), int(rng.integers(1, 5))
        q = np.concatenate([q[:c], ACGT[rng.integers(0, 4, d)], q[c:]])[:L] if kind & 1 else \
            np.concatenate([q[:c], q[c + d:], w[:d]])[:L]
    if kind % 5 == 2 and L > 40:
        # a block replaced by unrelated sequence of another length
        c, d, e = int(rng.integers(10, L - 20)), int(rng.integers(3, 9)), int(rng.integers(3, 9))
        q = np.concatenate([q[:c], ACGT[rng.integers(0, 4, d)], q[c + e:], w[:10]])[:L]
    if kind % 7 == 3 and L > 2:
        q[int(rng.integers(0, L))] = ord("N")
        w[int(rng.integers(0, len(w)))] = ord("N")
    if kind % 11 == 4:
        w = w[:max(1, len(w) // 3)]
    s = q.tobytes()
    return (s.lower() if kind % 13 == 5 else s), w.tobytes()


def _check(sa, queries, refs, scores, sample):
    kw = dict(zip(("match", "mismatch", "gap_open", "gap_extend"), scores)) if scores else {}
    got = sa.align_batch(queries, refs, sa.mapping_defaults(**kw))
    extra = dict(zip(("match", "mismatch", "go", "ge"), scores)) if scores else {}
    for i in sample:
        assert got[i] == aligner_oracle(queries[i], refs[i], **extra), (i, len(queries[i]), queries[i], refs[i])


EDGES = [1, 2, 7, 8, 9, 15, 16, 17, 23, 24, 25, 63, 64, 65, 95, 96, 97, 127, 128, 129, 143, 144, 145, 151, 152, 153, 159,
         160, 161, 175, 207, 208, 209, 239, 255, 256, 257, 271, 319, 320, 321, 415, 416, 417, 495, 496, 497, 510, 511, 512]


@pytest.mark.parametrize("scores", [None, (1, 4, 6, 1), (4, 6, 10, 2), (2, 64, 255, 16), (16, 64, 40, 31), (2, 8, 32, 17),
                                    (17, 8, 12, 1), (2, 65, 12, 1), (10, 8, 12, 1)])
def test_lengths_at_edges(scores):
    import strobealign_gb300 as sa
    rng = np.random.default_rng(11)
    # batches by their longest read: each row count and thread count has its own kernel
    for top in (96, 128, 160, 208, 256, 257, 320, 416, 512):
        lens = [e for e in EDGES if e <= top]
        lens = lens + [lens[-1], lens[-1]] * 8
        pairs = [_pair(rng, L, k) for k, L in enumerate(lens * (2 if scores is None else 1))]
        _check(sa, [p[0] for p in pairs], [p[1] for p in pairs], scores, range(len(pairs)))


@pytest.mark.parametrize("lo,hi", [(150, 150), (91, 91), (125, 125), (200, 200), (251, 251), (20, 256), (100, 160)])
def test_many_tasks(lo, hi):
    import strobealign_gb300 as sa
    rng = np.random.default_rng(lo * 1000 + hi)
    n = 17_000
    pairs = [_pair(rng, int(rng.integers(lo, hi + 1)), k) for k in range(n)]
    _check(sa, [p[0] for p in pairs], [p[1] for p in pairs], None, range(0, n, 13))
