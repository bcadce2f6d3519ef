"""Piecewise DP pieces at the edges of the wavefront's strips (32 rows of one, 64 of two rows a
lane), wider than the shared row buffer, and chains of more anchors than shared memory holds,
against the oracle's restatement; every field and CIGAR has to be equal."""

import numpy as np
import pytest

from test_unit_vectors import _mp, _ora_extend, _ora_piece

KINDS = {0: "global", 1: "xdrop_GlobalStartLocalEnd", 2: "xdrop_LocalStartGlobalEnd"}


@pytest.fixture(scope="module")
def sa():
    import strobealign_gb300

    return strobealign_gb300


def _noisy(rng, q, edits, alphabet="ACGT"):
    r = list(q)
    for _ in range(edits):
        p, op = int(rng.integers(0, max(1, len(r)))), rng.integers(0, 3)
        if op == 0 and r:
            r[min(p, len(r) - 1)] = rng.choice(list(alphabet))
        elif op == 1:
            r[p:p] = rng.choice(list(alphabet), int(rng.integers(1, 40)))
        else:
            del r[p:p + int(rng.integers(1, 40))]
    return r


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 34, 63, 64, 65, 127, 128, 129, 200])
@pytest.mark.parametrize("scores", [(2, 8, 12, 1, 10), (1, 1, 2, 2, 0), (3, 2, 4, 1, 5)])
def test_pieces_at_strip_edges(sa, n, scores):
    rng = np.random.default_rng(1000 * n + scores[0])
    sc = dict(zip(("match", "mismatch", "gap_open", "gap_extend", "end_bonus"), scores))
    qs, rs, kinds = [], [], []
    for m in (1, 2, 31, 32, 33, n, n + 1, n + n // 10, 511, 512, 600):
        for kind in KINDS:
            # two letters only in a third of them: many equal scores
            letters = "AC" if rng.random() < 0.33 else "ACGTN"
            q = "".join(rng.choice(list(letters), n))
            r = _noisy(rng, q, int(rng.integers(0, 5)), letters) + list(rng.choice(list(letters), 600))
            qs.append(q)
            rs.append("".join(r[:m]))
            kinds.append(kind)
    got = sa.piecewise_pieces(qs, rs, kinds, _mp(sa, sc))
    for q, r, k, g in zip(qs, rs, kinds, got):
        assert g == _ora_piece(dict(query=q, ref=r, kind=KINDS[k], scores=sc)), (q, r, k)


@pytest.mark.gpu
@pytest.mark.parametrize("stride", [1, 3, 17, 60])
@pytest.mark.parametrize("length", [70, 300, 900])
def test_chains_against_oracle(sa, stride, length):
    # every k-mer (900 nt: hundreds of anchors), every third, and gaps between anchors, with
    # indels on either side of what the pruning tolerates
    rng = np.random.default_rng(length + stride)
    sc = {"match": 2, "mismatch": 8, "gap_open": 12, "gap_extend": 1, "end_bonus": 10}
    k = 15
    cases = []
    for indel in (0, 1, 4, 6, 30):
        for _ in range(6):
            q = "".join(rng.choice(list("ACGT"), length))
            cut = int(rng.integers(k, length - k))
            body = list(q)
            for _ in range(int(rng.integers(0, 1 + length // 40))):
                body[int(rng.integers(0, length))] = "ACGT"[int(rng.integers(0, 4))]
            extra = "".join(rng.choice(list("ACGT"), indel))
            lead = "".join(rng.choice(list("ACGT"), int(rng.integers(0, 40))))
            back = length - cut
            gap = indel if rng.random() < 0.5 else -min(indel, back - 1)
            tail = body[cut:] if gap >= 0 else body[cut - gap:]
            ref = lead + "".join(body[:cut]) + (extra if gap > 0 else "") + "".join(tail) + \
                "".join(rng.choice(list("ACGT"), int(rng.integers(0, 40))))
            anchors = []
            for a in range(0, length - k + 1, stride):
                b = len(lead) + a + (gap if a >= cut else 0)
                if 0 <= b and b + k <= len(ref) and q[a:a + k] == ref[b:b + k] and (a + k <= cut or a >= cut):
                    anchors.append((a, b))
            if anchors:
                cases.append((q, ref, anchors[::-1]))
    assert cases
    got = sa.piecewise_batch([c[0] for c in cases], [c[1] for c in cases], [c[2] for c in cases], k, _mp(sa, sc))
    for (q, ref, anchors), g in zip(cases, got):
        want = _ora_extend(dict(query=q, ref=ref, k=k, padding=length // 10, xdrop=500, scores=sc,
                                anchors=[dict(ref_id=0, ref_start=b, query_start=a) for a, b in anchors]), 1)
        assert g == want, (q, ref, anchors)
