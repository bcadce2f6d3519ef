"""The banded traceback at the band widths where its kernels change hands: indels of 0 to 70
bases (a thread per task up to bands of 11 cells, the row wavefront from there on, in the
task's scratch up to 31 cells, in one or several 32-cell words per row beyond), two indels
that leave equal spans (no ungapped shortcut), spans shorter than a band, and ungapped
spans with scores on both sides of the shortcut's rule (mismatch <= gap_open + gap_extend).
Scores, spans and CIGARs equal the oracle's."""
import numpy as np
import pytest

from oracle_lib import aligner_oracle

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", np.uint8)


def _case(rng, L, d, where, sub):
    """L bases with an indel of d (negative: deleted from the query) at a fraction."""
    w = ACGT[rng.integers(0, 4, L + 140)]
    o, c = 40, int(L * where)
    ref = w[o:o + L + 80]
    q = np.concatenate([ref[:c], ACGT[rng.integers(0, 4, d)], ref[c:L - d]]) if d >= 0 else \
        np.concatenate([ref[:c], ref[c - d:L - d]])
    q = q.copy()
    m = rng.random(len(q)) < sub
    q[m] = ACGT[rng.integers(0, 4, int(m.sum()))]
    return q.tobytes(), w.tobytes()


def _check(sa, pairs, scores=None):
    names = ("match", "mismatch", "gap_open", "gap_extend")
    got = sa.align_batch([p[0] for p in pairs], [p[1] for p in pairs],
                         sa.mapping_defaults(**(dict(zip(names, scores)) if scores else {})))
    kw = dict(zip(("match", "mismatch", "go", "ge"), scores)) if scores else {}
    for p, g in zip(pairs, got):
        assert g == aligner_oracle(*p, **kw), p


@pytest.mark.parametrize("L", [60, 150, 300, 500])
def test_indel_sizes(L):
    import strobealign_gb300 as sa
    rng = np.random.default_rng(L)
    sizes = [d for d in (0, 1, 2, 3, 4, 5, 6, 7, 8, 10, 13, 14, 15, 16, 17, 20, 30, 31, 32, 33, 47, 48, 62, 63, 64, 70)
             if 3 * d < L]
    pairs = [_case(rng, L, s * d, w, sub) for d in sizes for s in (1, -1) for w in (0.3, 0.5, 0.7) for sub in (0, 0.02)]
    _check(sa, pairs)


def test_two_indels_and_short_spans():
    import strobealign_gb300 as sa
    rng = np.random.default_rng(3)
    pairs = []
    for _ in range(400):
        L, d = int(rng.integers(90, 400)), int(rng.integers(1, 25))
        w = ACGT[rng.integers(0, 4, L + 120)]
        r = w[30:30 + L]
        a, b = L // 3, 2 * L // 3
        # an insertion and a deletion of the same size: equal spans, a gapped path between
        q = np.concatenate([r[:a], ACGT[rng.integers(0, 4, d)], r[a:b], r[b + d:]])
        pairs.append((q.tobytes(), w.tobytes()))
    for n in range(1, 30):
        w = ACGT[rng.integers(0, 4, 60)]
        pairs.append((w[20:20 + n].tobytes(), w.tobytes()))
        pairs.append((w.tobytes(), w[20:20 + n].tobytes()))
    _check(sa, pairs)


@pytest.mark.parametrize("scores", [(2, 13, 12, 1), (2, 14, 12, 1), (2, 30, 12, 1), (1, 3, 2, 1), (2, 60, 5, 1)])
def test_ungapped_rule(scores):
    import strobealign_gb300 as sa
    rng = np.random.default_rng(sum(scores))
    pairs = [_case(rng, int(rng.integers(40, 250)), int(rng.integers(-3, 4)) if k & 1 else 0, 0.5, (0.02, 0.08)[k // 2 % 2])
             for k in range(600)]
    _check(sa, pairs, scores)
