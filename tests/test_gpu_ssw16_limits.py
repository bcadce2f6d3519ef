"""SSW at the largest gap extension that the packed 16-bit kernel takes for a read length:
with match 3 and extension 24, reads up to 336 nt (42 rows a lane) fit in 16 bits and longer
ones do not."""
import numpy as np
import pytest

from oracle_lib import aligner_oracle

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", np.uint8)


@pytest.mark.parametrize("length", [320, 328, 329, 335, 336, 337, 338, 340, 341])
@pytest.mark.parametrize("scores", [(3, 8, 30, 24), (3, 8, 25, 24), (2, 8, 30, 16)])
def test_raise_at_its_lower_bound(scores, length):
    import strobealign_gb300 as sa
    rng = np.random.default_rng(length)
    queries, refs = [], []
    for k in range(48):
        pad = int(rng.integers(0, 40))
        w = ACGT[rng.integers(0, 4, length + 2 * pad + 4)]
        q = w[pad:pad + length].copy()
        sub = rng.random(length) < (0.01, 0.1, 0.4, 0.75)[k % 4]
        q[sub] = ACGT[rng.integers(0, 4, int(sub.sum()))]
        if k % 3 == 1:
            c = int(rng.integers(10, length - 10))
            q = np.concatenate([q[:c], q[c + 2:], w[:2]])
        queries.append(q.tobytes())
        refs.append(w.tobytes())
    got = sa.align_batch(queries, refs, sa.mapping_defaults(
        **dict(zip(("match", "mismatch", "gap_open", "gap_extend"), scores))))
    for i in range(len(queries)):
        want = aligner_oracle(queries[i], refs[i], **dict(zip(("match", "mismatch", "go", "ge"), scores)))
        assert got[i] == want, (i, queries[i], refs[i])
