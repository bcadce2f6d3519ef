"""The smallest cluster limit of a mapper's tuning: 1 is taken as 2, which the tuning then
reports, and 2 sends every cluster of three anchors or more to the large-cluster kernel, with
the same output as all other limits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", np.uint8)


def test_smallest_cluster_limit():
    import strobealign_gb300 as sa
    rng = np.random.default_rng(17)
    rnd = lambda n: ACGT[rng.integers(0, 4, n)]  # noqa: E731
    # families far apart, a few anchors each, and a tandem array
    family, unit = rnd(60), rnd(31)
    seq = np.concatenate([np.concatenate([rnd(900), family]) for _ in range(80)] + [rnd(500), np.tile(unit, 60)])
    refs = sa.References.from_sequences(["c"], [seq.tobytes()])
    idx = sa.StrobemerIndex.build(refs, sa.SeedingParameters.from_read_length(150))
    seqs = []
    for i in range(300):
        n = int(rng.integers(150, 700))
        o = int(rng.integers(0, len(seq) - n))
        s = np.concatenate([family, seq[o:o + n]])
        s[rng.random(len(s)) < 0.01] = ord("A")
        seqs.append(s.tobytes())
    reads = sa.Reads.from_lists([f"r{i}" for i in range(len(seqs))], seqs)
    m = sa.Mapper(idx, refs, mode=sa.MODE_PAF)
    out = {}
    for limit in (1, 2, 3, 48, 4096):
        m.set_tuning(chain_lane_cluster_max=limit)
        assert m.tuning()["chain_lane_cluster_max"] == max(limit, 2)
        out[limit] = m.map(reads)
    assert len(out[1]) > 10_000 and len(set(out.values())) == 1
