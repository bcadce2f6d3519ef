"""Chaining of long read orientations: clusters of thousands of anchors (tandem arrays),
many clusters per orientation (families whose copies hold an array) and reads that cross
from unique sequence into an array, so that the best-index re-check fires early, late and
while another cluster holds the running best.  NAMs equal the oracle's bit for bit, and
the output does not depend on how many anchors a cluster needs for a warp of its own
(chain_lane_cluster_max: 1 sends every cluster there, 4096 scores them a thread each),
for lookbacks on both sides of the 32 and 64 slots that the warps' rings have."""
import numpy as np
import pytest

from oracle_lib import OracleIndex

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", np.uint8)


def _mutate(rng, s, rate):
    s = s.copy()
    m = rng.random(len(s)) < rate
    s[m] = ACGT[rng.integers(0, 4, int(m.sum()))]
    return s


@pytest.fixture(scope="module")
def tandem(tmp_path_factory):
    rng = np.random.default_rng(5)
    rnd = lambda n: ACGT[rng.integers(0, 4, n)]  # noqa: E731
    unit = rnd(37)
    family = np.concatenate([rnd(300), np.tile(unit, 12), rnd(250)])
    parts = []
    for c in range(60):
        parts += [rnd(700), _mutate(rng, family, 0.01 * (c % 4))]
    arrays = [rnd(2000)]
    for period, copies, rate in ((2, 400, 0.02), (7, 150, 0.03), (23, 90, 0.02), (37, 120, 0.01), (50, 60, 0.03),
                                 (171, 30, 0.05)):
        arrays += [_mutate(rng, np.tile(rnd(period), copies), rate), rnd(1200)]
    seqs = [np.concatenate(parts), np.concatenate(arrays), _mutate(rng, np.tile(unit, 200), 0.01)]
    d = tmp_path_factory.mktemp("tandem")
    fa = str(d / "t.fa")
    with open(fa, "w") as f:
        for i, s in enumerate(seqs):
            f.write(f">t{i}\n{s.tobytes().decode()}\n")
    reads = []
    for i in range(700):
        s = seqs[int(rng.integers(0, 3))]
        n = int(rng.choice([100, 150, 250, 500, 1000, 2000]))
        o = int(rng.integers(0, len(s) - n))
        r = _mutate(rng, s[o:o + n], 0.01)
        if i % 5 == 0:
            # two places in one read
            o2 = int(rng.integers(0, len(s) - n))
            r = np.concatenate([r[:n // 2], s[o2:o2 + n // 2]])
        if i & 1:
            r = np.frombuffer(r.tobytes().translate(bytes.maketrans(b"ACGT", b"TGCA")), np.uint8)[::-1]
        reads.append(r.tobytes())
    return dict(fa=fa, reads=reads)


@pytest.mark.parametrize("read_length", [100, 150, 400])
def test_nams_of_tandem_repeats(tandem, read_length):
    import strobealign_gb300 as sa
    refs = sa.References.from_fasta(tandem["fa"])
    idx = sa.StrobemerIndex.build(refs, sa.SeedingParameters.from_read_length(read_length))
    reads = tandem["reads"]
    nams, det = sa.nams_batch(idx, sa.Reads.from_lists([f"n{i}" for i in range(len(reads))], reads))
    assert int(det["n_anchors"].max()) > 2000  # long orientations are there
    o = OracleIndex(tandem["fa"], read_length)
    for i, s in enumerate(reads):
        rows, _ = o.nams(s, 0)
        got = [(int(x["nam_id"]), int(x["ref_id"]), int(x["ref_start"]), int(x["ref_end"]), int(x["query_start"]),
                int(x["query_end"]), int(x["matching_bases"]), int(x["n_anchors"]),
                np.float32(x["score"]).view(np.uint32), int(x["is_revcomp"])) for x in nams[i]]
        assert got == [r[:8] + (np.float32(r[8]).view(np.uint32), r[9]) for r in rows], i


@pytest.mark.parametrize("lookback", [0, 1, 2, 31, 32, 33, 50, 63, 64, 100])
def test_cluster_split_does_not_change_output(tandem, lookback):
    import strobealign_gb300 as sa
    refs = sa.References.from_fasta(tandem["fa"])
    idx = sa.StrobemerIndex.build(refs, sa.SeedingParameters.from_read_length(150))
    cp = sa.chaining_defaults()
    cp.max_lookback = lookback
    m = sa.Mapper(idx, refs, chaining=cp, mode=sa.MODE_PAF)
    reads = sa.Reads.from_lists([f"r{i}" for i in range(len(tandem["reads"]))], tandem["reads"])
    out = {}
    for lane_max in (4096, 1, 3, 48):
        m.set_tuning(chain_lane_cluster_max=lane_max)
        out[lane_max] = m.map(reads)
    assert len(out[4096]) > 10000
    assert out[1] == out[4096] and out[3] == out[4096] and out[48] == out[4096]
