"""The index build at the sizes where its kernels can go wrong: contigs shorter than a
k-mer, around the 32-lane windows of the syncmer kernel and its 28-, 26- and 24-position
steps, empty contigs in between, runs of equal hashes far beyond the histogram's last bin
and over several contigs (ties of hash and position), one contig (no position pass in the
sort) and many.  All integers: compared for equality with the oracle's table, directory
and cutoff."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", np.uint8)


def _genome(kind):
    rng = np.random.default_rng(77)
    rnd = lambda n: ACGT[rng.integers(0, 4, n)]  # noqa: E731
    if kind == "one":
        return [rnd(70_001)]
    if kind == "edges":
        return [rnd(n) for n in (0, 1, 15, 16, 19, 20, 21, 23, 27, 28, 29, 31, 32, 33, 47, 55, 56, 57, 0, 64, 2003, 3)]
    if kind == "runs":
        # one segment at the same positions of many contigs, a homopolymer and a tandem array
        seg = rnd(500)
        return [np.concatenate([seg, rnd(50)]) for _ in range(300)] + [np.full(4000, ord("A"), np.uint8),
                                                                     np.tile(rnd(23), 400), rnd(10_000)]
    # contigs on both sides of 2^16 nt: two and three position passes' worth of bits
    return [rnd(n) for n in (65_535, 65_536, 65_537, 40)]


@pytest.mark.parametrize("read_length", [70, 150, 250, 400])
@pytest.mark.parametrize("kind", ["one", "edges", "runs", "bits"])
def test_index_build_edges(kind, read_length):
    import strobealign_gb300 as sa
    from oracle.binding import OracleIndex
    seqs = _genome(kind)
    names = [f"c{i}" for i in range(len(seqs))]
    refs = sa.References.from_sequences(names, [s.tobytes() for s in seqs])
    idx = sa.StrobemerIndex.build(refs, sa.SeedingParameters.from_read_length(read_length))
    rs, bs = idx.to_host()
    o = OracleIndex(names, seqs, read_length)
    n, bits, cutoff = o.info()
    ors, obs = o.arrays()
    assert (len(rs), idx.bits, idx.filter_cutoff) == (n, bits, cutoff)
    assert np.array_equal(rs.view(np.uint8), ors.view(np.uint8))
    assert np.array_equal(bs, obs)
