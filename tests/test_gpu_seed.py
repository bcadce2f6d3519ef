"""Seeding kernel at the edges of its layout: read lengths around its 32-base words and 32-word
rounds, as many syncmers as shared memory holds and one more or less, and every byte value as a
base; randstrobes of both orientations against the oracle."""

import numpy as np
import pytest

from oracle_lib import randstrobes_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("read_length", [50, 100, 150, 250, 400])
def test_randstrobes_at_the_edges(tmp_path, read_length):
    import strobealign_gb300 as sa

    rng = np.random.default_rng(read_length)
    fa = tmp_path / "ref.fa"
    fa.write_text(">c\n" + "".join(rng.choice(list("ACGT"), 5000)) + "\n")
    refs = sa.References.from_fasta(str(fa))
    idx = sa.StrobemerIndex.build(refs, sa.SeedingParameters.from_read_length(read_length))
    seqs = []
    for n in (1, 19, 20, 31, 32, 33, 63, 64, 65, 159, 160, 161, 480, 520, 560, 600, 1023, 1024, 1025, 1056, 2047, 2048):
        for letters in ("ACGT", "ACGTNacgtu", "AT"):
            seqs.append("".join(rng.choice(list(letters), n)).encode())
    # homopolymers: every k-mer (19 to 23 nt) is a syncmer, so 104 of them at 122 to 126 nt
    seqs += [b"C" * n for n in range(118, 130)] + [b"A" * 2048]
    base = rng.choice(list(b"ACGT"), 300).astype(np.uint8)
    for byte in range(1, 256):
        r = base.copy()
        r[150] = byte
        seqs.append(r.tobytes())
    got = sa.randstrobes_batch(idx, sa.Reads.from_lists([f"r{i}" for i in range(len(seqs))], seqs))
    for s, (f, r) in zip(seqs, got):
        for a, b in zip((f, r), randstrobes_oracle(s, read_length)):
            assert len(a) == len(b), s
            for column, field in enumerate(("hash", "hash_revcomp", "start", "end")):
                assert (a[field] == b[:, column]).all(), (s, field)
