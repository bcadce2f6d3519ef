"""Ungapped jobs of the extension waves (eight lanes a job, match bits 32 positions at a time) at
read lengths around the 32-base steps and up to the longest read, on both strands, with
mismatches at the ends, in runs and at word borders: SAM bytes against the oracle."""

import numpy as np
import pytest

from oracle_lib import run_oracle_cli
from test_gpu_parity import _first_diff, _map_files

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sa():
    import strobealign_gb300

    return strobealign_gb300


@pytest.mark.parametrize("length", [63, 64, 65, 95, 127, 129, 160, 255, 257, 500, 2047])
def test_ungapped_reads_match_oracle(sa, tmp_path, length):
    from strobealign_gb300 import synthetic as syn

    g = syn.make_genome(5, 60_000, 2, gc=0.45)
    fa, fq = str(tmp_path / "ref.fa"), str(tmp_path / "reads.fq")
    g.write_fasta(fa)
    rng = np.random.default_rng(length)
    comp = bytes.maketrans(b"ACGT", b"TGCA")
    with open(fq, "w") as f:
        for i in range(150):
            contig = g.seqs[i % 2].tobytes()
            # some reads at the very ends of their contig
            at = int(rng.integers(0, len(contig) - length)) if i % 10 else (len(contig) - length if i % 20 else 0)
            r = bytearray(contig[at:at + length])
            kind = i % 6
            places = []
            if kind == 1:
                places = [0, length - 1]
            elif kind == 2:
                places = list(range(min(4, length // 20)))
            elif kind == 3:
                places = [p for p in (31, 32, 63, 64) if p < length][: max(1, length // 25)]
            elif kind == 4:
                places = list(rng.integers(0, length, max(1, length // 25)))
            elif kind == 5:
                places = [length - 2, length - 3, 1]
            for p in places:
                r[p] = ord("N") if i % 17 == 0 else rng.choice([c for c in b"ACGT" if c != r[p]])
            r = bytes(r)
            if i & 8:
                r = r.translate(comp)[::-1]
            f.write(f"@r{i}\n{r.decode()}\n+\n{'I' * length}\n")
    want = run_oracle_cli(["--no-PG", "--eqx", fa, fq])
    got = _map_files(sa, fa, [fq], eqx=1)
    assert got == want, _first_diff(got, want)
