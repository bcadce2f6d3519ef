"""Clusters whose best score is lower with the best-index re-check than without it (a score
that the re-check raised ends a later anchor's scan on its diagonal before a better
predecessor).  An earlier cluster holds the read's best score, so the reference scores the
cluster without the re-check, and the chain threshold lies between the two maxima: the
cluster has a NAM only if it is scored that way.

chain_recheck_clusters.json holds such anchor sets, found by a search over random lattices
with the default chaining parameters: per case a read, the randstrobes (by number) of a
one-diagonal chain on reference 0, and the cluster's anchors (randstrobe number, position)
on reference 1.  The index tables are written to have just these anchors."""
import json

import numpy as np
import pytest

from conftest import GOLDEN
from oracle_lib import OracleIndex, randstrobes_oracle
from test_gpu_sti import reference_layout

pytestmark = pytest.mark.gpu

CASES = json.loads((GOLDEN / "chain_recheck_clusters.json").read_text())
RS = np.dtype([("hash_offset", "<u8"), ("position", "<u4"), ("ref_index", "<u4")])
BITS, CUTOFF = 8, 100


def directory(hashes: np.ndarray, bits: int) -> np.ndarray:
    """bucket_starts of a sorted table (src/indexer.rs:82-124)."""
    starts = [0]
    for pos in range(1, len(hashes)):
        if hashes[pos] != hashes[pos - 1]:
            top = int(hashes[pos]) >> (64 - bits)
            starts += [pos] * (top + 1 - len(starts))
    return np.array(starts + [len(hashes)] * ((1 << bits) + 1 - len(starts)), np.uint64)


def table_of(case):
    fwd, _ = randstrobes_oracle(case["read"].encode(), 150)
    mask = ~np.uint64(0xff)
    first, last = case["before"]
    entries = [(int(fwd[i][0] & mask), 1000 + int(fwd[i][2]), 0) for i in range(first, last + 1)]
    entries += [(int(fwd[i][0] & mask), pos, 1) for i, pos in case["anchors"]]
    t = np.array(sorted(entries), dtype=RS)
    return t, directory(t["hash_offset"] & mask, BITS)


@pytest.mark.parametrize("i", range(len(CASES)))
def test_cluster_scored_without_the_recheck(i, tmp_path):
    import strobealign_gb300 as sa
    case = CASES[i]
    table, buckets = table_of(case)
    params = sa.SeedingParameters.from_read_length(150)
    f = tmp_path / "t.sti"
    f.write_bytes(reference_layout(params.c, CUTOFF, BITS, table, buckets))
    idx = sa.StrobemerIndex.read_sti(f, params)
    first_strobe = 3
    read = case["read"].encode()
    nams, det = sa.nams_batch(idx, sa.Reads.from_lists(["r"], [read]),
                              mapping=sa.mapping_defaults(mcs_strategy=first_strobe))
    rows, _ = OracleIndex.from_table(150, BITS, CUTOFF, table, buckets).nams(read, first_strobe)
    # the case is what it is meant to be: long, one chain before, and one in the cluster
    assert int(det["n_anchors"][0]) > 96 and {r[1] for r in rows} == {0, 1}
    got = [(int(x["nam_id"]), int(x["ref_id"]), int(x["ref_start"]), int(x["ref_end"]), int(x["query_start"]),
            int(x["query_end"]), int(x["matching_bases"]), int(x["n_anchors"]),
            np.float32(x["score"]).view(np.uint32), int(x["is_revcomp"])) for x in nams[0]]
    assert got == [r[:8] + (np.float32(r[8]).view(np.uint32), r[9]) for r in rows]
