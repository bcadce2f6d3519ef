"""The repeat filter of full and partial lookups (src/index.rs:298-337) at the edges that
a look at the neighbouring entry does not settle: a main hash mask with fewer leading bits
than the bucket directory (a run of equal masked hashes then goes on in the next bucket),
and filter cutoffs of 0 and 1 (as an index file may have them; 0 filters every hash that
is not one of the table's last).  Counts per read equal a restatement over the table."""
import numpy as np
import pytest

from test_gpu_sti import reference_layout

pytestmark = pytest.mark.gpu

HASH_MASK = ~np.uint64(0xff)


def _params(sa, mask_bits):
    p = sa.SeedingParameters.from_read_length(150)
    if mask_bits:
        pop = 64 - mask_bits - 1
        p.c.main_hash_mask = ((1 << mask_bits) - 1) << (64 - mask_bits)
        p.c.partial_orientation_pos = pop
        p.c.forward_main_hash_mask = p.c.main_hash_mask | (1 << pop)
    return p


def _first(hashes, mask, bits, h):
    """get_masked_from (src/index.rs:159-197): the first entry of h's bucket with its masked hash."""
    top = int(h) >> (64 - bits)
    lo = int(np.searchsorted(hashes >> np.uint64(64 - bits), np.uint64(top)))
    hi = int(np.searchsorted(hashes >> np.uint64(64 - bits), np.uint64(top), "right"))
    eq = np.flatnonzero((hashes[lo:hi] & mask) == (np.uint64(h) & mask))
    return lo + int(eq[0]) if len(eq) else None


def _counts(hashes, mask, bits, cutoff, rs):
    """(full not found, filtered, found, partial not found, filtered, found) of one orientation."""
    n, c = len(hashes), [0] * 6
    reaches = lambda p, m: p + cutoff < n and (hashes[p] & m) == (hashes[p + cutoff] & m)  # noqa: E731
    count = lambda p: int(np.searchsorted(hashes, hashes[p], "right")) - p  # noqa: E731
    for h, hrc in rs:
        p = _first(hashes, HASH_MASK, bits, h)
        if p is not None:
            rc = _first(hashes, HASH_MASK, bits, hrc)
            filtered = reaches(p, HASH_MASK)
            if not filtered and rc is not None:
                filtered = reaches(rc, HASH_MASK) or count(p) + count(rc) > cutoff
            c[1 if filtered else 2] += 1
            continue
        c[0] += 1
        p = _first(hashes, mask, bits, h)
        if p is None:
            c[3] += 1
        else:
            c[4 if reaches(p, mask) else 5] += 1
    return c


@pytest.mark.parametrize("mask_bits,bits,cutoff", [
    (8, 8, None), (8, 9, None), (8, 12, None), (8, 16, None), (12, 14, 1), (0, 12, None),
    (0, 12, 1), (8, 12, 1), (0, 12, 0), (8, 12, 0)])
def test_filtered_counts(mask_bits, bits, cutoff, tmp_path):
    import strobealign_gb300 as sa
    from strobealign_gb300 import synthetic as syn
    g = syn.make_genome(41, 60_000, 2, gc=0.45, repeat_fraction=0.3)
    refs = sa.References.from_sequences(g.names, g.seqs)
    params = _params(sa, mask_bits)
    idx = sa.StrobemerIndex.build(refs, params, bits=bits)
    table, buckets = idx.to_host()
    if cutoff is None:
        cutoff = idx.filter_cutoff
    else:
        f = tmp_path / "t.sti"
        f.write_bytes(reference_layout(params.c, cutoff, bits, table, buckets))
        idx = sa.StrobemerIndex.read_sti(f, params)
    r = syn.make_single_end(42, g, 60, 150, 0.06, 0.005)
    reads = sa.Reads.from_arrays(r.seq, r.offsets, r.names, r.name_offsets, r.qual)
    _, det = sa.nams_batch(idx, reads)
    hashes = table["hash_offset"] & HASH_MASK
    mask = np.uint64(params.c.main_hash_mask)
    names = ("full_not_found", "full_filtered", "full_found", "partial_not_found", "partial_filtered",
             "partial_found")
    total = np.zeros(6, int)
    for i, (fwd, rc) in enumerate(sa.randstrobes_batch(idx, reads)):
        want = np.sum([_counts(hashes, mask, bits, cutoff, [(int(x["hash"]), int(x["hash_revcomp"])) for x in o])
                       for o in (fwd, rc)], axis=0)
        assert [int(det[n][i]) for n in names] == want.tolist(), i
        total += want
    found = 1 if cutoff == 0 else 2
    assert total[0] and total[found] and total[found + 3], total
    if mask_bits:
        assert total[4], total
