"""Device memory of a batch too large for one NAM workspace: two parts are in work at once,
and together they hold no more bases than one part may alone."""
import pytest

pytestmark = pytest.mark.gpu


def test_two_lanes_share_the_limit():
    import torch

    import strobealign_gb300 as sa
    from strobealign_gb300 import synthetic as syn
    limit = 1 << 27  # bases
    g = syn.make_genome(3, 2_000_000, 2, gc=0.41)
    refs = sa.References.from_sequences(g.names, g.seqs)
    idx = sa.StrobemerIndex.build(refs, sa.SeedingParameters.from_read_length(150))
    r = syn.make_single_end(4, g, 2_000_000, 150, 0.01, 0.001)
    reads = sa.Reads.from_arrays(r.seq, r.offsets, r.names, r.name_offsets, r.qual)
    bases = int(reads.seq_offsets[-1])
    assert bases > 2 * limit
    sa.device_trim()
    before = torch.cuda.mem_get_info()[0]
    out = {}
    for parts in (1, 8):
        m = sa.Mapper(idx, refs, mode=sa.MODE_PAF)
        m.set_parts(parts)
        for _ in range(2):
            out[parts] = m.map(reads)
        sa.device_trim()
        held = before - torch.cuda.mem_get_info()[0]
        # the batch itself, then what a session counts for a workspace
        assert held <= 2 * bases + 160 * limit, (parts, held)
        del m
        sa.device_trim()
    assert out[1] == out[8] and len(out[1]) > 50 * len(reads)
