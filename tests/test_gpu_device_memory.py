"""The cache of freed device blocks: calls of several sizes from several threads at once give
what they give alone, an index outlives the buffers its build gave back, and what the
process keeps stays bounded."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _nams(sa, idx, reads):
    nams, det = sa.nams_batch(idx, reads)
    return [n.tobytes() for n in nams], det.tobytes()


def test_threads_and_sizes_share_blocks():
    import torch

    import strobealign_gb300 as sa
    from strobealign_gb300 import synthetic as syn
    g = syn.make_genome(91, 600_000, 3, gc=0.41, repeat_fraction=0.2)
    refs = sa.References.from_sequences(g.names, g.seqs)
    p = sa.SeedingParameters.from_read_length(150)
    idx = sa.StrobemerIndex.build(refs, p)
    table, buckets = idx.to_host()
    sets = []
    for i, n in enumerate((1, 37, 900, 901, 2500, 6000)):
        r = syn.make_single_end(92 + i, g, n, 150, 0.01, 0.001)
        sets.append(sa.Reads.from_arrays(r.seq, r.offsets, r.names, r.name_offsets, r.qual))
    want = [_nams(sa, idx, s) for s in sets]
    errors = []

    def work(t):
        try:
            for k in range(6):
                i = (t + k) % len(sets)
                assert _nams(sa, idx, sets[i]) == want[i]
                if k % 3 == t % 3:
                    again = sa.StrobemerIndex.build(refs, p)
                    rs, bs = again.to_host()
                    assert np.array_equal(rs, table) and np.array_equal(bs, buckets)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    th = [threading.Thread(target=work, args=(t,)) for t in range(5)]
    [t.start() for t in th]
    [t.join() for t in th]
    assert not errors, errors[0]
    # the index's own buffers were not among those given back
    rs, bs = idx.to_host()
    assert np.array_equal(rs, table) and np.array_equal(bs, buckets)
    free0 = torch.cuda.mem_get_info()[0]
    for _ in range(4):
        assert _nams(sa, idx, sets[-1]) == want[-1]
    assert free0 - torch.cuda.mem_get_info()[0] <= (8 << 30)
