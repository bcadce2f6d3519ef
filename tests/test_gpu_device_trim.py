"""Device memory of repeated calls and freed handles, as the device counts it: the same call
again takes no more of it, an index built after a larger call holds what it reports, and
sa_device_trim gives back all that is kept once the handles are freed."""
import ctypes as C
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SLACK = 8 << 20  # the driver's own allocations


def _free():
    import torch
    return torch.cuda.mem_get_info()[0]


@pytest.fixture(scope="module")
def work():
    import strobealign_gb300 as sa
    from strobealign_gb300 import synthetic as syn
    g = syn.make_genome(61, 40_000_000, 3, gc=0.41, repeat_fraction=0.2)
    refs = sa.References.from_sequences(g.names, g.seqs)
    r1, r2 = syn.make_paired_end(62, g, 40_000, 150, 300, 30, 0.01, 0.001)
    take = lambda r: sa.Reads.from_arrays(r.seq, r.offsets, r.names, r.name_offsets, r.qual)  # noqa: E731
    reads = (take(r1), take(r2))
    params = sa.SeedingParameters.from_read_length(150)

    def all_of_it():
        idx = sa.StrobemerIndex.build(refs, params)
        sa.nams_batch(idx, reads[0])
        sa.align_batch([b"ACGTTGCA" * 20] * 5000, [b"TTACGTTGCA" * 30] * 5000)
        m = sa.Mapper(idx, refs)
        out = m.map(*reads)
        s = sa.Session(idx, refs, max_inflight_bases=1 << 24)
        assert s.wait(s.submit(*reads))[0] == out
        s.close()
        del m, s, idx
        gc.collect()

    all_of_it()  # kernels and streams are loaded and made
    sa.device_trim()
    return sa, refs, params, reads, all_of_it


def test_all_is_given_back(work):
    sa, _, _, _, all_of_it = work
    before = _free()
    for _ in range(3):
        all_of_it()
        kept = before - _free()  # in whole pages, a block has at least one
        released = sa.device_trim()
        assert 0 < released <= min(kept + SLACK, 8 << 30)
        assert before - _free() <= SLACK
    assert sa.device_trim() == 0
    assert sa.lib().sa_device_trim(None) == 0


def test_the_same_call_takes_no_more(work):
    sa, refs, params, reads, _ = work
    idx = sa.StrobemerIndex.build(refs, params)

    def calls():
        sa.nams_batch(idx, reads[0])
        sa.align_batch([b"ACGTTGCA" * 20] * 5000, [b"TTACGTTGCA" * 30] * 5000)
        sa.StrobemerIndex.build(refs, params).lookup(np.arange(100_000, dtype=np.uint64) << np.uint64(44))

    for _ in range(2):
        calls()
    before = _free()
    for _ in range(6):
        calls()
    assert abs(before - _free()) <= SLACK


def test_an_index_holds_what_it_reports(work):
    sa, refs, params, reads, _ = work
    idx = sa.StrobemerIndex.build(refs, params)
    sa.nams_batch(idx, reads[0])  # leaves blocks of many sizes
    del idx
    gc.collect()
    idx = sa.StrobemerIndex.build(refs, params)
    sa.device_trim()
    before = _free()
    held = idx.info.device_bytes
    assert held > 10 * SLACK
    sa.lib().sa_index_free(idx.h)
    idx.h = C.c_void_p()
    sa.device_trim()
    # the device hands out memory in 2 MB pages
    assert abs(_free() - before - held) <= SLACK, (_free() - before, held)
