"""Batches of no reads whose arrays are null (a zeroed sa_read_batch) map to nothing, through
every entry point that takes a batch to a mapper or a session."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def indexed():
    import strobealign_gb300 as sa
    from strobealign_gb300 import synthetic as syn
    g = syn.make_genome(3, 50_000, 2)
    refs = sa.References.from_sequences(g.names, g.seqs)
    r = syn.make_single_end(4, g, 50, 150, 0.01, 0.001)
    return (sa, refs, sa.StrobemerIndex.build(refs, sa.SeedingParameters.from_read_length(150)),
            sa.Reads.from_arrays(r.seq, r.offsets, r.names, r.name_offsets, r.qual))


def test_null_arrays(indexed):
    sa, refs, idx, reads = indexed
    from strobealign_gb300 import _lib as L
    m = sa.Mapper(idx, refs)
    want = m.map(reads)
    lib, none = sa.lib(), L.ReadBatch()
    calls = [lambda o: lib.sa_map_batch(m.h, C.byref(none), None, o),
             lambda o: lib.sa_map_batch(m.h, C.byref(none), C.byref(none), o),
             lambda o: lib.sa_map_batch_interleaved(m.h, C.byref(none), o)]
    for r2 in (None, C.byref(none)):
        calls.append(lambda o, r2=r2: lib.sa_mapper_upload(m.h, C.byref(none), r2) or lib.sa_map_uploaded(m.h, o))
    for call in calls:
        out = L.Output()
        L.check(call(C.byref(out)))
        assert out.len == 0 and out.n_reads == 0 and out.n_mapped == 0
        lib.sa_output_free(C.byref(out))
    assert m.map(reads) == want


def test_null_arrays_in_a_session(indexed):
    sa, refs, idx, reads = indexed
    from strobealign_gb300 import _lib as L
    s = sa.Session(idx, refs)
    none = L.ReadBatch()
    for submit in (lambda t: sa.lib().sa_session_submit(s.h, C.byref(none), None, t),
                   lambda t: sa.lib().sa_session_submit(s.h, C.byref(none), C.byref(none), t),
                   lambda t: sa.lib().sa_session_submit_interleaved(s.h, C.byref(none), t)):
        ticket = C.c_uint64()
        L.check(submit(C.byref(ticket)))
        assert bytes(s.wait(ticket.value)[0]) == b""
    s.close()
