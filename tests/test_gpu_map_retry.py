"""A batch whose mapping ran out of device memory stays with the mapper: sa_map_uploaded maps
it once there is memory, to the bytes of a mapping that did not fail, after sa_map_batch as
after sa_mapper_upload."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("two_steps", [False, True])
def test_out_of_memory_then_again(two_steps):
    import torch

    import strobealign_gb300 as sa
    from strobealign_gb300 import synthetic as syn
    g = syn.make_genome(3, 2_000_000, 2, gc=0.41)
    refs = sa.References.from_sequences(g.names, g.seqs)
    idx = sa.StrobemerIndex.build(refs, sa.SeedingParameters.from_read_length(150))
    r = syn.make_single_end(4, g, 2_000_000, 150, 0.01, 0.001)
    reads = sa.Reads.from_arrays(r.seq, r.offsets, r.names, r.name_offsets, r.qual)
    want = sa.Mapper(idx, refs, mode=sa.MODE_PAF).map(reads)
    m = sa.Mapper(idx, refs, mode=sa.MODE_PAF)
    m.set_parts(1)  # as few parts as the limit allows: their workspaces take over 10 GB
    if two_steps:
        m.upload(reads)
    sa.device_trim()
    rest = 4 << 30
    held = torch.empty(torch.cuda.mem_get_info()[0] - rest, dtype=torch.uint8, device="cuda")
    try:
        for _ in range(2):
            with pytest.raises(sa.SaError) as e:
                m.map_uploaded() if two_steps else m.map(reads)
            assert e.value.code == -3  # SA_ERR_OOM
    finally:
        del held
        torch.cuda.empty_cache()
    assert m.map_uploaded() == want
    assert m.map_uploaded() == want
    assert m.map(reads) == want
