"""The bucket order of K3c where its branches meet: bucket counts around the two-per-thread
order (256, 512), partitions around the staged size (4096 keys), odd and tiny ones, and small
partitions whose buckets collide on most pilot counters (the collision test at the mark)."""
import pytest

import keygen
import oracle_lib as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lam,P,buckets", [(4.0, 1024, 256), (3.98, 1024, 258), (4.0, 2048, 512), (3.99, 2048, 514),
                                           (8.0, 4096, 512), (7.0, 6000, 858), (2.0, 48, 24), (8.0, 96, 12)])
def test_bucket_order_matches_oracle(phobic, lam, P, buckets):
    cfg = phobic.MPHFconfig(lam, P)
    assert cfg.bucketCountPerPartition == buckets
    for n in (1, P - 1, 37 * P + 5):
        keys = keygen.splitmix64(900 + buckets, n)
        want = O.build(O.hash_keys(keys, "u64"), P, buckets, cfg.getFulcs(), intermediates=True)
        with phobic.Context(0) as ctx:
            if want["status"] != 0:
                with pytest.raises(phobic.PhobicError) as e:
                    ctx.build(keys, cfg)
                assert e.value.status == want["status"]
                continue
            got, _, sizes = ctx.debug_build(keys, cfg)
            assert (got.pilots == want["pilots"]).all() and (got.partition_offsets == want["offsets"]).all()
            assert (sizes == want["bucket_sizes"]).all()


@pytest.mark.parametrize("group,pipe", [(1, 0), (2, 1), (4, 1), (8, 1), (4, 0)])
@pytest.mark.parametrize("P", [1024, 2048, 3072])
def test_round_edges_match_oracle(phobic, P, group, pipe):
    """Partitions on both sides of 1024, 2048 and 3072 slots: the edges of the offset search's
    rounds, and of the pipeline's one-, two- and three-round and general searches."""
    cfg = phobic.MPHFconfig(5.0, P)
    keys = keygen.splitmix64(7000 + P, 40 * P + 3)
    want = O.build(O.hash_keys(keys, "u64"), P, cfg.bucketCountPerPartition, cfg.getFulcs())
    assert want["status"] == 0
    with phobic.Context(0) as ctx:
        ctx.set_tuning(search_group=group, search_pipeline=pipe)
        got = ctx.build(keys, cfg)
    assert (got.pilots == want["pilots"]).all() and (got.partition_offsets == want["offsets"]).all()
