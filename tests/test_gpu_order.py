"""The bucket order of K3c where its branches meet: bucket counts around the two-per-thread
order (256, 512), partitions around the staged size (4096 keys), odd and tiny ones, and small
partitions whose buckets collide on most pilot counters (the collision test at the mark)."""
import numpy as np
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


@pytest.mark.parametrize("kind", ["u64", "bytes16", "prehashed"])
@pytest.mark.parametrize("P,n", [(2048, 12_288), (2048, 12_289), (64, 9_472), (64, 9_473), (64, 5_001), (2500, 1),
                                 (16_384, 12_288)])
def test_small_builds_match_oracle(phobic, kind, P, n):
    """Sizes on both sides of the one-launch path of small builds: 12,288 keys, 148 partitions."""
    cfg = phobic.MPHFconfig(4.0, P)
    if kind == "u64":
        keys = keygen.splitmix64(50 + P, n)
        keys4 = O.hash_keys(keys, "u64")
    else:
        keys = keygen.splitmix64(51 + P, 2 * n).reshape(n, 2)
        keys4 = O.hash_keys(keys, "pairs") if kind == "bytes16" else keys.view("uint32").reshape(n, 4)
    kid = {"u64": phobic.KEYS_U64, "bytes16": phobic.KEYS_BYTES16, "prehashed": phobic.KEYS_PREHASHED}[kind]
    want = O.build(keys4, P, cfg.bucketCountPerPartition, cfg.getFulcs())
    with phobic.Context(0) as ctx:
        if want["status"] != 0:
            with pytest.raises(phobic.PhobicError) as e:
                ctx.build(keys, cfg, kind=kid)
            assert e.value.status == want["status"]
            return
        got = ctx.build(keys, cfg, kind=kid)
        assert got.timings["kernels"] == (2 if n <= 12_288 and got.partitions <= 148 else 6)
    assert (got.pilots == want["pilots"]).all() and (got.partition_offsets == want["offsets"]).all()


def test_small_builds_report_errors_like_the_oracle(phobic):
    cfg = phobic.MPHFconfig(5.0, 2048)
    keys = keygen.splitmix64(60, 9_000)
    dup = keys.copy()
    dup[7] = dup[8_000]
    crowded = np.zeros((9_000, 4), np.uint32)  # every key in partition 0
    crowded[:, 1:] = keygen.splitmix64(61, 2 * 9_000).view(np.uint32).reshape(9_000, 4)[:, 1:]
    flat = crowded.copy()
    flat[:, 0] = keygen.splitmix64(62, 9_000).astype(np.uint32)
    flat[:, 1] = 0  # every key in bucket 0 of its partition
    with phobic.Context(0) as ctx:
        for k, kind, keys4 in ((dup, phobic.KEYS_U64, O.hash_keys(dup, "u64")), (crowded, phobic.KEYS_PREHASHED, crowded),
                               (flat, phobic.KEYS_PREHASHED, flat)):
            want = O.build(keys4, 2048, cfg.bucketCountPerPartition, cfg.getFulcs())["status"]
            assert want != 0
            with pytest.raises(phobic.PhobicError) as e:
                ctx.build(k, cfg, kind=kind)
            assert e.value.status == want
        got = ctx.build(keys, cfg)
        assert (got.pilots == O.build(O.hash_keys(keys, "u64"), 2048, cfg.bucketCountPerPartition, cfg.getFulcs())["pilots"]).all()


@pytest.mark.parametrize("group,pipe", [(1, 0), (4, 0), (2, 1), (4, 1), (8, 1), (0, 0)])
@pytest.mark.parametrize("P,n", [(16, 20), (32, 200), (64, 9_000), (128, 30_000), (256, 1_000), (300, 40_000), (512, 90_000), (520, 30_000)])
def test_small_partitions_match_oracle(phobic, P, n, group, pipe):
    """Partitions of few slots: most offsets of a bucket's windows are gone by its turn, most of its
    pilot counters put two keys on one slot, and a partition is ordered by one warp."""
    cfg = phobic.MPHFconfig(5.0, P)
    keys = keygen.splitmix64(8000 + P, n)
    want = O.build(O.hash_keys(keys, "u64"), P, cfg.bucketCountPerPartition, cfg.getFulcs())
    assert want["status"] == 0
    with phobic.Context(0) as ctx:
        ctx.set_tuning(search_group=group, search_pipeline=pipe)
        got = ctx.build(keys, cfg)
    assert (got.pilots == want["pilots"]).all() and (got.partition_offsets == want["offsets"]).all()


def test_crowded_buckets_match_oracle(phobic):
    """Large buckets that nearly always meet themselves: the first chunk of 32 keys ends most tries, the second
    one some, in the one-warp search of partitions of few slots (128 and fewer) and of more."""
    for lam, P, n in ((8.0, 100, 2_000), (7.0, 64, 640), (6.0, 160, 8_000), (10.0, 700, 14_000), (10.0, 160, 8_000)):
        cfg = phobic.MPHFconfig(lam, P)
        keys = keygen.splitmix64(8100 + P, n)
        want = O.build(O.hash_keys(keys, "u64"), P, cfg.bucketCountPerPartition, cfg.getFulcs(), max_k=20_000)
        cfg.params.max_pilot_counter = 20_000
        with phobic.Context(0) as ctx:
            for group, pipe in ((1, 0), (8, 1)):
                ctx.set_tuning(search_group=group, search_pipeline=pipe)
                if want["status"] != 0:
                    with pytest.raises(phobic.PhobicError) as e:
                        ctx.build(keys, cfg)
                    assert e.value.status == want["status"]
                    continue
                got = ctx.build(keys, cfg)
                assert (got.pilots == want["pilots"]).all() and (got.partition_offsets == want["offsets"]).all()


@pytest.mark.parametrize("group,pipe", [(1, 0), (4, 1), (8, 1), (2, 0)])
def test_more_one_key_buckets_than_are_listed(phobic, group, pipe):
    """Hundreds of buckets of one key per partition: the last 128 go by the list of free slots, those before them
    by the search."""
    cfg = phobic.MPHFconfig(1.5, 2048)
    keys = keygen.splitmix64(8200, 30_000)
    want = O.build(O.hash_keys(keys, "u64"), 2048, cfg.bucketCountPerPartition, cfg.getFulcs(), intermediates=True)
    assert want["status"] == 0
    assert (want["bucket_sizes"].reshape(-1, cfg.bucketCountPerPartition) == 1).sum(axis=1).min() > 128
    with phobic.Context(0) as ctx:
        ctx.set_tuning(search_group=group, search_pipeline=pipe)
        got = ctx.build(keys, cfg)
    assert (got.pilots == want["pilots"]).all() and (got.partition_offsets == want["offsets"]).all()
