"""What a build reports when its input is at fault, whatever the order in which the GPU comes to
the parts of it: the lowest oversized partition, keys that change while a small build runs."""
import numpy as np
import pytest

import keygen
import oracle_lib as O

pytestmark = pytest.mark.gpu


def partitioner_for(p, M):
    """A partitioner word of partition p of M (key_mapping.glsl:3-9)."""
    x = -(-(p << 32) // M)
    assert (x * M) >> 32 == p
    return x


def test_the_lowest_of_adjacent_oversized_partitions_is_reported(phobic):
    """64 oversized partitions side by side belong to as many CTAs, which by then have got to them
    at times of their own."""
    n, P, first = 600_000, 100, 5000
    cfg = phobic.MPHFconfig(5.0, P)
    cap = cfg.params.max_partition_size
    M = cfg.partitions(n)
    k4 = keygen.splitmix64(71, 2 * n).view(np.uint32).reshape(n, 4).copy()
    for i, p in enumerate(range(first, first + 64)):
        k4[3000 * i: 3000 * (i + 1), 0] = partitioner_for(p, M)
    sizes = np.bincount((k4[:, 0].astype(np.uint64) * M >> np.uint64(32)).astype(int), minlength=M)
    assert (np.flatnonzero(sizes > cap) == np.arange(first, first + 64)).all()
    want = O.build(k4, P, cfg.bucketCountPerPartition, cfg.getFulcs())
    assert want["status"] == phobic.ERR_PARTITION_OVERFLOW and want["stats"].err_partition == first
    good = keygen.splitmix64(72, 2 * 5_000).view(np.uint32).reshape(5_000, 4)
    assert O.build(good, P, cfg.bucketCountPerPartition, cfg.getFulcs())["status"] == phobic.OK
    with phobic.Context(0) as ctx:
        for _ in range(40):
            with pytest.raises(phobic.PhobicError) as e:
                ctx.build(k4, cfg, kind=phobic.KEYS_PREHASHED)
            assert e.value.status == phobic.ERR_PARTITION_OVERFLOW and f"partition {first})" in str(e.value)
        for _ in range(10):
            _, st = phobic.build_batch(ctx, [good, k4], cfg, kind=phobic.KEYS_PREHASHED)
            assert st == [phobic.OK, phobic.ERR_PARTITION_OVERFLOW] and f"set 1, partition {first})" in ctx.last_error


@pytest.mark.parametrize("way", ["down", "up", "from_first", "to_first", "same"])
def test_keys_changed_during_a_small_build_are_reported(phobic, way):
    """A small build reads its keys once per partition; here all readers but the first see one key
    changed (phobic_debug_change_key): moved to another partition, or, what no count can tell, to
    another place of its own partition.  The build of the keys as they then are is the oracle's."""
    torch = pytest.importorskip("torch")
    n = 9_000
    cfg = phobic.MPHFconfig(5.0, 2048)
    M = cfg.partitions(n)
    keys = keygen.splitmix64(73, n)

    def part(k):
        return (O.hash_keys(k, "u64")[:, 0].astype(np.uint64) * M >> np.uint64(32)).astype(int)

    old = part(keys)
    new = part(keys ^ np.uint64(0xFFFF))
    pick = {"down": (old > new) & (new > 0), "up": (old < new) & (old > 0), "from_first": (old == 0) & (new > 0),
            "to_first": (new == 0) & (old > 0), "same": (old == new) & (old > 0)}[way]
    index = int(np.flatnonzero(pick)[-1])
    dk = torch.from_numpy(keys.view(np.int64).copy()).cuda()
    with phobic.Context(0) as ctx:
        phobic.debug_change_key(index, 0xFFFF)
        with pytest.raises(phobic.PhobicError) as e:
            ctx.build(dk, cfg)
        assert e.value.status == phobic.ERR_KEYS_CHANGED
        now = dk.cpu().numpy().view(np.uint64)
        assert np.flatnonzero(now != keys).tolist() == [index] and now[index] == keys[index] ^ np.uint64(0xFFFF)
        got = ctx.build(now, cfg)
        want = O.build(O.hash_keys(now, "u64"), 2048, cfg.bucketCountPerPartition, cfg.getFulcs())
        assert got.timings["kernels"] == 2
        assert (got.pilots == want["pilots"]).all() and (got.partition_offsets == want["offsets"]).all()
