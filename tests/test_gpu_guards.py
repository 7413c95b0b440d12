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


def test_calls_after_a_timeout_leave_the_queued_build_alone(phobic, monkeypatch):
    """A build that timed out stays queued and still reads its pinned tables.  Calls that follow
    (a query with another configuration, a build of other keys) wait for it, time out like it
    while it is held back, and neither disturb it nor take over its status.  The work is held
    back by a bounded sleep kernel on the context's stream (about 0.3 s)."""
    torch = pytest.importorskip("torch")
    cfg, other = phobic.MPHFconfig(7.0, 2500), phobic.MPHFconfig(4.0, 1000)
    keys, twice = keygen.splitmix64(81, 100_000), keygen.splitmix64(82, 100_000)
    twice[9] = twice[8]

    def oracle(k, c):
        return O.build(O.hash_keys(k, "u64"), c.partitionSize, c.bucketCountPerPartition, c.getFulcs())

    want, want_other = oracle(keys, cfg), oracle(keys, other)
    dk, dt = (torch.from_numpy(k.view(np.int64)).cuda() for k in (keys, twice))

    def arrays(c):
        m = c.partitions(len(keys))
        return (torch.zeros(m * c.bucketCountPerPartition, dtype=torch.int32, device="cuda"),
                torch.zeros(m + 1, dtype=torch.int32, device="cuda"))

    def same(out, w):
        return ((out[0].cpu().numpy().view(np.uint32) == w["pilots"]).all()
                and (out[1].cpu().numpy().view(np.uint32) == w["offsets"]).all())

    first, late, built = arrays(cfg), arrays(cfg), arrays(other)
    with phobic.Context(0) as warm:  # loads every kernel
        r_other = warm.build(dk, other, out=built)
        slots = warm.query(dk, other, r_other)
        warm.build(dk, cfg, out=late)
        phobic.encode_gpu(warm, r_other, other, "interleaved_compact", "diff")
    assert same(built, want_other)
    monkeypatch.setenv("PHOBIC_TIMEOUT_MS", "40")
    with phobic.Context(0) as ctx:
        monkeypatch.delenv("PHOBIC_TIMEOUT_MS")
        for _ in range(2):  # arenas at their sizes
            ctx.build(dk, cfg, out=late)
            assert torch.equal(ctx.query(dk, other, r_other), slots)
        for t in late:
            t.zero_()
        torch.cuda.synchronize()

        def timed_out(call):
            with pytest.raises(phobic.PhobicError) as e:
                call()
            assert e.value.status == phobic.ERR_TIMEOUT

        with torch.cuda.stream(torch.cuda.ExternalStream(ctx.stream_handle())):
            torch.cuda._sleep(600_000_000)
        timed_out(lambda: ctx.build(dk, cfg, out=first))
        timed_out(lambda: ctx.query(dk, other, r_other))
        timed_out(lambda: ctx.build(dt, cfg, out=late))
        timed_out(lambda: phobic.encode_gpu(ctx, r_other, other, "interleaved_compact", "diff"))
        torch.cuda.synchronize()
        assert same(first, want)
        assert not late[0].any()  # never queued
        assert torch.equal(ctx.query(dk, other, r_other), slots)
        # A failing build left queued does not lend its status to the next one.
        with torch.cuda.stream(torch.cuda.ExternalStream(ctx.stream_handle())):
            torch.cuda._sleep(200_000_000)
        timed_out(lambda: ctx.build(dt, cfg, out=first))
        for _ in range(20):
            try:
                ctx.build(dk, cfg, out=late)
                break
            except phobic.PhobicError as e:
                assert e.status == phobic.ERR_TIMEOUT
        assert same(late, want)
