"""A sequence's block table on its way to the device: pinned rows that take turns, copied by streams that run as late as they may."""
import pytest
import torch

from rmlx_b200.kv.paged import PagedKvCache


class _Stream:
    """Does its queue only when somebody waits for it."""

    def __init__(self):
        self.queue, self.done = [], 0

    def run_to(self, n):
        while self.done < n:
            self.done += 1
            self.queue[self.done - 1]()

    def put(self, what):
        self.queue.append(what)

    def wait_event(self, event):
        self.put(event.synchronize)


class _Event:
    def record(self, stream):
        self.stream, self.at = stream, len(stream.queue)

    def synchronize(self):
        self.stream.run_to(self.at)


class _Device:
    """The device's table: a copy into a row is queued on the current stream and reads its source when it runs."""

    def __init__(self, table, current):
        self.table, self.current = table, current

    def __getitem__(self, slot):
        class Row:
            def copy_(_, src, non_blocking=False):
                assert non_blocking
                self.current[0].put(lambda: self.table[slot].copy_(src))
        return Row()


@pytest.fixture
def cache(monkeypatch):
    c = PagedKvCache(64, 1, 1, 64, max_seqs=2, max_blocks_per_seq=32)
    c.streams = [_Stream(), _Stream()]
    c.current = [c.streams[0]]
    c.on_device = c.block_table
    c.block_table, c.device = _Device(c.on_device, c.current), torch.device("cuda")
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: c.current[0])
    monkeypatch.setattr(torch.cuda, "Event", _Event)
    return c


def _look(cache, seen, seq):
    """What a kernel launched now on the current stream will find in the sequence's row, beside what it has to find."""
    slot, blocks = cache.slot_of[seq], list(cache.manager.block_table(seq))
    cache.current[0].put(lambda: seen.append((cache.on_device[slot, :len(blocks)].tolist(), blocks)))


def _all(cache):
    for s in cache.streams:
        s.run_to(len(s.queue))


def test_updates_behind_a_busy_stream(cache):
    """Every launch finds the table of its time, however many updates are queued, though pages given back go to another sequence; up to four
    updates wait for nothing."""
    cache.add_sequence(0)
    cache.add_sequence(1)
    seen = []
    for i in range(7):
        cache.reserve(0, 48)
        cache.commit(0, 48)
        _look(cache, seen, 0)
        cache.trim(0, 32)
        _look(cache, seen, 0)
        assert i > 1 or not seen
        cache.reserve(1, 16)                 # takes one of the pages
        cache.commit(1, 16)
    _all(cache)
    assert len(seen) == 14 and all(got == want for got, want in seen)


@pytest.mark.parametrize("first", [0, 1])
def test_updates_from_two_streams(cache, first):
    """They reach the device in the order in which they were made, whichever stream runs first."""
    cache.add_sequence(0)
    seen = []
    for i in range(9):
        cache.current[0] = cache.streams[i % 2 if i < 7 else 1]
        cache.reserve(0, 16)
        cache.commit(0, 16)
        _look(cache, seen, 0)
    for s in (cache.streams if first == 0 else cache.streams[::-1]):
        s.run_to(len(s.queue))
    assert cache.on_device[cache.slot_of[0], :9].tolist() == list(cache.manager.block_table(0))
    assert all(got[:len(want)] == want for got, want in seen)


def test_slot_taken_again_while_copies_are_queued(cache):
    """The next sequence of a slot starts from zeros and its tables follow those of the one before."""
    seen = []
    for seq in range(5):
        cache.add_sequence(seq)
        slot = cache.slot_of[seq]
        assert not cache._host_table[slot].any()
        for n in range(1 + seq % 3):
            cache.reserve(seq, 16 * (3 - n))
            cache.commit(seq, 16 * (3 - n))
            _look(cache, seen, seq)
        cache.free_sequence(seq)
    _all(cache)
    assert len(seen) == 9 and all(got == want for got, want in seen)
