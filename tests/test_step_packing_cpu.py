"""How a step's index arrays are packed, without a GPU: the batch's own arrays, one block table per
page group, and the arrays of every planner that the cache's users bring (the step function does
not know what they mean).  And what the engine does when a step raises."""
import numpy as np
import pytest
import torch

from mini_hisparse_b200.cache import CacheConfig, CacheManager
from mini_hisparse_b200.engine.step import BatchBuilder, StepEntry, StepError
from mini_hisparse_b200.parts import PartSpec, StepPlanner
from mini_hisparse_b200.parts.attention import ITEM_INTS, GQAttention
from mini_hisparse_b200.parts.spec import PagedKVNeed, PagedNeed, StateNeed
from dataclasses import dataclass


class CountingPlanner(StepPlanner):
    """A planner of a made-up mixer: one word per segment (its first position) and a running index."""

    def capacity(self, max_tokens, max_segments, fixed=None):
        return {"seg_first": max_segments, "tok_index": max_tokens + 3}

    def plan(self, segments, T, fixed=None):
        return ({"seg_first": np.asarray([s.start for s in segments], np.int32),
                 "tok_index": np.arange(T, dtype=np.int32)}, {"count": len(segments)})


class MadeUpMixer:
    def __init__(self, key):
        self.key = key

    def plan_key(self):
        return self.key

    def planner(self, page_size, sm_count):
        return CountingPlanner()


@dataclass(frozen=True)
class LatentNeed(PagedNeed):
    """A paged need with a page shape of its own: one vector of ``width`` per position."""

    width: int = 8
    window: int | None = None

    def page_shape(self, page_size):
        return (page_size, self.width)


def attention(nq, nkv, d=16):
    return GQAttention(PartSpec.make("gq_attention", hidden_size=32, q_heads=nq, kv_heads=nkv, head_dim=d,
                                     position=PartSpec.make("none")))


def test_packing_with_several_groups_and_planners():
    a4, a8 = attention(4, 2), attention(8, 2)          # same keys and values, other query heads
    needs = [a4.cache_need(), a8.cache_need(), LatentNeed(width=8), StateNeed((5,)), None]
    cache = CacheManager(needs, CacheConfig(num_pages=20, page_size=4, max_requests=3, dtype=torch.float32,
                                            device="cpu", allocate_storage=False))
    # equal needs share a pool and a block table whatever their query heads; the latent pages are a group of their own
    assert len(cache.page_groups) == 2 and len(cache.state_groups) == 1
    assert cache.page_groups[0].entries == [0, 1] and cache.page_groups[0].page_shape == (2, 2, 4, 16)
    assert cache.page_groups[1].page_shape == (4, 8) and cache.page_groups[1].page_bytes() == 4 * 8 * 4
    batch = BatchBuilder(cache, "cpu", sm_count=8)
    users = [batch.add_user(0, a4), batch.add_user(1, a8), batch.add_user(0, a4), batch.add_user(2, MadeUpMixer("m")),
             batch.add_user(3, MadeUpMixer("m")), batch.add_user(4, None)]
    # plans: one per (group, plan key): a4 (twice the same), a8, the made-up one over pages, and the made-up
    # one over the state group (a state's user may plan too: its group is another one); None plans nothing
    assert len(batch.slots) == 4 and [batch.users[u][1] for u in users] == [0, 1, 0, 2, 3, None]
    for name in ("x", "y"):
        cache.open(name)
    cache.ensure("x", 9), cache.advance("x", 9)
    entries = [StepEntry("x", [5, 6, 7], [0, 2]), StepEntry("y", [1, 2, 3, 4, 5, 6], [5])]
    segments, T = batch.segments(entries)
    assert T == 9 and [(s.start, s.count, s.offset) for s in segments] == [(9, 3, 0), (0, 6, 3)]
    for s in segments:
        cache.ensure(s.request, s.start + s.count)
    views = batch.eager(entries, segments)
    assert views["tokens"].tolist() == [5, 6, 7, 1, 2, 3, 4, 5, 6]
    assert views["positions"].tolist() == [9, 10, 11, 0, 1, 2, 3, 4, 5]
    assert views["tok_seg"].tolist() == [0, 0, 0, 1, 1, 1, 1, 1, 1]
    assert views["rows"].tolist() == [0, 2, 8]
    for gi, g in enumerate(cache.page_groups):
        table = views["tables"][gi]
        assert table.shape == (2, 3)                                   # 12 positions of 4 per page
        assert table[0].tolist() == g.tables[cache.slot("x")].pages
        assert table[1].tolist() == g.tables[cache.slot("y")].pages + [-1]
    v4, v8, vm = (batch.cache_view(u, views) for u in (users[0], users[1], users[3]))
    assert v4.meta["block_table"] is not None and v4.meta["n_small"] + v4.meta["n_big"] >= 2
    items4 = v4.meta["items"].view(-1, ITEM_INTS)[: v4.meta["n_small"] + v4.meta["n_big"]]
    items8 = v8.meta["items"].view(-1, ITEM_INTS)[: v8.meta["n_small"] + v8.meta["n_big"]]
    assert int(items4[:, 4].max()) == 2 and int(items8[:, 4].max()) == 4   # heads per KV group differ
    assert batch.cache_view(users[2], views).meta["items"].data_ptr() == v4.meta["items"].data_ptr()
    assert vm.meta["seg_first"].tolist() == [9, 0] and vm.meta["count"] == 2
    assert vm.meta["tok_index"].tolist() == list(range(9)) + [0, 0, 0]      # the rest of its capacity is zeroed
    assert vm.storage is None and vm.page_size == 4
    vs = batch.cache_view(users[4], views)
    assert vs.meta["seg_first"].tolist() == [9, 0] and vs.meta["count"] == 2 and "block_table" not in vs.meta
    assert batch.cache_view(users[5], views) is None


def test_a_plan_larger_than_its_capacity_is_refused():
    class Liar(CountingPlanner):
        def capacity(self, max_tokens, max_segments, fixed=None):
            return {"seg_first": 0, "tok_index": max_tokens}

    class LiarMixer(MadeUpMixer):
        def planner(self, page_size, sm_count):
            return Liar()

    cache = CacheManager([LatentNeed()], CacheConfig(num_pages=4, page_size=4, max_requests=2, dtype=torch.float32,
                                                     device="cpu", allocate_storage=False))
    batch = BatchBuilder(cache, "cpu", sm_count=8)
    batch.add_user(0, LiarMixer("l"))
    cache.open("x")
    entries = [StepEntry("x", [1, 2], [])]
    segments, _ = batch.segments(entries)
    cache.ensure("x", 2)
    with pytest.raises(StepError, match="seg_first"):
        batch.eager(entries, segments)


def test_engine_fails_the_requests_of_a_step_that_raised():
    """Engine.step with a runner whose status check raises: the step's requests end as failed, their
    pages come back, the runner is told to put its scratch back, and the next step serves the rest."""
    from mini_hisparse_b200.engine.engine import Engine
    from mini_hisparse_b200.engine.scheduler import Scheduler, SchedulerConfig

    cache = CacheManager([PagedKVNeed(2, 16)], CacheConfig(num_pages=16, page_size=4, max_requests=4,
                                                           dtype=torch.float32, device="cpu", allocate_storage=False))

    class FakeRunner:
        def __init__(self):
            self.fail_next = False
            self.resets = 0
            self.stats = {}
            self.device_tokens_seen = 0

        use_graphs = True

        def step(self, entries, device_tokens=None):
            self.device_tokens_seen += device_tokens is not None
            for e in entries:                  # what the real runner does before and after its launches
                cache.ensure(e.request, cache.length(e.request) + len(e.tokens))
                cache.advance(e.request, len(e.tokens))
            return torch.zeros(sum(len(e.want) for e in entries), 50) if any(e.want for e in entries) else None

        def queue_status(self):
            pass

        def prepare_decode_ahead(self, requests):
            pass

        def check_status(self, queued=False):
            if self.fail_next:
                self.fail_next = False
                raise StepError("a bounded wait in the tensor-core matrix product ran out")

        def reset_after_error(self):
            self.resets += 1

    class FakeSampler:
        """Tickets as the real one; request i's k-th token is 10 i + k (from the counter it is given)."""

        def __init__(self):
            self.rows = {}
            self.ticket = 0

        def launch(self, logits, temps, seeds, counters):
            self.ticket += 1
            self.rows[self.ticket] = [3 + c for c in counters]
            return self.ticket

        def device_tokens(self, ticket):
            return torch.tensor(self.rows[ticket], dtype=torch.int32)

        def reset(self):
            self.rows.clear()

        def collect(self, ticket):
            return self.rows.pop(ticket)

    def make_engine(pipeline):
        from collections import deque

        engine = object.__new__(Engine)
        engine.cache, engine.runner, engine.sampler, engine.timeline = cache, FakeRunner(), FakeSampler(), []
        engine.scheduler = Scheduler(cache, SchedulerConfig(max_tokens_per_step=6), 50, eos_token_id=6)
        engine.pipeline, engine._queued, engine.launch_log, engine.launches = pipeline, None, deque(maxlen=8), 0
        engine.stats = {"queued_steps": 0, "dropped_tokens": 0}
        engine.model = None
        return engine

    engine = make_engine(pipeline=False)
    engine.add_request("a", [1, 2, 3], max_new_tokens=3)
    engine.add_request("b", [4, 5], max_new_tokens=3)
    engine.add_request("c", [6, 7, 8, 9], max_new_tokens=2)
    assert [t for _, t in engine.step()] == [3, 3]          # a and b whole, the first token of c
    engine.runner.fail_next = True
    with pytest.raises(StepError, match="bounded wait"):
        engine.step()                                       # a, b decode, c prefills: all three fail
    assert engine.runner.resets == 1
    assert all(engine.requests[n].failed for n in "abc") and not cache.requests
    cache.assert_invariants()
    assert cache.snapshot()["page_groups"][0]["pages_free"] == 16
    engine.add_request("d", [1, 2], max_new_tokens=2)       # the engine goes on
    assert engine.run()["d"] == [3, 4]

    # Decode steps queued behind one another: a step's tokens reach the host's books one call later,
    # every call returns one step's tokens, and a request that draws its end token (6 = 3 + 3) while
    # the next step is already queued costs one dropped token and no more.
    engine = make_engine(pipeline=True)
    engine.add_request("x", [1, 2], max_new_tokens=8)
    engine.add_request("y", [4], max_new_tokens=5)
    out = []
    while not engine.scheduler.idle or engine._queued is not None:
        out.append(engine.step())
    assert engine.requests["x"].generated == [3, 4, 5, 6]        # ended by its end token, kept
    assert engine.requests["y"].generated == [3, 4, 5, 6]
    assert [len(o) for o in out[:4]] == [2, 2, 2, 2] and all(len(o) == 0 for o in out[4:])
    assert engine.stats["queued_steps"] >= 2 and engine.stats["dropped_tokens"] == 2
    assert engine.runner.device_tokens_seen == engine.stats["queued_steps"]
    assert not cache.requests
    cache.assert_invariants()
    assert cache.snapshot()["page_groups"][0]["pages_free"] == 16


def test_status_bits_have_messages():
    """Every bit a kernel can set has a text, several bits give several texts, unknown bits are named."""
    from mini_hisparse_b200.engine.step import ModelRunner

    for bit, text in ModelRunner.STATUS_BITS.items():
        assert ModelRunner.status_message(bit) == text
    both = ModelRunner.status_message(4 | 8)
    assert "matrix product" in both and "TMA-fed attention" in both
    assert "0x40" in ModelRunner.status_message(64 | 1) and "vocabulary" in ModelRunner.status_message(64 | 1)


@pytest.mark.parametrize("fixed", [(1, 1), (4, 1)])
@pytest.mark.parametrize("window", [None, 40])
def test_decode_arrays_written_again_into_a_graphs_buffers(fixed, window):
    """The buffers of a captured decode step are written in place step after step: every word is what a buffer written for the
    first time holds, and the plan's words are plan_decode's, whichever buffer of the ring has its turn."""
    from mini_hisparse_b200.engine.step import _DecodeBuffers, _Layout

    part = GQAttention(PartSpec.make("gq_attention", hidden_size=32, q_heads=40, kv_heads=2, head_dim=16, window=window,
                                     position=PartSpec.make("none")))
    cache = CacheManager([part.cache_need()], CacheConfig(num_pages=80, page_size=4, max_requests=3, dtype=torch.float32,
                                                          device="cpu", allocate_storage=False))
    batch = BatchBuilder(cache, "cpu", sm_count=8)
    batch.add_user(0, part)
    for name, n in zip("abc", (70, 1, 33)):
        cache.open(name), cache.ensure(name, n), cache.advance(name, n)
    planner = batch.slots[0].planner
    caps = [planner.capacity(3, 3, fixed)]
    layout = _Layout(3, 3, 3, [32], caps)
    ring = _DecodeBuffers(layout, torch.device("cpu"))
    for step in range(2 * ring.ring + 3):
        entries = [StepEntry(r, [step + i], [0]) for i, r in enumerate("cab")]
        segments, _ = batch.segments(entries)
        for s in segments:
            cache.ensure(s.request, s.start + 1)
        starts = np.asarray([s.start for s in segments])
        turn, fresh = ring.next(), _DecodeBuffers(layout, torch.device("cpu"))
        facts = batch._fill_decode(ring.views[turn], entries, segments, [fixed], starts)
        assert turn == step % ring.ring and facts == batch._fill_decode(fresh.views[0], entries, segments, [fixed], starts)
        assert torch.equal(ring.rows[turn], fresh.rows[0])
        arrays, plain = planner.plan_decode(starts, fixed)
        assert facts == [plain]
        for name, words in ring.views[turn]["plans"][0].items():
            assert np.array_equal(words, arrays[name].reshape(-1))
        assert ring.views[turn]["tables"][0].tolist() == cache.table_rows(0, [s.slot for s in segments], 32).tolist()
        for r in "abc":
            cache.advance(r, 1)


def test_a_decode_buffer_whose_plan_could_not_be_written(monkeypatch):
    """A plan of another size than the graph's layout is refused as a StepError, and what a planner that raised has left in the
    buffer does not count as written: the next step in its turn writes every word."""
    from mini_hisparse_b200.engine.step import _DecodeBuffers, _Layout

    part = attention(4, 2)
    cache = CacheManager([part.cache_need()], CacheConfig(num_pages=20, page_size=4, max_requests=2, dtype=torch.float32,
                                                          device="cpu", allocate_storage=False))
    batch = BatchBuilder(cache, "cpu", sm_count=8)
    batch.add_user(0, part)
    cache.open("a"), cache.ensure("a", 7), cache.advance("a", 6)
    planner, entries = batch.slots[0].planner, [StepEntry("a", [1], [0])]
    segments, _ = batch.segments(entries)
    layout, starts = _Layout(1, 1, 1, [16], [planner.capacity(1, 1, (1, 1))]), np.asarray([6])
    ring, fresh = (_DecodeBuffers(layout, torch.device("cpu")) for _ in range(2))
    write = type(planner).plan_decode

    def fails(self, starts, fixed):
        raise KeyError("a planner's own trouble")

    for plan, error in ((fails, KeyError), (lambda self, starts, fixed: write(self, starts, (2, 1)), StepError)):
        monkeypatch.setattr(type(planner), "plan_decode", plan)
        with pytest.raises(error):
            batch._fill_decode(ring.views[0], entries, segments, [(1, 1)], starts)
    monkeypatch.setattr(type(planner), "plan_decode", write)
    for buffers in (ring, fresh):
        batch._fill_decode(buffers.views[0], entries, segments, [(1, 1)], starts)
    assert torch.equal(ring.rows[0], fresh.rows[0])


def test_a_planner_derived_from_attentions_writes_its_own_plan_every_step():
    """The short cut that moves only the ends of the key ranges is for AttentionPlanner's own plans."""
    from mini_hisparse_b200.parts.attention import AttentionPlanner, AttentionShape

    class Backwards(AttentionPlanner):
        def plan_decode(self, starts, fixed):
            arrays, facts = super().plan_decode(starts, fixed)
            return dict(arrays, tok_part_row=(1000 + starts).astype(np.int32)), facts

    planner = Backwards(AttentionShape(4, 2), 8)
    regions = {name: np.zeros(n, np.int32) for name, n in planner.capacity(2, 2, (1, 1)).items()}
    for step in range(3):
        planner.write_decode(np.asarray([step, 9]), (1, 1), regions, step == 0)
        assert regions["tok_part_row"].tolist() == [1000 + step, 1009]


@pytest.mark.parametrize("pages,kernel", [(1 << 20, "attention_tokens"), ((1 << 29) - 1, "attention_tokens"), (1 << 29, "attention_simt")])
def test_pools_beyond_32_bit_rows_go_to_the_kernel_that_takes_them(monkeypatch, pages, kernel):
    """Decoded tokens over a pool of 2^31 rows and more: the kernel whose offsets are 64 bits wide, as before there was the other."""
    from types import SimpleNamespace

    from mini_hisparse_b200.kernels import api as K
    from mini_hisparse_b200.parts.base import Product

    part, ran = attention(2, 1), []
    part.rt, part.qkv_weight, part.o_weight = SimpleNamespace(dtype=torch.float32), None, None
    for name in ("attention_tokens", "attention_simt", "attention_rows", "attention_combine"):
        monkeypatch.setattr(K, name, lambda *a, name=name, **k: ran.append(name))
    rt = SimpleNamespace(dtype=torch.float32, linear=lambda *a, **k: Product(torch.zeros(1)), qkv_rope_append=lambda *a, **k: True)
    ctx = SimpleNamespace(rt=rt, ws=SimpleNamespace(get=lambda name, shape, dtype: torch.zeros(shape, dtype=dtype)), positions=None,
                          status=None, extras={})
    _, facts = part.planner(2, 148).plan_decode(np.asarray([5]), (1, 1))
    view = SimpleNamespace(meta=dict(facts, block_table=None, items=None, tok_part_row=None), page_size=2, writable=True,
                           storage=torch.empty(pages, 2, 1, 2, 16, device="meta"))
    part.forward(torch.zeros(1, 32), ctx, view)
    assert ran == [kernel]


class LazyGPU:
    """Streams that run what is queued on them as late as they may: at a synchronise, and at the end.  A copy remembers what its
    source held when it was queued, and looks again when it runs."""

    def __init__(self):
        self.queues, self.stream, self.stale, self.copies = {}, 1, 0, 0

    def queue(self, what):
        self.queues.setdefault(self.stream, []).append(what)

    def run(self, stream, until=None):
        queue = self.queues.get(stream, [])
        while queue:
            op = queue.pop(0)
            if op is until:
                return
            if not isinstance(op, Recorded):
                source, held = op
                self.stale += not torch.equal(source, held)

    def synchronize(self, device=None):
        for s in list(self.queues):
            self.run(s)

    def copy_(self, source, non_blocking=False):
        self.copies += 1
        self.queue((source, source.clone()))


class Recorded:
    pass


def lazy_gpu(monkeypatch):
    gpu = LazyGPU()

    class Event:
        def record(self, stream=None):
            self.at = (gpu.stream, Recorded())
            gpu.queue(self.at[1])

        def synchronize(self):
            if self.at[1] in gpu.queues.get(self.at[0], []):
                gpu.run(self.at[0], self.at[1])

    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(torch.cuda, "synchronize", gpu.synchronize)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: gpu.stream, raising=False)
    monkeypatch.setattr(torch.Tensor, "pin_memory", lambda t: t)
    return gpu


@pytest.mark.parametrize("width,ring", [(16, 8), (8192, 2)])
@pytest.mark.parametrize("where", ["one stream", "packed elsewhere", "steps change streams", "dropped"])
def test_no_host_buffer_is_written_while_its_copy_is_queued(monkeypatch, width, ring, where):
    """A captured graph's steps queued without waiting for any of them: packed at the step or ahead of it, on the stream of the
    step or on another, packed ahead and dropped, and steps that change streams.  Every copy finds what it was queued for."""
    from mini_hisparse_b200.engine.step import ModelRunner, _Layout

    gpu = lazy_gpu(monkeypatch)
    part = attention(4, 2)
    cache = CacheManager([part.cache_need()], CacheConfig(num_pages=8200, page_size=16, max_requests=3, dtype=torch.float32,
                                                          device="cpu", allocate_storage=False))
    runner = ModelRunner.__new__(ModelRunner)
    runner.cache, runner.device, runner.use_graphs, runner.graph_after = cache, torch.device("cuda", 0), True, 1
    runner.model = type("Model", (), {"spec": type("Spec", (), {"max_positions": None})})
    runner.batch = BatchBuilder(cache, "cpu", sm_count=8)
    runner.batch.add_user(0, part)
    runner.stats, runner._ahead = {"prepared_steps": 0, "graph_steps": 0}, None
    runner._table_width = lambda last: width
    lengths = dict(a=1, b=9, c=40)
    for name, n in lengths.items():
        cache.open(name), cache.ensure(name, n), cache.advance(name, n)
    key = runner._graph_key(runner.batch.segments([StepEntry(r, [0], [0]) for r in "abc"])[0], np.asarray([1, 9, 40]))
    layout = _Layout(3, 3, 3, [width], [runner.batch.slots[0].planner.capacity(3, 3, key[2][0])])
    graph = type("Graph", (), dict(layout=layout, fixed=list(key[2]), capturable=True, facts=None, meta=gpu, launches=0, logits=None,
                                   buffers=None, graph=type("Exec", (), {"replay": lambda self: None})()))()
    runner.graphs = {key: graph}
    for step in range(4 * 8):
        requests = ["abc", "bca", "cab"][step % 3]
        if step and (where == "packed elsewhere" or where == "dropped" and step % 5 < 3):
            gpu.stream = 1
            for _ in range(1 if where == "packed elsewhere" else 3):
                runner.prepare_decode_ahead(list(requests))
            assert runner._ahead is not None
        ahead, runner._ahead = runner._ahead, None
        entries = [StepEntry(r, [step + i], [0]) for i, r in enumerate(requests[::-1] if where == "dropped" else requests)]
        segments, _ = runner.batch.segments(entries)
        for s in segments:
            cache.ensure(s.request, s.start + 1)
        gpu.stream = {"packed elsewhere": 2, "steps change streams": 1 + step // 3 % 2}.get(where, 1)
        runner._step_graph(entries, segments, ahead)
        for r in "abc":
            cache.advance(r, 1)
    assert graph.buffers.ring == ring and gpu.copies == 32 and runner.stats["prepared_steps"] == (31 if where == "packed elsewhere" else 0)
    gpu.synchronize()
    assert gpu.stale == 0
