"""Host-side pieces of a step, without a GPU: the record a step's kernels read (ids, positions,
sequence of each token, first rows, tables; every part on a 16-byte boundary of one buffer) and
the replay loop's decisions (a slot a request, opened at its first step and given back at its end,
a file only where logits are wanted, one line a step)."""
import json
import os

import numpy as np
import pytest
import torch

from ultima_b200.engine.batch import DecodeRecord, build_step_batch
from ultima_b200.engine.trace import replay


def _tables(B, widths, seed=0):
    g = np.random.default_rng(seed)
    return [g.integers(0, 50, size=(B, w)).astype(np.int32) for w in widths]


def test_record_of_a_ragged_step():
    slots = [4, 0, 7]
    new = [[11, 12, 13, 14, 15], [21], [31, 32, 33]]
    before = [0, 70, 3]
    want = [0, 4, 5, 8]
    tables = _tables(3, [3, 2])
    b = build_step_batch(slots, new, before, want, tables, torch.device("cpu"))
    assert (b.n_tokens, b.n_seqs, b.max_new, b.max_after) == (9, 3, 5, 71)
    assert b.tok_ids.tolist() == [11, 12, 13, 14, 15, 21, 31, 32, 33]
    assert b.tok_seq.tolist() == [0, 0, 0, 0, 0, 1, 2, 2, 2]
    assert b.tok_pos.tolist() == [0, 1, 2, 3, 4, 70, 3, 4, 5]          # absolute positions: before + place
    assert b.seq_start.tolist() == [0, 5, 6, 9]
    assert b.seq_before.tolist() == before and b.seq_slot.tolist() == slots
    assert b.want_rows.tolist() == want
    for t, ref in zip(b.tables, tables):
        assert t.shape == ref.shape and np.array_equal(t.numpy(), ref)
    # one buffer, every part at a multiple of four 32-bit words (vector loads, bulk copies)
    base = b.tok_ids.data_ptr()
    for part in [b.tok_ids, b.tok_pos, b.tok_seq, b.seq_start, b.seq_before, b.seq_slot, b.want_rows] + b.tables:
        assert part.dtype == torch.int32 and (part.data_ptr() - base) % 16 == 0
    assert b.host["n_ints"] * 4 >= b.tables[-1].data_ptr() + b.tables[-1].numel() * 4 - base


def test_record_of_one_token_each_and_of_nothing_wanted():
    b = build_step_batch([2, 5], [[9], [8]], [63, 64], [], _tables(2, [4]), torch.device("cpu"))
    assert b.tok_pos.tolist() == [63, 64] and b.tok_seq.tolist() == [0, 1] and b.seq_start.tolist() == [0, 1, 2]
    assert b.want_rows.numel() == 0 and b.max_new == 1 and b.max_after == 65


def test_decode_record_keeps_its_layout_from_step_to_step():
    """The record of a captured decode step: the same places as ``build_step_batch`` makes for one
    token a sequence with every logit wanted, so a graph that was captured on it reads the right
    words after every update."""
    B, widths = 3, [2, 5]
    slots, before = [6, 1, 3], [10, 64, 127]
    tables = _tables(B, widths, seed=3)
    ref = build_step_batch(slots, [[5], [6], [7]], before, [0, 1, 2], tables, torch.device("cpu"))

    class Ring:                                           # stands in for the pinned buffers
        def take(self, n):
            return 0, torch.zeros(n, dtype=torch.int32)

        def copied(self, i):
            pass
    rec = DecodeRecord(B, widths, torch.device("cpu"), Ring())
    got = rec.update(slots, [5, 6, 7], before, tables)
    for name in ("tok_ids", "tok_pos", "tok_seq", "seq_start", "seq_before", "seq_slot", "want_rows"):
        assert getattr(got, name).tolist() == getattr(ref, name).tolist(), name
    for t, r in zip(got.tables, ref.tables):
        assert torch.equal(t, r)
    assert got.max_after == 128 and got.max_new == 1
    # the next step: same tensors (a graph holds their addresses), new contents
    again = rec.update(slots, [1, 2, 3], [11, 65, 128], tables)
    assert again.tok_ids.data_ptr() == got.tok_ids.data_ptr() and again.tok_ids.tolist() == [1, 2, 3]
    assert again.tok_pos.tolist() == [11, 65, 128] and again.max_after == 129


class ReplayEngine:
    """Logits are stand-ins: the row for a wanted place holds (slot, absolute position, token)."""

    def __init__(self, n_slots=3):
        self.free = list(range(n_slots))[::-1]
        self.held = {}
        self.steps, self.closed = [], []

    def open(self, n):
        assert n <= len(self.free), "more live requests than slots"
        got = [self.free.pop() for _ in range(n)]
        for s in got:
            self.held[s] = 0
        return got

    def close(self, slots):
        for s in slots:
            assert s in self.held, "slot given back twice"
            del self.held[s]
            self.free.append(s)
            self.closed.append(s)

    def step(self, slots, tokens, want):
        rows = []
        for s, t, w in zip(slots, tokens, want):
            assert s in self.held
            rows += [[s, self.held[s] + p, t[p]] for p in w]
            self.held[s] += len(t)
        self.steps.append((list(slots), [list(t) for t in tokens]))
        return torch.tensor(rows, dtype=torch.float32).reshape(len(rows), 3)

    def check_errors(self):
        pass


def test_replay_opens_a_slot_a_request_and_gives_it_back_at_its_end(tmp_path):
    lines = [
        {"step": 0, "entries": [{"id": "a", "tokens": [5, 17, 3], "want": [0, 2]},
                                {"id": "b", "tokens": [9], "want": []}], "end": []},
        {"step": 1, "entries": [{"id": "a", "tokens": [4], "want": [0]}, {"id": "b", "tokens": [8], "want": [0]}],
         "end": ["b"]},
        {"step": 2, "entries": [{"id": "a", "tokens": [6], "want": []}], "end": ["a", "never seen"]},
        # a second batch: its requests take the slots that came back
        {"step": 7, "entries": [{"id": "c", "tokens": [1, 2], "want": [1]}, {"id": "b", "tokens": [3], "want": [0]},
                                {"id": "d", "tokens": [4, 4, 4], "want": []}], "end": ["c", "b", "d"]},
    ]
    eng = ReplayEngine(n_slots=3)
    said = []
    n = replay(eng, [json.dumps(x) for x in lines] + ["", "  "], str(tmp_path), said.append)
    assert n == 4 and said == ["done 0", "done 1", "done 2", "done 7"]
    assert not eng.held and sorted(eng.free) == [0, 1, 2] and len(eng.closed) == 5
    # a request keeps its slot from step to step
    a_slot = eng.steps[0][0][0]
    assert eng.steps[1][0][0] == a_slot and eng.steps[2][0] == [a_slot]
    # files only where something was wanted, rows in the order of the entries and of ``want``
    assert sorted(os.listdir(tmp_path)) == ["0.f32", "1.f32", "7.f32"]
    f0 = np.fromfile(tmp_path / "0.f32", dtype="<f4").reshape(-1, 3)
    assert f0.tolist() == [[a_slot, 0, 5], [a_slot, 2, 3]]
    f1 = np.fromfile(tmp_path / "1.f32", dtype="<f4").reshape(-1, 3)
    b_slot = eng.steps[0][0][1]
    assert f1.tolist() == [[a_slot, 3, 4], [b_slot, 1, 8]]
    f7 = np.fromfile(tmp_path / "7.f32", dtype="<f4").reshape(-1, 3)
    assert [r[1:] for r in f7.tolist()] == [[1, 2], [0, 3]]             # "b" of the second batch starts at 0 again


def test_replay_stops_at_a_line_that_is_no_json(tmp_path):
    eng = ReplayEngine()
    with pytest.raises(json.JSONDecodeError):
        replay(eng, ['{"step": 0, "entries": [], "end": []}', "not json"], str(tmp_path), None)


def test_scratch_places_of_long_sequences_do_not_meet():
    """The records and chunks of the recurrent kernels: sequences from the length on that they are given lie apart and inside the
    scratch, whatever shorter ones lie between (first places as the kernels have them)."""
    import random

    from ultima_b200.kernels import ops
    rng = random.Random(3)
    for least, size, first, places in (
            (ops.DELTA_RECORDS_MIN, 4, lambda t: 9 * t >> 5, lambda T: ops.delta_records_floats(1, T, 1, 64, 16, ops.DELTA_RECORDS_MIN) // (13 * 64 + 32)),
            (ops.SSM_CHUNKS_MIN, 64, lambda t: 3 * t >> 7, lambda T: ops.ssm_chunk_places(1, T, 64, 128, ops.SSM_CHUNKS_MIN))):
        for n in range(least, 5 * least):                       # every length, from every residue
            for t in range(128):
                assert first(t + n) - first(t) >= -(-n // size)
        for _ in range(300):
            lens = [rng.choice([rng.randint(1, least - 1), rng.randint(least, 3 * least), least]) for _ in range(rng.randint(1, 40))]
            end, t = 0, 0
            for n in lens:
                if n >= least:
                    assert first(t) >= end
                    end = first(t) + -(-n // size)
                t += n
            assert end <= places(t)


def test_float32_attention_by_pages_leaves_what_its_grid_cannot_count():
    """Steps of more sequences than a grid has rows, and views off 16-byte boundaries, stay with the kernel that took them before."""
    from types import SimpleNamespace

    from ultima_b200.kernels import ops

    def fits(n_seqs, hd=64, shift=0):
        q = torch.zeros(n_seqs, 4 * hd + 4)[:, shift:shift + 4 * hd]
        pages = torch.zeros(1, 1, 64, hd)
        kv = SimpleNamespace(k=pages, v=pages, table=torch.zeros(n_seqs, 1, dtype=torch.int32), page=64)
        return ops.attn_f32_fits(q, kv, torch.zeros(n_seqs, 4 * hd), hd)
    assert fits(65535) and not fits(65536)
    assert not fits(3, shift=1) and not fits(3, hd=80)


# microseconds of the float32 product's forms on a chip of 148 multiprocessors, by tokens, weight rows and K
FORMS = {
    (780, 2048, 64): {32: 10.9, 64: 10.6, 128: 10.0, -32: 78.5, -64: 58.6},
    (100, 6144, 64): {32: 7.4, 64: 6.0, 128: 9.2, -32: 39.5, -64: 29.6},
    (389, 128, 256): {32: 13.3, 64: 17.1, 128: 30.1, -32: 6.5, -64: 8.1},
    (200, 2048, 512): {32: 41.9, 64: 33.0, 128: 57.6, -32: 31.4, -64: 24.3},
    (33, 6144, 512): {32: 38.5, 64: 33.0, 128: 57.2, -32: 26.3, -64: 21.5},
    (681, 512, 1024): {32: 74.8, 64: 63.9, 128: 111.7, -32: 42.2, -64: 33.0},
    (64, 2048, 2048): {32: 96.6, 64: 124.6, 128: 219.8, -32: 26.6, -64: 33.6},
    (681, 2048, 2048): {32: 260.8, 64: 250.1, 128: 224.3, -32: 253.4, -64: 177.9},
    (681, 6144, 2048): {32: 674.1, 64: 498.4, 128: 446.0, -32: 730.4, -64: 513.7},
    (100, 512, 6144): {32: 287.2, 64: 373.8, 128: 656.5, -32: 68.6, -64: 51.2},
    (389, 12288, 6144): {32: 2266.1, 64: 1842.7, 128: 1926.5, -32: 2416.5, -64: 1741.7},
}


@pytest.mark.parametrize("size", sorted(FORMS))
def test_the_float32_products_form_is_near_the_fastest_at_every_k(size):
    from ultima_b200.kernels import ops
    M, N, K = size
    form = ops.f32_form(M, N, K, ops.EPI_STORE, n_sms=148)
    assert FORMS[size][form] <= 1.12 * min(FORMS[size].values())


def test_the_float32_products_form_shares_k_only_where_there_are_slices():
    from ultima_b200.kernels import ops
    for M in (17, 40, 300, 3000):
        for N in (1, 64, 300, 32768):
            for epi in (ops.EPI_STORE, ops.EPI_ADD, ops.EPI_SWIGLU):
                assert ops.f32_form(M, N, 64, epi, n_sms=148) > 0 and ops.f32_form(9, N, 64, epi, n_sms=148) == 0
                assert ops.f32_form(M, N, 4096, epi, n_sms=148) in (32, 64, 128, -32, -64)
    assert [ops.f32_slice(k) for k in (4, 64, 68, 512, 516, 2048, 6144)] == [64, 64, 64, 64, 96, 256, 768]


@pytest.mark.parametrize("known", [True, False])
def test_portions_of_the_delta_rules_chunks_cover_a_step_and_fit_their_scratch(known):
    """Every token of every sequence of 512 or more in exactly one portion, portions begin at sixteens, and what a portion holds at any
    time fits the places; scratch follows neither tokens nor heads beyond what the records four at a time take."""
    from ultima_b200.kernels import ops
    rng = np.random.default_rng(3)
    for lens in ([2048], [512], [4096], [512] * 8, [2048] + [512] * 7, [40, 3000, 1, 511, 700, 512], [527, 528, 529] * 5,
                 [1] * 300 + [4000], rng.integers(1, 1500, 30).tolist()):
        lens = np.array(lens)
        T, B, longest = int(lens.sum()), len(lens), int(lens.max())
        long = lens[lens >= ops.DELTA_CHUNKS_MIN]
        for H, D, E in ((16, 128, 128), (64, 128, 128), (8, 64, 64), (64, 128, 256), (256, 128, 128)):
            floats = ops.delta_chunks_scratch(B, T, H, D, E)
            assert floats <= max(ops.DELTA_CHUNKS_SCRATCH // 4, ops.delta_records_floats(B, T, H, D, E, ops.DELTA_RECORDS_MIN))
            places = floats // (H * (73 * D + 36 * E))
            portions = ops.delta_chunk_portions(places, longest, B, T, ops.DELTA_CHUNKS_MIN, lens if known else None)
            seen = [0] * B
            for seq, seqs, first, most in portions:
                held = 0
                assert first % 16 == 0 and most >= 1 and 0 <= seq < seq + seqs <= B
                for b in range(seq, seq + seqs):
                    if lens[b] >= ops.DELTA_CHUNKS_MIN and lens[b] > first:
                        assert seen[b] == first
                        n = min(most, -(-(lens[b] - first) // 16))
                        seen[b], held = first + 16 * n, held + n
                assert 0 < held <= places
            assert all(s >= n if n >= ops.DELTA_CHUNKS_MIN else s == 0 for s, n in zip(seen, lens))
            if known and places >= sum(-(-n // 16) for n in long):
                assert len(portions) == 1


def test_a_long_steps_chunks_take_no_more_scratch_than_its_records():
    """4,096 tokens of 64 heads of 128 x 128: 0.5 GB of records; the chunks of the whole step would be 1.4 GB."""
    from types import SimpleNamespace as NS

    from ultima_b200.kernels import ops
    from ultima_b200.parts.delta import GatedDelta
    sizes = (64, 128, 128)
    assert ops.delta_chunks_floats(1, 4096, *sizes, ops.DELTA_CHUNKS_MIN) * 4 > 1.3e9
    asked = []

    class Arena:
        def mark(self):
            return 0

        def reset(self, mark):
            pass

        def alloc(self, shape, dtype):
            asked.append(int(np.prod(shape)) * 4)
            return torch.empty(shape, dtype=dtype, device="meta")
    part = GatedDelta(64, 64, 64, 128, 128, 4, decay_rank=8, gate_rank=8)
    rt = NS(dtype=torch.bfloat16, arena=Arena(), launches=0)
    batch = NS(n_seqs=1, max_new=4096, min_new=4096, host={"lens": np.array([4096])})
    calls = []
    old = ops.delta_scan_chunks
    ops.delta_scan_chunks = lambda *a, **k: calls.append(a) or 2
    try:
        part.recurrence(torch.empty(4096, 8192, device="meta"), None, None, None, None, None, None, batch, rt)
    finally:
        ops.delta_scan_chunks = old
    assert len(calls) == 1 and rt.launches == 2
    assert max(asked) <= 4 * ops.delta_records_floats(1, 4096, *sizes, ops.DELTA_RECORDS_MIN)


def test_the_float32_products_sums_follow_the_matrix_and_its_form_the_tokens():
    """Which sums a product has is a question of the matrix alone; which kernel forms them, of the tokens too
    (blocks for one and for two rounds of 148 multiprocessors, and one more, at the edges)."""
    import inspect

    from ultima_b200.kernels import ops
    assert list(inspect.signature(ops.f32_on_tensor_cores).parameters) == ["N", "K", "epilogue"]
    on = ops.f32_on_tensor_cores
    assert on(512, 1024, ops.EPI_STORE) and not on(511, 1024, ops.EPI_STORE) and not on(512, 1020, ops.EPI_STORE)
    assert on(256, 1024, ops.EPI_SWIGLU) and not on(8192, 252, ops.EPI_ADD) and on(2048, 256, ops.EPI_ADD)

    def form(M, N, K, epilogue=ops.EPI_STORE):
        return ops.f32_tc_form(M, N, K, epilogue, n_sms=148)
    assert [form(M, 2048, 2048) for M in (1, 8, 9, 16, 17, 48, 780)] == [4, 4, 3, 3, 3, 2, 0]
    assert [form(4, 16 * n, 4096) for n in (148, 149, 296, 297)] == [4, 3, 3, 2]
    assert [form(4, 8 * n, 4096, ops.EPI_SWIGLU) for n in (148, 149, 296, 297)] == [4, 3, 3, 2]
    assert [form(16, 4096, K) for K in (1024, 1792, 1796, 4096)] == [2, 2, 3, 3]
    assert [form(M, 4096, 4096) for M in (16, 17, 32, 33)] == [3, 1, 1, 1]
    assert [form(M, 32768, 2048) for M in (8, 16, 17, 681)] == [2, 2, 0, 0]
    assert form(681, 6144, 2048, ops.EPI_SWIGLU) == 0 and form(681, 2048, 6144) == 1 and form(780, 2048, 6144) == 0


def test_the_float32_products_scratch_is_bounded(monkeypatch):
    """4,096 tokens of 12,288 columns: 0.3 GB of parts, which go in portions of 64 MB; every token in one of them, in whole tiles.  Each is
    a launch for the parts and one for the product, the few tokens' kernel one, as the runtime counts them."""
    from types import SimpleNamespace as NS

    from ultima_b200.kernels import ops
    asked, calls = [], []
    rt = NS(launches=0, arena=NS(mark=lambda: 0, reset=lambda mark: None,
                     alloc=lambda shape, dtype: asked.append(shape) or torch.empty(shape, dtype=dtype, device="meta")))
    monkeypatch.setattr(ops, "_lib", lambda name: NS(ub_gemm_f32_tc=lambda *x: calls.append(x) or 0))
    monkeypatch.setattr(ops, "_ptr", lambda t: t)
    monkeypatch.setattr(ops, "_stream", lambda: None)
    monkeypatch.setattr(ops, "status_ptr", lambda rt: None)
    monkeypatch.setattr(ops, "sm_count", lambda: 148)
    for M, K in ((4096, 12288), (700, 2048), (20000, 100)):
        asked.clear(), calls.clear()
        a, w, out = (torch.empty(s, device="meta") for s in ((M, K), (4096, K), (M, 4096)))
        rt.launches = 1
        ops.gemm_f32_tc(a, w, out, ops.EPI_STORE, None, rt, 0)
        assert rt.launches == 2 * len(calls)
        assert all(2 * int(np.prod(s)) <= 64 << 20 for s in asked)
        at = 0
        for c in calls:
            x, y, rows = c[0], c[3], c[5]
            assert x.shape == (rows, K) and y.shape == (rows, 4096) and x.storage_offset() == at * K and y.storage_offset() == at * 4096
            assert rows <= asked[0][1] and (rows % 128 == 0 or at + rows == M)
            at += rows
        assert at == M and (len(calls) > 1) == (M == 4096)
    rt.launches = 1
    ops.gemm_f32_tc(a[:9], w, out[:9], ops.EPI_STORE, None, rt)
    assert rt.launches == 1


@pytest.mark.parametrize("lens", [[2048], [2048, 1, 1], [31, 600], [32, 600], [511], [40, 1, 512], [1, 1], [31]])
def test_the_delta_rules_forms_are_launched_for_the_sequences_that_take_them(lens, monkeypatch):
    """Token by token below 32 tokens, four at a time up to 511, sixteen from 512: a form that no sequence of the step takes is not launched."""
    from types import SimpleNamespace as NS

    from ultima_b200.kernels import ops
    from ultima_b200.parts.delta import GatedDelta
    part = GatedDelta(64, 2, 2, 64, 64, 4, decay_rank=8, gate_rank=8)
    arena = NS(mark=lambda: 0, reset=lambda mark: None, alloc=lambda shape, dtype: torch.empty(shape, dtype=dtype, device="meta"))
    called = []
    for name, n in (("delta_scan", None), ("delta_scan_records", None), ("delta_scan_chunks", 2)):
        monkeypatch.setattr(ops, name, lambda *a, _name=name, _n=n, **k: called.append(_name) or _n)
    rt = NS(dtype=torch.bfloat16, arena=arena, launches=0)
    batch = NS(n_seqs=len(lens), max_new=max(lens), min_new=min(lens), host={"lens": np.array(lens)})
    part.recurrence(torch.empty(sum(lens), 128, device="meta"), None, None, None, None, None, None, batch, rt)
    want = {"delta_scan": min(lens) < 32, "delta_scan_records": any(32 <= n < 512 for n in lens), "delta_scan_chunks": max(lens) >= 512}
    assert sorted(called) == sorted(k for k, v in want.items() if v)
    assert rt.launches == want["delta_scan"] + 2 * want["delta_scan_records"] + 2 * want["delta_scan_chunks"]
