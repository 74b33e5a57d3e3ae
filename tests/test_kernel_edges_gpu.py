"""Kernels at the sizes where their tiles, chunks and slices begin and end, against float64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def _within(got, ref, rel, floor):
    """|got - ref| <= rel * |ref| + floor, element by element."""
    got, ref = got.double(), ref.double()
    assert got.shape == ref.shape and bool(torch.isfinite(got).all())
    worst = float(((got - ref).abs() - rel * ref.abs()).max())
    assert worst <= floor, worst


@pytest.mark.parametrize("kind", ["plain", "gelu", "relu2", "cap", "gate a row", "gate an element", "product", "product clamped",
                                  "product rectified", "product with a gate a row"])
@pytest.mark.parametrize("T,N", [(1, 200), (16, 128), (17, 130), (31, 256), (33, 300), (64, 136), (65, 264), (129, 200), (257, 392),
                                 (1100, 4000)])
def test_stored_products_at_the_edges_of_a_chunk_of_tokens(kind, T, N):
    """Rounding of a bfloat16 result is 2^-9 of it; float32 sums of 96 terms of size about 1/10 are off by less than 1e-4 (the
    functions' slopes here are below 8)."""
    from ultima_b200.engine import Runtime
    from ultima_b200.kernels import gemm_tc, ops
    rt = Runtime(DEV, torch.bfloat16)
    g = torch.Generator(device=DEV).manual_seed(T * 1000 + N)
    K = 96
    if kind.startswith("product"):
        N = -(-N // 128) * 128
    a = torch.randn(T, K, generator=g, device=DEV).bfloat16()
    w = (torch.randn(N, K, generator=g, device=DEV) * 0.1).bfloat16()
    z = a.double() @ w.double().T
    gates = torch.randn(T, N, generator=g, device=DEV)
    if kind.startswith("product"):
        gu = z.view(T, N // 128, 2, 64)
        gg, uu = gu[:, :, 0].reshape(T, N // 2), gu[:, :, 1].reshape(T, N // 2)
        limit, alpha, shift = {"product clamped": (0.7, 1.702, 1.0), "product rectified": (math.inf, math.inf, 0.0)}.get(
            kind, (math.inf, 1.0, 0.0))
        gg, uu = gg.clamp(max=limit), uu.clamp(-limit, limit)
        ref = (gg.clamp(min=0) if math.isinf(alpha) else gg * torch.sigmoid(alpha * gg)) * (uu + shift)
        out = torch.full((T, N // 2), math.nan, dtype=torch.bfloat16, device=DEV)
        mul = (gates[:, 3], 0) if kind.endswith("row") else None
        if mul:
            ref = ref * torch.sigmoid(gates[:, 3].double())[:, None]
        gemm_tc.gemm(a, w, out, ops.EPI_SWIGLU_IL, None, rt, gate=(limit, alpha, shift), mul=mul)
        _within(out, ref, 2.0 ** -8, 2e-3)
    else:
        unary = {"gelu": 1, "relu2": 2, "cap": 3}.get(kind)
        gate = gemm_tc.unary_constants(unary, 2.5) if unary else None
        mul = {"gate a row": (gates[:, 3], 0), "gate an element": (gates, 1)}.get(kind)
        ref = z
        if kind == "gelu":
            ref = 0.5 * z * (1 + torch.erf(z / math.sqrt(2)))
        elif kind == "relu2":
            ref = z.clamp(min=0) ** 2
        elif kind == "cap":
            ref = 2.5 * torch.tanh(z / 2.5)
        elif mul:
            ref = z * torch.sigmoid(gates[:, 3:4].double() if mul[1] == 0 else gates.double())
        for dt, rel, floor in ((torch.float32, 1e-5, 1e-3), (torch.bfloat16, 2.0 ** -8, 2e-3)):
            out = torch.full((T, N), math.nan, dtype=dt, device=DEV)
            gemm_tc.gemm(a, w, out, ops.EPI_STORE, None, rt, gate=gate, mul=mul)
            _within(out, ref, rel, floor)
    gemm_tc.check_error(rt)


@pytest.mark.parametrize("epilogue", ["store", "add", "product"])
@pytest.mark.parametrize("M,N,K", [(1, 33, 68), (4, 130, 260), (5, 17, 36), (8, 64, 512), (9, 72, 1028), (16, 129, 96), (17, 40, 2048),
                                   (33, 200, 516), (64, 128, 64), (65, 257, 72), (129, 130, 640), (200, 1032, 1024)])
def test_float32_products_have_one_order_of_sums_in_every_form(M, N, K, epilogue):
    """Every form, and the rows alone, give the same bits; a sum of K terms of size 1 / sqrt(K) in eight chains is off by at most
    (K / 8 + 8) 2^-24 of the sum of sizes (below 0.8 sqrt(K)), and in fact by far less."""
    from ultima_b200.kernels import ops
    g = torch.Generator(device=DEV).manual_seed(M * 7 + N + K)
    a = torch.randn(M, K + 4, generator=g, device=DEV)[:, 4:]                 # rows with a stride of their own
    w = torch.randn(2 * N, K, generator=g, device=DEV) * K ** -0.5
    x = torch.randn(M, N, generator=g, device=DEV)
    epi = {"store": ops.EPI_STORE, "add": ops.EPI_ADD, "product": ops.EPI_SWIGLU}[epilogue]
    w2 = w[N:] if epilogue == "product" else None
    ref = a.double() @ w[:N].double().T
    if epilogue == "add":
        ref = ref + x.double()
    elif epilogue == "product":
        ref = torch.nn.functional.silu(ref) * (a.double() @ w[N:].double().T)
    assert ops.f32_fits(a, w[:N], x, epi, w2)
    first = None
    for form in ([0] if M <= 16 else []) + [32, 64, 128, -32, -64, -128]:
        out = x.clone()
        ops.gemm_f32(a, w[:N], out, epi, w2, form=form)
        if first is None:
            first = out
            _within(out, ref, 1e-5, (K / 8 + 8) * 2.0 ** -24 * 0.8 * K ** 0.5 * 8)
        assert torch.equal(out, first), form
    out = x.clone()
    for r in range(0, M, 3):                                                  # three rows at a time: the kernel of few rows
        ops.gemm_simt(a[r:r + 3], w[:N], out[r:r + 3], epi, w2)
    assert torch.equal(out, first)


class _Batch:
    def __init__(self, before, new):
        self.n_seqs, self.max_new, self.max_after = len(new), max(new), max(b + n for b, n in zip(before, new))
        i32 = dict(dtype=torch.int32, device=DEV)
        self.seq_start = torch.tensor([sum(new[:i]) for i in range(len(new) + 1)], **i32)
        self.seq_before = torch.tensor(before, **i32)
        self.tok_pos = torch.tensor([b + t for b, n in zip(before, new) for t in range(n)], **i32)
        self.tok_seq = torch.tensor([s for s, n in enumerate(new) for _ in range(n)], **i32)


class _View:
    def __init__(self, k, v, table, ring, window):
        self.k, self.v, self.table, self.ring, self.page, self.window = k, v, table, ring, 64, window


@pytest.mark.parametrize("nh,nkv,hd", [(8, 2, 128), (6, 2, 64), (3, 3, 64), (17, 1, 128)])
@pytest.mark.parametrize("window,ring_pages", [(None, 11), (70, 3), (300, 6)])
def test_float32_attention_across_pages_and_steps(nh, nkv, hd, window, ring_pages):
    """Lengths at the edges of pages (64), windows on wrapped rings, spare positions filled with NaN: against float64, and the
    same bits from blocks that walk their rows' keys, from pages shared out, and a token at a time."""
    from ultima_b200.engine import Runtime
    from ultima_b200.kernels import ops
    rt = Runtime(DEV, torch.float32)
    g = torch.Generator(device=DEV).manual_seed(nh * hd + (window or 0))
    ring = ring_pages * 64
    room = ring - (window or 0) if window else 10 ** 9
    before, new = [0, 0, 63, 250, 511, 640], [1, 64, 2, 7, 1, 33]
    new = [min(n, room) for n in new]
    n_pages = ring_pages * len(new) + 2
    kc = torch.full((n_pages, nkv, 64, hd), math.nan, device=DEV)
    vc = torch.full((n_pages, nkv, 64, hd), math.nan, device=DEV)
    table = torch.randperm(n_pages, generator=g, device=DEV)[:ring_pages * len(new)].view(len(new), -1).int().contiguous()
    batch = _Batch(before, new)
    q = torch.randn(sum(new), nh * hd + 8, generator=g, device=DEV)[:, :nh * hd]
    refs, row = [], 0
    for s, (b, n) in enumerate(zip(before, new)):
        k, v = torch.randn(b + n, nkv, hd, generator=g, device=DEV), torch.randn(b + n, nkv, hd, generator=g, device=DEV)
        for p in range(b + n):                               # (later laps of a ring lie over earlier ones)
            kc[table[s, (p % ring) // 64], :, p % 64], vc[table[s, (p % ring) // 64], :, p % 64] = k[p], v[p]
        for t in range(n):
            lo = max(0, b + t + 1 - window) if window else 0
            rep = nh // nkv
            kk, vv = (x[lo:b + t + 1].double().repeat_interleave(rep, 1) for x in (k, v))
            w = torch.softmax(torch.einsum("hd,shd->hs", q[row].double().view(nh, hd), kk) * hd ** -0.5, -1)
            refs.append(torch.einsum("hs,shd->hd", w, vv).reshape(-1))
            row += 1
    kv = _View(kc, vc, table, ring, window)
    got = []
    for split in (0, 1, 3, 64, None):
        rt.arena.reset(0)
        out = torch.full((sum(new), nh * hd), math.nan, device=DEV)
        assert ops.attn_f32_fits(q, kv, out, hd)
        ops.attn_f32(q, kv, out, batch, nh, nkv, hd, hd ** -0.5, rt, split=split)
        got.append(out)
    _within(got[0], torch.stack(refs), 1e-5, 2e-5)           # (values of size 1, weights that sum to 1, up to 673 of them)
    assert all(torch.equal(got[0], o) for o in got[1:])
    for t in range(max(new)):                                # the same tokens as steps of one token a sequence
        live = [s for s in range(len(new)) if t < new[s]]
        one = _Batch([before[s] + t for s in live], [1] * len(live))
        rows = [int(batch.seq_start[s]) + t for s in live]
        rt.arena.reset(0)
        out = torch.empty(len(live), nh * hd, device=DEV)
        sub = _View(kc, vc, table[live].contiguous(), ring, window)
        ops.attn_f32(q[rows].contiguous(), sub, out, one, nh, nkv, hd, hd ** -0.5, rt)
        assert torch.equal(out, got[0][rows])


class _Rows:
    """What the recurrent kernels read of a step's batch."""

    def __init__(self, starts, slots):
        i32 = dict(dtype=torch.int32, device=DEV)
        self.seq_start, self.seq_slot = torch.tensor(starts, **i32), torch.tensor(slots, **i32)
        self.n_seqs = len(slots)
        lens = [b - a for a, b in zip(starts[:-1], starts[1:])]
        self.tok_seq = torch.tensor([i for i, n in enumerate(lens) for _ in range(n)], **i32)
        self.max_new = max(lens)


@pytest.mark.parametrize("decay_per_head", [False, True])
@pytest.mark.parametrize("H,G,D,E,taps", [(4, 2, 64, 64, 4), (2, 1, 128, 64, 3), (3, 3, 64, 128, 2), (2, 2, 128, 128, 4), (2, 1, 128, 128, 1)])
def test_delta_rule_for_heads_of_64_and_128_in_any_portions(H, G, D, E, taps, decay_per_head):
    """Preparation and recurrence against float64 (sums of up to 128 products of unit vectors through 290 tokens), and the same
    bits for a sequence whole, in portions at the edges of a stage of eight tokens and of a run of eight, beside others, and
    beyond the 256 tokens from which a warp takes a run."""
    import plain_sugizen as P
    from ultima_b200.kernels import ops
    T = 290
    g = torch.Generator().manual_seed(H * D + E + taps)
    qk, C = G * D, 2 * G * D + H * E
    rows = torch.randn(T, C + H + (H if decay_per_head else 0) + 4, generator=g)
    cols = (0, qk, 2 * qk, C)
    conv_w = torch.randn(C, taps, generator=g) * 0.4
    dpre = torch.randn(T, H * D, generator=g)
    dt_bias = torch.randn(H if decay_per_head else H * D, generator=g) - 2
    a_log = torch.randn(H, generator=g) * 0.5
    x = rows.double()
    y = P.short_conv_silu(x[:, :C], conv_w.double())
    q, k = P.unit(y[:, :qk].view(T, G, D)) * D ** -0.5, P.unit(y[:, qk:2 * qk].view(T, G, D))
    v = y[:, 2 * qk:].reshape(T, H, E)
    beta = torch.sigmoid(x[:, C:C + H])
    pre = x[:, C + H:C + 2 * H, None].expand(T, H, D) + dt_bias.double()[None, :, None] if decay_per_head else \
        (dpre.double() + dt_bias.double()).view(T, H, D)
    dec = torch.exp(-torch.exp(a_log.double())[None, :, None] * P.softplus(pre))
    rep = H // G
    ref = P.delta_rule_scan(q.repeat_interleave(rep, 1), k.repeat_interleave(rep, 1), v, beta, dec)
    shape = ops.delta_shape(H, G, D, E, taps, cols, a_off=C + H if decay_per_head else -1)
    dev = [t.contiguous().to(DEV) for t in (rows, dpre, conv_w, dt_bias, a_log)]

    def run(sel, starts, slots, S, cs):
        p, dp = dev[0][sel].contiguous(), None if decay_per_head else dev[1][sel].contiguous()
        n, b = p.shape[0], _Rows(starts, slots)
        one = b.max_new == 1
        qn, kn = torch.empty(n, qk, device=DEV), torch.empty(n, qk, device=DEV)
        vc, o = torch.empty(n, H * E, device=DEV), torch.empty(n, H * E, device=DEV)
        bt, dc = torch.empty(n, H, device=DEV), torch.empty(n, H * D, device=DEV)
        ops.delta_prepare(p, shape, dev[2], cs, dp, dev[3], dev[4], b, qn, kn, vc, bt, dc, 1e-6, D ** -0.5, update_state=one)
        if not one:
            ops.conv_state_update(p, cs, b, C, taps)
        ops.delta_scan(qn, kn, vc, bt, dc, o, S, b, H, G, D, E)
        return o

    def fresh():
        return torch.zeros(3, H, D, E, device=DEV), torch.zeros(3, max(taps - 1, 1), C, device=DEV)
    S, cs = fresh()
    whole = run(torch.arange(T), [0, T], [1], S, cs)
    _within(whole, ref.reshape(T, -1).to(DEV), 3e-5, 3e-5)
    assert float(S[0].abs().max()) == 0.0 and float(S[2].abs().max()) == 0.0
    S2, cs2 = fresh()
    cuts = [0, 1, 2, 3, 10, 18, 26, 33, 290]
    cut = torch.cat([run(torch.arange(a, b), [0, b - a], [2], S2, cs2) for a, b in zip(cuts[:-1], cuts[1:])])
    assert torch.equal(cut, whole) and torch.equal(S2[2], S[1]) and torch.equal(cs2[2], cs[1])
    S3, cs3 = fresh()
    both = run(torch.cat([torch.arange(T), torch.arange(61)]), [0, T, T + 61], [2, 0], S3, cs3)
    assert torch.equal(both[:T], whole) and torch.equal(both[T:], whole[:61]) and torch.equal(S3[2], S[1])
