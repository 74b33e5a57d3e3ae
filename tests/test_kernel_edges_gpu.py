"""Kernels at the sizes where their tiles, chunks and slices begin and end, against float64."""
import math

import numpy as np
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


@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("T,N", [(5, 256), (40, 256), (200, 384), (1100, 8192)])
def test_gate_products_of_large_negative_gates(T, N, interleaved):
    """Gates of -87.5 to -88.5, where 1 + exp(-g) lies between 2^126 and 2^128 and the quotient is small but a normal number: every
    product is of one term, so only the sigmoid's exponential (32 bits; its argument of 127 is off by at most 2^-17) and the
    result's rounding to 2^-9 are left."""
    from ultima_b200.engine import Runtime
    from ultima_b200.kernels import gemm_tc, ops
    rt = Runtime(DEV, torch.bfloat16)
    g = torch.Generator().manual_seed(T + N)
    K, half = 64, N // 2
    a = torch.zeros(T, K)
    a[torch.arange(T), torch.arange(T) % 8] = 1
    w = torch.zeros(N, K)
    w[:half, :8] = -87.5 - 0.5 * torch.randint(0, 3, (half, 8), generator=g)
    w[half:, :8] = 2.0 ** 20 * torch.randint(1, 9, (half, 8), generator=g)
    gate, up = (a.double() @ m.double().T for m in (w[:half], w[half:]))
    if interleaved:                                          # 64 gate rows, then their 64 up rows
        w = torch.stack([w[:half].view(-1, 64, K), w[half:].view(-1, 64, K)], 1).reshape(N, K)
    a, w = (t.to(DEV, torch.bfloat16) for t in (a, w))
    out = torch.full((T, half), math.nan, dtype=torch.bfloat16, device=DEV)
    if interleaved:
        gemm_tc.gemm(a, w, out, ops.EPI_SWIGLU_IL, None, rt)
    else:
        gemm_tc.gemm(a, w[:half], out, ops.EPI_SWIGLU, w[half:], rt)
    gemm_tc.check_error(rt)
    ref = (gate / (1 + torch.exp(-gate)) * up).to(DEV)
    assert float(((out.double() - ref) / ref).abs().max()) < 2.0 ** -8


@pytest.mark.parametrize("epilogue", ["store", "add", "product"])
@pytest.mark.parametrize("M,N,K", [(1, 33, 68), (4, 130, 260), (5, 17, 36), (8, 64, 512), (9, 72, 1028), (16, 129, 96), (17, 40, 2048),
                                   (33, 200, 516), (64, 128, 64), (65, 257, 72), (129, 130, 640), (200, 1032, 1024)])
def test_float32_products_have_one_order_of_sums_in_every_form(M, N, K, epilogue):
    """Every form, and the rows alone, give the same bits.  A sum of K terms of size 1 / sqrt(K) in chains rounds K partial sums of size 1
    or less, each by up to 2^-24 of it and in either direction: sqrt(K) 2^-24 is the size of the error, four times that the bound, of
    either factor for the gate product (whose slopes are below 1.1).  Inputs rounded to 10 mantissa bits, which a product that is not
    float32 throughout would take, miss the bound at every K."""
    from ultima_b200.kernels import ops
    g = torch.Generator(device=DEV).manual_seed(M * 7 + N + K)
    a = torch.randn(M, K + 4, generator=g, device=DEV)[:, 4:]                 # rows with a stride of their own
    w = torch.randn(2 * N, K, generator=g, device=DEV) * K ** -0.5
    x = torch.randn(M, N, generator=g, device=DEV)
    epi = {"store": ops.EPI_STORE, "add": ops.EPI_ADD, "product": ops.EPI_SWIGLU}[epilogue]
    w2 = w[N:] if epilogue == "product" else None

    def plain(a, w):
        z, u = a.double() @ w[:N].double().T, a.double() @ w[N:].double().T
        return z + x.double() if epilogue == "add" else torch.nn.functional.silu(z) * u if epilogue == "product" else z
    ref = plain(a, w)
    factors = 1.0
    if epilogue == "product":
        z, u = a.double() @ w[:N].double().T, a.double() @ w[N:].double().T
        factors = torch.nn.functional.silu(z).abs() + 1.1 * u.abs()

    def over(got):                                                            # the largest error, in bounds
        return float(((got.double() - ref).abs() / (2e-6 * ref.abs() + 4 * K ** 0.5 * 2.0 ** -24 * factors)).max())

    def short(t):                                                             # 10 mantissa bits, to nearest
        return ((t.contiguous().view(torch.int32) + 0x1000) & -0x2000).view(torch.float32)
    assert over(plain(short(a), short(w))) > 1
    assert ops.f32_fits(a, w[:N], x, epi, w2)
    first = None
    for form in ([0] if M <= 16 else []) + [32, 64, 128, -32, -64]:
        out = x.clone()
        ops.gemm_f32(a, w[:N], out, epi, w2, form=form)
        if first is None:
            first = out
            assert over(out) <= 1, over(out)
        assert torch.equal(out, first), form
    out = x.clone()
    for r in range(0, M, 3):                                                  # three rows at a time: the kernel of few rows
        ops.gemm_simt(a[r:r + 3], w[:N], out[r:r + 3], epi, w2)
    assert torch.equal(out, first)


@pytest.mark.parametrize("epilogue", ["store", "add", "product"])
@pytest.mark.parametrize("M,N,K", [(17, 33, 4), (17, 130, 64), (31, 64, 68), (64, 65, 192), (65, 129, 260), (127, 200, 516), (128, 128, 1024),
                                   (129, 257, 300), (145, 70, 2052), (260, 384, 640)])
def test_float32_products_on_the_tensor_cores(M, N, K, epilogue):
    """A block of 64 terms is summed from zero and the blocks one after another, so fewer and smaller partial sums are rounded than in a
    chain of K terms: the bound of the test above (4 sqrt(K) 2^-24 of either factor) holds.  Clusters give the same bits, and so do other
    tokens beside these."""
    from ultima_b200.engine import Runtime
    from ultima_b200.kernels import ops
    rt = Runtime(DEV, torch.float32)
    g = torch.Generator(device=DEV).manual_seed(M * 7 + N + K)
    a = torch.randn(M, K + 8, generator=g, device=DEV)[:, 4:K + 4]
    w = torch.randn(2 * N, K + 4, generator=g, device=DEV)[:, :K] * K ** -0.5
    w = torch.nn.functional.pad(w, (0, 4))[:, :K]                             # rows with strides of their own
    wide = torch.randn(M, N + 3, generator=g, device=DEV)
    x = wide[:, 1:N + 1]
    epi = {"store": ops.EPI_STORE, "add": ops.EPI_ADD, "product": ops.EPI_SWIGLU}[epilogue]
    w2 = w[N:] if epilogue == "product" else None
    z, u = a.double() @ w[:N].double().T, a.double() @ w[N:].double().T
    ref = z + x.double() if epilogue == "add" else torch.nn.functional.silu(z) * u if epilogue == "product" else z
    factors = torch.nn.functional.silu(z).abs() + 1.1 * u.abs() if epilogue == "product" else 1.0
    assert ops.f32_fits(a, w[:N], x, epi, w2) and (K < 8 or w.stride(0) != K)
    got = []
    for split in (False, True):
        buf = wide.clone()
        out = buf[:, 1:N + 1]
        ops.gemm_f32_tc(a, w[:N], out, epi, w2, rt, split)
        over = float(((out.double() - ref).abs() / (2e-6 * ref.abs() + 4 * K ** 0.5 * 2.0 ** -24 * factors)).max())
        assert over <= 1, over
        assert torch.equal(buf[:, 0], wide[:, 0]) and torch.equal(buf[:, N + 1:], wide[:, N + 1:])
        got.append(out)
    assert torch.equal(*got)
    out = x[5:].clone()
    ops.gemm_f32_tc(a[5:], w[:N], out, epi, w2, rt)
    assert torch.equal(out, got[0][5:])
    rt.check_status()


@pytest.mark.parametrize("epilogue", ["store", "add", "product"])
@pytest.mark.parametrize("M,N,K", [(1, 33, 4), (3, 130, 64), (7, 16, 68), (8, 65, 192), (9, 129, 260), (15, 200, 516), (16, 8, 1024), (17, 257, 300),
                                   (33, 70, 2052), (40, 384, 640), (5, 40, 6148)])
def test_float32_products_of_few_tokens_have_the_sums_of_many(M, N, K, epilogue):
    """The kernels of few tokens, one, two and four warps a slice, whole and a row at a time, and tcgen05's tiles: the same bits, within the
    bound of the test above."""
    from ultima_b200.engine import Runtime
    from ultima_b200.kernels import ops
    rt = Runtime(DEV, torch.float32)
    g = torch.Generator(device=DEV).manual_seed(M * 7 + N + K)
    a = torch.randn(M, K + 8, generator=g, device=DEV)[:, 4:K + 4]
    w = torch.nn.functional.pad(torch.randn(2 * N, K, generator=g, device=DEV) * K ** -0.5, (0, 4))[:, :K]      # rows with strides of their own
    wide = torch.randn(M, N + 3, generator=g, device=DEV)
    epi = {"store": ops.EPI_STORE, "add": ops.EPI_ADD, "product": ops.EPI_SWIGLU}[epilogue]
    w2 = w[N:] if epilogue == "product" else None
    z, u = a.double() @ w[:N].double().T, a.double() @ w[N:].double().T
    x = wide[:, 1:N + 1].double()
    ref = z + x if epilogue == "add" else torch.nn.functional.silu(z) * u if epilogue == "product" else z
    factors = torch.nn.functional.silu(z).abs() + 1.1 * u.abs() if epilogue == "product" else 1.0
    first = None
    for form in (0, 2, 3) + ((4,) if M <= 8 else ()):
        buf = wide.clone()
        ops.gemm_f32_tc(a, w[:N], buf[:, 1:N + 1], epi, w2, rt, form)
        if first is None:
            first = buf
            assert float(((buf[:, 1:N + 1].double() - ref).abs() / (2e-6 * ref.abs() + 4 * K ** 0.5 * 2.0 ** -24 * factors)).max()) <= 1
            assert torch.equal(buf[:, 0], wide[:, 0]) and torch.equal(buf[:, N + 1:], wide[:, N + 1:])
        assert torch.equal(buf, first), form
    for form in (2, 3, 4):
        buf = wide.clone()
        for r in range(M):
            ops.gemm_f32_tc(a[r:r + 1], w[:N], buf[r:r + 1, 1:N + 1], epi, w2, rt, form)
        assert torch.equal(buf, first), form
    rt.check_status()


@pytest.mark.parametrize("M,N,K", [(16, 2048, 1024), (17, 2048, 1024), (64, 2048, 1024), (65, 2048, 1024), (681, 2048, 6144)])
def test_float32_products_of_a_runtime(M, N, K):
    """The way from ``Runtime.matmul`` to the kernels: within the bound of the tests above, what the arena holds beside the call untouched,
    its place given back, and a product with a small matrix on its FMA sums."""
    from ultima_b200.engine import Runtime
    from ultima_b200.kernels import ops
    rt = Runtime(DEV, torch.float32)
    g = torch.Generator(device=DEV).manual_seed(M)
    a, w = torch.randn(M, K, generator=g, device=DEV), torch.randn(N, K, generator=g, device=DEV) * K ** -0.5
    held = rt.arena.alloc((1000,), torch.float32).fill_(3.0)
    out, mark = rt.arena.alloc((M, N), torch.float32), rt.arena.mark()
    rt.matmul(a, w, out)
    behind = rt.arena.alloc((16,), torch.float32)
    assert mark <= rt.arena.mark() <= mark + 64 + rt.arena.ALIGN and behind.numel() == 16
    ref = a.double() @ w.double().T
    assert float(((out.double() - ref).abs() / (2e-6 * ref.abs() + 4 * K ** 0.5 * 2.0 ** -24)).max()) <= 1
    assert bool((held == 3.0).all())
    few, alone = torch.empty(M, 256, device=DEV), torch.empty(M, 256, device=DEV)
    rt.matmul(a, w[:256], few)
    ops.gemm_f32(a, w[:256], alone)
    assert torch.equal(few, alone)
    rt.check_status()


def test_float32_logits_do_not_depend_on_what_shares_a_step(tmp_path):
    """A model whose matrices are large enough for the float32 product on the tensor cores, and a router's worth of small ones beside them:
    a prompt of 140 tokens in one step, in steps of 16, 17, 64, 65 and single tokens and beside other prompts, and decode steps of 16 and 17
    sequences, give every logit the same bits."""
    import ultima_b200 as u
    from ultima_b200.engine import Engine
    from ultima_b200.kernels import ops
    cfg = u.config_from_dict(dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", vocab_size=1000, hidden_size=1024, intermediate_size=2304,
                                  num_hidden_layers=2, num_attention_heads=8, num_key_value_heads=2, head_dim=128, rms_norm_eps=1e-6,
                                  rope_theta=10000.0, max_position_embeddings=512, tie_word_embeddings=False, hidden_act="silu"))
    assert ops.f32_on_tensor_cores(1024, 1024, ops.EPI_ADD) and not ops.f32_on_tensor_cores(256, 1024, ops.EPI_STORE)
    eng = Engine.from_dir(u.write_random_model(str(tmp_path / "m"), cfg, 5, "bfloat16"), dtype="float32", max_tokens=40 * 256, max_seqs=40)
    rng = np.random.default_rng(7)
    ids = rng.integers(0, 1000, 157).tolist()

    def fed(cuts, others=()):
        """Logits of every position of ``ids``, fed in pieces of ``cuts`` tokens beside prompts of the lengths ``others``."""
        slots, out, at = eng.open(1 + len(others)), [], 0
        for i, n in enumerate(cuts):
            lists, want = [ids[at:at + n]], [list(range(n))]
            if i == 0:
                lists += [rng.integers(0, 1000, m).tolist() for m in others]
                want += [[] for _ in others]
            out.append(eng.step(slots[:len(lists)], lists, want=want).clone())
            at += n
        eng.close(slots)
        return torch.cat(out)
    whole = fed([157])
    for cuts, others in (([64, 65, 16, 12], ()), ([17, 140], ()), ([16, 1, 1, 17, 122], ()), ([140] + [1] * 17, (3, 90)), ([8, 9, 140], (60,)), ([1] * 40 + [117], ())):
        assert torch.equal(fed(cuts, others), whole), cuts
    prompts = [rng.integers(0, 1000, 5 + i).tolist() for i in range(17)]
    results = []
    for n in (16, 17):
        slots = eng.open(n)
        eng.step(slots, prompts[:n])
        results.append(torch.cat([eng.step(slots, [[t + i] for i in range(n)]).clone()[:16] for t in range(3)]))
        eng.close(slots)
    assert torch.equal(*results)
    eng.check_errors()


@pytest.mark.parametrize("ea,ew", [(-120, 60), (60, -120), (-126, 30), (-135, 70), (40, -133), (-66, -66), (-70, -70), (50, 45), (-149, 100)])
@pytest.mark.parametrize("M", [5, 70])
def test_float32_products_on_the_tensor_cores_over_the_range_of_the_exponents(M, ea, ew):
    """Operands of size 2^ea and 2^ew, down to denormal numbers, have all their bits in the sums: the error relative to 64 bits is the
    same as with operands of size one, below sqrt(K) 2^-24 of the row's largest (with results that are denormal, half of the smallest)."""
    from ultima_b200.engine import Runtime
    from ultima_b200.kernels import ops
    rt = Runtime(DEV, torch.float32)
    g = torch.Generator(device=DEV).manual_seed(M - ea)
    N, K = 150, 516
    a = (torch.randn(M, K, generator=g, device=DEV).double() * 2.0 ** ea).float()
    w = (torch.randn(N, K, generator=g, device=DEV).double() * 2.0 ** ew).float()
    ref = a.double() @ w.double().T
    bound = K ** 0.5 * 2.0 ** -24 * ref.abs().amax(1, keepdim=True) + 2.0 ** -150
    first = None
    for form in (0, 1, 2, 3):
        out = torch.empty(M, N, device=DEV)
        ops.gemm_f32_tc(a, w, out, ops.EPI_STORE, None, rt, form)
        assert bool(((out.double() - ref).abs() <= bound).all()), (form, float(((out.double() - ref).abs() / bound).max()))
        first = out if first is None else first
        assert torch.equal(out, first), form
    rt.check_status()


@pytest.mark.parametrize("epilogue", ["add", "product"])
def test_float32_products_of_many_tokens_in_portions(epilogue, monkeypatch):
    """Portions of 128 tokens: the bits of the whole."""
    from ultima_b200.engine import Runtime
    from ultima_b200.kernels import ops
    rt = Runtime(DEV, torch.float32)
    g = torch.Generator(device=DEV).manual_seed(2)
    M, N, K = 300, 130, 516
    a, w, x = (torch.randn(*s, generator=g, device=DEV) for s in ((M, K), (2 * N, K), (M, N)))
    epi, w2 = (ops.EPI_ADD, None) if epilogue == "add" else (ops.EPI_SWIGLU, w[N:])
    out = []
    for bound in (ops.F32_PLANES, 1 << 19):
        monkeypatch.setattr(ops, "F32_PLANES", bound)
        for form in (0, 1):
            out.append(x.clone())
            ops.gemm_f32_tc(a, w[:N], out[-1], epi, w2, rt, form)
    assert all(torch.equal(o, out[0]) for o in out[1:])
    rt.check_status()


def test_float32_products_on_the_tensor_cores_beyond_the_numbers():
    """Infinities, NaN and numbers that round up to infinity in bfloat16: what the FMA forms give, for the token or the weight row alone."""
    from ultima_b200.engine import Runtime
    from ultima_b200.kernels import ops
    rt = Runtime(DEV, torch.float32)
    g = torch.Generator(device=DEV).manual_seed(3)
    M, N, K = 70, 150, 516
    a, w = torch.randn(M, K, generator=g, device=DEV), torch.randn(N, K, generator=g, device=DEV)
    clean = torch.empty(M, N, device=DEV)
    ops.gemm_f32_tc(a, w, clean, ops.EPI_STORE, None, rt)
    a[3, 5], a[7, 500], w[11, 100], a[20, 300] = math.inf, math.nan, -math.inf, 3.3999e38
    w[30], w[31] = 0.0, 0.0
    ref, got = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    ops.gemm_f32(a, w, ref, form=64)
    for split in (False, True, 2, 3):
        ops.gemm_f32_tc(a, w, got, ops.EPI_STORE, None, rt, split)
        for r in (3, 7, 20):
            assert torch.equal(torch.nan_to_num(got[r], 7.0, 8.0, 9.0), torch.nan_to_num(ref[r], 7.0, 8.0, 9.0))
        assert torch.equal(torch.nan_to_num(got[:, 11], 7.0, 8.0, 9.0), torch.nan_to_num(ref[:, 11], 7.0, 8.0, 9.0))
        rows = [r for r in range(M) if r not in (3, 7, 20)]
        cols = [c for c in range(N) if c not in (11, 30, 31)]
        assert torch.equal(got[rows][:, cols], clean[rows][:, cols]) and not bool(got[rows][:, 30:32].any())


@pytest.mark.parametrize("N,K", [(64, 64), (192, 136), (328, 1032), (512, 320)])
def test_grouped_products_on_pairs_of_blocks(N, K):
    """Experts with no rows, one, up to and beyond one, two and three tiles of 256, N and K at the edges of blocks; rows of no expert are
    NaN.  bfloat16 results are rounded by 2^-9 (products of two rounded factors and their sum by less than 2^-7), float32 sums of K
    terms by sqrt(K) 2^-24 of the largest."""
    from ultima_b200.engine import Runtime
    from ultima_b200.kernels import gemm_tc, ops
    from ultima_b200.parts.routed import RoutePlan
    rt = Runtime(DEV, torch.bfloat16)
    counts = [0, 1, 257, 256, 31, 33, 513, 0, 300, 770, 128]
    E, rows, tile = len(counts), sum(counts), gemm_tc.PAIR_ROWS
    g = torch.Generator(device=DEV).manual_seed(N + K)
    a = torch.randn(rows + 40, K, generator=g, device=DEV).bfloat16()
    a[rows:] = math.nan
    w = (torch.randn(E, 2 * N, K, generator=g, device=DEV) * K ** -0.5).bfloat16()
    tiles, ws = (torch.zeros(n, dtype=torch.int32, device=DEV) for n in (4 * (-(-rows // tile) + E), 3 * E + 1))
    ws[:E] = torch.tensor(counts, dtype=torch.int32)
    ops.route_plan(ws[:E], ws[E:2 * E], ws[2 * E:3 * E], tiles, ws[3 * E:], E, tile)
    listed = tiles.view(-1, 4)[:int(ws[3 * E])].tolist()
    assert [sum(r[2] for r in listed if r[0] == e) for e in range(E)] == counts and all(0 < r[2] <= tile for r in listed)
    plan = RoutePlan(tiles, ws[3 * E:], None, tiles.numel() // 4, rows, gather=False, tile=tile)
    expert = torch.repeat_interleave(torch.arange(E, device=DEV), torch.tensor(counts, device=DEV))
    z = torch.cat([a[:rows][expert == e].double() @ w[e].double().T for e in range(E)])
    gate, up = z[:, :N], z[:, N:]
    consts = (1.3, 1.702, 1.0)
    clamped = gate.clamp(max=1.3)
    for kind, ref in (("product", gate * torch.sigmoid(gate) * up),
                      ("clamped", clamped * torch.sigmoid(1.702 * clamped) * (up.clamp(-1.3, 1.3) + 1.0)),
                      ("squared", up.clamp(min=0) ** 2), ("stored", up), ("float32", up)):
        out = torch.full((rows + 40, N), 7.0, device=DEV, dtype=torch.float32 if kind == "float32" else torch.bfloat16)
        if kind in ("product", "clamped"):
            gemm_tc.grouped(a, w[:, :N], out, plan, ops.EPI_SWIGLU, w[:, N:], rt, gate=consts if kind == "clamped" else None)
        else:
            gemm_tc.grouped(a, w[:, N:], out, plan, ops.EPI_STORE, None, rt, unary=ops.UNARY_RELU_SQUARED if kind == "squared" else 0)
        _within(out[:rows], ref, 2 ** -7 if kind != "float32" else 0.0, (2 ** -8 if kind != "float32" else K ** 0.5 * 2.0 ** -24) * float(ref.abs().max()))
        assert bool((out[rows:] == 7.0).all()), kind
    rt.check_status()


@pytest.mark.parametrize("tokens,experts,inner,width,tile", [(2048, 32, 1024, 2048, 256), (1024, 32, 1024, 2048, 128), (300, 2, 128, 256, 128),
                                                             (64, 8, 1024, 2048, 32)])
def test_rows_a_tile_of_the_grouped_products(tokens, experts, inner, width, tile):
    from ultima_b200.kernels import gemm_tc
    assert gemm_tc.row_tile(4 * tokens if experts > 2 else tokens, experts, inner, width, n_sms=148) == tile


@pytest.mark.parametrize("before", [2046, 2047, 2048, 4095, 4200])
def test_decode_attention_over_more_pages_than_the_loading_warp_has_lanes(before):
    """One slice of 32, 33, 64 and 66 pages that lie anywhere; float32 sums of bfloat16 products, results rounded to 2^-9."""
    from ultima_b200.engine import Runtime
    from ultima_b200.kernels import attn_tc
    rt = Runtime(DEV, torch.bfloat16)
    nh, nkv, hd, n = 4, 2, 64, before + 1
    g = torch.Generator(device=DEV).manual_seed(before)
    pages = -(-n // 64)
    q = torch.randn(1, nh * hd, generator=g, device=DEV).bfloat16()
    kc, vc = (torch.randn(pages + 2, nkv, 64, hd, generator=g, device=DEV).bfloat16() for _ in range(2))
    table = torch.randperm(pages + 2, generator=g, device=DEV)[:pages].int().view(1, -1)
    b, kv = _Batch([before], [1]), _View(kc, vc, table, pages * 64, None)
    out = torch.empty(1, nh * hd, dtype=torch.bfloat16, device=DEV)
    attn_tc.attention(q, kv, out, b, nh, nkv, hd, hd ** -0.5, rt, slices=1, kernel="tma")
    k, v = (c[table[0].long()].permute(1, 0, 2, 3).reshape(nkv, -1, hd)[:, :n].double().repeat_interleave(nh // nkv, 0) for c in (kc, vc))
    p = torch.softmax(torch.einsum("hd,hnd->hn", q.double().view(nh, hd), k) * hd ** -0.5, -1)
    ref = torch.einsum("hn,hnd->hd", p, v).reshape(1, -1)
    assert float((out.double() - ref).norm() / ref.norm()) < 2 ** -7
    rt.check_status()


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


@pytest.mark.parametrize("nh,nkv,hd,window,keep,slope,sink", [(8, 2, 128, 100, 4, 8.0, False), (4, 2, 64, 64, 64, None, False),
                                                              (6, 2, 64, 65, 65, 8.0, True), (4, 1, 128, 200, 130, 1.0, True),
                                                              (16, 1, 128, 63, 0, 8.0, False), (3, 3, 128, 0, 0, 2.0, True),
                                                              (4, 2, 128, 192, 0, None, True), (4, 2, 128, 0, 4, None, False),
                                                              (8, 2, 64, 0, 70, 8.0, True)])
def test_prompts_with_kept_positions_and_a_bias_by_distance(nh, nkv, hd, window, keep, slope, sink):
    """Tiles of kept positions ahead of the window's, windows at the edges of pages, kept positions without a window (they are what is
    visible anyway), new and continued prompts, every position that no sequence has reached NaN: bfloat16 probabilities and results, 2^-9 each, of sums in float32."""
    from ultima_b200.engine import Runtime
    from ultima_b200.kernels import attn_tc
    rt = Runtime(DEV, torch.bfloat16)
    before, new = [0, 0, 70, 321, 5], [1, 400, 130, 65, 64]
    g = torch.Generator(device=DEV).manual_seed(nh + hd + window)
    slopes = 2.0 ** (-slope * torch.arange(1, nh + 1, device=DEV, dtype=torch.float64) / nh) if slope else None
    lens, T = [b + n for b, n in zip(before, new)], sum(new)
    kc, vc = (torch.full((len(lens) * 7, nkv, 64, hd), math.nan, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    table = torch.randperm(len(lens) * 7, generator=g, device=DEV).int().view(len(lens), 7)
    k, v = ([torch.randn(n, nkv, hd, generator=g, device=DEV).bfloat16() for n in lens] for _ in range(2))
    for s, n in enumerate(lens):
        at = torch.arange(n, device=DEV)
        for c, x in ((kc, k), (vc, v)):
            c[table[s, at // 64].long(), :, at % 64] = x[s]
    q = torch.randn(T, nh * hd, generator=g, device=DEV).bfloat16()
    gate = torch.randn(T, nh * hd, generator=g, device=DEV) if sink else None
    out = torch.full((T, nh * hd), math.nan, device=DEV, dtype=torch.bfloat16)
    attn_tc.attention_ext(q, _View(kc, vc, table, 448, None), out, _Batch(before, new), nh, nkv, hd, 0.2, rt, window=window or None,
                          keep_first=keep, sink=sink, slopes_log2=None if slopes is None else (slopes * math.log2(math.e)).float(),
                          out_scale=1.3, gate=gate)
    rt.check_status()
    row = 0
    for s, (b, n) in enumerate(zip(before, new)):
        kd, vd = (x[s].double().repeat_interleave(nh // nkv, 1) for x in (k, v))
        z = torch.einsum("thd,jhd->htj", q[row:row + n].double().view(n, nh, hd), kd) * 0.2
        far = (torch.arange(b, b + n, device=DEV)[:, None] - torch.arange(b + n, device=DEV)[None]).double()
        if slopes is not None:
            z = z - slopes[:, None, None] * far
        seen = (far >= 0) & ((far < window) | (torch.arange(b + n, device=DEV) < keep)[None] if window else far >= 0)
        z = z.masked_fill(~seen, -math.inf)
        if sink:
            z = torch.cat([z, torch.zeros(nh, n, 1, device=DEV, dtype=torch.float64)], -1)
        ref = 1.3 * torch.einsum("htj,jhd->thd", torch.softmax(z, -1)[..., :b + n], vd).reshape(n, -1)
        if gate is not None:
            ref = ref * torch.sigmoid(gate[row:row + n].double())
        got = out[row:row + n].double()
        assert bool(torch.isfinite(got).all())
        assert float(((got - ref).norm(dim=1) / ref.norm(dim=1)).max()) < 2 ** -6
        row += n


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


@pytest.mark.parametrize("parts", [1, 3])
@pytest.mark.parametrize("hd,rd,inter,norm,gates", [(128, 128, False, True, "head"), (128, 64, False, True, "head"), (64, 32, False, False, None),
                                                    (64, 64, True, False, "element"), (128, 72, True, True, "element"), (128, None, False, True, None),
                                                    (64, 4, False, True, "head")])
def test_placement_of_heads_of_64_and_128(hd, rd, inter, norm, gates, parts):
    """Queries, cache and gates from projection rows (summed over parts) against float64; values that are the keys as they were
    for pairs of neighbours; a layer without keys of its own."""
    from ultima_b200.kernels import ops
    g = torch.Generator(device=DEV).manual_seed(hd + (rd or 0) + parts)
    nh, nkv, T, ring = 6, 2, 37, 192
    q_off, k_off = 4, 4 + nh * hd
    v_off = k_off if inter else k_off + nkv * hd
    g_off = k_off + 2 * nkv * hd
    g_width = {"head": nh, "element": nh * hd, None: 0}[gates]
    x = torch.randn(parts, T, g_off + g_width + (-g_width) % 4, generator=g, device=DEV)
    qw, kw = ((1 + 0.1 * torch.randn(hd, generator=g, device=DEV)) for _ in range(2)) if norm else (None, None)
    pos = torch.randint(0, 150, (T,), generator=g, device=DEV).int()
    pos = torch.arange(T, device=DEV).int() * 4 + pos % 4                     # no position twice
    cos = sin = None
    if rd:
        a = torch.rand(160, rd // 2, generator=g, device=DEV) * 6
        cos, sin = a.cos().contiguous(), a.sin().contiguous()
    table = torch.tensor([[2, 0, 3]], dtype=torch.int32, device=DEV)
    s = x.double().sum(0)

    def head(off, n, w):
        h = s[:, off:off + n * hd].view(T, n, hd)
        if w is not None:
            h = h * torch.rsqrt((h * h).mean(-1, keepdim=True) + 1e-5) * w.double()
        if rd:
            c, d = cos[pos.long()].double()[:, None], sin[pos.long()].double()[:, None]
            i, j = (slice(0, rd, 2), slice(1, rd, 2)) if inter else (slice(0, rd // 2), slice(rd // 2, rd))
            h, a, b = h.clone(), h[..., i].clone(), h[..., j].clone()
            h[..., i], h[..., j] = a * c - b * d, b * c + a * d
        return h
    for dt, tol in ((torch.float32, 1e-6), (torch.bfloat16, 2.0 ** -8)):
        for own in (True, False):
            q = torch.full((T, nh * hd), math.nan, dtype=dt, device=DEV)
            kc, vc = (torch.full((4, nkv, 64, hd), math.nan, dtype=dt, device=DEV) for _ in range(2))
            gate = torch.full((T, g_width), math.nan, device=DEV) if gates else None
            xs = x if parts > 1 else x[0]
            args = (pos, torch.zeros_like(pos), kc, vc, table, ring, 64, nh, nkv, hd, hd, 1e-5)
            if inter or gates == "element":
                ops.qkv_place_rows(xs, q_off, k_off if own else None, v_off, q, qw, kw, False, cos, sin, rd or 0, inter, *args,
                                   g_off if gates else None, gate)
            else:
                ops.qkv_place(xs, q_off, k_off if own else None, v_off, q, qw, kw, cos, sin, rd or 0, *args, g_off if gates else None, gate)
            _within(q, head(q_off, nh, qw).reshape(T, -1), tol, 4e-6)         # (sums of a few numbers of size 1)
            if gates:
                _within(gate, s[:, g_off:g_off + g_width], 0, 4e-6)
            if own:
                p = pos.long()
                got = [c[table[0].long()[p // 64], :, p % 64] for c in (kc, vc)]
                _within(got[0], head(k_off, nkv, kw), tol, 4e-6)
                _within(got[1], s[:, v_off:v_off + nkv * hd].view(T, nkv, hd), tol, 4e-6)
            assert int(torch.isfinite(kc).sum()) == (T * nkv * hd if own else 0)


@pytest.mark.parametrize("H,P,N,G,taps,groups", [(4, 64, 128, 2, 4, 2), (8, 16, 32, 1, 2, 1), (2, 64, 64, 2, 3, 1), (36, 64, 16, 1, 1, 1)])
def test_state_space_preparation_and_finish_of_long_prompts(H, P, N, G, taps, groups):
    """Beyond the 256 tokens from which a thread takes a run of eight: preparation, recurrence and finish against float64, and the
    same bits for a sequence whole, in portions and beside another."""
    import plain_tinuzen as Q
    from ultima_b200.kernels import ops
    T, eps = 290, 1e-5
    g = torch.Generator().manual_seed(H + P + N)
    inner, C = H * P, H * P + 2 * G * N
    rows = torch.randn(T, 2 * inner + 2 * G * N + H + (-H) % 4, generator=g)
    w, cb = torch.randn(C, taps, generator=g) * 0.4, torch.randn(C, generator=g) * 0.2
    dtb, al, ds = torch.randn(H, generator=g) - 1, torch.randn(H, generator=g) * 0.5, torch.randn(H, generator=g)
    nw = 1 + 0.1 * torch.randn(inner, generator=g)
    x = rows.double()
    z, dt = x[:, :inner], x[:, inner + C:inner + C + H]
    m = Q.silu(Q.causal_conv(x[:, inner:inner + C], w.double(), cb.double()))
    B, Cc = (m[:, inner + i * G * N:inner + (i + 1) * G * N].reshape(T, G, N).repeat_interleave(H // G, 1) for i in (0, 1))
    y = Q.state_space_scan(m[:, :inner].reshape(T, H, P), B, Cc, Q.softplus(dt + dtb.double()), al.double(), ds.double()).reshape(T, inner)
    y = (y * Q.silu(z)).view(T, groups, -1)
    ref = (y / torch.sqrt((y * y).mean(-1, keepdim=True) + eps)).reshape(T, inner) * nw.double()
    dev = [t.to(DEV) for t in (rows, w, cb, dtb, al, ds, nw)]
    shape = ops.ssm_shape(H, P, N, G, taps, (0, inner, 2 * inner, 2 * inner + G * N, inner + C))

    def run(sel, starts, slots, S, cs):
        p, b = dev[0][sel].contiguous(), _Rows(starts, slots)
        n, one = p.shape[0], b.max_new == 1
        xbc, dv, dc = (torch.empty(n, k, device=DEV) for k in (C, H, H))
        o, out = torch.empty(n, inner, device=DEV), torch.empty(n, inner, device=DEV)
        ops.ssm_prepare(p, shape, dev[1], dev[2], cs, dev[3], dev[4], b, xbc, dv, dc, update_state=one)
        if not one and taps > 1:
            ops.ssm_conv_state_update(p, shape, cs, b)
        ops.ssm_scan(xbc, dv, dc, dev[5], o, S, b, H, P, N, G)
        ops.ssm_finish(o, p, shape, dev[6], out, groups, eps)
        return out

    def fresh():
        return torch.zeros(3, H, N, P, device=DEV), torch.zeros(3, max(taps - 1, 1), C, device=DEV)
    S, cs = fresh()
    whole = run(torch.arange(T), [0, T], [1], S, cs)
    _within(whole, ref.to(DEV), 3e-5, 3e-5)
    S2, cs2 = fresh()
    cuts = [0, 1, 2, 3, 10, 19, T]
    cut = torch.cat([run(torch.arange(a, b), [0, b - a], [2], S2, cs2) for a, b in zip(cuts[:-1], cuts[1:])])
    assert torch.equal(cut, whole) and torch.equal(S2[2], S[1]) and torch.equal(cs2[2], cs[1])
    S3, cs3 = fresh()
    both = run(torch.cat([torch.arange(T), torch.arange(60)]), [0, T, T + 60], [2, 0], S3, cs3)
    assert torch.equal(both[:T], whole) and torch.equal(both[T:], whole[:60])


@pytest.mark.parametrize("H,G,D,E", [(2, 1, 64, 16), (4, 2, 128, 64), (1, 1, 128, 128), (6, 2, 64, 48)])
@pytest.mark.parametrize("decays", ["slow", "fast", "mixed"])
def test_delta_rule_four_tokens_at_a_time(H, G, D, E, decays):
    """Against float64 and the token-by-token kernel: sequences of 1 to 9 and 130 tokens side by side from states that are not
    zero, decays next to 1, next to 0 and both.  Sums of up to 128 products of unit vectors, through up to 130 tokens."""
    import plain_sugizen as P
    from ultima_b200.kernels import ops
    g = torch.Generator().manual_seed(H + D + E)
    lens = [130, 1, 2, 3, 4, 5, 7, 8, 9]
    T, n, rep = sum(lens), len(lens), H // G
    q = torch.nn.functional.normalize(torch.randn(T, G, D, generator=g), dim=-1) * D ** -0.5
    k = torch.nn.functional.normalize(torch.randn(T, G, D, generator=g), dim=-1)
    v, beta = torch.randn(T, H, E, generator=g), torch.sigmoid(torch.randn(T, H, generator=g))
    r = torch.rand(T, H, D, generator=g)
    dec = {"slow": torch.exp(-r * 1e-3), "fast": torch.exp(-r * 30), "mixed": torch.exp(-r ** 8 * 40)}[decays]
    S0 = torch.randn(n + 1, H, D, E, generator=g) * 0.3
    starts = [sum(lens[:i]) for i in range(n + 1)]
    slots = [(i * 3 + 1) % (n + 1) for i in range(n)]
    assert len(set(slots)) == n
    b = _Rows(starts, slots)
    dev = [t.reshape(T, -1).contiguous().to(DEV) for t in (q, k, v, beta, dec)]
    out, one = (torch.full((T, H * E), math.nan, device=DEV) for _ in range(2))
    S, S1 = S0.to(DEV), S0.to(DEV)
    records = torch.full((ops.delta_records_floats(n, T, H, D, E),), math.nan, device=DEV)
    ops.delta_scan_records(*dev, out, S, records, b, H, G, D, E)
    ops.delta_scan(*dev, one, S1, b, H, G, D, E)
    for i in range(n):
        sl = slice(starts[i], starts[i + 1])
        St, o = S0[slots[i]].double(), []
        for t in range(starts[i], starts[i + 1]):
            kk, qq = (x[t].double().repeat_interleave(rep, 0) for x in (k, q))
            St = dec[t].double()[:, :, None] * St
            u = beta[t].double()[:, None] * (v[t].double() - torch.einsum("hde,hd->he", St, kk))
            St = St + kk[:, :, None] * u[:, None, :]
            o.append(torch.einsum("hde,hd->he", St, qq).reshape(-1))
        for got, state in ((out, S), (one, S1)):
            _within(got[sl], torch.stack(o).to(DEV), 1e-5, 1e-5)
            _within(state[slots[i]], St.to(DEV), 1e-5, 1e-5)
    idle = [i for i in range(n + 1) if i not in slots]
    assert torch.equal(S[idle].cpu(), S0[idle])


@pytest.mark.parametrize("H,G,D,E", [(4, 2, 128, 128), (2, 2, 64, 32), (3, 1, 128, 16), (2, 1, 64, 208)])
@pytest.mark.parametrize("decays", ["slow", "fast", "mixed"])
def test_delta_rule_sixteen_tokens_at_a_time(H, G, D, E, decays):
    """Against float64 as the test above, and closer to it than the token-by-token kernel is (both rounding errors are averages over
    some 100,000 outputs; a tenth is left for the draw): sequences at the edges of sixteen tokens side by side, from states that are
    not zero."""
    from ultima_b200.kernels import ops
    g = torch.Generator().manual_seed(H + D + E)
    lens = [200, 1, 2, 15, 16, 17, 31, 32, 33, 64]
    T, n, rep = sum(lens), len(lens), H // G
    q = torch.nn.functional.normalize(torch.randn(T, G, D, generator=g), dim=-1) * D ** -0.5
    k = torch.nn.functional.normalize(torch.randn(T, G, D, generator=g), dim=-1)
    v, beta = torch.randn(T, H, E, generator=g), torch.sigmoid(torch.randn(T, H, generator=g))
    r = torch.rand(T, H, D, generator=g)
    dec = {"slow": torch.exp(-r * 1e-3), "fast": torch.exp(-r * 30), "mixed": torch.exp(-r ** 8 * 40)}[decays]
    S0 = torch.randn(n + 1, H, D, E, generator=g) * 0.3
    starts, slots = [sum(lens[:i]) for i in range(n + 1)], [(i * 3 + 1) % (n + 1) for i in range(n)]
    dev = [t.reshape(T, -1).contiguous().to(DEV) for t in (q, k, v, beta, dec)]
    for least in (1, 32):
        some = [i for i in range(n) if lens[i] >= least]
        b = _Rows(starts, slots)
        out, one = (torch.full((T, H * E), math.nan, device=DEV) for _ in range(2))
        S, S1 = S0.to(DEV), S0.to(DEV)
        chunks = torch.full((ops.delta_chunks_floats(n, T, H, D, E, least),), math.nan, device=DEV)
        ops.delta_scan_chunks(*dev, out, S, chunks, b, H, G, D, E, min_new=least)
        ops.delta_scan(*dev, one, S1, b, H, G, D, E)
        errors = [0.0, 0.0]
        for i in some:
            St, o = S0[slots[i]].double(), []
            for t in range(starts[i], starts[i + 1]):
                kk, qq = (x[t].double().repeat_interleave(rep, 0) for x in (k, q))
                St = dec[t].double()[:, :, None] * St
                u = beta[t].double()[:, None] * (v[t].double() - torch.einsum("hde,hd->he", St, kk))
                St = St + kk[:, :, None] * u[:, None, :]
                o.append(torch.einsum("hde,hd->he", St, qq).reshape(-1))
            o, sl = torch.stack(o).to(DEV), slice(starts[i], starts[i + 1])
            _within(out[sl], o, 1e-5, 1e-5)
            _within(S[slots[i]], St.to(DEV), 1e-5, 1e-5)
            for at, x in enumerate((out, one)):
                errors[at] += float((x[sl].double() - o).norm() ** 2)
        assert errors[0] ** 0.5 <= 1.1 * errors[1] ** 0.5, errors
        idle = [i for i in range(n + 1) if i not in [slots[j] for j in some]]
        assert torch.equal(S[idle].cpu(), S0[idle]) and bool(torch.isnan(out).any()) == (least > 1)


@pytest.mark.parametrize("H,G,D,E", [(4, 2, 128, 128), (2, 2, 64, 48)])
def test_delta_rule_of_sixteen_in_portions(H, G, D, E):
    """Scratch for fewer records than the step has: portions one after another, of whole sequences and of a sequence's tokens, the bits of the
    whole, and nothing written behind the scratch; with scratch that was miscounted the status word is raised."""
    from ultima_b200.engine import Runtime
    from ultima_b200.kernels import ops
    rt = Runtime(DEV, torch.bfloat16)
    g = torch.Generator(device=DEV).manual_seed(H + D)
    lens = [200, 1, 33, 64, 31, 47, 100]
    T, n = sum(lens), len(lens)
    starts = [sum(lens[:i]) for i in range(n + 1)]
    q, k = (torch.nn.functional.normalize(torch.randn(T, G, D, generator=g, device=DEV), dim=-1).reshape(T, -1) for _ in range(2))
    v, beta, dec = torch.randn(T, H * E, generator=g, device=DEV), torch.rand(T, H, generator=g, device=DEV), torch.rand(T, H * D, generator=g, device=DEV)
    S0, b, one = torch.randn(n, H, D, E, generator=g, device=DEV), _Rows(starts, list(range(n))), H * (73 * D + 36 * E)

    def run(places, lens=None):
        b.host = {} if lens is None else {"lens": lens}
        out, S = torch.full((T, H * E), math.nan, device=DEV), S0.clone()
        buf = torch.full((places * one + 64,), 7.0, device=DEV)
        launched = ops.delta_scan_chunks(q, k, v, beta, dec, out, S, buf[:places * one], b, H, G, D, E, min_new=32, rt=rt)
        assert bool((buf[places * one:] == 7.0).all())
        return out, S, launched
    whole = run(3 * T // 32)
    assert whole[2] == 2
    for places in (7, 11, 20, 29):
        for known in (None, np.array(lens)):
            out, S, launched = run(places, known)
            assert launched > 2
            assert torch.equal(S, whole[1]) and torch.equal(torch.isnan(out), torch.isnan(whole[0]))
            assert torch.equal(out.nan_to_num(), whole[0].nan_to_num())
    rt.check_status()
    run(7, np.array([33, 1, 32, 32]))                        # (the lengths are not this step's)
    with pytest.raises(RuntimeError):
        rt.check_status()


@pytest.mark.parametrize("least,below", [(1, 33), (32, 40), (32, 0)])
def test_delta_rule_of_four_leaves_longer_sequences_alone(least, below):
    """Sequences below ``least`` tokens, and of ``below`` or more, keep their states and outputs; the others have the bits they have alone."""
    from ultima_b200.kernels import ops
    H, G, D, E = 4, 2, 64, 32
    g = torch.Generator(device=DEV).manual_seed(below)
    lens = [31, 32, 33, 64, 39, 5, 40, 41]
    T, n = sum(lens), len(lens)
    starts = [sum(lens[:i]) for i in range(n + 1)]
    q, k = (torch.nn.functional.normalize(torch.randn(T, G, D, generator=g, device=DEV), dim=-1).reshape(T, -1) for _ in range(2))
    x = [q, k, torch.randn(T, H * E, generator=g, device=DEV), torch.rand(T, H, generator=g, device=DEV), torch.rand(T, H * D, generator=g, device=DEV)]
    S0 = torch.randn(n, H, D, E, generator=g, device=DEV)

    def run(seqs):
        rows = torch.cat([torch.arange(starts[i], starts[i + 1], device=DEV) for i in seqs])
        cut = [0]
        for i in seqs:
            cut.append(cut[-1] + lens[i])
        out, S = torch.full((len(rows), H * E), math.nan, device=DEV), S0.clone()
        records = torch.empty(ops.delta_records_floats(len(seqs), len(rows), H, D, E, least), device=DEV)
        ops.delta_scan_records(*(t[rows].contiguous() for t in x), out, S, records, _Rows(cut, seqs), H, G, D, E, min_new=least, below=below)
        return out, S
    out, S = run(list(range(n)))
    for i, m in enumerate(lens):
        mine = out[starts[i]:starts[i + 1]]
        if m < least or (below and m >= below):
            assert torch.equal(S[i], S0[i]) and bool(torch.isnan(mine).all()), m
        else:
            alone, S1 = run([i])
            assert torch.equal(alone, mine) and torch.equal(S1[i], S[i]) and bool(torch.isfinite(mine).all()), m


@pytest.mark.parametrize("place", [16, 17, 24, 31, 34])
def test_delta_rule_of_sixteen_keeps_later_tokens_out(place):
    """As the test of four below; an infinite value reaches its own column of the state alone, as infinities, not NaN."""
    from ultima_b200.kernels import ops
    H, G, D, E, T = 2, 1, 128, 64, 35
    g = torch.Generator(device=DEV).manual_seed(place)
    q, k = (torch.nn.functional.normalize(torch.randn(T, G, D, generator=g, device=DEV), dim=-1).reshape(T, -1) for _ in range(2))
    v, beta = torch.randn(T, H * E, generator=g, device=DEV), torch.rand(T, H, generator=g, device=DEV)
    dec, S0 = torch.rand(T, H * D, generator=g, device=DEV), torch.randn(1, H, D, E, generator=g, device=DEV)
    b = _Rows([0, T], [0])

    def run(inputs):
        out, S = torch.empty(T, H * E, device=DEV), S0.clone()
        chunks = torch.empty(ops.delta_chunks_floats(1, T, H, D, E), device=DEV)
        ops.delta_scan_chunks(*inputs, out, S, chunks, b, H, G, D, E)
        return out, S
    clean, _ = run((q, k, v, beta, dec))
    for which in range(5):
        for what in (math.inf, math.nan):
            bad = [x.clone() for x in (q, k, v, beta, dec)]
            bad[which][place] = what
            assert torch.equal(run(bad)[0][:place], clean[:place]), (which, what)
    bad = v.clone()
    bad[T - 1, 5] = math.inf                                 # (the last sixteen hold three tokens)
    out, S = run((q, k, bad, beta, dec))
    one, S1 = torch.empty(T, H * E, device=DEV), S0.clone()
    ops.delta_scan(q, k, bad, beta, dec, one, S1, b, H, G, D, E)
    assert torch.equal(torch.isnan(S[0, 0, :, 5]), torch.isnan(S1[0, 0, :, 5])) and torch.equal(torch.isinf(S[0]), torch.isinf(S1[0]))
    assert not math.isfinite(out[T - 1, 5]) and not math.isfinite(one[T - 1, 5])
    assert bool(torch.isfinite(S[0, 0][:, torch.arange(E, device=DEV) != 5]).all())


@pytest.mark.parametrize("H,N,G", [(2, 64, 1), (4, 128, 2), (3, 128, 3)])
@pytest.mark.parametrize("decays", ["slow", "fast", "mixed"])
def test_state_space_recurrence_in_chunks(H, N, G, decays):
    """Against float64 and the token-by-token kernel: sequences at the edges of chunks of 64 and of their halves, side by side,
    from states that are not zero, decays next to 1, next to 0 and both.  Sums of up to 128 and 260 terms relative to the largest
    result of the sequence."""
    from ultima_b200.kernels import ops
    P = 64
    g = torch.Generator().manual_seed(H + N + G)
    lens = [260, 1, 31, 32, 33, 63, 64, 65, 128, 129, 2]
    T, n = sum(lens), len(lens)
    C = H * P + 2 * G * N
    xbc = torch.randn(T, C, generator=g)
    dt = torch.nn.functional.softplus(torch.randn(T, H, generator=g))
    r = torch.rand(T, H, generator=g)
    dec = {"slow": torch.exp(-r * 1e-3), "fast": torch.exp(-r * 30), "mixed": torch.exp(-r ** 8 * 40)}[decays]
    Dw, S0 = torch.randn(H, generator=g), torch.randn(n + 1, H, N, P, generator=g)
    starts = [sum(lens[:i]) for i in range(n + 1)]
    slots = [(i * 5 + 1) % (n + 1) for i in range(n)]
    assert len(set(slots)) == n
    b = _Rows(starts, slots)
    dev = [t.contiguous().to(DEV) for t in (xbc, dt, dec, Dw)]
    out, one = (torch.full((T, H * P), math.nan, device=DEV) for _ in range(2))
    S, S1 = S0.to(DEV), S0.to(DEV)
    places = ops.ssm_chunk_places(n, T, P, N)
    scratch = [torch.full(sh, math.nan, device=DEV) for sh in ((places, H, N, P), (places, H), (places, G, 64, 64))]
    ops.ssm_scan_chunks(*dev, out, S, *scratch, b, H, P, N, G)
    ops.ssm_scan(*dev, one, S1, b, H, P, N, G)
    for i in range(n):
        St, o = S0[slots[i]].double(), []
        for t in range(starts[i], starts[i + 1]):
            x = xbc[t, :H * P].double().view(H, P)
            B, Cc = (xbc[t, H * P + k * G * N:H * P + (k + 1) * G * N].double().view(G, N).repeat_interleave(H // G, 0) for k in (0, 1))
            St = dec[t].double()[:, None, None] * St + (dt[t].double()[:, None] * B)[:, :, None] * x[:, None, :]
            o.append((torch.einsum("hnp,hn->hp", St, Cc) + Dw.double()[:, None] * x).reshape(-1))
        o = torch.stack(o).to(DEV)
        for got, state in ((out, S), (one, S1)):
            _within(got[starts[i]:starts[i + 1]], o, 2e-6, 2e-6 * float(o.abs().max()))
            _within(state[slots[i]], St.to(DEV), 2e-6, 2e-6 * float(St.abs().max()))
    idle = [i for i in range(n + 1) if i not in slots]
    assert torch.equal(S[idle].cpu(), S0[idle])


def _f32_attention(k, v, q, before, new, nh, nkv, hd, window=None, split=None):
    """One sequence whose positions lie in pages in order: attention of the ``new`` last of ``before + new`` tokens."""
    from ultima_b200.engine import Runtime
    from ultima_b200.kernels import ops
    rt = Runtime(DEV, torch.float32)
    n_pages = -(-(before + new) // 64)
    kc, vc = (torch.zeros(n_pages, nkv, 64, hd, device=DEV) for _ in range(2))
    for cache, x in ((kc, k), (vc, v)):
        for pg in range(n_pages):
            part = x[pg * 64:(pg + 1) * 64]
            cache[pg, :, :part.shape[0]] = part.permute(1, 0, 2)
    kv = _View(kc, vc, torch.arange(n_pages, device=DEV, dtype=torch.int32)[None].contiguous(), n_pages * 64, window)
    out = torch.full((new, nh * hd), 7.0, device=DEV)
    assert ops.attn_f32_fits(q, kv, out, hd)
    ops.attn_f32(q, kv, out, _Batch([before], [new]), nh, nkv, hd, hd ** -0.5, rt, split=split)
    return out


@pytest.mark.parametrize("split", [0, 3])
@pytest.mark.parametrize("before,new", [(200, 1), (130, 40)])
def test_float32_attention_shows_a_page_of_nan(before, new, split):
    """A page whose keys are NaN, as unwritten pages are in a poisoned cache, makes every row that sees it NaN: first, between and
    last, with one row a head and with many."""
    nh, nkv, hd = 8, 2, 64
    g = torch.Generator(device=DEV).manual_seed(before)
    n = before + new
    k, v = torch.randn(n, nkv, hd, generator=g, device=DEV), torch.randn(n, nkv, hd, generator=g, device=DEV)
    q = torch.randn(new, nh * hd, generator=g, device=DEV)
    assert bool(torch.isfinite(_f32_attention(k, v, q, before, new, nh, nkv, hd, split=split)).all())
    for page in range(-(-n // 64)):
        bad = k.clone()
        bad[page * 64:(page + 1) * 64] = math.nan
        got = _f32_attention(bad, v, q, before, new, nh, nkv, hd, split=split)
        sees = torch.arange(before, n, device=DEV) >= page * 64
        assert bool(torch.isnan(got[sees]).all()) and bool(torch.isfinite(got[~sees]).all())


@pytest.mark.parametrize("split", [0, 2])
@pytest.mark.parametrize("window", [None, 70])
@pytest.mark.parametrize("new", [3, 40])
def test_float32_attention_keeps_other_tokens_values_out(new, window, split):
    """A value that a row does not see, because it comes later or has left the window, does not reach the row though the block reads
    it for another: rows that do not see it keep their bits, whatever it is."""
    nh, nkv, hd, before = 4, 1, 128, 90
    g = torch.Generator(device=DEV).manual_seed(new)
    n = before + new
    k, v = torch.randn(n, nkv, hd, generator=g, device=DEV), torch.randn(n, nkv, hd, generator=g, device=DEV)
    q = torch.randn(new, nh * hd, generator=g, device=DEV)
    clean = _f32_attention(k, v, q, before, new, nh, nkv, hd, window, split)
    pos = torch.arange(before, n, device=DEV)
    for place in (n - 1, before + 1, before + 1 - (window or n), before + new // 2 - (window or n)):
        if place < 0:
            continue
        for what in (math.inf, math.nan):
            bad = v.clone()
            bad[place] = what
            got = _f32_attention(k, bad, q, before, new, nh, nkv, hd, window, split)
            sees = (pos >= place) & (place > pos - (window or n))
            assert torch.equal(got[~sees], clean[~sees]) and not bool(torch.isfinite(got[sees]).any())


@pytest.mark.parametrize("place", [3, 37, 63, 70])
def test_state_space_chunks_keep_later_tokens_out(place):
    """Infinite and undefined numbers of a token, in every input of the recurrence, leave the tokens before it their bits."""
    from ultima_b200.kernels import ops
    H, P, N, G, T = 4, 64, 128, 2, 129
    g = torch.Generator(device=DEV).manual_seed(place)
    xbc = torch.randn(T, H * P + 2 * G * N, generator=g, device=DEV)
    dt, dec = torch.rand(T, H, generator=g, device=DEV), torch.rand(T, H, generator=g, device=DEV)
    Dw, S0 = torch.randn(H, generator=g, device=DEV), torch.randn(1, H, N, P, generator=g, device=DEV)
    places, b = ops.ssm_chunk_places(1, T, P, N), _Rows([0, T], [0])

    def run(*inputs):
        out = torch.empty(T, H * P, device=DEV)
        scratch = [torch.empty(sh, device=DEV) for sh in ((places, H, N, P), (places, H), (places, G, 64, 64))]
        ops.ssm_scan_chunks(*inputs, Dw, out, S0.clone(), *scratch, b, H, P, N, G)
        return out
    clean = run(xbc, dt, dec)
    for which in range(3):
        for what in (math.inf, math.nan):
            bad = [xbc.clone(), dt.clone(), dec.clone()]
            bad[which][place] = what
            assert torch.equal(run(*bad)[:place], clean[:place]), (which, what)


@pytest.mark.parametrize("place", [4, 5, 6, 7, 34])
def test_delta_rule_of_four_keeps_later_tokens_out(place):
    """Infinite and undefined numbers of a token, in every input of the recurrence, leave the tokens before it their bits; an infinite
    value behind a closed gate in the last, partly filled four leaves the other columns of the state theirs."""
    from ultima_b200.kernels import ops
    H, G, D, E, T = 2, 1, 128, 64, 35
    g = torch.Generator(device=DEV).manual_seed(place)
    q, k = (torch.nn.functional.normalize(torch.randn(T, G, D, generator=g, device=DEV), dim=-1).reshape(T, -1) for _ in range(2))
    v, beta = torch.randn(T, H * E, generator=g, device=DEV), torch.rand(T, H, generator=g, device=DEV)
    dec, S0 = torch.rand(T, H * D, generator=g, device=DEV), torch.randn(1, H, D, E, generator=g, device=DEV)
    b = _Rows([0, T], [0])

    def run(inputs):
        out, S = torch.empty(T, H * E, device=DEV), S0.clone()
        records = torch.empty(ops.delta_records_floats(1, T, H, D, E), device=DEV)
        ops.delta_scan_records(*inputs, out, S, records, b, H, G, D, E)
        return out, S
    clean, _ = run((q, k, v, beta, dec))
    for which in range(5):
        for what in (math.inf, math.nan):
            bad = [x.clone() for x in (q, k, v, beta, dec)]
            bad[which][place] = what
            assert torch.equal(run(bad)[0][:place], clean[:place]), (which, what)
    bad = v.clone()
    bad[T - 1, 5] = math.inf                                 # (the last four hold three tokens)
    out, S = run((q, k, bad, beta, dec))
    one, S1 = torch.empty(T, H * E, device=DEV), S0.clone()
    ops.delta_scan(q, k, bad, beta, dec, one, S1, b, H, G, D, E)
    assert torch.equal(torch.isnan(S[0, 0, :, 5]), torch.isnan(S1[0, 0, :, 5]))
    assert not math.isfinite(out[T - 1, 5]) and not math.isfinite(one[T - 1, 5])      # (a sum of infinities of both signs, or of one)
    assert bool(torch.isfinite(S[0, 0][:, torch.arange(E, device=DEV) != 5]).all())


@pytest.mark.parametrize("decay", [0.2, 6.0])
@pytest.mark.parametrize("N", [64, 128])
def test_state_space_chunks_are_as_close_to_64_bits_as_token_by_token(N, decay):
    """The error of 320 tokens' outputs, as a 2-norm over 640,000 of them, for which both kernels' rounding errors are averages: the
    chunks' is no larger than the token-by-token kernel's (a tenth is left for the draw; one chain of N terms was off by 1.6 to 2.3
    times as much)."""
    from ultima_b200.kernels import ops
    H, G, P, T = 32, 2, 64, 320
    g = torch.Generator(device=DEV).manual_seed(N)
    xbc = torch.randn(T, H * P + 2 * G * N, generator=g, device=DEV)
    dt = torch.nn.functional.softplus(torch.randn(T, H, generator=g, device=DEV) - 2)
    dec = torch.exp(-decay * torch.rand(T, H, generator=g, device=DEV))
    Dw, S0 = torch.randn(H, generator=g, device=DEV), torch.randn(1, H, N, P, generator=g, device=DEV)
    b, places = _Rows([0, T], [0]), ops.ssm_chunk_places(1, T, P, N)
    St, ref = S0[0].double(), []
    for t in range(T):
        x = xbc[t, :H * P].double().view(H, P)
        B, Cc = (xbc[t, H * P + i * G * N:H * P + (i + 1) * G * N].double().view(G, N).repeat_interleave(H // G, 0) for i in (0, 1))
        St = dec[t].double()[:, None, None] * St + (dt[t].double()[:, None] * B)[:, :, None] * x[:, None, :]
        ref.append((torch.einsum("hnp,hn->hp", St, Cc) + Dw.double()[:, None] * x).reshape(-1))
    ref = torch.stack(ref)
    out, one = (torch.empty(T, H * P, device=DEV) for _ in range(2))
    scratch = [torch.empty(sh, device=DEV) for sh in ((places, H, N, P), (places, H), (places, G, 64, 64))]
    ops.ssm_scan_chunks(xbc, dt, dec, Dw, out, S0.clone(), *scratch, b, H, P, N, G)
    ops.ssm_scan(xbc, dt, dec, Dw, one, S0.clone(), b, H, P, N, G)
    chunks, tokens = (float((y.double() - ref).norm() / ref.norm()) for y in (out, one))
    assert chunks <= 1.1 * tokens, (chunks, tokens)


@pytest.mark.parametrize("kind", ["delta", "space"])
def test_a_sequences_recurrence_follows_its_own_tokens(kind):
    """In a 16-bit run, sequences on both sides of the lengths from which the forms for prompts are taken have, beside one another, the
    bits they have alone: outputs and states."""
    from ultima_b200.engine import Runtime
    from ultima_b200.kernels import ops
    from ultima_b200.parts.delta import GatedDelta
    from ultima_b200.parts.ssm import StateSpaceDual
    rt = Runtime(DEV, torch.bfloat16)
    g = torch.Generator(device=DEV).manual_seed(5)
    rand, randn = (lambda *s: torch.rand(*s, generator=g, device=DEV)), (lambda *s: torch.randn(*s, generator=g, device=DEV))
    if kind == "delta":
        least, H, G, D, E = ops.DELTA_RECORDS_MIN, 4, 2, 64, 128
        part = GatedDelta(256, H, G, D, E, 4, decay_rank=8, gate_rank=8)
        long = ops.DELTA_CHUNKS_MIN
        lens = [1, least + 5, long, least - 1, 3, long - 1, least, 1, long + 17, 2 * least + 1, 7]
    else:
        least, H, G, D, E = ops.SSM_CHUNKS_MIN, 4, 2, 64, 64
        part = StateSpaceDual(256, H, E, D, G, 4, 2, 1e-5)
        part.d_skip = randn(H)
        lens = [1, least - 1, least + 1, 2, least, 65, 2 * least + 3]
    T = sum(lens)
    starts = [sum(lens[:i]) for i in range(len(lens) + 1)]
    unit = lambda x: torch.nn.functional.normalize(x, dim=-1).reshape(T, -1)                # noqa: E731
    inputs = [unit(randn(T, G, D)), unit(randn(T, G, D)), randn(T, H * E), rand(T, H), rand(T, H * D)] if kind == "delta" else \
        [randn(T, H * E + 2 * G * D), rand(T, H), rand(T, H)]
    S0 = randn(len(lens), H, D, E)

    def run(seqs):
        rows = torch.cat([torch.arange(starts[i], starts[i + 1], device=DEV) for i in seqs])
        n = [lens[i] for i in seqs]
        b = _Rows([sum(n[:i]) for i in range(len(n) + 1)], seqs)
        b.min_new = min(n)
        S, out = S0.clone(), torch.full((len(rows), H * E), math.nan, device=DEV)
        rt.arena.reset(0)
        part.recurrence(*(x[rows].contiguous() for x in inputs), out, S, b, rt)
        return out, S
    together, S = run(list(range(len(lens))))
    assert bool(torch.isfinite(together).all())
    for i in range(len(lens)):
        alone, S1 = run([i])
        assert torch.equal(alone, together[starts[i]:starts[i + 1]]) and torch.equal(S1[i], S[i]), lens[i]


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="one device only")
def test_float32_kernels_on_a_second_device():
    """A kernel's leave to use more than 48 KB of shared memory belongs to a device: a program that moves to another one asks again."""
    from ultima_b200.kernels import ops
    for device in (0, 1):
        with torch.cuda.device(device):
            g = torch.Generator(device=f"cuda:{device}").manual_seed(1)
            a, w = (torch.randn(n, 256, generator=g, device=f"cuda:{device}") for n in (40, 130))
            for form in (32, 64, 128, -32, -64):
                out = torch.empty(40, 130, device=f"cuda:{device}")
                ops.gemm_f32(a, w, out, form=form)
                assert float((out.double() - a.double() @ w.double().T).abs().max()) < 1e-3
