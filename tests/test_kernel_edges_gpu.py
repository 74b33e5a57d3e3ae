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
