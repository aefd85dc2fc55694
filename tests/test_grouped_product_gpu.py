"""The pipelined grouped product at the edges of its tiles, against float64."""
import pytest
import torch

from test_attention_tc_gpu import launch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes, N, K", [((17,), 64, 64), ((0, 1, 31, 0), 66, 8), ((33, 0, 64, 65), 62, 72), ((127, 128, 129), 130, 136), ((3, 300, 0, 1, 200), 192, 1000), ((300, 210), 2, 264)])
def test_grouped(sizes, N, K):
    from qwen3_tts_cuda_graphs_b200 import codec as C

    torch.manual_seed(N)
    E, M, T = len(sizes), sum(sizes), 40
    A, B = torch.randn(T, K + 8, device="cuda").bfloat16(), torch.randn(E, N, K, device="cuda").bfloat16()
    seg = torch.tensor([sum(sizes[:e]) for e in range(E + 1)], dtype=torch.int32, device="cuda")
    rows = torch.randint(0, T, (M,), dtype=torch.int32, device="cuda")
    w = torch.rand(M, device="cuda")
    a = A[:, :K].double()[rows.long()]
    want, mag = torch.empty(M, N, dtype=torch.float64, device="cuda"), torch.empty(M, N, dtype=torch.float64, device="cuda")
    for e in range(E):
        s = slice(int(seg[e]), int(seg[e + 1]))
        want[s], mag[s] = a[s] @ B[e].double().T, a[s].abs() @ B[e].double().abs().T
    err = K * 2.0 ** -23 * mag      # exact products, f32 sums (the tensor cores' may truncate)
    for flags in (0, C.F_OUT_F32, C.F_OUT_F32 | C.F_RELU2, C.F_SWIGLU, C.F_SWIGLU | C.F_OUT_F32):
        glu, f32 = bool(flags & C.F_SWIGLU), bool(flags & C.F_OUT_F32)
        out = torch.full((M + 1, N // 2 if glu else N), 5.0, device="cuda", dtype=torch.float32 if f32 else torch.bfloat16)
        o = C.Op()
        o.kind, o.flags, o.M, o.N, o.K, o.i0, o.lda, o.ldc = C.K_GGEMM, flags, M, N, K, E, K + 8, out.shape[1]
        o.A, o.B, o.C, o.p0, o.p1 = A.data_ptr(), B.data_ptr(), out.data_ptr(), seg.data_ptr(), rows.data_ptr()
        if glu:
            o.scale = w.data_ptr()
        launch(o)
        if glu:      # silu's slope is at most 1.1: the two sums' errors, and a few roundings of the unit
            g, u, c = want[:, 0::2] * w.double()[:, None], want[:, 1::2] * w.double()[:, None], w.double()[:, None]
            y = g * torch.sigmoid(g) * u
            tol = 1.1 * c * (err[:, 0::2] * u.abs() + err[:, 1::2] * g.abs()) + 2.0 ** -20 * y.abs() + 1e-6
        elif flags & C.F_RELU2:
            y = want.clamp(min=0) ** 2
            tol = 2 * err * want.abs() + err ** 2 + 2.0 ** -22 * y
        else:
            y, tol = want, err + 2.0 ** -23 * want.abs()
        assert ((out[:M].double() - y).abs() <= tol + (0 if f32 else 2.0 ** -8 * (y.abs() + tol))).all()
        assert (out[M].float() == 5).all()
