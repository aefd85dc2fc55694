"""The pipelined true 32-bit product and attention at the edges of their tiles, against float64."""
import pytest
import torch

from test_attention_tc_gpu import exact, launch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M, N, K", [(9, 64, 4), (64, 65, 36), (65, 63, 32), (200, 130, 1000), (384, 1536, 1024), (77, 48, 64)])
def test_product(M, N, K):
    from qwen3_tts_cuda_graphs_b200 import codec as C

    torch.manual_seed(M)
    A, B, bias = torch.randn(M, K, device="cuda"), torch.randn(N, K, device="cuda"), torch.randn(N, device="cuda")
    want, mag = A.double() @ B.double().T, A.double().abs() @ B.double().abs().T
    for flags in (C.F_OUT_F32, C.F_OUT_F32 | C.F_BIAS) + ((C.F_OUT_F32 | C.F_SWIGLU,) if N % 2 == 0 else ()):
        glu = bool(flags & C.F_SWIGLU)
        out = torch.full((M + 1, N // 2 if glu else N), 5.0, device="cuda")
        o = C.Op()
        o.kind, o.flags, o.M, o.N, o.K, o.taps, o.cin, o.a_rows, o.lda, o.ldc, o.col_mod = C.K_GEMM, flags | C.F_F32 | C.F_NOROUND, M, N, K, 1, K, M, K, out.shape[1], N
        o.A, o.B, o.C, o.bias = A.data_ptr(), B.data_ptr(), out.data_ptr(), bias.data_ptr()
        launch(o)
        y = want + bias.double() if flags & C.F_BIAS else want
        if glu:      # silu's slope is at most 1.1: the two sums' errors, and a few roundings of the unit
            e = K * 2.0 ** -24 * mag
            unit = y[:, 0::2] * torch.sigmoid(y[:, 0::2]) * y[:, 1::2]
            assert ((out[:M].double() - unit).abs() <= 1.1 * e[:, 0::2] * y[:, 1::2].abs() + e[:, 1::2] * y[:, 0::2].abs() + 2.0 ** -20 * unit.abs() + 1e-6).all()
        else:
            assert ((out[:M].double() - y).abs() <= K * 2.0 ** -24 * mag + 2.0 ** -23 * y.abs()).all()
        assert (out[M] == 5).all()


@pytest.mark.parametrize("M, N, K", [(768, 768, 20), (769, 736, 100), (2100, 320, 64), (640, 960, 1024)])      # 144, 156, 165, 150 tiles
def test_product_of_a_wave_and_more(M, N, K):
    test_product(M, N, K)


# rows, positions in front, heads, key heads, key splits, options
@pytest.mark.parametrize("rows, first, heads, kv, splits, opt", [(9, 0, 4, 2, 1, {}), (33, 31, 8, 2, 1, {}), (64, 64, 6, 2, 3, {}), (100, 300, 8, 2, 4, dict(window=64)), (90, 200, 4, 4, 1, dict(window=40, keep=3)),
                                                                  (200, 100, 2, 1, 2, dict(chunk=70)), (40, 500, 12, 4, 16, dict(cap=30.0)), (384, 300, 8, 2, 3, dict(window=512)), (12, 0, 32, 1, 5, {})])
def test_attention(rows, first, heads, kv, splits, opt):
    from qwen3_tts_cuda_graphs_b200 import codec as C

    torch.manual_seed(rows + heads)
    L = first + rows
    q, sink = torch.randn(rows, heads * 128, device="cuda"), torch.randn(heads, device="cuda")
    kc = torch.full((L + 70, kv * 128), float("nan"), device="cuda")      # rows beyond the last position are never used
    vc = kc.clone()
    kc[:L], vc[:L] = torch.randn(L, kv * 128, device="cuda"), torch.randn(L, kv * 128, device="cuda")
    pos, out = torch.tensor([first], dtype=torch.int32, device="cuda"), torch.zeros(rows, heads * 128, device="cuda")
    ws = torch.zeros(rows * heads * splits * 130, device="cuda")
    o = C.Op()
    o.kind, o.flags, o.M, o.N, o.i0, o.i1, o.i2, o.cin, o.f0, o.f1 = C.K_CACHE_ATTN, C.F_OUT_F32 | C.F_F32, rows, heads * 128, heads, kv, 128, 128, 128 ** -0.5, opt.get("cap", 0.0)
    o.K, o.a_rows, o.tap_off[0], o.m_begin = opt.get("window", 0), opt.get("keep", 0), opt.get("chunk", 0), splits
    o.A, o.lda, o.B, o.ldr, o.p1, o.taps, o.p0 = q.data_ptr(), heads * 128, kc.data_ptr(), kv * 128, vc.data_ptr(), kv * 128, pos.data_ptr()
    o.C, o.ldc, o.col_mod, o.scale, o.ws, o.ws_bytes = out.data_ptr(), heads * 128, 1, sink.data_ptr(), ws.data_ptr(), ws.numel() * 4
    launch(o)
    want = exact(q.double().view(rows, heads, 128), kc[:L].double().view(L, kv, 128), vc[:L].double().view(L, kv, 128), first, 128 ** -0.5, opt.get("cap", 0.0),
                 opt.get("window", 0), opt.get("keep", 0), opt.get("chunk", 0), sink.double())
    # scores of about 1 from 128 products and weights from expf: a few 2^-23 each
    assert float((out.double() - want.reshape(rows, -1)).norm() / want.norm()) < 1e-6
