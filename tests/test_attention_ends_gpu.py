"""Attention of many rows where a CTA takes a row group from either end, or one group while there are a few more groups than SMs: against float64, ragged rows, caps near and far."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,pos,H,G", [(1185, 0, 16, 4), (1500, 0, 16, 4), (1500, 600, 16, 4), (1601, 0, 16, 4), (2047, 1, 16, 4), (1217, 300, 8, 2), (40, 0, 296, 148), (129, 0, 110, 110), (2369, 0, 2, 1)])
@pytest.mark.parametrize("cap,spread", [(0.0, 1.0), (50.0, 1.0), (4.0, 1.0), (20.0, 3.0)])      # no cap; scores within 0.35 of it; beyond it in some warps; in most
def test_against_float64(M, pos, H, G, cap, spread):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    lib, D = K.load_lib(), 128
    g = torch.Generator(device="cuda").manual_seed(M + H)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    q, k, v, sink = (rnd(M, H * D) * spread).bfloat16().float(), rnd(pos + M, G * D).bfloat16(), rnd(pos + M, G * D).bfloat16(), rnd(H)
    out, where = torch.zeros(M, H * D, device="cuda"), torch.tensor([pos], device="cuda", dtype=torch.int32)
    a = K.Op()
    a.kind, a.M, a.N, a.i0, a.i1, a.i2, a.cin, a.f0, a.f1, a.lda, a.ldr, a.taps, a.ldc, a.flags = K.K_CACHE_ATTN, M, H * D, H, G, D, D, D ** -0.5, cap, H * D, G * D, G * D, H * D, K.F_OUT_F32
    a.A, a.B, a.p1, a.p0, a.C, a.scale = q.data_ptr(), k.data_ptr(), v.data_ptr(), where.data_ptr(), out.data_ptr(), sink.data_ptr()
    assert lib.fq3c_run((K.Op * 1)(a), 1, torch.cuda.current_stream().cuda_stream) == 0, lib.fq3c_last_error()
    torch.cuda.synchronize()
    assert lib.fq3c_wait_errors() == 0
    hide = torch.arange(pos + M, device="cuda")[None] > torch.arange(pos, pos + M, device="cuda")[:, None]
    for h in sorted({0, 1, H // 2, H - 1}):
        n = h // (H // G)
        s = q[:, h * D:(h + 1) * D].double() @ k[:, n * D:(n + 1) * D].double().T * D ** -0.5
        s = (cap * torch.tanh(s / cap) if cap else s).masked_fill(hide, -torch.inf)
        w = torch.cat([s, sink[h].double().expand(M, 1)], 1).softmax(-1)[:, :-1]
        vv = v[:, n * D:(n + 1) * D].double()
        # weights of 16 bits (2^-17 of each) and scores off by some 1e-6 of the cap or of their sum of 128 products
        bound = (2.0 ** -16 + 4e-6 * max(cap, 8.0 * spread)) * (w @ vv.abs()) + 1e-6
        assert ((out[:, h * D:(h + 1) * D].double() - w @ vv).abs() <= bound).all()


def capped(q, k, v, H, G, cap, scale, pos=0):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    lib, M, D = K.load_lib(), q.shape[0], 128
    out, where = torch.zeros(M, H * D, device="cuda"), torch.tensor([pos], device="cuda", dtype=torch.int32)
    a = K.Op()
    a.kind, a.M, a.N, a.i0, a.i1, a.i2, a.cin, a.f0, a.f1, a.lda, a.ldr, a.taps, a.ldc, a.flags = K.K_CACHE_ATTN, M, H * D, H, G, D, D, scale, cap, H * D, G * D, G * D, H * D, K.F_OUT_F32
    a.A, a.B, a.p1, a.p0, a.C = q.data_ptr(), k.data_ptr(), v.data_ptr(), where.data_ptr(), out.data_ptr()
    assert lib.fq3c_run((K.Op * 1)(a), 1, torch.cuda.current_stream().cuda_stream) == 0, lib.fq3c_last_error()
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("M,H,G", [(9, 4, 2), (200, 16, 4), (1500, 4, 4)])
def test_a_cap_under_a_negative_scale(M, H, G):
    """The products of q and k under -s are those of -q and k under s: same bits, wherever the scores lie under the cap."""
    g = torch.Generator(device="cuda").manual_seed(M)
    q, k, v = torch.randn(M, H * 128, device="cuda", generator=g) * 4, *(torch.randn(M, G * 128, device="cuda", generator=g).bfloat16() for _ in range(2))
    for cap in (4.0, 200.0):
        assert torch.equal(capped(q, k, v, H, G, cap, -(128 ** -0.5)), capped(-q, k, v, H, G, cap, 128 ** -0.5))


@pytest.mark.parametrize("pos", [0, 70])
@pytest.mark.parametrize("spread", [1.0, 8.0])      # all scores near, some of most warps far up the cap
def test_a_capped_score_that_is_nan(pos, spread):
    """It counts as -cap, whatever the scores beside it are."""
    M, H, G, cap = 300, 8, 2, 20.0
    g = torch.Generator(device="cuda").manual_seed(pos)
    q, k, v = (torch.randn(M, H * 128, device="cuda", generator=g) * spread).bfloat16().float(), *(torch.randn(pos + M, G * 128, device="cuda", generator=g).bfloat16() for _ in range(2))
    hide = torch.arange(pos + M, device="cuda")[None] > torch.arange(pos, pos + M, device="cuda")[:, None]
    for at in (pos + 1, pos + 40, pos + 201, pos + M - 1):
        bad = k.clone()
        bad[at, 5] = torch.nan
        out = capped(q, bad, v, H, G, cap, 128 ** -0.5, pos)
        for h in range(H):
            n = h // (H // G)
            s = cap * torch.tanh((q[:, h * 128:(h + 1) * 128].double() @ bad[:, n * 128:(n + 1) * 128].double().T * 128 ** -0.5) / cap)
            w = s.nan_to_num(-cap).masked_fill(hide, -torch.inf).softmax(-1)
            vv = v[:, n * 128:(n + 1) * 128].double()
            bound = (2.0 ** -16 + 4e-6 * cap) * (w @ vv.abs()) + 1e-6      # as above
            assert ((out[:, h * 128:(h + 1) * 128].double() - w @ vv).abs() <= bound).all()
