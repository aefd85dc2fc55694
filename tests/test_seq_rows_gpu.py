"""Many rows of the sequence models: rotation and cache rows without a warp per head, norms of groups by the pieces a lane needs, the delta rule in blocks of 16 tokens."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def play(*ops):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    lib = K.load_lib()
    assert lib.fq3c_run((K.Op * len(ops))(*ops), len(ops), torch.cuda.current_stream().cuda_stream) == 0, lib.fq3c_last_error()
    torch.cuda.synchronize()


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("M,pos,H,G,d,dv,turned,half", [(9, 0, 16, 4, 128, 128, 32, False), (20, 700, 3, 1, 64, 48, 64, True), (33, 5, 4, 2, 40, 7, 6, False), (12, 90, 2, 0, 128, 0, 128, True), (17, 3, 2, 2, 96, 96, 0, False)])
def test_rotation_of_many_rows_as_row_by_row(M, pos, H, G, d, dv, turned, half, f32):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    g = torch.Generator(device="cuda").manual_seed(M + d)
    dt = torch.float32 if f32 else torch.bfloat16
    cols = H * d + G * (d + dv) + 5
    rows = torch.randn(M, cols, device="cuda", generator=g)
    freq, lo = torch.rand(max(1, turned // 2), device="cuda", generator=g), torch.rand(max(1, turned // 2), device="cuda", generator=g) * 1e-8
    got = []
    for step in (M, 1):      # (a single row takes a warp per head)
        x, k, v = rows.clone(), torch.zeros(pos + M, max(1, G * d), device="cuda", dtype=dt), torch.zeros(pos + M, max(1, G * dv), device="cuda", dtype=dt)
        for m in range(0, M, step):
            where = torch.tensor([pos + m], device="cuda", dtype=torch.int32)
            r = K.Op()
            r.kind, r.M, r.i0, r.i1, r.i2, r.cin, r.taps, r.K, r.a_rows, r.lda = K.K_ROT_APPEND, step, H, G, d, dv, turned, H * d, (H + G) * d, cols
            r.flags, r.f1 = (K.F_F32 if f32 else 0) | (K.F_ROT_HALF if half else 0), 1.25
            r.A, r.p0 = x[m].data_ptr(), where.data_ptr()
            if turned:
                r.B, r.p1 = freq.data_ptr(), lo.data_ptr()
            if G:
                r.C, r.ldc, r.C2, r.ldr = k.data_ptr(), k.shape[1], v.data_ptr(), v.shape[1]
            play(r)
        got.append((x, k, v))
    assert all(torch.equal(a, b) for a, b in zip(*got))


@pytest.mark.parametrize("size", [4, 124, 128, 132, 256, 260, 384, 512])
@pytest.mark.parametrize("gate", [0, 1, 2])      # none, before the statistics, behind the weights
def test_group_norm_of_many_groups(size, gate):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    M, groups = 130, 8
    g = torch.Generator(device="cuda").manual_seed(size)
    x, z, w = torch.randn(M, groups * size, device="cuda", generator=g), torch.randn(M, groups * size, device="cuda", generator=g), torch.randn(size, device="cuda", generator=g)
    out = torch.zeros(M, groups * size, device="cuda")
    o = K.Op()
    o.kind, o.M, o.N, o.i0, o.f0, o.A, o.lda, o.C, o.ldc, o.scale, o.i2, o.flags = K.K_GNORM, M, groups * size, groups, 1e-5, x.data_ptr(), groups * size, out.data_ptr(), groups * size, w.data_ptr(), size, K.F_OUT_F32
    if gate:
        o.p1, o.i1, o.flags = z.data_ptr(), groups * size, o.flags | (K.F_GATE_PRE if gate == 1 else K.F_GATE_POST)
    play(o)
    y, s = x.double().view(M, groups, size), torch.nn.functional.silu(z.double()).view(M, groups, size)
    y = y * s if gate == 1 else y
    y = y / torch.sqrt((y * y).mean(-1, keepdim=True) + 1e-5) * w.double()
    y = (y * s if gate == 2 else y).view(M, -1)
    # an exponential and some ten 32-bit operations an entry, a sum of up to 512 squares in 32 chains
    assert ((out.double() - y).abs() <= 40 * 2.0 ** -24 * y.abs().clamp_min(1e-3)).all()


@pytest.mark.parametrize("M", [32, 33, 47, 48, 200])
@pytest.mark.parametrize("H,G,dk,dv", [(2, 1, 128, 128), (3, 3, 64, 40), (2, 2, 256, 24), (20, 4, 128, 64), (12, 12, 160, 136), (1, 1, 20, 5)])
def test_delta_rule_in_blocks_as_token_by_token(M, H, G, dk, dv):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    g = torch.Generator(device="cuda").manual_seed(M + dk)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    nc = 2 * G * dk + H * dv
    rows, raw, alog, dtb, st = rnd(M, nc), rnd(M, 2 * H), rnd(H), rnd(H), rnd(H * dk, dv)
    D = (dk + 31) // 32 * 32
    got = []
    for blocks in (True, False):
        ws = torch.zeros(-(-M // 16) * H * (48 * (D + 4) + D + 640) if blocks else M * (2 * G * dk + G + 2 * H + 4), device="cuda")
        y, s = torch.zeros(M, H * dv, device="cuda"), st.clone()
        o = K.Op()
        o.kind, o.M, o.N, o.taps, o.i0, o.i1, o.i2, o.cin, o.K, o.a_rows, o.A, o.lda = K.K_MSTATE_SCAN, M, H * dv, 0, H, G, dk, dv, G * dk, 2 * G * dk, rows.data_ptr(), nc
        o.res, o.ldr, o.col_mod, o.m_begin, o.scale, o.bias, o.flags = raw.data_ptr(), 2 * H, 0, H, alog.data_ptr(), dtb.data_ptr(), K.F_OUT_F32
        o.p0, o.C2, o.C, o.ldc, o.ws, o.ws_bytes = s.data_ptr(), s.data_ptr(), y.data_ptr(), H * dv, ws.data_ptr(), ws.numel() * 4
        if not blocks:
            assert ws.numel() < -(-M // 16) * H * (48 * (D + 4) + D + 640) or M < 40
            o.ws_bytes = min(o.ws_bytes, 4 * M * ((2 * G * dk + G + 2 * H + 3) // 4 * 4))
        play(o)
        got.append((y, s))
    # 32-bit sums of dk products and up to M steps of a contraction, in another order
    for a, b in zip(*got):
        assert float((a - b).norm()) <= 2e-6 * float(b.norm()) and float((a - b).abs().max()) <= 3e-5 * float(b.abs().max())
