"""Attention over a cache for up to eight rows (a cluster per row and key head): against the mechanism in float64, with the rotation in front in the same launch and by itself."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def reference(rows, kc, vc, pos, H, G, D, o):
    """rows f64 [M, (H + 2 G) D + H (D)]; caches f64 [pos + M, G D], as they were in front; returns outputs, turned queries, new keys and values."""
    M = rows.shape[0]
    p = torch.arange(pos, pos + M, dtype=torch.float64, device="cuda")
    q, k, v = rows[:, :H * D].reshape(M, H, D), rows[:, H * D:(H + G) * D].reshape(M, G, D), rows[:, (H + G) * D:(H + 2 * G) * D].reshape(M, G, D)
    if o.get("norm"):
        unit = lambda z, w: z / torch.sqrt((z * z).mean(-1, keepdim=True) + 1e-6) * w  # noqa: E731
        q, k = unit(q, o["qn"].double()), unit(k, o["kn"].double())
    if o.get("temp"):
        q = q * (0.3 * torch.log(torch.floor((p + 1) / 16) + 1) + 1)[:, None, None]
    n = o["rot"]
    f = o["freq"].double()
    cos, sin = (p[:, None] * f).cos()[:, None], (p[:, None] * f).sin()[:, None]

    def turn(z):
        a, b = (z[..., :n // 2], z[..., n // 2:n]) if o.get("half") else (z[..., 0:n:2], z[..., 1:n:2])
        x, y = a * cos - b * sin, b * cos + a * sin
        return torch.cat([torch.cat([x, y], -1) if o.get("half") else torch.stack([x, y], -1).flatten(-2), z[..., n:]], -1)

    q, k = turn(q), turn(k)
    kc, vc = kc.clone(), vc.clone()
    dt = o["dt"]
    if not o.get("borrowed"):
        kc[pos:], vc[pos:] = k.reshape(M, -1).to(dt).double(), v.reshape(M, -1).to(dt).double()
    out = torch.empty(M, H, D, dtype=torch.float64, device="cuda")
    j = torch.arange(pos + M, device="cuda")
    for m in range(M):
        i = pos + m
        see = j <= i
        if o.get("window"):
            see &= (i - j < o["window"]) | (j < o.get("keep", 0))
        if o.get("chunk"):
            see &= j >= i - i % o["chunk"]
        for h in range(H):
            g = h // (H // G)
            s = kc[:, g * D:(g + 1) * D] @ q[m, h] * D ** -0.5
            s = o["cap"] * torch.tanh(s / o["cap"]) if o.get("cap") else s
            if o.get("far"):
                s = s - o["r12"][h].double() * torch.log1p(o["r12"][H + h].double() * (i - j))
            s = s[see]
            w = torch.softmax(torch.cat([s, o["sink"][h].double()[None]]) if o.get("sink") is not None else s, 0)[:len(s)]
            out[m, h] = w @ vc[see, g * D:(g + 1) * D]
    g = rows[:, (H + 2 * G) * D:]
    if o.get("gate"):
        out = out * (torch.sigmoid(g[:, :H * D]).reshape(M, H, D) if o["gate"] == "entry" else torch.sigmoid(g[:, :H])[..., None])
    return out.reshape(M, -1) * o.get("mult", 1.0), q.reshape(M, -1), kc, vc


OPTIONS = [dict(), dict(cap=30.0, sink=True, gate="head"), dict(window=40, half=True, norm=True), dict(window=24, keep=9, far=True, mult=0.5), dict(chunk=64, gate="entry", temp=True),
           dict(borrowed=True, sink=True), dict(window=1)]


@pytest.mark.parametrize("D,f32", [(128, False), (64, False), (128, True), (64, True)])
@pytest.mark.parametrize("H,G", [(4, 4), (4, 2), (3, 1), (8, 2), (8, 1), (5, 1)])      # (five heads a key head: the other kernel)
@pytest.mark.parametrize("option", range(len(OPTIONS)))
def test_against_float64(D, f32, H, G, option):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    lib = K.load_lib()
    dt = torch.float32 if f32 else torch.bfloat16
    for M, pos in [(1, 0), (1, 7), (1, 8), (1, 63), (1, 64), (1, 511), (1, 700), (2, 6), (5, 62), (8, 0), (8, 509)]:
        g = torch.Generator(device="cuda").manual_seed(M * 1000 + pos + H)
        rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
        o = dict(OPTIONS[option], rot=32, dt=dt, freq=10000.0 ** (-torch.arange(16, device="cuda", dtype=torch.float32) / 16), qn=rnd(D), kn=rnd(D), r12=rnd(2 * H).abs() * 0.3)
        o["sink"] = rnd(H) if o.get("sink") else None
        cols = (H + 2 * G) * D + H * D
        rows, kc, vc = rnd(M, cols), rnd(pos + M + 3, G * D).to(dt), rnd(pos + M + 3, G * D).to(dt)
        if o.get("window") and H // G != 5:      # what no row sees stays out of the sums
            lo = max(0, pos - o["window"] + 1)
            kc[o.get("keep", 0):lo], vc[o.get("keep", 0):lo] = float("nan"), float("inf")
        want = reference(rows.double(), torch.nan_to_num(kc[:pos + M].double(), 0, 0, 0), torch.nan_to_num(vc[:pos + M].double(), 0, 0, 0), pos, H, G, D, o)
        if not o.get("borrowed"):
            kc[pos:], vc[pos:] = float("nan"), float("nan")
        where = torch.tensor([pos], device="cuda", dtype=torch.int32)
        results = []
        for together in (True, False):
            x, k2, v2, out = rows.clone(), kc.clone(), vc.clone(), torch.zeros(M, H * D, device="cuda")
            ws = torch.zeros(M * H * 4 * (D + 2), device="cuda")
            r = K.Op()
            r.kind, r.M, r.i0, r.i1, r.i2, r.cin, r.taps, r.K, r.a_rows, r.lda, r.flags = K.K_ROT_APPEND, M, H, 0 if o.get("borrowed") else G, D, D, 32, H * D, (H + G) * D, cols, K.F_F32 if f32 else 0
            r.A, r.B, r.p0 = x.data_ptr(), o["freq"].data_ptr(), where.data_ptr()
            if r.i1:
                r.C, r.ldc, r.C2, r.ldr = k2.data_ptr(), G * D, v2.data_ptr(), G * D
            r.flags |= K.F_ROT_HALF if o.get("half") else 0
            if o.get("norm"):
                r.scale, r.bias, r.f0 = o["qn"].data_ptr(), o["kn"].data_ptr(), 1e-6
            if o.get("temp"):
                r.f2, r.f3 = 0.3, 16.0
            a = K.Op()
            a.kind, a.M, a.N, a.i0, a.i1, a.i2, a.cin, a.f0, a.f1, a.f2 = K.K_CACHE_ATTN, M, H * D, H, G, D, D, D ** -0.5, o.get("cap", 0.0), o.get("mult", 1.0)
            a.K, a.a_rows, a.lda, a.ldr, a.taps, a.m_begin, a.ldc, a.flags = o.get("window", 0), o.get("keep", 0), cols, G * D, G * D, 4, H * D, (K.F_F32 if f32 else 0) | K.F_OUT_F32
            a.A, a.B, a.p1, a.p0, a.C, a.ws, a.ws_bytes = x.data_ptr(), k2.data_ptr(), v2.data_ptr(), where.data_ptr(), out.data_ptr(), ws.data_ptr(), ws.numel() * 4
            a.tap_off[0] = o.get("chunk", 0)
            if o["sink"] is not None:
                a.scale = o["sink"].data_ptr()
            if o.get("far"):
                a.bias = o["r12"].data_ptr()
            if o.get("gate"):
                a.res, a.col_mod = x.data_ptr() + 4 * (H + 2 * G) * D, cols
                a.flags |= K.F_GATE_ENTRY if o["gate"] == "entry" else 0
            before, stream = lib.fq3c_launch_count(), torch.cuda.current_stream().cuda_stream
            for part in ([[r, a]] if together else [[r], [a]]):
                assert lib.fq3c_run((K.Op * len(part))(*part), len(part), stream) == 0, lib.fq3c_last_error()
            torch.cuda.synchronize()
            results.append((out, x, k2, v2, lib.fq3c_launch_count() - before))
        assert [t[4] for t in results] == ([3, 3] if H // G == 5 else [1 if M == 1 else 2, 2])
        for out, x, k2, v2, _ in results:
            assert torch.equal(x[:, H * D:], rows[:, H * D:])
            # 32-bit sums of D products of unit size, the rotation's and the exponential's few units: the scores are off by some 1e-6 of their size (up to 20 with a norm's weights)
            assert (x[:, :H * D].double() - want[1]).abs().max() <= 2e-5 * want[1].abs().max()
            if r.i1:
                # a cache entry may round the other way: one unit of its type
                for got, ref in ((k2, want[2]), (v2, want[3])):
                    assert (got[pos:pos + M].double() - ref[pos:]).abs().max() <= (2e-5 if f32 else 2 ** -8) * max(1.0, float(ref[pos:].abs().max()))
                assert torch.isnan(k2[pos + M:].float()).all()
            # outputs are weighted means of values of size one; a new key that rounds the other way moves its score by 2^-8 of a term
            assert (out.double() - want[0]).abs().max() <= (5e-5 if f32 else 2e-2) * max(1.0, float(want[0].abs().max()))
            assert (out.double() - want[0]).norm() <= (1e-5 if f32 else 4e-3) * want[0].norm()
        assert all(torch.allclose(a, b, rtol=1e-4, atol=1e-5, equal_nan=True) for a, b in zip(results[0][:2], results[1][:2])) and torch.equal(results[0][2].float().nan_to_num(7.0), results[1][2].float().nan_to_num(7.0))


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("H,G", [(2, 2), (4, 2), (6, 2), (8, 2), (8, 1)])
@pytest.mark.parametrize("pos,low", [(64, [64]), (8, [8]), (200, list(range(96, 104))), (70, list(range(64, 71))), (15, list(range(8, 15))), (9, list(range(9)))])
@pytest.mark.parametrize("turned", [True, False])      # with the rotation in front in the same launch, and the attention by itself
def test_visible_keys_that_score_minus_infinity(f32, H, G, pos, low, turned):
    """Keys of weight zero: alone among the eight of their warp (the newest one too), all of the eight, all but the newest key."""
    from qwen3_tts_cuda_graphs_b200 import codec as K

    lib, D, dt = K.load_lib(), 128, torch.float32 if f32 else torch.bfloat16
    g = torch.Generator(device="cuda").manual_seed(pos + H)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    o = dict(rot=32, dt=dt, freq=10000.0 ** (-torch.arange(16, device="cuda", dtype=torch.float32) / 16), borrowed=not turned)
    cols = (H + 2 * G) * D
    rows, kc, vc = rnd(1, cols), rnd(pos + 1, G * D).to(dt), rnd(pos + 1, G * D).to(dt)
    rows[0, D - 1:H * D:D] = 0.5      # (an entry behind those that turn)
    kc[low, D - 1::D] = -torch.inf
    if pos in low:
        rows[0, (H + 1) * D - 1:(H + G) * D:D] = -torch.inf
    want = reference(rows.double(), kc.double(), vc.double(), pos, H, G, D, o)[0]
    out, where = torch.zeros(1, H * D, device="cuda"), torch.tensor([pos], device="cuda", dtype=torch.int32)
    r, a = K.Op(), K.Op()
    r.kind, r.M, r.i0, r.i1, r.i2, r.cin, r.taps, r.K, r.a_rows, r.lda, r.flags = K.K_ROT_APPEND, 1, H, G if turned else 0, D, D, 32, H * D, (H + G) * D, cols, K.F_F32 if f32 else 0
    r.A, r.B, r.p0 = rows.data_ptr(), o["freq"].data_ptr(), where.data_ptr()
    if turned:
        r.C, r.ldc, r.C2, r.ldr = kc.data_ptr(), G * D, vc.data_ptr(), G * D
    a.kind, a.M, a.N, a.i0, a.i1, a.i2, a.cin, a.f0, a.lda, a.ldr, a.taps, a.ldc, a.flags = K.K_CACHE_ATTN, 1, H * D, H, G, D, D, D ** -0.5, cols, G * D, G * D, H * D, (K.F_F32 if f32 else 0) | K.F_OUT_F32
    a.A, a.B, a.p1, a.p0, a.C = rows.data_ptr(), kc.data_ptr(), vc.data_ptr(), where.data_ptr(), out.data_ptr()
    for part in ([[r, a]] if turned else [[r], [a]]):
        assert lib.fq3c_run((K.Op * len(part))(*part), len(part), torch.cuda.current_stream().cuda_stream) == 0, lib.fq3c_last_error()
    # as in the test above; a new key that rounds the other way moves its score by 2^-8 of a term
    assert want.isfinite().all() and (out.double() - want).norm() <= (1e-5 if f32 else 4e-3) * want.norm()


@pytest.mark.parametrize("M,pos,H,G,D,f32,splits,launches", [
    (1, 5000, 4, 4, 128, False, 64, 1), (2, 2047, 2, 2, 64, True, 64, 1), (1, 9000, 1, 1, 128, True, 64, 1),      # one head a key head: any number of keys
    (1, 2015, 8, 2, 128, False, 63, 1), (1, 2016, 8, 2, 128, False, 64, 2),      # 63 splits say that there are at most 2016 keys, 64 say nothing
    (8, 100, 16, 8, 128, False, 4, 1), (8, 100, 9, 9, 128, False, 4, 2), (4, 70, 8, 8, 64, False, 3, 1), (3, 70, 11, 11, 64, False, 3, 2),      # clusters of the variants with two CTAs an SM
    (3, 33, 10, 5, 128, True, 1, 1), (4, 28, 8, 4, 128, True, 1, 1), (8, 500, 16, 4, 128, True, 63, 1), (4, 500, 8, 8, 128, True, 16, 1), (4, 530, 8, 8, 128, True, 17, 2), (3, 60, 11, 11, 128, True, 2, 2)])      # and of the others
def test_which_calls_take_a_cluster(M, pos, H, G, D, f32, splits, launches):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    lib, dt = K.load_lib(), torch.float32 if f32 else torch.bfloat16
    g = torch.Generator(device="cuda").manual_seed(pos + H)
    rows, kc, vc = torch.randn(M, H * D, device="cuda", generator=g), *(torch.randn(pos + M, G * D, device="cuda", generator=g).to(dt) for _ in range(2))
    out, ws, where = torch.zeros(M, H * D, device="cuda"), torch.zeros(M * H * splits * (D + 2), device="cuda"), torch.tensor([pos], device="cuda", dtype=torch.int32)
    a = K.Op()
    a.kind, a.M, a.N, a.i0, a.i1, a.i2, a.cin, a.f0, a.lda, a.ldr, a.taps, a.ldc, a.flags = K.K_CACHE_ATTN, M, H * D, H, G, D, D, D ** -0.5, H * D, G * D, G * D, H * D, (K.F_F32 if f32 else 0) | K.F_OUT_F32
    a.A, a.B, a.p1, a.p0, a.C, a.ws, a.ws_bytes, a.m_begin = rows.data_ptr(), kc.data_ptr(), vc.data_ptr(), where.data_ptr(), out.data_ptr(), ws.data_ptr(), ws.numel() * 4, splits
    before = lib.fq3c_launch_count()
    assert lib.fq3c_run((K.Op * 1)(a), 1, torch.cuda.current_stream().cuda_stream) == 0, lib.fq3c_last_error()
    assert lib.fq3c_launch_count() - before == launches
    see = torch.arange(pos + M, device="cuda")[None] <= torch.arange(pos, pos + M, device="cuda")[:, None]
    for h in range(H):
        n = h // (H // G)
        s = (rows[:, h * D:(h + 1) * D].double() @ kc[:, n * D:(n + 1) * D].double().T * D ** -0.5).masked_fill(~see, -torch.inf)
        p, v = s.softmax(-1), vc[:, n * D:(n + 1) * D].double()
        # every entry: scores of about 1 from D products in 32 bits (some 1e-6 of them), so each weight is off by that, an exponential and a rounding or two, and their sum as well
        assert ((out[:, h * D:(h + 1) * D].double() - p @ v).abs() <= 1e-5 * (p @ v.abs())).all()
        assert (out[:, h * D:(h + 1) * D].double() - p @ v).norm() <= 2e-6 * (p @ v).norm()
