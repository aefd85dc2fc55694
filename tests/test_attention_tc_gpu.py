"""Attention of many queries on tcgen05 (both of its callers) at the edges of its key tiles, query groups, windows, chunks and kept positions, against float64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def launch(op):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    lib = K.load_lib()
    assert lib.fq3c_run((K.Op * 1)(op), 1, torch.cuda.current_stream().cuda_stream) == 0, lib.fq3c_last_error()
    torch.cuda.synchronize()
    assert lib.fq3c_wait_errors() == 0


def exact(q, k, v, first, scale, cap=0.0, window=0, keep=0, chunk=0, sink=None, r12=None, rounded=False):
    M, H, _ = q.shape
    L, G, _ = k.shape
    i, j = torch.arange(first, first + M, device="cuda")[:, None], torch.arange(L, device="cuda")[None]
    seen = j <= i
    if window:
        seen = seen & ((i - j < window) | (j < keep))
    if chunk:
        seen = seen & (j >= i - i % chunk)
    out = torch.empty(M, H, 128, device="cuda", dtype=torch.float64)
    for h in range(H):
        s = q[:, h] @ k[:, h // (H // G)].T
        s = (s.bfloat16().double() * scale).bfloat16().double() if rounded else s * scale
        s = cap * torch.tanh(s / cap) if cap else s
        if r12 is not None:
            s = s - r12[h] * torch.log1p(r12[H + h] * (i - j).clamp(min=0).double())
        s = s.masked_fill(~seen, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(M, 1)], 1)
        out[:, h] = s.softmax(-1)[:, :L] @ v[:, h // (H // G)]
    return out


def rel(got, want):
    return float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("rows, heads, kv, window", [(81, 16, 8, 0), (128, 16, 8, 0), (129, 4, 4, 0), (262, 16, 8, 0), (300, 4, 4, 40), (700, 6, 2, 0), (1300, 16, 16, 0), (1290, 12, 12, 200)])      # (the last two: two row groups a CTA)
def test_prompt_rows(rows, heads, kv, window):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    torch.manual_seed(rows)
    n = (heads + 2 * kv) * 128
    a, out = torch.randn(rows, n, device="cuda").bfloat16(), torch.zeros(rows, heads * 128, device="cuda", dtype=torch.bfloat16)
    o = K.Op()
    o.kind, o.flags, o.M, o.N, o.A, o.lda, o.a_rows = K.K_ATTN, 1, rows, heads * 128, a.data_ptr(), n, rows
    o.C, o.ldc, o.col_mod, o.i0, o.i1, o.i2, o.K = out.data_ptr(), heads * 128, heads * 128, heads, kv, 128, window or 2048
    launch(o)
    d = a.double()
    want = exact(d[:, :heads * 128].view(rows, heads, 128), d[:, heads * 128:(heads + kv) * 128].view(rows, kv, 128), d[:, (heads + kv) * 128:].view(rows, kv, 128), 0,
                 128 ** -0.5, window=window, rounded=True)
    assert rel(out, want.reshape(rows, -1)) < 2.0 ** -9      # one rounding to bf16: 2^-9 at most, about 2^-9.3 on average


def test_prompt_weights_keep_32_bits():
    """Outputs that are small differences of large terms show the weights' own error past the rounding of the output: v = 1 behind one score and -e^(difference),
    as the sum of three bf16 values, behind another."""
    from qwen3_tts_cuda_graphs_b200 import codec as K

    torch.manual_seed(3)
    rows, scale = 384, 128 ** -0.5
    a = torch.zeros(rows, 3 * 128, device="cuda", dtype=torch.bfloat16)
    q, k, v = a[:, :128], a[:, 128:256], a[:, 256:]
    q[:, 0], q[:, 1], q[:, 2] = torch.rand(rows, device="cuda").bfloat16() * 30, torch.rand(rows, device="cuda").bfloat16() * 30, 1.0
    k[0, 0], k[1:4, 1], k[4:, 2] = 1.0, 1.0, -400.0      # the other keys' weights are nothing
    s = lambda x: (x.double() * scale).bfloat16().double()
    s1, s2 = s(q[:, 0]), s(q[:, 1])
    t = torch.arange(256, 384, device="cuda")      # the rows looked at, one column each
    rest = -torch.exp(s1 - s2)[t]
    v[0] = 1.0
    for j in (1, 2, 3):
        v[j, t - 256] = rest.bfloat16()
        rest = rest - v[j, t - 256].double()
    out = torch.zeros(rows, 128, device="cuda", dtype=torch.bfloat16)
    o = K.Op()
    o.kind, o.flags, o.M, o.N, o.A, o.lda, o.a_rows = K.K_ATTN, 1, rows, 128, a.data_ptr(), 384, rows
    o.C, o.ldc, o.col_mod, o.i0, o.i1, o.i2, o.K = out.data_ptr(), 128, 128, 1, 1, 128, 2048
    launch(o)
    w1, w2 = torch.exp(s1)[t], torch.exp(s2)[t]
    vs = v[:4, t - 256].double()
    want = (w1 * vs[0] + w2 * vs[1:].sum(0)) / (w1 + 3 * w2)
    err = (out[t, t - 256].double() - want).abs() / ((w1 + w2 * vs[1:].abs().sum(0)) / (w1 + 3 * w2))
    assert float(err.max()) < 2.0 ** -20      # two weights: an exponential within 2^-22 of an argument within 2^-22 (16 bits would be 2^-17)


# rows, positions in front, heads, key heads, options
CASES = [(9, 0, 4, 2, {}), (100, 0, 4, 1, {}), (300, 77, 6, 2, {}), (128, 128, 16, 4, dict(cap=50.0, sink=True, gate=1)), (513, 300, 16, 4, dict(cap=50.0, sink=True)),
         (200, 300, 8, 2, dict(window=64)), (200, 300, 8, 2, dict(window=64, keep=5, dist=True, cap=50.0)), (128, 128, 3, 1, dict(window=130, keep=200)), (400, 0, 8, 8, dict(window=1)),
         (700, 129, 4, 4, dict(chunk=100, sink=True)), (700, 129, 4, 4, dict(chunk=1000, gate=2)), (260, 260, 12, 4, dict(dist=True, spread=4.0)), (300, 0, 2, 2, dict(spread=8.0)), (40, 700, 2, 1, dict(rising=True)),
         (1300, 100, 16, 16, {}), (1285, 33, 16, 16, dict(window=300, keep=2)), (33, 0, 8, 2, dict(cap=50.0)), (17, 111, 4, 4, {}), (9, 7, 1, 1, {}),
         # with a cap and more row groups than SMs: one a CTA, two because of the positions in front, two from the start (a window; too many), an odd number of them, scores that climb
         (2048, 0, 16, 4, dict(cap=50.0)), (2048, 513, 16, 4, dict(cap=50.0)), (1300, 200, 16, 4, dict(cap=50.0, rising=True)), (1185, 900, 16, 4, dict(cap=50.0, sink=True, gate=2)),
         (1500, 300, 16, 4, dict(cap=50.0, window=700)), (1300, 0, 32, 32, dict(cap=50.0)), (2433, 100, 8, 2, dict(cap=50.0)), (1210, 20, 8, 8, dict(cap=50.0, gate=1)), (600, 151, 32, 8, dict(cap=50.0, rising=True))]


@pytest.mark.parametrize("rows, first, heads, kv, opt", CASES)
def test_cache_rows(rows, first, heads, kv, opt):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    torch.manual_seed(rows + first + heads)
    L = first + rows
    q = torch.randn(rows, heads * 128, device="cuda") * opt.get("spread", 1.0)
    kc = torch.full((L + 300, kv * 128), float("nan"), device="cuda", dtype=torch.bfloat16)      # rows beyond the last position are never used
    vc = kc.clone()
    kc[:L], vc[:L] = torch.randn(L, kv * 128, device="cuda").bfloat16(), torch.randn(L, kv * 128, device="cuda").bfloat16()
    if opt.get("rising"):      # scores climb from tile to tile, so that a row's reference moves
        q, kc[:L] = q.abs(), (kc[:L].float().abs() * torch.linspace(0.1, 3.0, L, device="cuda")[:, None]).bfloat16()
    pos = torch.tensor([first], dtype=torch.int32, device="cuda")
    out = torch.zeros(rows, heads * 128, device="cuda")
    o = K.Op()
    o.kind, o.flags, o.M, o.N, o.i0, o.i1, o.i2, o.cin, o.f0, o.f1 = K.K_CACHE_ATTN, K.F_OUT_F32, rows, heads * 128, heads, kv, 128, 128, 128 ** -0.5, opt.get("cap", 0.0)
    o.K, o.a_rows, o.tap_off[0], o.m_begin = opt.get("window", 0), opt.get("keep", 0), opt.get("chunk", 0), 1
    o.A, o.lda, o.B, o.ldr, o.p1, o.taps, o.p0 = q.data_ptr(), heads * 128, kc.data_ptr(), kv * 128, vc.data_ptr(), kv * 128, pos.data_ptr()
    o.C, o.ldc, o.col_mod = out.data_ptr(), heads * 128, 1
    sink = torch.randn(heads, device="cuda") if opt.get("sink") else None
    r12 = torch.rand(2 * heads, device="cuda") if opt.get("dist") else None
    gate = torch.randn(rows, heads * (128 if opt["gate"] == 2 else 1), device="cuda") if opt.get("gate") else None
    if sink is not None:
        o.scale = sink.data_ptr()
    if r12 is not None:
        o.bias = r12.data_ptr()
    if gate is not None:
        o.res, o.col_mod = gate.data_ptr(), gate.shape[1]
        o.flags |= K.F_GATE_ENTRY if opt["gate"] == 2 else 0
    launch(o)
    want = exact(q.bfloat16().double().view(rows, heads, 128), kc[:L].double().view(L, kv, 128), vc[:L].double().view(L, kv, 128), first, 128 ** -0.5, opt.get("cap", 0.0),
                 opt.get("window", 0), opt.get("keep", 0), opt.get("chunk", 0), None if sink is None else sink.double(), None if r12 is None else r12.double())
    if gate is not None:
        want = want * torch.sigmoid(gate.double()).view(rows, heads, -1)
    # weights of 16 mantissa bits (2^-17 each, falling either way), scores within 2^-22 of their size through the fast cap and exponential
    assert rel(out, want.reshape(rows, -1)) < 1.5e-5


def spoil(v, rows_bad):
    """Infinite and NaN values of the first key head in some rows; where they may show: a position, and the columns."""
    v[rows_bad[0], 3], v[rows_bad[1], 70], v[rows_bad[2], 127] = math.inf, math.nan, -math.inf
    return [(rows_bad[0], 3), (rows_bad[1], 70), (rows_bad[2], 127)]


def check_spoiled(got, clean, heads_of, bad, first, tol):
    """got [M, H, 128] with spoiled values, clean without: what does not see a spoiled row is as without it, what sees it is not finite."""
    M = got.shape[0]
    for row, col in bad:
        sees = torch.arange(first, first + M, device="cuda") >= row
        hit = got[:, :heads_of, col]
        assert not hit[sees].isfinite().any() and hit[~sees].isfinite().all()
        if col != 70:      # an infinite value stays one
            assert hit[sees].isinf().all()
    keep = torch.ones_like(clean, dtype=torch.bool)
    for row, col in bad:
        keep[max(0, row - first):, :heads_of, col] = False
    assert float((got.double() - clean.double())[keep].norm() / clean.double()[keep].norm()) < tol


def test_prompt_values_past_the_causal_edge():
    from qwen3_tts_cuda_graphs_b200 import codec as K

    torch.manual_seed(5)
    rows, heads, kv = 450, 4, 2
    n = (heads + 2 * kv) * 128
    a = torch.randn(rows, n, device="cuda").bfloat16()
    outs = []
    bad = []
    for spoiled in (False, True):
        if spoiled:
            bad = spoil(a[:, (heads + kv) * 128:], (130, 255, 400))
        out = torch.zeros(rows, heads * 128, device="cuda", dtype=torch.bfloat16)
        o = K.Op()
        o.kind, o.flags, o.M, o.N, o.A, o.lda, o.a_rows = K.K_ATTN, 1, rows, heads * 128, a.data_ptr(), n, rows
        o.C, o.ldc, o.col_mod, o.i0, o.i1, o.i2, o.K = out.data_ptr(), heads * 128, heads * 128, heads, kv, 128, 2048
        launch(o)
        outs.append(out.view(rows, heads, 128).float())
    check_spoiled(outs[1], outs[0], heads // kv, bad, 0, 2.0 ** -8)


@pytest.mark.parametrize("f32, splits", [(False, 1), (True, 1), (True, 3)])
@pytest.mark.parametrize("opt", [{}, dict(window=2000, keep=3), dict(cap=20.0), dict(dist=True)])
def test_cache_values_past_the_causal_edge(f32, splits, opt):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    torch.manual_seed(6)
    rows, first, heads, kv = 300, 70, 6, 2
    L = first + rows
    q = torch.randn(rows, heads * 128, device="cuda")
    kc, vc = (torch.randn(L, kv * 128, device="cuda").to(torch.float32 if f32 else torch.bfloat16) for _ in range(2))
    pos, r12 = torch.tensor([first], dtype=torch.int32, device="cuda"), torch.rand(2 * heads, device="cuda")
    ws = torch.zeros(rows * heads * splits * 130, device="cuda")
    outs, bad = [], []
    for spoiled in (False, True):
        if spoiled:
            bad = spoil(vc, (100, 201, 350))
        out = torch.zeros(rows, heads * 128, device="cuda")
        o = K.Op()
        o.kind, o.flags, o.M, o.N, o.i0, o.i1, o.i2, o.cin = K.K_CACHE_ATTN, K.F_OUT_F32 | (K.F_F32 if f32 else 0), rows, heads * 128, heads, kv, 128, 128
        o.f0, o.f1, o.K, o.a_rows, o.m_begin = 128 ** -0.5, opt.get("cap", 0.0), opt.get("window", 0), opt.get("keep", 0), splits
        o.A, o.lda, o.B, o.ldr, o.p1, o.taps, o.p0 = q.data_ptr(), heads * 128, kc.data_ptr(), kv * 128, vc.data_ptr(), kv * 128, pos.data_ptr()
        o.C, o.ldc, o.col_mod, o.ws, o.ws_bytes = out.data_ptr(), heads * 128, 1, ws.data_ptr(), ws.numel() * 4
        if opt.get("dist"):
            o.bias = r12.data_ptr()
        launch(o)
        outs.append(out.view(rows, heads, 128))
    check_spoiled(outs[1], outs[0], heads // kv, bad, first, 1e-5)
