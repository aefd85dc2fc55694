"""One decoded row of a delta-rule layer, convolution, recurrence and gated norm in one launch: every buffer as the ops leave it one by one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def build(H, G, dk, dv, taps, gate, bias, in_place, f32_out, seed):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    nc = 2 * G * dk + H * dv
    b = dict(raw=rnd(1, nc + H * dv + 2 * H), hist=rnd(taps - 1, nc), next=torch.zeros(taps - 1, nc, device="cuda"), w=rnd(nc, taps), cb=rnd(nc), cv=torch.zeros(1, nc, device="cuda"), s=rnd(H * dk, dv),
             s2=torch.zeros(H * dk, dv, device="cuda"), alog=rnd(H), dtb=rnd(H), y=torch.zeros(1, H * dv, device="cuda"), nw=rnd(dv),
             yn=torch.zeros(1, H * dv, device="cuda", dtype=torch.float32 if f32_out else torch.bfloat16))
    ws = torch.zeros(2 * G * dk + G + 2 * H + 8, device="cuda")
    c, o, n = K.Op(), K.Op(), K.Op()
    c.kind, c.M, c.N, c.taps, c.A, c.lda, c.B, c.C, c.ldc, c.flags, c.p0, c.p1 = K.K_TCONV, 1, nc, taps, b["raw"].data_ptr(), b["raw"].shape[1], b["w"].data_ptr(), b["cv"].data_ptr(), nc, K.F_OUT_F32 | K.F_SILU, b["hist"].data_ptr(), b["next"].data_ptr()
    if bias:
        c.bias, c.i0, c.flags = b["cb"].data_ptr(), G * dk, c.flags | K.F_BIAS | K.F_RESID      # the queries without silu
    o.kind, o.M, o.N, o.taps, o.i0, o.i1, o.i2, o.cin, o.K, o.a_rows, o.A, o.lda = K.K_MSTATE_SCAN, 1, H * dv, 0, H, G, dk, dv, G * dk, 2 * G * dk, b["cv"].data_ptr(), nc
    o.res, o.ldr, o.col_mod, o.m_begin, o.scale, o.flags = b["raw"].data_ptr(), b["raw"].shape[1], nc + H * dv, nc + H * dv + H, b["alog"].data_ptr(), K.F_OUT_F32
    o.bias = b["dtb"].data_ptr() if bias else None
    o.p0, o.C2, o.C, o.ldc, o.ws, o.ws_bytes = b["s"].data_ptr(), b["s" if in_place else "s2"].data_ptr(), b["y"].data_ptr(), H * dv, ws.data_ptr(), ws.numel() * 4
    n.kind, n.M, n.N, n.i0, n.f0, n.A, n.lda, n.C, n.ldc, n.i2, n.scale, n.flags = K.K_GNORM, 1, H * dv, H, 1e-5, b["y"].data_ptr(), H * dv, b["yn"].data_ptr(), H * dv, dv, b["nw"].data_ptr(), K.F_OUT_F32 if f32_out else 0
    if gate:
        n.p1, n.i1, n.flags = b["raw"].data_ptr() + 4 * nc, b["raw"].shape[1], n.flags | K.F_GATE_POST | (K.F_SIGMOID if gate == 2 else 0)
    return [c, o, n], b, ws


def run(ops, together):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    lib = K.load_lib()
    before = lib.fq3c_launch_count()
    for part in ([ops] if together else [[o] for o in ops]):
        assert lib.fq3c_run((K.Op * len(part))(*part), len(part), torch.cuda.current_stream().cuda_stream) == 0, lib.fq3c_last_error()
    torch.cuda.synchronize()
    return lib.fq3c_launch_count() - before


@pytest.mark.parametrize("H,G,dk,dv", [(8, 4, 128, 128), (2, 2, 128, 64), (3, 1, 64, 8), (4, 4, 64, 72), (6, 2, 256, 128), (1, 1, 128, 120)])
@pytest.mark.parametrize("taps,gate,bias,in_place,f32_out", [(4, 1, False, True, False), (2, 0, True, False, True), (4, 2, True, True, False)])
def test_same_bits_as_one_by_one(H, G, dk, dv, taps, gate, bias, in_place, f32_out):
    ops, b, _ = build(H, G, dk, dv, taps, gate, bias, in_place, f32_out, H + dk + dv)
    start = {k: t.clone() for k, t in b.items()}
    assert run(ops, False) == 4
    after = {k: t.clone() for k, t in b.items()}
    for _ in range(3):
        for k, t in start.items():
            b[k].copy_(t)
        assert run(ops, True) == 1
        assert all(torch.equal(after[k], b[k]) for k in after)


APART = ["history in place", "queries over the gate", "norm over the input", "another head width", "no history"]


@pytest.mark.parametrize("what", APART)
def test_other_layouts_stay_apart(what):
    ops, b, ws = build(4, 2, 96 if what == "another head width" else 64, 64, 1 if what == "no history" else 3, 1, False, True, True, 5)
    c, o, n = ops
    if what == "history in place":
        c.p1 = c.p0
    if what == "queries over the gate":      # the norm's gate is what the convolution writes
        n.p1 = b["cv"].data_ptr()
    if what == "norm over the input":
        n.C = b["raw"].data_ptr()
    start = {k: t.clone() for k, t in b.items()}
    launches = run(ops, False)
    after = {k: t.clone() for k, t in b.items()}
    for k, t in start.items():
        b[k].copy_(t)
    assert run(ops, True) == launches == 4
    if what != "history in place":      # (its rows move over one another within the op)
        assert all(torch.equal(after[k], b[k]) for k in after)
