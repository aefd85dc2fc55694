"""Grouped products of routed experts on tcgen05: against float64, at the edges of row tiles, columns, inputs and row lists."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [[200], [20], [9, 0, 0, 8, 1], [128, 0, 128], [1, 127, 129, 0, 2], [0, 0, 300, 0], [64] * 5, [31] * 12, [257, 255]])
@pytest.mark.parametrize("N,Kd", [(128, 64), (130, 72), (96, 128), (1024, 768), (272, 1000), (2, 512)])
@pytest.mark.parametrize("what", ["plain f32", "units", "weighted units", "relu2", "gelu rows"])
def test_against_float64(counts, N, Kd, what):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    lib = K.load_lib()
    E, rows = len(counts), sum(counts)
    g = torch.Generator(device="cuda").manual_seed(rows + N + Kd)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    top, glu = 2, "units" in what
    tokens = -(-rows // top) if what != "plain f32" else rows
    x, w = rnd(tokens, Kd + 8).bfloat16(), (rnd(E, N, Kd) / Kd ** 0.5).bfloat16()
    seg = torch.tensor([0] + torch.tensor(counts).cumsum(0).tolist(), device="cuda", dtype=torch.int32)
    # sorted row r is a choice of token list[r]; pos names a choice's row
    order = torch.randperm(tokens * top, device="cuda", generator=g)[:rows] if what != "plain f32" else torch.arange(rows, device="cuda")
    lst = (order // top if what != "plain f32" else order).to(torch.int32)
    pos = torch.full((tokens, top), -1, device="cuda", dtype=torch.int32)
    if what != "plain f32":
        pos.view(-1)[order] = torch.arange(rows, device="cuda", dtype=torch.int32)
    wt = torch.rand(tokens, top, device="cuda", generator=g) + 0.5
    ldc = (N // 2 if glu else N) + 6
    f32 = what == "plain f32"
    out = torch.full((rows + 1, ldc), 7.0, device="cuda", dtype=torch.float32 if f32 else torch.bfloat16)
    o = K.Op()
    o.kind, o.M, o.N, o.K, o.i0, o.lda, o.ldc = K.K_GGEMM, rows, N, Kd, E, Kd + 8, ldc
    o.A, o.B, o.p0, o.C = x.data_ptr(), w.data_ptr(), seg.data_ptr(), out.data_ptr()
    o.p1 = None if f32 else lst.data_ptr()
    o.flags = K.F_OUT_F32 if f32 else K.F_SWIGLU if glu else K.F_RELU2 if what == "relu2" else K.F_GELU
    if what == "weighted units":
        o.scale, o.ws, o.i1 = wt.data_ptr(), pos.data_ptr(), top
    assert lib.fq3c_run((K.Op * 1)(o), 1, torch.cuda.current_stream().cuda_stream) == 0, lib.fq3c_last_error()
    torch.cuda.synchronize()
    assert lib.fq3c_wait_errors() == 0
    e = torch.repeat_interleave(torch.arange(E, device="cuda"), torch.tensor(counts, device="cuda"))
    a = x[lst.long(), :Kd].double()
    z, size = torch.empty(rows, N, device="cuda", dtype=torch.float64), torch.empty(rows, N, device="cuda", dtype=torch.float64)
    for i in range(E):
        z[e == i], size[e == i] = a[e == i] @ w[i].double().T, a[e == i].abs() @ w[i].double().abs().T
    # 32-bit sums of Kd exact products, dropped below the accumulator's last place; then the result's rounding to bf16 (2^-9), for the units that of the activation's argument too
    err = (Kd / 16 + 4) * 2.0 ** -23 * size
    if glu:
        s = wt.view(-1)[order].double()[:, None] if what == "weighted units" else 1.0
        u, v = z[:, 0::2] * s, z[:, 1::2] * s
        want = torch.nn.functional.silu(u) * v
        err = (err[:, 0::2] * v.abs() * 1.1 + err[:, 1::2] * u.abs()) * (s * s if what == "weighted units" else 1.0) * 1.5
    elif what == "relu2":
        want, err = z.clamp_min(0) ** 2, err * (2 * z.abs() + err)
    elif what == "gelu rows":
        want, err = torch.nn.functional.gelu(z), err * 1.2 + 1e-6
    else:
        want = z
    got = out[:rows, :want.shape[1]].double()
    assert ((got - want).abs() <= err * 1.01 + (0 if f32 else 2.0 ** -8) * want.abs() + 1e-30).all()
    assert (out[rows] == 7.0).all() and (out[:rows, want.shape[1]:] == 7.0).all()
