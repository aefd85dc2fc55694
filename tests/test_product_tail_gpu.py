"""Products of few rows that go on with their entries through the dynamic-tanh norm, the depth mix or xIELU behind them: every buffer as the ops leave it one by one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def run(ops, together):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    lib = K.load_lib()
    before = lib.fq3c_launch_count()
    for part in ([ops] if together else [[o] for o in ops]):
        assert lib.fq3c_run((K.Op * len(part))(*part), len(part), torch.cuda.current_stream().cuda_stream) == 0, lib.fq3c_last_error()
    torch.cuda.synchronize()
    return lib.fq3c_launch_count() - before


def build(M, N, Kd, f32, what, pad):
    """The ops of one sublayer over a fixed set of buffers; what: xielu, dyt, mix, or one of the layouts that have to stay apart."""
    from qwen3_tts_cuda_graphs_b200 import codec as K

    g = torch.Generator(device="cuda").manual_seed(M * 1000 + N)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    dt = torch.float32 if f32 else torch.bfloat16
    b = dict(x=rnd(M, max(Kd, N)).to(dt), w=(rnd(N, Kd) / Kd ** 0.5).to(dt), y=torch.zeros(M, N + pad, device="cuda"), res=rnd(M, N), hist=rnd(4, M, N), mixed=torch.zeros(M, N, device="cuda"),
             out16=torch.zeros(M, N, device="cuda", dtype=torch.bfloat16), nxt=torch.zeros(M, N, device="cuda", dtype=torch.bfloat16), nxt2=torch.zeros(M, N, device="cuda"),
             scale=rnd(N), bias=rnd(N), wb=rnd(2 * N), p=rnd(4))
    o = K.Op()
    o.kind, o.flags, o.M, o.N, o.K, o.taps, o.cin, o.a_rows, o.lda, o.ldc, o.col_mod = K.K_GEMM, K.F_OUT_F32 | K.F_NOROUND | (K.F_F32 if f32 else 0), M, N, Kd, 1, Kd, M, b["x"].shape[1], N + pad, N
    o.A, o.B, o.C = b["x"].data_ptr(), b["w"].data_ptr(), b["y"].data_ptr()
    ops = [o]
    e = K.Op()
    e.M, e.N, e.A, e.lda, e.col_mod, e.ldc = M, N, b["y"].data_ptr(), N + pad, 1, N
    ops.append(e)
    if what == "xielu":
        e.kind, e.p0, e.C = K.K_XIELU, b["p"].data_ptr(), b["out16"].data_ptr()
        return ops, b
    e.kind, e.flags, e.f0, e.scale, e.bias = K.K_DYT, K.F_OUT_F32 | K.F_RESID, 0.7, b["scale"].data_ptr(), b["bias"].data_ptr()
    e.res, e.ldr, e.C, e.C2 = b["res"].data_ptr(), N, b["hist"][2].data_ptr(), b["out16"].data_ptr()
    e.norm_out, e.norm_w, e.norm_ld, e.norm_eps = b["nxt"].data_ptr(), b["wb"].data_ptr(), N, 0.9
    if what == "in place":      # the stream itself
        e.C = e.res
    if what == "over the input":      # the next norm goes where the product reads: a launch of its own
        e.norm_out, e.norm_ld = b["x"].data_ptr(), b["x"].shape[1]
        e.flags |= K.F_F32 if f32 else 0
    if what == "shifted":      # another entry's residual
        e.C = b["res"].data_ptr() + 4
        e.N = N
    if what in ("mix", "mix over its slices"):
        m = K.Op()
        m.kind, m.flags, m.M, m.N, m.i0, m.K, m.A, m.lda, m.p0, m.C, m.ldc, m.col_mod = K.K_DEPTH_MIX, K.F_OUT_F32 | K.F_F32, M, N, 4, M * N, b["hist"].data_ptr(), N, b["p"].data_ptr(), b["mixed"].data_ptr(), N, 1
        m.norm_out, m.norm_w, m.norm_ld, m.norm_eps = b["nxt2"].data_ptr(), b["wb"].data_ptr(), N, 1.1
        if what == "mix over its slices":
            m.C = b["hist"].data_ptr() + 4 * (M * N // 2)
        ops.append(m)
    return ops, b


@pytest.mark.parametrize("M,N,Kd,f32,pad", [(1, 1024, 1024, False, 0), (1, 3072, 1024, False, 0), (1, 1024, 3072, False, 0), (3, 1000, 2080, False, 8), (4, 7, 40, False, 0), (8, 130, 512, True, 4), (1, 96, 100, True, 0)])
@pytest.mark.parametrize("what", ["xielu", "dyt", "mix", "in place", "over the input", "shifted", "mix over its slices"])
def test_same_bits_as_one_by_one(M, N, Kd, f32, pad, what):
    if what == "shifted" and M > 1:
        pytest.skip("rows would overlap each other within one op")
    ops, one = build(M, N, Kd, f32, what, pad)
    keep = {k: t.clone() for k, t in one.items()}
    if what == "shifted":
        pass      # within one op entries of two threads meet too: only that the launches stay apart is looked at
    launches = run(ops, False)
    after = {k: t.clone() for k, t in one.items()}
    for k, t in keep.items():
        one[k].copy_(t)
    fused = run(ops, True)
    apart = what in ("over the input", "shifted")
    assert fused == (launches if apart else 2 if what == "mix over its slices" else 1)
    if what not in ("shifted", "mix over its slices"):
        assert all(torch.equal(after[k].float(), one[k].float()) for k in after)


# overlaps that the ops define one by one: of entry with the same entry (one launch), and of entries with others', where the launches stay apart
OVERLAPS = {"mix in a slice it reads": 1, "next norm over the residual": 1, "mix over the residual, one entry on": 2, "mix over the first norm's weights": 2, "weights in the product's row": 2, "mix weights in the first norm's copy": 2}


@pytest.mark.parametrize("M,N,Kd,f32", [(1, 1024, 1024, False), (3, 1000, 2080, False), (4, 24, 40, False), (8, 130, 512, True), (1, 96, 100, True)])
@pytest.mark.parametrize("what", list(OVERLAPS))
def test_overlapping_buffers_have_the_values_of_one_by_one(M, N, Kd, f32, what):
    ops, b = build(M, N, Kd, f32, "xielu" if what == "weights in the product's row" else "mix", 0)
    _, dyt, mix = ops if len(ops) == 3 else (*ops, None)
    b["res"] = torch.randn(M * N + 8, device="cuda", generator=torch.Generator(device="cuda").manual_seed(N))      # with room behind the rows
    if mix is not None:
        dyt.res = b["res"].data_ptr()
    if what == "mix in a slice it reads":
        mix.C = b["hist"][1].data_ptr()
    if what == "next norm over the residual":
        mix.norm_out = b["res"].data_ptr()
    if what == "mix over the residual, one entry on":
        mix.C = b["res"].data_ptr() + 4
    if what == "mix over the first norm's weights":      # (entries whose norm may still be to come)
        b["big"] = torch.randn(M * N + 2 * N, device="cuda")
        dyt.norm_w, mix.C = b["big"].data_ptr(), b["big"].data_ptr()
    if what == "weights in the product's row":
        dyt.p0 = b["y"].data_ptr() + 4 * (N - 2)
    if what == "mix weights in the first norm's copy":      # two bf16 entries are a weight
        mix.p0 = b["out16"].data_ptr()
    keep = {k: t.clone() for k, t in b.items()}
    apart = run(ops, False)
    after = {k: t.clone() for k, t in b.items()}
    for _ in range(5):
        for k, t in keep.items():
            b[k].copy_(t)
        assert run(ops, True) == OVERLAPS[what] <= apart
        assert all(torch.equal(after[k].nan_to_num(3.0), b[k].nan_to_num(3.0)) for k in after)
