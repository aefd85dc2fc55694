"""A kernel whose bounded wait runs out: the launch ends, all of its outputs are NaN and the host is told.  (In a process of its own: the error stays set.)"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import sys, torch
sys.path.insert(0, sys.argv[2])
from test_gemm_gpu import make_op
from qwen3_tts_cuda_graphs_b200 import codec as K
what, lib, dev = sys.argv[1], K.load_lib(), "cuda"
outs = []
if what.startswith("gemm"):
    M, N, kk = {"gemm": (700, 1000, 512), "gemm split": (39, 1024, 2048), "gemm gated": (39, 1024, 512), "gemm snake": (3000, 192, 192)}[what]
    A, B = torch.randn(M, kk, device=dev).bfloat16(), torch.randn(N, kk, device=dev).bfloat16()
    out = torch.zeros(M, N // 2 if what == "gemm gated" else N, device=dev, dtype=torch.bfloat16)
    o = make_op(A, B, out, M, N, kk, flags=K.F_SWIGLU if what == "gemm gated" else 0, ws=torch.zeros(8 * M * N, device=dev) if what == "gemm split" else None)
    outs = [out]
    if what == "gemm snake":
        out2, par = torch.zeros_like(out), torch.ones(N, device=dev)
        o.flags |= K.F_SNAKE2
        o.C2, o.p0, o.p1 = out2.data_ptr(), par.data_ptr(), par.data_ptr()
        outs.append(out2)
    o.reserved = 3
elif what == "prompt attention":
    M, H, G = 300, 4, 2
    a, out = torch.randn(M, (H + 2 * G) * 128, device=dev).bfloat16(), torch.zeros(M, H * 128, device=dev, dtype=torch.bfloat16)
    o = K.Op()
    o.kind, o.flags, o.M, o.N, o.A, o.lda, o.a_rows = K.K_ATTN, 1, M, H * 128, a.data_ptr(), a.shape[1], M
    o.C, o.ldc, o.col_mod, o.i0, o.i1, o.i2, o.K, o.reserved = out.data_ptr(), H * 128, H * 128, H, G, 128, 2048, 2
    outs = [out]
elif what.startswith("delta rule"):
    M, H, G, dk, dv = {"delta rule, two blocks": (32, 2, 1, 64, 40), "delta rule": (333, 8, 4, 128, 128)}[what]
    nc = 2 * G * dk + H * dv
    rows, raw, one, st = torch.randn(M, nc, device=dev), torch.randn(M, 2 * H, device=dev), torch.zeros(H, device=dev), torch.randn(H * dk, dv, device=dev)
    out, ws = torch.zeros(M, H * dv, device=dev), torch.zeros(-(-M // 16) * H * (48 * (dk + 4) + dk + 640), device=dev)
    o = K.Op()
    o.kind, o.M, o.N, o.i0, o.i1, o.i2, o.cin, o.K, o.a_rows, o.A, o.lda = K.K_MSTATE_SCAN, M, H * dv, H, G, dk, dv, G * dk, 2 * G * dk, rows.data_ptr(), nc
    o.res, o.ldr, o.col_mod, o.m_begin, o.scale, o.flags, o.reserved = raw.data_ptr(), 2 * H, 0, H, one.data_ptr(), K.F_OUT_F32, 2
    o.p0, o.C2, o.C, o.ldc, o.ws, o.ws_bytes = st.data_ptr(), st.data_ptr(), out.data_ptr(), H * dv, ws.data_ptr(), ws.numel() * 4
    outs = [out]
elif what.startswith("experts"):
    E, rows, N, kk = 3, 300, 272, {"experts": 512, "experts, one k-block": 64, "experts, units": 512}[what]
    glu = what == "experts, units"
    a, w, seg = torch.randn(rows, kk, device=dev).bfloat16(), torch.randn(E, N, kk, device=dev).bfloat16(), torch.tensor([0, 130, 130, rows], device=dev, dtype=torch.int32)
    out = torch.zeros(rows, N // 2 if glu else N, device=dev, dtype=torch.bfloat16 if glu else torch.float32)
    o = K.Op()
    o.kind, o.M, o.N, o.K, o.i0, o.lda, o.ldc, o.flags, o.reserved = K.K_GGEMM, rows, N, kk, E, kk, out.shape[1], K.F_SWIGLU if glu else K.F_OUT_F32, 2
    o.A, o.B, o.p0, o.C = a.data_ptr(), w.data_ptr(), seg.data_ptr(), out.data_ptr()
    outs = [out]
else:
    M, H, G = 200, 6, 2
    q, kv, pos = torch.randn(M, H * 128, device=dev), torch.randn(M, G * 128, device=dev).bfloat16(), torch.zeros(1, dtype=torch.int32, device=dev)
    out = torch.zeros(M, H * 128, device=dev)
    o = K.Op()
    o.kind, o.flags, o.M, o.N, o.i0, o.i1, o.i2, o.cin, o.f0, o.m_begin = K.K_CACHE_ATTN, K.F_OUT_F32, M, H * 128, H, G, 128, 128, 128 ** -0.5, 1
    o.A, o.lda, o.B, o.ldr, o.p1, o.taps, o.p0 = q.data_ptr(), H * 128, kv.data_ptr(), G * 128, kv.data_ptr(), G * 128, pos.data_ptr()
    o.C, o.ldc, o.col_mod, o.reserved = out.data_ptr(), H * 128, 1, 2
    outs = [out]
assert lib.fq3c_run((K.Op * 1)(o), 1, torch.cuda.current_stream().cuda_stream) == 0, lib.fq3c_last_error()
torch.cuda.synchronize()
assert all(bool(t.isnan().all()) for t in outs)
assert lib.fq3c_wait_failed() != 0 and lib.fq3c_wait_errors() != 0
try:
    K.check_waits()
except K.CodecError:
    print("raised")
x = torch.randn(300, 300, device=dev)      # the context stays usable
assert torch.allclose((x @ x).double(), x.double() @ x.double(), atol=1e-1)
"""


@pytest.mark.parametrize("what", ["gemm", "gemm split", "gemm gated", "gemm snake", "prompt attention", "cache attention", "experts", "experts, one k-block", "experts, units", "delta rule", "delta rule, two blocks"])
def test_a_wait_that_runs_out(what):
    here = os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, "-c", PROGRAM, what, here], cwd=os.path.dirname(here), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "raised" in r.stdout, r.stdout + r.stderr
