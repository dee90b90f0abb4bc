"""The SwiGLU adjoint epilogue on CTA pairs against the one-CTA kernel, and grouped GEMMs with long contractions (on pairs)
against an fp32 reference."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# ragged rows (the second CTA of the last pair partly or wholly outside), columns that end inside either epilogue group's halves
@pytest.mark.parametrize("T,Fs", [(256, 256), (300, 288), (385, 416), (1000, 480), (2048, 1024)])
def test_shared_adjoint_on_pairs(T, Fs):
    from swamla_b200 import _cabi
    lib = _cabi.load()
    D, E, dev = 320, 8, "cuda:0"
    g = torch.Generator(dev).manual_seed(T)
    rand = lambda *s: torch.randn(*s, device=dev, generator=g).to(torch.bfloat16)
    dy, wd, h1, hid = rand(T, D), rand(D, Fs), rand(T, 2 * Fs), rand(T, Fs)
    shape = _cabi.Shape(T=T, D=D, L=D, E=E, K=2, F=64, Fs=Fs, n_shared=1)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    out = []
    for on in (0, 1):
        before = lib.lmoe_pair_gemm_enable(on)
        try:
            ws = torch.empty(lib.lmoe_moe_wgrad_workspace_bytes(shape), dtype=torch.uint8, device=dev)
            cat = torch.full((T, 2 * Fs + E), 3.0, dtype=torch.bfloat16, device=dev)
            dw = torch.empty(D, Fs, device=dev)
            _cabi.call("lmoe_moe_shared_bwd", shape, dy.data_ptr(), wd.data_ptr(), h1.data_ptr(), hid.data_ptr(), cat.data_ptr(),
                       dw.data_ptr(), _cabi.F32, ws.data_ptr(), ws.numel(), status.data_ptr(), torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
        finally:
            lib.lmoe_pair_gemm_enable(before)
        out.append((cat, dw))
    assert status.item() == 0
    (a, dwa), (b, dwb) = out
    assert (b[:, 2 * Fs:] == 3.0).all()                              # nothing beyond the two halves
    # d_hidden before its bf16 rounding differs by fp32 summation order only: a flipped rounding is one bf16 ulp (2^-7), which
    # the adjoint passes on linearly
    a, b = a[:, :2 * Fs].float(), b[:, :2 * Fs].float()
    scale = torch.maximum(a.abs(), torch.tensor(1e-3, device=dev) * a.abs().max())
    assert ((a - b).abs() <= 2.0 ** -6 * scale).all()
    assert (dwa - dwb).norm() <= 1e-5 * dwa.norm()


@pytest.mark.parametrize("rows", [[0, 128, 200, 1], [700, 0, 130, 385]])   # odd and even tile counts, empty experts
@pytest.mark.parametrize("b_mn", [0, 1])
def test_grouped_long_contraction(rows, b_mn):
    """K = 768 through lmoe_grouped_fwd's down GEMM (b_mn = 1) and lmoe_grouped_bwd_dgrad's d_x GEMM (b_mn = 0)."""
    from swamla_b200 import _cabi
    dev, E, L, F = "cuda:0", 4, 128, 768
    pads = [(r + 127) // 128 * 128 for r in rows]
    off = torch.tensor([sum(pads[:i]) for i in range(E + 1)], dtype=torch.int32)
    P = int(off[-1]) + 128                                           # one unused tile of capacity
    te = torch.tensor([e for e in range(E) for _ in range(pads[e] // 128)] + [0], dtype=torch.int32, device=dev)
    nt = torch.tensor([int(off[-1]) // 128], dtype=torch.int32, device=dev)
    offd = off.to(dev)
    g = torch.Generator(dev).manual_seed(5)
    rand = lambda *s: torch.randn(*s, device=dev, generator=g).to(torch.bfloat16)
    x, wgu, wd = rand(P, L), 0.1 * rand(E, L, 2 * F), 0.05 * rand(E, F, L)
    h1, hid, y = torch.zeros(P, 2 * F, dtype=torch.bfloat16, device=dev), torch.zeros(P, F, dtype=torch.bfloat16, device=dev), torch.zeros(P, L, dtype=torch.bfloat16, device=dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    st = torch.cuda.current_stream().cuda_stream
    _cabi.call("lmoe_grouped_fwd", P, E, L, F, x.data_ptr(), wgu.data_ptr(), wd.data_ptr(), te.data_ptr(), nt.data_ptr(),
               offd.data_ptr(), h1.data_ptr(), hid.data_ptr(), y.data_ptr(), status.data_ptr(), st)
    if b_mn:
        got, a, w = y, hid, wd
    else:
        dh1, dx = torch.zeros_like(h1), torch.zeros_like(x)
        _cabi.call("lmoe_grouped_bwd_dgrad", P, E, L, F, x.data_ptr(), h1.data_ptr(), wgu.data_ptr(), wd.data_ptr(), te.data_ptr(),
                   nt.data_ptr(), offd.data_ptr(), None, dh1.data_ptr(), dx.data_ptr(), status.data_ptr(), st)
        got, a, w = dx, dh1, wgu.transpose(1, 2)
    torch.cuda.synchronize()
    assert status.item() == 0
    for e in range(E):
        lo, hi = int(off[e]), int(off[e + 1])
        if hi > lo:
            ref = a[lo:hi].float() @ w[e].float()
            err = (got[lo:hi].float() - ref).abs()
            assert (err <= 2.0 ** -8 * ref.abs() + 2.0 ** -16 * ref.abs().max()).all()   # bf16 output rounding, fp32 sums
    assert (got[int(off[-1]):] == 0).all()                           # nothing beyond the tiles in use


# whole tiles, several tiles, ragged edges (the second CTA's rows partly outside), an extent that stays with one CTA per tile
@pytest.mark.parametrize("M,N", [(256, 256), (1024, 264), (504, 520), (256, 1536), (384, 256)])
@pytest.mark.parametrize("rows", [[128, 0, 640, 64], [0, 0, 0, 129], [1, 256, 2000, 0]])   # empty experts, one k-block pair, long
def test_grouped_weight_gradient(M, N, rows):
    from swamla_b200 import _cabi
    dev, E = "cuda:0", 4
    pads = [(r + 127) // 128 * 128 for r in rows]
    off = [sum(pads[:i]) for i in range(E + 1)]
    P = off[-1] + 128                                                # one unused tile of capacity, never read
    g = torch.Generator(dev).manual_seed(M + N)
    a, b = (torch.randn(P, n, device=dev, generator=g).to(torch.bfloat16) for n in (M, N))
    a[off[-1]:] = float("nan")
    out = torch.full((E + 1, M, N), 3.0, dtype=torch.bfloat16, device=dev)
    offd = torch.tensor(off, dtype=torch.int32, device=dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    _cabi.call("lmoe_grouped_wgrad_bf16", P, E, M, N, a.data_ptr(), b.data_ptr(), offd.data_ptr(), out.data_ptr(), status.data_ptr(),
               torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert status.item() == 0
    for e in range(E):
        ref = a[off[e]:off[e + 1]].double().t() @ b[off[e]:off[e + 1]].double()
        err = (out[e].double() - ref).abs()
        assert (err <= 2.0 ** -8 * ref.abs() + 2.0 ** -16 * max(1.0, ref.abs().max().item())).all()   # bf16 rounding, fp32 sums
    assert (out[E] == 3.0).all()                                     # nothing behind the last expert's plane
