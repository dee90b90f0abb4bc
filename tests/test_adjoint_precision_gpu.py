"""SwiGLU adjoints in GEMM epilogues that give the bits of the separate kernels (GEMM to a bf16 d_hidden, then
lmoe_swiglu_bwd): the non-latent layer's shared and routed experts, the e4m3 routed experts.  The gates spread over
[-12, 12]: an approximation with a bounded absolute error of the sigmoid is off by percents at the negative ones."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _rand(g, *shape, scale=1.0):
    return (scale * torch.randn(*shape, device=DEV, generator=g)).to(torch.bfloat16)


def _gates(g, rows, H):
    """h1[rows, 2H] = (gate | up)"""
    h1 = _rand(g, rows, 2 * H)
    h1[:, :H] = (24.0 * torch.rand(rows, H, device=DEV, generator=g) - 12.0).to(torch.bfloat16)
    return h1


# ragged rows and columns, the one-CTA kernel and the CTA-pair kernel
@pytest.mark.parametrize("T,Fs", [(1, 32), (300, 288), (1000, 480)])
@pytest.mark.parametrize("pairs", [0, 1])
def test_non_latent_shared_adjoint(T, Fs, pairs):
    from swamla_b200 import _cabi
    lib = _cabi.load()
    D, E = 320, 8
    g = torch.Generator(DEV).manual_seed(T)
    dy, wd, h1, hid = _rand(g, T, D), _rand(g, D, Fs, scale=0.1), _gates(g, T, Fs), _rand(g, T, Fs)
    shape = _cabi.Shape(T=T, D=D, L=D, E=E, K=2, F=64, Fs=Fs, n_shared=1)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    ws = torch.empty(lib.lmoe_moe_wgrad_workspace_bytes(shape), dtype=torch.uint8, device=DEV)
    got = torch.full((T, 2 * Fs + E), 3.0, dtype=torch.bfloat16, device=DEV)
    want, d_hid, dw = got.clone(), torch.empty(T, Fs, dtype=torch.bfloat16, device=DEV), torch.empty(D, Fs, device=DEV)
    st = torch.cuda.current_stream().cuda_stream
    before = lib.lmoe_pair_gemm_enable(pairs)
    try:
        _cabi.call("lmoe_moe_shared_bwd", shape, dy.data_ptr(), wd.data_ptr(), h1.data_ptr(), hid.data_ptr(), got.data_ptr(),
                   dw.data_ptr(), _cabi.F32, ws.data_ptr(), ws.numel(), status.data_ptr(), st)
        _cabi.call("lmoe_gemm_bf16", T, Fs, D, dy.data_ptr(), D, 0, wd.data_ptr(), Fs, 1, d_hid.data_ptr(), Fs, _cabi.BF16, 1, None,
                   0, status.data_ptr(), st)
        _cabi.call("lmoe_swiglu_bwd", T, Fs, h1.data_ptr(), d_hid.data_ptr(), want.data_ptr(), 2 * Fs + E, None, st)
        torch.cuda.synchronize()
    finally:
        lib.lmoe_pair_gemm_enable(before)
    assert status.item() == 0 and torch.equal(got, want)


@pytest.mark.parametrize("rows", [[1], [0, 128, 200, 1], [700, 0, 130, 385]])
@pytest.mark.parametrize("fp8", [False, True])
def test_routed_adjoint(rows, fp8):
    from swamla_b200 import _cabi
    E, L, F = len(rows), 384, 256
    pads = [(r + 127) // 128 * 128 for r in rows]
    used = sum(pads)
    P = used + 128                                                   # one unused tile of capacity
    i32 = dict(dtype=torch.int32, device=DEV)
    off = torch.tensor([sum(pads[:i]) for i in range(E + 1)], **i32)
    te = torch.tensor([e for e in range(E) for _ in range(pads[e] // 128)] + [0], **i32)
    nt = torch.tensor([used // 128], **i32)
    g = torch.Generator(DEV).manual_seed(used)
    dy, wgu, wd, h1 = _rand(g, P, L), _rand(g, E, L, 2 * F, scale=0.1), _rand(g, E, F, L, scale=0.1), _gates(g, P, F)
    status = torch.zeros(1, **i32)
    st = torch.cuda.current_stream().cuda_stream
    d_hid, want, got = torch.zeros(P, F, dtype=torch.bfloat16, device=DEV), torch.zeros_like(h1), torch.zeros_like(h1)
    if fp8:
        def quant(t):
            q, scal = torch.zeros(t.shape, dtype=torch.uint8, device=DEV), torch.zeros(2, device=DEV)
            _cabi.call("lmoe_fp8_quantize", t.data_ptr(), t.numel() // t.shape[-1], t.shape[-1], None, q.data_ptr(),
                       scal[0:1].data_ptr(), scal[1:2].data_ptr(), st)
            return q, scal[1:2]
        (dyq, s_dy), (wdq, s_wd) = quant(dy), quant(wd)
        _cabi.call("lmoe_grouped_rows_fp8", P, E, L, F, dyq.data_ptr(), wdq.data_ptr(), 0, s_dy.data_ptr(), s_wd.data_ptr(),
                   te.data_ptr(), nt.data_ptr(), d_hid.data_ptr(), status.data_ptr(), st)
        _cabi.call("lmoe_swiglu_bwd", P, F, h1.data_ptr(), d_hid.data_ptr(), want.data_ptr(), 2 * F, nt.data_ptr(), st)
        _cabi.call("lmoe_grouped_swiglu_bwd_fp8", P, E, L, F, dyq.data_ptr(), wdq.data_ptr(), s_dy.data_ptr(), s_wd.data_ptr(),
                   te.data_ptr(), nt.data_ptr(), h1.data_ptr(), got.data_ptr(), None, status.data_ptr(), st)
    else:
        dx, dx_want = torch.zeros_like(dy), torch.zeros_like(dy)
        args = (P, E, L, F, dy.data_ptr(), h1.data_ptr(), wgu.data_ptr(), wd.data_ptr(), te.data_ptr(), nt.data_ptr(), off.data_ptr())
        _cabi.call("lmoe_grouped_bwd_dgrad", *args, d_hid.data_ptr(), want.data_ptr(), dx_want.data_ptr(), status.data_ptr(), st)
        _cabi.call("lmoe_moe_experts_bwd_dgrad", *args, got.data_ptr(), dx.data_ptr(), status.data_ptr(), st)
        assert torch.equal(dx, dx_want)
    torch.cuda.synchronize()
    assert status.item() == 0 and torch.equal(got, want)
    # and the adjoint of d_gate itself, in fp64 on the stored d_hidden: one bf16 rounding and a few fp32 ones
    g64, u64, dh = h1[:used, :F].double(), h1[:used, F:].double(), d_hid[:used].double()
    sg = torch.sigmoid(g64)
    for out, ref in ((got[:used, F:], dh * g64 * sg), (got[:used, :F], dh * u64 * sg * (1 + g64 * (1 - sg)))):
        # near the zero of 1 + g (1 - s) the two terms cancel: their sizes bound the fp32 error
        size = dh.abs() * torch.maximum(u64.abs(), torch.ones_like(g64)) * sg * (1 + g64.abs())
        assert ((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 2.0 ** -20 * size + 1e-38).all()
