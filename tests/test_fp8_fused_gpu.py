"""The fused pieces of the backward of the combine and of the e4m3 expert path against the separate entry points."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _route(T, E, K, L, seed):
    """Routing tables of a random selection (no expert twice per token)."""
    from swamla_b200 import _cabi
    from swamla_b200.functional import RouteTables, make_shape
    dev = torch.device("cuda:0")
    g = torch.Generator(dev).manual_seed(seed)
    shape = make_shape(T, 64, L, E, K, 128, 64)
    sel = torch.rand(T, E, device=dev, generator=g).topk(K, dim=1).indices.to(torch.int32).contiguous()
    route = RouteTables(shape, dev)
    ws = torch.empty(max(16, _cabi.load().lmoe_route_workspace_bytes(shape)), dtype=torch.uint8, device=dev)
    st = torch.cuda.current_stream().cuda_stream
    _cabi.call("lmoe_route_permute", shape, sel.data_ptr(), route.struct, ws.data_ptr(), ws.numel(), st)
    return shape, route, g, st


# one token, K above and not a multiple of the unroll of four, rows of one and several 32-lane passes, an unused expert
@pytest.mark.parametrize("T,E,K,L", [(1, 8, 1, 64), (130, 32, 3, 128), (1000, 128, 12, 256), (77, 64, 32, 1024), (3000, 8, 5, 256)])
def test_combine_adjoint_by_tokens(T, E, K, L):
    from swamla_b200 import _cabi
    shape, route, g, st = _route(T, E, K, L, T + K)
    P, dev = route.padded_rows, "cuda:0"
    d_routed = torch.randn(T, L, device=dev, generator=g).to(torch.bfloat16)
    y = torch.randn(P, L, device=dev, generator=g).to(torch.bfloat16)
    w = torch.rand(T, K, device=dev, generator=g) + 0.05
    out = []
    for by_tokens in (False, True):
        d_y, d_w = torch.full((P, L), 9.0, dtype=torch.bfloat16, device=dev), torch.full((T, K), 9.0, device=dev)
        if by_tokens:
            _cabi.call("lmoe_combine_bwd", shape, d_routed.data_ptr(), y.data_ptr(), w.data_ptr(), route.struct, d_y.data_ptr(),
                       d_w.data_ptr(), st)
        else:
            _cabi.call("lmoe_combine_bwd_rows", d_routed.data_ptr(), y.data_ptr(), w.data_ptr(), route.row_src.data_ptr(), P, K, L,
                       route.n_tiles.data_ptr(), d_y.data_ptr(), d_w.data_ptr(), st)
        out.append((d_y, d_w))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    # e4m3 form: the bytes and the scale that quantising the bf16 rows gives
    used = int(route.n_tiles.item()) * 128
    q_ref, scal_ref = torch.zeros(P, L, dtype=torch.uint8, device=dev), torch.zeros(2, device=dev)
    _cabi.call("lmoe_fp8_quantize", out[0][0].data_ptr(), P, L, route.n_tiles.data_ptr(), q_ref.data_ptr(), scal_ref[0:1].data_ptr(),
               scal_ref[1:2].data_ptr(), st)
    q, scal = torch.full((P, L), 77, dtype=torch.uint8, device=dev), torch.zeros(2, device=dev)
    d_w = torch.full((T, K), 9.0, device=dev)
    _cabi.call("lmoe_fp8_combine_bwd", shape, d_routed.data_ptr(), y.data_ptr(), w.data_ptr(), route.struct, scal[0:1].data_ptr(),
               scal[1:2].data_ptr(), q.data_ptr(), d_w.data_ptr(), st)
    assert torch.equal(scal, scal_ref) and torch.equal(d_w, out[0][1])
    # the sign of a zero may differ only where the bf16 row's does not: the conversion is the same code
    assert torch.equal(q[:used], q_ref[:used])


@pytest.mark.parametrize("T", [1, 200, 3000])
def test_e4m3_gemm_epilogues_with_adjoint_and_amax(T):
    from swamla_b200 import _cabi
    E, K, L, F = 8, 3, 128, 128
    shape, route, g, st = _route(T, E, K, L, T)
    P, dev = route.padded_rows, "cuda:0"
    used = int(route.n_tiles.item()) * 128
    status = torch.zeros(1, dtype=torch.int32, device=dev)

    def quant(t):
        q, scal = torch.zeros(t.shape, dtype=torch.uint8, device=dev), torch.zeros(2, device=dev)
        _cabi.call("lmoe_fp8_quantize", t.data_ptr(), t.numel() // t.shape[-1], t.shape[-1], None, q.data_ptr(),
                   scal[0:1].data_ptr(), scal[1:2].data_ptr(), st)
        return q, scal[1:2]

    rand = lambda *s: torch.randn(*s, device=dev, generator=g).to(torch.bfloat16)
    xq, dx = quant(rand(P, L))
    wq, dw = quant(rand(E, L, 2 * F))
    wdq, dwd = quant(rand(E, F, L))
    te, nt = route.tile_expert.data_ptr(), route.n_tiles.data_ptr()
    h1, hid, amax = torch.zeros(P, 2 * F, dtype=torch.bfloat16, device=dev), torch.zeros(P, F, dtype=torch.bfloat16, device=dev), torch.zeros(1, device=dev)
    _cabi.call("lmoe_grouped_gateup_fp8_amax", P, E, L, F, xq.data_ptr(), wq.data_ptr(), dx.data_ptr(), dw.data_ptr(), te, nt,
               h1.data_ptr(), hid.data_ptr(), amax.data_ptr(), status.data_ptr(), st)
    assert amax.item() == hid[:used].float().abs().max().item()
    d_hid, ref, got = torch.zeros_like(hid), torch.zeros_like(h1), torch.zeros_like(h1)
    dyq, ddy = quant(rand(P, L))
    _cabi.call("lmoe_grouped_rows_fp8", P, E, L, F, dyq.data_ptr(), wdq.data_ptr(), 0, ddy.data_ptr(), dwd.data_ptr(), te, nt,
               d_hid.data_ptr(), status.data_ptr(), st)
    _cabi.call("lmoe_swiglu_bwd", P, F, h1.data_ptr(), d_hid.data_ptr(), ref.data_ptr(), 2 * F, nt, st)
    amax.zero_()
    _cabi.call("lmoe_grouped_swiglu_bwd_fp8", P, E, L, F, dyq.data_ptr(), wdq.data_ptr(), ddy.data_ptr(), dwd.data_ptr(), te, nt,
               h1.data_ptr(), got.data_ptr(), amax.data_ptr(), status.data_ptr(), st)
    torch.cuda.synchronize()
    assert status.item() == 0
    assert amax.item() == got[:used].float().abs().max().item()
    assert torch.equal(got[:used], ref[:used])                       # the same d_hidden, the same adjoint
