"""lmoe_topk_hist_fwd + lmoe_route_gather_fwd against the separate router, permutation and gather entry points (bit-equal),
and the SwiGLU forwards without a saved gate / up against the ones with it (bit-equal)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one token, one top-k block of eight warps and its neighbours, the last size with such blocks and its neighbour (16 warps), the
# last one without the scan kernel and its neighbour, one token per warp with a ragged last chunk; two, three and four tokens per
# warp (chunks of two, three and four mask words) with ragged last chunks, and more chunks than 1,024
@pytest.mark.parametrize("T", [1, 7, 8, 9, 1024, 1025, 4096, 4097, 20001, 32769, 65567, 131089, 140007])
@pytest.mark.parametrize("E,K", [(128, 12), (256, 16), (32, 3), (40, 5), (256, 32)])
def test_fused_routing_equals_separate_entry_points(T, E, K):
    from swamla_b200 import _cabi
    lib = _cabi.load()
    dev = torch.device("cuda:0")
    L = 64
    shape = _cabi.Shape(T=T, D=64, L=L, E=E, K=K, F=64, Fs=64, n_shared=1)
    P = lib.lmoe_padded_rows(shape)
    st = torch.cuda.current_stream().cuda_stream
    g = torch.Generator(dev).manual_seed(T + E)
    logits = torch.randn(T, E, device=dev, generator=g)
    logits[:, : E // 4] += 1.0                                   # uneven load; some experts stay empty at small T
    logits[3::32] += 3000.0                                      # squares that absorb small ones: the z-loss sum's grouping shows
    bias = 0.1 * torch.randn(E, device=dev, generator=g)
    src = torch.randn(T, L, device=dev, generator=g).to(torch.bfloat16)
    got = []
    for fused in (False, True):
        i32 = dict(dtype=torch.int32, device=dev)
        t = dict(counts=torch.full((E,), -7, **i32), offsets=torch.full((E + 1,), -7, **i32),
                 perm=torch.full((T * K,), -7, **i32), pad_offsets=torch.full((E + 1,), -7, **i32),
                 pos=torch.full((T * K,), -7, **i32), row_src=torch.full((P,), -7, **i32),
                 tile_expert=torch.full((P // 128,), -7, **i32), n_tiles=torch.full((1,), -7, **i32))
        route = _cabi.Route(**{k: v.data_ptr() for k, v in t.items()})
        sel, w = torch.full((T, K), -7, **i32), torch.zeros(T, K, device=dev)
        lse, z = torch.zeros(T, device=dev), torch.zeros(1, device=dev)
        rows = torch.full((P, L), 3.0, dtype=torch.bfloat16, device=dev)
        if fused:
            ws = torch.empty(lib.lmoe_route_fwd_workspace_bytes(shape), dtype=torch.uint8, device=dev)
            _cabi.call("lmoe_topk_hist_fwd", shape, logits.data_ptr(), bias.data_ptr(), sel.data_ptr(), w.data_ptr(),
                       lse.data_ptr(), ws.data_ptr(), ws.numel(), st)
            _cabi.call("lmoe_route_gather_fwd", shape, sel.data_ptr(), ws.data_ptr(), ws.numel(), 1e-3, z.data_ptr(), route,
                       src.data_ptr(), 2 * L, rows.data_ptr(), st)
        else:
            ws = torch.empty(max(16, lib.lmoe_route_workspace_bytes(shape)), dtype=torch.uint8, device=dev)
            zp = torch.empty((T + 7) // 8, device=dev)
            _cabi.call("lmoe_gate_topk_fwd", shape, logits.data_ptr(), bias.data_ptr(), 1e-3, sel.data_ptr(), w.data_ptr(),
                       lse.data_ptr(), zp.data_ptr(), z.data_ptr(), st)
            _cabi.call("lmoe_route_permute", shape, sel.data_ptr(), route, ws.data_ptr(), ws.numel(), st)
            _cabi.call("lmoe_gather_rows", src.data_ptr(), t["row_src"].data_ptr(), K, P, L, t["n_tiles"].data_ptr(),
                       rows.data_ptr(), st)
        torch.cuda.synchronize()
        got.append(dict(t, sel=sel, w=w, lse=lse, z=z, rows=rows))
    a, b = got
    for k in a:
        assert torch.equal(a[k], b[k]), k


@pytest.mark.parametrize("M,H", [(1, 64), (129, 96), (300, 160), (1024, 1024)])   # one-CTA and CTA-pair kernels, ragged tiles
def test_swiglu_forward_without_saved_gate_up(M, H):
    from swamla_b200 import _cabi
    dev = torch.device("cuda:0")
    g = torch.Generator(dev).manual_seed(M)
    A = torch.randn(M, 256, device=dev, generator=g).to(torch.bfloat16)
    W = (0.1 * torch.randn(2 * H, 256, device=dev, generator=g)).to(torch.bfloat16)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    st = torch.cuda.current_stream().cuda_stream
    out = []
    for keep in (True, False):
        h1 = torch.empty(M, 2 * H, dtype=torch.bfloat16, device=dev)
        hid = torch.full((M, H), 5.0, dtype=torch.bfloat16, device=dev)
        _cabi.call("lmoe_gemm_swiglu_bf16", M, H, 256, A.data_ptr(), 256, W.data_ptr(), 256, h1.data_ptr() if keep else None,
                   2 * H, hid.data_ptr(), H, status.data_ptr(), st)
        out.append(hid)
    torch.cuda.synchronize()
    assert status.item() == 0 and torch.equal(out[0], out[1])


@pytest.mark.parametrize("name", ["tiny_ragged", "cfg1", "tiny_moe_ragged"])
def test_forward_without_grad_gives_the_training_forward_s_bits(name):
    from oracle import inputs
    from swamla_b200.layer import create_moe_layer
    w = inputs.WORKLOADS[name]
    params, buffers, x, _ = inputs.make_inputs(w)
    layer = create_moe_layer(w.config())
    layer.load_state_dict({**params, **buffers}, strict=True)
    layer = layer.to("cuda:0").to(torch.bfloat16).train()
    xg = x.to("cuda:0").to(torch.bfloat16).requires_grad_(True)
    y1 = layer(xg)
    aux1, counts1 = layer.get_aux_loss(), layer.router._last_counts
    with torch.no_grad():
        y2 = layer(xg)
    assert torch.equal(y1, y2) and torch.equal(aux1, layer.get_aux_loss()) and torch.equal(counts1, layer.router._last_counts)
    layer.check_status()
