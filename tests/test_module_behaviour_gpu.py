"""What the layers owe their callers as modules: hooks, dropout in its own mode, the accepted input shapes."""
import pytest
import torch

from oracle import inputs

pytestmark = pytest.mark.gpu
KINDS = ["latent", "moe"]


def _layer(kind, dropout=0.0):
    from swamla_b200.layer import create_moe_layer
    w = inputs.WORKLOADS["tiny_moe" if kind == "moe" else "tiny"]
    cfg = w.config()
    cfg.dropout = dropout
    torch.manual_seed(7)
    with torch.device("cuda:0"):
        return create_moe_layer(cfg).to(torch.bfloat16), torch.randn(2, 50, w.D).to(torch.bfloat16)


@pytest.mark.parametrize("kind", KINDS)
def test_other_ranks_of_input_are_refused(kind):
    layer, x = _layer(kind)
    for bad in (x[0], x[None]):
        for m in (layer.train(), layer.eval()):
            with torch.no_grad(), pytest.raises(ValueError):
                m(bad)


@pytest.mark.parametrize("tokens", [1, 50])                            # the few-token path and the padded one
@pytest.mark.parametrize("kind", KINDS)
def test_dropout_follows_its_own_mode(kind, tokens):
    layer, x = _layer(kind, 0.5)
    x = x[:, :tokens]
    with torch.no_grad():
        plain = layer.eval()(x)
        layer.dropout.train()                                          # left active in an evaluated layer
        y = layer(x)
        zero = (y == 0) & (plain != 0)
        assert 0.3 < zero.float().mean().item() < 0.7
        assert torch.equal(y[~zero], 2.0 * plain[~zero])
        layer.train().dropout.eval()                                   # and the other way round
        assert (layer(x) != 0).float().mean().item() > 0.99


@pytest.mark.parametrize("kind", KINDS)
def test_dropout_may_be_replaced_or_hooked(kind):
    from swamla_b200.block import NormedResidualFFN
    layer, x = _layer(kind)
    seen = []
    handle = layer.dropout.register_forward_hook(lambda m, a, out: seen.append(out.shape))
    with torch.no_grad():
        want = layer.train()(x)
        layer.eval()(x)
        handle.remove()
        assert len(seen) == 2
        layer.dropout = torch.nn.Identity()
        assert torch.equal(layer.train()(x), want)
        NormedResidualFFN(layer, x.shape[-1]).cuda()(x)


@pytest.mark.parametrize("how", ["forward hook", "pre-hook", "global hook", "forward"])
@pytest.mark.parametrize("kind", KINDS)
def test_whoever_looks_at_the_feed_forward_module_sees_the_stream_s_precision(kind, how):
    from swamla_b200.block import NormedResidualFFN
    layer, x = _layer(kind)
    block, x = NormedResidualFFN(layer, x.shape[-1]).cuda(), x.float()
    with torch.no_grad():
        plain = block(x)
    seen = []
    add = 2.0 ** -13                                                   # lost if the branch were rounded to bf16 after it

    def hook(m, args, out):
        if m is layer:
            seen.extend([args[0].dtype, out.dtype])
            return out + add

    if how == "forward hook":
        handle = layer.register_forward_hook(hook)
    elif how == "pre-hook":
        handle = layer.register_forward_pre_hook(lambda m, args: seen.append(args[0].dtype))
    elif how == "global hook":
        handle = torch.nn.modules.module.register_module_forward_hook(hook)
    else:
        inner = layer.forward
        layer.forward = lambda t: hook(layer, (t,), inner(t))
    try:
        with torch.no_grad():
            y = block(x)
    finally:
        if how != "forward":
            handle.remove()
    assert seen and set(seen) == {torch.float32}
    if how != "pre-hook":
        assert ((y - plain) - add).abs().max().item() <= 2.0 ** -21   # fp32 roundings of values of a few units
    else:
        assert torch.equal(y, plain)


@pytest.mark.parametrize("grad", [True, False])
@pytest.mark.parametrize("kind", KINDS + ["block"])
def test_tensors_on_another_device_are_refused(kind, grad):
    """By the host, before anything is launched."""
    from swamla_b200 import _cabi
    from swamla_b200.block import NormedResidualFFN
    layer, x = _layer("latent" if kind == "block" else kind)
    m = NormedResidualFFN(layer, x.shape[-1]).cuda() if kind == "block" else layer
    names = [n for n, _ in m.named_parameters()] + [n for n, _ in m.named_buffers() if n.endswith("expert_bias")]
    lib = _cabi.load()
    with torch.set_grad_enabled(grad):
        for mode in (m.train(), m.eval()):
            for n in names:
                owner = m.get_submodule(n.rpartition(".")[0])
                t = getattr(owner, n.rpartition(".")[2])
                on_gpu, t.data = t.data, t.data.cpu()
                before = lib.lmoe_launch_count()
                try:
                    with pytest.raises(_cabi.LmoeError, match="is on cpu"):
                        mode(x)
                    assert lib.lmoe_launch_count() - before <= (1 if kind == "block" else 0), n    # the block's norm
                finally:
                    t.data = on_gpu
            mode(x)
            mode.check_status() if kind != "block" else layer.check_status()


def test_conversion_of_a_misaligned_tensor_is_refused():
    from swamla_b200 import _cabi
    a, b = torch.zeros(65, device="cuda:0"), torch.zeros(64, dtype=torch.bfloat16, device="cuda:0")
    st = torch.cuda.current_stream().cuda_stream
    rc = _cabi.load().lmoe_cast_f32_to_bf16(a[1:].data_ptr(), b.data_ptr(), 64, st)
    assert rc == -3                                                     # LMOE_ERR_ALIGN


@pytest.mark.parametrize("kind", KINDS)
def test_a_call_that_fails_between_fork_and_join(kind):
    """A weight that does not begin at 16 bytes is refused by the shared expert's GEMM, when the side stream has work already:
    the streams are joined, and the calls after it give the bits of the ones before."""
    from swamla_b200 import _cabi
    layer, x = _layer(kind)
    w = layer.shared_experts[0].gate_up_proj.weight
    flat = torch.empty(w.numel() + 1, dtype=w.dtype, device=w.device)
    off = flat[1:].view(w.shape)
    off.copy_(w.detach())
    with torch.no_grad():
        want = layer.train()(x)
        for _ in range(5):
            good, w.data = w.data, off
            try:
                with pytest.raises(_cabi.LmoeError, match="aligned"):
                    layer(x)
            finally:
                w.data = good
            assert torch.equal(layer(x), want)
    layer.check_status()
