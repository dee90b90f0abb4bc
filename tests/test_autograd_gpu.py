"""What a module's caller may do with its inputs and outputs under autograd: nothing that a plain module allows may break or,
worse, be answered wrongly without a word."""
import pytest
import torch
import torch.autograd.forward_ad as fwd_ad

from oracle import inputs

pytestmark = pytest.mark.gpu


def _module(kind, dtype=torch.bfloat16):
    from swamla_b200.block import NormedResidualFFN
    from swamla_b200.layer import create_moe_layer
    w = inputs.WORKLOADS["tiny_moe" if kind == "moe" else "tiny"]
    torch.manual_seed(3)
    with torch.device("cuda:0"):
        m = create_moe_layer(w.config()).to(torch.bfloat16)
        if kind == "block":
            m = NormedResidualFFN(m, w.D)
        x = torch.randn(2, 70, w.D, dtype=dtype)
    return m, x


KINDS = ["latent", "moe", "block"]


@pytest.mark.parametrize("kind", KINDS)
def test_output_may_be_changed_in_place(kind):
    m, x = _module(kind)
    xg = x.clone().requires_grad_(True)
    m.train()(xg).sum().backward()
    want, xg.grad = 3.0 * xg.grad, None
    y = m(xg)
    y.mul_(3.0)
    y.sum().backward()
    assert torch.allclose(xg.grad.float(), want.float(), rtol=2e-2, atol=2e-2 * want.float().abs().max().item())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("kind", KINDS)
def test_gradient_in_another_layout(kind, dtype):
    m, x = _module(kind, dtype)
    xg = x.clone().requires_grad_(True)
    dy = torch.randn(70, 2, x.shape[-1], dtype=dtype, device=x.device)
    m.train()(xg).backward(dy.transpose(0, 1).contiguous())
    want, xg.grad = xg.grad, None
    m(xg).transpose(0, 1).backward(dy)             # reaches the module with strides of the transpose
    assert torch.equal(xg.grad, want)


@pytest.mark.parametrize("grad", [True, False])
@pytest.mark.parametrize("kind", KINDS)
def test_forward_mode_is_refused(kind, grad):
    m, x = _module(kind)
    with fwd_ad.dual_level(), torch.set_grad_enabled(grad):
        with pytest.raises((RuntimeError, NotImplementedError)):
            m.eval()(fwd_ad.make_dual(x, torch.ones_like(x)))


@pytest.mark.parametrize("kind", KINDS)
def test_trace_is_refused(kind):
    m, x = _module(kind)
    with torch.no_grad(), pytest.raises(RuntimeError):
        torch.jit.trace(m.eval(), (x,), check_trace=False)


def test_block_takes_flattened_and_broadcast_branches():
    from swamla_b200.block import NormedResidualFFN

    class Branch(torch.nn.Module):
        def __init__(self, f):
            super().__init__()
            self.f = f

        def forward(self, t):
            return self.f(t)

    x = torch.randn(2, 5, 64, device="cuda:0")
    flat = NormedResidualFFN(Branch(lambda t: t.flatten(0, 1).to(torch.bfloat16)), 64).cuda()
    full = NormedResidualFFN(Branch(lambda t: t.to(torch.bfloat16)), 64).cuda()
    one = NormedResidualFFN(Branch(lambda t: torch.ones(64, device=t.device)), 64).cuda()
    for m in (flat, full):
        xg = x.clone().requires_grad_(True)
        y = m(xg)
        y.sum().backward()
        if m is flat:
            want, want_grad = y.detach(), xg.grad
    assert torch.equal(y, want) and torch.equal(xg.grad, want_grad)
    assert torch.equal(one(x), x + 1.0)


@pytest.mark.parametrize("what", ["stream", "bf16 weight"])
@pytest.mark.parametrize("width", [256, 2048])
def test_block_s_inputs_may_change_before_the_backward(what, width):
    """An fp32 stream (the norm keeps its rows in bf16) and a bf16 norm weight (kept in fp32) changed in place between the two
    directions: the gradients are those of the values that the forward saw."""
    from swamla_b200.block import NormedResidualFFN
    torch.manual_seed(5)
    m = NormedResidualFFN(torch.nn.Linear(width, width), width).cuda()
    with torch.no_grad():
        m.ffn_norm.weight.normal_(1.0, 0.1)
    if what == "bf16 weight":
        m.ffn_norm.to(torch.bfloat16)
    x = torch.randn(3, 37, width, device="cuda:0")
    dy = torch.randn_like(x)
    got = []
    for change in (False, True):
        m.zero_grad()
        leaf = x.clone().requires_grad_(True)
        h = 1.0 * leaf
        kept = m.ffn_norm.weight.detach().clone()
        y = m(h)
        if change:
            with torch.no_grad():
                (h if what == "stream" else m.ffn_norm.weight).mul_(3.0)
        y.backward(dy)
        with torch.no_grad():
            m.ffn_norm.weight.copy_(kept)
        got.append((leaf.grad, m.ffn_norm.weight.grad.clone()))
    assert all(torch.equal(a, b) for a, b in zip(*got))


@pytest.mark.parametrize("own", [True, False])
def test_block_takes_a_gradient_that_begins_anywhere(own):
    """An fp32 upstream gradient that is contiguous but does not begin at 16 bytes (a slice of a flat buffer)."""
    from swamla_b200.block import NormedResidualFFN
    m, x = _module("block", torch.float32)
    if not own:                                     # (an element-wise branch: a library GEMM may choose by alignment)
        m = NormedResidualFFN(torch.nn.Tanh(), x.shape[-1]).cuda()
    dy = torch.randn(x.numel() + 1, device=x.device)[1:].view(x.shape)
    assert dy.is_contiguous() and dy.data_ptr() % 16
    grads = []
    for g in (dy, dy.clone()):
        xg = x.clone().requires_grad_(True)
        m.zero_grad()
        m.train()(xg).backward(g)
        grads.append([xg.grad, *[p.grad.clone() for p in m.parameters()]])
    assert all(torch.equal(a, b) for a, b in zip(*grads))
