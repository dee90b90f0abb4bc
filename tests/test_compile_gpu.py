"""The compiled layer against the eager one, bit for bit, in every mode."""
import pytest
import torch

from oracle import inputs

pytestmark = pytest.mark.gpu


def _layer():
    from swamla_b200.layer import create_moe_layer
    w = inputs.WORKLOADS["tiny"]
    torch.manual_seed(11)
    with torch.device("cuda:0"):
        return create_moe_layer(w.config()).to(torch.bfloat16), torch.randn(1, 200, w.D).to(torch.bfloat16)


# few enough tokens for the evaluation kernels, the first size beyond them; trained, evaluated, frozen with gradients enabled
@pytest.mark.parametrize("tokens", [1, 64, 65])
@pytest.mark.parametrize("mode", ["train", "train without gradients", "evaluation", "frozen evaluation"])
def test_compiled_layer_gives_the_eager_bits(mode, tokens):
    layer, x = _layer()
    x = x[:, :tokens]
    layer.train(mode.startswith("train"))
    layer.requires_grad_(mode != "frozen evaluation")
    torch._dynamo.reset()
    compiled = torch.compile(layer, backend="aot_eager", fullgraph=True)
    with torch.set_grad_enabled(mode in ("train", "frozen evaluation")):
        want, want_aux = layer(x), layer.get_aux_loss()
        got, aux = compiled(x), layer.get_aux_loss()
    layer.check_status()
    assert torch.equal(got, want) and torch.equal(aux, want_aux)
    assert got.requires_grad == want.requires_grad
