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
