"""The few-token forward (evaluation mode, no gradients) against the padded path of the same layer.

Both are bf16 pipelines with the same rounding points and fp32 sums in another order: they differ by single bf16 ulps of
intermediates, for which the layer tests allow 2.5e-3 relative Frobenius error and two ulps (2^-6) per element of the output's
scale.  A token whose K-th and (K+1)-th scores are within the fp32 rounding of the logits may select another expert; tokens
with such a near-tie (gap below 1e-5) are left out of the comparison.
"""
import pytest
import torch

from oracle import inputs

pytestmark = pytest.mark.gpu


# one token, the edges of every token-tile count (8, 16, 32, 64), and the first sizes beyond the path: 65, and 25 for wide experts
@pytest.mark.parametrize("T", [1, 2, 8, 9, 16, 17, 24, 25, 33, 64, 65])
# widths of one and several passes, fewer slots than experts and more, 4 to 256 experts, both layer classes
@pytest.mark.parametrize("name", ["tiny", "cfg1", "cfg5_2k", "cfg3", "tiny_moe", "moe_1b"])
def test_few_token_forward_matches_padded_path(name, T):
    from swamla_b200 import _cabi
    from swamla_b200.layer import create_moe_layer
    w = inputs.WORKLOADS[name]
    torch.manual_seed(T)
    with torch.device("cuda:0"):
        layer = create_moe_layer(w.config()).to(torch.bfloat16)
        with torch.no_grad():
            for p in layer.parameters():
                p.normal_(0.0, 0.05)
            layer.router.expert_bias.normal_(0.0, 0.05)
        x = torch.randn(T, 1, w.D).to(torch.bfloat16)
    lib = _cabi.load()
    shape = _cabi.Shape(T=T, D=w.D, L=w.L, E=w.E, K=w.K, F=w.F, Fs=w.Fs, n_shared=1)
    few = T <= (64 if max(2 * w.F, w.L) <= 512 else 24)
    assert lib.lmoe_few_applies(shape) == (1 if few else 0)
    with torch.no_grad():
        y_ref = layer.train()(x)
        z_ref = layer.get_aux_loss().clone()
        before = lib.lmoe_launch_count()
        y = layer.eval()(x)
        assert (lib.lmoe_launch_count() - before <= 4) == few
        if not few:
            assert torch.equal(y, y_ref)
        y2 = layer(x)
    layer.check_status()
    assert torch.equal(y, y2)                                             # deterministic
    scores = torch.sigmoid(x.reshape(T, -1).float() @ layer.router.gate.weight.float().t()) + layer.router.expert_bias.float()
    top = scores.topk(w.K + 1, dim=1).values if w.K < w.E else None
    clear = (top[:, w.K - 1] - top[:, w.K] > 1e-5) if top is not None else torch.ones(T, dtype=torch.bool, device=x.device)
    assert clear.float().mean().item() > 0.5
    a, b = y.reshape(T, -1)[clear].float(), y_ref.reshape(T, -1)[clear].float()
    assert ((a - b).norm() / b.norm()).item() <= 2.5e-3
    rms = b.square().mean().sqrt()
    assert ((a - b).abs() / torch.maximum(b.abs(), rms)).max().item() <= 2.0 ** -6
    assert abs(layer.get_aux_loss().item() - z_ref.item()) <= 1e-5 * abs(z_ref.item())


def test_gradients_and_training_mode_keep_the_padded_path():
    from swamla_b200 import _cabi
    from swamla_b200.layer import create_moe_layer
    w = inputs.WORKLOADS["tiny"]
    with torch.device("cuda:0"):
        layer = create_moe_layer(w.config()).to(torch.bfloat16).eval()
        x = torch.randn(2, 3, w.D).to(torch.bfloat16)
    lib = _cabi.load()
    before = lib.lmoe_launch_count()
    y = layer(x.requires_grad_(True))                                    # evaluation mode with gradients: a backward may follow
    assert lib.lmoe_launch_count() - before > 4
    y.sum().backward()
    assert x.grad is not None and layer.down_proj.weight.grad is not None


@pytest.mark.parametrize("T", [1, 64, 65])
def test_e4m3_layer_keeps_its_precision_at_every_size(T):
    """An e4m3 layer in evaluation gives the training forward's bits: the same token's output does not depend on whether the
    call holds few enough tokens for the bf16 kernels."""
    from swamla_b200.layer import create_moe_layer
    w = inputs.WORKLOADS["cfg1"]
    cfg = w.config()
    cfg.moe_fp8 = True
    torch.manual_seed(T)
    with torch.device("cuda:0"):
        layer = create_moe_layer(cfg).to(torch.bfloat16)
        x = torch.randn(1, T, w.D).to(torch.bfloat16)
    assert layer.fp8_experts
    with torch.no_grad():
        want = layer.train()(x)
        want_aux = layer.get_aux_loss()
        got = layer.eval()(x)
    layer.check_status()
    assert torch.equal(got, want) and torch.equal(layer.get_aux_loss(), want_aux)


@pytest.mark.parametrize("K", [1, 6, 7, 16])                             # the combine takes six slots at a time
def test_infinite_expert_output_stays_infinite(K):
    """The last slot's expert overflows bf16 in one latent column: infinities in the output, as on the padded path, no NaN."""
    from types import SimpleNamespace
    from swamla_b200.layer import create_moe_layer
    cfg = SimpleNamespace(n_embd=128, latent_n_experts=32, latent_n_activated=K, latent_dim=64, expert_dim=256, latent_ratio=4,
                          n_shared_experts=1, bias=False, dropout=0.0, use_latent_moe=True)
    torch.manual_seed(K)
    with torch.device("cuda:0"):
        layer = create_moe_layer(cfg).to(torch.bfloat16).train()
        x = torch.randn(1, 1, 128).to(torch.bfloat16)
    with torch.no_grad():
        layer(x)
        e = int(layer.router._last_selected_experts[0, K - 1])
        xl = (x[0, 0] @ layer.down_proj.weight.t()).float()
        layer.experts.gate_up_weight[e] = (xl / xl.square().sum())[:, None]      # gate = up = 1: every hidden value 0.73
        layer.experts.down_weight[e, :, 0] = 1e38
        want = layer(x)
        got = layer.eval()(x)
    assert want.isinf().any() and not want.isnan().any()
    assert torch.equal(got.isinf(), want.isinf()) and not got.isnan().any()
