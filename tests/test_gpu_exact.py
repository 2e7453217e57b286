"""The correctly rounded linears (fc1_latent, fc2_latent, the dense / scaled-FP8 shared expert and
the router's gate) against the oracle's FP64 sums, at the edges of their dispatch: the FP64 kernels
for few rows, the integer kernel's token tiles of 16 to 64 rows, weights that are no whole tile, and
rows whose sums the rounding test cannot decide."""
import numpy as np
import pytest
import torch

import helpers

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=["bf16", "fp8", "fp32"])
def latent_layer(request, package, synthetic):
    # latent 192: one and a half tiles of weight rows; hidden 320: five 64-byte chunks
    cfg = synthetic.baseline_config(max_tokens=160, experts=64, hidden=320, routed=64, shared=192,
                                    latent=192)
    data = synthetic.make_layer(cfg, seed=91, device="cuda", norm_weight_uniform=True,
                                latent_family=request.param, shared_up_family=request.param,
                                shared_down_family=request.param)
    layer = package.ExpertLayerSlice.create(cfg, data.bindings)
    assert layer is not None, package.ExpertLayerSlice.create_error
    yield layer, data, cfg
    layer.close()


@pytest.mark.parametrize("tokens", [1, 2, 4, 5, 16, 17, 48, 49, 64, 65, 160])
def test_linears_round_the_fp64_sum(latent_layer, synthetic, tokens):
    layer, data, cfg = latent_layer
    x = synthetic.make_tokens(tokens, cfg.hidden_size, seed=tokens, device="cuda").to(torch.float32)
    if tokens > 4:
        x[1] = 0.0                                   # a row of zeros
        x[2] *= 2.0 ** (-30 * torch.rand(cfg.hidden_size, device="cuda"))  # a wide range of sizes
        x[3, 1:] = 0.0                               # one value carries the row
    out = torch.empty_like(x)
    assert layer.run(x, out), layer.last_error
    rep = helpers.compare_layer_with_oracle(layer, data, x, out)
    print(rep.summary())
    assert rep.ok(), rep.summary()
    assert rep.latent_max_diff == 0.0 and rep.logits_max_diff == 0.0


def test_an_fp8_input_scale_of_zero_is_the_smallest_scale(package, synthetic):
    # the reference clamps the scale of the activations' round trip (scaled_fp8_linear.cu:27-33)
    cfg = synthetic.baseline_config(max_tokens=64, experts=64, hidden=320, routed=64, shared=704,
                                    latent=192)
    outs = []
    for scale in (0.0, 1.0 / 1024.0):
        data = synthetic.make_layer(cfg, seed=93, device="cuda", latent_family="fp8",
                                    shared_up_family="fp8", shared_down_family="fp8")
        for linear in (data.bindings.fc1_latent, data.bindings.shared_up_linear,
                       data.bindings.shared_down_linear):
            linear.input_scale = scale
        layer = package.ExpertLayerSlice.create(cfg, data.bindings)
        assert layer is not None, package.ExpertLayerSlice.create_error
        for tokens in (2, 40):  # FP64 and integer kernels
            x = synthetic.make_tokens(tokens, 320, seed=tokens, device="cuda").to(torch.float32)
            out = torch.empty_like(x)
            assert layer.run(x, out), layer.last_error
            outs.append((out, layer.trace(tokens).latent_output))
        layer.close()
    for zero, smallest in zip(outs[:2], outs[2:]):
        assert torch.equal(zero[1], smallest[1])
        assert torch.equal(zero[0], smallest[0])
