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


def _contraction_layer(package, synthetic, hidden, shared, seed, experts=32):
    cfg = synthetic.baseline_config(max_tokens=128, experts=experts, hidden=hidden, routed=64,
                                    shared=shared, latent=64)
    data = synthetic.make_layer(cfg, seed=seed, device="cuda", norm_weight_uniform=True,
                                latent_family="fp32", shared_up_family="fp8",
                                shared_down_family="fp32")
    return cfg, data


def test_router_on_both_sides_of_the_product_line(package, synthetic):
    # 512 x 4096: FP64 up to 90 million products, 42 rows
    cfg, data = _contraction_layer(package, synthetic, 4096, 64, 94, experts=512)
    layer = package.ExpertLayerSlice.create(cfg, data.bindings)
    assert layer is not None, package.ExpertLayerSlice.create_error
    for tokens in (42, 43):
        x = synthetic.make_tokens(tokens, 4096, seed=tokens, device="cuda")
        out = torch.empty(x.shape, dtype=torch.float32, device="cuda")
        assert layer.run(x, out), layer.last_error
        rep = helpers.compare_layer_with_oracle(layer, data, x, out)
        assert rep.ok(), rep.summary()
        assert rep.logits_max_diff == 0.0 and rep.latent_max_diff == 0.0
    layer.close()


def test_linears_of_the_checkpoints_lengths(package, synthetic, oracle):
    # contractions over 4096 and 5376: the shared expert's FP64 sums, rounded once
    cfg, data = _contraction_layer(package, synthetic, 4096, 5376, 95)
    layer = package.ExpertLayerSlice.create(cfg, data.bindings)
    assert layer is not None, package.ExpertLayerSlice.create_error
    ocfg, ow = helpers.oracle_config(cfg), helpers.oracle_weights(data)
    for tokens in (3, 65):
        x = synthetic.make_tokens(tokens, 4096, seed=tokens, device="cuda")
        out = torch.empty(x.shape, dtype=torch.float32, device="cuda")
        assert layer.run(x, out), layer.last_error
        trace = layer.trace(tokens)
        y = trace.normalized_input.cpu().numpy()
        up = oracle.router_logits(oracle.fp8_round_trip(y, ow.shared_up_input_scale),
                                  ow.shared_up_dense)
        hidden = np.where(up > 0, up * up, np.float32(0.0))
        want = oracle.router_logits(hidden, ow.shared_down_dense)
        assert np.array_equal(trace.shared_output.cpu().numpy(), want)
    layer.close()


def test_longest_contraction_with_digits_of_one_sign(package, synthetic):
    # 16384 equal products per sum, so that the digits' products add up instead of cancelling: the
    # level sums reach for 32 bits, and the sum is a power of two times one product, exact in FP64.
    # Rows of alternating sign sum to zero, which the rounding test leaves to the FP64 sum.
    cfg, data = _contraction_layer(package, synthetic, 192, 16384, 96)
    up = torch.zeros((16384, 192), device="cuda")
    up[:, 0] = 1.0
    column = torch.randn((192, 1), generator=torch.Generator(device="cuda").manual_seed(97),
                         device="cuda")
    down = column.expand(192, 16384).contiguous()
    down[::16, 1::2] *= -1.0
    data.bindings.shared_up_linear = package.DenseLinear(up)
    data.bindings.shared_down_linear = package.DenseLinear(down)
    layer = package.ExpertLayerSlice.create(cfg, data.bindings)
    assert layer is not None, package.ExpertLayerSlice.create_error
    for tokens in (2, 16, 65, 128):
        x = synthetic.make_tokens(tokens, 192, seed=tokens, device="cuda").to(torch.float32)
        x[:, 0] = x[:, 0].abs() + 0.5
        out = torch.empty_like(x)
        assert layer.run(x, out), layer.last_error
        trace = layer.trace(tokens)
        value = trace.normalized_input[:, :1]
        want = (16384.0 * (value * value).double() * column.double().T).float()
        want[:, ::16] = 0.0
        assert torch.equal(trace.shared_output, want)
    layer.close()


@pytest.mark.parametrize("fc1,up", [("fp8", "bf16"), ("bf16", "fp32")])
def test_roundings_four_to_a_thread_are_those_of_one(package, synthetic, fc1, up):
    # four values a thread from four blocks of 1024 columns per SM, from a third of one where the contraction
    # is 64 long (fc2_latent); 1088 and 1152 columns end inside a block
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    cfg = synthetic.baseline_config(max_tokens=4 * sms, experts=32, hidden=1088, routed=64, shared=1152,
                                    latent=64, top_k=2)
    data = synthetic.make_layer(cfg, seed=91, device="cuda", norm_weight_uniform=True, latent_family=fc1,
                                shared_up_family=up)
    layer = package.ExpertLayerSlice.create(cfg, data.bindings)
    assert layer is not None, package.ExpertLayerSlice.create_error
    x = synthetic.make_tokens(4 * sms, 1088, seed=92, device="cuda")
    for dtype in (torch.float32, torch.bfloat16):
        four = torch.empty(x.shape, dtype=dtype, device="cuda")
        assert layer.run(x, four), layer.last_error
        for rows in (sms // 3, sms // 3 + 1, 4 * sms - 1):
            one = torch.empty_like(four[:rows])
            assert layer.run(x[:rows], one), layer.last_error
            assert torch.equal(four[:rows], one)
    rep = helpers.compare_layer_with_oracle(layer, data, x[:-1], one, raw_run=False)
    assert rep.ok(), rep.summary()
    layer.close()
