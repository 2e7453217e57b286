"""The sizes at which a different kernel, or a different split of one, takes over: results on both
sides of each line against the CPU oracle, and layers that run beside each other on two streams."""
import numpy as np
import pytest
import torch

import helpers

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def small_layer(package, synthetic):
    cfg = synthetic.baseline_config(max_tokens=2049, experts=32, hidden=512, routed=256, shared=512)
    data = synthetic.make_layer(cfg, seed=41, device="cuda", norm_weight_uniform=True)
    layer = package.ExpertLayerSlice.create(cfg, data.bindings)
    assert layer is not None and layer.valid(), package.ExpertLayerSlice.create_error
    yield layer, data
    layer.close()


# 32 experts, top-6: few-row epilogue up to 16 rows a tile; two-pass router from 256; CTA pairs from 100
# rows per expert (534 tokens), and with them the shared expert beside the router; a block per row in the
# quantiser up to 888, per token in the exact selection up to 804
@pytest.mark.parametrize("tokens", [16, 17, 129, 255, 256, 394, 395, 533, 534, 640, 641, 804, 805, 888, 889,
                                    1184, 1185, 1280, 1281, 2048, 2049])
def test_layer_on_both_sides_of_each_line(small_layer, synthetic, tokens):
    layer, data = small_layer
    x = synthetic.make_tokens(tokens, 512, seed=300 + tokens, device="cuda")
    out = torch.empty(x.shape, dtype=torch.float32, device="cuda")
    assert layer.run(x, out), layer.last_error
    rep = helpers.compare_layer_with_oracle(layer, data, x, out)
    assert rep.ok(), rep.summary()


def test_shared_expert_on_both_sides_of_its_line(package, synthetic):
    # in the routed experts' launch up to 56 K blocks of its tiles per SM: 128 for every 128 tokens here, seven
    # times that on 18 SMs
    cfg = synthetic.baseline_config(max_tokens=897, experts=128, hidden=256, routed=64, shared=8192)
    data = synthetic.make_layer(cfg, seed=45, device="cuda", norm_weight_uniform=True)
    layer = package.ExpertLayerSlice.create(cfg, data.bindings)
    assert layer is not None, package.ExpertLayerSlice.create_error
    layer.reserve_sms(torch.cuda.get_device_properties(0).multi_processor_count - 18)
    for tokens in (896, 897):
        x = synthetic.make_tokens(tokens, 256, seed=tokens, device="cuda")
        out = torch.empty(x.shape, dtype=torch.float32, device="cuda")
        assert layer.run(x, out), layer.last_error
        rep = helpers.compare_layer_with_oracle(layer, data, x, out)
        assert rep.ok(), rep.summary()
    layer.close()


def test_pairs_share_rows_of_every_count(package, synthetic):
    # experts without rows, with fewer than a box of them and with several pairs of tiles
    cfg = synthetic.baseline_config(max_tokens=1501, experts=32, hidden=512, routed=256, shared=512)
    data = synthetic.make_layer(cfg, seed=43, device="cuda", skewed=True)
    layer = package.ExpertLayerSlice.create(cfg, data.bindings)
    assert layer is not None, package.ExpertLayerSlice.create_error
    for tokens in (534, 1501):
        x = synthetic.make_tokens(tokens, 512, seed=tokens, device="cuda")
        out = torch.empty(x.shape, dtype=torch.float32, device="cuda")
        assert layer.run(x, out), layer.last_error
        rep = helpers.compare_layer_with_oracle(layer, data, x, out)
        assert rep.ok(), rep.summary()
    layer.close()


# up to eight tokens, 4096 columns and two blocks of the gate per SM (one token: 512 experts; four: 256; eight:
# 148) have one launch in front of the experts; the stages are timed through the four launches it stands for
@pytest.mark.parametrize("experts,hidden,top_k,groups", [(32, 448, 6, 1), (256, 1024, 32, 4),
                                                         (96, 4096, 1, 1), (128, 4160, 8, 8),
                                                         (288, 448, 8, 1), (512, 512, 22, 1)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_front_end_of_a_few_tokens(package, synthetic, experts, hidden, top_k, groups, dtype):
    cfg = synthetic.baseline_config(max_tokens=16, experts=experts, hidden=hidden, routed=64,
                                    shared=128, top_k=top_k)
    cfg.n_group, cfg.topk_group = groups, max(1, groups // 2)
    data = synthetic.make_layer(cfg, seed=experts, device="cuda", norm_weight_uniform=True,
                                skewed=experts == 32)
    layer = package.ExpertLayerSlice.create(cfg, data.bindings)
    assert layer is not None, package.ExpertLayerSlice.create_error
    for tokens in (1, 2, 4, 5, 8, 9):
        x = synthetic.make_tokens(tokens, hidden, seed=tokens, device="cuda").to(dtype)
        for out_dtype in (torch.bfloat16, torch.float32):
            out, launches = (torch.empty(x.shape, dtype=out_dtype, device="cuda") for _ in range(2))
            layer.enable_stage_timing(True)
            assert layer.run(x, launches), layer.last_error
            layer.enable_stage_timing(False)
            for _ in range(2):
                assert layer.run(x, out), layer.last_error
                assert torch.equal(out, launches)
        rep = helpers.compare_layer_with_oracle(layer, data, x, out)
        assert rep.ok(), rep.summary()
    layer.close()


# one token of a latent layer: linears of every family join that launch, unfinished groups of eight outputs
# and all; the routed sum, fc2_latent and the mixer are one launch behind the experts
@pytest.mark.parametrize("experts,top_k,hidden,latent,shared,fc1,up", [
    (64, 6, 448, 192, 704, "fp8", "fp8"), (160, 8, 4096, 64, 64, "bf16", "fp32"),
    (512, 22, 1024, 320, 448, "fp32", "bf16"), (288, 32, 512, 64, 128, "fp8", "nvfp4")])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_one_token_of_a_latent_layer(package, synthetic, experts, top_k, hidden, latent, shared, fc1, up,
                                     dtype):
    cfg = synthetic.baseline_config(max_tokens=2, experts=experts, hidden=hidden, routed=64,
                                    shared=shared, top_k=top_k, latent=latent)
    data = synthetic.make_layer(cfg, seed=experts, device="cuda", norm_weight_uniform=True,
                                latent_family=fc1, shared_up_family=up)
    layer = package.ExpertLayerSlice.create(cfg, data.bindings)
    assert layer is not None, package.ExpertLayerSlice.create_error
    x = synthetic.make_tokens(1, hidden, seed=9, device="cuda").to(dtype)
    out, launches = (torch.empty(x.shape, device="cuda") for _ in range(2))
    layer.enable_stage_timing(True)
    assert layer.run(x, launches), layer.last_error
    layer.enable_stage_timing(False)
    for _ in range(2):
        assert layer.run(x, out), layer.last_error
        assert torch.equal(out, launches)
    rep = helpers.compare_layer_with_oracle(layer, data, x, out)
    assert rep.ok(), rep.summary()
    assert rep.latent_max_diff == 0.0
    layer.close()


# many experts are narrowed down first (from 11 to 23 selected ones, or beyond 256), unless too many share the
# bound
@pytest.mark.parametrize("experts,top_k,n_group", [(160, 1, 1), (256, 8, 8), (512, 22, 1), (512, 32, 4),
                                                   (160, 10, 1), (160, 11, 1), (256, 16, 8), (384, 1, 1),
                                                   (512, 23, 1), (512, 24, 1)])
@pytest.mark.parametrize("levels", [1, 3, 100000])
def test_selection_among_many_with_ties(package, oracle, experts, top_k, n_group, levels):
    g = torch.Generator().manual_seed(experts + levels)
    logits = torch.randint(-levels, levels, (9, experts), generator=g).float() / levels
    bias = torch.randint(0, 2, (experts,), generator=g).float() * 0.25
    index, weight = package.router_topk(logits.cuda(), bias.cuda(), top_k, n_group, max(1, n_group // 2),
                                        True, 2.5)
    want_index, want_weight = oracle.select_top_experts(logits.numpy(), bias.numpy(), top_k, n_group,
                                                        max(1, n_group // 2), True, 2.5)
    assert np.array_equal(index.cpu().numpy(), want_index)
    # (the host's exponential is within an ulp)
    assert np.allclose(weight.cpu().numpy(), want_weight, rtol=1e-6, atol=0)


@pytest.mark.parametrize("rows", [3, 1185])
@pytest.mark.parametrize("cols", [16, 1008, 2048, 2064, 4096, 4112, 5376, 6144, 6160])
def test_quantiser_row_lengths(package, oracle, rows, cols):
    x = torch.randn(rows, cols, generator=torch.Generator().manual_seed(rows + cols)) * 3.0
    packed, scales, ts, _ = package.quantize_nvfp4(x.cuda(), per_row=True, swizzled=True)
    w = torch.linspace(0.9, 1.1, cols)
    y = package.rmsnorm(x.cuda(), w.cuda(), 1e-5)
    torch.cuda.synchronize()
    for got, expected in zip((packed, scales, ts), oracle.pack_nvfp4_per_row(x.numpy())):
        assert np.array_equal(got.cpu().numpy(), expected)
    assert np.array_equal(y.cpu().numpy(), oracle.rmsnorm(x.numpy(), w.numpy(), 1e-5))


def test_placing_on_both_sides_of_its_line(package, synthetic):
    # a warp per pair up to 40 KB of pairs per SM: 5262 pairs of 1152 bytes, 877 tokens
    cfg = synthetic.baseline_config(max_tokens=1024, experts=32, hidden=2048, routed=64, shared=64)
    data = synthetic.make_layer(cfg, seed=84, device="cuda", norm_weight_uniform=True)
    layer = package.ExpertLayerSlice.create(cfg, data.bindings)
    assert layer is not None, package.ExpertLayerSlice.create_error
    for tokens in (877, 878):
        x = synthetic.make_tokens(tokens, 2048, seed=tokens, device="cuda")
        out = torch.empty(x.shape, dtype=torch.float32, device="cuda")
        assert layer.run(x, out), layer.last_error
        rep = helpers.compare_layer_with_oracle(layer, data, x, out)
        assert rep.ok(), rep.summary()
    layer.close()


# 148 SMs: a block per row up to 888 rows of 2816 columns at most, register rows of 4, 6, 8 and 11 steps
# of 256 from there; longer bf16 rows a block each up to 3552, then three reads of the row
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,cols", [(888, 2816), (889, 1024), (889, 1040), (889, 1536), (889, 1552),
                                       (889, 2048), (889, 2064), (889, 2816), (889, 2832),
                                       (3552, 2832), (3553, 2832), (3553, 6144)])
def test_quantiser_kernel_lines(package, oracle, rows, cols, dtype):
    x = torch.randn(rows, cols, generator=torch.Generator().manual_seed(rows + cols)).to(dtype)
    w = torch.linspace(0.9, 1.1, cols)
    packed, scales, ts, _ = package.quantize_nvfp4(x.cuda(), per_row=True, swizzled=True)
    y = package.rmsnorm(x.cuda(), w.cuda(), 1e-5)
    torch.cuda.synchronize()
    x = x.to(torch.float32).numpy()
    for got, expected in zip((packed, scales, ts), oracle.pack_nvfp4_per_row(x)):
        assert np.array_equal(got.cpu().numpy(), expected)
    assert np.array_equal(y.cpu().numpy(), oracle.rmsnorm(x, w.numpy(), 1e-5))


def test_two_layers_beside_each_other(package, synthetic):
    # chained launches and kernels whose tiles wait for one another, on two streams at once
    cfg = synthetic.baseline_config(max_tokens=512, experts=32, hidden=512, routed=256, shared=512)
    layers = []
    for seed in (51, 52):
        data = synthetic.make_layer(cfg, seed=seed, device="cuda")
        layers.append(package.ExpertLayerSlice.create(cfg, data.bindings))
    for tokens in (1, 40, 200, 500):
        xs = [synthetic.make_tokens(tokens, 512, seed=60 + i, device="cuda") for i in range(2)]
        alone = []
        for layer, x in zip(layers, xs):
            out = torch.empty(x.shape, dtype=torch.float32, device="cuda")
            assert layer.run(x, out), layer.last_error
            alone.append(out)
        torch.cuda.synchronize()
        streams = [torch.cuda.Stream() for _ in range(2)]
        outs = [torch.empty_like(a) for a in alone]
        for _ in range(10):
            for layer, x, out, stream in zip(layers, xs, outs, streams):
                with torch.cuda.stream(stream):
                    layer.run_async(x, out)
        for layer, out, want, stream in zip(layers, outs, alone, streams):
            with torch.cuda.stream(stream):
                assert layer.sync_status() == 0
            assert torch.equal(out, want)
    for layer in layers:
        layer.close()


@pytest.mark.parametrize("family", ["bf16", "fp8", "fp32"])
def test_integer_linears_at_the_edges_of_their_tiles(package, synthetic, family):
    # shared_up with 704 outputs (five and a half tiles of weight rows): too many for the FP64 kernels
    cfg = synthetic.baseline_config(max_tokens=160, experts=64, hidden=320, routed=64, shared=704,
                                    latent=192)
    data = synthetic.make_layer(cfg, seed=92, device="cuda", latent_family=family,
                                shared_up_family=family, shared_down_family=family)
    layer = package.ExpertLayerSlice.create(cfg, data.bindings)
    assert layer is not None, package.ExpertLayerSlice.create_error
    for tokens in (5, 16, 17, 48, 49, 64, 65, 160):
        x = synthetic.make_tokens(tokens, 320, seed=tokens, device="cuda").to(torch.float32)
        x[1] = 0.0
        x[3, 1:] = 0.0
        out = torch.empty_like(x)
        assert layer.run(x, out), layer.last_error
        rep = helpers.compare_layer_with_oracle(layer, data, x, out)
        assert rep.ok(), rep.summary()
        assert rep.latent_max_diff == 0.0 and rep.logits_max_diff == 0.0
    layer.close()


def test_threads_launch_one_kernel_with_different_shared_memory(package, synthetic):
    # row tiles of 32 and of 128 rows give the streaming kernel different stages; a thread must not
    # meet the other's limit between setting its own and launching
    import ctypes
    import threading
    lib, rows = package.load_library(), (8, 128)
    networks, inputs, outputs, wanted = [], [], [], []
    for i, count in enumerate(rows):
        up, down = synthetic.make_ffn_weights(256, 128, seed=70 + i, device="cuda")
        networks.append(package.ExpertFfn(up, down, max_rows=128))
        inputs.append(synthetic.make_tokens(count, 256, seed=72, device="cuda"))
        outputs.append(torch.zeros((count, 256), dtype=torch.float32, device="cuda"))
        wanted.append(networks[i].run(inputs[i], 3))
    torch.cuda.synchronize()
    refused = [None, None]

    def work(i):
        stream = torch.cuda.Stream()
        call = (networks[i]._handle, ctypes.c_void_p(stream.cuda_stream), inputs[i].data_ptr(),
                package.NMOE_BF16, rows[i], outputs[i].data_ptr(), 3)
        refused[i] = sum(lib.nmoe_ffn_run(*call) != 0 for _ in range(40000))
        stream.synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert refused == [0, 0]
    for ffn, out, want in zip(networks, outputs, wanted):
        assert torch.equal(out, want)
        ffn.close()


@pytest.mark.parametrize("tokens", [40, 300, 1100])
def test_a_row_that_is_not_a_number_stays_alone(small_layer, synthetic, tokens):
    # its scores are no numbers, so nor are its weights and its output (the reference's arithmetic);
    # no row of an earlier batch takes their place, and the other tokens do not change
    layer, _ = small_layer
    x = synthetic.make_tokens(tokens, 512, seed=500 + tokens, device="cuda")
    clean = torch.empty(x.shape, dtype=torch.float32, device="cuda")
    assert layer.run(x, clean), layer.last_error
    bad = x.clone()
    bad[7, 100] = float("nan")
    bad[30, 3] = float("inf")
    out = torch.empty_like(clean)
    assert layer.run(bad, out), layer.last_error
    index = layer.trace(tokens).selected_index
    assert int(index.min()) >= 0 and int(index.max()) < 32
    assert torch.isnan(out[[7, 30]]).all()
    others = [t for t in range(tokens) if t not in (7, 30)]
    assert torch.equal(out[others], clean[others])



@pytest.mark.parametrize("experts", [192, 224, 256])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_router_of_many_experts(package, synthetic, experts, dtype):
    # the gate tiles of pass 1 grow with the experts; its stages have to fit shared memory
    cfg = synthetic.baseline_config(max_tokens=300, experts=experts, hidden=320, routed=64, shared=64)
    data = synthetic.make_layer(cfg, seed=80, device="cuda", norm_weight_uniform=True)
    layer = package.ExpertLayerSlice.create(cfg, data.bindings)
    assert layer is not None, package.ExpertLayerSlice.create_error
    x = synthetic.make_tokens(300, 320, seed=81, device="cuda").to(dtype)
    out = torch.empty(x.shape, dtype=torch.float32, device="cuda")
    assert layer.run(x, out), layer.last_error
    rep = helpers.compare_layer_with_oracle(layer, data, x, out)
    layer.close()
    assert rep.ok(), rep.summary()


def test_gate_slices_exist_where_a_call_needs_them(package, synthetic, monkeypatch):
    # a gate of 128 x 2688 in front of the two-pass router stays with the FP64 kernels (up to 255
    # rows): its digits and their workspace (25 MB at 1024 tokens) are for layers without that router
    cfg = synthetic.baseline_config(max_tokens=1024, hidden=2688, routed=64, shared=64)
    data = synthetic.make_layer(cfg, seed=82, device="cuda")
    torch.cuda.synchronize()

    def create():
        free = torch.cuda.mem_get_info()[0]
        layer = package.ExpertLayerSlice.create(cfg, data.bindings)
        assert layer is not None, package.ExpertLayerSlice.create_error
        return layer, free - torch.cuda.mem_get_info()[0]

    create()[0].close()
    two_pass, two_pass_bytes = create()
    monkeypatch.setenv("NMOE_ROUTER_FP64_ONLY", "1")
    exact_only, exact_only_bytes = create()
    print(two_pass_bytes, exact_only_bytes)
    assert two_pass_bytes < exact_only_bytes
    x = synthetic.make_tokens(200, 2688, seed=83, device="cuda")
    results = []
    for layer, reserved in ((exact_only, 0), (two_pass, 0), (two_pass, 130), (two_pass, 0)):
        layer.reserve_sms(reserved)  # with 18 SMs left the gate's FP64 kernels no longer pay
        out = torch.empty(x.shape, dtype=torch.float32, device="cuda")
        assert layer.run(x, out), layer.last_error
        results.append((out, layer.trace(200).router_logits))
    for out, logits in results[1:]:
        assert torch.equal(logits, results[0][1])
        assert torch.equal(out, results[0][0])
    two_pass.close()
    exact_only.close()
