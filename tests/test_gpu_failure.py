"""Failure detection on the device without faulting, trapping or hanging it: a kernel that
waits for another GPU gives up after a limit and leaves an error status the host reads."""
import time

import pytest
import torch

pytestmark = pytest.mark.gpu

NMOE_ERR_DEVICE_TIMEOUT = 4


def test_bounded_flag_wait_runs_out_and_the_layer_stays_usable(package, synthetic):
    cfg = synthetic.baseline_config(max_tokens=64, experts=32, hidden=512, routed=256, shared=512)
    data = synthetic.make_layer(cfg, seed=11, device="cuda")
    layer = package.ExpertLayerSlice.create(cfg, data.bindings)
    assert layer is not None
    x = synthetic.make_tokens(16, cfg.hidden_size, seed=12, device="cuda")
    out = torch.empty((16, cfg.hidden_size), dtype=torch.float32, device="cuda")
    assert layer.run(x, out), layer.last_error
    before = out.clone()

    # a flag that nothing raises: the wait runs out after the (short) limit
    layer.set_wait_limit_ms(20.0)
    flag = torch.zeros((1,), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    start = time.perf_counter()
    layer.wait_flag(flag, 1)
    status = layer.sync_status()
    elapsed = time.perf_counter() - start
    assert status == NMOE_ERR_DEVICE_TIMEOUT
    assert elapsed < 2.0, f"the bounded wait took {elapsed:.3f} s"

    # a raised flag passes at once, and the error slot was cleared by the read above
    flag.fill_(1)
    layer.wait_flag(flag, 1)
    assert layer.sync_status() == 0

    # the context and the layer are intact
    assert layer.run(x, out), layer.last_error
    assert torch.equal(out, before)
    layer.close()


def test_a_refused_allocation_does_not_fail_the_next_call(package, synthetic):
    up, down = synthetic.make_ffn_weights(256, 128, seed=13, device="cuda")
    ffn = package.ExpertFfn(up, down, max_rows=64)
    x = synthetic.make_tokens(20, 256, seed=14, device="cuda")
    want = ffn.run(x)
    # more scratch than any GPU holds: refused at once
    cfg = synthetic.baseline_config(max_tokens=2 ** 30, experts=32, hidden=512, routed=64, shared=64)
    data = synthetic.make_layer(cfg, seed=15, device="cuda")
    assert package.ExpertLayerSlice.create(cfg, data.bindings) is None
    assert torch.equal(ffn.run(x), want)
    ffn.close()


def test_a_layer_keeps_its_scratch_when_it_cannot_grow(package, synthetic):
    cfg = synthetic.baseline_config(max_tokens=64, experts=32, hidden=512, routed=64, shared=64)
    data = synthetic.make_layer(cfg, seed=16, device="cuda")
    layer = package.ExpertLayerSlice.create(cfg, data.bindings)
    x = synthetic.make_tokens(64, 512, seed=17, device="cuda")
    out = torch.empty((64, 512), dtype=torch.float32, device="cuda")
    assert layer.run(x, out), layer.last_error
    with pytest.raises(package.NmoeError):
        layer.reserve_tokens(2 ** 30)
    again = torch.empty_like(out)
    assert layer.run(x, again), layer.last_error
    assert torch.equal(again, out)
    layer.reserve_tokens(200)
    layer.set_unfused_activation(True)
    assert layer.run(x, again), layer.last_error
    assert torch.equal(again, out)
    layer.close()


def test_a_layer_keeps_its_workspace_when_fewer_sms_need_a_larger_one(package, synthetic):
    # with 4 SMs left the gate goes through the integer kernel, whose digits of 1024 rows of 11008 are
    # 56 MB; fc2_latent uses the same workspace
    cfg = synthetic.baseline_config(max_tokens=1024, experts=32, hidden=11008, routed=64, shared=64,
                                    latent=64, top_k=2)
    data = synthetic.make_layer(cfg, seed=20, device="cuda")
    layer = package.ExpertLayerSlice.create(cfg, data.bindings)
    assert layer is not None, package.ExpertLayerSlice.create_error
    x = synthetic.make_tokens(200, 11008, seed=21, device="cuda")
    out, again = (torch.empty((200, 11008), dtype=torch.float32, device="cuda") for _ in range(2))
    assert layer.run(x, out), layer.last_error
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - (40 << 20), dtype=torch.uint8, device="cuda")
    with pytest.raises(package.NmoeError):
        layer.reserve_sms(144)
    del held
    torch.cuda.empty_cache()
    for reserved in (0, 144):
        layer.reserve_sms(reserved)
        assert layer.run(x, again), layer.last_error
        assert torch.equal(again, out)
    # scratch made for all SMs has no room for the gate, although its digits are there
    layer.reserve_sms(0)
    layer.reserve_tokens(1025)
    layer.reserve_sms(144)
    assert layer.run(x, again), layer.last_error
    assert torch.equal(again, out)
    layer.close()


def test_unfused_rows_follow_the_scratch(package, synthetic):
    # enabled, disabled, grown, enabled: the FP32 rows have to be the larger scratch's
    cfg = synthetic.baseline_config(max_tokens=16, experts=32, hidden=512, routed=256, shared=256)
    data = synthetic.make_layer(cfg, seed=18, device="cuda")
    layer = package.ExpertLayerSlice.create(cfg, data.bindings)
    x = synthetic.make_tokens(700, 512, seed=19, device="cuda")
    out = torch.empty((700, 512), dtype=torch.float32, device="cuda")
    layer.set_unfused_activation(True)
    assert layer.run(x[:16], out[:16]), layer.last_error
    layer.set_unfused_activation(False)
    layer.reserve_tokens(700)
    assert layer.run(x, out), layer.last_error
    free = torch.cuda.mem_get_info()[0]
    layer.set_unfused_activation(True)
    # 4200 pairs in row tiles of 128: at least their FP32 rows
    assert free - torch.cuda.mem_get_info()[0] >= 4200 * 256 * 4
    again = torch.empty_like(out)
    assert layer.run(x, again), layer.last_error
    assert torch.equal(again, out)
    layer.close()
