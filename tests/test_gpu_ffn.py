"""GPU parity of one routed-expert NVFP4 FFN: y = W_down relu(W_up x)^2 with
dynamic per-16-block activation quantisation, against the reference's host FP32
dequantise-then-matmul path as restated by the oracle."""
import numpy as np
import pytest
import torch

import helpers

pytestmark = pytest.mark.gpu


def _run_case(package, oracle, synthetic, rows, hidden, inter, variant, seed=0):
    up, down = synthetic.make_ffn_weights(hidden, inter, seed=seed, device="cuda")
    x = synthetic.make_tokens(rows, hidden, seed=seed + 100, device="cuda")
    ffn = package.ExpertFfn(up, down, max_rows=max(rows, 128))
    out = ffn.run(x, variant).cpu().numpy()
    gp, gs = ffn.hidden_codes(rows)
    gp, gs = gp.cpu().numpy(), gs.cpu().numpy()
    ffn.close()
    x_np = x.to(torch.float32).cpu().numpy()
    oup = oracle.Nvfp4Weight(up.packed.cpu().numpy(), up.block_scales.cpu().numpy(), up.tensor_scale)
    odn = oracle.Nvfp4Weight(down.packed.cpu().numpy(), down.block_scales.cpu().numpy(),
                             down.tensor_scale)
    # the oracle as it is, and with the device's intermediate bytes adopted where they are
    # rounding ties (the only admissible difference)
    raw = oracle.expert_ffn_forward(x_np, oup, odn)
    tied = oracle.expert_ffn_forward(x_np, oup, odn, candidates=(gp, gs),
                                     override_limit=helpers.OVERRIDE_LIMIT)
    raw_max_abs, raw_cosine = helpers.max_abs_and_cosine(out, raw.out)
    max_abs, cosine = helpers.max_abs_and_cosine(out, tied.out)
    over = np.abs(out.astype(np.float64) - raw.out).max(axis=1) > helpers.MAX_ABS_TOL
    return dict(max_abs=max_abs, cosine=cosine, raw_max_abs=raw_max_abs, raw_cosine=raw_cosine,
                code_mismatch=helpers.nibble_mismatches(gp, raw.hid_packed),
                scale_mismatch=int(np.count_nonzero(gs != raw.hid_scales)),
                adopted=tied.adopted_codes + tied.adopted_scales,
                inadmissible=tied.inadmissible_codes + tied.inadmissible_scales,
                tie_distance=tied.max_noise_units,
                rows_over_tol_without_tie=int(np.count_nonzero(over & ~tied.adopted_row)),
                total_codes=int(gp.size * 2))


def _check(r):
    # the stated gate (max-abs 2e-2, cosine 0.9995) against the oracle with admissible ties
    # adopted; nothing but ties may differ, ties are rare and within accumulation noise,
    # and against the oracle as it is only rows that own a tie may exceed the tolerance
    assert r["inadmissible"] == 0
    assert r["adopted"] == r["code_mismatch"] + r["scale_mismatch"]
    assert r["adopted"] <= max(4, int(helpers.ADOPTED_FRACTION_MAX * r["total_codes"]))
    assert r["tie_distance"] <= helpers.OVERRIDE_LIMIT
    assert r["max_abs"] <= 1e-3 <= helpers.MAX_ABS_TOL  # accumulation-order noise only
    assert r["cosine"] >= helpers.COSINE_TOL and r["raw_cosine"] >= helpers.COSINE_TOL
    assert r["rows_over_tol_without_tie"] == 0


@pytest.mark.parametrize("rows,variant", [(64, 0), (64, 1), (64, 3), (20, 2), (130, 3), (300, 1),
                                          (300, 0), (64, 4), (130, 4), (300, 4), (700, 4)])
def test_single_expert_ffn_baseline_shape(package, oracle, synthetic, rows, variant):
    r = _run_case(package, oracle, synthetic, rows, 2688, 1856, variant)
    print(rows, variant, r)
    _check(r)


@pytest.mark.parametrize("hidden,inter", [(64, 64), (256, 128), (512, 1024)])
def test_single_expert_ffn_small_shapes(package, oracle, synthetic, hidden, inter):
    for rows, variant in [(3, 1), (3, 2), (40, 1), (40, 3), (40, 4), (300, 4)]:
        r = _run_case(package, oracle, synthetic, rows, hidden, inter, variant, seed=hidden)
        print(hidden, inter, rows, variant, r)
        _check(r)


# 64 columns are stored together: weight tiles of 208 columns that start inside such a group and end in
# one (832 = 4 tiles), last tiles of 16 to 192 columns, one row and the rows around a tile's edge
@pytest.mark.parametrize("hidden,inter", [(832, 448), (448, 832), (1088, 192)])
def test_ffn_where_tiles_end(package, oracle, synthetic, hidden, inter):
    for rows, variant in [(1, 1), (129, 1), (255, 4), (16, 3), (17, 3), (129, 3)]:
        _check(_run_case(package, oracle, synthetic, rows, hidden, inter, variant, seed=inter))


@pytest.mark.parametrize("variant", [1, 3])
def test_ffn_rows_on_a_16_byte_boundary(package, synthetic, variant):
    # whole sectors are stored only to rows that start on one
    up, down = synthetic.make_ffn_weights(448, 192, seed=5, device="cuda")
    x = synthetic.make_tokens(70, 448, seed=6, device="cuda")
    ffn = package.ExpertFfn(up, down, max_rows=128)
    expected = ffn.run(x, variant)
    room = torch.zeros(70 * 448 + 8, device="cuda")
    lib, stream = package.load_library(), torch.cuda.current_stream().cuda_stream
    assert lib.nmoe_ffn_run(ffn._handle, stream, x.data_ptr(), package._dtype_code(x), 70,
                            room[4:].data_ptr(), variant) == 0
    assert lib.nmoe_ffn_sync_status(ffn._handle, stream) == 0
    assert torch.equal(room[4:-4].view(70, 448), expected)
    assert not room[:4].any() and not room[-4:].any()
    ffn.close()


@pytest.mark.parametrize("variants", [(3, 3), (1, 3), (3, 1)])
def test_ffn_status_is_that_of_the_runs_since_the_last_one(package, synthetic, variants):
    # rows beyond 6 * 448 are reported once, whichever kernel found them and whichever ran after it
    up, down = synthetic.make_ffn_weights(448, 192, seed=5, device="cuda")
    ffn = package.ExpertFfn(up, down, max_rows=128)
    up.tensor_scale *= 400.0
    beyond = package.ExpertFfn(up, down, max_rows=128)
    x = synthetic.make_tokens(40, 448, seed=6, device="cuda")
    out = torch.empty(40, 448, device="cuda")
    lib, stream = package.load_library(), package._stream()
    for f, expected in ((beyond, 5), (ffn, package.NMOE_OK)):  # (5: NMOE_ERR_ACTIVATION_RANGE)
        for _ in range(2):
            for variant in variants:
                assert lib.nmoe_ffn_run(f._handle, stream, x.data_ptr(), package._dtype_code(x), 40,
                                        out.data_ptr(), variant) == 0
            assert lib.nmoe_ffn_sync_status(f._handle, stream) == expected
        assert lib.nmoe_ffn_sync_status(f._handle, stream) == package.NMOE_OK
        f.close()


@pytest.mark.parametrize("captured", [1, 3])
def test_ffn_status_is_that_of_a_replayed_run(package, synthetic, captured):
    # what ran last is a graph of the caller's, not the run that was launched last
    up, down = synthetic.make_ffn_weights(448, 192, seed=5, device="cuda")
    up.tensor_scale *= 400.0
    ffn = package.ExpertFfn(up, down, max_rows=128)
    ordinary = synthetic.make_tokens(40, 448, seed=6, device="cuda") * 0.01
    x = ordinary.clone()
    out = torch.empty(40, 448, device="cuda")
    lib, stream = package.load_library(), torch.cuda.Stream()

    def launch(rows, variant):
        return lib.nmoe_ffn_run(ffn._handle, stream.cuda_stream, rows.data_ptr(),
                                package._dtype_code(rows), 40, out.data_ptr(), variant)

    def status():
        return lib.nmoe_ffn_sync_status(ffn._handle, stream.cuda_stream)

    torch.cuda.synchronize()
    assert launch(x, captured) == 0 and status() == 0  # (its kernels are loaded)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        assert launch(x, captured) == 0
    x.mul_(100.0)  # beyond 6 * 448 from here on
    torch.cuda.synchronize()
    for variant in (3, 1, 3):
        assert launch(ordinary, variant) == 0
        with torch.cuda.stream(stream):
            graph.replay()
        assert status() == 5  # NMOE_ERR_ACTIVATION_RANGE
        assert launch(ordinary, variant) == 0
        assert status() == 0
    ffn.close()
