"""GPU parity of the tensor-memory (tcgen05) GEMM against the CPU oracle."""

from __future__ import annotations

import threading

import numpy as np
import pytest
import torch

from alignquant_b200 import _lib
from alignquant_b200.quantization.exact import metadata_stack
from alignquant_b200.synthetic import synthetic_module_tensors
from oracle import alignquant_oracle as oc
from tests import helpers

pytestmark = pytest.mark.gpu

REL, ABS = 1e-3, 1e-2


@pytest.fixture(scope="module")
def ext():
    from alignquant_b200.kernels.cuda import extension

    extension.load_extension()
    return extension


@pytest.fixture()
def options(ext):
    """Library options are process-wide: put the defaults back after the test."""
    yield ext
    ext.set_gemm_tile("auto")
    ext.set_gemm_split(0)
    ext.set_gemm_rounding(False)


def _case(ext, m, n, k, scale_mode, seed, fraction=0.6, act_dtype=torch.bfloat16):
    n_j, n_k = n // 64, k // 64
    packed, states, tiles, scales = oc.synthetic_layer(n, k, seed=seed, w4_fraction=fraction)
    weights, _ = helpers.prepare_layer(packed, n_k)
    x = oc.synthetic_activation(m, k, seed=seed + 1, dtype="bfloat16" if act_dtype == torch.bfloat16 else np.float16)
    xt = helpers.torch_activation(x, act_dtype)
    xq, a_s = ext.alignquant_activation_quantize_cuda(xt, None, scale_mode=scale_mode)
    if scale_mode == "token":
        a_mk = oc.expand_act_scales(a_s.cpu().numpy(), m, n_k, "token")
    else:
        a_mk = np.repeat(a_s.cpu().numpy().reshape(-1, n_k), 16, axis=0)[:m]
    return weights, tiles, scales, xq, a_s, a_mk


@pytest.mark.parametrize("scale_mode", ["tile", "token"])
@pytest.mark.parametrize("m", [2, 64, 128, 130, 300])
@pytest.mark.parametrize("n,k", [(64, 64), (192, 192), (256, 1024), (320, 128)])
def test_gemm_matches_oracle(ext, n, k, m, scale_mode):
    n_j, n_k = n // 64, k // 64
    weights, tiles, scales, xq, a_s, a_mk = _case(ext, m, n, k, scale_mode, seed=n + k + m)
    dump = torch.full((m, n_j, n_k, 64), -7, dtype=torch.int32, device="cuda")
    out = ext.alignquant_linear_prepared(xq, a_s, weights, None, schedule="forced_prefill_m64",
                                         scale_mode=scale_mode, acc_dump=dump)
    ext.device_status()
    xq_np = xq.cpu().numpy()
    assert np.array_equal(dump.cpu().numpy(), oc.tile_accumulators_c(xq_np, tiles)), "int32 tile accumulators differ"
    got = out.cpu().numpy()
    want = helpers.planned_fp32(ext, xq_np, a_mk, tiles, scales, m, n_j, n_k, schedule="forced_prefill_m64")
    assert np.array_equal(got, want), "fp32 not in the planned operation order"
    assert np.allclose(got, oc.dequant_matmul_fp64(xq_np, a_mk, tiles, scales), rtol=REL, atol=ABS)


@pytest.mark.parametrize("tile", ["paired", "narrow", "wide"])
@pytest.mark.parametrize("m,n,k", [(130, 192, 192), (300, 320, 1024)])
def test_gemm_separate_rounding_is_the_reference_order(options, tile, m, n, k):
    """AQ_GEMM_ROUNDING_SEPARATE: multiply and add rounded separately, K tiles in increasing order."""
    ext = options
    ext.set_gemm_rounding(True)
    ext.set_gemm_tile(tile)
    n_j, n_k = n // 64, k // 64
    weights, tiles, scales, xq, a_s, a_mk = _case(ext, m, n, k, "tile", seed=n + k + m)
    out = ext.alignquant_linear_prepared(xq, a_s, weights, None, schedule="forced_prefill_m64")
    ext.device_status()
    splits = ext.linear_plan(m, n_j, n_k, schedule="forced_prefill_m64")["splits"]
    want = oc.linear_fp32_c(xq.cpu().numpy(), a_mk, tiles, scales, splits)
    assert np.array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("fraction", [0.0, 1.0])
def test_gemm_uniform_precision_layers(ext, fraction):
    m, n, k = 256, 256, 256
    weights, tiles, scales, xq, a_s, a_mk = _case(ext, m, n, k, "token", seed=3, fraction=fraction)
    out = ext.alignquant_linear_prepared(xq, a_s, weights, None, schedule="forced_prefill_m64", scale_mode="token")
    ext.device_status()
    want = helpers.planned_fp32(ext, xq.cpu().numpy(), a_mk, tiles, scales, m, n // 64, k // 64, schedule="forced_prefill_m64")
    assert np.array_equal(out.cpu().numpy(), want)


def test_gemm_auto_schedule_bf16_output_and_bounds(ext):
    m, n, k = 200, 384, 512
    weights, tiles, scales, xq, a_s, a_mk = _case(ext, m, n, k, "token", seed=21)
    canvas = torch.full((m + 2, n), 77.0, dtype=torch.bfloat16, device="cuda")
    out = ext.alignquant_linear_prepared(xq, a_s, weights, None, scale_mode="token",
                                         output_dtype=torch.bfloat16, out=canvas[1 : m + 1])
    ext.device_status()
    assert bool((canvas[0] == 77.0).all()) and bool((canvas[m + 1] == 77.0).all())
    want = torch.from_numpy(helpers.planned_fp32(ext, xq.cpu().numpy(), a_mk, tiles, scales, m, n // 64, k // 64)).to(torch.bfloat16)
    assert torch.equal(out.cpu(), want)


def test_gemm_reference_fixture_with_output_transform(ext, golden_dir):
    g = dict(np.load(golden_dir / "linear_transformed.npz"))
    m, k = g["x"].shape
    n_j, n_k = g["states"].shape
    packed = {key[len("packed_"):]: v for key, v in g.items() if key.startswith("packed_")}
    weights, _ = helpers.prepare_layer(packed, n_k)
    xq = torch.from_numpy(g["xq"]).cuda()
    a_s = torch.from_numpy(np.ascontiguousarray(g["act_scales"])).cuda()
    u_meta = torch.from_numpy(g["u_metadata"]).cuda()
    dump = torch.zeros((m, n_j, n_k, 64), dtype=torch.int32, device="cuda")
    out = ext.alignquant_linear_prepared(xq, a_s, weights, u_meta, schedule="forced_prefill_m64", acc_dump=dump)
    ext.device_status()
    assert np.array_equal(dump.cpu().numpy(), g["acc"])
    assert np.allclose(out.cpu().numpy(), g["y"], rtol=REL, atol=ABS)


def test_gemm_agrees_with_streaming_kernel_bit_for_bit(options):
    ext = options
    ext.set_gemm_rounding(True)  # the streaming kernel rounds multiply and add separately
    m, n, k = 96, 256, 384
    weights, tiles, scales, xq, a_s, a_mk = _case(ext, m, n, k, "tile", seed=8)
    splits = ext.linear_plan(m, n // 64, k // 64, schedule="forced_prefill_m64")["splits"]
    a = ext.alignquant_linear_prepared(xq, a_s, weights, None, schedule="forced_prefill_m64")
    b = ext.alignquant_linear_prepared(xq, a_s, weights, None, schedule="forced_prefill",
                                       decode_splits=splits if splits in (1, 2, 4, 8) else 1)
    if splits not in (1, 2, 4, 8):
        pytest.skip(f"the GEMM chose {splits} K ranges, which the streaming kernel cannot be forced to")
    ext.device_status()
    assert torch.equal(a, b)


@pytest.mark.parametrize("tile", ["paired", "narrow", "wide"])
def test_gemm_all_cta_tiles(options, tile):
    """The three CTA tiles give the same bits (K long enough to wrap the stage ring)."""
    ext = options
    ext.set_gemm_tile(tile)
    m, n, k = 260, 448, 1280
    weights, tiles, scales, xq, a_s, a_mk = _case(ext, m, n, k, "tile", seed=31)
    dump = torch.zeros((m, n // 64, k // 64, 64), dtype=torch.int32, device="cuda")
    out = ext.alignquant_linear_prepared(xq, a_s, weights, None, schedule="forced_prefill_m64", acc_dump=dump)
    plain = ext.alignquant_linear_prepared(xq, a_s, weights, None, schedule="forced_prefill_m64")
    ext.device_status()
    xq_np = xq.cpu().numpy()
    assert np.array_equal(dump.cpu().numpy(), oc.tile_accumulators_c(xq_np, tiles))
    want = helpers.planned_fp32(ext, xq_np, a_mk, tiles, scales, m, n // 64, k // 64, schedule="forced_prefill_m64")
    assert np.array_equal(out.cpu().numpy(), want)
    assert np.array_equal(plain.cpu().numpy(), want)


@pytest.mark.parametrize("tile", ["paired", "narrow", "wide", "auto"])
@pytest.mark.parametrize("split", ["2", "3", "8"])
@pytest.mark.parametrize("m", [40, 128, 200])
def test_gemm_split_k_clusters(options, m, split, tile):
    """K ranges over a thread-block cluster, with every tile width and (automatic width, up to 128 rows) the kernel for few
    rows: integer sums exact, FP32 in split order, output transform applied to those sums."""
    ext = options
    ext.set_gemm_split(int(split))
    ext.set_gemm_tile(tile)
    n, k = 320, 2048
    weights, tiles, scales, xq, a_s, a_mk = _case(ext, m, n, k, "tile", seed=77 + m)
    n_j, n_k = n // 64, k // 64
    plan = ext.linear_plan(m, n_j, n_k, schedule="forced_prefill_m64")
    assert plan["kernel"] == 1 and plan["splits"] == int(split)
    dump = torch.zeros((m, n_j, n_k, 64), dtype=torch.int32, device="cuda")
    out = ext.alignquant_linear_prepared(xq, a_s, weights, None, schedule="forced_prefill_m64", acc_dump=dump)
    ext.device_status()
    xq_np = xq.cpu().numpy()
    assert np.array_equal(dump.cpu().numpy(), oc.tile_accumulators_c(xq_np, tiles))
    sums = oc.linear_fp32_c(xq_np, a_mk, tiles, scales, int(split), fused=True)
    assert np.array_equal(out.cpu().numpy(), sums)
    u = metadata_stack([-1 if i % 3 == 1 else i + 1 for i in range(n_j)], "cuda")
    turned = ext.alignquant_linear_prepared(xq, a_s, weights, u, schedule="forced_prefill_m64")
    ext.device_status()
    exact = oc.inverse_output(sums, u.cpu().numpy())  # another order of the FP64 additions: the FP32 results are those or their neighbours
    assert np.allclose(turned.cpu().numpy(), exact, rtol=2.0**-23, atol=2.0**-45 * np.abs(sums).max())


@pytest.mark.parametrize("tile", ["paired", "narrow", "wide", "auto"])
@pytest.mark.parametrize("m,n,k", [(1190, 2368, 192), (33, 2624, 32768), (1999, 1088, 64)])
def test_gemm_many_tiles_per_cta_and_column_passes(options, tile, m, n, k):
    """More output tiles than SMs (a CTA walks several, with an odd number of K steps and ragged last
    row and column blocks), the longest K and a single K step; every result type through the tensor-map stores.  FP32 sums are
    compared bit for bit, the 16-bit results with their rounding of them."""
    ext = options
    ext.set_gemm_tile(tile)
    ext.set_gemm_split(1)
    weights, tiles, scales, xq, a_s, a_mk = _case(ext, m, n, k, "token", seed=m + n)
    xq_np = xq.cpu().numpy()
    want = torch.from_numpy(oc.linear_fp32_c(xq_np, a_mk, tiles, scales, 1, fused=True))
    for dtype in (torch.float32, torch.bfloat16, torch.float16):
        out = ext.alignquant_linear_prepared(xq, a_s, weights, None, schedule="forced_prefill_m64", scale_mode="token",
                                             output_dtype=dtype)
        ext.device_status()
        assert torch.equal(out.cpu(), want.to(dtype))


@pytest.mark.parametrize("scale_mode", ["tile", "token"])
@pytest.mark.parametrize("m", [2, 17, 32, 33, 64, 65, 100, 128])
@pytest.mark.parametrize("n,k,split", [(64, 64, 1), (192, 320, 1), (320, 1088, 3), (448, 2176, 8), (640, 4096, 0)])
def test_gemm_of_few_rows_has_the_bits_of_the_other_gemm(options, scale_mode, m, n, k, split):
    """Up to 128 rows: every row width, an odd number of tile rows, stages that are not full and K ranges of
    unequal length, against the kernel for many rows with the same K ranges; integer sums against the oracle."""
    ext = options
    ext.set_gemm_split(split)
    weights, tiles, _, xq, a_s, _ = _case(ext, m, n, k, scale_mode, seed=m + n + k)
    n_j, n_k = n // 64, k // 64
    u = metadata_stack([-1 if i % 3 == 1 else i + 1 for i in range(n_j)], "cuda")
    ranges = ext.linear_plan(m, n_j, n_k, schedule="forced_prefill_m64")["splits"]
    dump = torch.full((m, n_j, n_k, 64), -7, dtype=torch.int32, device="cuda")
    got = [ext.alignquant_linear_prepared(xq, a_s, weights, meta, schedule="forced_prefill_m64", scale_mode=scale_mode,
                                          output_dtype=dtype, acc_dump=d)
           for meta, dtype, d in ((None, torch.float32, dump), (None, torch.bfloat16, None), (u, torch.float16, None))]
    ext.device_status()
    assert np.array_equal(dump.cpu().numpy(), oc.tile_accumulators_c(xq.cpu().numpy(), tiles))
    ext.set_gemm_tile("wide")
    ext.set_gemm_split(ranges)
    for have, (meta, dtype) in zip(got, ((None, torch.float32), (None, torch.bfloat16), (u, torch.float16))):
        want = ext.alignquant_linear_prepared(xq, a_s, weights, meta, schedule="forced_prefill_m64", scale_mode=scale_mode,
                                              output_dtype=dtype)
        assert torch.equal(have, want)
    ext.device_status()


def test_captured_gemms_do_not_share_scratch(ext):
    """Two graphs captured one after the other (torch captures both on one stream) and replayed at the
    same time on two streams: each has its own expanded weights."""
    cases = [_case(ext, 256, 1024, 1024, "token", seed=s) for s in (5, 6)]
    graphs, results, wants = [], [], []
    for weights, _, _, xq, a_s, _ in cases:
        wants.append(ext.alignquant_linear_prepared(xq, a_s, weights, None, scale_mode="token"))
        torch.cuda.synchronize()
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1]):
            results.append(ext.alignquant_linear_prepared(xq, a_s, weights, None, scale_mode="token"))
    streams = [torch.cuda.Stream() for _ in graphs]
    for _ in range(20):
        for graph, stream in zip(graphs, streams):
            with torch.cuda.stream(stream):
                graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(have, want) for have, want in zip(results, wants))


def test_options_set_by_another_thread_meet_whole_calls(options):
    """A call is planned once: with an option changing all the time, each call without a workspace runs the
    kernel that needs none or is refused, and never launches what its workspace was not checked for."""
    ext = options
    ext.set_gemm_split(1)
    m, n, k = 100, 640, 1024
    weights, _, _, xq, a_s, _ = _case(ext, m, n, k, "token", seed=12)
    want = ext.alignquant_linear_prepared(xq, a_s, weights, None, scale_mode="token")
    lib, stop = _lib.load(), threading.Event()

    def toggle():
        while not stop.is_set():
            for tile in (_lib.GEMM_TILES["wide"], _lib.GEMM_TILES["auto"]):
                lib.aq_set_option(_lib.AQ_OPT_GEMM_TILE, tile)

    thread = threading.Thread(target=toggle)
    thread.start()
    try:
        seen = {0: 0, -3: 0}
        for _ in range(2000):
            out = torch.zeros_like(want)
            status = lib.aq_linear(xq.data_ptr(), a_s.data_ptr(), _lib.AQ_SCALE_TOKEN, m, weights.image.data_ptr(), n // 64, k // 64,
                                   None, 0, 0, _lib.AQ_F32, out.data_ptr(), None, 0, None, torch.cuda.current_stream().cuda_stream)
            seen[status] += 1  # 0, or AQ_ERR_WORKSPACE
            assert status != 0 or torch.equal(out, want)
    finally:
        stop.set()
        thread.join()
    ext.device_status()
    assert seen[0] > 0


@pytest.mark.parametrize("tile", ["paired", "narrow", "wide", "auto"])
@pytest.mark.parametrize("transforms", [False, True])
@pytest.mark.parametrize("m,n,k", [(1190, 2368, 192), (700, 16448, 32768 // 4), (2100, 640, 320)])
def test_gemm_many_tiles_per_cta_under_tile_scales(options, tile, transforms, m, n, k):
    """Tile scales, transformed and plain tile rows mixed in one CTA, integer sums and every result type while a CTA walks
    several output tiles (ragged last ones), against calls of 64 rows, which the kernel for few rows answers; the second
    shape has more output tiles than SMs with every width."""
    ext = options
    n_j, n_k = n // 64, k // 64
    t = synthetic_module_tensors(n, k, m)
    weights = ext.prepare_weights(*(t[name] for name in ("state_bits", "w4_payload", "w4_scales", "w8_payload", "w8_scales",
                                                         "w4_row_offsets", "w8_row_offsets")), n_k=n_k)
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    x = torch.randn(m, k, generator=gen, device="cuda").to(torch.bfloat16)
    xq, a_s = ext.alignquant_activation_quantize_cuda(x, None, scale_mode="tile")
    u = metadata_stack([-1 if i % 3 == 1 else i + 1 for i in range(n_j)], "cuda") if transforms else None
    ext.set_gemm_split(1)
    few = dict(schedule="forced_prefill_m64", scale_mode="tile")
    dumps = m * n_j * n_k < 1 << 21
    for dtype in (torch.float32, torch.bfloat16, torch.float16):
        ext.set_gemm_tile("auto")
        want, sums = [], []
        for row in range(0, m, 64):
            rows = xq[row : row + 64]
            part = torch.empty((rows.size(0), n_j, n_k, 64), dtype=torch.int32, device="cuda") if dumps else None
            scales = a_s.reshape(-1, n_k)[row // 16 : (row + rows.size(0) + 15) // 16].contiguous()
            want.append(ext.alignquant_linear_prepared(rows, scales, weights, u, output_dtype=dtype, acc_dump=part, **few))
            sums.append(part)
        ext.set_gemm_tile(tile)
        dump = torch.empty((m, n_j, n_k, 64), dtype=torch.int32, device="cuda") if dumps else None
        have = ext.alignquant_linear_prepared(xq, a_s, weights, u, output_dtype=dtype, acc_dump=dump, **few)
        ext.device_status()
        assert torch.equal(have, torch.cat(want))
        assert not dumps or torch.equal(dump, torch.cat(sums))


def test_gemm_transforms_in_several_column_passes(options):
    """A layer above the scratch: the second pass transforms with the metadata of its own tile rows."""
    ext = options
    n, k, m = 34816, 8192, 160
    n_j, n_k = n // 64, k // 64
    assert n_j * n_k * 4096 > 256 << 20
    t = synthetic_module_tensors(n, k, 1)
    weights = ext.prepare_weights(*(t[name] for name in ("state_bits", "w4_payload", "w4_scales", "w8_payload", "w8_scales",
                                                         "w4_row_offsets", "w8_row_offsets")), n_k=n_k)
    x = torch.randn(m, k, generator=torch.Generator(device="cuda").manual_seed(2), device="cuda").to(torch.bfloat16)
    xq, a_s = ext.alignquant_activation_quantize_cuda(x, None, scale_mode="token")
    ext.set_gemm_split(1)
    for u in (None, metadata_stack([-1 if i % 3 == 1 else i + 1 for i in range(n_j)], "cuda")):
        have = ext.alignquant_linear_prepared(xq, a_s, weights, u, scale_mode="token", output_dtype=torch.bfloat16)
        want = [ext.alignquant_linear_prepared(xq[row : row + 64], a_s[row : row + 64], weights, u, scale_mode="token",
                                               schedule="forced_prefill_m64", output_dtype=torch.bfloat16) for row in range(0, m, 64)]
        assert torch.equal(have, torch.cat(want))
    ext.device_status()
