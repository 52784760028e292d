"""The tcgen05 / TMEM path (TF32 and BF16 operands, fp32 accumulate) through the C ABI.

Two checks per case: (1) against the CPU model of exactly that computation (fp32 transforms,
operands rounded once, exact contraction) with a tight tolerance, which catches layout and
indexing errors; (2) against the fp64 direct convolution with the tolerance the arithmetic
allows, which is the accuracy claim of the path.  Inputs and filters are themselves rounded to
the operand type first (the tensor-core benchmark configuration prescribes operands rounded once
from the seeded fp32 tensors)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from opencnn_b200 import api  # noqa: E402

pytestmark = pytest.mark.gpu

# These small maps are one round of tiles: the deep ones take the CTA-pair kernel in both types, also with an odd number of 32-image
# blocks, with K not a multiple of 128 and with 64 filters, the others the single-CTA kernel.  (test_dispatch_cpu.py checks what the
# comments here say of the automatic choice.)
SHAPES = [(32, 16, 128, 8, 8), (32, 8, 64, 7, 7), (64, 40, 192, 5, 9), (32, 64, 64, 14, 14), (96, 32, 256, 6, 6),
          (64, 512, 128, 4, 4), (96, 512, 192, 3, 5), (128, 520, 64, 2, 2), (64, 1024, 128, 3, 3), (96, 1040, 192, 2, 3)]
MODEL_REL = 2e-4                     # device vs model: fp32 accumulation order inside the tensor core
TRUTH_REL = {"tf32": 4e-3, "bf16": 3e-2}   # device vs fp64 truth, relative to rms(truth)


def run_tc(x, g, precision):
    C, H, W, N = x.shape
    K = g.shape[3]
    dx, dg = torch.from_numpy(x).cuda(), torch.from_numpy(g).cuda()
    dy = torch.full((K, H, W, N), float("nan"), device="cuda")
    dws = torch.empty((C, 4, 4, K), device="cuda")
    err = api.conv3x3(dx, dg, dy, dws, N, C, H, W, K, precision=precision,
                      stream=torch.cuda.current_stream().cuda_stream)
    assert err == 0, f"cudaError {err}"
    assert api.last_device_status() == 0
    return dy.cpu().numpy()


@pytest.mark.parametrize("precision", ["tf32", "bf16"])
@pytest.mark.parametrize("shape", SHAPES)
def test_tensor_core_path(oracle, libs, precision, shape):
    N, C, K, H, W = shape
    rnd = oracle.round_tf32 if precision == "tf32" else oracle.round_bf16
    x = rnd(oracle.input_chwn(N, C, H, W)).reshape(C, H, W, N)
    g = rnd(oracle.filter_crsk(C, K)).reshape(C, 3, 3, K)
    y = run_tc(x, g, precision)
    assert np.isfinite(y).all()
    model = oracle.tc_model(x, g, precision)
    rms = float(np.sqrt(np.mean(model.astype(np.float64) ** 2)))
    worst = float(np.abs(y - model).max())
    assert worst <= MODEL_REL * max(rms, 1e-30), f"vs model: {worst / rms:.3e} of rms"
    truth = oracle.direct_f64(x, g)
    trms = float(np.sqrt(np.mean(truth ** 2)))
    tworst = float(np.abs(y - truth).max())
    assert tworst <= TRUTH_REL[precision] * trms, f"vs fp64: {tworst / trms:.3e} of rms"


# Ragged last image block (N % 8 == 0 on this path), single-CTA kernel and (C >= 512) CTA-pair kernel.
RAGGED = [(40, 16, 128, 6, 6), (72, 32, 64, 5, 7), (8, 16, 128, 4, 4), (72, 512, 128, 4, 4), (104, 512, 128, 3, 3),
          (72, 1024, 128, 2, 2),
          (32, 3, 64, 6, 6), (40, 21, 128, 5, 5), (64, 515, 128, 3, 3)]   # and channel counts that are not a multiple of 8


@pytest.mark.parametrize("precision", ["tf32", "bf16"])
@pytest.mark.parametrize("shape", RAGGED)
def test_ragged_batch_on_tensor_cores(oracle, libs, precision, shape):
    N, C, K, H, W = shape
    rnd = oracle.round_tf32 if precision == "tf32" else oracle.round_bf16
    x = rnd(oracle.input_chwn(N, C, H, W)).reshape(C, H, W, N)
    g = rnd(oracle.filter_crsk(C, K)).reshape(C, 3, 3, K)
    y = run_tc(x, g, precision)
    assert np.isfinite(y).all()
    model = oracle.tc_model(x, g, precision)
    rms = float(np.sqrt(np.mean(model.astype(np.float64) ** 2)))
    worst = float(np.abs(y - model).max())
    assert worst <= MODEL_REL * max(rms, 1e-30), f"vs model: {worst / rms:.3e} of rms"
    dx = torch.zeros((C, H, W, N + 4), device="cuda")
    assert api.conv3x3(dx, torch.from_numpy(g).cuda(), torch.empty((K, H, W, N + 4), device="cuda"),
                       torch.empty((C, 4, 4, K), device="cuda"), N + 4, C, H, W, K, precision=precision) != 0, \
        "N % 8 != 0 must be refused on the tensor-core path"


@pytest.mark.parametrize("precision", ["tf32", "bf16"])
def test_integer_tensors_are_exact_on_tensor_cores(oracle, libs, precision):
    """Small integers are exact in both operand types and in the fp32 accumulator."""
    N, C, K, H, W = 32, 16, 128, 6, 6
    x, g = oracle.input_int(N, C, H, W), oracle.filter_int(C, K)
    y = run_tc(x, g, precision)
    assert np.array_equal(y.astype(np.float64), oracle.direct_f64(x, g))


@pytest.mark.parametrize("precision", ["tf32", "bf16"])
def test_tensor_core_results_are_repeatable(libs, precision):
    """Same bits run after run, from the single-CTA kernel (the first size) and the CTA-pair kernel (the other)."""
    for (N, C, K, H, W) in [(64, 64, 64, 9, 9), (64, 1024, 128, 3, 3)]:
        x = torch.rand((C, H, W, N), device="cuda") * 2 - 1
        g = torch.randn((C, 3, 3, K), device="cuda") * 0.05
        ws = torch.empty((C, 4, 4, K), device="cuda")
        first = torch.empty((K, H, W, N), device="cuda")
        again = torch.empty_like(first)
        assert api.conv3x3(x, g, first, ws, N, C, H, W, K, precision=precision) == 0
        for _ in range(3):
            assert api.conv3x3(x, g, again, ws, N, C, H, W, K, precision=precision) == 0
            torch.cuda.synchronize()
            assert torch.equal(first, again)
    assert api.last_device_status() == 0


# The benchmark shapes at full size (the N=128 layer sweep and the two wide stress layers): error of both
# operand types against 10^5 sampled fp64 outputs, relative to rms(truth).  All take the CTA-pair kernel but the
# two layers with 64 filters, which take the image-rows kernel.
FULL = [(128, 64, 64, 56), (128, 128, 128, 28), (128, 256, 256, 14), (128, 512, 512, 7), (64, 1024, 1024, 14),
        (256, 32, 64, 112)]


@pytest.mark.parametrize("precision", ["tf32", "bf16"])
@pytest.mark.parametrize("shape", FULL)
def test_tensor_core_error_at_benchmark_sizes(oracle, libs, precision, shape):
    N, C, K, HW = shape
    rnd = oracle.round_tf32 if precision == "tf32" else oracle.round_bf16
    x = rnd(oracle.input_chwn(N, C, HW, HW)).reshape(C, HW, HW, N)
    g = rnd(oracle.filter_crsk(C, K)).reshape(C, 3, 3, K)
    dx, dg = torch.from_numpy(x).cuda(), torch.from_numpy(g).cuda()
    dy = torch.full((K, HW, HW, N), float("nan"), device="cuda")
    dws = torch.empty((C, 4, 4, K), device="cuda")
    assert api.conv3x3(dx, dg, dy, dws, N, C, HW, HW, K, precision=precision) == 0
    assert api.last_device_status() == 0
    assert bool(torch.isfinite(dy).all().item()), "an output was not written"
    idx = np.random.default_rng(11).integers(0, dy.numel(), 100000)
    truth = oracle.direct_f64_sampled(x, g, idx)
    got = dy.view(-1)[torch.from_numpy(idx).cuda()].cpu().numpy()
    trms = float(np.sqrt(np.mean(truth ** 2)))
    worst = float(np.abs(got - truth).max())
    assert worst <= TRUTH_REL[precision] * trms, f"vs fp64: {worst / trms:.3e} of rms"
    # a second run gives the same bits
    dy2 = torch.empty_like(dy)
    assert api.conv3x3(dx, dg, dy2, dws, N, C, HW, HW, K, precision=precision) == 0
    torch.cuda.synchronize()
    assert torch.equal(dy, dy2)


# Every tensor-core kernel on its own, chosen by the caller (opencnn_winograd_forward_kernel), whatever the
# library's own rule would take: small and deep problems, an odd number of 32-image blocks, a ragged last block,
# K not a multiple of 128, channel counts that are not a multiple of the K-step.
KERNEL_SHAPES = [(32, 16, 128, 8, 8), (64, 40, 192, 5, 9), (96, 32, 256, 6, 6), (64, 512, 128, 4, 4), (128, 64, 64, 14, 14),
                 (72, 48, 64, 5, 7), (104, 515, 128, 3, 3), (8, 16, 128, 4, 4), (160, 24, 320, 7, 7)]


@pytest.mark.parametrize("kernel", ["single", "pair_local"])
@pytest.mark.parametrize("precision", ["tf32", "bf16"])
def test_each_tensor_core_kernel(oracle, libs, precision, kernel):
    rnd = oracle.round_tf32 if precision == "tf32" else oracle.round_bf16
    for (N, C, K, H, W) in KERNEL_SHAPES:
        x = rnd(oracle.input_chwn(N, C, H, W)).reshape(C, H, W, N)
        g = rnd(oracle.filter_crsk(C, K)).reshape(C, 3, 3, K)
        dx, dg = torch.from_numpy(x).cuda(), torch.from_numpy(g).cuda()
        dws = torch.empty((C, 4, 4, K), device="cuda")
        assert api.filter_transform(dg, dws, C, K, precision=precision) == 0
        outs = []
        for _ in range(2):
            dy = torch.full((K, H, W, N), float("nan"), device="cuda")
            assert api.winograd_forward_kernel(dx, dws, dy, N, C, H, W, K, precision=precision, kernel=kernel) == 0
            assert api.last_device_status() == 0, (kernel, precision, (N, C, K, H, W))
            outs.append(dy)
        assert torch.equal(outs[0], outs[1]), "not repeatable"
        y = outs[0].cpu().numpy()
        assert np.isfinite(y).all(), (kernel, precision, (N, C, K, H, W))
        model = oracle.tc_model(x, g, precision)
        rms = float(np.sqrt(np.mean(model.astype(np.float64) ** 2)))
        worst = float(np.abs(y - model).max())
        assert worst <= MODEL_REL * max(rms, 1e-30), f"{kernel} {precision} {(N, C, K, H, W)}: {worst / rms:.3e} of rms"
    bad = torch.zeros(16, device="cuda")
    assert api.winograd_forward_kernel(bad, bad, bad, 32, 8, 4, 4, 64, precision="fp32", kernel=kernel) != 0


# The stacked-blocks kernel (at most 64 filters): even and odd numbers of 32-image blocks, a ragged last block,
# channel counts that are not a multiple of the K-step, one K-step and many, more tiles than SMs (so that both
# stages of the filter ring are reused).
STACKED_SHAPES = [(64, 16, 64, 8, 8), (96, 40, 64, 5, 9), (128, 64, 64, 14, 14), (72, 3, 64, 6, 6), (32, 32, 64, 7, 7),
                  (200, 72, 64, 3, 5), (256, 32, 64, 12, 12), (256, 32, 64, 30, 30)]


@pytest.mark.parametrize("precision", ["tf32", "bf16"])
def test_stacked_blocks_kernel(oracle, libs, precision):
    rnd = oracle.round_tf32 if precision == "tf32" else oracle.round_bf16
    for (N, C, K, H, W) in STACKED_SHAPES:
        x = rnd(oracle.input_chwn(N, C, H, W)).reshape(C, H, W, N)
        g = rnd(oracle.filter_crsk(C, K)).reshape(C, 3, 3, K)
        dx, dg = torch.from_numpy(x).cuda(), torch.from_numpy(g).cuda()
        dws = torch.empty((C, 4, 4, K), device="cuda")
        assert api.filter_transform(dg, dws, C, K, precision=precision) == 0
        outs = []
        for _ in range(2):
            dy = torch.full((K, H, W, N), float("nan"), device="cuda")
            assert api.winograd_forward_kernel(dx, dws, dy, N, C, H, W, K, precision=precision, kernel="stacked") == 0
            assert api.last_device_status() == 0, (N, C, K, H, W)
            outs.append(dy)
        assert torch.equal(outs[0], outs[1]), "not repeatable"
        # the single-CTA kernel issues the same products in the same order: the two must agree bit for bit
        single = torch.full((K, H, W, N), float("nan"), device="cuda")
        assert api.winograd_forward_kernel(dx, dws, single, N, C, H, W, K, precision=precision, kernel="single") == 0
        assert torch.equal(outs[0], single), (N, C, K, H, W)
        y = outs[0].cpu().numpy()
        assert np.isfinite(y).all(), (N, C, K, H, W)
        model = oracle.tc_model(x, g, precision)
        rms = float(np.sqrt(np.mean(model.astype(np.float64) ** 2)))
        worst = float(np.abs(y - model).max())
        assert worst <= MODEL_REL * max(rms, 1e-30), f"{(N, C, K, H, W)}: {worst / rms:.3e} of rms"
    # refused: more than 64 filters
    z = torch.zeros(1 << 16, device="cuda")
    assert api.winograd_forward_kernel(z, z, z, 64, 16, 4, 4, 128, precision=precision, kernel="stacked") != 0


# The CTA-pair kernel against the single-CTA kernel, which issues the same products in the same order: one image block
# (the pair's second half is empty), an odd number of them, a pair that spans two tiles, a second CTA without filters,
# fewer K-steps than ring stages, more pairs than fit on the device at once.
PAIR_SHAPES = [(8, 16, 128, 2, 2), (32, 24, 128, 5, 5), (40, 3, 192, 3, 5), (96, 72, 64, 3, 3), (24, 100, 320, 9, 4),
               (160, 40, 192, 17, 23)]


@pytest.mark.parametrize("precision", ["tf32", "bf16"])
@pytest.mark.parametrize("shape", PAIR_SHAPES)
def test_pair_kernel_gives_the_bits_of_the_single_cta_kernel(libs, precision, shape):
    N, C, K, H, W = shape
    x = torch.rand((C, H, W, N), device="cuda") * 2 - 1
    ws = torch.empty((C, 4, 4, K), device="cuda")
    assert api.filter_transform(torch.randn((C, 3, 3, K), device="cuda") * 0.05, ws, C, K, precision=precision) == 0
    out = {}
    for kernel in ("single", "pair_local"):
        out[kernel] = torch.full((K, H, W, N), float("nan"), device="cuda")
        assert api.winograd_forward_kernel(x, ws, out[kernel], N, C, H, W, K, precision=precision, kernel=kernel) == 0
        assert api.last_device_status() == 0
    assert bool(torch.isfinite(out["single"]).all().item())
    assert torch.equal(out["single"], out["pair_local"])


# The kernel with the images in the accumulator rows, likewise: one block of columns (three quarters of the
# pair's tile empty), five, a tile that spans two output tiles, more filter blocks than one, fewer K-steps than ring stages, more
# tiles than pairs fit on the device at once.
IMAGE_ROWS_SHAPES = [(8, 16, 64, 2, 2), (32, 24, 128, 5, 5), (40, 3, 192, 3, 5), (96, 72, 64, 3, 3), (24, 100, 320, 9, 4), (160, 40, 64, 17, 23),
                     (64, 16, 64, 31, 30)]


@pytest.mark.parametrize("precision", ["tf32", "bf16"])
@pytest.mark.parametrize("shape", IMAGE_ROWS_SHAPES)
def test_image_rows_kernel_gives_the_bits_of_the_single_cta_kernel(libs, precision, shape):
    N, C, K, H, W = shape
    x = torch.rand((C, H, W, N), device="cuda") * 2 - 1
    ws = torch.empty((C, 4, 4, K), device="cuda")
    assert api.filter_transform(torch.randn((C, 3, 3, K), device="cuda") * 0.05, ws, C, K, precision=precision) == 0
    single, rows = (torch.full((K, H, W, N), float("nan"), device="cuda") for _ in range(2))
    assert api.winograd_forward_kernel(x, ws, single, N, C, H, W, K, precision=precision, kernel="single") == 0
    assert api.winograd_forward_kernel(x, ws, rows, N, C, H, W, K, precision=precision, kernel="image_rows") == 0
    assert api.last_device_status() == 0
    assert bool(torch.isfinite(single).all().item())
    assert torch.equal(single, rows)


# Batches that are not a multiple of 32 and whose blocks of columns the automatic choice packs (single-CTA kernel): the bits that the
# same images have in a batch filled up to a multiple of 32.  Blocks within one tile, across two and across four; odd maps.  The batches of 40 and
# more have blocks within a tile, which TMA loads, between others; of these (40, 20, 64, 35, 31), and in TF32 the others with 64 filters but
# (40, 3, 64, 13, 21), are another kernel's.
PACKED = [(8, 40, 128, 28, 28), (8, 3, 64, 57, 56), (16, 66, 192, 39, 38), (24, 64, 128, 28, 28), (40, 20, 64, 35, 31), (72, 24, 64, 33, 30),
          (40, 20, 192, 41, 37), (72, 8, 192, 35, 33), (104, 12, 192, 21, 27), (40, 24, 64, 41, 33), (104, 100, 64, 30, 30), (40, 3, 64, 13, 21)]


@pytest.mark.parametrize("precision", ["tf32", "bf16"])
@pytest.mark.parametrize("shape", PACKED)
def test_packed_columns_give_the_bits_of_a_full_batch(libs, precision, shape):
    N, C, K, H, W = shape
    full = (N + 31) // 32 * 32
    x = torch.zeros((C, H, W, full), device="cuda")
    x[..., :N] = torch.rand((C, H, W, N), device="cuda") * 2 - 1
    ws = torch.empty((C, 4, 4, K), device="cuda")
    assert api.filter_transform(torch.randn((C, 3, 3, K), device="cuda") * 0.05, ws, C, K, precision=precision) == 0
    expect = torch.empty((K, H, W, full), device="cuda")
    assert api.winograd_forward_kernel(x, ws, expect, full, C, H, W, K, precision=precision, kernel="single") == 0
    guard = 4096                                    # floats after the output that must stay untouched
    flat = torch.full((K * H * W * N + guard,), float("nan"), device="cuda")
    y = flat[:K * H * W * N].view(K, H, W, N)
    assert api.winograd_forward(x[..., :N].contiguous(), ws, y, N, C, H, W, K, precision=precision) == 0
    assert api.last_device_status() == 0
    assert torch.equal(y, expect[..., :N])
    assert bool(torch.isnan(flat[K * H * W * N:]).all())


# The fused kernel is launched so that its set-up overlaps the filter transform: back-to-back calls that reuse one
# workspace with other filters, and the same under stream capture, give what a transform waited for gives.  Every kernel of the
# automatic choice, the packed ones of both paths too.
ORDERED = [("fp32", (32, 16, 64, 9, 9)), ("fp32", (36, 5, 68, 6, 5)), ("bf16", (64, 16, 64, 30, 30)), ("bf16", (32, 256, 256, 6, 6)),
           ("tf32", (64, 64, 192, 7, 7)), ("tf32", (8, 3, 64, 4, 4)),
           ("fp32", (20, 64, 64, 31, 45)), ("fp32", (4, 20, 20, 49, 11)), ("bf16", (8, 64, 64, 27, 21)), ("bf16", (40, 20, 192, 41, 37)),
           ("tf32", (72, 20, 192, 17, 5)), ("bf16", (64, 16, 192, 25, 5)), ("tf32", (64, 64, 64, 21, 13)), ("tf32", (128, 8, 64, 5, 29)),
           ("bf16", (32, 64, 64, 6, 6))]


@pytest.mark.parametrize("precision,shape", ORDERED)
def test_transform_and_kernel_stay_ordered(libs, precision, shape):
    N, C, K, H, W = shape
    x = torch.rand((C, H, W, N), device="cuda") * 2 - 1
    filters = [torch.randn((C, 3, 3, K), device="cuda") * 0.05 for _ in range(4)]
    ws = torch.empty((C, 4, 4, K), device="cuda")
    expect = []
    for g in filters:
        y = torch.empty((K, H, W, N), device="cuda")
        assert api.filter_transform(g, ws, C, K, precision=precision) == 0
        torch.cuda.synchronize()
        assert api.winograd_forward(x, ws, y, N, C, H, W, K, precision=precision) == 0
        torch.cuda.synchronize()
        expect.append(y)
    got = [torch.full_like(y, float("nan")) for y in expect]
    stream = torch.cuda.Stream()

    def calls():
        for g, y in zip(filters, got):
            assert api.conv3x3(x, g, y, ws, N, C, H, W, K, precision=precision, stream=stream.cuda_stream) == 0

    torch.cuda.synchronize()
    calls()
    stream.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, expect))
    for y in got:
        y.fill_(float("nan"))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        calls()
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, expect))
    assert api.last_device_status() == 0


# An infinity or a NaN in the data must not come out as a number: the outputs that are not finite are those of the fp32 path,
# which does the same additions (no transformed filter value is zero here, and none overflows).  The NaNs include the bit
# patterns that rounding by integer addition would carry into the exponent or the sign.
@pytest.mark.parametrize("precision", ["tf32", "bf16"])
@pytest.mark.parametrize("bits", [0x7F800000, 0xFF800000, 0x7FC00000, 0x7FFFFFFF, 0xFFFFFFFF, 0x7F800001])
def test_nonfinite_values_are_not_lost(libs, precision, bits):
    N, C, K, H, W = 64, 24, 64, 7, 8
    x = torch.rand((C, H, W, N), device="cuda") * 2 - 1
    g = torch.randn((C, 3, 3, K), device="cuda") * 0.05
    for where in ("input", "filter"):
        xb, gb = x.clone(), g.clone()
        word = torch.tensor(bits - (1 << 32) if bits >= 1 << 31 else bits, dtype=torch.int32, device="cuda")
        if where == "input":
            xb.view(torch.int32)[3, 2, 5, 7] = word
        else:
            gb.view(torch.int32)[3, 0, 0, 9] = word          # the tap that the filter transform copies unchanged
        finite = {}
        for p in ("fp32", precision):
            ws = torch.empty((C, 4, 4, K), device="cuda")
            y = torch.zeros((K, H, W, N), device="cuda")
            assert api.conv3x3(xb, gb, y, ws, N, C, H, W, K, precision=p) == 0
            assert api.last_device_status() == 0
            finite[p] = torch.isfinite(y)
        assert not bool(finite["fp32"].all())
        assert torch.equal(finite["fp32"], finite[precision]), where


# Every image is a convolution of its own: an infinity or a NaN in one leaves the bits of all others as they are, whichever
# of a tile's two image blocks it sits in and whether the tile's other rows are another block's (K = 64, stacked), a
# repetition of the same filters (K = 64, single) or filters that do not exist (K = 192).  The automatic choice: stacked (image rows in TF32),
# CTA pair, packed columns twice, with more than 64 filters and with 64, and stacked.
CONTAINED = [("single", (64, 16, 64, 5, 6)), ("pair_local", (64, 24, 192, 5, 6)), ("stacked", (96, 24, 64, 5, 6)),
             ("image_rows", (96, 24, 64, 5, 6)), ("image_rows", (72, 24, 128, 5, 6)),
             ("auto", (64, 16, 64, 31, 30)), ("auto", (64, 40, 128, 31, 30)), ("auto", (72, 20, 192, 17, 5)), ("auto", (104, 8, 64, 15, 9)),
             ("auto", (128, 8, 64, 5, 29))]


@pytest.mark.parametrize("precision", ["tf32", "bf16"])
@pytest.mark.parametrize("kernel,shape", CONTAINED)
def test_nonfinite_values_stay_in_their_image(libs, precision, kernel, shape):
    N, C, K, H, W = shape
    x = torch.rand((C, H, W, N), device="cuda") * 2 - 1
    ws = torch.empty((C, 4, 4, K), device="cuda")
    assert api.filter_transform(torch.randn((C, 3, 3, K), device="cuda") * 0.05, ws, C, K, precision=precision) == 0

    def run(x):
        y = torch.zeros((K, H, W, N), device="cuda")
        assert api.winograd_forward_kernel(x, ws, y, N, C, H, W, K, precision=precision, kernel=kernel) == 0
        assert api.last_device_status() == 0
        return y

    clean = run(x)
    for image, value in [(5, float("inf")), (40, float("-inf")), (N - 1, float("nan"))]:
        bad = x.clone()
        bad[C - 2, 3, 2, image] = value
        y = run(bad)
        assert not bool(torch.isfinite(y[..., image]).all())
        others = [n for n in range(N) if n != image]
        assert torch.equal(y[..., others], clean[..., others]), (image, value)


# The automatic choice: the bits of the single-CTA kernel whatever it takes, which in each type is each of the kernels at some of these sizes.
CHOICES = [(32, 48, 128, 24, 12), (32, 128, 128, 24, 12), (64, 64, 192, 14, 20), (128, 16, 128, 41, 38), (128, 15, 256, 41, 39),
           (64, 64, 64, 16, 36), (64, 33, 64, 26, 26), (64, 33, 64, 30, 30), (200, 24, 64, 17, 23), (104, 100, 64, 30, 30), (160, 16, 64, 30, 30),
           (40, 400, 64, 30, 30), (8, 200, 64, 7, 5), (128, 8, 64, 5, 29), (24, 64, 128, 28, 28)]


@pytest.mark.parametrize("precision", ["tf32", "bf16"])
@pytest.mark.parametrize("shape", CHOICES)
def test_automatic_choice_gives_the_bits_of_the_single_cta_kernel(libs, precision, shape):
    N, C, K, H, W = shape
    x = torch.rand((C, H, W, N), device="cuda") * 2 - 1
    ws = torch.empty((C, 4, 4, K), device="cuda")
    assert api.filter_transform(torch.randn((C, 3, 3, K), device="cuda") * 0.05, ws, C, K, precision=precision) == 0
    out = {}
    for kernel in ("single", "auto"):
        out[kernel] = torch.full((K, H, W, N), float("nan"), device="cuda")
        assert api.winograd_forward_kernel(x, ws, out[kernel], N, C, H, W, K, precision=precision, kernel=kernel) == 0
        assert api.last_device_status() == 0
    assert bool(torch.isfinite(out["single"]).all().item())
    assert torch.equal(out["single"], out["auto"])


# The fused kernel reads its input before the transform it overlaps is over, so what it reads must be older than that
# transform: on one stream and without synchronisation the input buffer is rewritten before every call, and every call's
# output is the next one's input.  Sizes that reach each fused kernel, the packed ones too (those read the input with other instructions).
REWRITTEN = [("fp32", (32, 64, 64, 9, 9)), ("fp32", (36, 20, 20, 6, 5)), ("bf16", (32, 64, 64, 6, 6)), ("tf32", (40, 64, 64, 5, 5)),
             ("bf16", (64, 128, 128, 14, 20)), ("tf32", (72, 128, 128, 15, 20)), ("bf16", (64, 64, 64, 31, 30)), ("tf32", (56, 64, 64, 31, 30)),
             ("noalloc", (32, 64, 64, 9, 9)), ("fp32", (20, 64, 64, 31, 45)), ("fp32", (4, 20, 20, 49, 11)), ("bf16", (8, 64, 64, 27, 21)),
             ("bf16", (8, 128, 128, 28, 28)), ("tf32", (8, 64, 64, 21, 27)), ("bf16", (64, 64, 64, 29, 9)), ("noalloc", (20, 64, 64, 31, 45))]


@pytest.mark.parametrize("precision,shape", REWRITTEN)
def test_input_written_just_before_the_call(libs, precision, shape):
    N, C, K, H, W = shape
    sources = [torch.rand((C, H, W, N), device="cuda") * 2 - 1 for _ in range(4)]
    filters = [torch.randn((C, 3, 3, K), device="cuda") * 0.05 for _ in range(4)]
    x, ws = torch.empty((C, H, W, N), device="cuda"), torch.empty((C, 4, 4, K), device="cuda")
    stream = torch.cuda.Stream()

    def conv(x, g, y, wait):
        if precision == "noalloc":
            assert api.conv3x3_noalloc(x, g, y, N, C, H, W, K, stream=stream.cuda_stream) == 0
        else:
            assert api.conv3x3(x, g, y, ws, N, C, H, W, K, precision=precision, stream=stream.cuda_stream) == 0
        if wait:
            torch.cuda.synchronize()

    def calls(outs, wait):
        with torch.cuda.stream(stream):
            for s, g, y in zip(sources, filters, outs):
                x.copy_(s)
                if wait:
                    torch.cuda.synchronize()
                conv(x, g, y, wait)
            for g, a, b in zip(filters, outs[3:], outs[4:]):      # a chain: C == K, so an output is an input as it lies
                conv(a, g, b, wait)

    expect = [torch.full((K, H, W, N), float("nan"), device="cuda") for _ in range(8)]
    got = [torch.empty_like(y) for y in expect]
    torch.cuda.synchronize()
    calls(expect, wait=True)
    assert all(bool(torch.isfinite(y).all()) for y in expect)
    for _ in range(3):
        for y in got:
            y.fill_(float("nan"))
        torch.cuda.synchronize()
        calls(got, wait=False)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, expect))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        calls(got, wait=False)
    for _ in range(2):
        for y in got:
            y.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, expect))
    assert api.last_device_status() == 0
