"""The work that a user of this library has it do, as a list of sized cases: the 3x3 convolution
through each of its public entry points, in its three arithmetics, over the sizes of the
benchmark's layers and of the tests, from the smallest call to the largest layer.

A case is a dict: `entry` (which public calls), `precision`, and the problem's sizes
N images, C channels in, K filters, H x W pixels.

    stream   conv3x3: filter transform and fused kernel, every call
    legacy   call_like_reference: the same through the reference's own argument list
    cached   winograd_forward on a filter transformed once, as an inference program keeps it
    noalloc  conv3x3_noalloc: the caller has no workspace
    nchw     a program with NCHW tensors: layout adapters either side of conv3x3
    host     HostPlan.run: pinned host arrays in, pinned host array out
"""
import math

import torch

from opencnn_b200 import api

SIGMA = 0.05                                    # filters ~ N(0, 0.05^2), input ~ U(-1, 1)


def _case(name, entry, precision, N, C, K, H, W):
    return {"name": name, "entry": entry, "precision": precision, "N": N, "C": C, "K": K, "H": H, "W": W}


def listed():
    return [
        # the smallest call: one block of images, a small map; latency and launches are what it costs
        _case("stream fp32 9x9 c16 k64 n32", "stream", "fp32", 32, 16, 64, 9, 9),
        # the first shape of the reference's benchmark script, called as its main() calls it
        _case("legacy fp32 56x56 c64 n32", "legacy", "fp32", 32, 64, 64, 56, 56),
        # last stage of a ResNet at batch 128, weights fixed: odd extent, few tiles, many channels
        _case("cached fp32 7x7 c512 n128", "cached", "fp32", 128, 512, 512, 7, 7),
        # sizes that fit no block: ragged batch, odd channels, filters not a multiple of 64, a rectangle
        _case("noalloc fp32 23x31 ragged", "noalloc", "fp32", 100, 61, 132, 23, 31),
        # a wide layer: the most arithmetic of the list
        _case("stream fp32 14x14 c1024 n64", "stream", "fp32", 64, 1024, 1024, 14, 14),
        # second stage of a ResNet at batch 128 in a program that holds NCHW tensors
        _case("nchw fp32 28x28 c128 n128", "nchw", "fp32", 128, 128, 128, 28, 28),
        # data that lives on the host: upload, operator, download
        _case("host fp32 56x56 c64 n32", "host", "fp32", 32, 64, 64, 56, 56),
        # tensor-core arithmetic on a ResNet's first stage: large map, few channels and filters
        _case("stream bf16 56x56 c64 n128", "stream", "bf16", 128, 64, 64, 56, 56),
        # inference on a third stage with fixed weights
        _case("cached bf16 14x14 c256 n128", "cached", "bf16", 128, 256, 256, 14, 14),
        # the most memory of the list: a first-layer-like map
        _case("stream bf16 112x112 c32 n256", "stream", "bf16", 256, 32, 64, 112, 112),
        # TF32: second stage, and the wide layer with fixed weights
        _case("stream tf32 28x28 c128 n128", "stream", "tf32", 128, 128, 128, 28, 28),
        _case("cached tf32 14x14 c1024 n64", "cached", "tf32", 64, 1024, 1024, 14, 14),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _multiple(value, of):
    return max(of, of * int(value / of + 0.5))


def draw(rng):
    """One more case: every entry and arithmetic, batches of 8 to 256, 3 to 1024 channels, up to
    1024 filters, maps of 7 to 112 pixels a side, ragged wherever the entry takes it; never more
    arithmetic or memory than the largest listed cases have."""
    while True:
        entry = rng.choice(["stream", "stream", "legacy", "cached", "cached", "noalloc", "nchw", "host"])
        precision = "fp32" if entry in ("legacy", "noalloc") else rng.choice(["fp32", "tf32", "bf16"])
        n_of, c_of, k_of = (32, 8, 64) if entry == "legacy" else (4, 1, 4) if precision == "fp32" else (8, 1, 64)
        H = int(_log(rng, 7, 113))
        W = H if entry == "legacy" or rng.random() < 0.5 else int(_log(rng, 7, 113))
        c = {"entry": entry, "precision": precision, "N": _multiple(_log(rng, 8, 256), n_of),
             "C": _multiple(_log(rng, 3, 1024), c_of), "K": _multiple(_log(rng, 32, 1024), k_of), "H": H, "W": W}
        if entry == "noalloc" and c["C"] * c["K"] > api.NOALLOC_MAX_CK:
            continue
        w = work(c)
        if not 1e7 <= w["flops"] <= (2e10 if entry == "host" else 1e11):
            continue
        if w["bytes"] > (5.5e7 if entry == "host" else 1.2e9):
            continue
        return c


def _random(shape, generator, normal):
    t = torch.empty(shape, device="cuda")
    return t.normal_(0.0, SIGMA, generator=generator) if normal else t.uniform_(-1.0, 1.0, generator=generator)


def _inputs(case, seed):
    N, C, K, H, W = (case[k] for k in "NCKHW")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    x = _random((N, C, H, W) if case["entry"] == "nchw" else (C, H, W, N), gen, False)
    return x, _random((C, 3, 3, K), gen, True)


def prepare(case, seed):
    N, C, K, H, W = (case[k] for k in "NCKHW")
    entry, precision = case["entry"], case["precision"]
    x, g = _inputs(case, seed)
    s = {"entry": entry, "precision": precision, "size": (N, C, H, W, K),
         "stream": torch.cuda.current_stream().cuda_stream}
    if entry == "host":
        s["x"], s["g"] = x.cpu().pin_memory(), g.cpu().pin_memory()
        s["y"] = torch.zeros((K, H, W, N)).pin_memory()
        s["plan"] = api.HostPlan(N, C, H, W, K, precision=precision)
        return s
    s["x"], s["g"] = x, g
    s["y"] = torch.zeros((K, H, W, N), device="cuda")
    if entry != "noalloc":
        s["ws"] = torch.zeros(api.workspace_bytes(C, K) // 4, device="cuda")
    if entry == "nchw":
        s["x_chwn"] = torch.zeros((C, H, W, N), device="cuda")
        s["y_nkhw"] = torch.zeros((N, K, H, W), device="cuda")
    if entry == "cached":
        _ok(api.filter_transform(g, s["ws"], C, K, precision=precision, stream=s["stream"]))
    return s


def _ok(err):
    if err != 0:
        raise RuntimeError(f"the library returned cudaError {err}")


def run(s):
    N, C, H, W, K = s["size"]
    entry, stream = s["entry"], s["stream"]
    if entry == "stream":
        _ok(api.conv3x3(s["x"], s["g"], s["y"], s["ws"], N, C, H, W, K, precision=s["precision"], stream=stream))
    elif entry == "legacy":
        _ok(api.call_like_reference(s["x"], s["g"], s["y"], s["ws"], N, C, H, W, K))
    elif entry == "cached":
        _ok(api.winograd_forward(s["x"], s["ws"], s["y"], N, C, H, W, K, precision=s["precision"], stream=stream))
    elif entry == "noalloc":
        _ok(api.conv3x3_noalloc(s["x"], s["g"], s["y"], N, C, H, W, K, stream=stream))
    elif entry == "nchw":
        _ok(api.nchw_to_chwn(s["x"], s["x_chwn"], N, C, H, W, stream=stream))
        _ok(api.conv3x3(s["x_chwn"], s["g"], s["y"], s["ws"], N, C, H, W, K, precision=s["precision"], stream=stream))
        _ok(api.khwn_to_nkhw(s["y"], s["y_nkhw"], N, K, H, W, stream=stream))
        return s["y_nkhw"]
    else:
        _ok(s["plan"].run(s["x"].data_ptr(), s["g"].data_ptr(), s["y"].data_ptr()))
    return s["y"]


def work(case):
    """Bytes: input, filter (for `cached` the transformed filter in its operand type) and output,
    once each.  Flops: the sixteen products of F(2x2,3x3)."""
    N, C, K, H, W = (case[k] for k in "NCKHW")
    f = 16 * C * K * (2 if case["precision"] == "bf16" else 4) if case["entry"] == "cached" else 9 * C * K * 4
    return {"bytes": 4 * N * H * W * (C + K) + f,
            "flops": 2 * 16 * N * ((H + 1) // 2) * ((W + 1) // 2) * C * K}


def tolerance(case):
    """fp32: sums of 9 C products of 32-bit values.  TF32 and BF16: the operands carry 11 and 8
    significant bits; the sums are kept in 32."""
    return {"rel": {"fp32": 1e-5, "tf32": 1e-3, "bf16": 1e-2}[case["precision"]]}


def exact(case, seed):
    """The convolution of the unrounded inputs in 64 bits: one matrix product per filter tap."""
    N, C, K, H, W = (case[k] for k in "NCKHW")
    x, g = _inputs(case, seed)
    if case["entry"] == "nchw":
        x = x.permute(1, 2, 3, 0)
    padded = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1))
    y = torch.zeros((K, H * W * N), dtype=torch.float64, device="cuda")
    for r in range(3):
        for t in range(3):
            y.addmm_(g[:, r, t].double().T, padded[:, r:r + H, t:t + W].reshape(C, H * W * N))
    y = y.view(K, H, W, N)
    if case["entry"] == "nchw":
        return y.permute(3, 0, 1, 2).contiguous()
    return y.cpu() if case["entry"] == "host" else y
