"""The many-row kernel (prompts, evaluation batches, convolutions) against the oracle: edges of its 128-row tiles, of the
token tiles (32 to 256, one or two accumulators), of the 128-code groups, of the K split over a cluster, and every way
of folding scales (128, 64 and 32 codes at once, none, folded into fp16 weights)."""
import numpy as np
import pytest
import torch

import if_i_could_turn_back_time_b200 as jq
from if_i_could_turn_back_time_b200 import ops
from oracle import formats
from test_gpu_parity import DEV, TOL, _check_gemv, _weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt,N,K,g,had,rows,dtype", [
    ("gf4", 10, 100, 0, 0, 17, torch.float32),          # one ragged group, odd row count
    ("gf4", 300, 784, 0, 0, 64, torch.float32),         # seven groups, the last one an eighth full
    ("gf4", 129, 333, 0, 0, 130, torch.float16),        # odd K; two token halves
    ("gf4", 128, 640, 128, 128, 129, torch.bfloat16),   # K % 256 != 0: an odd number of groups
    ("gf4", 257, 1024, 64, 0, 256, torch.bfloat16),     # 64-code scales, a full token tile
    ("gf4", 70, 960, 32, 0, 257, torch.float32),        # 32-code scales, two token tiles
    ("gf4", 200, 1024, 256, 128, 33, torch.float16),    # one scale for two groups
    ("gf4", 64, 11008, 128, 128, 40, torch.bfloat16),   # K split eight ways
    ("gf4", 1100, 512, 128, 0, 700, torch.bfloat16),
    ("e2m1", 33, 256, 32, 128, 24, torch.bfloat16),     # too short for the folded weights: exact
    ("e2m1", 130, 1152, 32, 0, 100, torch.float32),     # K % 256 != 0: exact
    ("e2m1", 96, 1024, 64, 0, 300, torch.float16),
    ("e2m1", 140, 384, 96, 0, 20, torch.bfloat16),      # a group that is not a power of two
    ("e2m1", 256, 2048, 128, 128, 65, torch.bfloat16),
    ("e2m1", 300, 4096, 32, 0, 65, torch.bfloat16),     # folded
    ("e2m1", 129, 512, 32, 128, 513, torch.float32),    # folded, three token tiles
])
def test_many_rows_against_the_oracle(fmt, N, K, g, had, rows, dtype):
    spec = jq.QuantSpec(fmt, g, had)
    assert ops.many_rows(spec.fmt_id, K, g, rows)
    pw = jq.pack_weight(_weights(N, K, N + K), spec)
    gen = torch.Generator("cpu").manual_seed(rows)
    x = (torch.randn(rows, K, generator=gen) * torch.logspace(-2, 2, rows)[:, None]).to(dtype)
    _check_gemv(pw, x / 100, torch.randn(N, generator=gen))
    y32 = ops.linear(x.to(DEV), pw.to(DEV), out_dtype=torch.float32)
    assert torch.equal(ops.linear(x.to(DEV), pw.to(DEV)), y32.to(dtype))      # rounded once


def test_many_rows_unit_vectors_read_back_columns_and_misaligned_rows():
    """x = e_k is exact: every output is an entry of the dequantised matrix, bit for bit; also from an activation that
    starts 2 bytes off a vector boundary."""
    pw = jq.pack_weight(_weights(150, 700, 5), jq.QuantSpec("gf4", 0, 0)).to(DEV)
    ks = [0, 1, 7, 8, 127, 128, 511, 512, 640, 698, 699] * 3
    raw = torch.zeros(len(ks) * 700 + 1, dtype=torch.float16, device=DEV)
    x = raw[1:].view(len(ks), 700)
    for i, k in enumerate(ks):
        x[i, k] = 1.0
    y = ops.linear(x, pw, out_dtype=torch.float32)
    assert torch.equal(y, ops.dequantize(pw)[:, ks].t())
    assert ops.check_status(raise_on_error=False) == 0


def test_many_rows_in_parts_and_from_a_cuda_graph(monkeypatch):
    pw = jq.pack_weight(_weights(130, 512, 6), jq.QuantSpec("gf4", 128, 128)).to(DEV)
    x = torch.randn(600, 512, generator=torch.Generator("cpu").manual_seed(1)).bfloat16().to(DEV)
    whole = ops.linear(x, pw, out_dtype=torch.float32)
    monkeypatch.setattr(ops, "MAX_ROWS_SCRATCH", 256 * 512 * 2)               # 256 rows at a time
    parts = ops.linear(x, pw, out_dtype=torch.float32)
    assert formats.rel_err(parts.cpu().numpy(), whole.cpu().numpy()) <= 2e-6  # fp32 summation order (K split) may differ
    monkeypatch.undo()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ops.linear(x, pw)
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        y = ops.linear(x, pw)
    x2 = torch.randn(600, 512, generator=torch.Generator("cpu").manual_seed(2)).bfloat16().to(DEV)
    x.copy_(x2)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, ops.linear(x2, pw))


@pytest.mark.parametrize("cin,cout,k,stride,pad,dilation,hw,batch,dtype", [
    (3, 8, 3, 1, 1, 1, (9, 11), 2, torch.float32), (16, 130, 5, 2, 2, 1, (17, 8), 3, torch.float16),
    (48, 24, 1, 1, 0, 1, (7, 7), 5, torch.bfloat16), (20, 40, (3, 2), (2, 1), (0, 3), (2, 3), (14, 13), 2, torch.float32),
    (96, 16, 3, 1, 1, 1, (6, 7), 2, torch.float32)])          # fields too long for shared memory
def test_convolution_gathers_receptive_fields(cin, cout, k, stride, pad, dilation, hw, batch, dtype):
    """Against float64 conv2d on the dequantised weight; contiguous, channels-last and sliced images give the same bits."""
    torch.manual_seed(cin)
    q = jq.JenksQuantConv2d(torch.nn.Conv2d(cin, cout, k, stride, pad, dilation), 4).to(DEV)
    x = torch.randn(batch, cin, *hw, device=DEV).to(dtype)
    y = q(x)
    ref = torch.nn.functional.conv2d(x.double(), q.dequantized_weight().double(), q.bias.double(), stride, pad, dilation)
    assert y.shape == ref.shape and y.dtype == dtype
    limit = TOL + (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11 if dtype == torch.float16 else 0)
    assert np.abs(y.double().cpu().numpy() - ref.cpu().numpy()).max() <= limit * ref.abs().max().item()
    assert torch.equal(q(x.to(memory_format=torch.channels_last)), y)
    wide = torch.zeros(batch, cin + 1, hw[0] + 2, hw[1] + 3, device=DEV, dtype=dtype)
    wide[:, 1:, 1:-1, 2:-1] = x
    assert torch.equal(q(wide[:, 1:, 1:-1, 2:-1]), y)
    assert ops.check_status(raise_on_error=False) == 0


@pytest.mark.parametrize("fmt,g", [("gf4", 0), ("gf4", 32)])
def test_convolution_refuses_other_channel_counts(fmt, g):
    """From the module's forward, as torch.nn.Conv2d does; the refusal is the host's, nothing is launched."""
    q = jq.JenksQuantConv2d(torch.nn.Conv2d(32, 8, 3, padding=1), 4, fmt=fmt, group_size=g).to(DEV)
    q.commit()
    for channels in (31, 33, 64):
        with pytest.raises(RuntimeError, match=f"{channels} channels"):
            q(torch.randn(2, channels, 9, 9, device=DEV))
    assert q(torch.randn(2, 32, 9, 9, device=DEV)).shape == (2, 8, 9, 9)


def test_captured_calls_survive_a_larger_call_on_their_stream():
    """Between capture and replay a call that needs more scratch replaces the stream's buffer, and other tensors are
    allocated and filled: the replay still gives the right results and leaves the others alone."""
    gen = torch.Generator("cpu").manual_seed(4)
    flat = jq.pack_weight(_weights(130, 700, 8), jq.QuantSpec("gf4", 0, 0)).to(DEV)
    grouped = jq.pack_weight(_weights(192, 1024, 9), jq.QuantSpec("gf4", 128, 128)).to(DEV)
    wide = jq.pack_weight(_weights(64, 34048, 10).to(DEV), jq.QuantSpec("e2m1", 32, 0))
    conv = jq.JenksQuantConv2d(torch.nn.Conv2d(16, 24, 3), 4).to(DEV)
    conv.commit()
    xs = [torch.randn(40, 700, generator=gen).to(DEV), torch.randn(12, 1024, generator=gen).bfloat16().to(DEV),
          torch.randn(2, 16, 9, 9, generator=gen).to(DEV)]
    calls = [lambda x: ops.linear(x, flat), lambda x: ops.linear(x, grouped), conv]
    x_wide = torch.randn(64, 34048, generator=gen).bfloat16().to(DEV)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        for call, x in zip(calls, xs):
            call(x)
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        ys = [call(x) for call, x in zip(calls, xs)]
    with torch.cuda.stream(stream):
        ops.linear(x_wide, wide)
        fill = [torch.full((4 << 20,), 7, dtype=torch.uint8, device=DEV) for _ in range(4)]
    stream.synchronize()
    for _ in range(2):
        for x in xs:
            x.copy_(torch.randn(x.shape, generator=gen))
        graph.replay()
        torch.cuda.synchronize()
        for call, x, y in zip(calls, xs, ys):
            assert torch.equal(y, call(x))
        assert all(bool((f == 7).all()) for f in fill)
    with torch.cuda.stream(stream):
        assert ops.check_status(raise_on_error=False) == 0


@pytest.mark.parametrize("fmt,g,rows", [("gf4", 128, 24), ("gf4", 128, 70), ("e2m1", 32, 40), ("e2m1", 32, 65), ("e2m1", 32, 130)])
def test_scales_off_a_16_byte_boundary(fmt, g, rows):
    """The tensor-memory kernel reads scales in 16-byte pieces: such a view goes to the row loops or to the many-row kernel,
    which then keeps E2M1 weights exact at a shape where it would have folded the scales."""
    pw = jq.pack_weight(_weights(140, 1024, 11), jq.QuantSpec(fmt, g, 0))
    dev = pw.to(DEV)
    room = torch.zeros(dev.scales.numel() + 8, dtype=dev.scales.dtype, device=DEV)
    off = room[1:1 + dev.scales.numel()].view(dev.scales.shape)
    off.copy_(dev.scales)
    assert off.data_ptr() % 16 == 2
    shifted = jq.PackedWeight(dev.spec, dev.N, dev.K, dev.qweight, off, dev.codebook)
    x = torch.randn(rows, 1024, generator=torch.Generator("cpu").manual_seed(rows)).bfloat16()
    y = ops.linear(x.to(DEV), shifted, out_dtype=torch.float32).cpu().numpy()
    w = ops.dequantize(dev).cpu().double().numpy()
    # 11 bits of the activation, 1024 products summed in fp32; no rounding of the weights
    exact = x.double().numpy() @ w.T
    assert np.abs(y - exact).max() <= 1e-3 * np.abs(exact).max()
    assert formats.rel_err(y, ops.linear(x.to(DEV), dev, out_dtype=torch.float32).cpu().numpy()) <= 1e-3
    assert ops.check_status(raise_on_error=False) == 0


@pytest.mark.parametrize("fmt,K,g,had", [("gf4", 700, 0, 0), ("gf4", 1024, 128, 0), ("e2m1", 1024, 32, 0), ("e2m1", 1152, 64, 128)])
def test_rows_that_are_not_finite_stay_among_themselves(fmt, K, g, had):
    """A row with an infinity or a NaN gives no finite output (every product with it is one of these, or the sum is); the
    rows beside it are what they are without it."""
    spec = jq.QuantSpec(fmt, g, had)
    pw = jq.pack_weight(_weights(130, K, 12), spec).to(DEV)
    x = torch.randn(80, K, generator=torch.Generator("cpu").manual_seed(7)).to(DEV)
    clean = ops.linear(x, pw)
    bad = [0, 31, 32, 79]
    for i, v in zip(bad, (float("nan"), float("inf"), float("-inf"), float("nan"))):
        x[i, (i * 37) % K] = v
    y = ops.linear(x, pw)
    good = [i for i in range(80) if i not in bad]
    assert torch.equal(y[good], clean[good])
    assert not torch.isfinite(y[[0, 79]]).any()
    hit = ops.dequantize(pw)[:, [(31 * 37) % K, (32 * 37) % K]] != 0
    if not had:
        assert not torch.isfinite(y[31][hit[:, 0]]).any() and not torch.isfinite(y[32][hit[:, 1]]).any()


def test_convolution_with_group_scales():
    """Groups of 64 and 96 values of the unfolded field, gathered and unfolded, against float64 conv2d."""
    for cin, k, g, fmt in ((64, 3, 64, "gf4"), (32, 3, 96, "e2m1"), (256, 3, 128, "gf4")):
        torch.manual_seed(cin)
        q = jq.JenksQuantConv2d(torch.nn.Conv2d(cin, 20, k, padding=1), 4, fmt=fmt, group_size=g).to(DEV)
        assert q.spec.group_size == g
        x = torch.randn(2, cin, 7, 9, device=DEV)
        y = q(x)
        ref = torch.nn.functional.conv2d(x.double(), q.dequantized_weight().double(), q.bias.double(), padding=1)
        assert (y.double() - ref).abs().max() <= TOL * ref.abs().max()


def test_convolution_of_a_lazily_negated_image():
    q = jq.JenksQuantConv2d(torch.nn.Conv2d(6, 8, 3, padding=1), 4).to(DEV)
    x = torch.randn(2, 6, 9, 9, dtype=torch.complex64, device=DEV).conj().imag
    assert x.is_neg()
    assert torch.equal(q(x), q(x + 0.0))


@pytest.mark.parametrize("positions", [31, 4736, 4737, 9472, 9473])
@pytest.mark.parametrize("cin,dtype", [(4, torch.float32), (88, torch.float16)])       # fields kept in shared memory, or not
def test_convolution_gathered_by_more_or_fewer_warps(positions, cin, dtype):
    """Up to 148 blocks of 32 positions, up to 296 and beyond have 32, 16 and 8 warps each: row 1 of a two-row image whose
    kernel reaches over both edges, against float64 conv2d."""
    torch.manual_seed(cin)
    q = jq.JenksQuantConv2d(torch.nn.Conv2d(cin, 12, 3, stride=(2, 1), padding=1), 4).to(DEV)
    x = torch.randn(1, cin, 2, positions, device=DEV).to(dtype)
    y = ops.conv2d(x, q.packed, q.bias, q.kernel_size, q.stride, q.padding, q.dilation)
    ref = torch.nn.functional.conv2d(x.double(), q.dequantized_weight().double(), q.bias.double(), (2, 1), 1)
    assert y.shape == ref.shape == (1, 12, 1, positions)
    limit = TOL + (2.0 ** -11 if dtype == torch.float16 else 0)
    assert (y.double() - ref).abs().max() <= limit * ref.abs().max()
