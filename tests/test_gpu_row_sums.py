"""The tensor-memory kernel's row sums: parts of K, folded group by group, spread over a cluster or not."""
import pytest
import torch

import if_i_could_turn_back_time_b200 as jq
from if_i_could_turn_back_time_b200 import ops
from test_gpu_parity import DEV, _check_gemv, _weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K", [(40, 512), (129, 2048), (320, 2304), (130, 11008), (9600, 2048)])
@pytest.mark.parametrize("fmt,g,B", [("gf4", 128, 2), ("gf4", 256, 16), ("gf4", 128, 17), ("gf4", 128, 33), ("gf4", 128, 64),
                                     ("e2m1", 32, 9), ("e2m1", 32, 23), ("e2m1", 32, 48)])
def test_single_calls_groups_and_row_shards_agree(fmt, g, B, N, K):
    """Fewer than 8 steps (one part) and more (four parts of unequal length), clusters of 4, 2 and no cluster: against the
    oracle, and the same bits from a grouped launch (never split) and from a row shard (split differently)."""
    spec = jq.QuantSpec(fmt, g, 0)
    pw = jq.pack_weight(_weights(N, K, N + K).to(DEV), spec)
    # (a copy: rows of a shard whose scales start off a 16-byte boundary would be left to the row loops)

    def half(i):
        part, copy = pw.rows(i * (N // 2), (i + 1) * (N // 2)), lambda t: None if t is None else t.clone()
        return jq.PackedWeight(spec, part.N, K, copy(part.qweight), copy(part.scales), copy(part.codebook))

    gen = torch.Generator("cpu").manual_seed(B)
    x = torch.randn(B, K, generator=gen).bfloat16()
    if N < 1000:
        _check_gemv(pw.to("cpu"), x, torch.randn(N, generator=gen))
    grp = ops.GroupedGemv([pw, half(0)], B, torch.float32)
    for gx in grp.xs:
        gx.copy_(x)
    grp.run()
    assert grp.status() == 0 and grp._ta
    assert torch.equal(grp.ys[1], grp.ys[0][:, :N // 2])
    if not ops.many_rows(spec.fmt_id, K, g, B):
        y = ops.linear(x.to(DEV).float(), pw)
        assert torch.equal(y, grp.ys[0])
        assert torch.equal(ops.linear(x.to(DEV).float(), half(1)), y[:, N // 2:2 * (N // 2)])
    else:
        assert (ops.linear(x.to(DEV).float(), pw) - grp.ys[0]).abs().max() <= 3e-6 * grp.ys[0].abs().max()


@pytest.mark.parametrize("fmt,g,B", [("gf4", 128, 3), ("gf4", 256, 16), ("gf4", 128, 20), ("gf4", 128, 64), ("e2m1", 32, 16), ("e2m1", 32, 40)])
@pytest.mark.parametrize("shift", [0, 1])
def test_tiles_of_odd_step_counts_and_scales_off_a_word(fmt, g, B, shift):
    """Rows of 3 and 5 steps, several tiles per CTA: the warps' turns, the weight stages, the operand slots and the
    accumulators all run across tile boundaries out of step.  GF4 scales may start at any 2-byte boundary."""
    import ctypes
    from if_i_could_turn_back_time_b200 import _lib
    spec = jq.QuantSpec(fmt, g, 0)
    gen = torch.Generator("cpu").manual_seed(B)
    packed = [jq.pack_weight(_weights(N, K, N + K).to(DEV), spec) for N, K in ((20000, 768), (9000, 1280), (18950, 768))]
    grp = ops.GroupedGemv(packed, B, torch.float32)
    for x in grp.xs:
        x.copy_(torch.randn(x.shape, generator=gen))
    grp.run()
    assert grp.status() == 0 and grp._ta
    for w, x, y in zip(packed, grp.xs, grp.ys):
        # (fp16 rounding of the activation, 2^-12 of a term, and of value x scale for E2M1; sums of at most 1280 terms)
        ref = x.double() @ ops.dequantize(w).double().t()
        assert (y - ref).abs().max() <= 1e-3 * ref.abs().max()
    if fmt == "gf4" and shift:
        w, x = packed[1], grp.xs[1]
        raw = torch.empty(w.scales.numel() + 1, dtype=torch.float16, device=DEV)
        raw[1:] = w.scales.reshape(-1)
        y, ws = torch.empty_like(grp.ys[1]), torch.zeros(4 << 20, dtype=torch.uint8, device=DEV)
        p = lambda t, off=0: ctypes.c_void_p(t.data_ptr() + off)
        _lib.check(_lib.load().jq_gemm_ta(w.spec.fmt_id, p(w.qweight), p(raw, 2), p(w.codebook), p(x), None, p(y), w.N, w.K, B, g, 0,
                                          _lib.JQ_F32, _lib.JQ_F32, p(ws), ws.numel(), ops._stream()), "jq_gemm_ta")
        assert torch.equal(y, grp.ys[1])


@pytest.mark.parametrize("K", [512, 2304, 4096, 12288])
@pytest.mark.parametrize("had,dtype", [(0, torch.float32), (128, torch.float16), (128, torch.bfloat16)])
def test_one_row_prepared_in_the_kernel_or_in_front_of_it(K, had, dtype):
    """A single call of one row prepares its activation itself, a grouped launch reads one that a kernel of its own has
    prepared: the same bits, for the shortest and longest rows, blocks that do not divide over the warps, a row of zeros, one
    with an infinity and one that starts off a vector boundary."""
    pw = jq.pack_weight(_weights(200, K, K).to(DEV), jq.QuantSpec("gf4", 128, had))
    gen = torch.Generator("cpu").manual_seed(K)
    grp = ops.GroupedGemv([pw], 1, dtype)
    raw = torch.zeros(K + 1, dtype=dtype, device=DEV)
    for scale in (1.0, 1e-3, 0.0, float("inf")):
        row = torch.randn(1, K, generator=gen)
        row[0, 0] *= scale if scale == float("inf") else 1.0
        raw[1:] = (row * (1.0 if scale == float("inf") else scale))[0].to(dtype).to(DEV)
        x = raw[1:].view(1, K)
        grp.xs[0].copy_(x)
        grp.run()
        y = ops.linear(x, pw)
        assert torch.equal(y.view(torch.uint8), grp.ys[0].view(torch.uint8))
    assert grp.status() == 0 and ops.check_status(raise_on_error=False) == 0


@pytest.mark.parametrize("xt,yt", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16), (torch.bfloat16, torch.float32),
                                   (torch.float32, torch.float16)])
@pytest.mark.parametrize("N,K", [(4096, 4096), (12000, 2048), (200, 12288)])
def test_one_row_may_be_written_over_its_activation(xt, yt, N, K):
    """jq_gemm_ta with y on x, and with y reaching over x's first and last element: the bits of the call with y elsewhere (the
    row is read as a whole before anything is written).  With y right before or right behind x nothing overlaps."""
    import ctypes
    from if_i_could_turn_back_time_b200 import _lib
    pw = jq.pack_weight(_weights(N, K, K).to(DEV), jq.QuantSpec("gf4", 128, 128))
    lib, dt = _lib.load(), {torch.float32: _lib.JQ_F32, torch.float16: _lib.JQ_F16, torch.bfloat16: _lib.JQ_BF16}
    p = lambda t, off=0: ctypes.c_void_p(t.data_ptr() + off)
    ws = torch.zeros(1 << 20, dtype=torch.uint8, device=DEV)
    xb, yb = K * xt.itemsize, N * yt.itemsize
    x = torch.randn(1, K, generator=torch.Generator("cpu").manual_seed(N)).to(xt).to(DEV)

    def call(x_ptr, y_ptr):
        _lib.check(lib.jq_gemm_ta(pw.spec.fmt_id, p(pw.qweight), p(pw.scales), p(pw.codebook), x_ptr, None, y_ptr, N, K, 1, 128, 128,
                                  dt[xt], dt[yt], p(ws), ws.numel(), ops._stream()), "jq_gemm_ta")

    want = torch.empty(1, N, dtype=yt, device=DEV)
    call(p(x), p(want))
    for at in (0, 4 - yb, xb - 4, -yb, xb):                 # byte offset of y from x
        arena = torch.zeros(xb + 2 * yb, dtype=torch.uint8, device=DEV)
        arena[yb:yb + xb] = x.view(torch.uint8)[0]
        call(p(arena, yb), p(arena, yb + at))
        assert torch.equal(arena[yb + at:2 * yb + at], want.view(torch.uint8)[0])
    assert lib.jq_ta_status(p(ws), 1, ops._stream()) == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("K", [512, 4352, 16640])
def test_activation_prepared_by_wide_and_narrow_blocks(K, dtype):
    """Few rows are prepared by blocks of 32 warps, the 320 of a large step by blocks of 8, which keep fewer of a row's values
    between their passes (up to 16384 and 4096): the same bits, also from an activation that starts off a vector boundary."""
    pw = jq.pack_weight(_weights(40, K, K).to(DEV), jq.QuantSpec("gf4", 128, 128))
    grp = ops.GroupedGemv([pw] * 40, 8, dtype)
    gen = torch.Generator("cpu").manual_seed(K)
    for x in grp.xs:
        x.copy_(torch.randn(x.shape, generator=gen))
    grp.run()
    assert grp.status() == 0
    for i in (0, 17, 39):
        raw = torch.zeros(8 * K + 1, dtype=dtype, device=DEV)
        off = raw[1:].view(8, K)
        off.copy_(grp.xs[i])
        assert torch.equal(ops.linear(grp.xs[i], pw), grp.ys[i]) and torch.equal(ops.linear(off, pw), grp.ys[i])


@pytest.mark.parametrize("fmt,g,B", [("gf4", 128, 2), ("gf4", 256, 16), ("gf4", 128, 20), ("gf4", 128, 40), ("e2m1", 32, 9), ("e2m1", 32, 16),
                                     ("e2m1", 32, 24), ("e2m1", 32, 40)])
def test_parts_of_odd_step_counts_over_several_tiles(fmt, g, B):
    """Rows of 9, 3 and 11 steps, two to three tiles per CTA: the four parts of a row's sum begin and end at another stage,
    slot and accumulator in every tile.  Against 64 bits, and the bits of single calls, whole and by row shards."""
    spec = jq.QuantSpec(fmt, g, 0)
    gen = torch.Generator("cpu").manual_seed(B)
    packed = [jq.pack_weight(_weights(N, K, N + K).to(DEV), spec) for N, K in ((20000, 2304), (18950, 768), (9000, 2816))]
    grp = ops.GroupedGemv(packed, B, torch.float32)
    for x in grp.xs:
        x.copy_(torch.randn(x.shape, generator=gen))
    grp.run()
    assert grp.status() == 0 and grp._ta
    for w, x, y in zip(packed, grp.xs, grp.ys):
        # (fp16 rounding of the activation, 2^-12 of a term, and of value x scale for E2M1; sums of at most 2816 terms)
        ref = x.double() @ ops.dequantize(w).double().t()
        assert (y - ref).abs().max() <= 1e-3 * ref.abs().max()
        if ops.many_rows(spec.fmt_id, w.K, g, B):
            continue
        assert torch.equal(ops.linear(x, w), y)
        first = w.N // 3 // 64 * 64             # (a shard's tiles start elsewhere; its scales still on a 16-byte boundary)
        part = w.rows(first, w.N)
        assert torch.equal(ops.linear(x, part), y[:, first:])
    assert ops.check_status(raise_on_error=False) == 0
