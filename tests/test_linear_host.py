"""Host-side mirror of the reference's QuantLinear / quantize_module surface
(no GPU: nothing here launches a kernel)."""
import inspect

import pytest
import torch
import torch.nn as nn

import if_i_could_turn_back_time_b200 as jq


def test_constructor_signature_matches_reference():
    params = list(inspect.signature(jq.JenksQuantLinear.__init__).parameters.values())
    assert [p.name for p in params[:4]] == ["self", "linear_module", "bitwidth", "mask"]
    assert params[2].default == 4 and params[3].default is None
    assert all(p.kind is inspect.Parameter.KEYWORD_ONLY for p in params[4:])


def test_attributes_and_commit():
    lin = nn.Linear(256, 24)
    q = jq.JenksQuantLinear(lin, 4, fmt="e2m1", group_size=32)
    assert isinstance(q, nn.Linear) and q.in_features == 256 and q.out_features == 24
    assert q.hard_quant is False and not q.weight.requires_grad
    assert torch.equal(q.weight.data, lin.weight.data) and torch.equal(q.bias.data, lin.bias.data)
    assert torch.equal(q.mask, torch.ones_like(lin.weight))
    q.commit()
    assert q.hard_quant is True and q._parameters["weight"] is None
    sd = q.state_dict()
    assert {"qweight", "scales", "bias", "mask"} <= set(sd) and "weight" not in sd
    assert sd["qweight"].dtype == torch.uint8 and sd["qweight"].shape == (24, 128)


def test_bitwidth_other_than_4_is_rejected():
    with pytest.raises(ValueError):
        jq.JenksQuantLinear(nn.Linear(64, 8), 8)


def test_quantize_module_swaps_linears_and_keeps_sparsity_mask():
    model = nn.Sequential(nn.Flatten(), nn.Linear(784, 300), nn.ReLU(), nn.Linear(300, 100), nn.ReLU(),
                          nn.Linear(100, 10))
    with torch.no_grad():
        model[1].weight[:, ::2] = 0
    qm = jq.quantize_module(model, 4, fmt="gf4", group_size=0)
    assert isinstance(qm[1], jq.JenksQuantLinear) and isinstance(qm[3], jq.JenksQuantLinear)
    assert isinstance(model[1], nn.Linear) and not isinstance(model[1], jq.JenksQuantLinear)  # deep copy
    assert torch.equal(qm[1].mask, (model[1].weight != 0).float())
    leaf = jq.quantize_module(nn.Linear(128, 4), 4, fmt="e2m1", group_size=32)
    assert isinstance(leaf, jq.JenksQuantLinear)


def test_forward_without_cuda_fails_loudly():
    q = jq.JenksQuantLinear(nn.Linear(64, 8), 4, fmt="e2m1", group_size=32)
    with pytest.raises(RuntimeError, match="CUDA"):
        q(torch.randn(2, 64))


def test_spec_validation():
    with pytest.raises(ValueError):
        jq.QuantSpec("e2m1", 0, 0)
    with pytest.raises(ValueError):
        jq.QuantSpec("gf4", 48, 0)
    with pytest.raises(ValueError):
        jq.QuantSpec("gf4", 128, 64)
    assert jq.algorithmic_bytes(jq.QuantSpec("e2m1", 32, 0), 4096, 4096, 1, 2, 2) == 9453568
    assert jq.algorithmic_bytes(jq.QuantSpec("gf4", 128, 128), 11008, 4096, 1, 2, 2) == 23631360


def test_status_helpers_without_any_workspace():
    """No GPU work has run: nothing to read, nothing raised; checked mode is a plain switch."""
    from if_i_could_turn_back_time_b200 import ops
    ops.set_checked(True)
    assert ops._checked is True
    ops.set_checked(False)
    assert ops._checked is False


def test_scratch_buffers_are_per_thread():
    """Calls from different host threads never share a workspace: the cache lives in thread-local storage."""
    import threading
    from if_i_could_turn_back_time_b200 import ops
    mine = ops._ws_cache()
    mine["probe"] = 1
    seen = {}

    def other():
        seen["cache"] = ops._ws_cache()
        seen["empty"] = "probe" not in seen["cache"]

    t = threading.Thread(target=other)
    t.start()
    t.join()
    del mine["probe"]
    assert seen["empty"] and seen["cache"] is not mine


def test_grouped_plan_partitions_the_row_space_evenly():
    """jq_grouped_plan is host-only: its partition of the concatenated row-group space into one contiguous range
    per CTA can be checked without a GPU (fake, aligned device addresses; nothing is dereferenced).  Layout of the
    plan: 8 header ints [magic, n, grid, largest K, rows per group, batch, format, ...], then the first row group
    of every problem (n + 1 ints) and of every CTA (grid + 1 ints)."""
    import ctypes
    import numpy as np
    from if_i_could_turn_back_time_b200 import _lib
    lib = _lib.load()
    shapes = [(4096, 4096)] * 4 + [(11008, 4096)] * 2 + [(4096, 11008)]
    n = len(shapes) * 4
    arr = (_lib.jq_problem * n)()
    for i in range(n):
        N, K = shapes[i % len(shapes)]
        arr[i].qweight = 0x10000000 + i * 0x4000000
        arr[i].scales = 0x20000000 + i * 0x400000
        arr[i].x = 0x30000000
        arr[i].y = 0x40000000
        arr[i].N, arr[i].K, arr[i].g, arr[i].had_block = N, K, 32, 0
    nbytes = lib.jq_grouped_plan_bytes(n)
    plan = np.zeros((nbytes + 3) // 4, dtype=np.int32)
    st = lib.jq_grouped_plan(_lib.JQ_FMT_E2M1, ctypes.byref(arr), n, 1, plan.ctypes.data, plan.nbytes)
    assert st == 0, _lib.strerror(st)
    grid, rows_per_group = int(plan[2]), int(plan[4])
    assert int(plan[1]) == n and grid > 0 and rows_per_group > 0
    rg_start = plan[8:8 + n + 1]
    cta_first = plan[8 + n + 1:8 + n + 1 + grid + 1]
    groups = [(-(-shapes[i % len(shapes)][0] // rows_per_group)) for i in range(n)]
    assert list(np.diff(rg_start)) == groups
    assert cta_first[0] == 0 and cta_first[-1] == rg_start[-1] and np.all(np.diff(cta_first) >= 0)
    # cost of every CTA's range in row-group x K units: within two row groups of the mean
    k_of = np.repeat([shapes[i % len(shapes)][1] for i in range(n)], groups)
    cost = np.array([k_of[a:b].sum() for a, b in zip(cta_first[:-1], cta_first[1:])], dtype=np.float64)
    assert abs(cost - cost.mean()).max() <= 2 * 11008
    # a misaligned weight pointer is refused before anything else happens
    arr[3].qweight += 8
    st = lib.jq_grouped_plan(_lib.JQ_FMT_E2M1, ctypes.byref(arr), n, 1, plan.ctypes.data, plan.nbytes)
    assert st != 0 and "align" in _lib.strerror(st)


@pytest.mark.parametrize("fmt,g", [("gf4", 0), ("gf4", 32)])
@pytest.mark.parametrize("shape", [(2, 31, 9, 9), (2, 33, 9, 9), (2, 64, 9, 9), (32, 9, 9)])
def test_convolution_refuses_an_image_that_is_not_the_layers(fmt, g, shape):
    """The check comes before the devices are looked at, so that it needs no GPU."""
    q = jq.JenksQuantConv2d(nn.Conv2d(32, 4, 3, padding=1), 4, fmt=fmt, group_size=g)
    with pytest.raises(RuntimeError, match="channels|dimensions"):
        jq.ops.conv2d(torch.randn(*shape), q.packed, q.bias, q.kernel_size, q.stride, q.padding, q.dilation)


@pytest.mark.parametrize("make", [lambda: jq.JenksQuantLinear(nn.Linear(256, 8), 4),
                                  lambda: jq.JenksQuantConv2d(nn.Conv2d(16, 8, 4), 4, group_size=128)], ids=["linear", "conv"])
def test_packed_tensors_are_read_as_attributes(make):
    """A packed tensor that has become a parameter, is computed by a parametrisation or by a property of another class is
    what `packed` returns, as any other reader of the layer sees it."""
    class Doubled(nn.Module):
        def forward(self, t):
            return t * 2

    layer = make()
    layer.commit()
    q, s, c = layer.qweight, layer.scales, layer.codebook
    assert layer.packed.qweight is q and layer.packed.scales is s and layer.packed.codebook is c
    layer.qweight = nn.Parameter(q.clone(), requires_grad=False)
    assert layer.packed.qweight is layer.qweight and torch.equal(layer.packed.qweight, q)
    assert layer.packed.scales is s and layer.packed.codebook is c

    layer = make()
    layer.commit()
    s = layer.scales.clone()
    nn.utils.parametrize.register_parametrization(layer, "scales", Doubled(), unsafe=True)
    assert torch.equal(layer.packed.scales, s * 2)

    layer = make()
    layer.commit()
    c = layer.codebook.clone()
    layer.__class__ = type("Other", (type(layer),), {"codebook": property(lambda self: self._buffers["codebook"] + 1)})
    assert torch.equal(layer.packed.codebook, c + 1)


@pytest.fixture
def scratch(monkeypatch):
    """ops' scratch buffers on the CPU: one device, one stream, and a switch that says whether a graph is being captured."""
    import threading
    from if_i_could_turn_back_time_b200 import ops
    state = {"capturing": False}
    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: 0, raising=False)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda index: 7, raising=False)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: state["capturing"])
    monkeypatch.setattr(ops, "check_status", lambda raise_on_error=True: 0)
    monkeypatch.setattr(ops, "_tls", threading.local())
    monkeypatch.setattr(ops, "_captured", {}, raising=False)
    return ops, state


@pytest.mark.parametrize("kind", ["ta", "gemv"])
def test_a_scratch_buffer_that_a_graph_holds_is_not_freed(scratch, kind):
    import weakref
    ops, state = scratch
    cpu = torch.device("cpu")
    plain = weakref.ref(ops._workspace(cpu, 1024, kind))
    held = weakref.ref(ops._workspace(cpu, 6 << 20, kind))
    assert plain() is None                              # nothing but eager calls used it
    state["capturing"] = True
    assert ops._workspace(cpu, 1024, kind) is held()
    state["capturing"] = False
    largest = ops._workspace(cpu, 7 << 20, kind)
    assert held() is not None and largest is not held()
    assert largest.numel() >= 2 * held().numel()        # what is kept stays below the buffer in use


def test_captured_many_row_calls_have_scratch_of_their_own(scratch):
    ops, state = scratch
    cpu = torch.device("cpu")
    own, ptr, size, status = ops._rows_scratch(cpu, 4096)
    assert own is None and ptr == status + 1024 and size >= 4096
    state["capturing"] = True
    own, ptr, size, captured_status = ops._rows_scratch(cpu, 4096)
    assert own is not None and ptr == own.data_ptr() and size == own.numel() == 4096 and captured_status == status


def test_routes_of_calls_with_several_rows():
    """GF4 on the tensor-memory kernel's shapes leaves it at 33 rows, E2M1 at 65, everything else the row loops at 17."""
    from if_i_could_turn_back_time_b200 import _lib, ops
    gf4, e2m1 = _lib.JQ_FMT_GF4, _lib.JQ_FMT_E2M1
    for fmt, K, g, last in [(gf4, 4096, 128, 32), (gf4, 512, 256, 32), (gf4, 4096, 64, 16), (gf4, 784, 0, 16), (gf4, 384, 128, 16),
                            (e2m1, 4096, 32, 64), (e2m1, 4096, 64, 16), (e2m1, 1152, 32, 16)]:
        assert [ops.many_rows(fmt, K, g, b) for b in (1, last, last + 1, 4096)] == [False, False, True, True]


def test_calls_of_up_to_64_rows_fit_in_the_first_scratch_buffer(scratch):
    """A call in a graph capture cannot replace the stream's buffer (its status word would have to be read first)."""
    import ctypes
    from if_i_could_turn_back_time_b200 import _lib
    ops, _ = scratch
    prob = _lib.jq_problem()
    prob.K = 28672
    need = _lib.load().jq_ta_workspace_bytes(ctypes.byref(prob), 1, 64)
    first = ops._workspace(torch.device("cpu"), 1024, "ta")
    assert ops._workspace(torch.device("cpu"), need, "ta") is first


def test_long_fields_at_few_positions_are_unfolded():
    from if_i_could_turn_back_time_b200 import _lib, ops
    gf4, e2m1 = _lib.JQ_FMT_GF4, _lib.JQ_FMT_E2M1
    assert [ops.conv_gathers(gf4, 576, 0, p) for p in (1, 16, 17, 4096)] == [False, False, True, True]
    assert [ops.conv_gathers(gf4, 1024, 128, p) for p in (16, 17)] == [False, True]
    assert [ops.conv_gathers(e2m1, 1024, 32, p) for p in (64, 65)] == [False, True]
    assert [ops.conv_gathers(gf4, 4608, 0, p) for p in (17, 32, 2048, 2049)] == [False, False, False, True]
    assert [ops.conv_gathers(gf4, K, 0, 100) for K in (1536, 1537)] == [True, False]
