"""What linear.matmul describes and keeps, without a GPU: the descriptors' formats and addresses, and which calls a kept one
serves. Tensors are host ones and no launch is made."""

import contextlib
import ctypes

import numpy as np
import pytest
import torch

from common import ttnn_like as ttnn
from dense_reader import _tkd, linear


class Device:
    """Stands in for a GPU: tensors made on it are the host's."""

    id, sms, torch = 0, 148, torch.device("cpu")

    def dram_grid_size(self):
        return ttnn.Grid(8, 1)


DEVICE = Device()


class DeviceScale(torch.Tensor):
    """A host tensor where the device's is asked for."""

    is_cuda = True


def weight(k, n, dtype=ttnn.bfloat8_b, wide=False):
    fmt = _tkd.FMT_BF16 if wide else ttnn.FMT[dtype]
    stream = torch.zeros(_tkd.lib().tkd_packed_bytes(fmt, k, n), dtype=torch.uint8)
    emax = None if fmt == _tkd.FMT_BF16 else torch.zeros(_tkd.lib().tkd_padded_cols(n) // 16, dtype=torch.uint8)
    return ttnn.Weight(stream, emax, k, n, dtype, DEVICE, linear.sharded_memcfg(DEVICE, k, n), fmt=fmt)


def tensor(*shape, dtype=ttnn.bfloat16):
    return ttnn.Tensor(torch.zeros(*shape, dtype=ttnn._TORCH[dtype]), dtype, ttnn.TILE_LAYOUT, DEVICE, None)


@pytest.fixture
def ran(monkeypatch):
    """The calls that linear.matmul would have launched, in order."""
    calls = []

    def run(call, x, out, residual):
        calls.append(call)
        return out.t if out is not None else torch.zeros(1, 1, x.t.shape[-2], call.launches[0][1].ldo)

    def twin(w):
        if w.fmt == _tkd.FMT_BF16:
            return w
        if getattr(w, "_bf16_twin", None) is None:
            w._bf16_twin = weight(w.k, w.n, w.dtype, wide=True)
        return w._bf16_twin

    monkeypatch.setattr(linear._Call, "run", run)
    monkeypatch.setattr(ttnn, "as_bf16_stream", twin)
    return calls


@pytest.mark.parametrize("m", [1, 16, 64])
@pytest.mark.parametrize("dtype", [ttnn.bfloat8_b, ttnn.bfloat4_b])
@pytest.mark.parametrize("which", ["gate", "up"])
def test_a_gate_and_an_up_weight_of_two_stream_formats(ran, m, dtype, which):
    """A wide weight is held as a bf16 stream: its partner is streamed as bf16 too, since a launch is told one format."""
    gate, up = weight(256, 128, dtype, wide=which == "gate"), weight(256, 128, dtype, wide=which == "up")
    x = tensor(1, 1, m, 256)
    for _ in range(2):
        linear.matmul(x, gate, None, w_up=up, glu=True)
    linear.linear(x, (gate, up), None, activation="swiglu")
    for call in ran:
        ((_, a),) = call.launches
        assert a.fmt == _tkd.FMT_BF16 and a.epilogue == _tkd.EPI_GLU2
        assert a.block[0].w == ttnn.as_bf16_stream(gate).t.data_ptr() and a.block[0].w_up == ttnn.as_bf16_stream(up).t.data_ptr()
        assert not a.block[0].emax and not a.block[0].emax_up
    assert len(ran) == 3


@pytest.mark.parametrize("form", ["list", "pairs", "w_up"])
def test_a_kept_call_is_its_weights_own(ran, form):
    """The first weight wide, another not, so that the other is launched as its bf16 twin: a later weight in its place (at its
    object's address too, once it is gone) is another call, and a freed one's call is not run again."""
    k, n, x = 256, 128, tensor(1, 1, 4, 256)
    first, g2 = weight(k, n, wide=True), weight(k, n, wide=True)

    def call(w):
        if form == "w_up":
            linear.matmul(x, first, None, w_up=w, glu=True)
        else:
            linear.matmul(x, [((first, g2), 0), ((w, w), n // 32)] if form == "pairs" else [(first, 0), (w, n // 32)], None)
        ((_, a),) = ran[-1].launches
        at = {"list": a.block[1].w, "pairs": a.block[1].w_up, "w_up": a.block[0].w_up}[form]
        assert at == ttnn.as_bf16_stream(w).t.data_ptr()

    for _ in range(20):
        w = weight(k, n)
        call(w)
        call(w)
        assert ran[-1] is ran[-2]
        del w
    w = weight(k, n)
    call(w)
    kept = ran[-1]
    ttnn.deallocate(w)
    assert not kept.fits(x, None)


def test_options_that_a_kept_call_does_not_hold(ran):
    """Options that are no plain values (a number of another type, whose object is gone after the call) and lists that change
    name no kept call; a residual that is refused is refused beside a kept call too."""
    k, n, x = 256, 128, tensor(1, 1, 4, 256)
    gate, up = weight(k, n), weight(k, n)
    for i in range(40):
        linear.matmul(x, gate, None, w_up=up, glu=True, glu_act=np.int64(i & 1))
        assert ran[-1].launches[0][1].act == i & 1
    scales = [torch.ones(n), torch.ones(n)]
    for t in scales:
        t.__class__ = DeviceScale
    linear.matmul(x, gate, None, w_up=up, glu=True, col_scales=scales)
    other = torch.ones(n)
    other.__class__ = DeviceScale
    scales[1] = other
    linear.matmul(x, gate, None, w_up=up, glu=True, col_scales=scales)
    assert ran[-1].launches[0][1].scale_up == other.data_ptr()
    linear.matmul(x, gate, None, residual=tensor(1, 1, 4, n))
    sharded = tensor(1, 1, 4, n)
    sharded._mc = gate.memory_config()
    with pytest.raises(AssertionError):
        linear.matmul(x, gate, None, residual=sharded)


def test_an_error_zeroes_every_workspace(monkeypatch):
    """A kernel that gave up a wait may leave counters mid-count, in linear's workspaces (one outgrown, which a graph may hold,
    among them) and in a mixture-of-experts layer's: check_status zeroes them all in place."""
    from moe import moe8

    for name in ("_WORKSPACE", "_STATUS"):
        monkeypatch.setattr(linear, name, {})
    for name in ("_OUTGROWN", "_COUNTED"):
        monkeypatch.setattr(linear, name, [])
    monkeypatch.setattr(torch.cuda, "synchronize", lambda *a: None)
    layer, op = {"_ws": {}, "_device": DEVICE}, type("Op", (), {"need": 4096})
    small = linear._workspace(DEVICE, 1 << 20)
    large = linear._workspace(DEVICE, 3 << 20)
    own = moe8._workspace(layer, "gu rows", op)
    assert small is not large
    gone = linear.new_workspace(DEVICE, 64)
    del gone
    for ws in (small, large, own):
        ws.fill_(3)
    linear.check_status(DEVICE)  # (no error: nothing is touched)
    assert all((ws == 3).all() for ws in (small, large, own))
    linear.status_word(DEVICE).fill_(3)
    with pytest.raises(_tkd.TkdError):
        linear.check_status(DEVICE)
    assert not any(ws.any() for ws in (small, large, own)) and not linear.status_word(DEVICE).any()
    assert linear._workspace(DEVICE, 64) is large and moe8._workspace(layer, "gu rows", op) is own
    linear.check_status(DEVICE)


@pytest.mark.parametrize("rows,n,two", [(33, 128, False), (2048, 151936, False), (2048, 1 << 20, False), (512, 1 << 20, True),
                                        (700, 6291456, False), (2049, 4096, True)])
def test_rows_of_wide_outputs_are_launched_as_they_can_be(rows, n, two):
    """More than 32 rows over so many columns that a launch has no counter for every tile of them: fewer rows a launch."""
    panels = -(-n // 128) * (2 if two else 1)
    at = 0
    for row0, m in linear._launch_rows(rows, panels, _tkd.FMT_BFP4, None, None, None):
        assert row0 == at and m >= 1
        at += m
        a, need = _tkd.TkdMatmul(), ctypes.c_uint64()
        a.fmt, a.m, a.k, a.nblocks, a.out_dtype = _tkd.FMT_BFP4, m, 64, 1, _tkd.DT_BF16
        a.epilogue = _tkd.EPI_GLU2 if two else _tkd.EPI_PLAIN
        a.block[0].n = n
        L = _tkd.lib()
        _tkd.check((L.tkd_matmul_workspace if m <= 32 else L.tkd_matmul_rows_workspace)(ctypes.byref(a), ctypes.byref(need)), "workspace")
    assert at == rows


@pytest.mark.parametrize("adjacent", [True, False])
@pytest.mark.parametrize("unit,launches", [(2048, 1), (128, 2)])
def test_records_of_many_columns_are_launched_as_they_can_be(monkeypatch, adjacent, unit, launches):
    """A head's blocks in one launch only as far as it has counters for their units; every block's slots and indices once."""
    made = []
    host = type("Host", (), {"matmul": staticmethod(lambda a, *rest: made.append(_tkd.TkdMatmul.from_buffer_copy(
        (ctypes.c_char * ctypes.sizeof(_tkd.TkdMatmul)).from_address(a))))})
    monkeypatch.setattr(_tkd, "host", lambda: host)
    monkeypatch.setattr(linear, "TOPK_UNIT", unit)
    monkeypatch.setattr(linear, "_workspace", lambda device, need: torch.zeros(1))
    k, n, count = 32, 1 << 20, 3
    L = _tkd.lib()
    streams = torch.zeros(count, L.tkd_packed_bytes(_tkd.FMT_BFP4, k, n), dtype=torch.uint8)
    emaxes = torch.zeros(count, n // 16, dtype=torch.uint8)
    order = range(count) if adjacent else (2, 0, 1)
    mc = linear.sharded_memcfg(DEVICE, k, n)
    weights = tuple(ttnn.Weight(streams[i], emaxes[i], k, n, ttnn.bfloat4_b, DEVICE, mc) for i in order)
    units = linear.topk_units(n)
    r = tensor(1, 1, count * units, 2, dtype=ttnn.uint32)
    topk = {"r": r, "k": 1, "rows": 1, "slot0": 5, "base": 7, "n": n}
    for _ in range(2):
        linear.records_together(tensor(1, 1, 1, k), weights, topk, tensor(1, 1, 1, n))
    assert len(made) == 2 * launches
    got = []
    for a in made[: len(made) // 2]:
        for b in range(max(a.nblocks, a.repeats)):
            at = a.block[0].w + b * streams.shape[1] if a.repeats else a.block[b].w
            got.append((at, a.topk_slot0 + b * units, a.topk_base + b * n))
    assert got == [(w.t.data_ptr(), 5 + b * units, 7 + b * n) for b, w in enumerate(weights)]


def test_settings_given_as_arrays(monkeypatch):
    """head_pick.pick and moe8.route keep their checked settings by value: numbers given as arrays and tensors serve as before, and
    an array changed in place is read anew."""
    from lm_head_topk import head_pick
    from moe import moe8

    made = []
    host = type("Host", (), {"pick": staticmethod(lambda *a: made.append(a[5])), "route": staticmethod(lambda *a: made.append(a[5]))})
    monkeypatch.setattr(_tkd, "host", lambda: host)
    records, x = tensor(1, 1, 4, 16, dtype=ttnn.uint32), tensor(1, 1, 1, 64)
    rows_t = ttnn.Tensor(torch.zeros(1, 1, 128, 64, dtype=torch.bfloat16), ttnn.bfloat16, ttnn.ROW_MAJOR_LAYOUT, DEVICE, None)
    valid = np.array(100)
    for v in (100, 90):
        valid[...] = v
        head_pick.pick(records, x, rows_t, 1, 8, valid=valid)
        assert made[-1][4] == v
    logits, ids, w = tensor(1, 1, 1, 64, dtype=ttnn.float32), tensor(1, 1, 1, 8, dtype=ttnn.uint16), tensor(1, 1, 1, 8)
    bias, scale = tensor(1, 1, 1, 64, dtype=ttnn.float32), torch.tensor(1.0)
    for v in (1.0, 2.5):
        scale.fill_(v)
        moe8.route(logits, ids, w, 8, kind="sigmoid", bias=bias, scale=scale, groups=np.array([4, 2]))
        assert made[-1][4] == v and made[-1][6:8] == (4, 2)


def test_records_together_refuses_what_matmul_refuses(monkeypatch):
    monkeypatch.setattr(_tkd, "host", lambda: type("Host", (), {"matmul": staticmethod(lambda *a: None)}))
    weights = (weight(64, 128), weight(64, 128))
    topk = {"r": tensor(1, 1, 2, 2, dtype=ttnn.uint32), "k": 1, "rows": 1, "slot0": 0, "base": 0, "n": 128}
    x, out = tensor(1, 1, 1, 64), tensor(1, 1, 1, 128)
    x._mc = weights[0].memory_config()
    with pytest.raises(AssertionError):
        linear.records_together(x, weights, topk, out)
    monkeypatch.setattr(linear.dev, "MAX_BANKS", 4)
    with pytest.raises(ValueError):
        linear.records_together(tensor(1, 1, 1, 64), weights, topk, out)


@pytest.mark.parametrize("m", [33, 64, 300])
def test_fixed_sums_are_slices_of_32_rows(ran, m):
    w, x = weight(256, 128), tensor(1, 1, m, 256)
    linear.matmul(x, w, None)
    assert [a.m for _, a in ran[-1].launches] == [m]
    linear.matmul(x, w, None, fixed_sums=True)
    assert [(at, a.m) for at, a in ran[-1].launches] == [(at, min(32, m - at)) for at in range(0, m, 32)]
    linear.matmul(x, w, None, fixed_sums=False)
    assert [a.m for _, a in ran[-1].launches] == [m]


def test_a_moe_layers_workspaces_go_by_slot(monkeypatch):
    """Calls on one layer that may overlap pick their workspaces as linear's do: gate_up_rows counts in one too."""
    from moe import moe8

    monkeypatch.setattr(linear, "_COUNTED", [])
    layer, op = {"_ws": {}, "_device": DEVICE}, type("Op", (), {"need": 4096})
    own = {}
    for slot in (0, 1, 0, 1):
        monkeypatch.setattr(linear, "WORKSPACE_SLOT", slot)
        for what in ("gu rows", "dn rows", "dn"):
            ws = moe8._workspace(layer, what, op)
            assert own.setdefault((slot, what), ws) is ws
    assert len({ws.data_ptr() for ws in own.values()}) == 6


def test_prompts_of_many_lengths_leave_the_decode_calls(ran):
    """A weight keeps so many calls; a new one takes the oldest prompt's place, and the oldest's where there is none."""
    w = weight(64, 128)
    xs = [tensor(1, 1, m, 64) for m in (1, 8, *range(33, 133))]
    for x in xs:
        linear.matmul(x, w, None)
    assert len(w.calls) == linear._WEIGHT_CALLS
    decode = ran[:2]
    for x in xs[:2]:
        linear.matmul(x, w, None)
    assert ran[-2:] == decode and ran[-3].launches[0][1].m == 132
    linear.matmul(xs[-linear._WEIGHT_CALLS + 2], w, None)
    assert ran[-1] in ran[:-1]
    for col0 in range(2 * linear._WEIGHT_CALLS):
        linear.matmul(xs[0], w, None, out=tensor(1, 1, 1, 32 * (col0 + 4)), col0=col0)
    assert len(w.calls) == linear._WEIGHT_CALLS and all(c.launches[0][1].m == 1 for c in w.calls.values())


def test_matmul_host_sees_a_list_and_a_dict_change(ran, monkeypatch):
    """matmul_host's calls go by what a block list and a top-k's dict hold, not by the list and the dict."""
    made = []
    lib = _tkd.lib()
    stream = type("Stream", (), {"cuda_stream": 0})

    class Lib:
        def __getattr__(self, name):
            return getattr(lib, name)

        def tkd_matmul_host(self, a, x, out, sp):
            made.append(_tkd.TkdMatmul.from_buffer_copy(a._obj))
            return 0

    monkeypatch.setattr(_tkd, "lib", lambda: Lib())
    monkeypatch.setattr(torch.cuda, "stream", lambda s: contextlib.nullcontext())
    monkeypatch.setattr(linear, "_CALLS", {})
    monkeypatch.setattr(linear, "_WORKSPACE", {})
    x, out, host = tensor(1, 1, 1, 64), tensor(1, 1, 1, 256), torch.zeros(1, 64, dtype=torch.bfloat16)
    ws = [weight(64, 128) for _ in range(3)]
    entries = [(ws[0], 0), (ws[1], 4)]
    topk = {"r": tensor(1, 1, 4, 2, dtype=ttnn.uint32), "k": 1, "rows": 1, "slot0": 0, "base": 0, "n": 128}

    def call(w, **kw):
        linear.matmul_host(host, host, x, w, None, out=out, stream=stream, **kw)
        return made[-1]

    assert call(entries).block[1].w == ws[1].t.data_ptr()
    entries[1] = (ws[2], 4)
    assert call(entries).block[1].w == ws[2].t.data_ptr()
    assert call(ws[0], topk=topk).topk_slot0 == 0
    topk["slot0"] = 3
    assert call(ws[0], topk=topk).topk_slot0 == 3
    assert len(linear._CALLS) == 4 and call(entries).block[1].w == ws[2].t.data_ptr() and len(linear._CALLS) == 4


def test_the_log_and_the_plans_are_of_what_runs(ran, monkeypatch, capsys):
    """A call of more than 32 rows in one launch makes no plans of slices and logs none; its options are checked all the same."""
    w, x = weight(256, 128), tensor(1, 1, 512, 256)
    monkeypatch.setattr(linear, "LOG", True)
    monkeypatch.setattr(linear, "_CHOICE", {})
    linear.matmul(x, w, None)
    assert [type(v) for v in linear._CHOICE.values()] == [dict] and "rows 512: 1 launch(es)" in capsys.readouterr().out
    with pytest.raises(ValueError):
        linear.matmul(x, w, None, kb=3)
    linear.matmul(x, w, None, fixed_sums=True)
    assert len(linear._CHOICE) == 2 and "ctas" in capsys.readouterr().out


def test_linears_own_arguments_find_the_kept_call(ran, monkeypatch):
    """linear.linear without options goes straight to the call its weight keeps: the same one for the same arguments, another for
    another scale, activation, output type, shape or setting, none of a freed or moved tensor's; the described calls stay 64."""
    w, x = weight(64, 128), tensor(1, 1, 3, 64)
    scales = [ttnn.Tensor(torch.ones(1, 1, 1, 128, dtype=torch.bfloat16), ttnn.bfloat16, ttnn.TILE_LAYOUT, DEVICE, None) for _ in range(2)]
    seen = []
    for args in ({"scale": None}, {"scale": scales[0]}, {"scale": scales[1]}, {"scale": None, "activation": "silu"},
                 {"scale": None, "activation": "swiglu"}, {"scale": None, "out_dtype": ttnn.float32}, {"scale": scales[0], "activation": "silu"}):
        for _ in range(3):
            linear.linear(x, w, **args)
        assert ran[-1] is ran[-2] is ran[-3] and ran[-1] not in seen
        seen.append(ran[-1])
    assert ran[-1].launches[0][1].epilogue == _tkd.EPI_SILU and len(w.calls) == len(w.short) == len(seen)
    linear.linear(tensor(1, 1, 4, 64), w, None)
    assert ran[-1] not in seen
    monkeypatch.setattr(linear, "MAX_CTAS", 5)
    linear.linear(x, w, None)
    assert ran[-1] not in seen and ran[-1].launches[0][1].max_ctas == 5
    monkeypatch.setattr(linear, "MAX_CTAS", None)
    linear.linear(x, w, scales[0])
    assert ran[-1] is seen[1]
    scales[0].t = torch.ones(1, 1, 1, 256, dtype=torch.bfloat16)[..., :128]  # (moved; some tensor freed)
    monkeypatch.setattr(ttnn, "EPOCH", ttnn.EPOCH + 1)
    linear.linear(x, w, scales[0])
    assert ran[-1] not in seen and ran[-1].launches[0][1].scale == scales[0].t.data_ptr()
    with pytest.raises(AssertionError):
        linear.linear(x, w, None, activation="relu")
    with pytest.raises(AssertionError):
        linear.linear(x, w, None, out_dtype=ttnn.uint32)
    for m in range(1, 2 * linear._WEIGHT_CALLS):
        linear.linear(tensor(1, 1, m, 64), w, None)
    assert len(w.calls) <= linear._WEIGHT_CALLS and len(w.short) <= linear._WEIGHT_CALLS


@pytest.mark.parametrize("out_dtype", [None, ttnn.bfloat16, ttnn.float32])
@pytest.mark.parametrize("activation", [None, "silu", "swiglu", "geglu", "relu", ""])
@pytest.mark.parametrize("scaled", [False, True])
def test_a_repeated_linear_gives_what_the_first_gave(ran, monkeypatch, activation, out_dtype, scaled):
    """linear.linear three times with the same arguments, for every activation and output type: equal outputs, the activation among
    them, or a refusal each time. The launch is stood in for by the product 2 with what its output stage adds."""
    act = lambda v, which: torch.nn.functional.silu(v) if which == 0 else torch.nn.functional.gelu(v, approximate="tanh")  # noqa: E731

    def run(call, x, out, residual):
        ran.append(call)
        a = call.launches[0][1]
        v = torch.full((1, 1, x.t.shape[-2], a.ldo), 2.0)
        return act(v, 0) if a.epilogue == _tkd.EPI_SILU else act(v, a.act) * 2.0 if a.epilogue == _tkd.EPI_GLU_IL else v

    monkeypatch.setattr(linear._Call, "run", run)
    # (the first call's launch writes into a tensor made before it: described calls return that one)
    described = linear._described

    def with_output(*args):
        y, call = described(*args)
        return ttnn.Tensor(run(call, args[0], None, None), y.dtype, y.layout, y._device, y._mc), call

    monkeypatch.setattr(linear, "_described", with_output)
    w, x = weight(64, 128), tensor(1, 1, 3, 64)
    scale = ttnn.Tensor(torch.ones(1, 1, 1, 128, dtype=torch.bfloat16), ttnn.bfloat16, ttnn.TILE_LAYOUT, DEVICE, None) if scaled else None
    two = torch.tensor(2.0)
    want = {None: two, "silu": act(two, 0), "swiglu": act(two, 0) * 2, "geglu": act(two, 1) * 2}.get(activation)
    if want is None or (scaled and activation in ("swiglu", "geglu")) or (out_dtype == ttnn.float32 and (scaled or activation in ("swiglu", "geglu"))):
        for _ in range(3):
            with pytest.raises(AssertionError):
                linear.linear(x, w, scale, activation=activation, out_dtype=out_dtype)
        return
    for _ in range(3):
        y = linear.linear(x, w, scale, activation=activation, out_dtype=out_dtype)
        assert y.dtype == (out_dtype or ttnn.bfloat16)
        assert torch.equal(y.t, torch.full_like(y.t, float(want))), (activation, out_dtype)
