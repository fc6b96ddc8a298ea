"""Parity of the CUDA path with the CPU oracle, through the package's API (which calls libtkd's C-ABI): bit-exact for
the quantiser, the packed weights' held values and the top-k indices; 1e-2 relative (compared in bf16) for the sums."""

from pathlib import Path

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from common import ttnn_like as ttnn  # noqa: E402
from dense_reader import linear  # noqa: E402
from oracle import oracle as orc  # noqa: E402

DT = {"bfp8": ttnn.bfloat8_b, "bfp4": ttnn.bfloat4_b, "bf16": ttnn.bfloat16}
GOLDEN = Path(__file__).resolve().parent / "golden"


def dev_x(device, x):
    return ttnn.from_torch(x.reshape(1, 1, *x.shape).to(torch.bfloat16), dtype=ttnn.bfloat16, layout=ttnn.TILE_LAYOUT,
                           device=device)


def host(y):
    return ttnn.to_torch(y).float().reshape(-1, y.shape[-1])


def close_bf16(got, want, tol=1e-2):
    """|got - want| within tol relative to the row's scale, both seen in bf16."""
    g, w = got.to(torch.bfloat16).float(), torch.as_tensor(want).to(torch.bfloat16).float()
    scale = w.abs().amax(dim=-1, keepdim=True).clamp(min=1e-30)
    err = ((g - w).abs() / scale).max().item()
    assert err < tol, err


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4", "bf16"])
@pytest.mark.parametrize("k,n", [(64, 32), (96, 48), (1024, 2048), (4096, 1024 + 16)])
def test_held_values_bit_exact(device, fmt, k, n):
    g = torch.Generator().manual_seed(k * 7 + n)
    w = torch.randn(n, k, generator=g) * 0.02 * torch.exp2(torch.randint(-6, 7, (n, 1), generator=g).float())
    w[0] = 0
    w[3, 5], w[7 % n, 9] = 0.0, -1e-30
    n_ok = n if n % 32 == 0 else n  # (native_weight takes any N; the stream pads to 16)
    tw, _ = linear.native_weight(device, w, DT[fmt])
    got = ttnn.to_torch(tw)[0, 0, :, :n_ok].numpy()
    want = orc.block_float(w.T.contiguous().numpy(), fmt)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    # padded columns hold zeros
    assert not ttnn.to_torch(tw)[0, 0, :, n_ok:].any()


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4"])
def test_col_scale_and_block_float(device, fmt):
    g = torch.Generator().manual_seed(11)
    w = torch.randn(256, 128, generator=g) * 0.02
    w[:100] *= 40
    tw, ts = linear.native_weight(device, w, DT[fmt], col_scale=True)
    want_w, want_c = orc.native_values(w, fmt, col_scale=True)
    assert np.array_equal(ttnn.to_torch(tw)[0, 0, :, :256].numpy().view(np.uint32), want_w.view(np.uint32))
    assert np.array_equal(ttnn.to_torch(ts).float().reshape(-1).numpy(), want_c)
    t = torch.randn(2, 64, 96, generator=g)
    got = linear.block_float(t, DT[fmt])
    for i in range(2):
        assert np.array_equal(got[i].numpy().view(np.uint32), orc.block_float(t[i].numpy(), fmt).view(np.uint32))


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4"])
def test_wide_weight_runs(device, fmt):
    """A weight whose exponents inside a group of 16 columns spread further than the block-float stream encodes (the
    reference takes any float matrix, linear.py:144-156): here a dead input channel of 1e-17-size noise beside
    0.02-size rows, and the quantiser golden file's wide-spread matrix (zeros, denormals, huge values). The weight holds
    the oracle's values bit for bit and the matmul matches the oracle, also when only the tiny rows see activations."""
    g = torch.Generator().manual_seed(66)
    n, k = 256, 512
    w = torch.randn(n, k, generator=g) * 0.02
    w[:, 7] = torch.randn(n, generator=g) * 1e-17
    tw, _ = linear.native_weight(device, w, DT[fmt])
    assert tw.wide and tw.dtype == DT[fmt]
    wk = orc.native_values(w, fmt)[0]
    assert np.array_equal(ttnn.to_torch(tw)[0, 0, :, :n].numpy().view(np.uint32), wk.view(np.uint32))
    x = torch.randn(3, k, generator=g)
    x[1] = 0
    x[1, 7] = 3.0   # only the dead channel: the sums are of 1e-17 size
    x[2, 7] = 2.0 ** 60
    y = host(linear.matmul(dev_x(device, x), tw, None))
    want = orc.matmul_f64(x, wk)
    close_bf16(y, want)
    assert y[1].abs().max() > 0
    # a block list with a weight that is not wide: one launch, one stream format
    w2 = torch.randn(128, k, generator=g) * 0.02
    t2, _ = linear.native_weight(device, w2, DT[fmt])
    assert not t2.wide
    both = host(linear.matmul(dev_x(device, x), [(tw, 0), (t2, n // 32)], None))
    assert torch.equal(both[:, :n], y)
    close_bf16(both[:, n:], orc.matmul_f64(x, orc.native_values(w2, fmt)[0]))
    if fmt == "bfp4":
        gold = np.load(GOLDEN / "quantiser_bfp4.npz")
        w4 = torch.from_numpy(gold["w4"].astype(np.float32))  # [K, N]
        t4 = ttnn.from_torch(w4, dtype=ttnn.bfloat4_b, device=device)
        held = ttnn.to_torch(t4)[0, 0, :, : w4.shape[1]].numpy()
        assert np.array_equal(held.view(np.uint32), orc.block_float(w4.numpy(), "bfp4").view(np.uint32))
    linear.check_status(device)


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4"])
@pytest.mark.parametrize("m", [1, 16, 64])
@pytest.mark.parametrize("which", ["gate", "up"])
def test_wide_gate_or_up_weight(device, fmt, m, which):
    """Two weights of which one is wide (a bf16 stream) and one is not: one launch streams both as bf16."""
    g = torch.Generator().manual_seed(67 + m)
    n, k = 192, 512
    w = [torch.randn(n, k, generator=g) * 0.02 for _ in range(2)]
    w[which == "up"][:, 7] = torch.randn(n, generator=g) * 1e-17
    gate, up = (linear.native_weight(device, v, DT[fmt])[0] for v in w)
    assert (gate.wide, up.wide) == (which == "gate", which == "up")
    x = torch.randn(m, k, generator=g)
    G, U = (torch.from_numpy(orc.matmul_f64(x, orc.native_values(v, fmt)[0])) for v in w)
    want = (torch.nn.functional.silu(G) * U).numpy()
    for _ in range(2):  # (described, then kept)
        close_bf16(host(linear.matmul(dev_x(device, x), gate, None, w_up=up, glu=True)), want)
    close_bf16(host(linear.linear(dev_x(device, x), (gate, up), None, activation="swiglu")), want)
    linear.check_status(device)


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4", "bf16"])
@pytest.mark.parametrize("m", [1, 4, 8, 13, 32])
def test_matmul_against_oracle(device, fmt, m):
    k, n = 2048 + 32, 1024 + 32  # K not a multiple of the slice, N not of the panel
    g = torch.Generator().manual_seed(100 + m)
    w = torch.randn(n, k, generator=g) * 0.02
    x = torch.randn(m, k, generator=g)
    tw, _ = linear.native_weight(device, w, DT[fmt])
    wk, _ = orc.native_values(w, fmt)
    y = host(linear.matmul(dev_x(device, x), tw, None))
    assert y.shape == (m, n)
    want = orc.matmul_f64(x, wk)
    close_bf16(y, want)
    linear.check_status(device)


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4", "bf16"])
@pytest.mark.parametrize("m,n", [(9, 1024 + 16), (17, 1024 + 128), (32, 2048 + 80)])
def test_many_rows_epilogues_against_oracle(device, fmt, m, n):
    """The kernel for 9 to 32 rows: every epilogue, N with a ragged last panel, K with a short last slice."""
    k = 1024 + 96
    g = torch.Generator().manual_seed(7 * m + n)
    w, w2 = torch.randn(n, k, generator=g) * 0.02, torch.randn(n, k, generator=g) * 0.02
    x = torch.randn(m, k, generator=g)
    tx = dev_x(device, x)
    tw, _ = linear.native_weight(device, w, DT[fmt])
    tw2, _ = linear.native_weight(device, w2, DT[fmt])
    wk, _ = orc.native_values(w, fmt)
    wk2, _ = orc.native_values(w2, fmt)
    plain = orc.matmul_f64(x, wk)
    close_bf16(host(linear.matmul(tx, tw, None)), plain)
    # fp32 output with an fp32 residual
    res = torch.randn(m, n, generator=g)
    tr = ttnn.from_torch(res.reshape(1, 1, m, n), dtype=ttnn.float32, layout=ttnn.TILE_LAYOUT, device=device)
    y32 = host(linear.matmul(tx, tw, None, residual=tr, out32=True)).double().numpy()
    np.testing.assert_allclose(y32, plain + res.double().numpy(), rtol=2e-3, atol=2e-3)
    # bf16 residual
    resb = res.to(torch.bfloat16)
    trb = ttnn.from_torch(resb.reshape(1, 1, m, n), dtype=ttnn.bfloat16, layout=ttnn.TILE_LAYOUT, device=device)
    close_bf16(host(linear.matmul(tx, tw, None, residual=trb)), plain + resb.double().numpy())
    # column scales
    sc = (torch.rand(n, generator=g) + 0.5).to(torch.bfloat16)
    close_bf16(host(linear.matmul(tx, tw, linear.scale_tensor(device, sc.float()))), plain * sc.double().numpy()[None, :])
    # SwiGLU from two weights
    gate, up = torch.from_numpy(plain), torch.from_numpy(orc.matmul_f64(x, wk2))
    close_bf16(host(linear.matmul(tx, tw, None, w_up=tw2, glu=True)), (torch.nn.functional.silu(gate) * up).numpy())
    linear.check_status(device)


@pytest.mark.parametrize("m", [9, 12, 13])
def test_a_panels_sums_as_large_as_the_ring(device, m):
    """9 to 12 rows of a panel of 24 slices, a CTA each: their sums, three lots of four rows a slice, take the whole of the ring
    that they are added up in (72 times 2 KB), and the lots are read in pairs."""
    g = torch.Generator().manual_seed(68 + m)
    n, k = 128, 24 * 512
    w, x = torch.randn(n, k, generator=g) * 0.02, torch.randn(m, k, generator=g)
    tw, _ = linear.native_weight(device, w, ttnn.bfloat4_b)
    plan = linear.plan(device, dev_x(device, x), tw, noscale=True, ks=512)
    assert (plan["SLICES"], plan["PANELS"], plan["GRID"]) == (24, 1, 24)
    close_bf16(host(linear.matmul(dev_x(device, x), tw, None, ks=512)), orc.matmul_f64(x, orc.native_values(w, "bfp4")[0]))
    linear.check_status(device)


def test_config_shapes_full_size(device):
    """The benchmark configurations at their own sizes against the oracle over every column: the README example
    (one token through a [4096, 2048] bfloat8_b weight), the MLP gate/up pair (two [14336, 4096] bfloat4_b weights,
    float32 column scales, SwiGLU; as two weights and as one interleaved weight) and the down projection ([4096, 14336]
    bfloat8_b, float32 residual and output) at 1, 8 and 32 rows."""
    g = torch.Generator().manual_seed(0)
    w = torch.randn(4096, 2048, generator=g) * 0.02
    x = torch.randn(1, 2048, generator=g)
    tw, _ = linear.native_weight(device, w, ttnn.bfloat8_b)
    close_bf16(host(linear.matmul(dev_x(device, x), tw, None)), orc.matmul_f64(x, orc.native_values(w, "bfp8")[0]))
    # the gate/up pair: silu((x Wg) sg) * ((x Wu) su), bfloat4_b
    k, n = 4096, 14336
    wg, wu = torch.randn(n, k, generator=g) * 0.02, torch.randn(n, k, generator=g) * 0.02
    sg, su = torch.rand(n, generator=g) + 0.5, torch.rand(n, generator=g) + 0.5
    x = torch.randn(1, k, generator=g)
    tg, _ = linear.native_weight(device, wg, ttnn.bfloat4_b)
    tu, _ = linear.native_weight(device, wu, ttnn.bfloat4_b)
    cs = (sg.to(device.torch), su.to(device.torch))
    y = host(linear.matmul(dev_x(device, x), tg, None, w_up=tu, glu=True, col_scales=cs))
    assert y.shape == (1, n)
    ag = orc.matmul_f64(x, orc.native_values(wg, "bfp4")[0])
    au = orc.matmul_f64(x, orc.native_values(wu, "bfp4")[0])
    close_bf16(y, orc.epilogue(ag, 2, acc2=au, scale=sg.numpy(), scale2=su.numpy()))
    # the same through an interleaved weight
    ti, _ = linear.native_weight(device, linear.interleave_glu(wg, wu), ttnn.bfloat4_b)
    si = linear.interleave_glu(sg[:, None], su[:, None]).reshape(-1).to(device.torch)
    y2 = host(linear.matmul(dev_x(device, x), ti, None, glu=True, col_scales=si))
    assert torch.equal(y, y2)
    del tg, tu, ti, wg, wu
    # the down projection: x W^T + residual in float32
    k, n = 14336, 4096
    w = torch.randn(n, k, generator=g) * 0.02
    tw, _ = linear.native_weight(device, w, ttnn.bfloat8_b)
    wk = orc.native_values(w, "bfp8")[0]
    for m in (1, 8, 32):
        x = torch.randn(m, k, generator=g)
        res = torch.randn(m, n, generator=g)
        tr = ttnn.from_torch(res.reshape(1, 1, m, n), dtype=ttnn.float32, layout=ttnn.TILE_LAYOUT, device=device)
        y = linear.matmul(dev_x(device, x), tw, None, residual=tr, out32=True)
        want = orc.epilogue(orc.matmul_f64(x, wk), 4, res32=res.numpy())
        got = host(y)[:m]
        assert got.dtype == torch.float32
        close_bf16(got, want)
        rel = ((got.double() - torch.from_numpy(want)).norm() / torch.from_numpy(want).norm()).item()
        assert rel < 1e-5, rel
    linear.check_status(device)


def test_lm_head_full_size(device):
    """The LM head at its own size: x [1, 4096] through a [151936, 4096] bfloat8_b weight, one top-8 record per 2048
    columns (74 full units and one of 384 columns), then the best 32 of them all. Every record equals the oracle's
    canonical top-k of the call's own bf16 outputs bit for bit, the merged 32 equal the oracle's merge of those
    records (and the canonical top-32 of the whole row), and the outputs match the oracle's sums over every column."""
    k, n, kk, top = 4096, 151936, 8, 32
    g = torch.Generator().manual_seed(5)
    w = torch.randn(n, k, generator=g) * 0.02
    x = torch.randn(1, k, generator=g)
    tw, _ = linear.native_weight(device, w, ttnn.bfloat8_b)
    units = linear.topk_units(n)
    assert units == 75
    r = linear.topk_result(device, units, 1, kk)
    out = ttnn.allocate_tensor_on_device([1, 1, 1, n], ttnn.bfloat16, ttnn.TILE_LAYOUT, device)
    spec = {"r": r, "k": kk, "rows": 1, "slot0": 0, "base": 0, "n": n, "write_y": True}
    tx = dev_x(device, x)
    linear.matmul(tx, tw, None, topk=spec, out=out)
    merged = linear.topk_merge(r, 1, kk, top)
    linear.check_status(device)
    y = host(out)
    rec = ttnn.to_torch(r).reshape(units, 2, 1, kk).numpy().view(np.uint32)
    bits = orc.bf16_bits(y[0])
    for u in range(units):
        c0, c1 = u * 2048, min((u + 1) * 2048, n)
        keys, idx = orc.topk_canonical(bits[c0:c1], c1 - c0, kk, c0)
        assert np.array_equal(rec[u, 0, 0], keys), u
        assert np.array_equal(rec[u, 1, 0], idx), u
    got = ttnn.to_torch(merged).numpy().view(np.uint32).reshape(2, 1, top)
    assert np.array_equal(got, orc.topk_merge_ref(rec, 1, kk, top))
    keys, idx = orc.topk_canonical(bits, n, top, 0)
    assert np.array_equal(got[0, 0], keys) and np.array_equal(got[1, 0], idx)
    # the same records with write_y False (the outputs stay in the call's scratch buffer)
    r2 = linear.topk_result(device, units, 1, kk)
    linear.matmul(tx, tw, None, topk={**spec, "r": r2, "write_y": False}, out=out)
    assert torch.equal(ttnn.to_torch(r2), ttnn.to_torch(r))
    del tw
    wk = orc.native_values(w, "bfp8")[0]
    close_bf16(y, orc.matmul_f64(x, wk))
    linear.check_status(device)


def test_records_as_bfloat16(device):
    """RECORDS_BF16 (the reference's linear.py:77-78, 775-778): the result tensor is bfloat16 with the same bytes as
    the uint32 words. The op, the host decode, the device merge and the LM head's pick take it unchanged."""
    from lm_head_topk import head_pick

    k, n, kk, rows = 1024, 2048 * 2 + 384, 8, 2
    g = torch.Generator().manual_seed(51)
    w = torch.randn(n, k, generator=g) * 0.02
    x = torch.randn(rows, k, generator=g)
    tw, _ = linear.native_weight(device, w, ttnn.bfloat8_b)
    tx = dev_x(device, x)
    units = linear.topk_units(n)
    spec = {"k": kk, "rows": rows, "slot0": 0, "base": 0, "n": n, "write_y": True}
    r32 = linear.topk_result(device, units, rows, kk)
    linear.matmul(tx, tw, None, topk={**spec, "r": r32})
    linear.RECORDS_BF16 = True
    try:
        r16 = linear.topk_result(device, units, rows, kk)
        assert r16.dtype == ttnn.bfloat16 and r16.shape[-1] == 4 * rows * kk
        linear.matmul(tx, tw, None, topk={**spec, "r": r16})
        a, b = ttnn.to_torch(r16), ttnn.to_torch(r32)
        assert torch.equal(a.contiguous().view(torch.int32).reshape(-1), b.reshape(-1))
        v16, i16 = linear.topk_records(r16, rows, kk)
        v32, i32 = linear.topk_records(r32, rows, kk)
        assert torch.equal(v16, v32) and torch.equal(i16, i32)
        m16 = linear.topk_merge(r16, rows, kk, 32)
        assert m16.dtype == ttnn.bfloat16
    finally:
        linear.RECORDS_BF16 = False
    m32 = linear.topk_merge(r32, rows, kk, 32)
    assert torch.equal(ttnn.to_torch(m16).contiguous().view(torch.int32).reshape(-1), ttnn.to_torch(m32).reshape(-1))
    p16 = ttnn.to_torch(head_pick.pick_records(r16, rows, kk, n))
    p32 = ttnn.to_torch(head_pick.pick_records(r32, rows, kk, n))
    assert torch.equal(p16.reshape(32, 32)[:rows, :3], p32.reshape(32, 32)[:rows, :3])
    linear.check_status(device)


def test_block_list_config4(device):
    """One launch over an attention layer's four projections (config 4) equals one call per weight, bit for bit, and
    matches the oracle."""
    k = 4096
    g = torch.Generator().manual_seed(40)
    shapes = [(4096, 0), (1024, 128), (1024, 160), (4096, 192)]
    ws = [torch.randn(n, k, generator=g) * 0.02 for n, _ in shapes]
    tws = [linear.native_weight(device, w, ttnn.bfloat8_b)[0] for w in ws]
    for m in (1, 4):
        x = torch.randn(m, k, generator=g)
        tx = dev_x(device, x)
        one = host(linear.matmul(tx, [(tw, c0) for tw, (_, c0) in zip(tws, shapes)], None))
        assert one.shape == (m, 32 * 192 + 4096)
        for tw, w, (n, c0) in zip(tws, ws, shapes):
            own = host(linear.matmul(tx, tw, None))
            assert torch.equal(one[:, 32 * c0 : 32 * c0 + n], own)
            close_bf16(own, orc.matmul_f64(x, orc.native_values(w, "bfp8")[0]))
    linear.check_status(device)


def test_topk_indices_exact(device):
    """Top-k candidate indices equal the oracle's canonical order (key descending, lower index first among ties) on
    the op's own bf16 outputs, including heavy ties, a last partial unit and write_y False."""
    k, n = 1024, 2048 * 2 + 384
    g = torch.Generator().manual_seed(50)
    w = (torch.randn(n, k, generator=g) * 4).round() / 64  # few distinct values: many exact ties in y
    x = (torch.randn(2, k, generator=g) * 2).round()
    tw, _ = linear.native_weight(device, w, ttnn.bfloat8_b)
    tx = dev_x(device, x)
    y = host(linear.matmul(tx, tw, None))
    units, kk, rows = 3, 8, 2
    for n_valid, base, write_y in ((n, 0, True), (n - 100, 5000, False)):
        r = linear.topk_result(device, units + 1, rows, kk)
        spec = {"r": r, "k": kk, "rows": rows, "slot0": 1, "base": base, "n": n_valid, "write_y": write_y}
        out = ttnn.from_torch(torch.full((1, 1, 2, n), -7.0, dtype=torch.bfloat16), dtype=ttnn.bfloat16,
                              layout=ttnn.TILE_LAYOUT, device=device)
        linear.matmul(tx, tw, None, topk=spec, out=out)
        if write_y:
            assert torch.equal(host(out), y)
        else:
            assert bool((host(out) == -7.0).all())  # never written
        rec = ttnn.to_torch(r).reshape(units + 1, 2, rows, kk).numpy().view(np.uint32)
        assert not rec[0].any()  # slot 0 untouched
        for u in range(units):
            for t in range(rows):
                c0, c1 = u * 2048, min((u + 1) * 2048, n_valid)
                keys, idx = orc.topk_canonical(orc.bf16_bits(y[t, c0:c1]), c1 - c0, kk, base + c0)
                assert np.array_equal(rec[1 + u, 0, t], keys), (u, t)
                assert np.array_equal(rec[1 + u, 1, t], idx), (u, t)
    linear.check_status(device)


@pytest.mark.parametrize("nrec,rows,k,top", [(75, 1, 8, 32), (7, 4, 8, 32), (300, 2, 16, 64), (3, 1, 4, 32)])
def test_topk_merge_exact(device, nrec, rows, k, top):
    """The device merge of records (any rank's, gathered) equals the oracle's: key descending, lower index first among
    the many equal keys, empty slots skipped, fewer candidates than `top` leave empty slots."""
    g = np.random.default_rng(nrec * 31 + rows)
    words = np.zeros((nrec, 2, rows, k), np.uint32)
    words[:, 0] = g.integers(0x8000, 0x8040, size=(nrec, rows, k))  # 64 distinct keys: heavy ties
    words[:, 0][g.random((nrec, rows, k)) < 0.2] = 0                 # empty slots
    words[:, 1] = g.permutation(nrec * rows * k).reshape(nrec, rows, k).astype(np.uint32) + 1000
    words[:, 1][words[:, 0] == 0] = 0xFFFFFFFF
    r = linear.topk_result(device, nrec, rows, k)
    r.t.copy_(torch.from_numpy(words.view(np.int32)).reshape(r.t.shape))
    got = ttnn.to_torch(linear.topk_merge(r, rows, k, top)).numpy().view(np.uint32).reshape(2, rows, top)
    assert np.array_equal(got, orc.topk_merge_ref(words, rows, k, top))
    linear.check_status(device)


def test_packed_weight_cache_round_trip(device, tmp_path):
    """A weight loaded from its cache directory is the packed weight bit for bit (stream, side array, scales), gives
    the same outputs, and a cache of other weights is refused."""
    from dense_reader import cache

    g = torch.Generator().manual_seed(77)
    w = torch.randn(384, 256, generator=g) * 0.02
    for fmt, col_scale in ((ttnn.bfloat8_b, True), (ttnn.bfloat4_b, False), (ttnn.bfloat16, False)):
        path = tmp_path / f"w_{fmt}"
        tw, ts = cache.native_weight_cached(device, w, fmt, path, col_scale=col_scale)   # packs and writes
        tw2, ts2 = cache.native_weight_cached(device, w, fmt, path, col_scale=col_scale)  # loads
        assert torch.equal(tw.t, tw2.t) and (tw.emax is None or torch.equal(tw.emax, tw2.emax))
        assert torch.equal(ts.t, ts2.t)
        tx = dev_x(device, torch.randn(3, 256, generator=g))
        assert torch.equal(host(linear.matmul(tx, tw, ts)), host(linear.matmul(tx, tw2, ts2)))
        other = torch.randn(384, 256, generator=g) * 0.02
        with pytest.raises(cache.PackCacheMismatch):
            cache.native_weight_cached(device, other, fmt, path, col_scale=col_scale)
        tw3, _ = cache.native_weight_cached(device, other, fmt, path, col_scale=col_scale, rebuild=True)
        assert not torch.equal(tw3.t, tw.t)
        tw4, _ = cache.native_weight_cached(device, other, fmt, path, col_scale=col_scale)  # the rebuilt cache, loaded
        assert torch.equal(tw4.t, tw3.t)


def test_full_size_properties(device):
    """At the benchmark configurations' full sizes (the gate weight, 14336 x 4096 bfloat4_b; the down projection's 4096 x 14336 bfloat8_b)
    the oracle is too slow for every column; size-independent properties stand in: linearity in x (power-of-two
    scaling is exact), a zero row of x gives zeros, columns of a sub-matrix equal the same columns computed alone,
    and a sample of columns against the oracle."""
    g = torch.Generator().manual_seed(60)
    for fmt, n, k in (("bfp4", 14336, 4096), ("bfp8", 4096, 14336)):
        w = torch.randn(n, k, generator=g) * 0.02
        tw, _ = linear.native_weight(device, w, DT[fmt])
        x = torch.randn(2, k, generator=g).to(torch.bfloat16).float()
        x[1] = 0
        y = host(linear.matmul(dev_x(device, x), tw, None))
        assert not y[1].any()
        y4 = host(linear.matmul(dev_x(device, x * 4), tw, None))
        assert torch.equal(y4, y * 4)
        cols = torch.randperm(n // 16, generator=g)[:24] * 16
        sub = torch.cat([w[c : c + 16] for c in cols.tolist()])
        ts, _ = linear.native_weight(device, sub, DT[fmt])
        ysub = host(linear.matmul(dev_x(device, x), ts, None))
        pick = torch.cat([y[:, c : c + 16] for c in cols.tolist()], dim=1)
        assert torch.equal(ysub, pick)
        close_bf16(ysub[:1], orc.matmul_f64(x[:1], orc.native_values(sub, fmt)[0]))
    linear.check_status(device)


def test_matmul_host_equals_matmul(device):
    """The host-buffer call (pinned x in, pinned y out, one library call) gives what matmul gives."""
    g = torch.Generator().manual_seed(70)
    k, n, m = 2048, 1024, 3
    tw, _ = linear.native_weight(device, torch.randn(n, k, generator=g) * 0.02, ttnn.bfloat8_b)
    x = torch.randn(m, k, generator=g).to(torch.bfloat16)
    tx = dev_x(device, torch.zeros(m, k))
    out = ttnn.allocate_tensor_on_device([1, 1, m, n], ttnn.bfloat16, ttnn.TILE_LAYOUT, device)
    x_pin, y_pin = x.contiguous().pin_memory(), torch.empty(m, n, dtype=torch.bfloat16).pin_memory()
    for _ in range(2):
        linear.matmul_host(x_pin, y_pin, tx, tw, None, out=out)
        torch.cuda.synchronize()
        want = host(linear.matmul(dev_x(device, x.float()), tw, None))
        assert torch.equal(y_pin.float(), want)
    linear.check_status(device)


def test_launch_cache_survives_freed_weights(device):
    """The launch caches hold raw addresses. A weight is freed, another of the same shape is packed (its stream
    usually lands on the freed one's address) and the same call objects are used again: the result is the new
    weight's, with and without ttnn.deallocate having been told."""
    g = torch.Generator().manual_seed(81)
    k, n = 1024, 512
    x = dev_x(device, torch.randn(2, k, generator=g))
    out = ttnn.allocate_tensor_on_device([1, 1, 2, n], ttnn.bfloat16, ttnn.TILE_LAYOUT, device)
    for told in (False, True):
        w1, w2 = torch.randn(n, k, generator=g) * 0.02, torch.randn(n, k, generator=g) * 0.02
        t1, _ = linear.native_weight(device, w1, ttnn.bfloat8_b)
        y1 = host(linear.matmul(x, t1, None, out=out)).clone()
        y1b = host(linear.matmul(x, t1, None, out=out))  # the replayed call
        assert torch.equal(y1, y1b)
        addr = t1.t.data_ptr()
        if told:
            ttnn.deallocate(t1)
        del t1
        t2, _ = linear.native_weight(device, w2, ttnn.bfloat8_b)
        y2 = host(linear.matmul(x, t2, None, out=out)).clone()
        close_bf16(y2, orc.matmul_f64(ttnn.to_torch(x).reshape(2, k).float(), orc.native_values(w2, "bfp8")[0]))
        assert not torch.equal(y1, y2), addr
    linear.check_status(device)


def test_pack_then_matmul_in_stream_order(device):
    """Through the C-ABI: a weight packed and multiplied by on one stream with no synchronisation in between. The
    matmul's first weight loads may start before the work ahead of it has finished (programmatic dependent launch)
    unless the call says the weights are fresh (TkdMatmul.weights_fresh): with it, the result equals the synchronised
    one bit for bit."""
    import ctypes

    from dense_reader import _tkd

    L = _tkd.lib()
    k, n, m = 4096, 2048, 2
    g = torch.Generator().manual_seed(91)
    npad = L.tkd_padded_cols(n)
    src = [(torch.randn(k, n, generator=g) * 0.02).to(device.torch) for _ in range(2)]
    x = torch.randn(m, k, generator=g).to(torch.bfloat16).to(device.torch)
    exps = torch.empty(k * npad // 16, dtype=torch.uint8, device=device.torch)
    codes = torch.empty(k * npad, dtype=torch.uint8, device=device.torch)
    packed = torch.zeros(L.tkd_packed_bytes(_tkd.FMT_BFP8, k, n), dtype=torch.uint8, device=device.torch)
    emax = torch.zeros(npad // 16, dtype=torch.uint8, device=device.torch)
    info = torch.zeros(1, dtype=torch.int32, device=device.torch)
    st = torch.cuda.current_stream().cuda_stream

    def pack(w):
        _tkd.check(L.tkd_quantise(_tkd.FMT_BFP8, w.data_ptr(), 1, k, n, None, exps.data_ptr(), codes.data_ptr(), st), "quantise")
        _tkd.check(L.tkd_pack(_tkd.FMT_BFP8, k, n, exps.data_ptr(), codes.data_ptr(), packed.data_ptr(), emax.data_ptr(),
                              info.data_ptr(), st), "pack")

    def describe(out, fresh):
        a = _tkd.TkdMatmul()
        a.fmt, a.m, a.k, a.x, a.ldx = _tkd.FMT_BFP8, m, k, x.data_ptr(), k
        a.nblocks, a.epilogue, a.out_dtype, a.out, a.ldo = 1, _tkd.EPI_PLAIN, _tkd.DT_BF16, out.data_ptr(), n
        a.block[0].w, a.block[0].emax, a.block[0].n = packed.data_ptr(), emax.data_ptr(), n
        a.weights_fresh = fresh
        need = ctypes.c_uint64(0)
        _tkd.check(L.tkd_matmul_workspace(ctypes.byref(a), ctypes.byref(need)), "workspace")
        ws = torch.zeros(need.value, dtype=torch.uint8, device=device.torch)
        a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
        return a, ws

    outs = [torch.empty(m, n, dtype=torch.bfloat16, device=device.torch) for _ in range(3)]
    pack(src[0])
    torch.cuda.synchronize()
    a, ws = describe(outs[0], 0)
    _tkd.check(L.tkd_matmul(ctypes.byref(a), st), "tkd_matmul")  # the first weight, packed and synchronised
    torch.cuda.synchronize()
    # the second weight over the same stream, no synchronisation before its matmul
    pack(src[1])
    b, ws2 = describe(outs[1], 1)
    _tkd.check(L.tkd_matmul(ctypes.byref(b), st), "tkd_matmul")
    torch.cuda.synchronize()
    c, ws3 = describe(outs[2], 0)
    _tkd.check(L.tkd_matmul(ctypes.byref(c), st), "tkd_matmul")  # ... and after a synchronisation
    torch.cuda.synchronize()
    assert torch.equal(outs[1], outs[2]) and not torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("m,out32", [(1, False), (5, True), (70, False)])
def test_kept_calls_take_new_tensors(device, m, out32):
    """A call kept with its weight runs again on other activations, residuals and outputs (given or new), on another stream,
    and not once a tensor it names was freed: every result is what a call described anew gives, bit for bit."""
    g = torch.Generator().manual_seed(95 + m)
    k, n = 512, 160
    tw, ts = linear.native_weight(device, torch.randn(n, k, generator=g) * 0.02, ttnn.bfloat8_b, col_scale=True)
    rdt = ttnn.float32 if out32 else ttnn.bfloat16

    def call(x, r, out=None, scale=None):
        opts = {"out32": out32, "residual": r} if scale is None else {}
        return host(linear.matmul(x, tw, scale, out=out, **opts))

    side = torch.cuda.Stream()
    for rnd in range(3):
        x = dev_x(device, torch.randn(m, k, generator=g))
        r = ttnn.from_torch(torch.randn(1, 1, m, n, generator=g), dtype=rdt, layout=ttnn.TILE_LAYOUT, device=device)
        out = ttnn.allocate_tensor_on_device([1, 1, m, n], rdt, ttnn.TILE_LAYOUT, device)
        torch.cuda.synchronize()
        with torch.cuda.stream(side if rnd == 1 else torch.cuda.current_stream()):
            got = [call(x, r), call(x, r, out), call(x, None, scale=ts)]
            torch.cuda.synchronize()
        linear.CACHE = False
        try:
            want = [call(x, r), call(x, r, out), call(x, None, scale=ts)]
        finally:
            linear.CACHE = True
        assert all(torch.equal(a, b) for a, b in zip(got, want)), rnd
    assert len(tw.calls) == 3
    ttnn.deallocate(ts)
    with pytest.raises(Exception):
        call(x, None, scale=ts)
    assert torch.equal(call(x, r), want[0])
    linear.check_status(device)


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4", "bf16"])
@pytest.mark.parametrize("k,n", [(32, 1), (96, 40), (544, 130), (4096, 272)])
def test_packing_in_one_pass_equals_the_passes(device, fmt, k, n):
    """tkd_pack_weight against tkd_quantise and tkd_pack, bytes and scales: K inside a super-atom and a chunk, N inside a group
    and a panel, zero rows and denormals, both orientations (one with a wider leading dimension), with and without the
    columns' own scales (against bf16_ceil's on the host)."""
    from dense_reader import _tkd

    g = torch.Generator().manual_seed(k + n)
    w = torch.randn(n, k, generator=g) * 0.02 * torch.exp2(torch.randint(-6, 7, (n, 1), generator=g).float())
    w[:, 1] = 0
    w[:, 3] = 1e-41
    w[0, 0] = 0.0 if n > 1 else w[0, 0]
    wide = torch.zeros(k, n + 5)
    wide[:, :n] = w.T
    for scaled in (False, True):
        c = linear.bf16_ceil(w.abs().amax(dim=1).clamp(min=1e-8))
        div = c.to(device.torch) if scaled else None
        want, emax, f = ttnn._pack_in_passes(device, w.to(device.torch), _tkd.__dict__["FMT_" + fmt.upper()], 0, k, n, div)
        own, cs = ttnn.pack_weight_scaled(device, w, DT[fmt]) if scaled else (ttnn.pack_weight(device, w, DT[fmt], 0), None)
        got = [own, ttnn.pack_weight(device, w, DT[fmt], 0, col_div=div),
               ttnn.pack_weight(device, wide.to(device.torch)[:, :n], DT[fmt], 1, col_div=div)]
        for t in got:
            assert t.fmt == f and torch.equal(t.t, want)
            assert emax is None or torch.equal(t.emax, emax)
        if scaled:
            assert torch.equal(cs.float().cpu().reshape(-1), c)


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4", "bf16"])
@pytest.mark.parametrize("m,k,n", [(33, 32, 16), (64, 1024 + 96, 144), (128, 2048, 1024 + 48), (129, 96, 320), (256, 4096, 208),
                                   (257, 512, 64), (515, 1024 + 32, 640)])
def test_prefill_rows_and_epilogues_against_oracle(device, fmt, m, k, n):
    """tkd_matmul_rows: every output stage at the edges of its row tiles (one and two MMA warps, one and two sets of
    accumulators, a last tile with rows to spare), K inside a tile of 64, a unit and a chunk, N inside a panel, and few CTAs
    (whole tiles) against all (tiles cut between them). bf16 outputs within a rounding and the fp32 sums' error; the float32
    ones within K products of relative error 2^-24 each, added at random: 1e-5 of the result's size."""
    g = torch.Generator().manual_seed(m + k + n)
    w, w2 = torch.randn(n, k, generator=g) * 0.02, torch.randn(n, k, generator=g) * 0.02
    x = torch.randn(m, k, generator=g)
    tx = dev_x(device, x)
    (tw, ts), (tw2, _) = linear.native_weight(device, w, DT[fmt], col_scale=True), linear.native_weight(device, w2, DT[fmt])
    wk, wk2 = (torch.from_numpy(orc.native_values(w, fmt, col_scale=True)[0]).double(), torch.from_numpy(orc.native_values(w2, fmt)[0]).double())
    sc = ttnn.to_torch(ts).double().reshape(-1)
    xd = x.to(torch.bfloat16).double()
    plain, other = (xd @ wk), xd @ wk2
    res = torch.randn(m, n, generator=g)
    t32 = ttnn.from_torch(res.reshape(1, 1, m, n), dtype=ttnn.float32, layout=ttnn.TILE_LAYOUT, device=device)
    tbf = ttnn.from_torch(res.to(torch.bfloat16).reshape(1, 1, m, n), dtype=ttnn.bfloat16, layout=ttnn.TILE_LAYOUT, device=device)
    for ctas in (None, 3):
        close_bf16(host(linear.matmul(tx, tw, ts, max_ctas=ctas)), (plain * sc).numpy())
        y32 = host(linear.matmul(tx, tw, None, residual=t32, out32=True, max_ctas=ctas)).double()
        want = plain + res.double()
        assert ((y32 - want).norm() / want.norm()).item() < 1e-5
        close_bf16(host(linear.matmul(tx, tw2, None, residual=tbf, max_ctas=ctas)), (other + res.to(torch.bfloat16).double()).numpy())
        glu = torch.nn.functional.silu(plain) * other
        close_bf16(host(linear.matmul(tx, tw, None, w_up=tw2, glu=True, max_ctas=ctas)), glu.numpy())
        if n % 64 == 0:
            act = torch.nn.functional.gelu(plain, approximate="tanh")
            half = act.reshape(m, -1, 2, 32)[:, :, 0].reshape(m, -1) * plain.reshape(m, -1, 2, 32)[:, :, 1].reshape(m, -1)
            close_bf16(host(linear.matmul(tx, tw, None, glu=True, glu_act=1, max_ctas=ctas)), half.numpy())
    linear.check_status(device)


def test_graph_keeps_its_workspace(device):
    """A captured call replays rightly after larger calls have outgrown its workspace, whose memory others may have by then."""
    g = torch.Generator().manual_seed(96)
    k, n = 4096, 1024 + 128
    tw, _ = linear.native_weight(device, torch.randn(n, k, generator=g) * 0.02, ttnn.bfloat8_b)
    slot, linear.WORKSPACE_SLOT = linear.WORKSPACE_SLOT, "graph"
    try:
        x = dev_x(device, torch.randn(2, k, generator=g))
        want = host(linear.matmul(x, tw, None)).clone()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            y = linear.matmul(x, tw, None)
        before = linear._WORKSPACE[(device.id, "graph")].numel()
        linear.matmul(dev_x(device, torch.randn(300, k, generator=g)), tw, None)
        assert linear._WORKSPACE[(device.id, "graph")].numel() >= 2 * before
        junk = [torch.full((1 << 20,), 7, dtype=torch.int32, device=device.torch) for _ in range(8)]
        y.t.zero_()
        graph.replay()
        assert torch.equal(host(y), want)
        del junk, graph
    finally:
        linear.WORKSPACE_SLOT = slot
    linear.check_status(device)


@pytest.mark.parametrize("dtype,k", [(ttnn.bfloat8_b, 1024), (ttnn.bfloat8_b, 3616), (ttnn.bfloat8_b, 4096), (ttnn.bfloat4_b, 2048),
                                     (ttnn.bfloat4_b, 4000), (ttnn.bfloat16, 992), (ttnn.bfloat16, 5632), (ttnn.bfloat8_b, 14336)])
@pytest.mark.parametrize("m", [1, 2, 8, 9, 17, 32])
def test_plain_calls_equal_the_counted_kernels(device, dtype, k, m):
    """Plain calls of four slices run as items of 32 columns over all of K (up to 8 rows) or in clusters of a CTA a slice (9 to 32);
    tkd_matmul_noalloc stays with the kernels that add panels up through their workspace. Both add the same sums in the same order:
    equal bits, in every epilogue, at shapes with more and fewer items than SMs, on few CTAs, with the last columns of a panel
    missing and a K that ends inside a chunk."""
    import ctypes

    from dense_reader import _tkd

    L, g = _tkd.lib(), torch.Generator().manual_seed(k + m)
    put = lambda t: t.to(device.torch)
    x = put(torch.randn(m, k, generator=g).bfloat16())
    W = lambda n: linear.native_weight(device, torch.randn(n, k, generator=g) * 0.02, dtype)[0]
    big = 5000 if m <= 8 else 2500  # (the fixed scratch holds no more)
    w1, w2, w3, w4 = W(big), W(big), W(64), W(176)
    ws = torch.zeros(64 << 20, dtype=torch.uint8, device=device.torch)
    status = torch.zeros(1, dtype=torch.int32, device=device.torch)
    scale, scale2 = (put(0.5 + torch.rand(big, generator=g)) for _ in range(2))
    for epi, blocks, ctas in ((_tkd.EPI_PLAIN, [(w1, None, big)], 0), (_tkd.EPI_PLAIN, [(w4, None, 161), (w3, None, 64)], 8),
                              (_tkd.EPI_GLU_IL, [(w3, None, 64)], 0), (_tkd.EPI_GLU2, [(w1, w2, big)], 100),
                              (_tkd.EPI_RESIDUAL, [(w4, None, 176)], 0), (_tkd.EPI_OUT32, [(w1, None, big - 1)], 0)):
        f32 = epi == _tkd.EPI_OUT32
        cols = 32 if epi == _tkd.EPI_GLU_IL else sum(b[2] for b in blocks)
        outs = [torch.full((m, cols), 7.0, dtype=torch.float32 if f32 else torch.bfloat16, device=device.torch) for _ in range(2)]
        res = put(torch.randn(m, cols, generator=g)).to(outs[0].dtype)
        for out, counted in zip(outs, (False, True)):
            a = _tkd.TkdMatmul()
            a.fmt, a.m, a.k, a.x, a.ldx, a.nblocks, a.epilogue = w1.fmt, m, k, x.data_ptr(), k, len(blocks), epi
            at = 0
            for b, (w, up, n) in enumerate(blocks):
                a.block[b].w, a.block[b].n, a.block[b].out_col0 = w.t.data_ptr(), n, at
                a.block[b].emax = w.emax.data_ptr() if w.emax is not None else None
                if up is not None:
                    a.block[b].w_up, a.block[b].emax_up = up.t.data_ptr(), up.emax.data_ptr() if up.emax is not None else None
                at += n
            if len(blocks) == 1 and epi != _tkd.EPI_GLU_IL and blocks[0][2] == big:
                a.scale, a.scale_dtype, a.scale_up = scale.data_ptr(), _tkd.DT_F32, scale2.data_ptr()
            if epi in (_tkd.EPI_RESIDUAL, _tkd.EPI_OUT32):
                a.residual, a.residual_dtype, a.ldr = res.data_ptr(), _tkd.DT_F32 if f32 else _tkd.DT_BF16, cols
            a.out, a.out_dtype, a.ldo, a.max_ctas = out.data_ptr(), _tkd.DT_F32 if f32 else _tkd.DT_BF16, cols, ctas
            a.status = status.data_ptr()
            a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
            stream = torch.cuda.current_stream().cuda_stream
            _tkd.check((L.tkd_matmul_noalloc if counted else L.tkd_matmul)(ctypes.byref(a), stream), "matmul")
        torch.cuda.synchronize()
        assert status.item() == 0 and torch.isfinite(outs[0]).all() and not (outs[0] == 7.0).all()
        assert torch.equal(outs[0], outs[1]), (epi, cols)


@pytest.mark.parametrize("m", [1, 3, 20, 40])
@pytest.mark.parametrize("act", [0, 1])
def test_activations_over_their_range(device, m, act):
    """act(gate) * up, the gates any float32 (a weight of 1 times its column's scale), up 1: within a rounding to bf16 of the
    float64 value over the whole range, and at the edges: where e^-u passes 2^64 and the largest float32, at infinities and NaN.
    2^-8 for the rounding (8 significant bits), and for e^t in float32 2^-23 |t| (t's rounding and its product's with log2 e) and 2^-21 (the
    exponential's own two units, the sum and the quotient)."""
    g = torch.Generator().manual_seed(99)
    edges = torch.tensor([0.0, -0.0, 44.36, -44.36, -44.37, -88.69, -88.7, -88.71, -88.72, -88.7228, -88.7229, -88.73, -104.0, 88.7, 1e30, -1e30,
                          7.9, -7.9, -7.91, -10.0, -10.1, -10.2, float("inf"), float("-inf"), float("nan")])
    gates = torch.cat([edges, torch.rand(2000, generator=g) * 200 - 100, torch.randn(2000, generator=g) * 4,
                       torch.randn(71, generator=g) * torch.exp2(torch.rand(71, generator=g) * 60 - 40)])
    n, k = gates.numel(), 32
    one = torch.zeros(n, k)
    one[:, 0] = 1.0
    gate, up = (linear.native_weight(device, one, ttnn.bfloat16)[0] for _ in range(2))
    x = torch.zeros(m, k)
    x[:, 0] = 1.0
    scales = (gates.to(device.torch), torch.ones(n, device=device.torch))
    got = host(linear.matmul(dev_x(device, x), gate, None, w_up=up, glu=True, glu_act=act, col_scales=scales)).double()
    v = gates.double()
    t = -v if act == 0 else -(v * (1.5957691216 + 0.0713548162 * v * v))
    want = v / (1 + torch.exp(t))  # (-inf / inf: no number)
    for row in got:
        assert torch.equal(row.isnan(), want.isnan()) and torch.equal(row.isinf(), want.isinf())
        ok = want.isfinite()
        # (past e^88.72 the float32 sum has no end and the quotient is zero: below 2^-119 anything counts as zero)
        bound = want[ok].abs() * (2.0**-8 + 2.0**-23 * t[ok].abs().clamp(max=90) + 2.0**-21) + 2.0**-119
        assert ((row[ok] - want[ok]).abs() <= bound).all()
    linear.check_status(device)


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4", "bf16"])
@pytest.mark.parametrize("m", [7, 32, 40, 100])
def test_column_shards_give_the_whole_weights_bits(device, fmt, m):
    """A weight's columns in parts, as the GPUs of a box hold them, give what the whole weight gives bit for bit: up to 32 rows, and
    with fixed_sums for more."""
    g = torch.Generator().manual_seed(97 + m)
    k, n = 4096, 2560
    w = torch.randn(n, k, generator=g) * 0.02
    x = dev_x(device, torch.randn(m, k, generator=g))
    opts = {"fixed_sums": True} if m > 32 else {}
    whole = host(linear.matmul(x, linear.native_weight(device, w, DT[fmt])[0], None, **opts))
    for parts in (2, 5):
        cols = n // parts
        got = [host(linear.matmul(x, linear.native_weight(device, w[i * cols : (i + 1) * cols], DT[fmt])[0], None, **opts)) for i in range(parts)]
        assert torch.equal(torch.cat(got, dim=1), whole), parts
    linear.check_status(device)


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4", "bf16"])
@pytest.mark.parametrize("m,k,n", [(1, 4096, 1072), (5, 544, 176), (8, 32, 16), (9, 1056, 144), (32, 4096, 208), (33, 96, 320), (300, 1056, 144)])
def test_linear_silu_in_the_output_stage(device, fmt, m, k, n):
    """linear(activation="silu") against the oracle for the kernels that have the output stage (long rows: the test of that name), with and without column scales:
    within a rounding to bf16 of the float64 value and float32's sums. With an out the product stays in it and the activation is a
    tensor of its own; a residual is added before the activation."""
    g = torch.Generator().manual_seed(m + k + n)
    w, x = torch.randn(n, k, generator=g) * 0.06, torch.randn(m, k, generator=g)
    tx, silu = dev_x(device, x), torch.nn.functional.silu
    for scaled in (False, True):
        tw, ts = linear.native_weight(device, w, DT[fmt], col_scale=scaled)
        plain = x.to(torch.bfloat16).double() @ torch.from_numpy(orc.native_values(w, fmt, col_scale=scaled)[0]).double()
        if scaled:
            plain = plain * ttnn.to_torch(ts).double().reshape(-1)
        y = linear.linear(tx, tw, ts if scaled else None, activation="silu")
        assert y.dtype == ttnn.bfloat16 and tuple(y.shape) == (1, 1, m, n)
        close_bf16(host(y), silu(plain).numpy())
    out = ttnn.allocate_tensor_on_device([1, 1, m, n], ttnn.bfloat16, ttnn.TILE_LAYOUT, device)
    y = linear.linear(tx, tw, ts, activation="silu", out=out)
    close_bf16(host(out), plain.numpy())
    close_bf16(host(y), silu(host(out).double()).numpy())
    unit, _ = linear.native_weight(device, w, DT[fmt])
    plain = x.to(torch.bfloat16).double() @ torch.from_numpy(orc.native_values(w, fmt)[0]).double()
    res = torch.randn(m, n, generator=g).to(torch.bfloat16)
    tr = ttnn.from_torch(res.reshape(1, 1, m, n), dtype=ttnn.bfloat16, layout=ttnn.TILE_LAYOUT, device=device)
    close_bf16(host(linear.linear(tx, unit, None, activation="silu", residual=tr)), silu(plain + res.double()).numpy())
    linear.check_status(device)


@pytest.mark.parametrize("dtype,k", [(ttnn.bfloat8_b, 32), (ttnn.bfloat8_b, 288), (ttnn.bfloat8_b, 544), (ttnn.bfloat8_b, 2080), (ttnn.bfloat8_b, 4128),
                                     (ttnn.bfloat4_b, 480), (ttnn.bfloat4_b, 1056), (ttnn.bfloat4_b, 5120), (ttnn.bfloat16, 160), (ttnn.bfloat16, 1280),
                                     (ttnn.bfloat8_b, 8960), (ttnn.bfloat8_b, 8992), (ttnn.bfloat4_b, 8704), (ttnn.bfloat4_b, 8736),
                                     (ttnn.bfloat16, 7168), (ttnn.bfloat16, 7200)])
@pytest.mark.parametrize("m", [1, 2, 8])
def test_items_of_one_to_four_slices_equal_the_counted_kernel(device, dtype, k, m):
    """The same for one to three slices (of one, the smallest weights only), for four whose last is short, and at both sides of the
    longest eight rows that fit beside the ring, where the plain call is the counting kernel too."""
    test_plain_calls_equal_the_counted_kernels(device, dtype, k, m)


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4"])
@pytest.mark.parametrize("n", [16, 112, 144])
def test_own_scales_with_zero_and_tiny_inputs(device, fmt, n):
    """Columns divided by their own scales where inputs are zero, denormal or near it: quotients that are no normal numbers, or come
    of a shared exponent below 100, are the division's, and zeros are zeros, also in the columns that pad N to a panel. Bit for bit
    the oracle's."""
    g = torch.Generator().manual_seed(n)
    k = 128
    w = torch.randn(n, k, generator=g) * 0.1
    for i, size in enumerate((0.0, 1e-45, 3e-42, 2e-39, 1.2e-38, 1e-37, 1e-36, 1e-33, 1e-30, 1e-20, 1e-10)):
        w[:, 3 * i] = torch.randn(n, generator=g) * size
    w[:, 40] = torch.where(torch.arange(n) % 16 == 3, torch.randn(n, generator=g) * 1e-39, torch.zeros(n))
    w[5] = 0.0
    tw, ts = linear.native_weight(device, w, DT[fmt], col_scale=True)
    want, scale = orc.native_values(w, fmt, col_scale=True)
    assert torch.equal(ttnn.to_torch(ts).float().reshape(-1), torch.as_tensor(scale).float().reshape(-1))
    held = ttnn.to_torch(tw).float().reshape(k, -1)[:, :n]
    assert torch.equal(held, torch.from_numpy(want))


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4", "bf16"])
@pytest.mark.parametrize("n,k", [(1, 32), (40, 96), (130, 544), (4096, 1024)])
def test_unit_scales_come_with_the_pack(device, fmt, n, k):
    """native_weight without column scales: the same weight as the packer's alone, and a one for every column, of a wide weight too."""
    g = torch.Generator().manual_seed(n)
    w = torch.randn(n, k, generator=g) * 0.1
    for wide in (False, True):
        if wide:
            w[:, 1] = 1e-30
        tw, ts = linear.native_weight(device, w, DT[fmt])
        alone = ttnn.pack_weight(device, w, DT[fmt], 0)
        assert tw.fmt == alone.fmt and torch.equal(tw.t, alone.t) and (tw.emax is None) == (alone.emax is None)
        assert tw.emax is None or torch.equal(tw.emax, alone.emax)
        assert ts.t.dtype == torch.bfloat16 and tuple(ts.t.shape) == (1, 1, 1, n) and bool((ts.t == 1).all())


@pytest.mark.parametrize("m", [1, 16, 64])
def test_silu_behind_a_float32_product(device, m):
    """linear(activation="silu") into float32 applies the activation to the float32 product, each time it is called alike."""
    g = torch.Generator().manual_seed(m)
    tw, ts = linear.native_weight(device, torch.randn(144, 544, generator=g) * 0.06, ttnn.bfloat8_b)
    tx = dev_x(device, torch.randn(m, 544, generator=g))
    want = torch.nn.functional.silu(host(linear.matmul(tx, tw, None, out32=True)))
    for _ in range(3):
        y = linear.linear(tx, tw, None, activation="silu", out_dtype=ttnn.float32)
        # (exponentials of the CPU and the GPU: a few units in the last place)
        assert y.dtype == ttnn.float32 and torch.allclose(host(y), want, rtol=1e-6, atol=1e-7)
        with pytest.raises(AssertionError):
            linear.linear(tx, tw, None, activation="relu")
    linear.check_status(device)


@pytest.mark.parametrize("fmt,m,k", [("bf16", 8, 7168), ("bf16", 8, 7200), ("bf16", 8, 8192), ("bfp8", 8, 8960), ("bfp8", 8, 8992), ("bfp8", 6, 14336),
                                     ("bfp4", 8, 8704), ("bfp4", 8, 8736), ("bfp4", 7, 14336), ("bfp8", 8, 9632), ("bfp4", 8, 9632), ("bf16", 6, 9632),
                                     ("bfp8", 1, 114688), ("bfp8", 32, 20480), ("bfp4", 20, 20512), ("bf16", 12, 20480), ("bfp8", 40, 9632)])
def test_linear_silu_of_long_rows(device, fmt, m, k):
    """linear(activation="silu") of long rows: where x leaves tkd_narrow_kernel's ring no room, and then tkd_stream_kernel's (on both
    sides of that limit, and a K that ends inside a chunk), slices past four, more than 32 rows."""
    g = torch.Generator().manual_seed(m + k)
    w, x = torch.randn(80, k, generator=g) * 0.02, torch.randn(m, k, generator=g)
    for scaled in (False, True):
        tw, ts = linear.native_weight(device, w, DT[fmt], col_scale=scaled)
        plain = x.to(torch.bfloat16).double() @ torch.from_numpy(orc.native_values(w, fmt, col_scale=scaled)[0]).double()
        if scaled:
            plain = plain * ttnn.to_torch(ts).double().reshape(-1)
        close_bf16(host(linear.linear(dev_x(device, x), tw, ts if scaled else None, activation="silu")), torch.nn.functional.silu(plain).numpy())
    linear.check_status(device)


@pytest.mark.parametrize("m,k", [(1, 1024), (5, 544), (8, 14336), (16, 1056), (32, 1056), (32, 4096), (40, 1056), (300, 4096)])
def test_the_silu_output_stage_has_no_other_activation(device, m, k):
    """TKD_EPI_SILU is silu whatever `act` (a GLU's) says, in every kernel: the same bits with act 1."""
    g = torch.Generator().manual_seed(m + k)
    tw, _ = linear.native_weight(device, torch.randn(144, k, generator=g) * 0.06, ttnn.bfloat8_b)
    tx = dev_x(device, torch.randn(m, k, generator=g))
    first = host(linear.linear(tx, tw, None, activation="silu"))
    (call,) = tw.calls.values()
    for _, a in call.launches:
        a.act = 1
    assert torch.equal(host(linear.linear(tx, tw, None, activation="silu")), first)
    linear.check_status(device)


@pytest.mark.parametrize("fmt", ["bfp8", "bf16"])
@pytest.mark.parametrize("m", [33, 64, 300])
def test_more_rows_in_place(device, fmt, m):
    """More than 32 rows whose output is x's own memory, or overlaps it: what an output of its own gets, within the rounding of other
    sums (such a call runs the kernel that reads a copy of x)."""
    g = torch.Generator().manual_seed(m)
    k = n = 288
    tw, _ = linear.native_weight(device, torch.randn(n, k, generator=g) * 0.06, DT[fmt])
    x = torch.randn(m, k, generator=g)
    want = host(linear.matmul(dev_x(device, x), tw, None))
    tx = dev_x(device, x)
    for _ in range(2):
        linear.matmul(tx, tw, None, out=tx)
        close_bf16(host(tx), want)
        tx.t.copy_(x.reshape(1, 1, m, k))
    # (the output's first row is x's last)
    both = torch.empty(1, 1, 2 * m - 1, k, dtype=torch.bfloat16, device=device.torch)
    both[..., :m, :] = x.to(device.torch)
    view = lambda t: ttnn.Tensor(t, ttnn.bfloat16, ttnn.TILE_LAYOUT, device, ttnn.DRAM_MEMORY_CONFIG)  # noqa: E731
    out = view(both[..., m - 1 :, :])
    linear.matmul(view(both[..., :m, :]), tw, None, out=out)
    close_bf16(host(out), want)
    linear.check_status(device)
