"""The kernel that keeps 9 to 32 rows of x in shared memory (csrc/tkd_rows.cuh): its outputs, its records and its exchanged calls."""

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from common import ttnn_like as ttnn  # noqa: E402
from dense_reader import _tkd, linear, sharded  # noqa: E402
from oracle import oracle as orc  # noqa: E402
from test_exchange_gpu import fake_rank  # noqa: E402
from test_parity_gpu import DT, close_bf16, dev_x, host  # noqa: E402


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4", "bf16"])
@pytest.mark.parametrize("m,k,n", [(9, 32, 16), (9, 4096, 208), (12, 288, 144), (16, 544, 320), (16, 3360, 1056), (17, 1024, 64),
                                   (24, 1184, 5008), (25, 160, 144), (32, 1056, 272), (20, 3136, 144)])
def test_outputs_against_oracle(device, fmt, m, k, n):
    """Every output stage, K inside a super-atom, a chunk and a stage, N inside a panel and past one item a CTA, few CTAs and all.
    bf16 results within a rounding and the float32 sums' error; float32 ones within K products of relative error 2^-24, added at
    random: 1e-5 of the result's size."""
    g = torch.Generator().manual_seed(m + k + n)
    w, w2, x = (torch.randn(r, k, generator=g) * s for r, s in ((n, 0.03), (n, 0.03), (m, 1.0)))
    tx, xd = dev_x(device, x), x.to(torch.bfloat16).double()
    (tw, ts), (tw2, _) = linear.native_weight(device, w, DT[fmt], col_scale=True), linear.native_weight(device, w2, DT[fmt])
    plain = xd @ torch.from_numpy(orc.native_values(w, fmt, col_scale=True)[0]).double()
    other = xd @ torch.from_numpy(orc.native_values(w2, fmt)[0]).double()
    sc = ttnn.to_torch(ts).double().reshape(-1)
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


def runs_in_tensor_memory(fmt, m, k, n, ctas):
    """Whether a plain call of 9 to 32 rows runs the tensor-memory kernel: given its slice size, which the other kernel does not serve, it is
    the same launch."""
    a, plans = _tkd.TkdMatmul(), []
    a.fmt, a.m, a.k = {"bfp8": _tkd.FMT_BFP8, "bfp4": _tkd.FMT_BFP4, "bf16": _tkd.FMT_BF16}[fmt], m, k
    a.nblocks, a.epilogue, a.out_dtype = 1, _tkd.EPI_PLAIN, _tkd.DT_BF16
    a.block[0].n, a.max_ctas = n, ctas or 0
    for _ in range(2):
        p = _tkd.TkdPlan()
        assert _tkd.lib().tkd_matmul_plan(ctypes.byref(a), ctypes.byref(p)) == 0
        plans.append((p.smem_bytes, p.stages, p.grid))
        a.ks = p.ks
    return plans[0] == plans[1]


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4", "bf16"])
@pytest.mark.parametrize("m,k,n", [(17, 3104, 208), (24, 4128, 144), (31, 6560, 2064), (32, 8224, 272), (9, 14368, 80)])
def test_units_of_the_tensor_memory_kernel(device, fmt, m, k, n):
    """K that ends inside a unit of 128, a tile of 64 and a chunk, more units than there are slots, in clusters and without; the rows
    past the call's, which hold what a call before left in shared memory (here NaN), show nowhere. float32 results within K products
    of relative error 2^-24, added at random: 1e-5 of the result's size."""
    g = torch.Generator().manual_seed(m + k + n)
    w, x = torch.randn(n, k, generator=g) * 0.03, torch.randn(m, k, generator=g)
    tw, _ = linear.native_weight(device, w, DT[fmt])
    tx, nan = dev_x(device, x), dev_x(device, torch.full((32, k), float("nan")))
    want = x.to(torch.bfloat16).double() @ torch.from_numpy(orc.native_values(w, fmt)[0]).double()
    for ctas in (None, 3):
        for rows in (m, 32):
            assert runs_in_tensor_memory(fmt, rows, k, n, ctas), (rows, ctas)
        assert bool(host(linear.matmul(nan, tw, None, max_ctas=ctas)).isnan().all())
        y = host(linear.matmul(tx, tw, None, out32=True, max_ctas=ctas)).double()
        assert ((y - want).norm() / want.norm()).item() < 1e-5
    linear.check_status(device)


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4", "bf16"])
@pytest.mark.parametrize("m,k,n", [(17, 3104, 192), (32, 4128, 144), (9, 14368, 64)])
def test_every_output_of_a_k_that_ends_inside_a_chunk(device, fmt, m, k, n):
    """The tensor-memory kernel has an instance for each kind of output, outside clusters and (for fewer kinds) in them."""
    assert runs_in_tensor_memory(fmt, m, k, n, None) and runs_in_tensor_memory(fmt, m, k, n, 3)
    test_outputs_against_oracle(device, fmt, m, k, n)
    g = torch.Generator().manual_seed(m)
    w, x = torch.randn(n, k, generator=g) * 0.05, torch.randn(m, k, generator=g)
    tw, _ = linear.native_weight(device, w, DT[fmt])
    plain = x.to(torch.bfloat16).double() @ torch.from_numpy(orc.native_values(w, fmt)[0]).double()
    for ctas in (None, 3):
        close_bf16(host(linear.linear(dev_x(device, x), tw, None, activation="silu", max_ctas=ctas)), torch.nn.functional.silu(plain).numpy())
    linear.check_status(device)


@pytest.mark.parametrize("m,k", [(9, 1024), (16, 288), (24, 1056), (30, 1056)])
def test_records_of_the_plain_calls_outputs(device, m, k):
    """Records are the canonical top-k of the outputs that a plain call gives, with and without y written, of one weight and of a
    block list, with ties and a last unit in part."""
    g = torch.Generator().manual_seed(m + k)
    n, rows, kk, units = 2048 + 416, 9, 7, 2
    ws = [(torch.randn(n, k, generator=g) * 4).round() / 64 for _ in range(2)]
    tws = [linear.native_weight(device, w, ttnn.bfloat8_b)[0] for w in ws]
    tx = dev_x(device, (torch.randn(m, k, generator=g) * 2).round())
    ys = [host(linear.matmul(tx, tw, None)) for tw in tws]
    # (one weight with y, one without, and several by one launch)
    for base, write_y in ((0, True), (5000, False)):
        r = linear.topk_result(device, units + 1, rows, kk)
        out = ttnn.from_torch(torch.full((1, 1, m, n), -7.0, dtype=torch.bfloat16), dtype=ttnn.bfloat16, layout=ttnn.TILE_LAYOUT, device=device)
        linear.matmul(tx, tws[0], None, topk={"r": r, "k": kk, "rows": rows, "slot0": 1, "base": base, "n": n - 100, "write_y": write_y}, out=out)
        assert torch.equal(host(out), ys[0]) if write_y else bool((host(out) == -7.0).all())
        check_records(ttnn.to_torch(r).reshape(units + 1, 2, rows, kk)[1:], ys[0], n - 100, base)
    r = linear.topk_result(device, 2 * units, rows, kk)
    linear.records_together(tx, tuple(tws), {"r": r, "k": kk, "rows": rows, "slot0": 0, "base": 0, "n": n, "write_y": False}, out)
    rec = ttnn.to_torch(r).reshape(2, units, 2, rows, kk)
    for b in range(2):
        check_records(rec[b], ys[b], n, b * n)
    linear.check_status(device)


def check_records(rec, y, n, base):
    rec = rec.numpy().view(np.uint32)
    for u in range(rec.shape[0]):
        for t in range(rec.shape[2]):
            c0, c1 = u * 2048, min((u + 1) * 2048, n)
            keys, idx = orc.topk_canonical(orc.bf16_bits(y[t, c0:c1]), c1 - c0, rec.shape[3], base + c0)
            assert np.array_equal(rec[u, 0, t], keys) and np.array_equal(rec[u, 1, t], idx), (u, t)


@pytest.mark.parametrize("m,out32", [(9, False), (16, True), (20, False), (31, False)])
def test_exchanged_calls_give_the_plain_calls_bits(device, m, out32):
    """Column shards of 9 and more rows, their outputs stored into every rank's buffer: the whole weight's bits, and the flags."""
    world, k = 3, 1056
    shards = sharded.column_shards(1024 * 3 - 96, world)
    n = shards[-1][1]
    g = torch.Generator().manual_seed(5)
    w = torch.randn(n, k, generator=g) * 0.02
    tx = dev_x(device, torch.randn(m, k, generator=g))
    full = ttnn.to_torch(linear.matmul(tx, linear.native_weight(device, w, ttnn.bfloat8_b)[0], None, out32=out32))
    nbytes = 1 << 20
    bufs = [torch.zeros(nbytes + 256, dtype=torch.uint8, device=device.torch) for _ in range(world)]
    ranks = [fake_rank(device, r, world, bufs, nbytes) for r in range(world)]
    outs = [ex.tensor([1, 1, m, n], ttnn.float32 if out32 else ttnn.bfloat16) for ex in ranks]
    tws = [linear.native_weight(device, sharded.shard_rows(w, shards, r), ttnn.bfloat8_b)[0] for r in range(world)]
    status = torch.zeros(1, dtype=torch.int32, device=device.torch)
    for r, ex in enumerate(ranks):
        linear.matmul(tx, tws[r], None, out=outs[r], col0=shards[r][0] // 32, out32=out32, exchange=ex)
    for ex in ranks:
        ex.wait_all(status)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    for r in range(world):
        assert torch.equal(ttnn.to_torch(outs[r]), full), r
        assert bufs[r][: 4 * world].view(torch.int32).tolist() == [1] * world
    linear.check_status(device)


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4", "bf16"])
@pytest.mark.parametrize("m,k,n", [(33, 96, 16), (47, 544, 320), (64, 2080, 144), (97, 1056, 512), (100, 4096, 80), (250, 288, 64)])
def test_tiles_of_rows(device, fmt, m, k, n):
    """More than 32 rows of a small weight, tiles of sixteen rows (twelve at K 4096) with a team of CTAs each: every output stage, a
    last tile in part, a team of one CTA, more items than CTAs."""
    test_outputs_against_oracle(device, fmt, m, k, n)
    g = torch.Generator().manual_seed(m)
    w, x = torch.randn(n, k, generator=g) * 0.05, torch.randn(m, k, generator=g)
    tw, _ = linear.native_weight(device, w, DT[fmt])
    plain = x.to(torch.bfloat16).double() @ torch.from_numpy(orc.native_values(w, fmt)[0]).double()
    for ctas in (None, 17):
        close_bf16(host(linear.linear(dev_x(device, x), tw, None, activation="silu", max_ctas=ctas)), torch.nn.functional.silu(plain).numpy())
    linear.check_status(device)


@pytest.mark.parametrize("fmt,m,k", [("bfp8", 32, 1056), ("bfp4", 25, 544), ("bfp4", 24, 2816), ("bfp8", 31, 2304)])
def test_two_tiles_of_rows_on_one_cta(device, fmt, m, k):
    """17 to 32 rows as two tiles of sixteen where max_ctas leaves one CTA: it takes one tile after the other. The same bits as with
    two, three and all CTAs, of the outputs, their float32 form, the records and an exchanged call."""
    g = torch.Generator().manual_seed(m + k)
    n, rows, kk = 2048 + 176, 9, 7
    w, x = torch.randn(n, k, generator=g) * 0.05, torch.randn(m, k, generator=g)
    tw, _ = linear.native_weight(device, w, DT[fmt])
    tx, res = dev_x(device, x), torch.randn(m, n, generator=g)
    t32 = ttnn.from_torch(res.reshape(1, 1, m, n), dtype=ttnn.float32, layout=ttnn.TILE_LAYOUT, device=device)
    plain = x.to(torch.bfloat16).double() @ torch.from_numpy(orc.native_values(w, fmt)[0]).double()
    whole, whole32 = host(linear.matmul(tx, tw, None)), host(linear.matmul(tx, tw, None, residual=t32, out32=True))
    close_bf16(whole, plain.numpy())
    for ctas in (1, 2, 3, 1):
        assert torch.equal(host(linear.matmul(tx, tw, None, max_ctas=ctas)), whole), ctas
        assert torch.equal(host(linear.matmul(tx, tw, None, residual=t32, out32=True, max_ctas=ctas)), whole32), ctas
        for write_y in (True, False):
            r = linear.topk_result(device, 2, rows, kk)
            out = ttnn.from_torch(torch.full((1, 1, m, n), -7.0, dtype=torch.bfloat16), dtype=ttnn.bfloat16, layout=ttnn.TILE_LAYOUT, device=device)
            spec = {"r": r, "k": kk, "rows": rows, "slot0": 0, "base": 0, "n": n, "write_y": write_y}
            linear.matmul(tx, tw, None, topk=spec, out=out, max_ctas=ctas)
            assert torch.equal(host(out), whole) if write_y else bool((host(out) == -7.0).all())
            check_records(ttnn.to_torch(r).reshape(2, 2, rows, kk), whole, n, 0)
    nbytes = 1 << 20
    bufs = [torch.zeros(nbytes + 256, dtype=torch.uint8, device=device.torch) for _ in range(2)]
    ranks = [fake_rank(device, r, 2, bufs, nbytes) for r in range(2)]
    outs = [ex.tensor([1, 1, m, n], ttnn.bfloat16) for ex in ranks]
    half = 1024
    parts = [linear.native_weight(device, w[:half], DT[fmt])[0], linear.native_weight(device, w[half:], DT[fmt])[0]]
    status = torch.zeros(1, dtype=torch.int32, device=device.torch)
    for r, ex in enumerate(ranks):
        linear.matmul(tx, parts[r], None, out=outs[r], col0=r * half // 32, exchange=ex, max_ctas=1)
    for ex in ranks:
        ex.wait_all(status)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    for r in range(2):
        assert torch.equal(host(outs[r]), whole), r
    linear.check_status(device)
