# SPDX-License-Identifier: Apache-2.0
# Copyright 2026 Xylolabs
# Ported from XylolabsInc/tensix-kernels, lm_head_topk/tests/test_lm_head.py (Apache-2.0): the test cases, shapes, seeds and bars are that
# file's; the imports and the device API under them are this package's.
"""The top-k LM head (lm_head_topk/lmhead.py, head_pick.py) against torch, case for case the reference's
lm_head_topk/tests/test_lm_head.py: a random bf16 head [8192, 1024] as four bfloat4_b blocks and random x rows;
- the records hold the block matmul's own bf16 logits at their ids, and each row's best k over the records are its best
  k over all logits, bit for bit;
- the host rescore's tokens against a bf16 host head, token for token;
- the device pick against the host rescore on the same records in bf16 and float32 logits (token for token, or, where
  the sum orders part a near tie, exact logits equal to 1e-6 / one bf16 step), also on a head whose rows
  repeat in pairs (exact ties: the lowest id wins) and on a padded head (valid=), its table also the valid rows only;
- the records-only pick with and without a token map against the host's argmax over the same records;
- both picks with k 4 at 1 and 3 rows.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from common import ttnn_like as ttnn  # noqa: E402
from common.testing import same  # noqa: E402
from dense_reader import linear  # noqa: E402
from lm_head_topk import head_pick, lmhead  # noqa: E402
from oracle import oracle as orc  # noqa: E402

VOCAB, DIM, CHUNKS = 8192, 1024, 4


def head(seed, pairs=False):
    g = torch.Generator().manual_seed(seed)
    w = (torch.randn(VOCAB, DIM, generator=g) * 0.05).to(torch.bfloat16)
    if pairs:
        w[1::2] = w[0::2]  # rows 2i and 2i + 1 equal: every logit ties with its pair
    return w


def x_rows(device, rows, seed):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(rows, DIM, generator=g).to(torch.bfloat16)
    return x, ttnn.from_torch(x.reshape(1, 1, rows, DIM), dtype=ttnn.bfloat16, layout=ttnn.TILE_LAYOUT, device=device)


def host_tokens(x, w, logits="bf16"):
    z = x.float() @ w.float().T
    if logits == "bf16":
        z = z.to(torch.bfloat16).float()
    return lmhead.pick_token(z, torch.arange(VOCAB).expand(x.shape[0], -1), VOCAB)


def agree(what, got, want, x, w, tol=2.0 ** -7, pairs=False):
    """Tokens equal, or, where they differ, a near tie: the float32 sums behind two logits come out in another order on
    the device than in torch (whose own order varies with the host's thread count), so two candidates whose exact
    logits are within `tol` (relative; one bf16 step for rounded logits) may be picked either way. pairs: rows 2i and
    2i + 1 of the head are equal, an exact tie, and of those the lower id must have won."""
    if torch.equal(got, want):
        print(f"ok   {what}: token for token", flush=True)
        return
    z = x.double() @ w.double().T
    for t in range(got.shape[0]):
        a, b = z[t, got[t]].item(), z[t, want[t]].item()
        assert abs(a - b) <= tol * max(abs(a), abs(b)), (what, t, int(got[t]), int(want[t]), a, b)
        assert not pairs or int(got[t]) % 2 == 0, (what, t, int(got[t]))
    print(f"ok   {what}: equal up to near ties", flush=True)


def test_records(device):
    w = head(1)
    rows, k = 3, 8
    x, tx = x_rows(device, rows, 2)
    dh = lmhead.DeviceHead(device, w, fmt="bfp4", chunks=CHUNKS, k=k, rescore=False)
    vals, ids = dh.candidates(tx, rows)
    y = torch.cat([ttnn.to_torch(linear.matmul(tx, tw, None)).float().reshape(-1, dh.step)[:rows] for tw, _ in dh.blocks], 1)
    for t in range(rows):
        ok = ids[t] >= 0
        same(f"records row {t}: values at their ids", y[t][ids[t][ok]], vals[t][ok])
        top = torch.sort(vals[t][ok], descending=True).values[:k]
        same(f"records row {t}: the best {k} of all logits", top, torch.topk(y[t], k).values)
    dh.deallocate()


def test_host_rescore(device):
    w = head(3)
    dh = lmhead.DeviceHead(device, w, fmt="bfp4", chunks=CHUNKS)
    for rows in (1, 5):
        x, tx = x_rows(device, rows, 4 + rows)
        agree(f"host rescore rows {rows}: tokens against the bf16 host head", dh(tx, rows), host_tokens(x, w), x, w)
    dh.deallocate()


@pytest.mark.parametrize("kind,seed,pairs", [("random", 5, False), ("ties", 6, True)])
@pytest.mark.parametrize("logits", ["bf16", "float32"])
def test_device_pick(device, kind, seed, pairs, logits):
    w = head(seed, pairs)
    host = lmhead.DeviceHead(device, w, fmt="bfp4", chunks=CHUNKS, logits=logits)
    dev = lmhead.DeviceHead(device, w, fmt="bfp4", chunks=CHUNKS, logits=logits, device_pick=True)
    for rows in (1, 4):
        x, tx = x_rows(device, rows, 7 + rows)
        want, got = host(tx, rows), dev(tx, rows)
        agree(f"device pick ({kind}, {logits} logits) rows {rows}: tokens against the host rescore", got, want, x, w,
              1e-6 if logits == "float32" else 2.0 ** -7, pairs)
        if kind == "random" and logits == "bf16":
            agree(f"device pick rows {rows}: tokens against the bf16 host head", got, host_tokens(x, w), x, w)
    dev.deallocate()
    host.deallocate()


def test_small_records(device):
    w = head(14)
    for rows in (1, 3):
        x, tx = x_rows(device, rows, 15 + rows)
        host = lmhead.DeviceHead(device, w, fmt="bfp4", chunks=CHUNKS, k=4)
        dev = lmhead.DeviceHead(device, w, fmt="bfp4", chunks=CHUNKS, k=4, device_pick=True)
        agree(f"device pick, k 4, rows {rows}: tokens against the host rescore", dev(tx, rows), host(tx, rows), x, w)
        plain = lmhead.DeviceHead(device, w, fmt="bfp4", chunks=CHUNKS, k=4, rescore=False)
        vals, ids = plain.candidates(tx, rows)
        picked = lmhead.DeviceHead(device, w, fmt="bfp4", chunks=CHUNKS, k=4, rescore=False, device_pick=True)
        best = ids[torch.arange(rows), vals.argmax(dim=1)]
        same(f"records pick, k 4, rows {rows}: rows against the host's argmax over the records", picked(tx, rows), best)
        for h in (host, dev, plain, picked):
            h.deallocate()


def test_padded_head(device):
    w = head(9)
    valid = VOCAB - 3 * 32 - 5  # the last rows are padding: never candidates
    rows, k = 2, 8
    x, tx = x_rows(device, rows, 10)
    dh = lmhead.DeviceHead(device, w, fmt="bfp4", chunks=CHUNKS, k=k, rescore=False)
    r = dh.logits_topk(tx, rows)
    rows_t = head_pick.head_rows(device, w)
    tok, _, _ = head_pick.tokens(head_pick.pick(r, tx, rows_t, rows, k, valid=valid), rows)
    vals, ids = linear.topk_records(r, rows, k)
    vals = torch.where(ids >= valid, torch.full_like(vals, float("-inf")), vals)
    cand = ids.gather(1, vals.topk(16, dim=1).indices)
    z = torch.einsum("rd,rcd->rc", x.float(), w[cand.clamp(min=0).reshape(-1)].float().reshape(rows, 16, DIM))
    z = z.to(torch.bfloat16).float()
    z = torch.where((cand >= 0) & (cand < valid), z, torch.full_like(z, float("-inf")))
    want = lmhead.pick_token(z, cand, VOCAB)
    same(f"padded head (valid {valid}): tokens against the host rescore of the valid candidates", tok, want)
    assert int(tok.max()) < valid
    short = head_pick.head_rows(device, w[:valid])  # a table of the valid rows only serves the padded head
    dv = lmhead.DeviceHead(device, w, fmt="bfp4", chunks=CHUNKS, k=k, device_pick=True, valid=valid, rows=short)
    same(f"padded head (valid {valid}), a table of the valid rows only: tokens", dv(tx, rows), want)
    dv.deallocate()
    ttnn.deallocate(short)
    ttnn.deallocate(rows_t)
    dh.deallocate()


def test_records_pick(device):
    w = head(11)
    rows, k = 3, 8
    g = torch.Generator().manual_seed(12)
    tmap = torch.randperm(1 << 20, generator=g)[:VOCAB]  # row i of the sub-head is token tmap[i]
    x, tx = x_rows(device, rows, 13)
    plain = lmhead.DeviceHead(device, w, fmt="bfp4", chunks=CHUNKS, k=k, rescore=False)
    vals, ids = plain.candidates(tx, rows)
    best = ids[torch.arange(rows), vals.argmax(dim=1)]  # the host's argmax over the same records
    picked = lmhead.DeviceHead(device, w, fmt="bfp4", chunks=CHUNKS, k=k, rescore=False, device_pick=True)
    same("records pick: rows against the host's argmax over the records", picked(tx, rows), best)
    mapped = lmhead.DeviceHead(device, w, fmt="bfp4", chunks=CHUNKS, k=k, rescore=False, device_pick=True,
                               token_map=tmap.tolist())
    same("records pick with a token map: tokens", mapped(tx, rows), tmap[best])
    ids_out = ttnn.from_torch(torch.zeros(1, 1, dtype=torch.int32), dtype=ttnn.uint32, layout=ttnn.ROW_MAJOR_LAYOUT,
                              device=device)
    mapped.logits_topk(tx, rows, ids_out=ids_out)
    assert int(ttnn.to_torch(ids_out).reshape(-1)[0]) == int(tmap[best][0])
    for h in (plain, picked, mapped):
        h.deallocate()


@pytest.mark.parametrize("adjacent", [False, True])
@pytest.mark.parametrize("fmt", ["bfp8", "bfp4"])
@pytest.mark.parametrize("blocks,step,rows,k,unit", [(2, 96, 1, 8, 2048), (5, 2048 + 160, 16, 4, 2048), (17, 288, 5, 8, 128), (4, 2048, 1, 64, 512)])
def test_blocks_together_equal_a_call_each(device, fmt, blocks, step, rows, k, unit, adjacent):
    """The head's blocks in one launch (back to back in memory; else one for four) leave the records that a call for each leaves, bit for bit, and those are
    the canonical top-k of the outputs: blocks that end inside a panel and a unit, one row and more than the four warps that
    merge, lists of one lane and of many, equal logits by the dozen, ids that count from a block's base."""
    g = torch.Generator().manual_seed(blocks + step)
    dim = 256
    w = (torch.randn(blocks * step, dim, generator=g) * 4).round() / 64
    x = (torch.randn(rows, dim, generator=g) * 2).round().to(torch.bfloat16)
    tx = ttnn.from_torch(x.reshape(1, 1, rows, dim), dtype=ttnn.bfloat16, layout=ttnn.TILE_LAYOUT, device=device)
    ws = tuple(linear.native_weight(device, w[i * step : (i + 1) * step], lmhead.FORMATS[fmt])[0] for i in range(blocks))
    if adjacent:
        streams, emaxes = torch.stack([t.t for t in ws]), torch.stack([t.emax for t in ws])
        for i, t in enumerate(ws):
            t.t, t.emax = streams[i], emaxes[i]
        torch.cuda.synchronize()
    was, linear.TOPK_UNIT = linear.TOPK_UNIT, unit
    try:
        units = linear.topk_units(step)
        one, each = (linear.topk_result(device, 1 + blocks * units, rows, k) for _ in range(2))
        y = ttnn.allocate_tensor_on_device([1, 1, rows, step], ttnn.bfloat16, ttnn.TILE_LAYOUT, device)
        spec = {"k": k, "rows": rows, "n": step - 7, "write_y": False}
        for _ in range(2):  # (described, then as kept)
            linear.records_together(tx, ws, {**spec, "r": one, "slot0": 1, "base": 50}, y)
        for b, tw in enumerate(ws):
            linear.matmul(tx, tw, None, out=y, topk={**spec, "r": each, "slot0": 1 + b * units, "base": 50 + b * step})
            out = ttnn.to_torch(linear.matmul(tx, tw, None)).reshape(rows, step)
            rec = ttnn.to_torch(each).reshape(-1, 2, rows, k).numpy().view(np.uint32)
            for u in range(units):
                c0, c1 = u * unit, min((u + 1) * unit, step - 7)
                for r in range(rows):
                    keys, idx = orc.topk_canonical(orc.bf16_bits(out[r, c0:c1].float()), max(0, c1 - c0), k, 50 + b * step + c0)
                    assert np.array_equal(rec[1 + b * units + u, 0, r], keys) and np.array_equal(rec[1 + b * units + u, 1, r], idx), (b, u, r)
    finally:
        linear.TOPK_UNIT = was
    assert torch.equal(ttnn.to_torch(one), ttnn.to_torch(each))
    linear.check_status(device)


@pytest.mark.parametrize("nrec,rows,k,top", [(1, 1, 4, 1), (75, 3, 8, 16), (600, 2, 8, 32), (40, 32, 16, 5)])
def test_pick_takes_the_earliest_of_equal_keys(device, nrec, rows, k, top):
    """The pick's candidates against the host's stable order over records full of equal keys, empty slots and ids past the
    vocabulary, with fewer and more slots than the warps take at a time: the first candidate, the count and the token."""
    gen = np.random.default_rng(nrec + top)
    dim, vocab = 64, nrec * rows * k // 2 + 8
    words = np.zeros((nrec, 2, rows, k), np.uint32)
    words[:, 0] = gen.integers(0x8000, 0x8010, size=(nrec, rows, k))
    words[:, 0][gen.random((nrec, rows, k)) < 0.2] = 0
    words[:, 1] = gen.permutation(nrec * rows * k).reshape(nrec, rows, k)
    r = linear.topk_result(device, nrec, rows, k)
    r.t.copy_(torch.from_numpy(words.view(np.int32)).reshape(r.t.shape))
    g = torch.Generator().manual_seed(nrec)
    table = (torch.randn(vocab, dim, generator=g) * 4).round().to(torch.bfloat16)
    x = (torch.randn(rows, dim, generator=g) * 2).round().to(torch.bfloat16)  # (whole numbers: exact sums, whatever their order)
    tx = ttnn.from_torch(x.reshape(1, 1, rows, dim), dtype=ttnn.bfloat16, layout=ttnn.TILE_LAYOUT, device=device)
    tok, best, count = head_pick.tokens(head_pick.pick(r, tx, head_pick.head_rows(device, table), rows, k, top=top, logits="float32"), rows)
    rtok, _, rcount = head_pick.tokens(head_pick.pick_records(r, rows, k, vocab), rows)
    for t in range(rows):
        keys, ids = words[:, 0, t].reshape(-1).astype(np.int64), words[:, 1, t].reshape(-1).astype(np.int64)
        keys[ids >= vocab] = 0
        order = np.argsort(-keys, kind="stable")
        order = order[keys[order] > 0]
        cand = ids[order][:top]
        z = (x[t].float() @ table[torch.from_numpy(cand)].float().T).numpy()
        want = cand[z == z.max()].min()
        assert (int(tok[t]), int(best[t]), int(count[t])) == (want, cand[0], len(cand)), t
        assert (int(rtok[t]), int(rcount[t])) == (ids[order][0], len(order)), t


@pytest.mark.parametrize("nrec,rows,k,top", [(1, 1, 4, 1), (3, 2, 4, 32), (75, 1, 8, 16), (300, 3, 4, 9), (512, 1, 4, 32), (513, 2, 2, 16), (300, 2, 8, 32),
                                            (180, 2, 4, 9), (181, 2, 4, 9)])
def test_picks_from_records_with_ties_and_holes(device, nrec, rows, k, top):
    """The best slots of arbitrary records (few distinct keys, empty slots, ids past the vocabulary, a record's slots in no order), by
    counting and, past 2048 slots, 512 records or twenty records for each of the top, in rounds: the first candidate and how many are
    held, and the pick among their exact logits, as numpy finds them."""
    g = np.random.default_rng(nrec + k)
    dim, vocab = 64, 4000
    keys = g.integers(0x8000, 0x8000 + 60, (nrec, rows, k)).astype(np.uint32)
    keys[g.random(keys.shape) < 0.2] = 0
    ids = g.integers(0, vocab + 400, (nrec, rows, k)).astype(np.uint32)
    rec = np.stack([keys, ids], axis=1).reshape(1, 1, nrec, 2 * rows * k)
    tr = ttnn.from_torch(torch.from_numpy(rec.view(np.int32)), dtype=ttnn.uint32, layout=ttnn.ROW_MAJOR_LAYOUT, device=device)
    head = torch.from_numpy(g.standard_normal((vocab, dim))).float().bfloat16()
    x = torch.from_numpy(g.standard_normal((rows, dim))).float().bfloat16()
    tx = ttnn.from_torch(x.reshape(1, 1, rows, dim), dtype=ttnn.bfloat16, layout=ttnn.TILE_LAYOUT, device=device)
    exact = x.double() @ head.double().T
    tok, first, count = head_pick.tokens(head_pick.pick(tr, tx, head_pick.head_rows(device, head), rows, k, top=top, logits="float32"), rows)
    best, own, valid = head_pick.tokens(head_pick.pick_records(tr, rows, k, vocab), rows)
    for r in range(rows):
        kk, ii = keys[:, r].reshape(-1).astype(np.int64), ids[:, r].reshape(-1).astype(np.int64)
        ok = (kk > 0) & (ii < vocab)
        order = np.lexsort((np.arange(kk.size), -kk, ~ok))[: min(top, int(ok.sum()))]
        assert int(count[r]) == len(order) and int(valid[r]) == int(ok.sum())
        if len(order):
            assert int(first[r]) == ii[order[0]] == int(own[r]) == int(best[r])
            logits = exact[r, torch.from_numpy(ii[order])]
            assert int(tok[r]) in ii[order] and float(exact[r, int(tok[r])]) >= float(logits.max()) - 1e-4
